"""tg_tractogram_noalloc's forms: one streamline per lane, and lanes that take more.

With at most as many seeds as the GPU has lanes each lane tracks one by itself;
with more, lanes take the next seed when theirs ends, joined with their warp or
by themselves.  Every form equals the tracker's own run bit for bit, at one seed,
on either side of a warp per scheduler and with more seeds than lanes.
"""

import numpy as np
import pytest

import tractography_b200 as tg
from tractography_b200 import synthetic

from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,lmax", [("transport", 8), ("transport", 4), ("diffusion", 8), ("philox", 2)])
@pytest.mark.parametrize("n", [1, 18944, 18945, 100003, 300007])
def test_forms_equal_the_tracker(runtime, kind, lmax, n):
    shape = (20, 20, 20)
    mask = tg.Nifti1Image(np.ones(shape, np.uint8), np.diag([2.0, 2.0, 2.0, 1.0]))
    field = tg.field.Image(synthetic.bundle_field(shape, lmax=lmax, seed=1)[0])
    domain = tg.domain.Image(mask)
    model = tg.local.RealSymmetricSphericalHarmonics((lmax + 1) * (lmax + 2) // 2)
    if kind == "transport":
        alg = tg.algorithm.Transport(model, step_size=0.2, gamma=1.0)
    else:
        alg = tg.algorithm.Diffusion(model, step_size=0.05, gamma=1.0, noise_variance=0.2, seed=3,
                                     rng="philox" if kind == "philox" else "mwc64x")
    seeds = synthetic.uniform_seeds(mask, n, seed=4)
    batches = np.arange(5, 5 + (n + 49999) // 50000, dtype=np.uint32)
    save_at, n_steps = 1.0, 8
    out, lengths = _noalloc(runtime, alg, domain, field, seeds, 50000, batches, save_at, n_steps)
    want = tg.tracking.track_packed(alg, domain, field, seeds, save_at=save_at, n_steps=n_steps, batch_size=50000,
                                    batch_rng_seeds=batches, runtime=runtime)
    assert np.array_equal(lengths, want.lengths)
    kept = out[..., :3][np.arange(n_steps)[None] < lengths[:, None]]
    order = np.argsort(want.offsets, kind="stable")
    assert np.array_equal(order, np.arange(n))
    assert np.array_equal(kept, want.points)
