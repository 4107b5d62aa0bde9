"""Sparse warps merging at the end of a sliced launch.

Once the seeds are taken, warps with few live lanes save their streamlines and
leave, and warps with idle lanes take them.  Every streamline must still be tracked
once and to the end: results equal the unsliced run's bit for bit, whether the
launch starts with full warps, with a part of each warp, or with queued seeds.
"""

import numpy as np
import pytest

import tractography_b200 as tg

from helpers import small_config0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["diffusion", "philox", "transport"])
@pytest.mark.parametrize("n", [700, 25000, 94720, 130000])
def test_merged_runs_equal_the_unsliced_run(kind, n):
    field, domain, seeds = small_config0(n_voxels=16, n_seeds=n, seed=2)
    model = tg.local.RealSymmetricSphericalHarmonics(45)
    out = []
    for steps in (0, 4096):
        if kind == "transport":
            alg = tg.algorithm.Transport(model, step_size=0.02, gamma=1.0)
        else:
            alg = tg.algorithm.Diffusion(model, step_size=0.02, gamma=1.0, noise_variance=0.2, seed=3,
                                         rng="philox" if kind == "philox" else "mwc64x")
        runtime = tg.CudaRuntime()
        runtime.set_slicing(steps)
        for _ in range(2 if steps else 1):        # the merge order differs from run to run
            out.append(tg.tracking.track_packed(alg, domain, field, seeds, save_at=0.05, n_steps=2000, batch_size=n,
                                                batch_rng_seeds=[9], runtime=runtime, philox_key=5))
    plain = out[0]
    for sliced in out[1:]:
        assert np.array_equal(plain.lengths, sliced.lengths)
        assert plain.steps == sliced.steps
        assert np.array_equal(plain.points, sliced.points)
