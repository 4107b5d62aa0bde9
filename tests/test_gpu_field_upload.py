"""Field creation: coefficients padded and folded on the device, every row length.

A field's coefficients go up packed and are padded to float4 rows there; rows
that are whole float4s already go up in place.  Each length must evaluate to
the coefficients it was made from.
"""

import numpy as np
import pytest

import tractography_b200 as tg
from tractography_b200 import local, tracking

from helpers import bits_equal, oracle_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,C", [("sh", c) for c in (1, 2, 3, 4, 5, 6, 8, 15, 16, 27, 28, 44, 45)] + [("dti", 6)])
def test_field_rows_of_any_length(runtime, model, C):
    rng = np.random.default_rng(C)
    shape = (5, 7, 3)
    values = rng.normal(size=shape + (C,)).astype(np.float32) * 0.1
    values[..., 0] += 0.5
    if model == "dti":
        values[..., :3] += 1.0
    field = tg.field.Image(tg.Nifti1Image(values, np.eye(4)))
    m = local.DiffusionTensorImaging() if model == "dti" else local.RealSymmetricSphericalHarmonics(C)
    field.device(runtime, local.model_id(m))
    points = rng.uniform(-1, 7, (400, 3)).astype(np.float32)
    if model == "sh":
        assert bits_equal(tg.field.evaluate(field, points, runtime), field.evaluate(points))
    # and the trackers' copy: one step from every voxel
    domain = tg.domain.Image(tg.Nifti1Image(np.ones(shape, np.uint8), np.eye(4)))
    seeds = np.zeros((105, 8), np.float32)
    seeds[:, :3] = np.argwhere(np.ones(shape))
    seeds[:, 3] = 1.0
    o = rng.normal(size=(105, 3))
    seeds[:, 4:7] = o / np.linalg.norm(o, axis=1, keepdims=True)
    alg = tg.algorithm.Transport(m, step_size=0.2, gamma=1.0)
    res = tracking.track_packed(alg, domain, field, seeds, save_at=0.2, n_steps=4, batch_size=105, batch_rng_seeds=[0],
                                runtime=runtime)
    want, lengths = oracle_case(alg, domain, field, save_at=0.2, n_steps=4).tractogram(seeds)
    assert np.array_equal(res.lengths, lengths)
    assert bits_equal(res.points, np.concatenate([w[:k, :3] for w, k in zip(want, lengths)]))
