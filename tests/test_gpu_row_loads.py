"""Rows of the standalone model and update calls, bit for bit against the oracle.

Rows of up to six coefficients are read directly, longer ones through shared
memory a block at a time; a row may hold fewer coefficients than its band.
"""

import numpy as np
import pytest

import tractography_b200 as tg

from helpers import bits_equal, random_orientations

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
@pytest.mark.parametrize("model,C", [("tensor", 6), ("sh", 1), ("sh", 3), ("sh", 6), ("sh", 7), ("sh", 15), ("sh", 44),
                                     ("sh", 45)])
def test_rows_of_any_length(runtime, oracle, model, C, n):
    rng = np.random.default_rng([C, n])
    rows = (rng.normal(size=(n, C)) * 0.2).astype(np.float32)
    rows[:, 0] = np.abs(rows[:, 0]) + 0.5
    o = random_orientations(rng, n)
    tensor = model == "tensor"
    local = tg.local.DiffusionTensorImaging() if tensor else tg.local.RealSymmetricSphericalHarmonics(C)
    which = oracle.MODEL_DTI if tensor else oracle.MODEL_SH
    assert bits_equal(tg.local.evaluate(local, rows, o, runtime), oracle.local_evaluate(which, rows, o))
    alg = tg.algorithm.Transport(local, step_size=0.05, gamma=1.0)
    case = oracle.Case(model=which, algorithm=oracle.ALGO_TRANSPORT, step_size=0.05, gamma=1.0)
    assert bits_equal(tg.algorithm.update_orientation(alg, rows, o, runtime), case.update_orientation(rows, o))
