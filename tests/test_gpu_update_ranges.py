"""The update's device forms against the oracle over the whole binary32 range.

On the device the step's reciprocal, Box-Muller's square roots and its pair
of normals are written differently from the shared math layer (a Newton step
on the hardware's estimates, two values per instruction), and a reciprocal
above 2^125 takes the division.  Coefficients from 1e-38 to the largest
floats, infinities and NaN reach every side of those rules; results equal the
oracle's bit for bit.
"""

import numpy as np
import pytest

import tractography_b200 as tg

from helpers import bits_equal, random_orientations

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rng_mode", ["mwc64x", "philox"])
@pytest.mark.parametrize("C", [1, 6, 15, 45])
def test_updates_of_any_magnitude_equal_the_oracle(oracle, C, rng_mode):
    rng = np.random.default_rng(C)
    n = 20011
    rows = rng.normal(size=(n, C)).astype(np.float32)
    rows *= (10.0 ** rng.uniform(-38, 37.9, (n, 1))).astype(np.float32)
    rows[:6] = 0.0
    rows[6:12] = np.finfo(np.float32).max
    rows[12:14, 0], rows[14:16, -1], rows[16:18, 0] = np.inf, -np.inf, np.nan
    rows[18:40, 0] = np.float32(2.0) ** np.arange(116, 138).clip(max=127).astype(np.float32)
    o = random_orientations(rng, n)
    dti = C == 6
    model = tg.local.DiffusionTensorImaging() if dti else tg.local.RealSymmetricSphericalHarmonics(C)
    alg = tg.algorithm.Diffusion(model, step_size=0.01, gamma=1.0, noise_variance=0.2, seed=4, rng=rng_mode)
    twin = tg.algorithm.Diffusion(model, step_size=0.01, gamma=1.0, noise_variance=0.2, seed=4, rng=rng_mode)
    with np.errstate(all="ignore"):
        got = tg.algorithm.update_orientation(alg, rows, o)
        stream = twin.get_rng_seed()
        key = twin.philox_key() if rng_mode == "philox" else 0
        case = oracle.Case(model=oracle.MODEL_DTI if dti else oracle.MODEL_SH, algorithm=oracle.ALGO_DIFFUSION,
                           step_size=0.01, gamma=1.0, noise_variance=0.2, rng_mode=alg.rng_mode(), rng_seed=stream,
                           philox_key=key)
        assert bits_equal(got, case.update_orientation(rows, o))
        assert bits_equal(tg.local.evaluate(model, rows, o),
                          oracle.local_evaluate(oracle.MODEL_DTI if dti else oracle.MODEL_SH, rows, o))
