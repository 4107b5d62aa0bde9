"""FOD seeding at the edges of its launch forms, against the oracle.

One seed per thread up to two warps per scheduler, two beyond; directions in
tiles of 16 with a shorter last one; the last block's threads repeat the last
seed.  Coefficients that overflow or are not numbers select no direction, as in
the oracle.
"""

import numpy as np
import pytest

import tractography_b200 as tg
from tractography_b200 import seeds as S

from helpers import bits_equal

pytestmark = pytest.mark.gpu

EDGE = 148 * 128 * 2


@pytest.mark.parametrize("n", [1, 128, 129, EDGE, EDGE + 1, EDGE + 257])
@pytest.mark.parametrize("C", [1, 6, 15, 28, 45])
def test_any_seed_count_equals_the_oracle(oracle, C, n):
    rng = np.random.default_rng(100 * C + n)
    tensor = C == 6
    nnz = 400
    fod = (rng.normal(size=(nnz, C)) * 0.1).astype(np.float32)
    fod[:, 0] += 0.3
    if tensor:
        fod[:, :3] = np.abs(fod[:, :3]) + 0.1
    fod[0], fod[1], fod[2], fod[3] = np.nan, np.inf, 3e38, -3e38
    fod[4], fod[5] = 0.0, -5.0
    voxels = np.hstack([rng.integers(0, 9, (nnz, 3)), np.ones((nnz, 1))]).astype(np.float32)
    affine = np.array([[2, 0.1, 0, -4], [0, 1.5, 0.2, 3], [0.1, 0, 2.5, 1], [0, 0, 0, 1]], np.float32)
    states = rng.integers(1, 4294967295, (n, 2), dtype=np.uint32)
    mid = oracle.MODEL_DTI if tensor else oracle.MODEL_SH
    got = S.seeds_from_sparse_fod(mid, fod, voxels, affine, states, tg.CudaRuntime())
    sample = np.unique(np.concatenate([np.arange(min(n, 600)), np.arange(max(0, n - 600), n),
                                       rng.integers(0, n, 600)]))
    with np.errstate(all="ignore"):
        want = oracle.seeds_from_fod(mid, fod, voxels, affine, states[sample])
    assert bits_equal(got[sample], want)
