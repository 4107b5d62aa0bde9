"""Points next to a voxel's faces, mask and field on one grid, bit for bit.

The tracker keeps the last voxel while the point stays within half a voxel of
its centre.  The mask's voxel is floor(fl(a + 0.5)), and for a = 0.5 - 2^-25 the
binary32 sum is 1: the point lies in mask voxel 1 and field voxel 0, whether a
streamline steps there out of voxel 0 or starts there.
"""

import numpy as np
import pytest

import tractography_b200 as tg

from helpers import bits_equal, oracle_case

pytestmark = pytest.mark.gpu

HALF = np.float32(0.5)
STEPS = [np.float32(0.25) - np.float32(2.0 ** -25), np.float32(0.25), np.float32(0.25) + np.float32(2.0 ** -24)]


@pytest.mark.parametrize("step", STEPS, ids=["below", "on", "above"])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_streamlines_that_meet_a_face(runtime, axis, step):
    shape = (4, 4, 4)
    mask = np.ones(shape, np.uint8)
    for edge in ((1,), (0, 2), (0, 1, 3), (3,)):
        mask[:] = 1
        mask[tuple(list(edge) if a == axis else slice(None) for a in range(3))] = 0
        field = tg.field.Image(tg.Nifti1Image(np.ones(shape + (1,), np.float32), np.eye(4)))
        domain = tg.domain.Image(tg.Nifti1Image(mask, np.eye(4)))
        alg = tg.algorithm.Transport(tg.local.RealSymmetricSphericalHarmonics(1), step_size=float(step), gamma=1.0)
        # along the axis, both ways, from quarter positions and from either side of each face
        at = np.array([b + d for b in range(4) for d in (-0.25, 0.0, 0.25)] +
                      [np.nextafter(HALF + b, np.float32(t)) for b in range(-1, 4) for t in (-9, 9)] +
                      [HALF + b for b in range(-1, 4)], np.float32)
        seeds = np.zeros((2 * len(at), 8), np.float32)
        seeds[:, :3], seeds[:, 3] = 1.0, 1.0
        seeds[:, axis] = np.tile(at, 2)
        seeds[:, 4 + axis] = np.repeat([1.0, -1.0], len(at))
        case = oracle_case(alg, domain, field, save_at=0.2, n_steps=30)
        want, want_len = case.tractogram(seeds)
        dense, lengths = tg.tracking.tractogram_dense(alg, domain, field, seeds, save_at=0.2,
                                                      maximum_streamline_length=6.1, runtime=runtime)
        assert np.array_equal(lengths, want_len)
        res = tg.tracking.track_packed(alg, domain, field, seeds, save_at=0.2, n_steps=30, batch_size=len(seeds),
                                       batch_rng_seeds=[0], runtime=runtime)
        assert np.array_equal(res.lengths, want_len)
        for i in range(len(seeds)):
            assert bits_equal(dense[i, : lengths[i]], want[i, : want_len[i]]), i
            assert bits_equal(res.points[res.offsets[i]: res.offsets[i] + res.lengths[i]], want[i, : want_len[i], :3]), i
