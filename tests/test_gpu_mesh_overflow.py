"""Segments whose extent overflows binary32, against the oracle, bit for bit.

End minus start rounds to infinity, its reciprocal to zero, and where only one
bound of a box lies more than the largest float from the start, that bound's
slab value alone is NaN (infinity times zero): the reference's comparisons
skip it and keep the other bound's.
"""

import numpy as np
import pytest

import tractography_b200 as tg
from oracle import oracle as O
from tractography_b200 import synthetic

from helpers import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("infinite_axes", [1, 2, 3])
def test_segments_that_overflow(runtime, infinite_axes):
    v, f = synthetic.geodesic_sphere(5)
    mesh, bvh = tg.domain.Mesh(v * 1e38, f), O.BoundaryBvh.build(v * 1e38, f)
    rng = np.random.default_rng(infinite_axes)
    n = 4000
    starts = rng.uniform(-1.2e38, 1.2e38, (n, 3))
    ends = starts + rng.normal(0, 3e37, (n, 3))
    far = np.argsort(rng.random((n, 3)), axis=1) < infinite_axes
    side = rng.choice([-1.0, 1.0], (n, 3))
    starts = np.where(far, side * rng.uniform(2.3e38, 3.3e38, (n, 3)), starts).astype(np.float32)
    ends = np.where(far, -side * rng.uniform(1.5e38, 3.3e38, (n, 3)), ends).astype(np.float32)
    with np.errstate(over="ignore"):
        assert np.array_equal(np.isinf(ends - starts), far)
    found, tri, hit = mesh.segment_hits(starts, ends, runtime)
    want = bvh.segment_hits(starts, ends, n_threads=8)
    assert np.array_equal(found, want[0]) and np.array_equal(tri, want[1])
    assert bits_equal(hit, want[2])
    assert np.array_equal(mesh.segments_blocked(starts, ends, runtime), want[0])
