"""Edges of the surface kernels' forms against the oracle, bit for bit.

The box test has a branch-free form for segments with no parallel axis and
the reference's for the rest (a component below 1e-12), reciprocals are a
Newton step inside 2^-125 .. 2^125 and a division outside, and the inside
test's lanes go through several points each when there are more points than
lanes.
"""

import numpy as np
import pytest

import tractography_b200 as tg
from oracle import oracle as O
from tractography_b200 import synthetic

from helpers import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("component", [0.0, -0.0, 1e-45, 9e-13, 1.1e-12, 1e-6, 1e20, 3e38])
def test_segments_with_extreme_components(runtime, component):
    v, f = synthetic.geodesic_sphere(5)
    mesh, bvh = tg.domain.Mesh(v * 8.0, f), O.BoundaryBvh.build(v * 8.0, f)
    rng = np.random.default_rng(3)
    n = 1500
    starts = rng.uniform(-9, 9, (n, 3)).astype(np.float32)
    ends = starts + rng.normal(0, 6, (n, 3)).astype(np.float32)
    axis = np.arange(n) % 3
    starts[np.arange(n), axis] = 0.0 if abs(component) < 1e-3 else starts[np.arange(n), axis]
    ends[np.arange(n), axis] = starts[np.arange(n), axis] + np.float32(component)
    found, tri, hit = mesh.segment_hits(starts, ends, runtime)
    want = bvh.segment_hits(starts, ends, n_threads=8)
    assert np.array_equal(found, want[0]) and np.array_equal(tri, want[1])
    assert bits_equal(hit, want[2])
    assert np.array_equal(mesh.segments_blocked(starts, ends, runtime), want[0])


@pytest.mark.parametrize("n", [1, 127, 129, 400003])
def test_inside_test_of_any_number_of_points(runtime, n):
    v, f = synthetic.geodesic_sphere(4)
    mesh, bvh = tg.domain.Mesh(v * 8.0, f), O.BoundaryBvh.build(v * 8.0, f)
    points = np.random.default_rng(n).uniform(-9, 9, (n, 3)).astype(np.float32)
    points[n // 2:: 7] *= np.nan
    got = tg.domain.contains(mesh, points, runtime)
    sample = np.unique(np.linspace(0, n - 1, 5000).astype(int))
    assert np.array_equal(got[sample], bvh.contains(points[sample]))
