"""Blocks given up at the end of a sliced launch, where it is known that they were.

With no more seeds than lanes and more than one layer of blocks, nothing waits
until a block gives up its streamlines: the launch's first handover is one of
those.  Every kind of tracker must hand over, and its results equal the
unsliced run's bit for bit; so must those of waves that share a small pool.
"""

import ctypes

import numpy as np
import pytest

import tractography_b200 as tg
from tractography_b200 import _lib, synthetic

from test_gpu_own_grid import SHAPE, make, own_grid_mask

pytestmark = pytest.mark.gpu


def _handovers(runtime):
    n = ctypes.c_uint32()
    _lib.check(runtime.lib.tg_tracker_handovers(runtime.tracker(), ctypes.byref(n)))
    return n.value


def _problem(kind, n):
    algorithm, lmax = {"sh8": ("diffusion", 8), "own": ("diffusion", 8), "transport": ("transport", 4),
                       "philox": ("philox", 6), "tensor": ("diffusion", -1), "surface": ("transport", -1),
                       "surface_sde": ("diffusion", 8)}[kind]
    field, alg = make(algorithm, lmax, step=0.02)
    if kind.startswith("surface"):
        v, f = synthetic.config2_surface(shape=SHAPE, frequency=12)
        domain, rt = tg.domain.Mesh(v, f), tg.CudaRuntime()
        seeds = synthetic.seeds_inside(lambda p: tg.domain.contains(domain, p, rt), v.min(axis=0), v.max(axis=0), n,
                                       seed=7)
    else:
        mask = own_grid_mask() if kind == "own" else tg.Nifti1Image(np.ones(SHAPE, np.uint8),
                                                                    np.diag([2.0, 2.0, 2.0, 1.0]))
        domain, seeds = tg.domain.Image(mask), synthetic.uniform_seeds(mask, n, seed=7)
    return field, domain, alg, seeds


def _track(runtime, problem, batch=10000, n_steps=1500):
    field, domain, alg, seeds = problem
    return tg.tracking.track_packed(alg(), domain, field, seeds, save_at=0.05, n_steps=n_steps, batch_size=batch,
                                    batch_rng_seeds=np.arange(3, 3 + -(-len(seeds) // batch), dtype=np.uint32),
                                    runtime=runtime, philox_key=11)


@pytest.mark.parametrize("kind", ["sh8", "own", "transport", "philox", "tensor", "surface", "surface_sde"])
def test_every_tracker_hands_over(kind):
    problem = _problem(kind, 40000)          # three layers of blocks
    plain_rt = tg.CudaRuntime()
    plain_rt.set_slicing(0)
    plain = _track(plain_rt, problem)
    assert _handovers(plain_rt) == 0
    rt = tg.CudaRuntime()
    rt.set_slicing(2048)
    sliced = _track(rt, problem)
    assert _handovers(rt) > 0
    assert np.array_equal(plain.lengths, sliced.lengths) and plain.steps == sliced.steps
    assert np.array_equal(plain.points, sliced.points)


@pytest.mark.parametrize("kind", ["sh8", "surface"])
def test_waves_of_a_small_pool_hand_over(kind):
    problem = _problem(kind, 40000)
    plain_rt = tg.CudaRuntime()
    plain_rt.set_slicing(0)
    plain = _track(plain_rt, problem)
    rt = tg.CudaRuntime(pool_points=int(plain.lengths.sum() * 0.6) + 40000 * 32)
    rt.set_slicing(2048)
    waved = _track(rt, problem)
    kms, waves, launches = ctypes.c_float(), ctypes.c_uint32(), ctypes.c_uint32()
    _lib.check(rt.lib.tg_tracker_stats(rt.tracker(), ctypes.byref(kms), ctypes.byref(waves), ctypes.byref(launches)))
    assert waves.value > 1
    assert np.array_equal(plain.lengths, waved.lengths)
    for i in range(0, len(plain.lengths), 37):
        a, b = plain.offsets[i], waved.offsets[i]
        assert np.array_equal(plain.points[a: a + plain.lengths[i]], waved.points[b: b + plain.lengths[i]]), i
