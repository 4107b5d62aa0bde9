"""Masks on a grid of their own: other voxels, another extent, an oblique affine.

Every tracker has one form for a mask on the field's grid and one for any other;
the second keeps the mask's and the field's voxel apart.  Bit for bit against the
oracle through each entry point, and jobs and requests of both forms together.
"""

import numpy as np
import pytest

import tractography_b200 as tg
from tractography_b200 import jobs as jobs_module
from tractography_b200 import synthetic
from tractography_b200.serve import Server

from helpers import bits_equal, oracle_case
from test_gpu_connectome import _device_contributions
from test_gpu_tod import _compare
from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu

SHAPE = (14, 16, 12)


def own_grid_mask(shape=SHAPE, voxel=2.0):
    """An ellipsoid of the field's volume with a hole, in 1.4 mm voxels turned about
    an oblique axis."""
    a, b = 0.3, -0.2
    turn = np.array([[np.cos(a), -np.sin(a), 0], [np.sin(a), np.cos(a), 0], [0, 0, 1]]) @ \
        np.array([[1, 0, 0], [0, np.cos(b), -np.sin(b)], [0, np.sin(b), np.cos(b)]])
    n = np.array([27, 29, 25])
    centre = (np.array(shape) - 1) * voxel / 2
    affine = np.eye(4)
    affine[:3, :3] = turn * 1.4
    affine[:3, 3] = centre - affine[:3, :3] @ ((n - 1) / 2)
    at = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1) @ affine[:3, :3].T + affine[:3, 3]
    r = np.linalg.norm((at - centre) / (0.45 * voxel * np.array(shape)), axis=-1)
    hole = np.linalg.norm(at - centre - [3.0, 0, 0], axis=-1) < 2.0
    return tg.Nifti1Image(((r < 1) & ~hole).astype(np.uint8), affine)


def make(kind, lmax, step=0.2):
    if lmax < 0:
        fod, model = synthetic.dti_field(SHAPE, seed=3), tg.local.DiffusionTensorImaging()
    else:
        fod = synthetic.bundle_field(SHAPE, lmax=lmax, seed=3)[0]
        model = tg.local.RealSymmetricSphericalHarmonics((lmax + 1) * (lmax + 2) // 2)
    if kind == "transport":
        alg = lambda: tg.algorithm.Transport(model, step_size=step, gamma=1.0)                        # noqa: E731
    else:
        alg = lambda: tg.algorithm.Diffusion(model, step_size=step, gamma=1.0, noise_variance=0.15, seed=5,  # noqa: E731
                                             rng="philox" if kind == "philox" else "mwc64x")
    return tg.field.Image(fod), alg


CASES = [("transport", 8), ("diffusion", 8), ("philox", 6), ("diffusion", 4), ("transport", 2), ("transport", 0),
         ("transport", -1), ("diffusion", -1)]


@pytest.mark.parametrize("kind,lmax", CASES)
def test_trackers(kind, lmax):
    field, alg = make(kind, lmax)
    mask = own_grid_mask()
    domain = tg.domain.Image(mask)
    n, batch, save_at, n_steps, key = 1500, 700, 0.25, 60, 77
    seeds = synthetic.uniform_seeds(mask, n, seed=6)
    batches = np.array([31, 32, 33], np.uint32)
    want, lengths = [], []
    for b, r in enumerate(batches):
        w, l = oracle_case(alg(), domain, field, rng_seed=int(r), save_at=save_at, n_steps=n_steps, philox_key=key,
                           seed_offset=b * batch).tractogram(seeds[b * batch:(b + 1) * batch], n_threads=8)
        want.append(w)
        lengths.append(l)
    want, lengths = np.concatenate(want), np.concatenate(lengths)
    assert len(np.unique(lengths)) > 10
    kept = want[..., :3][np.arange(n_steps)[None] < lengths[:, None]]
    for slice_steps in (0, 16):
        runtime = tg.CudaRuntime()
        runtime.set_slicing(slice_steps)
        res = tg.tracking.track_packed(alg(), domain, field, seeds, save_at=save_at, n_steps=n_steps, batch_size=batch,
                                       batch_rng_seeds=batches, runtime=runtime, philox_key=key)
        assert np.array_equal(res.lengths, lengths)
        assert bits_equal(res.points, kept)
    dense, dense_lengths = tg.tracking.tractogram_dense(alg(), domain, field, seeds[:batch], save_at=save_at,
                                                        maximum_streamline_length=n_steps * save_at, runtime=runtime,
                                                        rng_seed=int(batches[0]), philox_key=key)
    assert np.array_equal(dense_lengths, lengths[:batch])
    held = np.arange(n_steps)[None] < dense_lengths[:, None]
    assert bits_equal(dense[held], want[:batch][held])
    if kind != "philox" and lmax >= 0:
        out, out_lengths = _noalloc(runtime, alg(), domain, field, seeds, batch, batches, save_at, n_steps)
        assert np.array_equal(out_lengths, lengths)
        assert bits_equal(out[..., :3][np.arange(n_steps)[None] < lengths[:, None]], kept)


@pytest.mark.parametrize("kind,lmax", [("transport", 8), ("diffusion", 4), ("diffusion", -1)])
def test_tod_and_connectome(runtime, kind, lmax):
    from oracle import oracle as O

    field, alg = make(kind, lmax, step=0.1)
    domain = tg.domain.Image(own_grid_mask())
    grid = tg.Nifti1Image(np.zeros(SHAPE), np.diag([2.0, 2.0, 2.0, 1.0]))
    got = tg.tracking.tod(alg(), domain, field, grid, 2000, maximum_streamline_length=8.0, runtime=runtime)
    twin = alg()
    raw = oracle_case(twin, domain, field, rng_seed=twin.get_rng_seed()).tod(
        domain.boundary_arrays(), 2000, 80, SHAPE, np.linalg.inv(grid.affine))
    _compare(np.asarray(got.dataobj), tg.utils.normalize_odf(raw))
    got = _device_contributions(alg(), domain, field, 3000, 100, 0.5, runtime, 99)
    boundary = domain.boundary_bvh()
    want = oracle_case(alg(), domain, field, rng_seed=99).connectome(
        O.BoundaryBvh.build(boundary.vertices, boundary.faces), domain.boundary_arrays(), 3000, 100, 0.5)
    valid = want[0] >= 0
    assert valid.any() and np.array_equal(got[0], want[0]) and np.array_equal(got[1][valid], want[1][valid])
    assert np.array_equal(got[2][valid].view(np.uint32), want[2][valid].view(np.uint32))


def test_both_forms_in_one_run_and_one_server(runtime):
    masks = {"own": own_grid_mask(), "field": None}
    jobs = []
    for k, (kind, lmax) in enumerate([("transport", 8), ("diffusion", 8), ("diffusion", 4), ("transport", -1)]):
        for form in masks:
            field, alg = make(kind, lmax)
            mask = masks[form] or tg.Nifti1Image(np.ones(SHAPE, np.uint8), np.diag([2.0, 2.0, 2.0, 1.0]))
            jobs.append(jobs_module.prepare(field, synthetic.uniform_seeds(mask, 300 + 50 * k, seed=k),
                                            tg.domain.Image(mask), alg(), save_at=0.25, maximum_streamline_length=15.0,
                                            batch_size=200))
    want = []
    for job in jobs:
        rows = []
        for b, r in enumerate(job.batch_rng_seeds):
            w, l = oracle_case(job.algorithm, job.domain, job.field, rng_seed=int(r), save_at=0.25,
                               n_steps=job.n_steps).tractogram(job.seeds[200 * b: 200 * (b + 1)], n_threads=8)
            rows += [w[i, : l[i], :3] for i in range(len(l))]
        want.append(rows)
    together = jobs_module.run_jobs_packed(jobs, runtime)
    with Server(runtime, hbm_budget_bytes=8e9, epoch_steps=64, reserve_bytes=int(1e9)) as server:
        ids = [server.submit(job) for job in jobs]
        done = {}
        while len(done) < len(ids):
            for rid in server.poll():
                done[rid] = server.take(rid)
    for j, rows in enumerate(want):
        r = together.job(j)
        points, offsets, lengths, _ = done[ids[j]]
        for i, row in enumerate(rows):
            assert bits_equal(r.points[r.offsets[i]: r.offsets[i] + r.lengths[i]], row), (j, i)
            assert bits_equal(points[offsets[i]: offsets[i] + lengths[i]], row), (j, i)
