"""Seed counts at the edges of the launch's spread over warps (spread_lanes).

A launch that does not fill the GPU uses as few warps per scheduler as hold
its streamlines, and as few lanes of each as those warps then need; a launch
of one streamline more than the lanes refills.  Whatever the shape, every
seed is tracked once: results equal the oracle's bit for bit, alone and
split over the jobs of one run.
"""

import numpy as np
import pytest

import tractography_b200 as tg
from tractography_b200 import jobs as jobs_module

from helpers import bits_equal, oracle_case, small_config0

pytestmark = pytest.mark.gpu

ROUND = 148 * 4                       # warps of one block per SM
SIZES = [1, ROUND - 1, ROUND + 1, 32 * ROUND, 32 * ROUND + 1, 32 * ROUND * 5 + 1]


@pytest.mark.parametrize("n", SIZES)
def test_any_seed_count_equals_the_oracle(n):
    field, domain, seeds = small_config0(n_voxels=16, n_seeds=n, seed=5)
    alg = tg.algorithm.Diffusion(tg.local.RealSymmetricSphericalHarmonics(45), step_size=0.2, gamma=1.0,
                                 noise_variance=0.1, seed=1)
    runtime = tg.CudaRuntime()
    n_steps, stream = 6, 77
    want, lengths = oracle_case(alg, domain, field, rng_seed=stream, save_at=0.25, n_steps=n_steps).tractogram(
        seeds, n_threads=8)
    kept = np.concatenate([w[:m, :3] for w, m in zip(want, lengths)])
    res = tg.tracking.track_packed(alg, domain, field, seeds, save_at=0.25, n_steps=n_steps, batch_size=n,
                                   batch_rng_seeds=[stream], runtime=runtime)
    assert np.array_equal(res.lengths, lengths)
    assert bits_equal(res.points, kept)
    # the same seeds as jobs of one run, cut at a warp's worth (stream ids restart per job: Transport draws none)
    transport = tg.algorithm.Transport(alg.local_model, step_size=0.2, gamma=1.0)
    want, lengths = oracle_case(transport, domain, field, save_at=0.25, n_steps=n_steps).tractogram(seeds, n_threads=8)
    parts = [p for p in (seeds[:33], seeds[33:]) if len(p)]
    jobs = [jobs_module.Job(field=field, domain=domain, algorithm=transport, seeds=p, save_at=0.25, n_steps=n_steps,
                            min_points=0, batch_size=len(p), batch_rng_seeds=np.zeros(1, np.uint32)) for p in parts]
    both = jobs_module.run_jobs_packed(jobs, runtime)
    assert np.array_equal(both.lengths, lengths)
    assert bits_equal(both.points, np.concatenate([w[:m, :3] for w, m in zip(want, lengths)]))
