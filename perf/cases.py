"""Cases that time the framework through its public entry points.

Each case is one call that a user's program makes, on synthetic data of the
generators in ``tractography_b200.synthetic``: tracking one set of seeds
(``tractogram``), several jobs at once (``jobs.run_jobs``), requests through the
continuous-batching server, the track orientation distribution, the boundary
connectome, seeding from a FOD, and the standalone model and orientation
updates.  Fields, domains, surfaces and seeds are in hand before the call, as in
a program that tracks several times in one volume.  Results come back to the host
(``tractogram`` and the rest of the Python calls), or stay on the device with the
seeds that were there (``resident``: the C ABI's tracker, for a program that goes
on working on the GPU).  Points are handed on in a device buffer that holds the
most a case can give, zero beyond its streamlines.
"""

from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import tractography_b200 as tg
from tractography_b200 import _lib, jobs, local, nifti, seeds, serve, synthetic, tracking

VOXEL_MM = 2.0

# Mean streamline lengths, as measured (only the counts of `work` depend on them):
# SDE streamlines and those stopped by a surface cover about this share of the
# volume's mean extent, Transport streamlines in a mask this share of the maximum.
MEAN_EXTENT = 0.45
MEAN_TRANSPORT = 0.8


def listed():
    return [
        # A preview while parameters are chosen: few seeds, where the call's fixed costs count.
        dict(name="track_preview", kind="track", shape="32x32x32", lmax=8, domain="image", n=1000,
             algorithm="transport", rng="mwc64x", step=0.2, save_at=0.25, max_mm=300.0, batch=50000, resident=False),
        # The smallest whole job of the benchmark: 10,000 Transport seeds in a 32^3 volume.
        dict(name="track_transport_10k", kind="track", shape="32x32x32", lmax=8, domain="image", n=10000,
             algorithm="transport", rng="mwc64x", step=0.2, save_at=0.25, max_mm=300.0, batch=50000, resident=False),
        # A slab of the headline job: the SDE at its default step in a whole-brain volume, two batches.
        dict(name="track_diffusion_brain", kind="track", shape="145x174x145", lmax=8, domain="image", n=100000,
             algorithm="diffusion", rng="mwc64x", step=0.001, save_at=0.25, max_mm=300.0, batch=50000, resident=False),
        # A coarse SDE run with the counter-based streams, odd seed count, ragged last batch, kept on the device.
        dict(name="track_diffusion_philox", kind="track", shape="64x64x64", lmax=6, domain="image", n=30011,
             algorithm="diffusion", rng="philox", step=0.05, save_at=1.0, max_mm=200.0, batch=7000, resident=True),
        # A whole-volume tractogram with default spacing: many seeds, long packed output, kept on the device.
        dict(name="track_transport_200k", kind="track", shape="96x96x60", lmax=8, domain="image", n=200000,
             algorithm="transport", rng="mwc64x", step=0.2, save_at=1.0, max_mm=300.0, batch=50000, resident=True),
        # Tensors inside a closed triangle surface (499,280 triangles) instead of a mask, points kept on the device.
        dict(name="track_tensor_surface", kind="track", shape="96x96x60", lmax=-1, domain="surface158", n=500000,
             algorithm="transport", rng="mwc64x", step=0.2, save_at=1.0, max_mm=300.0, batch=50000, resident=True),
        # Uneven jobs of a cohort tracked together: sizes, bands, algorithms and lengths drawn per job.
        dict(name="jobs_uneven", kind="jobs", shape="64x64x64", n=300000, jobs=16, step=0.2, save_at=1.0),
        # A burst of requests to the continuous-batching server.
        dict(name="serve_burst", kind="serve", shape="64x64x64", n=100000, jobs=12, step=0.2, save_at=1.0),
        # Track orientation distribution at the reference's default step, seeds on the mask's boundary.
        dict(name="tod", kind="tod", shape="96x96x60", lmax=8, n=40000, algorithm="transport", step=0.001,
             max_mm=60.0),
        # Boundary connectome, the SDE at its default step.
        dict(name="connectome", kind="connectome", shape="96x96x60", lmax=8, n=40000, algorithm="diffusion",
             step=0.001, max_mm=60.0),
        # Seeds importance-sampled from a FOD already reduced to its nonzero voxels.
        dict(name="seed_fod", kind="seed_fod", shape="64x64x64", lmax=8, n=100000),
        # The standalone entry points: model values and one SDE update per row.
        dict(name="update_rows", kind="update", shape="32x32x32", lmax=8, n=20000, algorithm="diffusion", step=0.001),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    shape = rng.choice(["32x32x32", "41x37x45", "64x64x64", "96x96x60"])
    algorithm = rng.choice(["transport", "diffusion"])
    kind = rng.choice(["track", "track", "track", "track", "jobs", "serve", "tod", "connectome", "seed_fod", "update"])
    if kind == "track":
        step = rng.choice([0.2, 0.1, 0.05, 0.01])
        surface = rng.random() < 0.3
        return dict(kind=kind, shape=shape, lmax=rng.choice([-1, 4, 6, 8]) if surface else rng.choice([-1, 2, 4, 6, 8, 8]),
                    domain="surface%d" % spread(20, 158) if surface else "image",
                    n=spread(300, 200000 if step >= 0.05 else 40000), algorithm=algorithm,
                    rng=rng.choice(["mwc64x", "philox"]), step=step, save_at=rng.choice([0.25, 0.5, 1.0]),
                    max_mm=round(rng.uniform(50.0, 150.0), 1), batch=rng.choice([50000, 7000, 999]),
                    resident=rng.random() < 0.5)
    if kind in ("jobs", "serve"):
        return dict(kind=kind, shape=rng.choice(["41x37x45", "64x64x64"]),
                    n=spread(2000, 300000 if kind == "jobs" else 100000), jobs=rng.randint(2, 20), step=0.2,
                    save_at=rng.choice([0.5, 1.0]))
    if kind in ("tod", "connectome"):
        step = rng.choice([0.2, 0.05, 0.01, 0.001])
        return dict(kind=kind, shape=shape, lmax=rng.choice([-1, 4, 8, 8]), n=spread(500, 40000),
                    algorithm=algorithm, step=step, max_mm=round(rng.uniform(20.0, 60.0), 1))
    if kind == "seed_fod":
        return dict(kind=kind, shape=rng.choice(["32x32x32", "64x64x64"]), lmax=rng.choice([-1, 8, 8]),
                    n=spread(500, 200000))
    return dict(kind=kind, shape="32x32x32", lmax=rng.choice([-1, 2, 4, 6, 8]), n=spread(100, 100000),
                algorithm=algorithm, step=rng.choice([0.2, 0.001]))


# ------------------------------------------------------------------ inputs


def _shape(case):
    return tuple(int(v) for v in case["shape"].split("x"))


def _n_coefficients(lmax):
    return 6 if lmax < 0 else (lmax + 1) * (lmax + 2) // 2


def _model(lmax):
    if lmax < 0:
        return local.DiffusionTensorImaging()
    return local.RealSymmetricSphericalHarmonics(_n_coefficients(lmax))


def _mask(shape):
    """Ellipsoid with semi-axes 0.45 of the volume's extents."""
    axes = [((np.arange(n, dtype=np.float32) - (n - 1) / 2.0) / (0.45 * n)) ** 2 for n in shape]
    inside = axes[0][:, None, None] + axes[1][None, :, None] + axes[2][None, None, :] <= 1.0
    return nifti.Nifti1Image(inside.astype(np.uint8), np.diag([VOXEL_MM, VOXEL_MM, VOXEL_MM, 1.0]))


def _volume(shape, lmax, seed):
    if lmax < 0:
        return synthetic.dti_field(shape, seed=seed)
    return synthetic.bundle_field(shape, lmax=lmax, seed=seed)[0]


@functools.lru_cache(maxsize=8)
def _surface(shape, frequency):
    return synthetic.config2_surface(shape=shape, frequency=frequency)


def _algorithm(case, seed):
    model = _model(case["lmax"])
    if case["algorithm"] == "transport":
        return tg.algorithm.Transport(model, step_size=case["step"], gamma=1.0)
    return tg.algorithm.Diffusion(model, step_size=case["step"], gamma=1.0,
                                  noise_variance=case.get("noise", 0.1), seed=seed, rng=case.get("rng", "mwc64x"))


def _job_specs(case, seed):
    """Uneven jobs: seed counts log-uniform and scaled to case["n"] in all."""
    rng = np.random.default_rng([seed, 17])
    sizes = np.exp(rng.uniform(0.0, math.log(100.0), case["jobs"]))
    sizes = np.maximum(1, (sizes / sizes.sum() * case["n"]).astype(int))
    sizes[-1] += case["n"] - sizes.sum()
    return [dict(n=int(n), lmax=int(rng.choice([4, 6, 8])), step=case["step"],
                 algorithm="transport" if rng.uniform() < 0.5 else "diffusion",
                 noise=float(rng.uniform(0.05, 0.2)), max_mm=float(rng.uniform(50.0, 300.0)),
                 seed=int(rng.integers(0, 2 ** 31))) for n in sizes]


def prepare(case, seed):
    runtime = tg.runtime.default_runtime()
    shape = _shape(case)
    kind = case["kind"]
    state = dict(case=case, seed=seed, runtime=runtime)
    if kind in ("track", "jobs", "serve"):
        longest = int(math.floor(case.get("max_mm", 300.0) / case["save_at"]))
        state["out"] = torch.zeros((case["n"] * longest, 3), dtype=torch.float32, device=runtime.device)
    if kind in ("jobs", "serve"):
        mask = _mask(shape)
        domain = tg.domain.Image(mask)
        domain.device(runtime)
        fields = {}
        state["requests"] = []
        for spec in _job_specs(case, seed):
            if spec["lmax"] not in fields:
                fields[spec["lmax"]] = tg.field.Image(_volume(shape, spec["lmax"], seed + spec["lmax"]))
                fields[spec["lmax"]].device(runtime, _lib.MODEL_SH)
            state["requests"].append((fields[spec["lmax"]], domain, spec,
                                      synthetic.uniform_seeds(mask, spec["n"], seed=spec["seed"])))
        if kind == "serve":
            state["server"] = serve.Server(runtime, hbm_budget_bytes=12e9, pool_points=32 << 20, epoch_steps=65536,
                                           epoch_seconds=6e-3, max_requests=32, reserve_bytes=int(3e9))
        return state
    volume = _volume(shape, case["lmax"], seed)
    if kind == "seed_fod":
        rng = np.random.default_rng([seed, 3])
        state["sparse"] = seeds.sparse_fod(volume)
        state["states"] = rng.integers(0, 4294967295, size=(case["n"], 2), dtype=np.uint32)
        return state
    if kind == "update":
        rng = np.random.default_rng([seed, 5])
        rows = np.asarray(volume.dataobj).reshape(-1, _n_coefficients(case["lmax"]))
        o = rng.normal(size=(case["n"], 3))
        state["rows"] = np.ascontiguousarray(rows[rng.integers(0, len(rows), case["n"])])
        state["orientations"] = (o / np.linalg.norm(o, axis=1, keepdims=True)).astype(np.float32)
        return state
    state["field"] = tg.field.Image(volume)
    state["field"].device(runtime, local.model_id(_model(case["lmax"])))
    if case.get("domain", "image") == "image":
        mask = _mask(shape)
        state["domain"] = tg.domain.Image(mask)
        state["domain"].device(runtime)
        if kind == "track":
            state["seeds"] = synthetic.uniform_seeds(mask, case["n"], seed=seed)
    else:
        vertices, faces = _surface(shape, int(case["domain"][len("surface"):]))
        state["domain"] = tg.domain.Mesh(vertices, faces)
        state["domain"].device(runtime)
        state["seeds"] = synthetic.seeds_inside(lambda p: tg.domain.contains(state["domain"], p, runtime),
                                                vertices.min(axis=0), vertices.max(axis=0), case["n"], seed=seed,
                                                chunk=max(1024, 2 * case["n"]))
    if case.get("resident"):
        state["device_seeds"] = runtime.to_device(state["seeds"])
    if kind in ("tod", "connectome"):
        state["domain"].boundary_arrays()
        state["domain"].boundary_bvh().device(runtime)
        state["grid"] = nifti.Nifti1Image(np.zeros(shape, np.float32), volume.affine)
    return state


# --------------------------------------------------------------------- run


def _handed_on(state, points):
    state["out"][:len(points)].copy_(torch.from_numpy(points), non_blocking=True)
    return state["out"]


def _run_resident(state):
    """tg_tracker_run on seeds in device memory, points copied to a device buffer."""
    case, runtime = state["case"], state["runtime"]
    n, lib, stream = case["n"], state["runtime"].lib, ctypes.c_void_p(state["runtime"].stream_handle)
    algorithm = _algorithm(case, state["seed"])
    batches = -(-n // case["batch"])
    stream_seeds = np.array([algorithm.get_rng_seed() for _ in range(batches)], dtype=np.uint32)
    key = algorithm.philox_key() if algorithm.rng_mode() == _lib.RNG_PHILOX else 0
    lengths, offsets = np.empty(n, np.uint32), np.empty(n, np.uint64)
    points, steps = ctypes.c_uint64(), ctypes.c_uint64()
    a = tg.algorithm.to_struct(algorithm, 0, key, 0)
    model = local.model_id(algorithm.local_model)
    _lib.check(lib.tg_tracker_run(
        runtime.tracker(), ctypes.byref(a), state["domain"].device(runtime), state["field"].device(runtime, model),
        ctypes.c_void_p(state["device_seeds"].data_ptr()), 0, n, case["batch"],
        stream_seeds.ctypes.data_as(ctypes.c_void_p), case["save_at"], int(math.floor(case["max_mm"] / case["save_at"])),
        lengths.ctypes.data_as(ctypes.c_void_p), offsets.ctypes.data_as(ctypes.c_void_p), ctypes.byref(points),
        ctypes.byref(steps), stream))
    _lib.check(lib.tg_tracker_copy_points(runtime.tracker(), ctypes.c_void_p(state["out"].data_ptr()), 0,
                                          points.value, 0, stream))
    return state["out"], lengths


def _in_order(state, results):
    """Points of the streamlines one after the other (a server packs them as they finish)."""
    device, base = state["out"].device, 0
    for points, offsets, lengths, _ in results:
        p = torch.from_numpy(points).to(device)
        o, n = torch.from_numpy(offsets).to(device), torch.from_numpy(lengths).to(device)
        starts = torch.cumsum(n, 0) - n
        at = torch.arange(len(points), device=device) + torch.repeat_interleave(o - starts, n, output_size=len(points))
        torch.index_select(p, 0, at, out=state["out"][base:base + len(points)])
        base += len(points)
    return state["out"], np.concatenate([lengths for _, _, lengths, _ in results])


def _run_serve(state):
    case, server = state["case"], state["server"]
    ids = []
    for field, domain, spec, rows in state["requests"]:
        job = jobs.prepare(field, rows, domain, _algorithm(spec, spec["seed"]), save_at=case["save_at"],
                           maximum_streamline_length=spec["max_mm"])
        ids.append(server.submit(job))
    done = {}
    while len(done) < len(ids):
        for rid in server.poll():
            done[rid] = server.take(rid)
    return _in_order(state, [done[rid] for rid in ids])


def run(state):
    case, runtime = state["case"], state["runtime"]
    kind = case["kind"]
    if kind == "track" and case["resident"]:
        return _run_resident(state)
    if kind == "track":
        t = tg.tractogram(state["field"], state["seeds"], state["domain"], _algorithm(case, state["seed"]),
                          save_at=case["save_at"], maximum_streamline_length=case["max_mm"],
                          batch_size=case["batch"], runtime=runtime)
        return _handed_on(state, t.streamlines.get_data()), t.streamlines.lengths
    if kind == "jobs":
        prepared = [jobs.prepare(field, rows, domain, _algorithm(spec, spec["seed"]), save_at=case["save_at"],
                                 maximum_streamline_length=spec["max_mm"])
                    for field, domain, spec, rows in state["requests"]]
        result = jobs.run_jobs_packed(prepared, runtime)
        return _handed_on(state, result.points), result.lengths
    if kind == "serve":
        return _run_serve(state)
    if kind == "tod":
        image = tracking.tod(_algorithm(case, state["seed"]), state["domain"], state["field"], state["grid"],
                             case["n"], maximum_streamline_length=case["max_mm"], runtime=runtime)
        return np.asarray(image.dataobj)
    if kind == "connectome":
        m = tracking.connectome(_algorithm(case, state["seed"]), state["domain"], state["field"], case["n"],
                                maximum_streamline_length=case["max_mm"], runtime=runtime)
        most = 9 * case["n"]          # a track adds at most nine entries
        return (np.pad(m.data, (0, most - m.nnz)), np.pad(m.indices, (0, most - m.nnz), constant_values=-1),
                m.indptr)
    if kind == "seed_fod":
        return seeds.seeds_from_sparse_fod(local.model_id(_model(case["lmax"])), *state["sparse"], state["states"],
                                           runtime)
    algorithm = _algorithm(case, state["seed"])
    return (local.evaluate(algorithm.local_model, state["rows"], state["orientations"], runtime),
            tg.algorithm.update_orientation(algorithm, state["rows"], state["orientations"], runtime))


# -------------------------------------------------------------------- work


def _step_flops(lmax, algorithm):
    """Binary32 operations of one step: model value and slopes (4 per folded
    coefficient, 11 per order), frame, exponential map and Euler step, softplus,
    and for the SDE two normal draws."""
    model = 60 if lmax < 0 else 4 * _n_coefficients(lmax) + 14 * lmax + 60
    return model + 90 + (90 if algorithm == "diffusion" else 0)


def _mean_mm(shape, max_mm, in_mask_transport=True):
    if in_mask_transport:
        return MEAN_TRANSPORT * max_mm
    return min(max_mm, MEAN_EXTENT * VOXEL_MM * sum(shape) / 3.0)


def work(case):
    shape, kind, n = _shape(case), case["kind"], case["n"]
    voxels = int(np.prod(shape))
    if kind == "update":
        C = _n_coefficients(case["lmax"])
        return {"bytes": float(n * (4 * C + 12 + 12 + 12)), "flops": float(n * 2 * _step_flops(case["lmax"], "transport"))}
    if kind == "seed_fod":
        C = _n_coefficients(case["lmax"])
        return {"bytes": float(min(n, voxels) * 4 * C + n * (8 + 16 + 32)), "flops": float(n * 1000 * (2 * C + 20))}
    if kind in ("jobs", "serve"):
        mean = _mean_mm(shape, 175.0)
        steps = n * mean / case["step"]
        flops = steps * np.mean([_step_flops(l, a) for l in (4, 6, 8) for a in ("transport", "diffusion")])
        return {"bytes": float(voxels * (4 * (15 + 28 + 45) + 1) + n * 32 + 12 * n * mean / case["save_at"]),
                "flops": float(flops)}
    C = _n_coefficients(case["lmax"])
    mean = _mean_mm(shape, case["max_mm"],
                    case["algorithm"] == "transport" and case["lmax"] >= 0 and case.get("domain", "image") == "image")
    flops = n * mean / case["step"] * _step_flops(case["lmax"], case["algorithm"])
    if kind == "track":
        return {"bytes": float(voxels * (4 * C + 1) + n * 32 + 12 * n * mean / case["save_at"]), "flops": float(flops)}
    if kind == "tod":
        return {"bytes": float(voxels * (4 * C + 1 + 180)), "flops": float(flops + n * mean / case["step"] * 150)}
    return {"bytes": float(voxels * (4 * C + 1) + n * 9 * 12), "flops": float(flops)}


# ------------------------------------------------------------------- exact


def _sh_rows(directions, lmax):
    """Real symmetric SH (even l <= lmax) at unit directions in 64 bits:
    values, d/dtheta and (d/dphi)/sin(theta), (n, C) each; coefficient
    l (l + 1) / 2 + m, Legendre functions with the Condon-Shortley phase."""
    x, y, z = directions.T
    st, ct = np.hypot(x, y), z
    phi = np.arctan2(y, x)
    # P[l][m] / sin^m, so that nothing divides by sin at the poles
    q = {}
    for m in range(lmax + 1):
        q[m, m] = np.full_like(ct, (-1.0) ** m * np.prod(np.arange(1, 2 * m, 2, dtype=float)))
        if m < lmax:
            q[m + 1, m] = ct * (2 * m + 1) * q[m, m]
        for l in range(m + 2, lmax + 1):
            q[l, m] = ((2 * l - 1) * ct * q[l - 1, m] - (l + m - 1) * q[l - 2, m]) / (l - m)
    C = (lmax + 1) * (lmax + 2) // 2
    Y, T, P = (np.zeros((len(ct), C)) for _ in range(3))
    for l in range(0, lmax + 1, 2):
        for m in range(l + 1):
            k = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            k *= math.sqrt(2.0) if m else 1.0
            value = st ** m * q[l, m]
            # dq_l^m/dx = -q_l^(m+1); d/dtheta of sin^m q(cos)
            slope = (m * st ** (m - 1) * ct * q[l, m] if m else 0.0) + (st ** (m + 1) * q[l, m + 1] if m < l else 0.0)
            over = m * st ** (m - 1) * q[l, m] if m else 0.0
            base = l * (l + 1) // 2
            Y[:, base + m], T[:, base + m] = k * value * np.cos(m * phi), k * slope * np.cos(m * phi)
            P[:, base + m] = -k * over * np.sin(m * phi)
            if m:
                Y[:, base - m], T[:, base - m] = k * value * np.sin(m * phi), k * slope * np.sin(m * phi)
                P[:, base - m] = k * over * np.cos(m * phi)
    return Y, T, P


def _softplus(v):
    return np.where(v * 100.0 < 30.0, np.log1p(np.exp(np.minimum(v * 100.0, 30.0))) / 100.0, v)


def _frame(o):
    rho = np.hypot(o[:, 0], o[:, 1])
    r = np.linalg.norm(o, axis=1)
    ct, st, cp, sp = o[:, 2] / r, rho / r, o[:, 0] / rho, o[:, 1] / rho
    return np.stack([ct * cp, ct * sp, -st], 1), np.stack([-sp, cp, 0 * cp], 1)


def _model_rows(lmax, rows, o):
    if lmax < 0:
        et, ep = _frame(o)
        D = rows[:, [0, 3, 4, 3, 1, 5, 4, 5, 2]].reshape(-1, 3, 3)
        du = np.einsum("nij,nj->ni", D, o)
        return np.stack([(o * du).sum(1), 2 * (du * et).sum(1), 2 * (du * ep).sum(1)], 1)
    Y, T, P = _sh_rows(o / np.linalg.norm(o, axis=1, keepdims=True), lmax)
    raw = (rows * Y).sum(1)
    slope = 1.0 / (1.0 + np.exp(-np.clip(100.0 * raw, -700.0, 700.0)))
    return np.stack([_softplus(raw), (rows * T).sum(1) * slope, (rows * P).sum(1) * slope], 1)


class _Mwc:
    """The MWC64X streams of many seeds at once."""

    def __init__(self, x, c):
        self.x, self.c = x.astype(np.uint64), c.astype(np.uint64)

    @classmethod
    def of(cls, seed, n):
        def mix(v):
            for shift, factor in ((16, 0x7feb352d), (15, 0x846ca68b)):
                v = (v ^ (v >> np.uint64(shift))) * np.uint64(factor) & np.uint64(0xffffffff)
            return v ^ (v >> np.uint64(16))

        i, low = np.arange(n, dtype=np.uint64), np.uint64(0xffffffff)
        x = mix(np.uint64(seed) ^ ((i + np.uint64(0x9e3779b9)) & low))
        c = mix((np.uint64(seed) + i * np.uint64(0x85ebca6b)) & low) % np.uint64(4294883355)
        return cls(np.maximum(x, 1), c)

    def bits(self, where=slice(None)):
        x, c = self.x[where], self.c[where]
        out = (x ^ c) >> np.uint64(8)
        t = x * np.uint64(4294883355) + c
        self.x[where], self.c[where] = t & np.uint64(0xffffffff), t >> np.uint64(32)
        return out

    def uniform(self):
        return self.bits().astype(np.float64) * 2.0 ** -24

    def normal(self):
        u = self.uniform()
        while np.any(u <= 0):
            zero = np.flatnonzero(u <= 0)
            u[zero] = self.bits(zero).astype(np.float64) * 2.0 ** -24
        return np.sqrt(-2.0 * np.log(u)) * np.cos(2 * math.pi * self.uniform())


def exact(case, seed):
    """In 64 bits where the path has such a value.  Tracking has none: a step
    divides by a model value that nearly vanishes in places, so rounding grows to
    whole voxels within a track, and what tracks share (tod, connectome, jobs,
    server) follows from their points."""
    if case["kind"] == "update":
        state = prepare(case, seed)
        rows, o = state["rows"].astype(np.float64), state["orientations"].astype(np.float64)
        mv = _model_rows(case["lmax"], rows, o)
        et, ep = _frame(o)
        t = case["step"] * (mv[:, 1:2] * et + mv[:, 2:3] * ep) / np.maximum(mv[:, :1], 1e-6)
        if case["algorithm"] == "diffusion":
            stream = int(np.random.default_rng(seed).integers(0, np.iinfo(np.uint32).max, dtype=np.uint32))
            mwc = _Mwc.of(stream, case["n"])
            n1, n2 = mwc.normal(), mwc.normal()
            t = t + math.sqrt(0.1 * case["step"]) * (n1[:, None] * et + n2[:, None] * ep)
        n = np.linalg.norm(t, axis=1, keepdims=True)
        return mv, np.cos(n) * o + np.sinc(n / math.pi) * t
    if case["kind"] == "seed_fod":
        state = prepare(case, seed)
        coefficients, voxels, affine = (np.asarray(v, np.float64) for v in state["sparse"])
        mwc = _Mwc(state["states"][:, 0], state["states"][:, 1])
        pick = np.minimum((mwc.uniform() * len(voxels)).astype(np.int64), len(voxels) - 1)
        at = voxels[pick]
        at[:, :3] += np.stack([mwc.uniform() - 0.5 for _ in range(3)], 1)
        i = np.arange(1000)
        turn = 2 * math.pi / ((1 + 5 ** 0.5) / 2) * i
        z = 1.0 - 2.0 * i / 999.0
        directions = np.stack([np.sqrt(1 - z * z) * np.cos(turn), np.sqrt(1 - z * z) * np.sin(turn), z], 1)
        u = mwc.uniform()
        basis = None if case["lmax"] < 0 else _sh_rows(directions, case["lmax"])[0].T
        out = np.zeros((case["n"], 8))
        out[:, :4] = at @ affine.T
        for lo in range(0, case["n"], 20000):
            c = coefficients[pick[lo:lo + 20000]]
            if basis is None:
                D = c[:, [0, 3, 4, 3, 1, 5, 4, 5, 2]].reshape(-1, 9)
                values = np.maximum(D @ np.einsum("ni,nj->ijn", directions, directions).reshape(9, -1), 0.0)
            else:
                values = _softplus(c @ basis)
            values = np.cumsum(values, axis=1)
            chosen = (values <= (u[lo:lo + 20000] * values[:, -1])[:, None]).sum(1)
            out[lo:lo + 20000, 4:7] = directions[np.minimum(chosen, 999)]
        return out
    return None
