"""The work that a user of this framework has it do, as cases for timing.

Whole steps: a 2-D channel (latency: ten thousand particles, some eighty
launches), the flow past a sphere (the benchmark scene, two million
particles), a batch of channels replayed from a CUDA graph.  Single stages:
the grid rebuild, the DFSPH solves, the DIMCV sweeps with the reference's
default sampler, the vortex-to-velocity sum (2-D and 3-D reference kernel,
3-D blob kernel), the full Biot-Savart sum, the differentiable velocity with
its gradients, and one step of the differentiable rollout.

Positions are the dispersed state a run reaches after its first steps: the
scene's lattice with every fluid particle moved by up to 2% of the
spacing, and a smooth velocity disturbance with some noise on the inflow.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from dimcv_sph_b200 import scenes
from dimcv_sph_b200.adjoint import MC, Plan, VortexBox
from dimcv_sph_b200.batch import SceneBatch, channel_batch_configs
from dimcv_sph_b200.config_builder import SimConfig
from dimcv_sph_b200.dimcv_sph import DIMCVSPHSolver
from dimcv_sph_b200.particle_system import ParticleSystem

RESTART = 32  # passes after which a stepped state starts again from its first state


def listed():
    return [
        # the small channel: what one interactive step of a 2-D scene costs
        {"name": "channel_step", "kind": "step", "dim": 2, "radius": 0.01, "sampler": "inverse_cdf",
         "blob": False, "vis": True, "tile": 0},
        # the benchmark scene of the framework: one step of the flow past a sphere
        {"name": "sphere_step", "kind": "step", "dim": 3, "radius": 0.004, "sampler": "inverse_cdf",
         "blob": False, "vis": True, "tile": 8},
        # a parameter sweep: many channels of 2k-60k particles, two steps per graph launch
        {"name": "channels_batch", "kind": "batch", "scenes": 24, "n_min": 2000, "n_max": 60000},
        # the per-step grid rebuild: sort, cell table, field permutation, neighbour lists
        {"name": "grid_3d", "kind": "grid", "dim": 3, "radius": 0.006},
        # densities, both Jacobi solves and the forces between them
        {"name": "dfsph_3d", "kind": "dfsph", "dim": 3, "radius": 0.006},
        # vorticity, smoothing, kinematic vorticity number, kernel density, birth and death of samples
        {"name": "dimcv_3d", "kind": "dimcv", "dim": 3, "radius": 0.006},
        # the velocity of the vortex samples, 2-D, as in a fine channel
        {"name": "vvpe_2d", "kind": "vvpe", "dim": 2, "side": 250, "every": 16, "blob": False, "periodic": False,
         "compensated": False},
        # the same sum with the reference kernel in 3-D (odd lattice, M = N/32)
        {"name": "vvpe_3d", "kind": "vvpe", "dim": 3, "side": 59, "every": 32, "blob": False, "periodic": False,
         "compensated": False},
        # the vortex ring with the regularised 3-D kernel, M = N/16
        {"name": "vvpe_ring", "kind": "vvpe", "dim": 3, "side": 64, "every": 16, "blob": True, "periodic": False,
         "compensated": False},
        # the full sum that the Monte-Carlo velocity is compared with
        {"name": "bs_ring", "kind": "bs", "n": 65536, "precision": 32, "compensated": False},
        # the differentiable velocity, forward and backward, on a kept plan
        {"name": "adjoint_velocity", "kind": "adjoint", "side": 256, "every": 16, "precision": 32},
        # one step of a differentiable rollout: plan, velocity, gradients
        {"name": "adjoint_step", "kind": "adjoint_step", "side": 128, "every": 16, "precision": 32},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step", "step", "batch", "grid", "dfsph", "dimcv", "vvpe", "vvpe", "vvpe", "bs", "adjoint",
                       "adjoint", "adjoint_step"])
    dim = rng.choice([2, 3])
    radius = round(_log(rng, 0.0025, 0.02), 5) if dim == 2 else round(_log(rng, 0.005, 0.03), 5)
    if kind == "step":
        return {"kind": kind, "dim": dim, "radius": radius,
                "sampler": rng.choice(["inverse_cdf", "stratified", "bernoulli"]),
                "blob": dim == 3 and rng.random() < 0.4, "vis": rng.random() < 0.7, "tile": 0}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 32), "n_min": int(_log(rng, 1500, 4000)),
                "n_max": int(_log(rng, 8000, 60000))}
    if kind in ("grid", "dfsph", "dimcv"):
        return {"kind": kind, "dim": dim, "radius": radius}
    if kind == "vvpe":
        blob = dim == 3 and rng.random() < 0.5
        return {"kind": kind, "dim": dim, "side": int(_log(rng, 40, 400)) if dim == 2 else int(_log(rng, 13, 68)),
                "every": rng.choice([8, 16, 32, 64]), "blob": blob,
                "periodic": not blob and rng.random() < 0.25, "compensated": rng.random() < 0.2}
    if kind == "bs":
        precision = 64 if rng.random() < 0.3 else 32
        return {"kind": kind, "n": int(_log(rng, 1000, 20000 if precision == 64 else 130000)), "precision": precision,
                "compensated": precision == 32 and rng.random() < 0.2}
    precision = 64 if rng.random() < 0.25 else 32
    return {"kind": kind, "side": int(_log(rng, 24, 80 if precision == 64 else 256)),
            "every": rng.choice([1, 4, 16]) if kind == "adjoint" else rng.choice([4, 16]), "precision": precision}


# ------------------------------------------------------------------ scenes
def _scene(case):
    r = case["radius"]
    if case["dim"] == 2:
        cfg = scenes.channel2d(radius=r, dt=4e-4 * r / 0.01, reserved=int(40 / r) + 2000)
    else:
        cfg = scenes.sphere3d(radius=r, dt=1.6e-4 * r / 0.004)
    conf = cfg.config["Configuration"]
    conf["samplerMode"] = case.get("sampler", "bernoulli")
    conf["computeVis"] = case.get("vis", True)
    if case.get("blob"):
        conf["kernel3D"] = True
    return cfg


def _generator(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed))


def _disturb(x, v, fluid, spacing, seed):
    """The dispersed state, in place: every fluid row moved by up to 2% of the
    spacing, its velocity disturbed by four Fourier modes and 1% noise."""
    g = _generator(seed)
    dim = x.shape[1]

    def rand(*shape):
        return torch.rand(*shape, device="cuda", generator=g)

    dx = (rand(x.shape[0], dim) - 0.5) * (0.04 * spacing)
    dv = 0.01 * torch.randn(x.shape[0], dim, device="cuda", generator=g)
    for _ in range(4):
        k, ph, a = 2 + 7 * rand(dim), 6.28 * rand(1), 0.05 * (2 * rand(dim) - 1)
        dv += a * torch.sin((x * k).sum(1, keepdim=True) + ph)
    x += torch.where(fluid[:, None], dx, torch.zeros_like(dx))
    v += torch.where(fluid[:, None], dv, torch.zeros_like(dv))


def _system(case, seed):
    ps = ParticleSystem(_scene(case))
    solver = ps.build_solver()
    solver.initialize()
    n = ps.particle_num[None]
    _disturb(ps.x[:n], ps.v[:n], ps.material[:n] == 1, ps.particle_diameter, seed)
    return ps, solver, n


def _prepare_step(case, seed):
    ps, solver, n = _system(case, seed)
    solver.seed = seed
    cnt = ps.counters()
    s = {"ps": ps, "solver": solver, "first": {k: t.clone() for k, t in ps.fields.t.items()},
         "counts": (cnt["n"], cnt["n_fluid"], cnt["n_solid"]), "passes": 0}
    if case["tile"]:  # the tile and chunk count that a user keeps from an earlier run
        solver.far_tile = case["tile"]
        ps.lib.dv_set_far_tile(ps.ctx, case["tile"])
        ps.lib.dv_set_far_chunks(ps.ctx, 8)
    solver.step()  # the solver tunes its far field on its first step
    _restart_step(s)
    return s


def _restart_step(s):
    ps, solver = s["ps"], s["solver"]
    for k, t in s["first"].items():
        ps.fields.t[k].copy_(t)
    ps.set_counts(*s["counts"])
    for k, t in ps.solver_buf.t.items():
        t.zero_()
    solver.cnt = solver.rng_step = 0
    s["passes"] = 0


def _run_step(s):
    if s["passes"] == RESTART:
        _restart_step(s)
    s["solver"].step()
    s["passes"] += 1
    ps, n = s["ps"], s["counts"][0]
    return {"x": ps.x[:n], "v": ps.v[:n], "density": ps.density[:n], "material": ps.material[:n]}


def _prepare_batch(case, seed):
    cfgs, _ = channel_batch_configs(n_scenes=case["scenes"], seed=11, n_min=case["n_min"], n_max=case["n_max"])
    b = SceneBatch(cfgs)
    cnt = b.counters()
    n, f = cnt["n"], b.fields
    _disturb(f["x"][:n, :2], f["v"][:n, :2], f["material"][:n] == 1, 0.02, seed)
    b.lib.dv_set_far_tile(b.ctx, 2)
    s = {"batch": b, "first": {k: t.clone() for k, t in f.t.items()}, "counts": (n, cnt["n_fluid"], cnt["n_solid"]),
         "passes": 0}
    b.capture(2)
    return s


def _run_batch(s):
    b = s["batch"]
    if s["passes"] == RESTART:
        for k, t in s["first"].items():
            b.fields.t[k].copy_(t)
        b.lib.dv_set_counts(b.ctx, *s["counts"])
        s["passes"] = 0
    b.replay()
    s["passes"] += 1
    n = s["counts"][0]
    return {"x": b.fields["x"][:n], "v": b.fields["v"][:n], "density": b.fields["density"][:n],
            "object_id": b.fields["object_id"][:n]}


# ------------------------------------------------------------------ stages
def _prepare_stage(case, seed):
    ps, solver, n = _system(case, seed)
    solver.seed = seed
    ps.initialize_particle_system()
    if case["kind"] == "dimcv":  # what the sweeps read of the stages before them
        solver.compute_densities()
        solver.compute_DFSPH_factor()
        solver.divergence_solve()
        solver.compute_non_pressure_forces()
    return {"ps": ps, "solver": solver, "n": ps.particle_num[None]}


def _run_grid(s):
    ps, n = s["ps"], s["n"]
    ps.initialize_particle_system()
    return {"x": ps.x[:n], "v": ps.v[:n], "m_V": ps.m_V[:n], "grid_ids": ps.grid_ids[:n],
            "object_id": ps.object_id[:n], "material": ps.material[:n]}


def _run_dfsph(s):
    ps, solver, n = s["ps"], s["solver"], s["n"]
    solver.compute_densities()
    solver.compute_DFSPH_factor()
    solver.divergence_solve()
    solver.compute_non_pressure_forces()
    solver.predict_velocity()
    solver.pressure_solve()
    return {"v": ps.v[:n], "density": ps.density[:n], "density_adv": ps.density_adv[:n],
            "factor": ps.dfsph_factor[:n], "acceleration": ps.acceleration[:n]}


def _run_dimcv(s):
    ps, solver, n = s["ps"], s["solver"], s["n"]
    solver.init()
    solver.compute_d_vorticity()
    solver.update_sample()
    solver.smooth_and_kernel_density()
    return {"vorticity": ps.vorticity[:n], "grad_v": solver.grad_v[:n], "d_vort": solver.d_vort[:n],
            "smoothed": solver.d_vort_smoothed[:n], "kvn": solver.kinematic_vort_num[:n],
            "kden": solver.kernel_density[:n], "is_sample": ps.is_sample[:n]}


# ------------------------------------------- vortex sums on a unit box
def _points(dim, side, uniform, seed):
    """Positions (float32, caller order) in the unit box: a jittered lattice,
    or uniform points as in the vortex ring."""
    g = _generator(seed)
    n = side ** dim
    if uniform:
        x = torch.rand(n, dim, device="cuda", generator=g)
    else:
        ax = torch.arange(side, device="cuda", dtype=torch.float32)
        x = torch.stack(torch.meshgrid(*[ax] * dim, indexing="ij"), -1).reshape(n, dim) + 0.5
        x = (x + (torch.rand(n, dim, device="cuda", generator=g) - 0.5) * 0.5) / side
    return torch.clamp(x, 0.0, 0.99999988), g


def _box_config(dim, side, blob=False, periodic=False, compensated=False):
    r = 0.5 / side
    return SimConfig(config={"Configuration": {
        "domainStart": [0.0] * dim, "domainEnd": [1.0] * dim, "particleRadius": r, "density0": 1000,
        "simulationMethod": 0, "gravitation": [0.0] * dim, "timeStepSize": 1e-3, "volumeScale": 1.25,
        "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False, "kernel3D": blob,
        "blobDelta": r, "samplerMode": "injected", "periodic": periodic, "compensated": compensated}})


def _cells(side, periodic):
    h = 2.0 / side
    return (int(math.floor(1.0 / h)), 1.0 / math.floor(1.0 / h)) if periodic else (int(np.ceil(1.0 / h)), h)


def _slot_order(x, side, periodic):
    """The particles in the framework's slot order: by the Morton key of the
    cell (last axis lowest), stable in the caller's order."""
    num, size = _cells(side, periodic)
    c = (x / torch.tensor(np.float32(size), device=x.device)).to(torch.int64).clamp(0, num - 1)
    key = torch.zeros(x.shape[0], dtype=torch.int64, device=x.device)
    dim = x.shape[1]
    for bit in range(max(1, (num - 1).bit_length())):
        for d in range(dim):
            key |= ((c[:, d] >> bit) & 1) << (bit * dim + (dim - 1 - d))
    return torch.sort(key, stable=True).indices


def _ring(x, g):
    """Vorticity of a Gaussian-core ring (3-D) or of two blobs (2-D), with noise."""
    n, dim = x.shape
    w = torch.zeros(n, 3, device="cuda")
    if dim == 2:
        for cx, cy, a, s in ((0.3, 0.6, 5.0, 0.08), (0.7, 0.4, -4.0, 0.06)):
            w[:, 2] += a * torch.exp(-((x[:, 0] - cx) ** 2 + (x[:, 1] - cy) ** 2) / s ** 2)
        w[:, 2] += 0.05 * torch.randn(n, device="cuda", generator=g)
        return w
    y = x - 0.5
    rho = torch.sqrt(y[:, 0] ** 2 + y[:, 1] ** 2).clamp_min(1e-6)
    m = 30.0 * torch.exp(-((rho - 0.25) ** 2 + y[:, 2] ** 2) / 0.08 ** 2)
    w[:, 0], w[:, 1] = -y[:, 1] / rho * m, y[:, 0] / rho * m
    return w + 0.3 * torch.randn(n, 3, device="cuda", generator=g)


def _vvpe_inputs(case, seed):
    """In the caller's order: positions, smoothed vorticity, KVN, drawn particles."""
    x, g = _points(case["dim"], case["side"], case["blob"], seed)
    n = x.shape[0]
    w = _ring(x, g)
    kvn = 0.5 + torch.rand(n, device="cuda", generator=g)
    drawn = torch.randint(n, (max(1, n // case["every"]),), device="cuda", generator=g)
    return x, w, kvn, drawn


def _fluid(cfg, x, speed):
    n, dim = x.shape
    ps = ParticleSystem(cfg, capacity=n)
    v = np.zeros((n, dim), np.float32)
    v[:, 0] = speed
    ps.add_particles(0, n, x.cpu().numpy(), v, np.full(n, 1000.0), np.zeros(n), np.ones(n, np.int32),
                     np.ones(n, np.int32), np.zeros((n, 3), np.int32))
    return ps


SPEED = 40.0  # of the flow that the vortices are carried by: the induced velocity is added to it


def _prepare_vvpe(case, seed):
    x, w, kvn, drawn = _vvpe_inputs(case, seed)
    n = x.shape[0]
    ps = _fluid(_box_config(case["dim"], case["side"], case["blob"], case["periodic"], case["compensated"]), x, SPEED)
    solver = DIMCVSPHSolver(ps)
    solver.initialize()
    perm = _slot_order(x, case["side"], case["periodic"])
    inv = torch.empty_like(perm)
    inv[perm] = torch.arange(n, device="cuda")
    solver.d_vort_smoothed[:n] = w[perm]
    solver.kinematic_vort_num[:n] = kvn[perm]
    solver.compute_kernel_density()
    m = drawn.shape[0]
    solver.sample_idx[:m] = inv[drawn].to(torch.int32)
    solver.num_samples[None] = m
    v = ps.v[:n].clone()
    solver.vort2vel()  # the solver tunes its far field on its first call
    ps.v[:n] = v
    return {"ps": ps, "solver": solver, "n": n}


def _run_vvpe(s):
    s["solver"].vort2vel()
    return {"v_vort": s["solver"].v_vort[:s["n"]], "v": s["ps"].v[:s["n"]]}


def _exact_vvpe(case, seed):
    x, w, kvn, drawn = _vvpe_inputs(case, seed)
    dim, side = case["dim"], case["side"]
    perm = _slot_order(x, side, case["periodic"])
    inv = torch.empty_like(perm)
    inv[perm] = torch.arange(perm.shape[0], device="cuda")
    x, w, kvn = x[perm], w[perm].double(), kvn[perm].double()
    n, h = x.shape[0], float(np.float32(2.0 / side))
    hd = 2.0 / side
    coef = 1.25 * 0.8 * (1.0 / side) ** dim * (1.0 / (4 * math.pi) if case["blob"] else 0.1592)
    delta2 = (0.5 / side) ** 2

    def rel(xi, xj):  # float32 differences decide who is a neighbour, as in the framework
        d = xi[:, None, :] - xj[None, :, :]
        dd = xi.double()[:, None, :] - xj.double()[None, :, :]
        if case["periodic"]:
            d = d - (d > 0.5).float() + (d < -0.5).float()
            dd = dd - torch.round(dd)
        r2 = d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]
        if dim == 3:
            r2 = r2 + d[..., 2] * d[..., 2]
        return dd, torch.sqrt(r2)

    def cross(dd, k, wj):
        dx, dy = dd[..., 0], dd[..., 1]
        a, b = k * dx, k * dy
        z = a @ wj[:, 1] - b @ wj[:, 0]
        if case["blob"]:
            e = k * dd[..., 2]
            return torch.stack([b @ wj[:, 2] - e @ wj[:, 1], e @ wj[:, 0] - a @ wj[:, 2], z], -1)
        return torch.stack([b @ wj[:, 2], -(a @ wj[:, 2]), z], -1)

    def kernel(r2):
        if case["blob"]:
            return (r2 + delta2) ** -1.5
        r = torch.sqrt(r2)
        e = torch.exp(-r / 1e-6)
        return (1 - e) / (r * (r + 1e-6 * e))

    step = max(1, int(6e7 // n))
    kden = torch.empty(n, dtype=torch.float64, device="cuda")
    near = torch.empty(n, 3, dtype=torch.float64, device="cuda")
    for i in range(0, n, step):
        dd, rn = rel(x[i:i + step], x)
        nb = rn < h
        rows = torch.arange(dd.shape[0], device="cuda")
        nb[rows, rows + i] = False
        q = (dd.abs() / hd).clamp_max(1.0)
        kden[i:i + step] = kvn[i:i + step] * 0.75 ** dim + (nb * (0.75 * (1 - q * q)).prod(-1)) @ kvn
        r2 = (dd * dd).sum(-1) if case["blob"] else dd[..., 0] ** 2 + dd[..., 1] ** 2
        near[i:i + step] = coef * cross(dd, torch.where(nb, kernel(torch.where(nb, r2, torch.ones_like(r2))),
                                                        torch.zeros_like(r2)), w)
    slots = inv[drawn]
    total = kden.sum()
    ws = w[slots] / (kden[slots] + 1e-8)[:, None]
    xs = x[slots]
    out = torch.empty(n, 3, dtype=torch.float64, device="cuda")
    for i in range(0, n, step):
        dd, rn = rel(x[i:i + step], x)
        nb = rn < h  # the particle itself among them
        S = nb.double() @ kden
        dd, rn = rel(x[i:i + step], xs)
        far = rn > h
        r2 = (dd * dd).sum(-1)
        k = torch.where(far, kernel(torch.where(far, r2, torch.ones_like(r2))), torch.zeros_like(r2))
        cnt = far.sum(1).clamp_min(1).double()
        out[i:i + step] = near[i:i + step] + coef * cross(dd, k, ws) * ((total - S) / cnt)[:, None]
    v = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    v[:, 0] = SPEED
    add = torch.where((out.norm(dim=1) < SPEED)[:, None], out, torch.zeros_like(out))
    return {"v_vort": out, "v": (v + add)[:, :dim]}


def _bs_inputs(case, seed):
    g = _generator(seed)
    x = torch.rand(case["n"], 3, device="cuda", generator=g).clamp_max(0.99999988)
    return x, _ring(x, g)


def _bs_side(n):
    return max(8, int(round(n ** (1.0 / 3.0))))


def _prepare_bs(case, seed):
    x, w = _bs_inputs(case, seed)
    n, side = x.shape[0], _bs_side(case["n"])
    ps = _fluid(_box_config(3, side, True, False, case["compensated"]), x, 0.0)
    ps.initialize_particle_system()
    omega = torch.zeros(n, 4, device="cuda")
    omega[:, :3] = w[_slot_order(x, side, False)]
    out = torch.zeros(n, 4, device="cuda", dtype=torch.float64 if case["precision"] == 64 else torch.float32)
    return {"ps": ps, "omega": omega, "out": out, "precision": case["precision"]}


def _run_bs(s):
    ps, n = s["ps"], s["omega"].shape[0]
    rc = ps.lib.dv_bs_full(ps.ctx, C.byref(ps.fields_struct), C.c_void_p(s["omega"].data_ptr()), None, n,
                           C.c_void_p(s["out"].data_ptr()), s["precision"])
    if rc:
        raise RuntimeError(ps.lib.dv_last_error(ps.ctx).decode())
    return s["out"][:, :3]


def _exact_bs(case, seed):
    x, w = _bs_inputs(case, seed)
    side = _bs_side(case["n"])
    perm = _slot_order(x, side, False)
    x, w = x[perm].double(), w[perm].double()
    # the regularisation and the volume factor as the parameters hold them, in float32
    d2 = float(np.float32((0.5 / side) ** 2))
    coef = float(np.float32(1.25 * 0.8 * (1.0 / side) ** 3 / (4 * math.pi)))
    out = torch.empty_like(x)
    step = max(1, int(1e8 // x.shape[0]))
    for i in range(0, x.shape[0], step):
        a = [x[i:i + step, d][:, None] - x[None, :, d] for d in range(3)]
        k = (a[0] * a[0] + a[1] * a[1] + a[2] * a[2] + d2) ** -1.5
        a = [k * t for t in a]
        out[i:i + step] = torch.stack([a[1] @ w[:, 2] - a[2] @ w[:, 1], a[2] @ w[:, 0] - a[0] @ w[:, 2],
                                       a[0] @ w[:, 1] - a[1] @ w[:, 0]], -1)
    return out * coef


# ------------------------------------------------- differentiable velocity
def _dtype(case):
    return torch.float64 if case["precision"] == 64 else torch.float32


def _adjoint_inputs(case, seed):
    """A plan and its inputs, from the seed alone: neighbour lists within the
    support radius, a sixteenth (or more) of the particles as sources."""
    side = case["side"]
    x, g = _points(2, side, False, seed)
    n, h = x.shape[0], 2.0 / side
    perm = _slot_order(x, side, True)
    xs = x[perm]
    rows, cols, step = [], [], max(1, int(2e8 // n))
    for i in range(0, n, step):
        d = xs[i:i + step, None, :] - xs[None, :, :]
        d = d - torch.round(d)
        r2 = d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]
        a, b = torch.nonzero(r2 < h * h, as_tuple=True)
        keep = a + i != b
        rows.append(a[keep] + i)
        cols.append(b[keep])
    rows, cols = torch.cat(rows), torch.cat(cols)
    m = max(1, n // case["every"])
    src = torch.sort(torch.randperm(n, device="cuda", generator=g)[:m]).values

    def rand(k):
        return torch.rand(k, device="cuda", generator=g)

    c = 0.1592 * 1.25 * 0.8 / n
    p = {"perm": perm, "rows": rows, "cols": cols, "src": src, "src_a": 0.5 + rand(m),
         "f": (0.9 + 0.2 * rand(n)) * (c * n / m), "m_V": (0.9 + 0.2 * rand(n)) / n}
    w = _ring(x, g)[:, 2]
    gu = torch.randn(n, 2, device="cuda", generator=g)
    return x, w, gu, p


def _prepare_adjoint(case, seed):
    x, w, gu, p = _adjoint_inputs(case, seed)
    n, m = x.shape[0], p["src"].shape[0]
    cfg = _box_config(2, case["side"], periodic=True)
    cfg.config["Configuration"]["samplerMode"] = "stratified"
    box = VortexBox(cfg, x.cpu().numpy())
    plan = Plan(n, m, box.nbr_cap, device="cuda")
    t = plan.t
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(p["rows"], minlength=n), 0)
    if int(off[-1]) > box.nbr_cap:
        raise RuntimeError("the neighbour lists do not fit the plan")
    t["n_src"][0] = m
    t["perm"].copy_(p["perm"])
    t["inv_perm"][p["perm"]] = torch.arange(n, device="cuda", dtype=torch.int32)
    t["nbr_off"].copy_(off)
    t["nbr"][:p["cols"].shape[0]] = p["cols"].to(torch.int32)
    t["src"].copy_(p["src"])
    t["src_a"].copy_(p["src_a"])
    t["slot_src"].fill_(-1)
    t["slot_src"][p["src"]] = torch.arange(m, device="cuda", dtype=torch.int32)
    t["slot_a"].zero_()
    t["slot_a"][p["src"]] = p["src_a"]
    t["f"].copy_(p["f"])
    t["m_V"].copy_(p["m_V"])
    d = _dtype(case)
    return {"box": box, "plan": plan, "x": x.to(d).requires_grad_(True), "w": w.to(d).requires_grad_(True),
            "g": gu.to(d)}


def _run_adjoint(s):
    u = s["box"].velocity(s["x"], s["w"], s["plan"])
    gx, gw = torch.autograd.grad(u, (s["x"], s["w"]), s["g"])
    return {"u": u, "gx": gx, "gw": gw}


def _exact_adjoint(case, seed):
    x, w, gu, p = _adjoint_inputs(case, seed)
    n, perm = x.shape[0], p["perm"]
    h = 2.0 / case["side"]
    c = float(np.float32(0.1592 * 1.25 * 0.8 / case["side"] ** 2))
    kw = 1.8189 / (h * h)
    xs, ws = x[perm].double().requires_grad_(True), w[perm].double().requires_grad_(True)
    f, mv, a = p["f"].double(), p["m_V"].double(), p["src_a"].double()
    rows, cols, src = p["rows"], p["cols"], p["src"]
    slot_a = torch.zeros(n, dtype=torch.float64, device="cuda")
    slot_a[src] = a
    xc = x[perm].to(_dtype(case))  # the periodic image of a pair is taken in the case's own precision
    d = xs[rows] - xs[cols]
    d = d - torch.round(xc[rows] - xc[cols]).double()
    r = torch.sqrt((d * d).sum(1))
    q = r / h
    W = kw * torch.where(q <= 0.5, 6 * q ** 3 - 6 * q ** 2 + 1, 2 * (1 - q).clamp_min(0) ** 3)
    wt = (mv * kw * ws).index_add(0, rows, mv[cols] * W * ws[cols])
    e = torch.exp(-r / 1e-6)
    F = c * (1 - e) / (r * (r + 1e-6 * e)) - f[rows] * slot_a[cols] / (r * r)
    Fw = F * wt[cols]
    u = torch.zeros(n, 2, dtype=torch.float64, device="cuda")
    u = u.index_add(0, rows, torch.stack([Fw * d[:, 1], -Fw * d[:, 0]], 1))
    gs = gu[perm].double()
    total = torch.zeros(n, 2, dtype=torch.float64, device="cuda")
    wd, xd = wt.detach().requires_grad_(True), xs.detach().requires_grad_(True)
    gwt, gxf = torch.zeros_like(wd), torch.zeros_like(xd)
    step = max(1, int(5e7 // src.shape[0]))
    for i in range(0, n, step):
        d = xd[i:i + step, None, :] - xd[src][None, :, :]
        d = d - torch.round(xc[i:i + step, None, :] - xc[src][None, :, :]).double()
        dx, dy = d[..., 0], d[..., 1]
        r2 = dx * dx + dy * dy
        k = torch.where(r2 > 0, 1 / torch.where(r2 > 0, r2, torch.ones_like(r2)), torch.zeros_like(r2))
        b = a * wd[src]
        fu = f[i:i + step, None] * torch.stack([(k * dy) @ b, -((k * dx) @ b)], 1)
        total[i:i + step] = fu.detach()
        g1, g2 = torch.autograd.grad(fu, (wd, xd), gs[i:i + step])
        gwt += g1
        gxf += g2
    gx, gw = torch.autograd.grad([u, wt], (xs, ws), [gs, gwt])
    inv = torch.empty_like(perm)
    inv[perm] = torch.arange(n, device="cuda")
    return {"u": (u.detach() + total)[inv], "gx": (gx + gxf)[inv], "gw": gw[inv]}


def _prepare_adjoint_step(case, seed):
    x, g = _points(2, case["side"], False, seed)
    cfg = _box_config(2, case["side"], periodic=True)
    cfg.config["Configuration"]["samplerMode"] = "stratified"
    box = VortexBox(cfg, x.cpu().numpy(), mc_fraction=1.0 / case["every"])
    w = _ring(x, g)[:, 2].contiguous()
    # the velocity of the step before: it sets the sampling density
    k = 6.2831853
    v = torch.stack([torch.sin(k * x[:, 1]) + 0.3 * torch.cos(2 * k * x[:, 0]), torch.cos(k * x[:, 0])], 1)
    v = v + 0.05 * torch.randn(x.shape[0], 2, device="cuda", generator=g)
    d = _dtype(case)
    return {"box": box, "x": x.to(d).requires_grad_(True), "w": w.to(d).requires_grad_(True), "v": v.contiguous(),
            "g": torch.randn(x.shape[0], 2, device="cuda", generator=g).to(d)}


def _run_adjoint_step(s):
    box = s["box"]
    plan = box.build_plan(s["x"], s["v"], 3, MC, seed=5)
    u = box.velocity(s["x"], s["w"], plan)
    gx, gw = torch.autograd.grad(u, (s["x"], s["w"]), s["g"])
    return {"u": u, "gx": gx, "gw": gw, "perm": plan.perm, "f": plan.t["f"], "slot_a": plan.t["slot_a"]}


# ------------------------------------------------------------- the interface
_PREPARE = {"step": _prepare_step, "batch": _prepare_batch, "grid": _prepare_stage, "dfsph": _prepare_stage,
            "dimcv": _prepare_stage, "vvpe": _prepare_vvpe, "bs": _prepare_bs, "adjoint": _prepare_adjoint,
            "adjoint_step": _prepare_adjoint_step}
_RUN = {"step": _run_step, "batch": _run_batch, "grid": _run_grid, "dfsph": _run_dfsph, "dimcv": _run_dimcv,
        "vvpe": _run_vvpe, "bs": _run_bs, "adjoint": _run_adjoint, "adjoint_step": _run_adjoint_step}


def prepare(case, seed):
    torch.cuda.set_device(0)
    s = _PREPARE[case["kind"]](case, seed)
    s["run"] = _RUN[case["kind"]]
    return s


def run(state):
    return state["run"](state)


def exact(case, seed):
    if case["kind"] == "vvpe":
        return _exact_vvpe(case, seed)
    if case["kind"] == "bs":
        return _exact_bs(case, seed)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    return None


def _particles(case):
    """(fluid, all) particles of a channel or sphere scene."""
    d = 2 * case["radius"]
    if case["dim"] == 2:
        return 3.8 / (d * d), 4.0 / (d * d)
    return 1.04 / d ** 3, 1.04 / d ** 3 + 22.0 / (d * d)


def work(case):
    kind = case["kind"]
    # bytes per particle: every field of the stage read once and written once;
    # operations per neighbour pair and per (target, sample) pair of the sums
    if kind in ("step", "grid", "dfsph", "dimcv"):
        nf, n = _particles(case)
        nb, s = (12, 2 / 3) if case["dim"] == 2 else (28, 1.0)
        per, ops = {"grid": (192, 10), "dfsph": (372, 240), "dimcv": (230, 120), "step": (960, 500)}[kind]
        pairs = 0.0
        if kind == "step" and case["sampler"] != "bernoulli":
            pairs = nf * nf / (16 if case["dim"] == 2 else 32)
        return {"bytes": per * s * n, "flops": ops * nb * nf + pairs * (12 if case["dim"] == 2 else 24)}
    if kind == "batch":
        a, b = case["n_min"], case["n_max"]
        mean = (b - a) / math.log(b / a)
        square = (b * b - a * a) / (2 * math.log(b / a))
        return {"bytes": 2 * 640 * mean * case["scenes"],
                "flops": 2 * case["scenes"] * (500 * 12 * mean + 12 * square / 16)}
    if kind == "vvpe":
        n = case["side"] ** case["dim"]
        per = 27 if case["blob"] else (24 if case["dim"] == 3 else 12)
        return {"bytes": 100.0 * n, "flops": float(per) * n * (n // case["every"])}
    if kind == "bs":
        return {"bytes": 48.0 * case["n"], "flops": 27.0 * case["n"] ** 2}
    n = case["side"] ** 2
    per = 12 + 30  # the velocity, and both sides of its derivative
    size = case["precision"] // 8
    return {"bytes": size * 14.0 * n + 12 * 8.0 * n, "flops": per * float(n) * (n // case["every"]) + 12 * 120.0 * n}
