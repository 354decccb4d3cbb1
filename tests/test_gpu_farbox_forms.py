"""The far field on boxes in each of its launch forms, against FP64 sums and the
direct loop: few, some and many boxes (4, 2 and 1 sets of sample stripes a
class), many and few near parts, both kernels, a small and a large regularisation
length, weights of one ring and of random signs; and a cloud that fills
more boxes than there are buffers for, which takes the direct loop.

Tolerance: the scheme is used because its error is not above the direct loop's,
so its RMS error against FP64 has to lie below that of the same call's direct
loop with 8 sample chunks (the most accurate it has; 2e-7 to 1.5e-6 here).  The
polynomials' truncation is at most 3e-7 of the sum at the documented degrees;
with two degrees less in the first or second distance class the random weights
are above the bound."""
import ctypes as C

import numpy as np
import pytest
import torch

from dimcv_sph_b200.config_builder import SimConfig

pytestmark = pytest.mark.gpu
D = 1.0 / 32.0


def make(shape, keep, every, blob=False, delta=0.5, weights="ring", seed=1):
    """A share of a jittered lattice (boxes of 16 points an axis)."""
    from dimcv_sph_b200.dimcv_sph import DIMCVSPHSolver
    from dimcv_sph_b200.particle_system import ParticleSystem
    conf = {"domainStart": [0.0] * 3, "domainEnd": [k * D for k in shape], "particleRadius": D / 2, "density0": 1000,
            "simulationMethod": 0, "gravitation": [0.0] * 3, "timeStepSize": 1e-3, "volumeScale": 1.25,
            "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False, "kernel3D": blob,
            "blobDelta": delta * D}
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(k) for k in shape], indexing="ij"), -1).reshape(-1, 3)
    g = g[np.sort(rng.choice(len(g), int(keep * len(g)), replace=False))]
    x = ((g + 0.5 + rng.uniform(-0.3, 0.3, g.shape)) * D).astype(np.float32)
    n = len(x)
    ps = ParticleSystem(SimConfig(config={"Configuration": conf}), capacity=n)
    v = np.zeros_like(x)
    v[:, 0] = 100.0
    ps.add_particles(0, n, x, v, np.full(n, 1000.0), np.zeros(n), np.ones(n, np.int32), np.ones(n, np.int32),
                     np.zeros((n, 3), np.int32))
    solver = DIMCVSPHSolver(ps)
    solver.initialize()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    c = ps.x[:n] - ps.x[:n].mean(0)
    solver.d_vort_smoothed[:n] = (torch.randn(n, 3, device="cuda", generator=gen) if weights == "random" else
                                  torch.stack([-c[:, 1], c[:, 0], 0.1 * c[:, 2]], 1))
    solver.kinematic_vort_num[:n] = 0.5 + torch.rand(n, device="cuda", generator=gen)
    solver.compute_kernel_density()
    idx = torch.randint(n, (n // every,), device="cuda", generator=gen)
    solver.sample_idx[:len(idx)] = idx.to(torch.int32)
    solver.num_samples[None] = len(idx)
    solver.far_tile = 8
    assert ps.lib.dv_set_far_tile(ps.ctx, 8) == 0 and ps.lib.dv_set_far_chunks(ps.ctx, 8) == 0
    return ps, solver, idx


def run(ps, solver):
    """(v_vort, whether the boxes carried the far field)"""
    ps.lib.dv_profile(ps.ctx, 1)
    solver.vort2vel()
    calls = C.c_int64()
    assert ps.lib.dv_profile_far(ps.ctx, C.byref(calls), None) == 0
    ps.lib.dv_profile(ps.ctx, 0)
    return solver.v_vort[:ps.particle_num[None]].double(), calls.value == 1


def direct(ps, solver, idx):
    """The direct loop's result: a particle that is no sample, moved to another
    box, makes the call take it; and the rows that its move touches."""
    n = ps.particle_num[None]
    drawn = set(idx.tolist())
    t = next(i for i in range(n // 2, n) if i not in drawn)
    here, there = ps.x[t].clone(), ps.x[0].clone()
    ps.x[t] = there + torch.tensor([0.001, 0.0, 0.0], device="cuda")
    got, boxes = run(ps, solver)
    ps.x[t] = here
    assert not boxes
    x = ps.x[:n]
    return got, ((x - here).norm(dim=1) < 3 * D) | ((x - there).norm(dim=1) < 3 * D)


def exact(ps, solver, idx, pick, blob):
    """v_vort of the picked targets in FP64 (reference: dimcv_sph.py:649-719)."""
    P, n = ps.params, ps.particle_num[None]
    x, w = ps.x[:n], solver.d_vort_smoothed[:n].double()
    kden = ps.solver_buf.t["kden"][:n].double()
    total = float(np.float32(ps.counters()["kden_sum"]))
    d2, eps, coef = P.blob_delta2, P.eps, P.blob_coef if blob else P.vvpe_coef
    xs, ws = x[idx], w[idx] / (kden[idx] + 1e-8)[:, None]

    def cross(dd, k, wj):
        a, b, e = k * dd[..., 0], k * dd[..., 1], k * dd[..., 2]
        z = a @ wj[:, 1] - b @ wj[:, 0]
        if blob:
            return torch.stack([b @ wj[:, 2] - e @ wj[:, 1], e @ wj[:, 0] - a @ wj[:, 2], z], -1)
        return torch.stack([b @ wj[:, 2], -(a @ wj[:, 2]), z], -1)

    def rel(i, xj):  # FP32 differences decide who is near, as in the library
        d = x[i][:, None] - xj[None]
        r2 = d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]
        return x[i].double()[:, None] - xj.double()[None], r2 + d[..., 2] * d[..., 2]

    out = []
    for i in pick.split(64):
        dd, r2 = rel(i, x)
        nb = r2 < P.nbr_r2_limit
        S = nb.double() @ kden
        nb[torch.arange(len(i)), i] = False
        rn = torch.sqrt(dd[..., 0] ** 2 + dd[..., 1] ** 2)
        e = torch.exp(-rn / eps)
        k = ((dd * dd).sum(-1) + d2) ** -1.5 if blob else (1 - e) / (rn * (rn + eps * e))
        near = coef * cross(dd, torch.where(nb, k, 0.0), w)
        dd, r2 = rel(i, xs)
        far, rr = r2 > P.far_r2_limit, (dd * dd).sum(-1)
        k = torch.where(far, (rr + d2) ** -1.5 if blob else 1 / rr.clamp_min(1e-30), 0.0)
        out.append(near + coef * cross(dd, k, ws) * ((total - S) / far.sum(1).clamp_min(1))[:, None])
    return torch.cat(out)


FORMS = {"few boxes": dict(shape=(96, 32, 24), keep=1.0, every=8),
         "some boxes": dict(shape=(128, 64, 64), keep=0.4, every=16),
         "many boxes": dict(shape=(128, 128, 128), keep=0.38, every=64)}


@pytest.mark.parametrize("weights", ["ring", "random"])
@pytest.mark.parametrize("blob", [False, True])
@pytest.mark.parametrize("form", FORMS)
def test_error_below_the_direct_loops(cuda, form, blob, weights):
    check(**FORMS[form], blob=blob, weights=weights)


@pytest.mark.parametrize("delta", [0.05, 4.0])
def test_regularisation_length(cuda, delta):
    check(**FORMS["some boxes"], blob=True, delta=delta)


def check(**case):
    ps, solver, idx = make(**case)
    n = ps.particle_num[None]
    box, on = run(ps, solver)
    assert on, "the boxes were not used"
    loop, touched = direct(ps, solver, idx)
    pick = torch.randperm(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))[:1024]
    pick = pick[~touched[pick]]
    ref = exact(ps, solver, idx, pick, case["blob"])

    def rms(a):
        return float((a[pick] - ref).norm() / ref.norm())

    assert rms(box) < rms(loop) < 1e-5, (rms(box), rms(loop))


def test_more_boxes_than_buffers(cuda):
    """256 boxes with targets, buffers for 136 (a 1,536th of the capacity)."""
    ps, solver, _ = make(shape=(128, 128, 64), keep=0.2, every=8)
    got, on = run(ps, solver)
    assert not on and bool(torch.isfinite(got).all()) and bool(got.any())
