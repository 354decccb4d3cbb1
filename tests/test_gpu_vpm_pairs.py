"""The FP32 pair kernels of the differentiable velocity (two targets in each
64-bit register, narrow and wide tiles, source chunks) against a plain FP64
evaluation of the same plan with torch's derivatives: part-filled tiles on both
sides of the width switch at 8,192 targets, one source up to every particle,
and the three image modes.  The reference takes each pair's periodic image
from the FP32 difference, as the FP32 kernels do: a pair half a box apart has
either image, and the two differ by their whole term.

Tolerance: both sides sum at most 2e4 terms; FP32 rounding of such sums with
random signs stays near 1e-6 of the result's norm (2e-6 measured for the
gradients, whose near terms cancel), so 2e-5 of the norm."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
RTOL = 2e-5


def make(k, fraction):
    from dimcv_sph_b200 import scenes
    from dimcv_sph_b200.adjoint import VortexBox
    cfg, x, w = scenes.periodic2d(k * k, seed=k, dt=0.01)
    return VortexBox(cfg, x, mc_fraction=fraction), torch.from_numpy(w).cuda()


def reference(box, w, plan, gu, periodic):
    """(u, gx, gw) of the plan's step (formulas: dv_vpm.cu) in FP64."""
    P, t = box.ps.params, plan.t
    n, ns, nnz = plan.n, plan.n_src, plan.nnz
    perm = plan.perm.long()
    x32 = box.x0.index_select(0, perm)
    xs = x32.double().requires_grad_(True)
    ws = w.double().index_select(0, perm).requires_grad_(True)
    gs = gu.double().index_select(0, perm)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), t["nbr_off"].diff().long())
    cols, src = t["nbr"][:nnz].long(), t["src"][:ns].long()
    f, a, mv, slot_a = (t[k].double() for k in ("f", "src_a", "m_V", "slot_a"))
    a = a[:ns]
    h, kw, c = 1.0 / P.inv_support_radius, P.kW, P.vvpe_coef

    def image(d):
        return torch.round(d).double() if periodic else 0.0

    d = xs[rows] - xs[cols] - image(x32[rows] - x32[cols])
    r = torch.sqrt((d * d).sum(1))
    q = r / h
    W = kw * torch.where(q <= 0.5, 6 * q ** 3 - 6 * q ** 2 + 1, 2 * (1 - q).clamp_min(0) ** 3)
    wt = (mv * kw * ws).index_add(0, rows, mv[cols] * W * ws[cols])
    e = torch.exp(-r * 1e6)
    Fw = (c * (1 - e) / (r * (r + 1e-6 * e)) - f[rows] * slot_a[cols] / (r * r)) * wt[cols]
    u = torch.zeros(n, 2, dtype=torch.float64, device="cuda")
    u = u.index_add(0, rows, torch.stack([Fw * d[:, 1], -Fw * d[:, 0]], 1))
    total = u.detach().clone()
    wd, xd = wt.detach().requires_grad_(True), xs.detach().requires_grad_(True)
    gwt, gxf = torch.zeros_like(wd), torch.zeros_like(xd)
    step = max(1, int(2e7 // ns))
    for i in range(0, n, step):
        d = xd[i:i + step, None] - xd[src][None] - image(x32[i:i + step, None] - x32[src][None])
        r2 = (d * d).sum(-1)
        k = torch.where(r2 > 0, 1 / torch.where(r2 > 0, r2, torch.ones_like(r2)), torch.zeros_like(r2))
        b = a * wd[src]
        fu = f[i:i + step, None] * torch.stack([(k * d[..., 1]) @ b, -((k * d[..., 0]) @ b)], 1)
        total[i:i + step] += fu.detach()
        g1, g2 = torch.autograd.grad(fu, (wd, xd), gs[i:i + step])
        gwt += g1
        gxf += g2
    gx, gw = torch.autograd.grad([u, wt], (xs, ws), [gs, gwt])
    inv = plan.inv_perm.long()
    return total[inv], (gx + gxf)[inv], gw[inv]


def check(box, w, plan, frozen=False, periodic=True):
    g = torch.randn(box.n, 2, device="cuda", generator=torch.Generator(device="cuda").manual_seed(0))
    x, q = box.x0.clone().requires_grad_(True), w.clone().requires_grad_(True)
    u = box.velocity(x, q, plan, frozen)
    got = (u.detach(), *torch.autograd.grad(u, (x, q), g))
    for name, s, t in zip(("u", "gx", "gw"), got, reference(box, w, plan, g, periodic)):
        err = float((s.double() - t).norm() / t.norm())
        assert err < RTOL, (name, err)


@pytest.mark.parametrize("k,fraction", [(11, 1.0), (11, 0.004), (33, 0.25), (90, 0.004), (91, 1.0 / 16.0), (91, 1.0),
                                        (128, 0.05)])
def test_fp32_pairs_match_fp64(cuda, k, fraction):
    from dimcv_sph_b200.adjoint import FULL, MC
    box, w = make(k, fraction)
    v = box.initial_velocity(w)
    plan = box.validate(box.build_plan(box.x0, v, 1, FULL if fraction == 1.0 else MC))
    assert 1 <= plan.n_src <= box.n
    check(box, w, plan)


@pytest.mark.parametrize("k", [33, 91])
def test_fp32_pairs_image_modes(cuda, k):
    """Nominal images (a kept plan) and no images (a box that is not periodic)."""
    box, w = make(k, 1.0 / 8.0)
    v = box.initial_velocity(w)
    plan = box.validate(box.build_plan(box.x0, v, 1))
    plan.xbar = box.x0.index_select(0, plan.perm).clone()
    check(box, w, plan, frozen=True)
    box.ps.params.periodic = 0
    assert box.lib.dv_set_params(box.ctx, C.byref(box.ps.params)) == 0
    check(box, w, plan, periodic=False)
