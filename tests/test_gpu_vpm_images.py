"""Which periodic image the FP32 pair kernels of the differentiable velocity
take for pairs half a box apart: rint of the rounded product of the difference
and 1/L, as the scalar FP32 kernels and the FP64 ones do.  On a lattice in a box
of length 3 the product of 1.5 and the FP32 1/3 is a little above a half and
rounds to a half; rint of the unrounded product would give those pairs the
other image, which turns their term round.  Narrow tiles (1,024 particles) and
wide ones (9,216), minimum and nominal images.

Tolerance: as the other tests of these kernels against FP64, 2e-5 of the norm;
one flipped pair a target is some 1e-2 of it."""
import numpy as np
import pytest
import torch

from dimcv_sph_b200.config_builder import SimConfig

pytestmark = pytest.mark.gpu
RTOL = 2e-5


@pytest.mark.parametrize("k", [32, 96])
@pytest.mark.parametrize("frozen", [False, True])
def test_half_box_pairs(cuda, k, frozen):
    from dimcv_sph_b200.adjoint import FULL, VortexBox
    sp = 3.0 / k  # exact, and so are all differences
    cfg = SimConfig(config={"Configuration": {
        "domainStart": [0.0, 0.0], "domainEnd": [3.0, 3.0], "particleRadius": sp / 2, "density0": 1000,
        "simulationMethod": 0, "gravitation": [0.0, 0.0], "timeStepSize": 1e-3, "volumeScale": 1.25,
        "GenProbPara": 5, "DelProbPara": 3.5, "periodic": True, "samplerMode": "stratified", "seed": 0}})
    x = np.stack(np.meshgrid(np.arange(k), np.arange(k), indexing="ij"), -1).reshape(-1, 2) * sp
    box = VortexBox(cfg, x.astype(np.float32))
    assert np.float32(1.5) * np.float32(1 / 3) == 0.5 and 1.5 * float(np.float32(1 / 3)) > 0.5
    gen = torch.Generator(device="cuda").manual_seed(k)
    w = torch.randn(box.n, device="cuda", generator=gen)
    g = torch.randn(box.n, 2, device="cuda", generator=gen)
    plan = box.validate(box.build_plan(box.x0, None, 0, FULL))
    plan.xbar = box.x0.index_select(0, plan.perm).clone() if frozen else None
    out = {}
    for t in (torch.float32, torch.float64):
        xs, ws = box.x0.to(t).requires_grad_(True), w.to(t).requires_grad_(True)
        u = box.velocity(xs, ws, plan, frozen)
        out[t] = (u.detach(), *torch.autograd.grad(u, (xs, ws), g.to(t)))
    for name, a, b in zip(("u", "gx", "gw"), out[torch.float32], out[torch.float64]):
        err = float((a.double() - b).norm() / b.norm())
        assert err < RTOL, (name, err)
