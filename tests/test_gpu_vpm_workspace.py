"""Scratch of the differentiable velocity: the partial sums of its two directions
share their place.  Forward, backward and forward again on one scratch buffer
give the same bits as on fresh ones."""
import pytest
import torch

from dimcv_sph_b200 import scenes

pytestmark = pytest.mark.gpu


def test_size(cuda):
    from dimcv_sph_b200.adjoint import VortexBox
    cfg, x, _ = scenes.periodic2d(16384, seed=0, dt=0.01)
    box = VortexBox(cfg, x)
    n, m = box.n, box.M
    assert m == 1024
    # sources and their gradients, and the larger direction's partial sums: the
    # backward one's, 32 chunks of three numbers a target
    sums = 4 * (3 * 32 * n)
    got = box.lib.dv_vpm_workspace_bytes(box.ctx, n, m, 32)
    assert sums < got < 1.1 * sums


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_shared_scratch(cuda, dtype):
    from dimcv_sph_b200.adjoint import VortexBox
    cfg, x, w = scenes.periodic2d(1600, seed=0, dt=0.01)
    box = VortexBox(cfg, x, mc_fraction=0.25)
    w = torch.from_numpy(w).cuda()
    plan = box.validate(box.build_plan(box.x0, box.initial_velocity(w), 1))
    gen = torch.Generator(device="cuda").manual_seed(0)
    g = torch.randn(box.n, 2, device="cuda", generator=gen).to(dtype)

    def both():
        xs, ws = box.x0.to(dtype).requires_grad_(True), w.to(dtype).requires_grad_(True)
        u = box.velocity(xs, ws, plan)
        return (u.detach().clone(), *torch.autograd.grad(u, (xs, ws), g))

    first = both()
    for _ in range(2):
        assert all(torch.equal(a, b) for a, b in zip(first, both()))
    box._ws.clear()
    assert all(torch.equal(a, b) for a, b in zip(first, both()))
