"""dv_launch_count counts every kernel: a 3-D sweep and the pass that packs its
fields are two, a 2-D sweep is one; dv_sweep_count counts both as one.  The
profiler's list of kernels agrees."""
import pytest
import torch

from dimcv_sph_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_launches_are_kernels(cuda, dim):
    from dimcv_sph_b200.particle_system import ParticleSystem
    ps = ParticleSystem(scenes.channel2d(length=2.0, reserved=200) if dim == 2 else
                        scenes.sphere3d(radius=0.016, dt=6.4e-4))
    solver = ps.build_solver()
    solver.initialize()
    calls = [lambda: solver._call("dv_densities_factor_change"), lambda: solver._call("dv_density_adv"),
             lambda: solver._call("dv_divergence_iteration"), lambda: solver._calls("dv_vorticity_dvort")]
    torch.cuda.synchronize()
    l0, s0 = ps.lib.dv_launch_count(ps.ctx), ps.lib.dv_sweep_count(ps.ctx)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        for f in calls:
            f()
        torch.cuda.synchronize()
    launches = ps.lib.dv_launch_count(ps.ctx) - l0
    assert launches == len(calls) * (dim - 1)
    assert ps.lib.dv_sweep_count(ps.ctx) - s0 == len(calls)
    kernels = [e.name for e in prof.events() if "k_" in e.name]
    assert len(kernels) == launches, kernels
