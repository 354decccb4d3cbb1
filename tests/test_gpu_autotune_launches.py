"""dv_autotune, which a solver calls on its first far field, times 32 forms with
68 launches of the loop (72 before it tried every chunk count) beside the few
that list targets and pack samples, and leaves a form that it timed."""
import ctypes as C

import pytest

from dimcv_sph_b200 import scenes

pytestmark = pytest.mark.gpu


def test_launches_of_the_first_call(cuda):
    from dimcv_sph_b200.particle_system import ParticleSystem
    ps = ParticleSystem(scenes.channel2d(length=2.0, reserved=200))
    solver = ps.build_solver()
    solver.initialize()
    solver.compute_densities()
    solver.init()
    solver.update_sample()
    solver.smooth_and_kernel_density()
    solver._calls("dv_sample", 1, 1, 1, 500)
    before = ps.lib.dv_launch_count(ps.ctx)
    tile, ms = C.c_int32(), C.c_float()
    solver._calls("dv_autotune", C.byref(tile), C.byref(ms))
    assert 68 <= ps.lib.dv_launch_count(ps.ctx) - before <= 72
    assert tile.value in (2, 4, 6, 8) and 0 < ms.value < 10
    assert 1 <= ps.lib.dv_get_far_chunks(ps.ctx) <= 8
