"""A context whose calls move between two streams, each ordered behind the other
by an event (dv_set_stream): scans, compactions, sort, solves and vortex sums
give the bits of one stream."""
import ctypes as C

import numpy as np
import pytest
import torch

from dimcv_sph_b200 import scenes

pytestmark = pytest.mark.gpu


def steps(streams):
    from dimcv_sph_b200.particle_system import ParticleSystem
    ps = ParticleSystem(scenes.channel2d(length=2.0, reserved=200))
    solver = ps.build_solver()
    solver.far_tile = 4
    main = torch.cuda.current_stream()
    turn = [0]

    def move():
        if not streams:
            return
        new, old = streams[turn[0] % 2], streams[(turn[0] + 1) % 2] if turn[0] else main
        new.wait_event(old.record_event())
        assert ps.lib.dv_set_stream(ps.ctx, C.c_void_p(new.cuda_stream)) == 0
        turn[0] += 1

    solver.initialize()
    for _ in range(3):
        for stage in (ps.initialize_particle_system, solver.compute_densities, solver.compute_DFSPH_factor,
                      solver.divergence_solve, solver.compute_non_pressure_forces, solver.dimcv,
                      solver.predict_velocity, solver.pressure_solve, solver.advect):
            move()
            stage()
    torch.cuda.synchronize()
    ps.counters()  # an error if a wait had run out
    return ps.snapshot()


def test_two_ordered_streams(cuda):
    a, b = steps(None), steps([torch.cuda.Stream(), torch.cuda.Stream()])
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k
