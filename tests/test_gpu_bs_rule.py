"""The full Biot-Savart sum's own choice between 4 and 8 targets a thread, at
counts where one of them leaves SMs idle: its time against the better of the
two (the other is 1.06 to 1.8 times slower there; the bound of 1.2 is between)."""
import ctypes as C

import numpy as np
import pytest
import torch

from dimcv_sph_b200.config_builder import SimConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [17000, 37000, 53865, 65536])
def test_choice(cuda, n):
    from dimcv_sph_b200.particle_system import ParticleSystem
    ps = ParticleSystem(SimConfig(config={"Configuration": {
        "domainStart": [-1.0] * 3, "domainEnd": [1.0] * 3, "particleRadius": 0.02, "density0": 1000,
        "timeStepSize": 1e-3, "gravitation": [0, 0, 0], "volumeScale": 1.0, "kernel3D": True,
        "cellOriginOffset": True, "skipCell0": False}}), capacity=n)
    x = np.random.default_rng(n).uniform(-0.9, 0.9, (n, 3)).astype(np.float32)
    ps.add_particles(0, n, x, np.zeros_like(x), np.full(n, 1000.0), np.zeros(n), np.ones(n, np.int32),
                     np.ones(n, np.int32), np.zeros((n, 3), np.int32))
    om = torch.randn(n, 4, device=ps.device)
    out = torch.zeros(n, 4, device=ps.device)

    def timed():
        best = float("inf")
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            assert ps.lib.dv_bs_full(ps.ctx, C.byref(ps.fields_struct), C.c_void_p(om.data_ptr()), None, n,
                                     C.c_void_p(out.data_ptr()), 32) == 0
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    own = timed()
    forced = []
    for tile in (4, 8):
        assert ps.lib.dv_set_far_tile(ps.ctx, tile) == 0
        forced.append(timed())
    assert own < 1.2 * min(forced), (own, forced)
