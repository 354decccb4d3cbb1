"""The full Biot-Savart sum while no far-field tile has been chosen: 4 or 8
targets a thread by the target count, at the edges of both tiles, against the
FP64 sum of the same call.  Tolerance: the contract of the N-body sums, 1e-5 of
the largest component."""
import ctypes as C

import numpy as np
import pytest
import torch

from dimcv_sph_b200.config_builder import SimConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [1, 1024, 1025, 2048, 2049, 3000])
def test_untuned_tile(cuda, nt):
    from dimcv_sph_b200.particle_system import ParticleSystem
    n = 3000
    rng = np.random.default_rng(nt)
    cfg = SimConfig(config={"Configuration": {
        "domainStart": [-1.0] * 3, "domainEnd": [1.0] * 3, "particleRadius": 0.02, "density0": 1000,
        "timeStepSize": 1e-3, "gravitation": [0, 0, 0], "volumeScale": 1.0, "kernel3D": True,
        "cellOriginOffset": True, "skipCell0": False, "reservedCapacity": n}})
    ps = ParticleSystem(cfg)
    x = rng.uniform(-0.9, 0.9, size=(n, 3)).astype(np.float32)
    ps.add_particles(0, n, x, np.zeros_like(x), np.full(n, 1000.0), np.zeros(n), np.ones(n, np.int32),
                     np.ones(n, np.int32), np.zeros((n, 3), np.int32))
    om = torch.from_numpy(rng.normal(size=(ps.particle_max_num, 4)).astype(np.float32)).to(ps.device)
    tl = torch.from_numpy(rng.permutation(n)[:nt].astype(np.int32)).to(ps.device)
    out = {}
    for prec, dt in ((32, torch.float32), (64, torch.float64)):
        out[prec] = torch.zeros(nt, 4, dtype=dt, device=ps.device)
        rc = ps.lib.dv_bs_full(ps.ctx, C.byref(ps.fields_struct), C.c_void_p(om.data_ptr()),
                               C.c_void_p(tl.data_ptr()), nt, C.c_void_p(out[prec].data_ptr()), prec)
        assert rc == 0, ps.lib.dv_last_error(ps.ctx)
    a, b = out[32][:, :3].double(), out[64][:, :3]
    assert float((a - b).abs().max() / b.abs().max()) < 1e-5
