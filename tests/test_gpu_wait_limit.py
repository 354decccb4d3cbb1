"""A wait between blocks that runs out (dv_set_wait_limit; a limit of 0 reads
wants a neighbour tile's word at the first read, which the hundreds of tiles
here, on the GPU together, do not all find).  The calls go on with nothing:
every slot keeps its place, no cell, list, target or sample is made, every
stage of a step runs on that, and the host's next reads are errors.  After
dv_clear_status a build is the oracle's again."""
import ctypes as C

import numpy as np
import pytest
import torch

from dimcv_sph_b200._abi import DV_EWAIT, DV_WARN_WAIT, DvCounters
from dimcv_sph_b200._lib import DimcvError
from dimcv_sph_b200.config_builder import SimConfig
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,k", [(2, 840), (3, 74)])
def test_wait_that_runs_out(cuda, dim, k):
    from dimcv_sph_b200.particle_system import ParticleSystem
    d, n = 1.0 / k, k ** dim
    ps = ParticleSystem(SimConfig(config={"Configuration": {
        "domainStart": [0.0] * dim, "domainEnd": [1.0] * dim, "particleRadius": d / 2, "density0": 1000,
        "simulationMethod": 0, "gravitation": [0.0] * dim, "timeStepSize": 1e-5, "volumeScale": 0.8,
        "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False}}), capacity=n)
    rng = np.random.default_rng(dim)
    x = rng.uniform(0.01, 0.99, (n, dim)).astype(np.float32)
    v = rng.normal(0, 0.1, (n, dim)).astype(np.float32)
    ps.add_particles(0, n, x, v, np.full(n, 1000.0), np.zeros(n), np.ones(n, np.int32), np.ones(n, np.int32),
                     np.zeros((n, 3), np.int32))
    solver = ps.build_solver()
    before = ps.snapshot()
    assert ps.lib.dv_set_wait_limit(ps.ctx, 0) == 0
    ps.initialize_particle_system()
    c = DvCounters()
    assert ps.lib.dv_get_counters(ps.ctx, C.byref(c)) == DV_EWAIT
    assert c.status & DV_WARN_WAIT and c.n == n and c.n_fluid == n
    assert np.array_equal(ps.x[:n].cpu().numpy(), x) and np.array_equal(ps.v[:n].cpu().numpy(), v)
    for read in (ps.counters, ps.permutation, ps.neighbor_lists, ps.stored_neighbor_lists):
        with pytest.raises(DimcvError):
            read()
    solver.track_iterations = False
    for name in ("dv_densities_factor_change", "dv_scale_factor", "dv_density_adv"):
        solver._call(name, *((1.0,) if name == "dv_scale_factor" else ()))
    solver._call("dv_divergence_solve", None)
    for name, *args in (("dv_vorticity_dvort",), ("dv_kvn_sample", 1, 1, 1), ("dv_smooth_akde",), ("dv_record_samples",),
                        ("dv_sample", 1, 1, 1, n // 16), ("dv_vvpe_mc",), ("dv_vis",)):
        solver._calls(name, *args)
    om = torch.ones(n, 4, device=ps.device)
    out = torch.full((n, 4), float("nan"), device=ps.device)
    solver._call("dv_bs_full", C.c_void_p(om.data_ptr()), None, 64, C.c_void_p(out.data_ptr()), 32)
    solver._call("dv_pressure_solve", None)
    solver._call("dv_advect")
    torch.cuda.synchronize()
    assert ps.lib.dv_get_counters(ps.ctx, C.byref(c)) == DV_EWAIT
    assert c.n == n and c.n_targets == 0 and c.num_samples == 0
    assert bool((out[:64] == 0).all())
    # all clear: the particles as they were, and the oracle's order and lists
    assert ps.lib.dv_clear_status(ps.ctx) == 0 and ps.lib.dv_set_wait_limit(ps.ctx, 1 << 22) == 0
    ps.x[:n] = torch.from_numpy(x).to(ps.device)
    ps.initialize_particle_system()
    o = OracleSim(ps.params, ps.particle_max_num, 0)
    o.load_snapshot(before, {**ps.counters(), "n": n, "n_fluid": n, "n_solid": 0})
    o.initialize_particle_system()
    assert np.array_equal(ps.permutation(), o.permutation())
    off, nbr = (t.cpu().numpy() for t in ps.stored_neighbor_lists())
    ooff, onbr = o.neighbor_lists()
    assert np.array_equal(off, ooff) and np.array_equal(nbr, onbr)
    solver._calls("dv_record_samples")
    assert ps.counters()["status"] == 0
