"""A 3-D scene batch through the C ABI (the Python class builds 2-D channels):
every scene after three steps has the bits of the same scene stepped alone.  The
3-D sweeps gather packed copies of their fields, which the batch's Jacobi loops
keep current and the pressure solve takes over from the sweep before it."""
import ctypes as C

import numpy as np
import pytest
import torch

from dimcv_sph_b200._abi import DV_SAMPLE_INVERSE_CDF, DvBatchScene, DvSceneState
from dimcv_sph_b200.config_builder import SimConfig
from dimcv_sph_b200.fields import particle_fields, solver_fields
from dimcv_sph_b200.params import make_params

pytestmark = pytest.mark.gpu
FIELDS = ("x", "v", "density", "dfsph_factor", "density_adv", "material", "m_V", "life_time", "acceleration")
END = 0.5


def scene(k):
    """A block of fluid over a floor of static solids, in motion; its (config, arrays)."""
    d = 1.0 / 32.0
    cfg = SimConfig(config={"Configuration": {
        "domainStart": [0.0] * 3, "domainEnd": [END] * 3, "particleRadius": d / 2, "density0": 1000,
        "simulationMethod": 0, "gravitation": [0.0, -9.8, 0.0], "timeStepSize": 5e-4, "volumeScale": 0.8,
        "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False,
        "samplerMode": "inverse_cdf", "mcSamples": 1.0 / 16.0, "seed": 11 + k, "computeVis": False}})
    rng = np.random.default_rng(k)
    g = np.stack(np.meshgrid(np.arange(16), np.arange(2, 6 + 2 * k), np.arange(14 - k), indexing="ij"), -1)
    x = (g.reshape(-1, 3) + 0.5 + rng.uniform(-0.2, 0.2, (g.size // 3, 3))) * d
    floor = np.stack(np.meshgrid(np.arange(16), np.arange(2), np.arange(16), indexing="ij"), -1).reshape(-1, 3)
    floor = (floor + 0.5) * d
    v = rng.normal(0, 0.3, x.shape)
    return cfg, (x.astype(np.float32), v.astype(np.float32), floor.astype(np.float32))


def alone(cfg, arrays):
    from dimcv_sph_b200.particle_system import ParticleSystem
    x, v, floor = arrays
    ps = ParticleSystem(cfg, capacity=len(x) + len(floor))
    for pos, vel, material, dyn in ((x, v, 1, 1), (floor, np.zeros_like(floor), 0, 0)):
        m = len(pos)
        ps.add_particles(0, m, pos, vel, np.full(m, 1000.0), np.zeros(m), np.full(m, material, np.int32),
                         np.full(m, dyn, np.int32), np.zeros((m, 3), np.int32))
    solver = ps.build_solver()
    solver.initialize()
    solver.far_tile = 4  # one sample chunk, as in the batch
    return ps, solver


def test_scenes_equal_lone_runs(cuda):
    S, steps = 3, 3
    made = [scene(k) for k in range(S)]
    lone = [alone(*m) for m in made]
    counts = [ps.counters() for ps, _ in lone]
    cap = sum(c["n"] for c in counts)
    p = make_params(made[0][0])
    p.n_scenes = S
    lib, ps0 = lone[0][0].lib, lone[0][0]
    ctx = lib.dv_create(C.byref(p), cap, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert ctx, lib.dv_last_error(None)
    try:
        sets = [particle_fields(cap, 3, ps0.device), particle_fields(cap, 3, ps0.device)]
        sb = solver_fields(cap, 3, ps0.device)
        o = 0
        for s, (ps, _) in enumerate(lone):
            n = counts[s]["n"]
            for k, t in ps.fields.t.items():
                sets[0][k][o:o + n] = t[:n]
            sets[0]["object_id"][o:o + n] = s
            o += n
        nf = sum(c["n_fluid"] for c in counts)
        assert lib.dv_set_counts(ctx, cap, nf, cap - nf) == 0
        tab = (DvBatchScene * S)()
        for s in range(S):
            for d in range(3):
                tab[s].domain_end[d] = END
            tab[s].cap = counts[s]["n"]
            tab[s].emit_density, tab[s].emit_volume, tab[s].seed = 1000.0, float(ps0.m_V0), 11 + s
        assert lib.dv_batch_setup(ctx, tab, S, None, 0, 1.0 / 16.0, DV_SAMPLE_INVERSE_CDF) == 0, lib.dv_last_error(ctx)
        for k in range(steps):
            rc = lib.dv_batch_step(ctx, C.byref(sets[k % 2].struct), C.byref(sets[1 - k % 2].struct),
                                   C.byref(sb.struct))
            assert rc == 0, lib.dv_last_error(ctx)
        states = (DvSceneState * S)()
        done = C.c_int64()
        assert lib.dv_batch_read(ctx, states, S, C.byref(done)) == 0 and done.value == steps
        cur = sets[steps % 2]
        for s, (ps, solver) in enumerate(lone):
            for _ in range(steps):
                ps.initialize_particle_system()
                solver.substep()
            c, st = ps.counters(), states[s]
            n = c["n"]
            assert st.end - st.start == n and st.n_fluid == c["n_fluid"] and st.num_samples == c["num_samples"] > 0
            assert (st.iters_div, st.iters_p) == (c["iters_div"], c["iters_p"])
            for k in FIELDS:
                a = cur[k][st.start:st.end].cpu().numpy()
                assert np.array_equal(a, ps.fields[k][:n].cpu().numpy()), (s, k)
    finally:
        lib.dv_destroy(ctx)
