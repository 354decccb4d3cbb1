"""The one-launch scans, compactions and sort passes (dv_lookback.cuh,
dv_grid.cu) at the sizes where their tiles and forms change: one element, the
edges of a block and of a tile, the narrow and wide forms of the scans
(131,072) and of the sort (296 and 592 tiles of 2,048 on 148 SMs, where the
keys kernel and the passes change), all in one cell, half of them inactive.
Order, lists and sample slots are whole numbers: equal to the oracle's."""
import numpy as np
import pytest
import torch

from dimcv_sph_b200.config_builder import SimConfig
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu


def scatter(n, clump=False, outside=0.0, seed=3):
    """n fluid particles at random in a square of one per spacing squared; a
    fraction beyond the domain's end (they turn inactive, sort last)."""
    from dimcv_sph_b200.dimcv_sph import DIMCVSPHSolver
    from dimcv_sph_b200.particle_system import ParticleSystem
    d = 1.0 / 32.0
    k = max(8, int(np.ceil(np.sqrt(n))))
    conf = {"domainStart": [0.0, 0.0], "domainEnd": [k * d, k * d], "particleRadius": d / 2, "density0": 1000,
            "simulationMethod": 0, "gravitation": [0.0, 0.0], "timeStepSize": 1e-3, "volumeScale": 0.8,
            "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False}
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.1 * d, (k - 0.1) * d, (n, 2))
    if clump:
        x = (k // 2 + 0.5 + 0.2 * rng.uniform(-1, 1, (n, 2))) * d
    x[rng.uniform(size=n) < outside] += k * d
    ps = ParticleSystem(SimConfig(config={"Configuration": conf}), capacity=n)
    ps.add_particles(0, n, x.astype(np.float32), np.zeros((n, 2), np.float32), np.full(n, 1000.0), np.zeros(n),
                     np.ones(n, np.int32), np.ones(n, np.int32), np.zeros((n, 3), np.int32))
    return ps, DIMCVSPHSolver(ps)


@pytest.mark.parametrize("n,outside", [(1, 0), (255, 0), (257, 0.5), (2047, 0), (2048, 0.5), (2049, 0), (131071, 0),
                                       (131073, 0.5), (296 * 2048 - 1, 0), (592 * 2048, 0), (592 * 2048 + 1, 0.25)])
def test_order_lists_and_compaction(cuda, n, outside):
    ps, solver = scatter(n, outside=outside)
    o = OracleSim(ps.params, ps.particle_max_num, 0)
    o.load_snapshot(ps.snapshot(), ps.counters())
    for _ in range(2):  # the second build finds what the first one left of the state
        ps.initialize_particle_system()
        o.initialize_particle_system()
        assert np.array_equal(ps.permutation(), o.permutation())
    m = ps.particle_num[None]
    assert m == o.counters()["n"] and (m < n) == (outside > 0)
    off, nbr = (t.cpu().numpy() for t in ps.stored_neighbor_lists())
    ooff, onbr = o.neighbor_lists()
    assert np.array_equal(off, ooff) and np.array_equal(nbr, onbr)
    pick = np.random.default_rng(n).uniform(size=m) < 0.5
    pick[-1] = True
    for flags in (pick, np.zeros(m, bool), np.ones(m, bool)):
        ps.is_sample[:m] = torch.from_numpy(flags).to(ps.is_sample)
        solver._calls("dv_record_samples")
        want = np.flatnonzero(flags)
        assert solver.num_samples[None] == len(want)
        assert np.array_equal(solver.sample_idx[:len(want)].cpu().numpy(), want)
    assert ps.counters()["status"] == 0


def test_sort_of_one_cell_is_the_identity(cuda):
    n = 5000
    ps, _ = scatter(n, clump=True)
    ps.initialize_particle_system()
    assert np.array_equal(ps.permutation(), np.arange(n))
