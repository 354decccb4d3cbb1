"""A particle of a material that list entries cannot hold (neither fluid nor
solid), in 3-D: the lists are off where it is a neighbour of a built row, also
when only a lane past the end of the particles tests it, and stay on where it
merely lies in the 27 cells around one.  Density and factor are the oracle's."""
import numpy as np
import pytest

from dimcv_sph_b200._lib import DimcvError
from dimcv_sph_b200.config_builder import SimConfig
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu
CELL = 1.0 / 16.0  # h


def system(groups):
    """groups: (positions in cells, material, dynamic)"""
    from dimcv_sph_b200.particle_system import ParticleSystem
    n = sum(len(g[0]) for g in groups)
    ps = ParticleSystem(SimConfig(config={"Configuration": {
        "domainStart": [0.0] * 3, "domainEnd": [1.0] * 3, "particleRadius": CELL / 4, "density0": 1000,
        "simulationMethod": 0, "gravitation": [0.0] * 3, "timeStepSize": 1e-3, "volumeScale": 0.8,
        "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False}}), capacity=n)
    for x, material, dyn in groups:
        m = len(x)
        ps.add_particles(0, m, (np.asarray(x) * CELL).astype(np.float32), np.zeros((m, 3), np.float32),
                         np.full(m, 1000.0), np.zeros(m), np.full(m, material, np.int32), np.full(m, dyn, np.int32),
                         np.zeros((m, 3), np.int32))
    ps.initialize_particle_system()
    return ps


def listed(ps):
    try:
        ps.stored_neighbor_lists()
        return True
    except DimcvError:
        return False


def check_sweep(ps):
    solver = ps.build_solver()
    o = OracleSim(ps.params, ps.particle_max_num, 0)
    o.load_snapshot(ps.snapshot(), ps.counters())
    o.counting_sort()
    solver._call("dv_densities_factor")
    o.call("densities")
    o.call("dfsph_factor")
    ref, n = o.snapshot(), ps.particle_num[None]
    for k in ("density", "dfsph_factor"):
        assert np.array_equal(getattr(ps, k)[:n].cpu().numpy(), ref[k][:n]), k


def spread(count):
    """Particles alone in cells of the low corner."""
    return [(2 * (k % 4) + 0.5, 2 * (k // 4 % 4) + 0.5, 2 * (k // 16) + 0.5) for k in range(count)]


def test_seen_by_a_lane_past_the_end(cuda):
    # the last warp holds a fluid particle and the odd one; the candidates before
    # them are static solids, whose own rows are not built
    solids = [(14.5 + 0.02 * k, 15.5, 15.5) for k in range(10)]
    ps = system([(spread(20), 1, 1), (solids, 0, 0), ([(15.1, 15.5, 15.5), (15.3, 15.5, 15.5)], 1, 1)])
    n = ps.particle_num[None]
    last = ps.x[n - 1].cpu().numpy() / CELL
    assert n % 32 == 0 and abs(last[0] - 15.3) < 1e-4
    ps = system([(spread(22), 1, 1), (solids, 0, 0), ([(15.1, 15.5, 15.5)], 1, 1), ([(15.3, 15.5, 15.5)], 2, 1)])
    n = ps.particle_num[None]
    last = ps.x[n - 1].cpu().numpy() / CELL
    assert n % 32 == 2 and abs(last[0] - 15.3) < 1e-4 and int(ps.material[n - 1]) == 2
    assert not listed(ps)
    check_sweep(ps)


@pytest.mark.parametrize("gap", [0.9, 1.1])
def test_within_and_beyond_the_support_radius(cuda, gap):
    ps = system([(spread(40), 1, 1), ([(12.95, 12.5, 12.5)], 1, 1), ([(12.95 + gap, 12.5, 12.5)], 2, 1)])
    assert listed(ps) == (gap > 1)
    check_sweep(ps)
