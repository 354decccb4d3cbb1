"""So many particles in one cell that the number of list entries wraps in 32
bits: 65,537 x 65,536 in 2-D is 2^32 + 65,536, which passed for lists that fit;
131,200 rows of 32,800 quads in 3-D pass 2^32.  Such lists are refused, and the
sweeps scan cells: the density of n coincident particles, the same FP32 sum.
And long rows beyond the room for long rows (51 entries a particle in all), while
every other row fits: densities and factors are the oracle's cell scans."""
import numpy as np
import pytest

from dimcv_sph_b200._lib import DimcvError
from dimcv_sph_b200.config_builder import SimConfig
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu


def system(dim, x):
    from dimcv_sph_b200.particle_system import ParticleSystem
    n = len(x)
    ps = ParticleSystem(SimConfig(config={"Configuration": {
        "domainStart": [0.0] * dim, "domainEnd": [1.0] * dim, "particleRadius": 1.0 / 64.0, "density0": 1000,
        "simulationMethod": 0, "gravitation": [0.0] * dim, "timeStepSize": 1e-3, "volumeScale": 0.8,
        "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False}}), capacity=n)
    ps.add_particles(0, n, x, np.zeros_like(x), np.full(n, 1000.0), np.zeros(n), np.ones(n, np.int32),
                     np.ones(n, np.int32), np.zeros((n, 3), np.int32))
    ps.initialize_particle_system()
    return ps, ps.build_solver()


@pytest.mark.parametrize("clump", [300, 400])
def test_room_for_long_rows(cuda, clump):
    rng = np.random.default_rng(clump)
    x = np.concatenate([0.53 + rng.uniform(0, 0.01, (clump, 3)), rng.uniform(0.05, 0.95, (2000 - clump, 3))])
    ps, solver = system(3, x.astype(np.float32))
    o = OracleSim(ps.params, ps.particle_max_num, 0)
    o.load_snapshot(ps.snapshot(), ps.counters())
    o.counting_sort()
    off, _ = o.neighbor_lists()
    rows = np.diff(off)
    long = int(((rows[rows > 64] + 3) // 4 * 4).sum())
    assert (long > 51 * 2000) == (clump == 400) and (rows <= 64).sum() > 1000
    if clump == 400:
        with pytest.raises(DimcvError, match="no valid lists"):
            ps.stored_neighbor_lists()
    else:
        assert np.array_equal(ps.stored_neighbor_lists()[0].cpu().numpy(), off)
    solver._call("dv_densities_factor")
    o.call("densities")
    o.call("dfsph_factor")
    ref = o.snapshot()
    for k in ("density", "dfsph_factor"):
        assert np.array_equal(getattr(ps, k)[:2000].cpu().numpy(), ref[k][:2000]), k


@pytest.mark.parametrize("dim,n", [(2, 65537), (3, 131200)])
def test_lists_longer_than_32_bits(cuda, dim, n):
    ps, solver = system(dim, np.full((n, dim), 0.53, np.float32))
    with pytest.raises(DimcvError, match="no valid lists"):
        ps.stored_neighbor_lists()
    with pytest.raises(DimcvError, match="pairs"):
        ps.neighbor_lists()
    solver.compute_densities()
    # n coincident particles: rho0 m_V (1 + (n - 1)) W(0), the sum in FP32 one by one
    P, m_V = ps.params, float(ps.m_V[0])
    w = np.float32(m_V) * np.float32(P.kW)
    den = np.add.accumulate(np.full(n - 1, w, np.float32), dtype=np.float32)[-1]
    want = (w + den) * np.float32(P.density0)
    got = ps.density[:n].cpu().numpy()
    assert np.all(got == got[0]) and abs(float(got[0]) - float(want)) < 1e-6 * float(want)
