"""The neighbour-list builds where their form depends on how the particles lie:
3-D warps whose slots lie in more cells than a warp handles together (each lane
then scans for its own particle, long rows among them) beside warps that work
cell by cell; 2-D scenes so dense that lists are counted before they are
written, with lists that fit all the same and lists that do not; 2-D rows longer
than a row in shared memory beside short ones.  Rows are whole numbers: equal to
the oracle's; densities of the sweeps that read or cannot read them too."""
import numpy as np
import pytest

from dimcv_sph_b200._lib import DimcvError
from dimcv_sph_b200.config_builder import SimConfig
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu


def system(x, cells, periodic=False):
    from dimcv_sph_b200.particle_system import ParticleSystem
    n, dim = x.shape
    ps = ParticleSystem(SimConfig(config={"Configuration": {
        "domainStart": [0.0] * dim, "domainEnd": [1.0] * dim, "particleRadius": 0.25 / cells, "density0": 1000,
        "simulationMethod": 0, "gravitation": [0.0] * dim, "timeStepSize": 1e-3, "volumeScale": 0.8,
        "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False, "periodic": periodic}}),
        capacity=n)
    ps.add_particles(0, n, x.astype(np.float32), np.zeros((n, dim), np.float32), np.full(n, 1000.0), np.zeros(n),
                     np.ones(n, np.int32), np.ones(n, np.int32), np.zeros((n, 3), np.int32))
    ps.initialize_particle_system()
    return ps


def check(ps, stored=True):
    o = OracleSim(ps.params, ps.particle_max_num, 0)
    o.load_snapshot(ps.snapshot(), ps.counters())
    o.counting_sort()
    n = o.counters()["n"]
    assert np.array_equal(o.permutation(), np.arange(n))
    off, nbr = o.neighbor_lists()
    if stored:
        goff, gnbr = (t.cpu().numpy() for t in ps.stored_neighbor_lists())
        assert np.array_equal(goff, off) and np.array_equal(gnbr, nbr)
    else:
        with pytest.raises(DimcvError, match="no valid lists"):
            ps.stored_neighbor_lists()
    ps.build_solver()._call("dv_densities_factor")
    o.call("densities")
    assert np.array_equal(ps.density[:n].cpu().numpy(), o.snapshot()["density"][:n])
    return np.diff(off)


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("per_cell", [0.05, 0.5, 1.2, 2.0, 8.0])
def test_sparse_to_dense_3d(cuda, per_cell, periodic):
    rng = np.random.default_rng(int(10 * per_cell))
    check(system(rng.uniform(0, 0.999, (int(per_cell * 12 ** 3) + 1, 3)), 12, periodic))


def test_long_rows_in_sparse_warps(cuda):
    """Clumps of 70 (long rows) and of 65 (a full row) among single particles."""
    rng = np.random.default_rng(0)
    x = [rng.uniform(0.02, 0.98, (900, 3))]
    for k, count in enumerate((70, 65, 70, 65)):
        x.append((np.array([3 * k + 1, 5, 7]) + 0.4 + rng.uniform(0, 0.2, (count, 3))) / 16)
    rows = check(system(np.concatenate(x), 16))
    assert rows.max() > 64 and np.median(rows) < 8


@pytest.mark.parametrize("per_cell,fits", [(5.0, True), (7.9, True), (14.0, False)])
def test_dense_2d(cuda, per_cell, fits):
    """7.9 a cell: more than the buffer's 24 entries a particle are expected
    (24.8), but the particles at the border of the box have fewer."""
    cells = 12
    rng = np.random.default_rng(3)
    rows = check(system(rng.uniform(0, 0.999, (int(per_cell * cells ** 2), 2)), cells), stored=fits)
    assert (rows.mean() <= 24) == fits and rows.max() > 24


def test_long_rows_beside_short_ones_2d(cuda):
    rng = np.random.default_rng(4)
    x = [rng.uniform(0.02, 0.98, (3000, 2)), 0.51 + rng.uniform(0, 0.01, (120, 2)), 0.2 + rng.uniform(0, 0.01, (34, 2))]
    rows = check(system(np.concatenate(x), 40))
    assert rows.max() > 100 and np.median(rows) < 10
