"""The neighbour-list builds (k_csr_rows in 3-D, k_csr_build in 2-D) where
their forms change: a periodic box, 1 to 13 particles a cell around the group
of 12, a particle with exactly 64 and 65 neighbours (a full row, a long one), pairs
within rounding of the support radius,
rows longer than 2-D's 32 slots, the part-filled last warp, lists too long for
their buffer and a material that the entries cannot hold (the sweeps then scan
cells).  Rows are whole numbers: equal to the oracle's."""
import numpy as np
import pytest

from dimcv_sph_b200.config_builder import SimConfig
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu
R = 1.0 / 64.0  # h = 1/16: 16 cells an axis


def system(dim, x, periodic=False, capacity=None, material=1):
    from dimcv_sph_b200.particle_system import ParticleSystem
    conf = {"domainStart": [0.0] * dim, "domainEnd": [1.0] * dim, "particleRadius": R, "density0": 1000,
            "simulationMethod": 0, "gravitation": [0.0] * dim, "timeStepSize": 1e-3, "volumeScale": 0.8,
            "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False, "periodic": periodic}
    n = len(x)
    ps = ParticleSystem(SimConfig(config={"Configuration": conf}), capacity=capacity or n)
    ps.add_particles(0, n, x.astype(np.float32), np.zeros((n, dim), np.float32), np.full(n, 1000.0), np.zeros(n),
                     np.full(n, material, np.int32), np.ones(n, np.int32), np.zeros((n, 3), np.int32))
    ps.initialize_particle_system()
    return ps


def oracle_lists(ps):
    o = OracleSim(ps.params, ps.particle_max_num, 0)
    o.load_snapshot(ps.snapshot(), ps.counters())
    o.counting_sort()
    assert np.array_equal(o.permutation(), np.arange(o.counters()["n"]))
    return o.neighbor_lists()


def crowded(dim, rng):
    """Cells of 1 to 13 particles, in every second cell of an axis."""
    rows = []
    for k, cell in enumerate(np.ndindex(*[8] * dim)):
        rows.append((2 * np.array(cell) + rng.uniform(0.05, 0.95, (1 + k % 13, dim))) / 16)
    return np.concatenate(rows)


def clump(dim, count, rng):
    return np.concatenate([0.53 + rng.uniform(0, 0.01, (count, dim)), rng.uniform(0.1, 0.4, (50, dim))])


def at_radius(dim, rng):
    """Pairs about h apart: their squared distances lie within rounding of its square."""
    a = rng.uniform(0.1, 0.9, (3000 if dim == 3 else 600, dim)).astype(np.float32)
    u = rng.normal(size=a.shape)
    return np.concatenate([a, a + u / np.linalg.norm(u, axis=1, keepdims=True) / 16])


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("shape", ["periodic", "crowded", "full row", "long row", "at radius", "one"])
def test_rows(cuda, dim, shape):
    rng = np.random.default_rng(7)
    full = 64 if dim == 3 else 32
    x = {"periodic": lambda: rng.uniform(0, 0.999, (3001, dim)), "crowded": lambda: crowded(dim, rng),
         "full row": lambda: clump(dim, full + 1, rng), "long row": lambda: clump(dim, full + 2, rng),
         "at radius": lambda: at_radius(dim, rng), "one": lambda: np.full((1, dim), 0.5)}[shape]()
    ps = system(dim, x, periodic=shape == "periodic", capacity=20000)
    off, nbr = (t.cpu().numpy() for t in ps.stored_neighbor_lists())
    ooff, onbr = oracle_lists(ps)
    assert np.array_equal(off, ooff) and np.array_equal(nbr, onbr)
    if shape in ("full row", "long row"):
        assert np.diff(off).max() == full + (shape == "long row")


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("why", ["length", "material"])
def test_lists_that_cannot_be_stored(cuda, dim, why):
    rng = np.random.default_rng(8)
    if why == "length":  # everything near everything: more entries than the buffer holds
        ps = system(dim, 0.53 + rng.uniform(0, 0.01, (400, dim)))
    else:
        ps = system(dim, rng.uniform(0, 0.2, (400, dim)), material=2)
    with pytest.raises(RuntimeError, match="no valid lists"):
        ps.stored_neighbor_lists()
    solver = ps.build_solver()
    solver.compute_densities()  # scans cells
    o = OracleSim(ps.params, ps.particle_max_num, 0)
    o.load_snapshot(ps.snapshot(), ps.counters())
    o.counting_sort()
    o.call("densities")
    n = ps.particle_num[None]
    assert np.array_equal(ps.density[:n].cpu().numpy(), o.snapshot()["density"][:n])
