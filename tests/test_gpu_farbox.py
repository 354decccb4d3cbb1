"""The 3-D far field by interpolation on boxes (dv_farbox.cu) against the CPU
oracle's FP64 sums, at the shapes where its boxes can go wrong: part-filled
boxes, axes of fewer cells than a box, samples drawn several times, targets in
part of the domain; and the calls that have to take the direct loop instead.

Tolerance: the contract of the N-body sums, 1e-5 of the largest component.
The scheme adds to the FP32 sums' 2e-7 to 4e-7 the truncation of its
polynomials, at most 3e-7 of the sum (RMS, random weights)."""
import ctypes as C

import numpy as np
import pytest
import torch

from dimcv_sph_b200.config_builder import SimConfig
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu
RTOL = 1e-5


def make(shape, every, blob=False, vortex_domain=None, origin=0.0, seed=0):
    """A jittered lattice of fluid (spacing 1/32) with random vorticity, KVN and
    draws (with replacement), sorted, with the kernel density computed."""
    from dimcv_sph_b200.dimcv_sph import DIMCVSPHSolver
    from dimcv_sph_b200.particle_system import ParticleSystem
    d = 1.0 / 32.0
    conf = {"domainStart": [origin] * 3, "domainEnd": [origin + k * d for k in shape], "particleRadius": d / 2,
            "density0": 1000, "simulationMethod": 0, "gravitation": [0.0] * 3, "timeStepSize": 1e-3,
            "volumeScale": 1.25, "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False,
            "kernel3D": blob, "blobDelta": d / 2}
    if vortex_domain:
        conf["vortexEnforcingDomainStart"], conf["vortexEnforcingDomainEnd"] = vortex_domain
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(k) for k in shape], indexing="ij"), -1).reshape(-1, 3)
    x = ((g + 0.5 + rng.uniform(-0.3, 0.3, g.shape)) * d + origin).astype(np.float32)
    n = len(x)
    ps = ParticleSystem(SimConfig(config={"Configuration": conf}), capacity=n)
    v = np.zeros_like(x)
    v[:, 0] = 100.0
    ps.add_particles(0, n, x, v, np.full(n, 1000.0), np.zeros(n), np.ones(n, np.int32), np.ones(n, np.int32),
                     np.zeros((n, 3), np.int32))
    solver = DIMCVSPHSolver(ps)
    solver.initialize()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    solver.d_vort_smoothed[:n] = torch.randn(n, 3, device="cuda", generator=gen)
    solver.kinematic_vort_num[:n] = 0.5 + torch.rand(n, device="cuda", generator=gen)
    solver.compute_kernel_density()
    M = n // every
    idx = torch.randint(n, (M,), device="cuda", generator=gen)
    if vortex_domain:  # draws come from the targets
        idx = idx[torch.from_numpy(np.all((ps.x[:n].cpu().numpy() >= vortex_domain[0]) &
                                          (ps.x[:n].cpu().numpy() <= vortex_domain[1]), axis=1)).to("cuda")[idx]]
    idx[:5] = idx[0]  # one particle drawn five times
    solver.sample_idx[:len(idx)] = idx.to(torch.int32)
    solver.num_samples[None] = len(idx)
    solver.far_tile = 8
    return ps, solver, idx


def run(ps, solver):
    """vort2vel; returns (v_vort, pair evaluations of the far field)."""
    ps.lib.dv_profile(ps.ctx, 1)
    solver.vort2vel()
    ms, launches, pairs = C.c_double(), C.c_int64(), C.c_double()
    ps.lib.dv_profile_read(ps.ctx, C.byref(ms), C.byref(launches), C.byref(pairs))
    ps.lib.dv_profile(ps.ctx, 0)
    return solver.v_vort[:ps.particle_num[None]].clone(), pairs.value


def direct_pairs(ps):
    q = ps.counters()
    return float(q["n_targets"]) * q["num_samples"]


CASES = {
    "cubes_ref": dict(shape=(96, 32, 24), every=8),
    "cubes_blob": dict(shape=(96, 32, 24), every=8, blob=True),
    "part_boxes": dict(shape=(71, 37, 29), every=4, origin=-1.25),
    "thin_axis": dict(shape=(128, 128, 5), every=8),
    "thin_axis_blob": dict(shape=(7, 96, 110), every=8, blob=True),
    "long_axis": dict(shape=(420, 16, 11), every=8),
    "vortex_domain": dict(shape=(96, 40, 32), every=4, vortex_domain=([0.4, 0.2, 0.1], [2.5, 1.1, 1.0])),
}


@pytest.mark.parametrize("case", CASES)
def test_boxes_match_fp64_oracle(cuda, case):
    ps, solver, _ = make(**CASES[case])
    o = OracleSim(ps.params, ps.particle_max_num, 0)
    o.load_snapshot(ps.snapshot(), ps.counters())
    o.counting_sort()
    assert np.array_equal(o.permutation(), np.arange(ps.particle_num[None]))
    got, pairs = run(ps, solver)
    assert pairs < 0.9 * direct_pairs(ps), "the boxes were not used"
    o.calls("vvpe_mc", 64)
    n = ps.particle_num[None]
    ref = o.snapshot()["solver.v_vort"][:n, :3].astype(np.float64)
    g = got.cpu().numpy().astype(np.float64)
    if CASES[case].get("vortex_domain"):
        lo, hi = CASES[case]["vortex_domain"]
        x = ps.snapshot()["x"][:, :3]
        inside = np.all((x >= np.float32(lo)) & (x <= np.float32(hi)), axis=1)
        assert 0 < inside.sum() < n
        g, ref = g[inside], ref[inside]
    assert np.all(np.isfinite(ref)) and np.max(np.abs(ref)) > 0
    assert np.max(np.abs(g - ref)) < RTOL * np.max(np.abs(ref))


def test_calls_that_take_the_direct_loop(cuda):
    """A target moved to another box after the sort, a weight that is not
    finite, positions changed by advect: every target with every sample."""
    ps, solver, idx = make(shape=(96, 32, 24), every=8)
    a, pairs = run(ps, solver)
    assert pairs < 0.9 * direct_pairs(ps)
    n = ps.particle_num[None]
    drawn = set(idx.tolist())
    t = next(i for i in range(n // 2, n) if i not in drawn)
    keep = ps.x[t].clone()
    ps.x[t] = ps.x[0] + torch.tensor([0.001, 0.0, 0.0], device="cuda")
    b, pairs = run(ps, solver)
    assert pairs == direct_pairs(ps)
    rows = torch.ones(n, dtype=torch.bool, device="cuda")
    off, nbr = ps.stored_neighbor_lists()
    rows[nbr[off[t]:off[t + 1]].long()] = False  # the lists still name the moved particle there
    rows[t] = False
    assert float((a - b)[rows].abs().max()) < RTOL * float(a.abs().max())
    ps.x[t] = keep
    j = int(idx[7])
    w = solver.d_vort_smoothed[j].clone()
    solver.d_vort_smoothed[j] = float("inf")
    _, pairs = run(ps, solver)
    assert pairs == direct_pairs(ps)
    solver.d_vort_smoothed[j] = w
    c, pairs = run(ps, solver)
    assert pairs < 0.9 * direct_pairs(ps) and torch.equal(c, a)
    solver.advect()
    _, pairs = run(ps, solver)
    assert pairs == direct_pairs(ps)


def test_no_samples_and_few_samples(cuda):
    """No sample: the far part is zero; few samples: too few pairs for boxes."""
    ps, solver, idx = make(shape=(96, 32, 24), every=8)
    for m in (0, 1, 40):
        solver.num_samples[None] = m
        got, pairs = run(ps, solver)
        assert pairs == direct_pairs(ps) and bool(torch.isfinite(got).all())
