"""Device memory of a 3-D context.  Per particle of capacity it is what it was
before sweeps packed fields and the far field had boxes (685 bytes by its
arrays) to within 2%; the boxes come on top only where they can be used and take
at most a quarter of what is free, so a context fits wherever it fitted."""
import ctypes as C

import pytest
import torch

from dimcv_sph_b200.config_builder import SimConfig

pytestmark = pytest.mark.gpu


def params(**extra):
    from dimcv_sph_b200.particle_system import ParticleSystem
    c = {"domainStart": [0.0] * 3, "domainEnd": [1.0] * 3, "particleRadius": 1.0 / 64.0, "density0": 1000,
         "simulationMethod": 0, "gravitation": [0.0] * 3, "timeStepSize": 1e-3, "volumeScale": 0.8,
         "GenProbPara": 5, "DelProbPara": 3.5, "cellOriginOffset": True, "skipCell0": False, **extra}
    ps = ParticleSystem(SimConfig(config={"Configuration": c}), capacity=64)
    return ps, ps.params


def used(ps, p, cap, keep=0):
    """Bytes that dv_create takes for `cap` particles with only `keep` bytes free (0: all that is)."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = None
    if keep:
        fill = torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device="cuda")
    a = torch.cuda.mem_get_info()[0]
    ctx = ps.lib.dv_create(C.byref(p), cap, None)
    assert ctx, ps.lib.dv_last_error(None)
    b = torch.cuda.mem_get_info()[0]
    ps.lib.dv_destroy(ctx)
    del fill
    torch.cuda.empty_cache()
    return a - b


def test_bytes_per_particle(cuda):
    ps, p = params(compensated=True)
    n = 4_000_000
    per = (used(ps, p, 2 * n) - used(ps, p, n)) / n
    assert per < 1.02 * 685, per
    ps, p = params(periodic=True)
    assert (used(ps, p, 2 * n) - used(ps, p, n)) / n < 1.02 * 685


def test_boxes_only_where_memory_allows(cuda):
    fine = {"particleRadius": 1.0 / 512.0}  # 16 x 16 x 16 boxes
    ps, p = params(**fine)
    n = 4_000_000
    full, plain = used(ps, p, n), used(ps, params(compensated=True, **fine)[1], n)
    assert full > plain + 60 * n
    assert used(ps, p, n, keep=plain + (64 << 20)) <= plain + (16 << 20)


def test_no_boxes_on_an_axis_too_long(cuda):
    """Squared gaps of 46,341 boxes and more along an axis do not fit 32 bits
    (a channel of 400,000 x 8 x 8 cells has 50,000): such grids have no boxes."""
    n = 17_000_000  # enough slots for 256 in each of 65,536 boxes
    h = 0.01
    shape = {"domainEnd": [400_000 * h, 8 * h, 8 * h], "particleRadius": h / 4}
    ps, p = params(**shape)
    assert p.grid_num[0] >= 400_000
    gap = p.grid_num[0] // 8 - 2
    assert gap * gap > 2 ** 31
    full, plain = used(ps, p, n), used(ps, params(compensated=True, **shape)[1], n)
    assert full <= plain + (16 << 20)
