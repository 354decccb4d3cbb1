"""The FP32 velocity of the differentiable step against its FP64 kernels on the
same plan, where the source chunks are many: the sum of the chunks' partial sums
adds next to nothing.  Without periodic images, as a pair half a box apart can
take another one in FP64 than its FP32 difference does.  Bound: a chunk of 32 terms and one rounding of the result
leave about 1e-7 of the norm (1.0e-7 to 1.2e-7 measured in FP64 against the
exact sum); a hundred partial sums added in FP32 leave 1.9e-7 to 2.5e-7."""
import ctypes as C

import pytest
import torch

from dimcv_sph_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [56, 92])
def test_error_of_many_chunks(cuda, k):
    from dimcv_sph_b200.adjoint import FULL, VortexBox, _Velocity
    errs = []
    for seed in range(4):
        cfg, x, w = scenes.periodic2d(k * k, seed=seed, dt=0.01)
        box = VortexBox(cfg, x)
        w = torch.from_numpy(w).cuda()
        plan = box.validate(box.build_plan(box.x0, None, 0, FULL))
        xs, wt = box.x0.index_select(0, plan.perm), w.index_select(0, plan.perm)
        box.ps.params.periodic = 0
        assert box.lib.dv_set_params(box.ctx, C.byref(box.ps.params)) == 0
        a = _Velocity.apply(xs, wt, box, plan, None).double()
        b = _Velocity.apply(xs.double(), wt.double(), box, plan, None)
        errs.append(float((a - b).norm() / b.norm()))
    assert sum(errs) / len(errs) < 1.5e-7, errs
