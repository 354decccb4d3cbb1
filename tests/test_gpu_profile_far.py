"""dv_profile_far counts the calls that the boxes carried and the pairs of all
calls, with the counts that each call had: a direct loop whose sample count
changes between calls is not taken for the boxes."""
import ctypes as C

import pytest

from test_gpu_farbox import make

pytestmark = pytest.mark.gpu


def test_calls_on_boxes_and_all_pairs(cuda):
    ps, solver, idx = make(shape=(96, 32, 24), every=8)
    n, M = ps.particle_num[None], len(idx)
    ps.lib.dv_profile(ps.ctx, 1)
    want = 0.0
    for m in (40, M, 10, M, 20):  # few samples: the direct loop
        solver.num_samples[None] = m
        solver.vort2vel()
        want += float(n) * m
    calls, pairs, ms, launches, evaluated = C.c_int64(), C.c_double(), C.c_double(), C.c_int64(), C.c_double()
    assert ps.lib.dv_profile_far(ps.ctx, C.byref(calls), C.byref(pairs)) == 0
    ps.lib.dv_profile_read(ps.ctx, C.byref(ms), C.byref(launches), C.byref(evaluated))
    assert calls.value == 2 and launches.value == 5 and pairs.value == want
    assert evaluated.value < want
    ps.lib.dv_profile(ps.ctx, 1)
    assert ps.lib.dv_profile_far(ps.ctx, C.byref(calls), C.byref(pairs)) == 0
    assert calls.value == 0 and pairs.value == 0.0
    ps.lib.dv_profile(ps.ctx, 0)
