"""How the host waits for a Jacobi solve follows the device's scheduling flag
(cudaSetDeviceFlags): with blocking synchronisation the thread sleeps while the
GPU is busy, as cudaStreamSynchronize does.  In a process of its own, as the
flag belongs to the device's context; the GPU is kept busy for about half a
second before the solve."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, sys, time
import torch
assert ctypes.CDLL("libcudart.so.12").cudaSetDeviceFlags(int(sys.argv[1])) == 0
from dimcv_sph_b200 import scenes
from dimcv_sph_b200.particle_system import ParticleSystem
ps = ParticleSystem(scenes.channel2d(length=2.0, reserved=200))
solver = ps.build_solver()
solver.initialize()
solver.compute_densities()
solver._call("dv_divergence_solve", None)
torch.cuda.synchronize()
cpu, wall = time.thread_time(), time.perf_counter()
torch.cuda._sleep(1_000_000_000)
solver._call("dv_divergence_solve", None)
print("used", time.thread_time() - cpu, time.perf_counter() - wall)
torch.cuda.synchronize()
"""


@pytest.mark.parametrize("flag", [4])  # cudaDeviceScheduleBlockingSync
def test_blocking_wait_sleeps(cuda, flag):
    r = subprocess.run([sys.executable, "-c", CHILD, str(flag)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    cpu, wall = (float(t) for t in r.stdout.split("used")[1].split())
    assert wall > 0.2 and cpu < 0.25 * wall, (cpu, wall)
