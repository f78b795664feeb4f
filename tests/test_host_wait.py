"""The host thread of an eager corrector waits the way the device is set to:
with cudaDeviceScheduleBlockingSync it sleeps. A kernel of half a second on the
context's stream ahead of the step makes the wait long; a thread that spins
through it uses as much processor time as it takes, one that sleeps next to
none (bound: a quarter). In a process of its own, since the flag belongs to
the device's context."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, time
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0
CU_CTX_SCHED_BLOCKING_SYNC = 4
assert cu.cuDevicePrimaryCtxSetFlags_v2(0, CU_CTX_SCHED_BLOCKING_SYNC) == 0
import torch
import psb_project_b200 as P
sc = P.dam_break((20, 18, 16), 0.01, (0.5, 0.4, 0.3), 0.02, dt=5e-4, seed=5)
pos = P.scene_positions(sc)
with P.Simulation(sc) as sim:
    st = torch.cuda.Stream()
    sim.set_stream(st.cuda_stream)
    sim.upload(pos)
    sim.step(2)
    with torch.cuda.stream(st):
        torch.cuda._sleep(1_000_000_000)
    wall, cpu = time.perf_counter(), time.thread_time()
    sim.step(1)
    wall, cpu = time.perf_counter() - wall, time.thread_time() - cpu
    sim.set_stream(0)
    assert sim.stats().iters >= sc.min_iters
print(wall, cpu)
"""


def test_blocking_schedule_does_not_spin():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    wall, cpu = map(float, r.stdout.split())
    assert wall > 0.2
    assert cpu < 0.25 * wall
