"""The host's wait for a step follows the scheduling the process chose: under
blocking waits a step leaves the calling thread's core to others."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, time
cuda = ctypes.CDLL("libcuda.so.1")
assert cuda.cuInit(0) == 0
assert cuda.cuDevicePrimaryCtxSetFlags_v2(0, {flag}) == 0  # CU_CTX_SCHED_*, of this process alone
import numpy as np
import partmc_b200 as pm
from partmc_b200 import aero_dist
pop = aero_dist.additive_exp(2000000, seed=1)
st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
st.add_particles(pop.vol, pop.group)
step = lambda n: pm.mc_coag_batch(pm.COAG_KERNEL_TYPE_ADDITIVE, 288.0, 1e5, 1000.0, st, 2.0, n_steps=n)
step(8)
w, c = time.perf_counter(), time.thread_time()
tests, coags = step(60)
print(time.thread_time() - c, time.perf_counter() - w, tests, coags, st.n_part())
"""


def test_blocking_waits_leave_the_core(gpu_lib):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = {}
    for name, flag in (("spin", 1), ("yield", 2), ("blocking", 4)):
        out = subprocess.run([sys.executable, "-c", CHILD.format(flag=flag)], cwd=root, check=True, timeout=300,
                             capture_output=True, text=True, env=dict(os.environ, PYTHONPATH=root)).stdout.split()
        res[name] = [float(x) for x in out]
    assert res["spin"][2:] == res["yield"][2:] == res["blocking"][2:]  # the same steps
    cpu, wall = res["blocking"][:2]
    print(res)
    # of a step of 0.4 ms the launch, some 20 us, is on the host
    assert cpu < 0.6 * wall, res
