"""Contexts that live for a few steps: what they cost beside one that stays, and
what the last one leaves behind."""
import ctypes
import gc
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def job(pop, n_steps):
    import partmc_b200 as pm
    env = pm.EnvState(288.0, 1e5, 1000.0)
    st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
    st.add_particles(pop.vol, pop.group)
    for _ in range(n_steps):
        pm.mc_coag(pm.COAG_KERNEL_TYPE_ADDITIVE, env, pop.aero_data, st, 1.0)
    n = st.n_part()
    st.close()
    return n


def test_a_context_alone_costs_little_more(gpu_lib):
    """The fastest of 25 short jobs with no other context alive, against the
    same beside one that has stepped: memory that contexts share is not made
    and freed with each (which took 2 to 4 ms of 6)."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    gc.collect()
    pop = aero_dist.additive_exp(1000, seed=1)

    def fastest():
        t = []
        for _ in range(25):
            t0 = time.perf_counter()
            job(pop, 3)
            t.append(time.perf_counter() - t0)
        return min(t)

    job(pop, 3)
    alone = fastest()
    st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
    st.add_particles(pop.vol, pop.group)
    for _ in range(6):
        pm.mc_coag(pm.COAG_KERNEL_TYPE_ADDITIVE, pm.EnvState(288.0, 1e5, 1000.0), pop.aero_data, st, 1.0)
    beside = fastest()
    assert alone < 1.35 * beside


def test_first_steps_run_from_the_host(gpu_lib):
    """No graph is made for a context's first two steps; from the third on a
    step is one."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pop = aero_dist.additive_exp(1000, seed=1)
    st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
    st.add_particles(pop.vol, pop.group)
    gpu_lib.pmc_coag_gpu_profile(st.ctx, 1)
    ms, n, u = ctypes.c_double(), ctypes.c_int64(), ctypes.c_int64()
    runs = []
    for _ in range(6):
        pm.mc_coag(pm.COAG_KERNEL_TYPE_ADDITIVE, pm.EnvState(288.0, 1e5, 1000.0), pop.aero_data, st, 1.0)
        assert gpu_lib.pmc_coag_gpu_profile_read(st.ctx, 2, ctypes.byref(ms), ctypes.byref(n), ctypes.byref(u)) == 0
        runs.append(n.value)
    assert runs == [0, 0, 1, 2, 3, 4]


def test_last_context_gives_its_memory_back(gpu_lib):
    import partmc_b200 as pm
    import torch
    gc.collect()
    st = pm.AeroState(pm.AeroData([1000.0]), pm.AeroWeightArray.flat())
    st.close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(2):  # a pool that was left is used again
        st = pm.AeroState(pm.AeroData([1000.0]), pm.AeroWeightArray.flat())
        st.add_particles(np.full((1000000, 1), 1e-18))
        assert torch.cuda.mem_get_info()[0] < before - (256 << 20)
        assert st.n_part() == 1000000
        st.close()
        gc.collect()
        assert torch.cuda.mem_get_info()[0] > before - (64 << 20)
