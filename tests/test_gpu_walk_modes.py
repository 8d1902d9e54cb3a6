"""A later round's walks and chains run a warp each while the launch has warps
for them, else a thread each: the same draws, so the same particles.  A small
population alone takes the warps; beside one with tens of thousands of events
a round it takes the threads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("case", ["additive_flat", "brown_power"])
def test_warp_and_thread_walks_agree(gpu_lib, case, mode):
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    m = pm.MODE_FP64 if mode == "fp64" else pm.MODE_MIXED
    if case == "brown_power":
        make, kernel, del_t = aero_dist.brown_bimodal, pm.COAG_KERNEL_TYPE_BROWN, 1800.0
    else:
        make, kernel, del_t = aero_dist.additive_exp, pm.COAG_KERNEL_TYPE_ADDITIVE, 40.0
    small, large = make(1500, seed=2), make(400000, seed=3)
    res, events = [], []
    for pops in ([small], [small, large]):
        n = len(pops)
        st = pm.AeroState(small.aero_data, small.awa, mode=m, n_pop=n, seeds=np.arange(5, 5 + n, dtype=np.uint64))
        for k, p in enumerate(pops):
            st.set_weight_pop(k, p.awa)
            st.add_particles(p.vol, p.group, pop=k)
        for _ in range(4):
            pm.mc_coag_batch(kernel, np.full(n, 288.0), np.full(n, 1e5), 1000.0, st, del_t)
            events.append(st.conflicts()["events"])
        res.append(st.particles(pop=0, components=True))
    # 148 SMs x 2 blocks x 8 warps = 2368 walks take a warp each
    assert min(events[4:]) > 2 * 2368 and max(events[:4]) < 2368
    for k in res[0]:
        assert np.array_equal(res[0][k], res[1][k]), k
