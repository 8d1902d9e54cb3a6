"""Chains of sedimenting drops, whose collectors absorb many partners, change
cells and draw absorbed partners again, by a warp each and by a thread each:
the same particles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def drops(n, seed, kind):
    from partmc_b200 import aero_dist
    if kind == "flat":
        return aero_dist.additive_exp(n, seed=seed)
    data, awa, vol, group = aero_dist._modes_population(np.random.default_rng(seed), n, [(1e9, 1e-5, 0.2)], "nummass",
                                                        0.0, [1000.0])
    return aero_dist.Population(data, awa, vol, group)


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("kind,n_large,del_t,n_steps", [("flat", 1500000, 20.0, 30), ("nummass", 1000000, 5.0, 3)])
def test_sedimentation_chains(gpu_lib, kind, n_large, del_t, n_steps, mode):
    """A small population alone takes the warps.  Beside a large one its walks
    take the threads; under number-and-mass weights, where most events of the
    large one come from chains over some 17 rounds a step, its chains too."""
    import partmc_b200 as pm
    m = pm.MODE_FP64 if mode == "fp64" else pm.MODE_MIXED
    small, large = drops(1500, 2, kind), drops(n_large, 3, kind)
    res, events, per_round = [], [], []
    for pops in ([small], [small, large]):
        n = len(pops)
        st = pm.AeroState(small.aero_data, small.awa, mode=m, n_pop=n, seeds=np.arange(5, 5 + n, dtype=np.uint64))
        for k, p in enumerate(pops):
            st.set_weight_pop(k, p.awa)
            st.add_particles(p.vol, p.group, pop=k)
        for _ in range(n_steps):
            pm.mc_coag_batch(pm.COAG_KERNEL_TYPE_SEDI, np.full(n, 288.0), np.full(n, 1e5), 0.0, st, del_t)
            events.append(st.conflicts()["events"])
            per_round.append(events[-1] / st.stats()["rounds"])
        res.append(st.particles(pop=0, components=True))
    # 148 SMs x 2 blocks x 8 warps = 2368 walks or chains of a launch take a warp each
    assert max(events[:n_steps]) < 2368 < min(events[n_steps:]) / 2
    if kind == "nummass":
        assert min(per_round[n_steps:]) > 2 * 2368
    assert res[0]["n_comp"].max() == 20  # long chains: their component lists overflowed
    for k in res[0]:
        assert np.array_equal(res[0][k], res[1][k]), k
