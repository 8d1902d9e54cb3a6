"""A step that a device scan's give-up ends: reported before a particle has
changed, with the step as one graph or run from the host, and the context
steps on as if that step had not been asked for (its random streams are
used up)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["power", "target_ops"])
def test_steps_after_a_scan_that_gave_up(gpu_lib, case):
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    if case == "power":
        pop, del_t = aero_dist.brown_bimodal(20000, seed=4), 600.0
    else:
        modes = [(1e11, 0.5e-8, np.log10(1.3)), (1e8, 0.25e-6, np.log10(1.3))]
        pop, del_t = aero_dist.brown_bimodal(4000, seed=11, modes=modes), 150.0
    env = pm.EnvState(288.0, 1e5)
    res = []
    for graphs in (True, False):
        st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
        st.set_graphs(graphs)
        st.add_particles(pop.vol, pop.group)
        counts = []
        for _ in range(3):
            for _ in range(12):
                counts.append(pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, del_t))
            before = st.particles(components=True)
            assert gpu_lib.pmc_coag_gpu_test_scan_give_up(st.ctx) == 0
            with pytest.raises(pm.PmcError) as e:
                pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, del_t)
            assert e.value.code == 5  # PMC_ERR_TIMEOUT
            after = st.particles(components=True)
            for k in before:
                assert np.array_equal(before[k], after[k]), (graphs, k)
        for _ in range(3):
            counts.append(pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, del_t))
        res.append((counts, st.particles(components=True)))
    assert res[0][0] == res[1][0]
    for k in res[0][1]:
        assert np.array_equal(res[0][1][k], res[1][1][k]), k
