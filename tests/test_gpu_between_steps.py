"""Calls between steps that run as one graph: the graph counts steps and reads
parameters from the device's copies, so whatever a call changes has to reach
them, and the particles are those of a context whose steps run from the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("call", ["sort", "record", "rebalance", "none"])
def test_new_seed_then_a_call_that_copies_the_population(gpu_lib, call):
    """A new seed restarts the population's step count, also where another call
    copies the population to the device before the next step."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pop = aero_dist.brown_bimodal(3000, seed=4)
    env = pm.EnvState(288.0, 1e5)
    res = []
    for graphs in (True, False):
        st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
        st.set_graphs(graphs)
        st.add_particles(pop.vol, pop.group)
        counts = []
        for block in range(2):
            for _ in range(12):
                counts.append(pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, 600.0))
            st.set_seed(21 + block)
            if call == "sort":
                st.sort()
            elif call == "record":
                st.set_record_removals(block == 0)
            elif call == "rebalance":
                st.rebalance(2500.0)
            counts.append(pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, 600.0))
        res.append((st.particles(components=True), counts))
    assert res[0][1] == res[1][1]
    same(res[0][0], res[1][0])


@pytest.mark.parametrize("steps,expect", [(0, (3128, 1585, 2488598, 2617649246)), (5, (3100, 1532, 2334703, 2397525976))])
def test_halving_after_a_new_seed(gpu_lib, steps, expect):
    """A halving draws by the seed and the steps taken before it; which
    particles stay (recorded: count before and after, sums over the IDs) does
    not change with how the steps are run."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pop = aero_dist.brown_bimodal(3000, seed=4)
    st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
    st.add_particles(pop.vol, pop.group)
    for _ in range(steps):
        pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, pm.EnvState(288.0, 1e5), pop.aero_data, st, 600.0)
    n = st.n_part()
    st.set_seed(21)
    st.rebalance(900.0)
    ids = st.particles()["id"]
    assert (n, ids.size, int(ids.sum()), int((ids * np.arange(ids.size)).sum())) == expect
