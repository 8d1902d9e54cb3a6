"""More populations in a context than the sort keeps chunk counts for in shared
memory (2048): each steps as it does alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pop", [2048, 2049])
def test_populations_around_the_sorts_map(gpu_lib, n_pop):
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pops = [aero_dist.brown_bimodal(n, seed=n) for n in (30, 400, 5000)]  # 5000: several chunks
    at = {0: 2, 1: 1, 700: 0, 1023: 2, 1500: 1, n_pop - 2: 2, n_pop - 1: 1}
    temps = np.linspace(270.0, 300.0, n_pop)

    def fill(st, k, p):
        st.set_weight_pop(k, p.awa)
        st.add_particles(p.vol, p.group, pop=k)

    st = pm.AeroState(pops[0].aero_data, pops[0].awa, n_pop=n_pop, seeds=np.arange(5, 5 + n_pop, dtype=np.uint64))
    for k in range(n_pop):
        fill(st, k, pops[at.get(k, 0)])
    for n in (1, 5):
        pm.mc_coag_batch(pm.COAG_KERNEL_TYPE_BROWN, temps, np.full(n_pop, 1e5), 0.0, st, 1800.0, n_steps=n)
    for k, which in at.items():
        p = pops[which]
        one = pm.AeroState(p.aero_data, p.awa, seed=5 + k)
        fill(one, 0, p)
        for _ in range(6):
            pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, pm.EnvState(float(temps[k]), 1e5), p.aero_data, one, 1800.0)
        a, b = st.particles(pop=k, components=True), one.particles(components=True)
        assert which == 0 or not np.array_equal(a["id"], np.arange(1, p.n_part + 1))  # it coagulated
        for key in a:
            assert np.array_equal(a[key], b[key]), (k, key)
