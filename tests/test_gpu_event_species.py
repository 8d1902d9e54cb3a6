"""Events move their particles' species in blocks of 8 loads: numbers of species
around the blocks and the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_spec", [7, 8, 9, 16, 17, 64])
def test_events_of_split_species(gpu_lib, n_spec):
    """Each volume split evenly over n_spec species of one density: the same
    particles as with one species, volumes to rounding (sums of at most 64
    equal parts and of the particles' merges, a thousand additions at 1e-16)."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pop = aero_dist.additive_exp(6000, seed=7)
    env = pm.EnvState(288.0, 1e5, 1000.0)
    res = []
    for ns in (1, n_spec):
        data = pm.AeroData(np.full(ns, 1000.0))
        st = pm.AeroState(data, pop.awa, seed=3)
        st.add_particles(np.repeat(pop.vol / ns, ns, axis=1), pop.group)
        counts = [pm.mc_coag(pm.COAG_KERNEL_TYPE_ADDITIVE, env, data, st, 20.0) for _ in range(5)]
        assert sum(c[1] for c in counts) > 1000
        res.append((counts, st.particles(components=True)))
    a, b = res[0][1], res[1][1]
    assert res[0][0] == res[1][0]
    for k in ("id", "n_primary_parts", "n_comp", "comp_source"):
        assert np.array_equal(a[k], b[k]), k
    assert np.allclose(b["vol"], a["vol"] / n_spec, rtol=1e-13, atol=0.0)
