"""Target operations (per-particle path) carried out by a warp: species lie
with the lanes, so the result may not depend on how a particle's volume is
split into species."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scavenging(n_part, n_spec):
    """Fine particles (10 nm) with coarse ones (0.5 um) that collect them,
    power weights; each volume split evenly over n_spec species of one
    density."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    modes = [(1e11, 0.5e-8, np.log10(1.3)), (1e8, 0.25e-6, np.log10(1.3))]
    pop = aero_dist.brown_bimodal(n_part, seed=11, modes=modes)
    data = pm.AeroData(np.full(n_spec, 1800.0))
    st = pm.AeroState(data, pop.awa, seed=7)
    st.add_particles(np.repeat(pop.vol / n_spec, n_spec, axis=1), pop.group)
    return pm, data, st


@pytest.mark.parametrize("n_spec", [2, 31, 32, 33, 64])
def test_species_split_over_lanes(n_spec):
    """The same particles (IDs, component and primary counts) as with one
    species, and total volumes to rounding: sums of at most 64 equal parts,
    a few thousand additions at 1e-16 each."""
    env, res = None, {}
    for ns in (1, n_spec):
        pm, data, st = scavenging(3000, ns)
        env = pm.EnvState(288.0, 1e5)
        ops = 0
        for _ in range(4):
            pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, data, st, 150.0)
            ops += st.conflicts()["target_ops"]
        assert ops > 100  # the per-particle path ran
        res[ns] = st.particles(components=True)
    a, b = res[1], res[n_spec]
    assert np.array_equal(a["id"], b["id"])
    assert np.array_equal(a["n_primary_parts"], b["n_primary_parts"])
    assert np.array_equal(a["n_comp"], b["n_comp"])
    assert a["n_comp"].max() == 20  # component lists overflowed: the selection ran
    assert np.allclose(b["vol"].sum(1), a["vol"][:, 0], rtol=1e-12, atol=0.0)
