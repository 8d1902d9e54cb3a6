"""A round's events are flagged, ranked, decided and applied by tiled kernels:
sample counts below, at and past one tile (1024 flags) and past the 32 tiles
that one look-back step covers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_part,del_t", [(50, 0.5), (2000, 60.0), (2000, 120.0), (60000, 120.0), (300000, 90.0)])
def test_flat_events_conserve(gpu_lib, n_part, del_t):
    """Flat weights: every coagulation replaces two particles by one, so the
    count falls by the coagulations, the volume stays (to rounding: sums of
    n_part terms), the primary particles stay, and IDs stay unique."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pop = aero_dist.additive_exp(n_part, seed=7)
    st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
    st.add_particles(pop.vol, pop.group)
    tests, coags = pm.mc_coag(pm.COAG_KERNEL_TYPE_ADDITIVE, pm.EnvState(288.0, 1e5, 1000.0), pop.aero_data, st, del_t)
    got = st.particles()
    assert coags > 0 or n_part < 100
    assert got["id"].size == st.n_part() == pop.n_part - coags
    assert np.unique(got["id"]).size == got["id"].size
    assert got["n_primary_parts"].sum() == pop.n_part
    assert abs(got["vol"].sum() - pop.vol.sum()) <= 1e-12 * pop.vol.sum()
    assert tests >= coags
