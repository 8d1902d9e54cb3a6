"""Downloads gather live slots by warps; the host mirror copies slot arrays as
they are.  Both give the same particles for species counts around a warp's
lanes, with dead slots among the live ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_spec", [1, 3, 31, 32, 33, 64])
@pytest.mark.parametrize("n_part", [1, 33, 4001])
def test_download_matches_slot_copy(gpu_lib, n_spec, n_part):
    import partmc_b200 as pm
    rng = np.random.default_rng(n_spec + n_part)
    vol = 4.2e-15 * rng.exponential(size=(n_part, 1)) * rng.dirichlet(np.ones(n_spec), size=n_part)
    data = pm.AeroData(np.full(n_spec, 1000.0))
    st = pm.AeroState(data, pm.AeroWeightArray.flat(magnitude=1e9 / n_part), seed=3)
    st.add_particles(vol)
    _, coags = pm.mc_coag(pm.COAG_KERNEL_TYPE_ADDITIVE, pm.EnvState(288.0, 1e5, 1000.0), data, st, 30.0)
    assert n_part < 4000 or coags > 100  # dead slots
    m = pm.HostMirror(st)
    m.sync()
    a, b = st.particles(components=True), m.particles()
    for k in b:
        assert np.array_equal(a[k], b[k]), k
    assert np.array_equal(a["n_comp"], np.minimum(a["n_primary_parts"], 20))
    filled = np.arange(20)[None, :] < a["n_comp"][:, None]
    assert np.array_equal(a["comp_source"], filled.astype(np.int32))  # source 1 where there is a component
    assert np.all(a["comp_create_time"] == 0.0)
