"""Size distributions over species counts around a warp's lanes and over grids
whose sums do and do not fit one warp's share of shared memory, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_spec,n_bin", [(1, 50), (1, 4000), (3, 160), (31, 40), (32, 40), (33, 100), (64, 160)])
@pytest.mark.parametrize("n_part", [1, 31, 5003])
def test_size_dist_shapes(gpu_lib, n_spec, n_bin, n_part):
    """Relative 1e-12: sums of at most 5003 positive terms in any order."""
    import partmc_b200 as pm
    rng = np.random.default_rng(n_spec * 7 + n_bin + n_part)
    vol = rng.lognormal(-48.0, 1.5, size=(n_part, n_spec))
    dens = rng.uniform(1000.0, 2000.0, size=n_spec)
    awa = pm.AeroWeightArray.power(-1.0, magnitude=3.0)
    st = pm.AeroState(pm.AeroData(dens), awa)
    st.add_particles(vol)
    d = 2.0 * (vol.sum(1) * 3.0 / (4.0 * np.pi)) ** (1.0 / 3.0)
    lo, hi = 0.9 * np.quantile(d, 0.02), 1.1 * np.quantile(d, 0.98)  # particles off both ends
    num, mass = st.size_dist(n_bin, lo, hi)
    b = np.floor((np.log(d) - np.log(lo)) / (np.log(hi) - np.log(lo)) * n_bin).astype(int)
    ok = (b >= 0) & (b < n_bin)
    nc = awa.num_conc_at_radius(1, d / 2.0) * n_bin / (np.log(hi) - np.log(lo))
    ref = np.bincount(b[ok], weights=nc[ok], minlength=n_bin)
    assert np.allclose(num, ref, rtol=1e-12, atol=0.0)
    for k in range(n_spec):
        r = np.bincount(b[ok], weights=(nc * vol[:, k] * dens[k])[ok], minlength=n_bin)
        assert np.allclose(mass[:, k], r, rtol=1e-12, atol=0.0)


@pytest.mark.parametrize("n_spec", [8, 9])
@pytest.mark.parametrize("n_part", [1025, 160000])
def test_size_dist_either_way(gpu_lib, n_spec, n_part):
    """Both kernels around the number of species and slots where the choice
    changes.  At most n_part positive terms a sum, each side rounding each."""
    import partmc_b200 as pm
    rng = np.random.default_rng(n_spec + n_part)
    vol = rng.lognormal(-48.0, 1.5, size=(n_part, n_spec))
    dens = rng.uniform(1000.0, 2000.0, size=n_spec)
    awa = pm.AeroWeightArray.power(-1.0, magnitude=3.0)
    st = pm.AeroState(pm.AeroData(dens), awa)
    st.add_particles(vol)
    d = 2.0 * (vol.sum(1) * 3.0 / (4.0 * np.pi)) ** (1.0 / 3.0)
    num, mass = st.size_dist(20, 0.5 * d.min(), 2.0 * d.max())
    width = (np.log(2.0 * d.max()) - np.log(0.5 * d.min())) / 20
    nc = awa.num_conc_at_radius(1, d / 2.0)
    tol = 4.0 * n_part * 2.0 ** -53 + 1e-12
    assert abs(num.sum() * width / nc.sum() - 1.0) < tol
    assert np.all(np.abs(mass.sum(0) * width / (nc[:, None] * vol * dens).sum(0) - 1.0) < tol)
