"""Size distributions of large populations bin by bin, with dead slots and slot
counts that end inside a tile, for the numbers of species around a warp's
lanes and around the two kernels' limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_spec,n_bin", [(8, 60), (9, 60), (20, 160), (32, 90), (33, 90), (64, 100)])
def test_every_bin_of_a_large_population(gpu_lib, n_spec, n_bin):
    """More slots than two half tiles an SM (151,552 on 148 SMs).  Each sum has
    at most n positive terms, rounded on either side."""
    import partmc_b200 as pm
    n = 190123
    rng = np.random.default_rng(n_spec)
    dens = rng.uniform(1000.0, 2000.0, size=n_spec)
    vol = rng.lognormal(-34.0, 1.0, size=(n, 1)) * rng.dirichlet(np.ones(n_spec), size=n)
    data = pm.AeroData(dens)
    awa = pm.AeroWeightArray.flat(magnitude=1e9 / n)
    st = pm.AeroState(data, awa, seed=4)
    st.add_particles(vol)
    pm.mc_coag(pm.COAG_KERNEL_TYPE_ADDITIVE, pm.EnvState(288.0, 1e5, 1000.0), data, st, 1.0)
    got = st.particles()
    v = got["vol"]
    assert 0.5 * n < v.shape[0] < n - 100  # dead slots between the live ones
    vt = v[:, 0].copy()
    for k in range(1, n_spec):  # in species order, as the library sums
        vt = vt + v[:, k]
    d = 2.0 * (vt * 3.0 / (4.0 * np.pi)) ** (1.0 / 3.0)
    lo, hi = 0.9 * np.quantile(d, 0.01), 1.1 * np.quantile(d, 0.99)  # particles off both ends
    num, mass = st.size_dist(n_bin, lo, hi)
    b = np.floor((np.log(d) - np.log(lo)) / (np.log(hi) - np.log(lo)) * n_bin).astype(int)
    ok = (b >= 0) & (b < n_bin)
    assert 0 < (~ok).sum() < 0.1 * n
    nc = awa.num_conc_at_radius(1, d / 2.0) * n_bin / (np.log(hi) - np.log(lo))
    tol = 4.0 * n * 2.0 ** -53 + 1e-12
    ref = np.bincount(b[ok], weights=nc[ok], minlength=n_bin)
    assert ref.min() > 0.0
    assert np.all(np.abs(num / ref - 1.0) < tol)
    for k in range(n_spec):
        r = np.bincount(b[ok], weights=(nc * v[:, k] * dens[k])[ok], minlength=n_bin)
        assert np.all(np.abs(mass[:, k] / r - 1.0) < tol), k
