"""Contexts that share the device's memory pool: side by side in two threads, and
made and closed between one another's steps."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def job(seed, n_jobs):
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pop = aero_dist.brown_bimodal(2000 + 1000 * seed, seed=seed)
    env = pm.EnvState(288.0, 1e5)
    out = []
    for j in range(n_jobs):
        st = pm.AeroState(pop.aero_data, pop.awa, seed=3 + j)
        for n in (1, 3):  # slots freed and taken again in between
            st.add_particles(np.repeat(pop.vol, n, axis=0), np.repeat(pop.group, n))
            st.set_seed(7 + j)
            counts = [pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, 600.0) for _ in range(6)]
            out.append((counts, st.particles(components=True)))
        st.close()
    return out


def same(a, b):
    assert len(a) == len(b)
    for (ca, pa), (cb, pb) in zip(a, b):
        assert ca == cb
        for k in pa:
            assert np.array_equal(pa[k], pb[k]), k


def test_two_threads(gpu_lib):
    ref = [job(s, 6) for s in (1, 2)]
    got = [None, None]

    def work(i):
        got[i] = job(i + 1, 6)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    for i in range(2):
        assert got[i] is not None
        same(got[i], ref[i])


def test_contexts_come_and_go(gpu_lib):
    """One context steps on while others are made, filled and closed."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pop = aero_dist.brown_bimodal(8000, seed=5)
    env = pm.EnvState(288.0, 1e5)
    res = []
    for others in (False, True):
        st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
        st.add_particles(pop.vol, pop.group)
        counts = []
        for i in range(10):
            counts.append(pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, 600.0))
            if others:
                job(1 + i % 3, 1)
        res.append([(counts, st.particles(components=True))])
    same(*res)
