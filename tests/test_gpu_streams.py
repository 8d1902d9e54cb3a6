"""Contexts in a process whose default stream is busy: a context works on a
stream of its own, which does not wait for the default one."""
import glob
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def queue_work():
    """Some 0.4 s of an ordinary, bounded kernel on the default stream."""
    import torch
    torch.cuda.synchronize()
    torch.cuda._sleep(int(0.4 * 1.9e9))
    e = torch.cuda.Event()
    e.record()
    return e


def test_context_made_behind_queued_work(gpu_lib):
    """Made and filled while the default stream is busy; every particle is
    there after that work has ended, and the steps are those of a context made
    on an idle device."""
    import partmc_b200 as pm
    import torch
    from partmc_b200 import aero_dist
    pop = aero_dist.brown_bimodal(20000, seed=4)
    env = pm.EnvState(288.0, 1e5)
    res, kept = [], []  # a context that goes would wait for the device
    for busy in (False, True):
        e = queue_work() if busy else None
        st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
        kept.append(st)
        st.add_particles(pop.vol, pop.group)
        if busy:
            assert not e.query()  # the work was still queued: nothing here waited for it
        torch.cuda.synchronize()
        assert st.n_part() == pop.n_part and st.next_id() == pop.n_part + 1
        counts = [pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, 600.0) for _ in range(5)]
        res.append((counts, st.particles(components=True)))
    assert res[0][0] == res[1][0] and sum(c[1] for c in res[0][0]) > 0
    for k in res[0][1]:
        assert np.array_equal(res[0][1][k], res[1][1][k]), k


def test_replay_stream_set_behind_queued_work(gpu_lib):
    import partmc_b200 as pm
    import torch
    g = np.load(sorted(glob.glob(os.path.join(os.path.dirname(__file__), "golden", "replay_*.npz")))[0])
    data = pm.AeroData(g["density"])
    env = pm.EnvState(float(g["temp"]), float(g["pressure"]), float(g["coeff"]))
    queue_work()
    st = pm.AeroState(data, pm.AeroWeightArray(g["w_type"], g["w_mag"], g["w_exp"]), mode=pm.MODE_REPLAY)
    st.add_particles(g["vol0"], g["group0"], ids=g["id0"])
    st.set_next_id(len(g["vol0"]) + 1)
    st.set_replay(g["uniforms"])
    counters = [pm.mc_coag(int(g["kernel"]), env, data, st, float(g["del_t"])) for _ in range(int(g["steps"]))]
    assert np.array_equal(np.array(counters), g["counters"])
    torch.cuda.synchronize()
    p = st.particles()
    for k, ref in (("vol", "vol"), ("id", "id"), ("weight_group", "weight_group")):
        assert np.array_equal(p[k], g[ref]), k
