"""A step run as one graph against the same step with every round launched
from the host: the same particles, counters and IDs bit for bit, across what
sends a step the long way (new grids, changed parameters, uploads, slot
growth, per-particle pairs) and back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def run(pop, kernel, del_t, n_steps, graphs, seed=3, temps=None, upload_at=(), rebalance=None):
    import partmc_b200 as pm
    st = pm.AeroState(pop.aero_data, pop.awa, seed=seed)
    st.set_graphs(graphs)
    st.add_particles(pop.vol, pop.group)
    counts, n_bins = [], set()
    for i in range(n_steps):
        env = pm.EnvState(288.0 if temps is None else temps[i], 1e5, 1000.0)
        counts.append(pm.mc_coag(kernel, env, pop.aero_data, st, del_t) + (st.stats()["rounds"],))
        n_bins.add(float(st.sort()[0][0]))
        if i in upload_at:  # the host takes the particles and gives them back
            p = st.particles()
            st.add_particles(p["vol"], p["weight_group"], ids=p["id"], n_primary_parts=p["n_primary_parts"])
        if rebalance:
            st.rebalance(rebalance)
    return st.particles(components=True), counts, n_bins


@pytest.mark.parametrize("case", ["flat_regrid", "power", "nummass", "temps", "uploads", "rebalance", "tiny"])
def test_step_graph_matches_host_rounds(gpu_lib, case):
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    kw = {}
    if case in ("flat_regrid", "uploads", "tiny"):
        pop = aero_dist.additive_exp(30 if case == "tiny" else 5000, seed=4)
        args = (pm.COAG_KERNEL_TYPE_ADDITIVE, 10.0, 60)
        if case == "uploads":
            kw = dict(upload_at=(5, 6, 20))
    elif case == "nummass":
        pop = aero_dist.brown_20spec(20000, seed=4)
        args = (pm.COAG_KERNEL_TYPE_BROWN, 60.0, 12)
    else:
        pop = aero_dist.brown_bimodal(20000, seed=4)
        args = (pm.COAG_KERNEL_TYPE_BROWN, 600.0, 14)
        if case == "temps":
            kw = dict(temps=[288.0] * 4 + [280.0] * 5 + [270.0] * 5)
        if case == "rebalance":
            kw = dict(rebalance=18000.0)
    a, ca, ga = run(pop, *args, True, **kw)
    b, cb, _ = run(pop, *args, False, **kw)
    assert ca == cb
    same(a, b)
    if case == "flat_regrid":
        assert len(ga) > 1  # the grid was made anew on the way


@pytest.mark.parametrize("n_part", [4000, 60000])
def test_step_graph_with_target_operations(gpu_lib, n_part):
    """Coarse particles scavenging fine ones, at step lengths that take the
    target operations from few to many more than the step before (and past
    the bounds a graph was captured for) and back."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    modes = [(1e11, 0.5e-8, np.log10(1.3)), (1e8, 0.25e-6, np.log10(1.3))]
    pop = aero_dist.brown_bimodal(n_part, seed=11, modes=modes)
    env = pm.EnvState(288.0, 1e5)
    res = []
    for graphs in (True, False):
        st = pm.AeroState(pop.aero_data, pop.awa, seed=7)
        st.set_graphs(graphs)
        st.add_particles(pop.vol, pop.group)
        counts = []
        for del_t in (20.0, 20.0, 20.0, 20.0, 150.0, 20.0, 150.0, 150.0, 150.0, 5.0, 5.0, 600.0, 5.0):
            counts.append(pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, del_t))
            counts.append((st.stats()["rounds"], st.conflicts()["target_ops"], st.conflicts()["target_op_losers"]))
        res.append((st.particles(components=True), counts))
    assert res[0][1] == res[1][1]
    ops = [c[1] for c in res[0][1][1::2]]
    assert max(ops) > 4 * min(ops)
    same(res[0][0], res[1][0])


def test_batched_step_graph(gpu_lib):
    """Populations of uneven sizes, one of them empty, in one context."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pops, temps, press = aero_dist.batched_bimodal(n_pop=5, seed=8, n_min=500, n_max=2e4)
    res = []
    for graphs in (True, False):
        st = pm.AeroState(pops[0].aero_data, pops[0].awa, n_pop=6)
        st.set_graphs(graphs)
        for k, p in enumerate(pops):
            st.set_weight_pop(k, p.awa)
            st.add_particles(p.vol, p.group, pop=k)
        t, q = np.append(temps, 288.0), np.append(press, 1e5)
        c = [pm.mc_coag_batch(pm.COAG_KERNEL_TYPE_BROWN, t, q, 0.0, st, 600.0, n_steps=3) for _ in range(4)]
        res.append((c, [st.particles(pop=k) for k in range(6)]))
    assert res[0][0] == res[1][0]
    for a, b in zip(res[0][1], res[1][1]):
        same(a, b)


def test_claim_generations_restart_after_a_smaller_upload(gpu_lib):
    """Claim generations restart after about 2000 rounds.  A population
    uploaded again starts with fewer slots than it ended with, so slots above
    them hold claims of old generations when that happens; events on those
    slots must not lose to them."""
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pop = aero_dist.brown_bimodal(20000, seed=6)
    st = pm.AeroState(pop.aero_data, pop.awa, seed=5)
    env = pm.EnvState(288.0, 1e5)
    first, rounds = None, 0
    while rounds < 5000:  # at least two restarts
        st.set_next_id(1)
        st.add_particles(pop.vol, pop.group)
        st.set_seed(9)
        for _ in range(6):
            pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, 600.0)
            rounds += st.stats()["rounds"]
        got = st.particles()
        if first is None:
            first = got
            assert got["id"].max() > pop.n_part  # new slots were made
        same(first, got)
