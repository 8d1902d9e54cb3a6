"""Removal records of steps that run as one graph, read after several of them,
against those of steps run from the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["flat", "target_ops", "batch"])
def test_records_over_graph_steps(gpu_lib, case):
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    modes = [(1e11, 0.5e-8, np.log10(1.3)), (1e8, 0.25e-6, np.log10(1.3))]
    if case == "flat":
        pops, kernel, del_t = [aero_dist.additive_exp(5000, seed=4)], pm.COAG_KERNEL_TYPE_ADDITIVE, 4.0
    elif case == "target_ops":
        pops, kernel, del_t = [aero_dist.brown_bimodal(4000, seed=11, modes=modes)], pm.COAG_KERNEL_TYPE_BROWN, 100.0
    else:
        pops = [aero_dist.brown_bimodal(n, seed=n) for n in (3000, 700, 9000)]
        kernel, del_t = pm.COAG_KERNEL_TYPE_BROWN, 600.0
    n = len(pops)
    res = []
    for graphs in (True, False):
        st = pm.AeroState(pops[0].aero_data, pops[0].awa, n_pop=n, seeds=np.arange(3, 3 + n, dtype=np.uint64))
        st.set_graphs(graphs)
        for k, p in enumerate(pops):
            st.set_weight_pop(k, p.awa)
            st.add_particles(p.vol, p.group, pop=k)
        st.set_record_removals(True)
        out = []
        for steps in (1, 6, 9, 2, 7):
            coags = pm.mc_coag_batch(kernel, np.full(n, 288.0), np.full(n, 1e5), 1000.0, st, del_t, n_steps=steps)[1]
            for k in range(n):
                r = st.removals(pop=k)
                o = np.lexsort((r["other_id"], r["id"]))
                out.append((coags, [r[f][o].tolist() for f in ("id", "action", "other_id")]))
        assert sum(len(x[1][0]) for x in out) > 100
        res.append((out, [st.particles(pop=k) for k in range(n)]))
    assert res[0][0] == res[1][0]
    for a, b in zip(res[0][1], res[1][1]):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
