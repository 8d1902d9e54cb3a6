"""Target operations that come and go from step to step, in one population or
in some of a batch: the steps stay graphs, with the particles of steps run
from the host."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = [(1e11, 0.5e-8, np.log10(1.3)), (1e8, 0.25e-6, np.log10(1.3))]  # fine particles, coarse collectors


def graph_runs(gpu_lib, st):
    """Steps whose later rounds ran as a graph since profiling began."""
    ms, n, u = ctypes.c_double(), ctypes.c_int64(), ctypes.c_int64()
    assert gpu_lib.pmc_coag_gpu_profile_read(st.ctx, 2, ctypes.byref(ms), ctypes.byref(n), ctypes.byref(u)) == 0
    return n.value


def steps(pops, del_ts, graphs, gpu_lib=None):
    import partmc_b200 as pm
    n = len(pops)
    st = pm.AeroState(pops[0].aero_data, pops[0].awa, n_pop=n, seeds=np.arange(7, 7 + n, dtype=np.uint64))
    st.set_graphs(graphs)
    for k, p in enumerate(pops):
        st.set_weight_pop(k, p.awa)
        st.add_particles(p.vol, p.group, pop=k)
    if gpu_lib:
        gpu_lib.pmc_coag_gpu_profile(st.ctx, 1)
    out, ops = [], []
    for dt in del_ts:
        out.append(pm.mc_coag_batch(pm.COAG_KERNEL_TYPE_BROWN, np.full(n, 288.0), np.full(n, 1e5), 0.0, st, dt) +
                   (st.stats()["rounds"],))
        ops.append(st.conflicts()["target_ops"])
    return out, ops, [st.particles(pop=k, components=True) for k in range(n)], graph_runs(gpu_lib, st) if gpu_lib else 0


@pytest.mark.parametrize("sizes", [[4000], [4000, 1500, 4000], [1500, 4000]])
def test_operations_that_come_and_go(gpu_lib, sizes):
    from partmc_b200 import aero_dist
    pops = [aero_dist.brown_bimodal(n, seed=11 + k, modes=MODES) for k, n in enumerate(sizes)]
    del_ts = [150.0, 150.0, 150.0, 150.0] + [0.01, 150.0, 20.0, 150.0, 0.01, 0.01, 20.0, 150.0] * 3 + [0.01] * 24 + [150.0] * 6
    a = steps(pops, del_ts, True, gpu_lib)
    b = steps(pops, del_ts, False)
    assert a[:2] == b[:2]
    for pa, pb in zip(a[2], b[2]):
        for k in pa:
            assert np.array_equal(pa[k], pb[k]), k
    ops = a[1]
    flips = sum((x > 0) != (y > 0) for x, y in zip(ops, ops[1:]))
    assert flips >= 12 and max(ops) > 100
    # the long way: the first steps, the change to the graph without target
    # operations and back after the long pause, and where bounds are outgrown
    assert a[3] >= len(del_ts) - 12, a[3]
