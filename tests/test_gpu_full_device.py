"""A device with little memory left: a call whose memory does not fit is refused
and the populations stay usable; a step that fits without its graph runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CAPACITY = 3  # PMC_ERR_CAPACITY


class Full:
    """Blocks that leave at most `left` bytes of device memory."""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        import torch
        torch.cuda.empty_cache()
        self.blocks = []
        for mib in (4096, 256, 32):
            while torch.cuda.mem_get_info()[0] > (mib << 20) + self.left:
                try:
                    self.blocks.append(torch.empty(mib << 20, dtype=torch.uint8, device="cuda"))
                except torch.OutOfMemoryError:
                    break
        return self

    def __exit__(self, *_):
        import torch
        self.blocks = None
        torch.cuda.empty_cache()


def same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def additive(n, seed=3):
    import partmc_b200 as pm
    from partmc_b200 import aero_dist
    pop = aero_dist.additive_exp(n, seed=2)
    st = pm.AeroState(pop.aero_data, pop.awa, seed=seed)
    st.add_particles(pop.vol, pop.group)
    env = pm.EnvState(288.0, 1e5, 1000.0)
    return pm, pop, st, lambda dt: pm.mc_coag(pm.COAG_KERNEL_TYPE_ADDITIVE, env, pop.aero_data, st, dt)


@pytest.mark.parametrize("call", ["rebalance", "step"])
def test_slots_that_cannot_grow(gpu_lib, call):
    """Twice the slots (some 280 MB) do not fit: the particles are as before,
    and go on as those of a context that was never refused."""
    pm, pop, st, step = additive(200000)
    _, _, twin, twin_step = additive(200000)
    for f in (step, twin_step):
        for _ in range(4):
            f(1.0)
    before = st.particles(components=True)
    with Full(40 << 20):
        with pytest.raises(pm.PmcError) as e:
            if call == "rebalance":
                st.rebalance(10.0 * st.n_part())
            else:
                step(400.0)  # more samples than free slots
        assert e.value.code == CAPACITY
    same(before, st.particles(components=True))
    res = []
    for s, f in ((st, step), (twin, twin_step)):
        s.set_seed(77)
        res.append(([f(1.0) for _ in range(6)], s.particles(components=True)))
    assert res[0][0] == res[1][0]
    same(res[0][1], res[1][1])


def test_upload_that_does_not_fit(gpu_lib):
    """The population is left empty, and takes the next upload."""
    pm, pop, st, step = additive(5000)
    step(1.0)
    with Full(40 << 20):
        with pytest.raises(pm.PmcError) as e:
            st.add_particles(np.full((2000000, 1), 1e-15))
        assert e.value.code == CAPACITY
        assert st.n_part() == 0 and st.particles()["id"].size == 0
        step(1.0)
    res = []
    for s, f in ((st, step), additive(5000)[2:]):
        s.set_next_id(1)
        s.add_particles(pop.vol, pop.group)
        s.set_seed(5)
        res.append(([f(1.0) for _ in range(5)], s.particles()))
    assert res[0][0] == res[1][0]
    same(res[0][1], res[1][1])


def test_step_whose_graph_does_not_fit(gpu_lib):
    """A step graph's bounds are the power of two above 1.25 of the last step's
    samples, its host-run step's the one above the samples: with 1.7 to 2.1
    million samples the graph's buffers take 2 GB, twice the others, which the
    device has no room for here."""
    import partmc_b200 as pm
    import torch
    from partmc_b200 import aero_dist
    pop = aero_dist.brown_bimodal(2000000, seed=2)
    env = pm.EnvState(288.0, 1e5)
    res = []
    for full in (False, True):
        st = pm.AeroState(pop.aero_data, pop.awa, seed=3)
        st.add_particles(pop.vol, pop.group)
        counts = [pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, dt) for dt in (600.0, 37000.0)]
        assert 2 ** 21 / 1.25 < counts[1][0] < 2.05 * 2 ** 20
        if full:
            with Full(300 << 20):
                counts += [pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, 20000.0) for _ in range(2)]
        else:
            counts += [pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, 20000.0) for _ in range(2)]
        counts += [pm.mc_coag(pm.COAG_KERNEL_TYPE_BROWN, env, pop.aero_data, st, 600.0) for _ in range(40)]
        res.append((counts, st.particles()))
        del st
        torch.cuda.synchronize()
    assert res[0][0] == res[1][0]
    same(res[0][1], res[1][1])
