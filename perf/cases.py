"""Timed cases of the coagulation library: what its users have it do.

Each case is one pass through the package's public entry points, as a
program around them makes it: host arrays in, a number of mc_coag steps (or
the device sampler, or the size distributions), results out.  A pass with
steps is one job as the server runs it: the population admitted into a
context that is kept, its steps, the particles back in the caller's
page-locked arrays, and the slot emptied.

  kind      what it stands for
  member    one population: an ensemble member, a served job, or (one step)
            a host model that owns its particles
  mirror    the same with the host's copy brought up to date after every
            step (HostMirror), the drop-in for a coagulation-only run_part
  batch     many populations in one context, advanced together
  run_part  the loop of run_part: step, rebalance, size distributions
  sample    the initial condition drawn on the device, then read back
  size_dist the size distributions of a resident population

Populations follow this repository's configurations: exponential volumes
under the additive kernel, cloud drops under sedimentation, bimodal
log-normals under the Brownian kernel with power weights, three modes of 20
species under number-and-mass weights, and the fine-and-coarse population
whose coarse particles take the per-particle path.
"""
import math

import numpy as np
import torch

import partmc_b200 as pm

LN10 = math.log(10.0)
TEMP, PRESSURE, ADDITIVE_COEFF = 288.0, 1e5, 1000.0
KERNEL = {"additive": pm.COAG_KERNEL_TYPE_ADDITIVE, "brown": pm.COAG_KERNEL_TYPE_BROWN,
          "sedi": pm.COAG_KERNEL_TYPE_SEDI}
# exponents of the weight groups
GROUPS = {"flat": (0.0,), "power": (-1.0,), "nummass": (0.0, -3.0)}


def listed():
    return [
        # the smallest call: a host model that owns its 1000 particles takes
        # one step (the reference's tests run 1000 to 10,000 particles)
        dict(name="host_step_1e3", kind="member", pop="exp", kernel="additive", mode="fp64", n_part=1000, n_spec=1,
             del_t=1.0, n_steps=1),
        # the additive validation run (1e4 particles, flat weights, 1 s steps)
        dict(name="member_additive_1e4", kind="member", pop="exp", kernel="additive", mode="fp64", n_part=10000,
             n_spec=1, del_t=1.0, n_steps=100),
        # the bimodal Brownian run, power weights, 60 s steps
        dict(name="member_brown_1e5", kind="member", pop="bimodal", kernel="brown", mode="fp64", n_part=100000,
             n_spec=1, del_t=60.0, n_steps=60),
        # a served sedimentation job: collectors that absorb many droplets a step
        dict(name="member_sedi_37003", kind="member", pop="drops", kernel="sedi", mode="mixed", n_part=37003,
             n_spec=1, del_t=5.0, n_steps=80),
        # coarse particles scavenging fine ones: the per-particle path
        dict(name="member_scavenge_2e4", kind="member", pop="scavenge", kernel="brown", mode="mixed", n_part=20011,
             n_spec=1, del_t=150.0, n_steps=16),
        # the largest single population: 1e6 particles of 20 species
        dict(name="member_20spec_1e6", kind="member", pop="modes3", kernel="brown", mode="mixed", n_part=1000000,
             n_spec=20, del_t=60.0, n_steps=40),
        # the drop-in with the host's copy current after every step
        dict(name="mirror_20spec_6e5", kind="mirror", pop="modes3", kernel="brown", mode="fp64", n_part=611953,
             n_spec=20, del_t=60.0, n_steps=16),
        # 256 populations of 3e3 to 1e5 particles at their own T and p
        dict(name="batch_256", kind="batch", pop="bimodal", kernel="brown", mode="mixed", n_pop=256, n_min=3000,
             n_max=100000, n_spec=1, del_t=60.0, n_steps=150),
        # a few large populations side by side
        dict(name="batch_20spec_4x4e5", kind="batch", pop="modes3", kernel="brown", mode="mixed", n_pop=4,
             n_min=350000, n_max=450000, n_spec=20, del_t=60.0, n_steps=20),
        # run_part's loop on a small cloud: step, rebalance, output every 10 steps
        dict(name="run_part_sedi_4e3", kind="run_part", pop="drops_ln", kernel="sedi", mode="fp64", n_part=4000,
             n_spec=1, del_t=5.0, n_steps=20, n_out=10, n_bin=100),
        # the initial condition of the 20-species population, on the device
        dict(name="sample_20spec_5e5", kind="sample", n_part=500000, n_spec=20),
        # run_part's output of a large population
        dict(name="size_dist_20spec_1e6", kind="size_dist", pop="modes3", mode="fp64", n_part=1000000, n_spec=20,
             n_bin=160),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["member"] * 5 + ["mirror", "batch", "run_part", "sample", "size_dist"])
    mode = rng.choice(["fp64", "mixed"])
    if kind == "member":
        pop = rng.choice(["exp", "bimodal", "drops", "scavenge", "modes3"])
        n, steps, n_spec, del_t, kernel = {
            "exp": (_log_int(rng, 1e3, 1e6), rng.randint(1, 100), 1, 1.0, "additive"),
            "bimodal": (_log_int(rng, 3e3, 1e6), rng.randint(1, 60), 1, rng.choice([60.0, 600.0]), "brown"),
            "drops": (_log_int(rng, 1e3, 4e4), rng.randint(10, 80), 1, 5.0, "sedi"),
            "scavenge": (_log_int(rng, 3e3, 2e4), rng.randint(4, 16), 1, rng.choice([37.5, 150.0]), "brown"),
            "modes3": (_log_int(rng, 1e4, 1e6), rng.randint(5, 40), rng.randint(2, 20), 60.0, "brown"),
        }[pop]
        return dict(kind=kind, pop=pop, kernel=kernel, mode=mode, n_part=n, n_spec=n_spec, del_t=del_t, n_steps=steps)
    if kind == "mirror":
        return dict(kind=kind, pop="modes3", kernel="brown", mode=mode, n_part=_log_int(rng, 1e4, 6e5),
                    n_spec=rng.randint(2, 20), del_t=60.0, n_steps=rng.randint(4, 16))
    if kind == "batch":
        return dict(kind=kind, pop="bimodal", kernel="brown", mode=mode, n_pop=_log_int(rng, 8, 200), n_min=3000,
                    n_max=_log_int(rng, 1e4, 1e5), n_spec=1, del_t=60.0, n_steps=rng.randint(10, 100))
    if kind == "run_part":
        return dict(kind=kind, pop="drops_ln", kernel="sedi", mode=mode, n_part=_log_int(rng, 3e3, 1e4), n_spec=1,
                    del_t=5.0, n_steps=rng.randint(4, 16), n_out=4, n_bin=100)
    if kind == "sample":
        return dict(kind=kind, n_part=_log_int(rng, 1e4, 5e5), n_spec=rng.randint(2, 20))
    return dict(kind=kind, pop="modes3", mode="fp64", n_part=_log_int(rng, 1e4, 1e6), n_spec=rng.randint(1, 20),
                n_bin=rng.randint(60, 220))


# ---------------------------------------------------------------------------
# populations (host arrays, drawn from the seed)

def _sphere_volume(r):
    return 4.0 * math.pi / 3.0 * r ** 3


def _modes_of(pop, rng):
    """Log-normal modes (number concentration, median radius, log10 sigma)."""
    if pop == "scavenge":
        return [(1e11, 0.5e-8, math.log10(1.3)), (1e8, 0.25e-6, math.log10(1.3))]
    if pop == "drops_ln":
        return [(1e9, 1e-5, 0.2)]
    if pop == "modes3":
        sig = rng.uniform(1.5, 2.0, size=3)
        return [(nc, d / 2.0, math.log10(s)) for nc, d, s in zip((1e10, 1e9, 1e8), (0.02e-6, 0.1e-6, 0.5e-6), sig)]
    if pop == "bimodal":
        return [(3.2e9, 0.025e-6, math.log10(1.6)), (1e8, 0.1e-6, math.log10(1.8))]
    da, db = rng.uniform(0.03e-6, 0.08e-6), rng.uniform(0.15e-6, 0.3e-6)  # one of a batch
    sa, sb = rng.uniform(1.4, 1.9, size=2)
    return [(3.2e9, da / 2.0, math.log10(sa)), (1e8, db / 2.0, math.log10(sb))]


def _population(pop, n_part, n_spec, density, seed):
    """Species volumes (n, n_spec), weight groups and weights of one
    population of about n_part particles."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator("cuda").manual_seed(int(rng.integers(1 << 62)))
    f64 = dict(dtype=torch.float64, device="cuda", generator=gen)
    if pop in ("exp", "drops"):  # exponential volumes, mean radius 10 um, 1e9 m^-3
        vol = (-_sphere_volume(1e-5) * torch.log1p(-torch.rand(n_part, **f64)))[:, None]
        return vol.cpu().numpy(), np.ones(n_part, np.int32), pm.AeroWeightArray.flat(magnitude=1e9 / n_part)
    modes = _modes_of(pop, rng)
    kind = "nummass" if pop in ("modes3", "drops_ln") else "power"
    vols, group, mags = [], [], []
    for g, expo in enumerate(GROUPS[kind]):
        # computational particles per unit magnitude, and the weighted median
        share, median = [], []
        for nc, r, s in modes:
            x = math.log10(r)
            xp = x - expo * s * s * LN10
            share.append(nc * math.exp((xp * xp - x * x) / (2.0 * s * s)) if expo else nc)
            median.append(xp)
        mags.append(sum(share) / (n_part / len(GROUPS[kind])))
        for (nc, r, s), sh, xp in zip(modes, share, median):
            n = max(1, int(round(sh / mags[-1])))
            vols.append(_sphere_volume(10.0 ** (xp + s * torch.randn(n, **f64))))
            group.append(np.full(n, g + 1, np.int32))
    vtot = torch.cat(vols)
    if n_spec == 1:
        vol = vtot[:, None]
    else:  # Dirichlet(1) mass fractions, as volume fractions
        phi = -torch.log1p(-torch.rand(vtot.numel(), n_spec, **f64)) / torch.from_numpy(density).cuda()
        vol = phi / phi.sum(1, keepdim=True) * vtot[:, None]
    awa = pm.AeroWeightArray.power(-1.0, magnitude=mags[0]) if kind == "power" else \
        pm.AeroWeightArray.nummass(magnitudes=mags)
    return vol.cpu().numpy(), np.concatenate(group), awa


def _density(case, seed):
    if case["n_spec"] > 1:
        return np.random.default_rng([seed, 1]).uniform(1000.0, 2000.0, size=case["n_spec"])
    return np.array([1800.0 if case.get("kernel") == "brown" else 1000.0])


def _pinned(shape, dtype):
    t = torch.zeros(shape, dtype=torch.from_numpy(np.empty(0, dtype)).dtype, pin_memory=True)
    return t.numpy()


def _out_arrays(n, n_spec):
    return {"vol": _pinned((n, n_spec), np.float64), "weight_group": _pinned((n,), np.int32),
            "weight_class": _pinned((n,), np.int32), "id": _pinned((n,), np.int64),
            "n_primary_parts": _pinned((n,), np.int32)}


def _to_pinned(a):
    b = _pinned(a.shape, a.dtype)
    b[...] = a
    return b


def _mode_of(case):
    return pm.MODE_MIXED if case.get("mode") == "mixed" else pm.MODE_FP64


# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    density = _density(case, seed)
    s = {"case": case, "kind": kind, "seed": int(seed) + 17, "data": pm.AeroData(density),
         "env": pm.EnvState(TEMP, PRESSURE, ADDITIVE_COEFF)}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        n_pop = case["n_pop"]
        # log-uniform sizes, one in each of n_pop equal strata, in seeded order
        at = (rng.permutation(n_pop) + 0.5) / n_pop
        sizes = np.round(case["n_min"] * (case["n_max"] / case["n_min"]) ** at).astype(int)
        if case["pop"] == "modes3":
            temps, press = np.full(n_pop, TEMP), np.full(n_pop, PRESSURE)
        else:
            temps, press = rng.uniform(250.0, 300.0, size=n_pop), rng.uniform(5e4, 1e5, size=n_pop)
        name = "modes3" if case["pop"] == "modes3" else "bimodal_any"
        s["pops"] = []
        for n in sizes:
            vol, group, awa = _population(name, int(n), case["n_spec"], density, int(rng.integers(1 << 62)))
            s["pops"].append((_to_pinned(vol), _to_pinned(group), awa))
        s["temps"], s["press"] = temps, press
        s["empty"] = np.zeros((0, case["n_spec"]))
        s["st"] = pm.AeroState(s["data"], s["pops"][0][2], mode=_mode_of(case), n_pop=n_pop)
        s["out"] = _out_arrays(int(1.25 * sizes.sum()) + 64 * n_pop, case["n_spec"])
        return s
    if kind == "sample":
        rng = np.random.default_rng(seed)
        frac = np.full(case["n_spec"], 1.0 / case["n_spec"])
        modes = [pm.AeroMode(pm.AERO_MODE_TYPE_LOG_NORMAL, r, sg, nc, vol_frac=frac, vol_frac_std=0.1 * frac)
                 for nc, r, sg in _modes_of("modes3", rng)]
        s["dist"], s["awa"] = pm.AeroDist(modes), pm.AeroWeightArray.nummass()
        s["st"] = pm.AeroState(s["data"], s["awa"], seed=s["seed"])
        s["st"].set_n_part_ideal(case["n_part"])
        s["empty"] = np.zeros((0, case["n_spec"]))
        s["out"] = _out_arrays(2 * case["n_part"] + case["n_part"] // 2 + 1024, case["n_spec"])
        return s
    vol, group, awa = _population(case["pop"], case["n_part"], case["n_spec"], density, seed)
    s["vol"], s["group"], s["awa"] = _to_pinned(vol), _to_pinned(group), awa
    s["empty"] = np.zeros((0, case["n_spec"]))
    s["st"] = pm.AeroState(s["data"], awa, seed=s["seed"], mode=_mode_of(case))
    if kind == "size_dist":
        s["st"].add_particles(s["vol"], s["group"])
        d = 2.0 * (vol.sum(1) * 3.0 / (4.0 * math.pi)) ** (1.0 / 3.0)
        s["d_min"], s["d_max"] = 0.5 * float(d.min()), 2.0 * float(d.max())
        return s
    if kind == "mirror":
        s["mirror"] = pm.HostMirror(s["st"], cap=2 * case["n_part"] + 1024, alloc=_pinned)
        return s
    if kind == "run_part":
        s["ideal"] = case["n_part"] / len(GROUPS["nummass"])
    s["out"] = _out_arrays(4 * case["n_part"] + 1024, case["n_spec"])
    return s


def _load(s):
    """The population into the context, as a server admits a job."""
    s["st"].set_next_id(1)
    s["st"].add_particles(s["vol"], s["group"])
    s["st"].set_seed(s["seed"])


def run(s):
    case, st, kind = s["case"], s["st"], s["kind"]
    if kind == "size_dist":
        num, mass = st.size_dist(case["n_bin"], s["d_min"], s["d_max"])
        return {"num": num, "mass": mass}
    if kind == "sample":
        st.set_weight_pop(0, s["awa"])
        st.set_next_id(1)
        st.add_particles(s["empty"])
        st.set_seed(s["seed"])
        n_add = st.add_aero_dist_sample(s["dist"])
        st.particles(out=s["out"])
        return dict(s["out"], n_add=n_add, magnitude=st.weight_magnitudes())
    kernel = KERNEL[case["kernel"]]
    if kind == "batch":
        for k, (vol, group, awa) in enumerate(s["pops"]):
            st.set_weight_pop(k, awa)
            st.set_next_id(1, pop=k)
            st.add_particles(vol, group, pop=k)
            st.set_seed(s["seed"] + k, pop=k)
        tests, coags = pm.mc_coag_batch(kernel, s["temps"], s["press"], ADDITIVE_COEFF, st, case["del_t"],
                                        n_steps=case["n_steps"])
        at, counts = 0, []
        for k in range(case["n_pop"]):
            got = st.particles(pop=k, out={key: a[at:] for key, a in s["out"].items()})
            counts.append(got["id"].shape[0])
            at += counts[-1]
            st.add_particles(s["empty"], pop=k)
        return dict(s["out"], n_part=np.array(counts), tests=tests, coags=coags)
    if kind == "run_part":
        st.set_weight_pop(0, s["awa"])
    _load(s)
    tests, coags, dists = [], [], []
    for i in range(case["n_steps"]):
        a, b = pm.mc_coag(kernel, s["env"], s["data"], st, case["del_t"])
        tests.append(a)
        coags.append(b)
        if kind == "mirror":
            s["mirror"].sync()
        if kind == "run_part":
            st.rebalance(s["ideal"])
            if (i + 1) % case["n_out"] == 0:
                dists.append(st.size_dist(case["n_bin"], 1e-7, 1.0))
    res = {"tests": np.array(tests), "coags": np.array(coags)}
    if kind == "mirror":
        m = s["mirror"]
        res.update(vol=m.vol, weight_group=m.group, weight_class=m.cls, id=m.id, n_primary_parts=m.n_primary,
                   alive=m.alive, n_slots=m.n_slots)
    else:
        res.update(s["out"], n_part=st.particles(out=s["out"])["id"].shape[0])
    if kind == "run_part":
        res.update(num=np.array([d[0] for d in dists]), mass=np.array([d[1] for d in dists]),
                   magnitude=st.weight_magnitudes())
    st.add_particles(s["empty"])
    return res


def work(case):
    """The particles in and out once, and per step the cells of the size-bin
    sort (8 bytes a particle, aero_sorted's bin lists)."""
    part = 8 * case["n_spec"] + 20  # species volumes, group, class, id, primary particles
    kind = case["kind"]
    if kind == "size_dist":
        return {"bytes": case["n_part"] * (8 * case["n_spec"] + 16) + 8 * case["n_bin"] * (1 + case["n_spec"]),
                "flops": case["n_part"] * (3.0 * case["n_spec"] + 60)}
    if kind == "sample":
        return {"bytes": 2.0 * case["n_part"] * part, "flops": 2.0 * case["n_part"] * (60.0 * case["n_spec"] + 200)}
    if kind == "batch":
        lo, hi = case["n_min"], case["n_max"]
        n = case["n_pop"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)
    else:
        n = case["n_part"]
    return {"bytes": n * (2.0 * part + 8.0 * case["n_steps"]), "flops": n * 20.0 * case["n_steps"]}


def exact(case, seed):
    """The size distributions in 64 bits; the other cases' results are draws
    of a stochastic process, which have no such value."""
    if case["kind"] != "size_dist":
        return None
    density = _density(case, seed)
    vol, _, awa = _population(case["pop"], case["n_part"], case["n_spec"], density, seed)
    d = 2.0 * (vol.sum(1) * 3.0 / (4.0 * math.pi)) ** (1.0 / 3.0)
    lo, hi, n_bin = math.log(0.5 * float(d.min())), math.log(2.0 * float(d.max())), case["n_bin"]
    b = np.floor((np.log(d) - lo) / (hi - lo) * n_bin).astype(np.int64)
    inv = sum(1.0 / (m * (d / 2.0) ** e) for m, e in zip(awa.magnitude[:, 0], awa.exponent[:, 0]))
    nc = 1.0 / inv * n_bin / (hi - lo)
    num = np.bincount(b, weights=nc, minlength=n_bin)
    mass = np.stack([np.bincount(b, weights=nc * vol[:, k] * density[k], minlength=n_bin)
                     for k in range(case["n_spec"])], axis=1)
    return {"num": num, "mass": mass}
