"""Performance cases of the engine: what a program that uses it has it do.

Each case is one call, or one short sequence of calls, of the public entry
points, on the systems that the configurations, tests and benchmark of this
repository use: Kob-Andersen 80:20 mixtures at density 1.2 and
single-component Lennard-Jones liquids at density 0.8442, from 256 particles
to 2^20, alone, in batches of uneven replicas and as a served mix.

kinds of case
  run       Engine.run (Simulation.Run of one system), then the final
            configuration and energies: the plain method
  sim       the same through the RUMD classes (rumd_b200.rumd.Simulation)
  stepwise  RunStepwise: one CalcF and one Integrate call per step, for
            programs with their own work between steps
  batch     run_queued on many uneven replicas in one engine
  served    resident jobs advanced by an asynchronous chunk while a new job
            is admitted, read and removed
  forces    new positions set, list, forces, energies and stress of them
  f64       the double-precision engine's run
  noalloc   b2md_forces_noalloc on the caller's own device buffers

Positions are returned unwrapped (position + image * box), so that a particle
that sits on the box face to within rounding compares equal on either side.
"""
import ctypes
import math

import numpy as np
import torch

from rumd_b200 import capi, initconf

DEV = "cuda"
DENSITY = {"ka": 1.2, "lj": 0.8442}
PAIRS = {"ka": initconf.KA, "lj": initconf.LJ}
TAU = 0.2
IPL_EXPONENT = 18.0


def listed():
    return [
        # the smallest job of the serving stream, run alone through the RUMD
        # classes with their default launch shape: launches and barriers only
        dict(name="sim_lj256", kind="sim", model="lj", n=256, T=0.722, dt=0.004, steps=64, cutoff="SF"),
        # the plain small configuration
        dict(name="run_ka1000", kind="run", model="ka", n=1000, T=0.73, dt=0.005, skin=0.3, steps=128, cutoff="SF",
             pot="LJ_12_6", pb=64, tp=4, nvt=True),
        # an ordinary odd size: another pair function, NVE, shifted potential
        dict(name="run_smooth9973", kind="run", model="ka", n=9973, T=0.8, dt=0.005, skin=0.3, steps=64,
             cutoff="SP", pot="LJ_12_6_smooth_2_4", pb=64, tp=2, nvt=False),
        # the benchmark's headline: one large supercooled system
        dict(name="run_ka65536", kind="run", model="ka", n=65536, T=0.45, dt=0.005, skin=0.3, steps=128, cutoff="SF",
             pot="LJ_12_6", pb=64, tp=2, nvt=True),
        # the HBM-scale configuration
        dict(name="run_lj1m", kind="run", model="lj", n=1048576, T=0.722, dt=0.004, skin=0.3, steps=96, cutoff="SF",
             pot="LJ_12_6", pb=64, tp=2, nvt=True),
        # the batching configuration, with its tuned shape and skin
        dict(name="batch_ka256", kind="batch", replicas=256, n_min=512, n_max=8192, T_min=0.45, T_max=2.0, dt=0.005,
             skin=0.4, steps=96, pb=256, tp=1),
        # the server's mix of Kob-Andersen and LJ jobs of 256 to 32768 particles
        dict(name="served_mix24", kind="served", replicas=24, n_min=256, n_max=32768, T_min=0.5, T_max=2.0, dt=0.005,
             skin=0.4, steps=64, pb=256, tp=1),
        # a program's own loop over CalcF and Integrate
        dict(name="stepwise_ka4096", kind="stepwise", model="ka", n=4096, T=0.8, dt=0.005, steps=16, cutoff="SF"),
        # new configurations evaluated from outside: upload, sort, list, forces, stress
        dict(name="forces_ka32000", kind="forces", model="ka", n=32000, cutoff="SF", pot="LJ_12_6", skin=0.3, pb=64,
             tp=4, stress=True),
        # the double-precision engine on the size its accuracy is stated at
        dict(name="f64_lj32000", kind="f64", model="lj", n=32000, T=0.722, dt=0.004, skin=0.3, steps=16, cutoff="SF"),
        # a plugin with its own device buffers: a small system, and the largest but odd
        dict(name="noalloc_ka1000", kind="noalloc", model="ka", n=1000, cutoff="SF"),
        dict(name="noalloc_ka65521", kind="noalloc", model="ka", n=65521, cutoff="SP"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds, sizes spread over their ranges."""
    kind = rng.choice(["run", "run", "run", "sim", "stepwise", "batch", "served", "forces", "f64", "noalloc"])
    model = rng.choice(["ka", "lj"])
    cutoff = rng.choice(["SF", "SF", "SP"])
    pot = rng.choice(["LJ_12_6", "LJ_12_6", "LJ_12_6_smooth_2_4", "IPL_n"])
    T = round(rng.uniform(0.5, 1.5), 3)
    dt = 0.005 if model == "ka" else 0.004
    skin = rng.choice([0.3, 0.4])
    if kind == "run":
        return dict(kind=kind, model=model, n=_log_int(rng, 500, 700000), T=T, dt=dt, skin=skin,
                    steps=rng.randint(48, 96), cutoff=cutoff, pot=pot, pb=rng.choice([32, 64, 128]),
                    tp=rng.choice([1, 2, 4]), nvt=rng.random() < 0.7)
    if kind == "sim":
        return dict(kind=kind, model=model, n=_log_int(rng, 256, 20000), T=T, dt=dt, steps=rng.randint(48, 96),
                    cutoff=cutoff)
    if kind == "stepwise":
        return dict(kind=kind, model=model, n=_log_int(rng, 500, 60000), T=T, dt=dt, steps=rng.randint(8, 24),
                    cutoff=cutoff)
    if kind == "batch":
        return dict(kind=kind, replicas=rng.randint(32, 200), n_min=512, n_max=_log_int(rng, 2048, 8192), T_min=0.45,
                    T_max=2.0, dt=0.005, skin=0.4, steps=rng.randint(48, 96), pb=rng.choice([128, 256]),
                    tp=rng.choice([1, 2]))
    if kind == "served":
        return dict(kind=kind, replicas=rng.randint(6, 40), n_min=256, n_max=_log_int(rng, 4096, 32768), T_min=0.5,
                    T_max=2.0, dt=0.005, skin=0.4, steps=rng.randint(48, 96), pb=256, tp=1)
    if kind == "forces":
        return dict(kind=kind, model=model, n=_log_int(rng, 500, 300000), cutoff=cutoff, pot=pot, skin=skin, pb=64,
                    tp=rng.choice([2, 4]), stress=rng.random() < 0.5)
    if kind == "f64":
        return dict(kind=kind, model=model, n=_log_int(rng, 1000, 60000), T=T, dt=dt, skin=skin,
                    steps=rng.randint(8, 24), cutoff=cutoff)
    return dict(kind=kind, model=model, n=_log_int(rng, 500, 65536), cutoff=cutoff)


# ---- inputs ----------------------------------------------------------------

def _params(model, pot="LJ_12_6"):
    ntypes = 2 if model == "ka" else 1
    if pot == "LJ_12_6":
        p = initconf.lj_params(ntypes, PAIRS[model])
    elif pot == "LJ_12_6_smooth_2_4":
        p = initconf.smooth_params(ntypes, PAIRS[model])
    else:
        p = initconf.ipl_n_params(ntypes, IPL_EXPONENT, PAIRS[model])
    return p, ntypes


def _config(model, n, T, seed):
    """A disordered start: n of the sites of the smallest FCC lattice with at
    least n sites (vacancies at random), displaced by thermal noise; random
    types; Maxwell-Boltzmann velocities without net momentum."""
    g = torch.Generator().manual_seed(int(seed) * 1000003 + n)
    m = 1
    while 4 * m ** 3 < n:
        m += 1
    L = np.float32((n / DENSITY[model]) ** (1.0 / 3.0))
    a = float(L) / m
    k = torch.arange(m, dtype=torch.float64)
    cell = torch.stack(torch.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 1, 3)
    basis = torch.tensor([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]], dtype=torch.float64)
    sites = (cell + basis).reshape(-1, 3)
    keep = torch.randperm(len(sites), generator=g)[:n].sort().values
    pos = (sites[keep] + 0.25) * a - float(L) / 2
    pos += 0.03 * torch.randn(n, 3, generator=g)
    pos -= float(L) * torch.round(pos / float(L))
    types = np.zeros(n, np.int32)
    if model == "ka":
        types[torch.randperm(n, generator=g)[: n // 5].numpy()] = 1
    vel = torch.randn(n, 3, generator=g) * math.sqrt(T)
    vel -= vel.mean(0)
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :3] = pos.numpy()
    pos4[:, 3] = types.view(np.float32)
    vel4 = np.ones((n, 4), np.float32)
    vel4[:, :3] = vel.numpy()
    return dict(pos4=pos4, vel4=vel4, box=np.array([L, L, L], np.float32), types=types)


def _replicas(case, seed):
    """(model, n, T) of the replicas of a batch or served mix (a served mix
    draws KA or LJ for each job; its last one is the job that comes and goes).
    The sizes belong to the case; the configurations follow the seed."""
    rng = np.random.default_rng(case["replicas"] * 7919 + case["n_max"])
    R = case["replicas"] + (1 if case["kind"] == "served" else 0)
    ns = np.floor(np.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]), R))).astype(int)
    if case["kind"] == "batch":
        Ts = np.exp(np.linspace(math.log(case["T_min"]), math.log(case["T_max"]), R))
        models = ["ka"] * R
    else:
        Ts = rng.uniform(case["T_min"], case["T_max"], R)
        models = [("ka", "lj")[int(k)] for k in rng.integers(0, 2, R)]
    return [(m, int(n), float(T), _config(m, int(n), float(T), seed * 1009 + k))
            for k, (m, n, T) in enumerate(zip(models, ns, Ts))]


def _rumd_sample(case, conf):
    from rumd_b200 import rumd
    s = rumd.Sample()
    s.SetVerbose(False)
    masses = [1.0, 1.0] if case["model"] == "ka" else [1.0]
    s.SetConfiguration(conf["pos4"][:, :3], conf["types"].tolist(), conf["box"].tolist(), masses,
                       conf["vel4"][:, :3])
    pot = rumd.Pot_LJ_12_6(cutoff_method={"SF": rumd.ShiftedForce, "SP": rumd.ShiftedPotential}[case["cutoff"]])
    for (i, j), (sigma, eps, rc) in PAIRS[case["model"]].items():
        pot.SetParams(i, j, sigma, eps, rc)
    pot.SetNbListSkin(0.3)
    sim = rumd.Simulation(sample=s, verbose=False)
    sim.SetPotential(pot)
    sim.SetIntegrator(rumd.IntegratorNVT(timeStep=case["dt"], targetTemperature=case["T"],
                                         thermostatRelaxationTime=TAU))
    return sim


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind in ("batch", "served"):
        reps = _replicas(case, seed)
        e = capi.Engine(max_particles=int(sum(r[1] for r in reps) + 64 * len(reps)), max_replicas=len(reps),
                        pb=case["pb"], tp=case["tp"])
        if kind == "served":
            e.set_variant(capi.VARIANT_PERSISTENT, 3)
        st.update(e=e, reps=reps, ids=[])
        for r in reps[: case["replicas"]]:
            st["ids"].append(_add(e, case, r))
        e.sync()
        return st
    conf = _config(case["model"], case["n"], case.get("T", 1.0), seed)
    st["conf"] = conf
    if kind in ("sim", "stepwise"):
        st["sim"] = _rumd_sample(case, conf)
        st["sim"].sample.CalcF()
        return st
    params, ntypes = _params(case["model"], case.get("pot", "LJ_12_6"))
    if kind in ("run", "forces"):
        e = capi.Engine(pb=case["pb"], tp=case["tp"])
        rid = e.add(conf["pos4"], conf["box"], params, ntypes, cutoff=case["cutoff"], skin=case["skin"],
                    dt=case.get("dt", 0.005), T=case.get("T", 1.0), tau=TAU, thermostat=case.get("nvt", True),
                    vel4=conf["vel4"], potential=case["pot"])
        e.sync()
        st.update(e=e, rid=rid)
    elif kind == "f64":
        st["e"] = capi.F64Engine(conf["pos4"], conf["box"].astype(np.float64), params, ntypes, cutoff=case["cutoff"],
                                 skin=case["skin"], dt=case["dt"], T=case["T"], tau=TAU,
                                 vel4=conf["vel4"].astype(np.float64))
    else:
        st.update(pos=torch.from_numpy(conf["pos4"]).to(DEV), force=torch.empty(case["n"], 4, device=DEV),
                  sums=torch.zeros(2, dtype=torch.float64, device=DEV), params=params, ntypes=ntypes)
    return st


def _add(e, case, r):
    model, n, T, c = r
    params, ntypes = _params(model)
    return e.add(c["pos4"], c["box"], params, ntypes, cutoff="SF", skin=case["skin"], dt=case["dt"], T=T, tau=TAU,
                 vel4=c["vel4"])


# ---- one pass --------------------------------------------------------------

def _state(e, rid, n, box):
    p, v, im = e.read(rid, n)
    return p[:, :3] + im.astype(np.float32) * box, v[:, :3]


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "run":
        e, rid = st["e"], st["rid"]
        e.run(case["steps"])
        pos, vel = _state(e, rid, case["n"], st["conf"]["box"])
        s = e.stats(rid)
        return dict(pos=pos, vel=vel, energy=np.array([s["pe"], s["virial"], s["ke"]]))
    if kind == "sim":
        sim = st["sim"]
        sim.Run(case["steps"])
        s = sim.sample
        return dict(pos=s.GetPositions() + np.asarray(s.GetImages(), np.float32) * st["conf"]["box"],
                    vel=s.GetVelocities(), energy=np.array([s.GetPotentialEnergy(), s.GetVirial()]))
    if kind == "stepwise":
        sim, pe = st["sim"], []
        sim.RunStepwise(case["steps"], lambda i, s: pe.append(s.GetPotentialEnergy()))
        s = sim.sample
        return dict(pos=s.GetPositions() + np.asarray(s.GetImages(), np.float32) * st["conf"]["box"],
                    vel=s.GetVelocities(), pe=np.array(pe), force=s.GetForces())
    if kind == "batch":
        e = st["e"]
        for rid in st["ids"]:
            e.queue(rid, case["steps"])
        _, snap = e.wait(e.run_queued_async())
        cols = [capi.CHUNK_FIELDS.index(k) for k in ("pe", "virial", "ke")]
        got = [_state(e, rid, r[1], r[3]["box"]) for rid, r in zip(st["ids"], st["reps"])]
        return dict(pos=np.concatenate([g[0] for g in got]), vel=np.concatenate([g[1] for g in got]),
                    energy=snap[st["ids"]][:, cols])
    if kind == "served":
        e = st["e"]
        for rid in st["ids"]:
            e.queue(rid, case["steps"])
        ticket = e.run_queued_async(case["steps"] // 2)
        # a job arrives while the chunk runs, joins the next one and leaves
        r = st["reps"][-1]
        new = _add(e, case, r)
        e.queue(new, case["steps"])
        t2 = e.run_queued_async()
        e.wait(ticket)
        _, snap = e.wait(t2)
        pos, vel = _state(e, new, r[1], r[3]["box"])
        e.remove(new)
        cols = [capi.CHUNK_FIELDS.index(k) for k in ("pe", "virial", "ke")]
        got = [_state(e, rid, x[1], x[3]["box"]) for rid, x in zip(st["ids"], st["reps"])]
        return dict(pos=np.concatenate([g[0] for g in got] + [pos]), vel=np.concatenate([g[1] for g in got] + [vel]),
                    energy=snap[st["ids"] + [new]][:, cols])
    if kind == "forces":
        e, rid, n = st["e"], st["rid"], case["n"]
        e.set(rid, "pos", st["conf"]["pos4"])
        e.calc_f(case["stress"])
        s = e.stats(rid)
        out = dict(force=e.get(rid, "force", n), energy=np.array([s["pe"], s["virial"]]))
        if case["stress"]:
            out["stress"] = e.stress(rid)
        return out
    if kind == "f64":
        e = st["e"]
        en = e.run(case["steps"], energies=True)
        return dict(pos=e.get("pos")[:, :3] + e.get("images") * st["conf"]["box"].astype(np.float64),
                    vel=e.get("vel")[:, :3], energy=en[:, :3])
    rc = capi.lib().b2md_forces_noalloc(
        ctypes.c_void_p(st["pos"].data_ptr()), case["n"], st["conf"]["box"].ctypes.data_as(ctypes.c_void_p),
        st["ntypes"], st["params"].ctypes.data_as(ctypes.c_void_p), capi.CUTOFF[case["cutoff"]],
        ctypes.c_void_p(st["force"].data_ptr()), ctypes.c_void_p(st["sums"].data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    capi.check(rc)
    return dict(force=st["force"], sums=st["sums"])


# ---- what a pass cannot do without ------------------------------------------

def _pairs_in_range(model, n):
    """Mean neighbours of a particle inside the cut-off, at uniform density."""
    rho = DENSITY[model]
    x = (0.8, 0.2) if model == "ka" else (1.0,)
    tot = 0.0
    for i, xi in enumerate(x):
        for j, xj in enumerate(x):
            sigma, _, rc = PAIRS[model][(min(i, j), max(i, j))]
            tot += xi * xj * rho * 4.0 / 3.0 * math.pi * (rc * sigma) ** 3
    return min(tot, n - 1.0)


def work(case):
    """Bytes: state read and written, and the list of neighbours in range (4 B
    each) read once a step; flops: 30 per ordered pair in range and step."""
    kind = case["kind"]
    if kind in ("batch", "served"):
        reps = [(m, n) for m, n, _, _ in _sizes(case)]
    else:
        reps = [(case["model"], case["n"])]
    steps = case.get("steps", 1)
    wide = 2 if kind == "f64" else 1
    by = fl = 0.0
    for m, n in reps:
        nb = _pairs_in_range(m, n)
        fl += 30.0 * n * nb * steps
        if kind == "noalloc":
            by += 32.0 * n
        elif kind == "forces":
            by += n * (16 + 16 + 4 * nb)
        else:
            by += n * steps * (wide * 96.0 + 4 * nb)
    return dict(bytes=by, flops=fl)


def _sizes(case):
    rng = np.random.default_rng(case["replicas"] * 7919 + case["n_max"])
    R = case["replicas"] + (1 if case["kind"] == "served" else 0)
    ns = np.floor(np.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]), R))).astype(int)
    if case["kind"] == "batch":
        return [("ka", int(n), 0.0, None) for n in ns]
    rng.uniform(case["T_min"], case["T_max"], R)
    return [(("ka", "lj")[int(k)], int(n), 0.0, None) for n, k in zip(ns, rng.integers(0, 2, R))]


def tolerance(case):
    """About four times what another order of the pair sums (other threads per
    particle) shows after two passes: rounding differences of one evaluation
    (1e-7) grow along a trajectory, the more the longer it is; velocities show
    the most (6e-5 after 2 x 64 steps, 3e-4 after 2 x 128).  Single force
    evaluations are 2e-6 to 4e-6 from the 64-bit sums."""
    kind = case["kind"]
    if kind == "f64":
        return {"rel": 1e-9, "max": 1e-6}
    if kind in ("forces", "noalloc"):
        return {"rel": 1e-5, "max": 1e-3}
    if kind == "stepwise":
        return {"rel": 2e-5, "max": 2e-3}
    return {"rel": 1.5e-3, "max": 0.05} if case["steps"] > 72 else {"rel": 5e-4, "max": 0.02}


# ---- the same in 64 bits ----------------------------------------------------

class _Exact:
    """Systems side by side in float64 torch: full Verlet lists, the pair
    functions, Nose-Hoover leap-frog."""

    SKIN = 0.5

    def __init__(self, systems, cutoff, pot, dt, nvt, params_of):
        self.cutoff, self.pot, self.dt, self.nvt = cutoff, pot, dt, nvt
        T64 = dict(dtype=torch.float64, device=DEV)
        self.r = torch.cat([torch.from_numpy(c["pos4"][:, :3]).to(DEV).double() for _, _, _, c in systems])
        self.v = torch.cat([torch.from_numpy(c["vel4"][:, :3]).to(DEV).double() for _, _, _, c in systems])
        self.n = [s[1] for s in systems]
        self.sys = torch.repeat_interleave(torch.arange(len(systems), device=DEV), torch.tensor(self.n, device=DEV))
        self.Ls = torch.tensor([float(s[3]["box"][0]) for s in systems], **T64)
        self.Ts = torch.tensor([s[2] for s in systems], **T64)
        self.L = self.Ls[self.sys][:, None]
        # one table for all systems: KA types 0, 1 and LJ type 2
        tab = torch.zeros(3, 3, 12, **T64)
        for m, off in (("ka", 0), ("lj", 2)):
            p, nt = params_of(m)
            tab[off:off + nt, off:off + nt] = torch.from_numpy(p.reshape(nt, nt, 12)).to(DEV).double()
        self.tab = tab.reshape(9, 12)
        self.types = torch.cat([torch.from_numpy(c["types"]).to(DEV).long() + (2 if m == "lj" else 0)
                                for m, _, _, c in systems])
        self.models = [s[0] for s in systems]
        self.xi = torch.zeros(len(systems), **T64)
        self.ref = None

    def _lists(self):
        rc = [float(max(x[2] * x[0] for x in PAIRS[m].values())) + self.SKIN for m in self.models]
        rows, base = [], 0
        for m, n, c in zip(self.models, self.n, rc):
            r = self.r[base:base + n]
            L = float(self.Ls[len(rows)])
            rows.append(self._one_list(r - L * torch.round(r / L), L, c) + base)
            base += n
        K = max(x.shape[1] for x in rows)
        self.nbr = torch.cat([torch.cat([x, (x[:, :1] * 0 - 1).expand(-1, K - x.shape[1])], 1) for x in rows])
        base = 0
        for x, n in zip(rows, self.n):   # padding (base - 1 in a row) to -1
            part = self.nbr[base:base + n]
            part[part < base] = -1
            base += n
        self.ref = self.r.clone()

    @staticmethod
    def _one_list(r, L, rc):
        """[n, K] neighbours within rc, padded with -1."""
        n = len(r)
        nc = int(L / rc)
        rows = []
        if nc < 4 or n < 3000:
            cand = torch.arange(n, device=DEV)[None, :]
            cells = None
        else:
            c3 = torch.clamp(((r / L + 0.5) * nc).long(), 0, nc - 1)
            key = c3[:, 0] + nc * (c3[:, 1] + nc * c3[:, 2])
            order = torch.argsort(key)
            cnt = torch.bincount(key, minlength=nc ** 3)
            occ = int(cnt.max())
            start = torch.cumsum(cnt, 0) - cnt
            slots = torch.arange(occ, device=DEV)[None, :]
            cells = torch.where(slots < cnt[:, None], order[torch.clamp(start[:, None] + slots, max=n - 1)], -1)
            k = torch.arange(-1, 2, device=DEV)
            off = torch.stack(torch.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
        step = max(1, 30_000_000 // (n if cells is None else 27 * cells.shape[1]))
        for b in range(0, n, step):
            i = torch.arange(b, min(n, b + step), device=DEV)
            if cells is not None:
                o = (c3[i][:, None, :] + off[None]) % nc
                cand = cells[o[..., 0] + nc * (o[..., 1] + nc * o[..., 2])].reshape(len(i), -1)
            j = cand.expand(len(i), -1)
            d = r[i][:, None, :] - r[torch.clamp(j, min=0)]
            d -= L * torch.round(d / L)
            ok = ((d * d).sum(-1) < rc * rc) & (j >= 0) & (j != i[:, None])
            K = int(ok.sum(1).max())
            idx = torch.argsort((~ok).to(torch.int8), dim=1, stable=True)[:, :K]
            rows.append(torch.where(torch.gather(ok, 1, idx), torch.gather(j, 1, idx), -1))
        K = max(x.shape[1] for x in rows)
        return torch.cat([torch.nn.functional.pad(x, (0, K - x.shape[1]), value=-1) for x in rows])

    def forces(self):
        if self.ref is None or float((self.r - self.ref).square().sum(1).max()) > (0.5 * self.SKIN) ** 2:
            self._lists()
        N = len(self.r)
        f = torch.empty_like(self.r)
        u = torch.empty(N, dtype=torch.float64, device=DEV)
        w = torch.empty_like(u)
        stress = torch.zeros(6, dtype=torch.float64, device=DEV)
        step = max(1, 40_000_000 // self.nbr.shape[1])
        for b in range(0, N, step):
            i = slice(b, min(N, b + step))
            j = self.nbr[i]
            jj = torch.clamp(j, min=0)
            L = self.L[i]
            dx = []
            d2 = 0
            for k in range(3):
                x = self.r[i, k][:, None] - self.r[:, k][jj]
                x -= L * torch.round(x / L)
                dx.append(x)
                d2 = d2 + x * x
            p = self.types[i][:, None] * 3 + self.types[jj]
            q = lambda k: self.tab[:, k][p]  # noqa: E731
            rc = q(0)
            s, e = self._pair(d2, q)
            if self.cutoff in ("SF", "SP"):
                sc, uc = self._pair(rc * rc, q)
                if self.cutoff == "SF":
                    d = d2.sqrt()
                    s = s - sc * rc / d
                    e = e + sc * rc * (d - rc)
                e = e - uc
            ok = (d2 < rc * rc) & (j >= 0)
            s = torch.where(ok, s, 0.0)
            u[i] = 0.5 * torch.where(ok, e, 0.0).sum(1)
            w[i] = (d2 * s).sum(1)
            for k in range(3):
                f[i, k] = (dx[k] * s).sum(1)
            for m, (k, l) in enumerate(((0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1))):
                stress[m] -= (dx[k] * dx[l] * s).sum()
        self.u, self.w, self.f, self.stress = u, w, f, stress
        return f

    def _pair(self, d2, q):
        if self.pot == "LJ_12_6":
            i2 = 1.0 / d2
            i6 = i2 * i2 * i2
            return i6 * i2 * (12.0 * q(1) * i6 + 6.0 * q(2)), i6 * (q(1) * i6 + q(2))
        if self.pot == "LJ_12_6_smooth_2_4":
            x = d2 * q(1)
            i2 = 1.0 / x
            i6 = i2 * i2 * i2
            s = q(2) * q(1) * (i2 * i6 * (12.0 * i6 - 6.0) - 2.0 * q(3) - 4.0 * q(4) * x)
            return s, q(2) * (i6 * (i6 - 1.0) + q(3) * x + q(4) * x * x)
        i2 = 1.0 / (d2 * q(1))
        t = i2 ** (0.5 * q(3))
        return q(1) * q(2) * q(3) * t * i2, q(2) * t

    def sums(self, x):
        return torch.zeros_like(self.Ls).index_add_(0, self.sys, x)

    def step(self, reset):
        if reset:
            p = torch.zeros(len(self.n), 3, dtype=torch.float64, device=DEV).index_add_(0, self.sys, self.v)
            self.v = self.v - (p / torch.tensor(self.n, dtype=torch.float64, device=DEV)[:, None])[self.sys]
        self.forces()
        h = (0.5 * self.xi * self.dt if self.nvt else self.xi * 0)[self.sys][:, None]
        vb = (self.v * self.v).sum(1)
        self.v = ((1.0 - h) * self.v + self.f * self.dt) / (1.0 + h)
        self.r = self.r + self.v * self.dt
        vf = (self.v * self.v).sum(1)
        self.ke = self.sums(0.25 * (vb + vf))
        if self.nvt:
            dof = torch.tensor([3.0 * n - 3.0 for n in self.n], dtype=torch.float64, device=DEV)
            dev = torch.clamp(self.sums(vf) / (dof * self.Ts) - 1.0, max=10.0)
            self.xi = self.xi + self.dt * (4.0 * math.pi ** 2 / TAU ** 2) * dev

    def energy(self):
        return torch.stack([self.sums(self.u), self.sums(self.w) / 6.0, self.ke], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "served"):
        reps = _replicas(case, seed)
    else:
        reps = [(case["model"], case["n"], case.get("T", 1.0), _config(case["model"], case["n"], case.get("T", 1.0),
                                                                        seed))]
    pot = case.get("pot", "LJ_12_6")
    x = _Exact(reps, case.get("cutoff", "SF"), pot, float(np.float32(case.get("dt", 0.005))), case.get("nvt", True),
               lambda m: _params(m, pot))
    if kind == "f64":
        x.dt = case["dt"]
    if kind in ("forces", "noalloc"):
        x.forces()
        f4 = torch.cat([x.f, x.u[:, None]], 1)
        sums = torch.stack([x.u.sum(), x.w.sum() / 6.0])
        if kind == "noalloc":
            return dict(force=f4, sums=sums)
        out = dict(force=f4, energy=sums)
        if case["stress"]:
            out["stress"] = 0.5 * x.stress / x.Ls[0] ** 3
        return out
    rows = []
    for k in range(case["steps"]):
        x.step(k % 100 == 0)
        rows.append(x.energy())
    if kind == "f64":
        return dict(pos=x.r, vel=x.v, energy=torch.cat(rows))
    if kind == "stepwise":
        x.forces()
        return dict(pos=x.r, vel=x.v, pe=torch.cat(rows)[:, 0], force=x.f)
    if kind in ("batch", "served"):
        # the snapshot's energies are those of the last step's force evaluation
        return dict(pos=x.r, vel=x.v, energy=rows[-1])
    x.forces()
    return dict(pos=x.r, vel=x.v, energy=x.energy()[0, :2] if kind == "sim" else x.energy()[0])
