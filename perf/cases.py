"""What the speed of this framework is measured on: a dozen uses of its public entry points.

Five kinds of work, over the sizes of the repository's own workloads (beep_gb300.synth),
tests and benchmark:

sim      one batch of particles simulated and scored (``DeviceModel.simulate``,
         ``DeviceBatch.run`` / ``run_graph``): an ABC-SMC generation, a PMCMC batch, a
         scenario with trajectories; in the fast form and in the plain FP64 form
pf       a particle-filter likelihood estimate (``DeviceModel.pf_loglik``)
mbp      a sweep of MBP proposals and their acceptance (``MbpChains``)
weights  ABC-SMC importance weights of a generation (``abcsmc_weights``)
serve    a stream of requests of mixed sizes through a ``Server``, from its start to its end

A case is a dict of sizes.  The synthetic epidemics (populations, mixing, observed data)
come from the sizes alone; the seed draws the parameter sets and the variates.
"""
import functools
import math
import random

import numpy as np
import torch

from beep_gb300 import capi, model_builder, synth

T, C = 6, 6                       # transitions and compartments of the SEIR-H-D family
FORMS = {"fast": capi.FORM_FAST, "plain": capi.FORM_PLAIN_FP64}
MBP_ALL = ",".join("%dx%d" % s for s in synth.MBP_SIZES)


def sim(name, **kw):
    case = dict(kind="sim", recipe="small", areas=10, ages=3, days=100, spd=4, particles=16, sets=16, form="fast",
                call="simulate", traj=False, pop=False)
    case.update(kw)
    return dict(case, name=name)


def listed():
    return [
        # one PMCMC likelihood estimate, the inner loop of PMCMC: 256 particles, 400 dependent
        # steps of a small model, where latency and launches count
        dict(kind="pf", name="pf_estimate", areas=10, ages=3, days=100, spd=4, particles=256, section=28, form="fast"),
        # the same estimate in the form that reproduces the CPU program bit for bit (the default form)
        dict(kind="pf", name="pf_estimate_fp64", areas=10, ages=3, days=100, spd=4, particles=256, section=28,
             form="plain"),
        # a scenario run: a few trajectories of a small model brought back whole, the smallest call
        sim("scenario_trajectories", particles=16, traj=True, pop=True),
        # a generation of ABC-SMC on a regional model, each particle with its own parameters
        sim("abc_generation_40x4", recipe="abc", areas=40, ages=4, days=180, spd=2, particles=2048, sets=2048),
        # a large generation: the headline workload, staged and replayed as a graph as a sampler does
        sim("abc_generation_150x4", recipe="abc", areas=150, ages=4, days=180, spd=2, particles=16384, sets=16384,
            call="graph"),
        # a PMCMC batch of the largest model, one parameter set, a year at four steps a day
        sim("pmcmc_batch_350x10", recipe="precision", areas=350, ages=10, days=365, spd=4, particles=1024, sets=1,
            call="run"),
        # two strains, of odd sizes, with the final populations read back
        sim("two_strains_71x2", recipe="strains", areas=71, ages=2, days=60, spd=4, particles=901, sets=7, call="run",
            pop=True),
        # an ordinary batch in the FP64 form, of odd sizes
        sim("batch_fp64_77x5", areas=77, ages=5, days=90, spd=2, particles=187, sets=11, form="plain", call="run",
            pop=True),
        # a sweep of MBP chains over four models of uneven size
        dict(kind="mbp", name="mbp_sweep_uneven", sizes=MBP_ALL, days=200, spd=2, chains=128, form="fast"),
        # a sweep of a few FP64 chains, with the likelihood of their states under new parameters
        dict(kind="mbp", name="mbp_sweep_fp64", sizes="33x3", days=200, spd=2, chains=48, form="plain"),
        # the importance weights of a large ABC-SMC generation
        dict(kind="weights", name="abc_weights_16384", new=16384, last=16384, nvar=3),
        # requests of mixed sizes and kinds through the serving engine
        dict(kind="serve", name="serve_mixed", requests=16, mix=7, areas=200, ages=8, days=150, particles=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("pf", "sim", "sim", "sim", "sim", "mbp", "weights", "serve"))
    form = rng.choice(("fast", "fast", "plain"))
    if kind == "pf":
        return dict(kind=kind, areas=_log_int(rng, 3, 40), ages=rng.randint(1, 5), days=rng.randint(30, 100),
                    spd=rng.choice((2, 4)), particles=_log_int(rng, 32, 1024 if form == "fast" else 300),
                    section=rng.randint(7, 60), form=form)
    if kind == "weights":
        return dict(kind=kind, new=_log_int(rng, 64, 16384), last=_log_int(rng, 64, 16384), nvar=rng.randint(1, 9))
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(2, 16), mix=rng.randint(0, 1 << 20), areas=rng.randint(20, 200),
                    ages=rng.randint(1, 8), days=rng.randint(60, 150), particles=_log_int(rng, 64, 1024))
    if kind == "mbp":
        n = rng.randint(1, 4 if form == "fast" else 1)
        hi = 200 if form == "fast" else 60
        sizes = ["%dx%d" % (_log_int(rng, 10, hi), rng.randint(1, 6)) for _ in range(n)]
        return dict(kind=kind, sizes=",".join(sizes), days=rng.randint(60, 200), spd=2,
                    chains=_log_int(rng, 8, 128 if form == "fast" else 48), form=form)
    recipe = rng.choice(("small", "abc", "precision", "strains"))
    areas, ages = _log_int(rng, 5, 350), rng.randint(1, 10)
    days, spd = rng.randint(40, 200), rng.choice((2, 4))
    if recipe == "precision":
        ages, days = max(3, ages), max(90, days)
    if recipe == "strains":
        areas, ages = min(areas, 150), min(ages, 4)
    if form == "plain":                 # its particles take about a second per million steps of an area and age
        areas = max(3, min(areas, 250000 // (ages * days * spd)))
    units = areas * ages * days * spd
    particles = min(_log_int(rng, 1, 16384), max(1, int((1.5e9 if form == "fast" else 1.2e7) / units)))
    traj = rng.random() < 0.25 and particles * units * (T + C) < 2e7
    call = rng.choice(("simulate", "run", "graph"))
    sets = rng.choice((1, min(particles, rng.randint(2, 40)), particles)) if recipe in ("small", "abc") else 1
    return dict(kind="sim", recipe=recipe, areas=areas, ages=ages, days=days, spd=spd, particles=particles, sets=sets,
                form=form, call=call, traj=traj, pop=rng.random() < 0.5)


# ---- inputs ---------------------------------------------------------------

@functools.lru_cache(maxsize=16)
def _epidemic(recipe, areas, ages, days, spd):
    """(workload, model arrays): the observed data are one simulated epidemic plus noise."""
    if recipe == "abc":
        w = synth.abc_smc_large(narea=areas, nage=ages, days=days, steps_per_day=spd)
    elif recipe == "precision":
        w = synth.precision_large(narea=areas, nage=ages, days=days, steps_per_day=spd)
    elif recipe == "strains":
        w = synth.seir_hd_strains(narea=areas, nage=ages, days=days)
        w.steps_per_day = spd
    else:
        w = synth.seir_hd_small(narea=areas, nage=ages, days=days, steps_per_day=spd)
        if recipe == "hosp":
            w.obs_kind = "hosp_pop"
    arr = model_builder.model_arrays(w)
    m = capi.Model(arr)
    dm = capi.DeviceModel(m)
    truth = dm.simulate(capi.Batch(m, [capi.Tables(model_builder.param_tables(w))], 1, 17, want_transnum=True,
                                   want_pop_traj=True, want_L=False, form=capi.FORM_FAST))
    dm.close()
    y, sd = model_builder.observed_from_trajectory(arr, truth.transnum[0], truth.pop_traj[0], np.random.default_rng(1))
    return w, dict(arr, obs_value=y, obs_sd=sd)


def _table_arrays(w, recipe, sets, rng):
    if recipe in ("precision", "strains"):      # one proposal each around the workload's own parameters
        return [model_builder.param_tables(w, w.sigma_inv * rng.uniform(0.9, 1.1), w.gamma_inv * rng.uniform(0.9, 1.1),
                                           rng.uniform(0.9, 1.1)) for _ in range(sets)]
    return model_builder.param_tables_batch(w, *synth.abc_smc_priors(rng, sets))


def _sections(S, k):
    return [(a, min(a + k, S)) for a in range(0, S, k)]


def _sim_inputs(case, seed):
    w, arr = _epidemic(case["recipe"], case["areas"], case["ages"], case["days"], case["spd"])
    tabs = _table_arrays(w, case["recipe"], case["sets"], np.random.default_rng(seed))
    return arr, tabs, np.arange(case["particles"]) % case["sets"]


def _mbp_inputs(case, seed):
    """Per model: (arrays, current tables, proposed tables)."""
    rng, n, out = np.random.default_rng(seed), case["chains"], []
    for size in case["sizes"].split(","):
        A, G = map(int, size.split("x"))
        w, arr = _epidemic("hosp", A, G, case["days"], case["spd"])
        th = np.stack([rng.uniform(2.2, 2.8, n), rng.uniform(3.6, 4.4, n), rng.uniform(4.5, 5.5, n)], 1)
        tp = th * np.exp(rng.normal(0, 0.05, th.shape))
        out.append((arr, model_builder.param_tables_batch(w, *th.T), model_builder.param_tables_batch(w, *tp.T)))
    return out


def _weights_inputs(case, seed):
    rng, nv = np.random.default_rng(seed), case["nvar"]
    lo, hi = np.linspace(1.0, 3.0, nv), np.linspace(4.0, 8.0, nv)
    tl = rng.uniform(lo, hi, (case["last"], nv))
    wl = rng.uniform(0.2, 2.0, case["last"])
    tn = np.clip(tl[rng.integers(0, case["last"], case["new"])] + rng.normal(0, 0.2, (case["new"], nv)), lo, hi)
    ic = np.linalg.inv(np.atleast_2d(np.cov(tl.T, aweights=wl)) + 1e-9 * np.eye(nv))
    return tn, np.full(case["new"], -np.log(np.prod(hi - lo))), tl, wl, ic


def _serve_sizes(case):
    """The requests' sizes: areas, ages, days, steps a day, particles, kind."""
    rng, out = random.Random(case["mix"]), []
    for k in range(case["requests"]):
        out.append((rng.randint(10, case["areas"]), rng.randint(1, case["ages"]), rng.randint(60, max(60, case["days"])),
                    rng.choice((2, 4)), _log_int(rng, 64, case["particles"]), k % 3))
    return out


def prepare(case, seed):
    st = dict(case=case)
    form = FORMS.get(case.get("form"))
    if case["kind"] == "sim":
        arr, tabs, group_of = _sim_inputs(case, seed)
        st["m"] = capi.Model(arr)
        st["dm"] = capi.DeviceModel(st["m"])
        st["batch"] = capi.Batch(st["m"], [capi.Tables(t) for t in tabs], case["particles"], seed, group_of=group_of,
                                 want_pop=case["pop"], want_transnum=case["traj"], want_pop_traj=case["traj"], form=form)
        if case["call"] != "simulate":
            st["db"] = capi.DeviceBatch(st["dm"], st["batch"])
    elif case["kind"] == "pf":
        w, arr = _epidemic("small", case["areas"], case["ages"], case["days"], case["spd"])
        rng = np.random.default_rng(seed)
        st["m"] = capi.Model(arr)
        st["dm"] = capi.DeviceModel(st["m"])
        st["tables"] = capi.Tables(_table_arrays(w, "strains", 1, rng)[0])
        st["sections"], st["seed"] = _sections(st["m"].ndivision, case["section"]), seed
    elif case["kind"] == "mbp":
        n, st["sets"] = case["chains"], []
        for arr, t0, t1 in _mbp_inputs(case, seed):
            m = capi.Model(arr)
            dm = capi.DeviceModel(m)
            ch = capi.MbpChains(dm, n, form=form)
            ch.initialise([capi.Tables(t) for t in t0], seed, group_of=np.arange(n), stream_of=np.arange(n))
            st["sets"].append((m, dm, ch, dict(tables=[capi.Tables(t) for t in t1], seed=seed, group_of=np.arange(n),
                                               stream_of=np.arange(n) + n)))
    elif case["kind"] == "weights":
        st["args"] = _weights_inputs(case, seed)
    else:
        rng, st["requests"] = np.random.default_rng(seed), []
        for k, (A, G, days, spd, P, kind) in enumerate(_serve_sizes(case)):
            w = synth.seir_hd_small(seed=k, narea=A, nage=G, days=days, steps_per_day=spd)
            m = capi.Model(model_builder.model_arrays(w))
            tabs = [capi.Tables(t) for t in _table_arrays(w, "small", min(16, P), rng)]
            more = dict(group_of=np.arange(P) % len(tabs), form=capi.FORM_FAST, want_pop=kind != capi.REQ_LIKELIHOOD)
            if kind == capi.REQ_PREDICTION:     # continued from given populations
                p0 = np.rint(m.arr["pop_init"]).astype(np.int32).reshape(1, -1)
                more.update(ti=m.ndivision // 2, pop_in=np.repeat(p0, P, 0))
            st["requests"].append((m, capi.Batch(m, tabs, P, seed + k, **more), kind))
    return st


# ---- one pass -------------------------------------------------------------

def run(st):
    case = st["case"]
    if case["kind"] == "sim":
        b = st["batch"]
        if case["call"] == "simulate":
            st["dm"].simulate(b)
        else:
            st["db"].run_graph() if case["call"] == "graph" else st["db"].run()
        return {k: v for k, v in (("L", b.L), ("pop", b.pop), ("transnum", b.transnum), ("pop_traj", b.pop_traj))
                if v is not None}
    if case["kind"] == "pf":
        ll, terms, L, ancestors = st["dm"].pf_loglik(st["tables"], case["particles"], st["seed"], 5, 1.0, st["sections"],
                                                     form=FORMS[case["form"]])
        return {"loglik": ll, "terms": terms, "L": L, "ancestors": ancestors}
    if case["kind"] == "mbp":
        chains = [s[2] for s in st["sets"]]
        if case["form"] == "fast":
            out = {"L": capi.MbpChains.propose_fused(chains, [s[3] for s in st["sets"]])}
        else:
            q = st["sets"][0][3]
            out = {"L": [chains[0].propose(**q)],
                   "Li": chains[0].state_likelihood(q["tables"], group_of=q["group_of"])}
        everyone = np.ones(case["chains"], np.uint8)
        chains[0].accept(everyone)
        out["state"] = chains[0].read_state(0)
        chains[0].accept(everyone)              # back to the state that the next pass starts from
        return out
    if case["kind"] == "weights":
        tn, lp, tl, wl, ic = st["args"]
        return capi.abcsmc_weights(tn, lp, tl, wl, ic, 1.3)
    srv = capi.Server(100 << 30, 8)             # a stream of requests, start to end
    tickets = [srv.submit(*r) for r in st["requests"]]
    done = [srv.wait(t) for t in tickets]
    srv.close()
    return [(b.L, b.pop) if b.pop is not None else (b.L,) for b in done]


# ---- the work that a pass cannot do without --------------------------------

def _sim_work(A, G, S, P, sets, strains=1, traj=False, pop=False, obs=0):
    """Area and age mixing (two operations per pair), and per draw ten Philox rounds of
    eight operations and some twenty of the sampler; each table, observation and output once."""
    col = A * G * strains
    flops = float(P) * S * col * (2 * A + 2 * G + 100 * T)
    by = 8.0 * (sets * (T * G * strains + S) + S * (A / 4 + G * G + 2) + A * A + C * col) + 32.0 * obs + 8.0 * P
    by += 4.0 * P * col * (C * pop + S * (C + T) * traj)
    return flops, by


def work(case):
    if case["kind"] == "sim":
        strains = 2 if case["recipe"] == "strains" else 1
        S, A, G = case["days"] * case["spd"], case["areas"], case["ages"]
        obs = A * case["days"] * (G if case["recipe"] == "abc" else 8 / 7)
        f, b = _sim_work(A, G, S, case["particles"], case["sets"], strains, case["traj"], case["pop"], obs)
    elif case["kind"] == "pf":
        S, A = case["days"] * case["spd"], case["areas"]
        f, b = _sim_work(A, case["ages"], S, case["particles"], 1, obs=A * case["days"] * 8 / 7)
        b += 12.0 * case["particles"] * math.ceil(S / case["section"])
    elif case["kind"] == "mbp":
        f = b = 0.0
        S, n = case["days"] * case["spd"], case["chains"]
        wide = 8 if case["form"] == "fast" else 12
        for size in case["sizes"].split(","):
            A, G = map(int, size.split("x"))
            x, y = _sim_work(A, G, S, n, n, obs=A * case["days"] / 7)
            f, b = f + x, b + y + 2.0 * wide * n * S * T * A * G      # the current state read, the proposal written
    elif case["kind"] == "weights":
        nv = case["nvar"]
        f = float(case["new"]) * case["last"] * (3 * nv + 12)
        b = 8.0 * (case["new"] * (nv + 2) + case["last"] * (nv + 1))
    else:
        f = b = 0.0
        for A, G, days, spd, P, kind in _serve_sizes(case):
            S = days * spd // (2 if kind == capi.REQ_PREDICTION else 1)
            x, y = _sim_work(A, G, S, P, min(16, P), pop=kind != capi.REQ_LIKELIHOOD, obs=A * days * 8 / 7)
            f, b = f + x, b + y
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits ---------------------------------------------------

_M32 = 0xFFFFFFFF


def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 on int64 tensors holding 32-bit words."""
    k0, k1 = seed & _M32, (seed >> 32) & _M32

    def mul(a, x):                   # high and low words of a * x
        return ((a >> 16) * x + (((a & 0xFFFF) * x) >> 16)) >> 16, (a * x) & _M32
    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c0)
        h1, l1 = mul(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return c0, c1, c2, c3


def _u01(w):
    return w.double() * 2.0 ** -32 + 2.0 ** -33


def _poisson(mean, col, tr, sett, stream, seed):
    """Keyed Poisson draws: inversion below 10, Hoermann's PTRS from 10 on."""
    n = torch.zeros_like(mean)
    at = torch.nonzero((mean > 0) & (mean < 10), as_tuple=True)
    if at[0].numel():
        m, t = mean[at], tr[at]
        words = torch.stack(_philox(col[at], torch.full_like(t, sett), stream[at], t >> 2, seed))
        u = _u01(words.gather(0, (t & 3)[None])[0])
        p = torch.exp(-m)
        F, k = p.clone(), torch.zeros_like(m)
        for j in range(1, 80):
            k += u > F
            p = p * m / j
            F = F + p
        n[at] = k
    at = torch.nonzero(mean >= 10, as_tuple=True)
    m, t, cl, sm, it = mean[at], tr[at], col[at], stream[at], 0
    got = torch.full_like(m, -1.0)
    todo = torch.arange(m.numel(), device=m.device)
    while todo.numel():
        mm, tt = m[todo], t[todo]
        w = _philox(cl[todo], torch.full_like(tt, sett), sm[todo], (1 << 24) | (tt << 16) | it, seed)
        U, V = _u01(w[0]) - 0.5, _u01(w[1])
        b = 0.931 + 2.53 * mm.sqrt()
        a = -0.059 + 0.02483 * b
        us = 0.5 - U.abs()
        k = torch.floor((2.0 * a / us + b) * U + mm + 0.43)
        lhs = V.log() + (1.1239 + 1.1328 / (b - 3.4)).log() - (a / (us * us) + b).log()
        good = (lhs <= -mm + k * mm.log() - torch.lgamma(k + 1)) & (k >= 0) & ~((us < 0.013) & (V > us))
        good |= (us >= 0.07) & (V <= 0.9277 - 3.6224 / (b - 2.0))
        got[todo[good]] = k[good]
        todo, it = todo[~good], it + 1
    n[at] = got
    return n


class _Exact:
    """The tau-leap of a batch of particles and the log-likelihood of its observations in 64 bits."""

    def __init__(self, arr, tabs, group_of, seed):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        f = lambda x: torch.as_tensor(np.asarray(x, np.float64), device=dev)   # noqa: E731
        self.dev, self.seed = dev, seed
        d = [int(x) for x in arr["dims"]]
        self.A, self.G, self.DP, self.NS, self.C, self.T, self.S, _, self.spd = d
        self.P, self.DPS = len(group_of), self.DP // self.NS
        self.dt, self.popsize = float(arr["dt"][0]), float(arr["popsize"][0])
        M = np.zeros((self.A, self.A))
        ptr = arr["M_rowptr"]
        for c in range(self.A):
            M[c, arr["M_to"][ptr[c]:ptr[c + 1]]] = arr["M_val"][ptr[c]:ptr[c + 1]]
        self.M, self.diag, self.fac = f(M), f(arr["M_diag"]), f(arr["M_factor"])
        self.frm, self.to, self.itr = arr["trans_from"], arr["trans_to"], int(arr["infection_trans"][0])
        self.arr = arr
        self.pop = f(arr["pop_init"]).reshape(1, self.A, self.C, self.DP).repeat(self.P, 1, 1, 1)
        self.stream = torch.arange(self.P, device=dev)[:, None, None, None].expand(self.P, self.A, self.T, self.DP)
        col = torch.arange(self.A * self.DP, device=dev).reshape(1, self.A, 1, self.DP)
        self.col = col.expand(self.P, self.A, self.T, self.DP)
        self.tr = torch.arange(self.T, device=dev).reshape(1, 1, self.T, 1).expand(self.P, self.A, self.T, self.DP)
        self.set_tables(tabs, group_of)
        cells, cptr = arr["obs_cells"], arr["obs_cell_ptr"]
        oid = np.repeat(np.arange(len(arr["obs_sett_i"])), np.diff(cptr))
        self.at = []                    # per step: observation and cell of each active pair
        for s in range(self.S):
            k = np.flatnonzero((arr["obs_sett_i"][oid] <= s) & (s < arr["obs_sett_f"][oid]))
            self.at.append([torch.as_tensor(x, device=dev) for x in (oid[k], cells[k].astype(np.int64))])
        self.acc = torch.zeros(self.P, len(arr["obs_sett_i"]), dtype=torch.float64, device=dev)
        self.y, self.var = f(arr["obs_value"]), f(arr["obs_sd"]) ** 2

    def set_tables(self, tabs, group_of):
        f = lambda x: torch.as_tensor(np.asarray(x, np.float64), device=self.dev)   # noqa: E731
        g = torch.as_tensor(np.asarray(group_of), device=self.dev)
        self.rate = f(np.stack([t["transrate"] for t in tabs]))[g]                      # [P][T][DP]
        self.beta = f(np.stack([t["beta_rows"] for t in tabs]))[g]                      # [P][row][S]
        t = tabs[0]
        self.brow = torch.as_tensor(np.asarray(t["beta_row_of"]).reshape(self.NS, self.A).astype(np.int64), device=self.dev)
        self.sus, self.inf, self.af = f(t["susceptibility"]), f(t["infectivity"]), f(t["areafactor"])
        self.N, self.geo, self.efoi = f(t["Ntime"]), f(t["geo_spline"]), f(t["efoi_spline"])[0]

    def means(self, s):
        P, A, G, NS, DPS = self.P, self.A, self.G, self.NS, self.DPS
        src = int(self.frm[self.itr])
        I = torch.einsum("pacd,c->pad", self.pop, self.inf).reshape(P, A, NS, G)
        if NS > 1:                      # the susceptibles of all strains are in the first one's place
            S0 = self.pop[:, :, src].reshape(P, A, NS, DPS).sum(2)
            self.pop[:, :, src] = 0
            self.pop[:, :, src, :DPS] = S0
        Im = torch.einsum("pcsg,ct->ptsg", I, self.M)
        Id = I * self.diag[None, :, None, None]
        d = self.geo[s]
        X = (Id + Im) * d + self.fac[None, :, None, None] * Id * (1 - d)
        nmi = torch.einsum("pasg,hg->pash", X, self.N[s].reshape(G, G)).clamp(min=0)
        be = self.beta[:, :, s][:, self.brow].permute(0, 2, 1) * self.af[s // self.spd][None, :, None]     # [P][A][NS]
        lam = be[..., None] * nmi + self.efoi[s] / self.popsize
        pop = self.pop[:, :, src, :DPS].clamp(min=0)[:, :, None, :]
        m = self.dt * self.pop[:, :, [int(x) for x in self.frm]].clamp(min=0) * self.rate[:, None]
        m[:, :, self.itr] = (self.dt * pop * self.sus.reshape(NS, DPS) * lam).reshape(P, A, self.DP)
        return m

    def steps(self, ti, tf, each=None):
        P = self.P
        for s in range(ti, tf):
            m = self.means(s)
            n = _poisson(m, self.col, self.tr, s, self.stream, self.seed)
            if each is not None:
                each(s, m, n)
            oid, cell = self.at[s]
            flat = torch.cat([n.reshape(P, -1), self.pop.reshape(P, -1)], 1)
            where = torch.where(cell >= 0, cell, n[0].numel() - 1 - cell)
            self.acc.index_add_(1, oid, flat[:, where])
            for k in range(self.T):
                self.pop[:, :, int(self.frm[k])] -= n[:, :, k]
                self.pop[:, :, int(self.to[k])] += n[:, :, k]

    def loglik(self, ti, tf):
        on = torch.as_tensor((self.arr["obs_sett_i"] >= ti) & (self.arr["obs_sett_f"] <= tf), device=self.dev)
        lp = -0.5 * torch.log(2 * math.pi * self.var) - (self.y - self.acc.clamp(min=0)) ** 2 / (2 * self.var)
        return (lp * on).sum(1)


def _exact_pf(case, seed):
    w, arr = _epidemic("small", case["areas"], case["ages"], case["days"], case["spd"])
    tabs = _table_arrays(w, "strains", 1, np.random.default_rng(seed))
    N = case["particles"]
    e = _Exact(arr, tabs, np.zeros(N, np.int64), seed)
    terms, Ls = [], []
    for k, (ti, tf) in enumerate(_sections(e.S, case["section"])):
        e.acc.zero_()
        e.steps(ti, tf)
        L = e.loglik(ti, tf).cpu().numpy()
        wsum = np.cumsum(np.exp(L - L.max()))
        j = torch.arange(N)
        one = torch.ones_like(j)
        z = _u01(_philox(j, k * one, 5 * one, (3 << 24) * one, seed)[0]).numpy() * wsum[-1]
        place, extra = np.full(N, -1), []
        for p in np.searchsorted(wsum, z):      # a selected particle keeps its slot
            if place[p] < 0:
                place[p] = p
            else:
                extra.append(p)
        for p in range(N):
            if place[p] < 0:
                place[p] = extra.pop()
        e.pop = e.pop[torch.as_tensor(place, device=e.dev)]
        terms.append(L.max() + math.log(wsum[-1] / N))
        Ls.append(L)
    return {"loglik": float(sum(terms)), "terms": np.array(terms), "L": np.array(Ls), "ancestors": None}


def exact(case, seed):
    """What ``run`` returns, in 64 bits.  The fast form has no such value: its FP32 means send a
    particle to another trajectory wherever a variate falls on a near tie."""
    if case["kind"] == "weights":
        tn, lp, tl, wl, ic = _weights_inputs(case, seed)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        tn, lp, tl, wl, ic = (torch.as_tensor(x, device=dev) for x in (tn, lp, tl, wl, ic))
        sums = []
        for k in range(0, case["new"], 256):
            d = (tn[k:k + 256, None] - tl[None]) / 1.3
            sums.append(torch.logsumexp(wl.log() - 0.5 * torch.einsum("ijv,vw,ijw->ij", d, ic, d), 1))
        lw = lp - torch.cat(sums)
        w = torch.exp(lw - lw.max())
        return (w / w.mean()).cpu().numpy()
    if case.get("form") != "plain":
        return None
    if case["kind"] == "pf":
        return _exact_pf(case, seed)
    if case["kind"] == "mbp":                   # the likelihood of the current state; not the coupled proposal
        n = case["chains"]
        arr, t0, t1 = _mbp_inputs(case, seed)[0]
        e = _Exact(arr, t0, np.arange(n), seed)
        Li = torch.zeros(n, dtype=torch.float64, device=e.dev)

        def score(s, m, cnt):
            e.set_tables(t1, np.arange(n))
            m = e.means(s)
            e.set_tables(t0, np.arange(n))
            lp = torch.where(m > 0, cnt * m.clamp(min=1e-300).log() - m - torch.lgamma(cnt + 1), torch.zeros_like(m))
            Li.add_(lp.sum((1, 2, 3)))
        e.steps(0, e.S, score)
        return {"L": None, "Li": Li.cpu().numpy(), "state": None}
    if case["particles"] * case["areas"] * case["ages"] * case["days"] * case["spd"] > 2e7:
        return None
    arr, tabs, group_of = _sim_inputs(case, seed)
    e = _Exact(arr, tabs, group_of, seed)
    e.steps(0, e.S)
    return {"L": e.loglik(0, e.S).cpu().numpy(), "pop": None, "transnum": None, "pop_traj": None}
