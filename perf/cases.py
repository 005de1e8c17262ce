"""Performance cases of the vacancy-hop engine, through its public Python binding.

A case is a dict of plain values; `kind` names the call a user's program makes:

  hop       one hop through the per-hop boundary (calculate, then select_and_perform), the way the
            reference's own time loop drives its backend: host in charge of sectors, draws and clock;
  rates     a new lattice into a resident job, then every vacancy's 8 energy changes and rates, sector
            by sector (energetics and precision reports are made of these calls);
  run       sector rounds of one job on the device, then its lattice and sector clocks read back;
            with `load`, a new lattice comes from pinned host memory before each pass;
  replicas  the same for many independent boxes of uneven size in one context;
  clusters  the Cu cluster statistics of a resident lattice, sampled during a run;
  serve     a burst of jobs through the job server, from submission to the last result.

Lattices, draws and job streams come from the seed given to prepare(); the potential is the
synthetic EAM of the repository's workloads, or the reference's pair-bond model.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "misa-akmc-gpu_b200", "python")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import akmc_b200 as ak  # noqa: E402

POT_SEED = 42
WINDOW_S = 3.0e-7
NU = 6.0e12
KB = 8.617330350e-5
E0 = {ak.FE: 0.62, ak.CU: 0.54, ak.NI: 0.68, ak.MN: 1.03}


def listed():
    return [
        # the drop-in boundary at its usual size: one domain of 20^3 cells, one hop per pass.  The
        # smallest call: latency and launches are all there is
        dict(name="hop_20_pairbond", kind="hop", nx=20, ny=20, nz=20, model="pairbond", vacancies=20, temperature=573.0,
             cu=134, ni=0, mn=0),
        # energetics of a sampled state: a 20^3 window uploaded, all of its vacancies evaluated
        dict(name="rates_20_fp32c", kind="rates", nx=20, ny=20, nz=20, model="fp32c", vacancies=20, temperature=563.0,
             cu=134, ni=70, mn=30),
        # the plain serial box: 20^3 cells, 20 vacancies, single domain, FP64
        dict(name="serial_20_fp64", kind="run", nx=20, ny=20, nz=20, block=32, model="fp64", vacancies=20,
             temperature=573.0, cu=134, ni=0, mn=0, rounds=256, load=False),
        # the reference's energy model on a box with odd edges and uneven domain blocks
        dict(name="ragged_97_pairbond", kind="run", nx=97, ny=83, nz=71, block=16, model="pairbond", vacancies=114,
             temperature=563.0, cu=134, ni=70, mn=30, rounds=512, load=False),
        # the serial box's vacancy concentration over several domain blocks: more than 32 vacancies
        # to a block, so the rounds run block-synchronously
        dict(name="dense_48_fp64", kind="run", nx=48, ny=48, nz=48, block=24, model="fp64", vacancies=276,
             temperature=573.0, cu=134, ni=70, mn=30, rounds=256, load=False),
        # a sweep over starting lattices: each pass uploads one, runs one sublattice time step, reads it back
        dict(name="restart_150_fp64", kind="run", nx=150, ny=131, nz=117, block=16, model="fp64", vacancies=92,
             temperature=563.0, cu=134, ni=70, mn=30, rounds=8, load=True),
        # an ensemble of 64 small boxes in double precision
        dict(name="replicas_64_fp64", kind="replicas", boxes=64, lo=16, hi=48, block=24, model="fp64", fraction=1e-4,
             rounds=256, load=False),
        # 512 boxes of 16^3 to 48^3 cells, FP32-compensated, lattices up and down on every pass
        dict(name="replicas_512_fp32c", kind="replicas", boxes=512, lo=16, hi=48, block=20, model="fp32c", fraction=1e-4,
             rounds=256, load=True),
        # the large lattice in double precision, end to end: upload, 1024 rounds, read-back
        dict(name="scale_256_fp64", kind="run", nx=256, ny=256, nz=256, block=16, model="fp64", vacancies=671,
             temperature=563.0, cu=134, ni=70, mn=30, rounds=1024, load=True),
        # the same lattice resident, FP32-compensated, sampled every 256 rounds
        dict(name="scale_256_fp32c", kind="run", nx=256, ny=256, nz=256, block=16, model="fp32c", vacancies=671,
             temperature=563.0, cu=134, ni=70, mn=30, rounds=256, load=False),
        # cluster statistics of the large lattice
        dict(name="clusters_256", kind="clusters", nx=256, ny=256, nz=256, vacancies=671, cu=134, ni=70, mn=30),
        # a burst of jobs on the server, the serving workload's sizes and the low end of its budgets
        dict(name="serve_96_fp32c", kind="serve", jobs=96, lo=16, hi=96, budget_lo=10000, budget_hi=100000, model="fp32c"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _edges(rng, lo, hi):
    e = _log(rng, lo, hi)
    return [max(int(lo), min(int(hi), int(round(e * rng.uniform(0.8, 1.25))))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["hop", "rates", "run", "run", "run", "run", "replicas", "replicas", "clusters", "serve"])
    c = dict(kind=kind)
    if kind in ("hop", "rates"):
        c["nx"], c["ny"], c["nz"] = _edges(rng, 16, 26)
        c["model"] = rng.choice(["pairbond", "fp64", "fp32c"]) if kind == "hop" else rng.choice(["fp64", "fp32c"])
        c["vacancies"] = int(round(_log(rng, 4, 60)))
    elif kind == "run":
        c["block"] = rng.choice([12, 16, 16, 20, 24])
        c["model"] = rng.choice(["pairbond", "fp64", "fp32c"])
        c["nx"], c["ny"], c["nz"] = _edges(rng, 16, 240)
        sites = 2 * c["nx"] * c["ny"] * c["nz"]
        c["vacancies"] = max(2, int(round(sites * min(_log(rng, 2e-5, 1.5e-3), 671.0 / sites if sites > 1 << 20 else 1.0))))
        c["load"] = rng.random() < 0.5
        c["rounds"] = 8 * max(1, int(min(_log(rng, 1, 128), 671 * 128 / c["vacancies"])))
    elif kind == "replicas":
        c["boxes"] = int(round(_log(rng, 8, 512)))
        c["lo"], c["hi"] = 16, rng.choice([24, 32, 48])
        c["block"] = rng.choice([16, 20, 24])
        c["model"] = rng.choice(["fp64", "fp32c", "fp32c"])
        c["fraction"] = round(_log(rng, 1e-4, 4e-4), 6)
        c["load"] = rng.random() < 0.5
        c["rounds"] = 8 * int(round(_log(rng, 4, 32)))
    elif kind == "clusters":
        c["nx"], c["ny"], c["nz"] = _edges(rng, 24, 240)
        c["vacancies"] = 4
    else:
        c["jobs"] = int(round(_log(rng, 8, 96)))
        c["lo"], c["hi"] = 16, rng.choice([32, 64, 96])
        c["budget_lo"], c["budget_hi"] = 10000, rng.choice([20000, 50000, 100000])
        c["model"] = rng.choice(["fp64", "fp32c"])
    if "nx" in c:
        c["cu"], c["ni"], c["mn"] = rng.randint(50, 150), rng.randint(0, 100), rng.randint(0, 50)
        if kind != "clusters":
            c["temperature"] = float(rng.randint(473, 673))
    return c


# --- inputs ---------------------------------------------------------------------------------
def _blocks(edge, block):
    """Domain blocks along an edge: blocks of at most `block` cells, none below 8."""
    return max(1, min(-(-edge // block), edge // 8))


def _alloy(cu, ni, mn):
    return ((ak.FE, 10000 - cu - ni - mn), (ak.CU, cu), (ak.NI, ni), (ak.MN, mn))


def _config(box, blocks, model, temperature, seed, eam, hop_budget=0):
    pair = model == "pairbond"
    return ak.job_config(box, blocks=blocks, energy_model=ak.MODEL_PAIRBOND if pair else ak.MODEL_EAM,
                         precision=ak.FP32C if model == "fp32c" else ak.FP64, temperature=temperature, seed=seed,
                         window=WINDOW_S, hop_budget=hop_budget, eam=None if pair else eam)


def _box(case):
    return (case["nx"], case["ny"], case["nz"])


def _lattice(case, seed):
    return ak.create_lattice(_box(case), _alloy(case["cu"], case["ni"], case["mn"]), case["vacancies"], seed)


def _many(case, seed):
    """The boxes of an ensemble or the jobs of a burst: edge, composition and temperature drawn per
    job as the batched and serving workloads draw them.  The sizes are the case's, the rest the seed's."""
    n = case["boxes"] if case["kind"] == "replicas" else case["jobs"]
    sizes = random.Random("%s %d %d %d" % (case["kind"], n, case["lo"], case["hi"]))
    rng = random.Random("%d %s" % (seed, case["kind"]))
    jobs = []
    for i in range(n):
        edge = int(round(_log(sizes, case["lo"], case["hi"])))
        j = dict(edge=edge, cu=rng.randint(50, 150), ni=rng.randint(0, 100), mn=rng.randint(0, 50),
                 temperature=rng.uniform(473.0, 673.0), seed=seed * 1000 + i)
        if case["kind"] == "serve":
            j["vacancies"] = max(2, int(round(1e-4 * 2 * edge ** 3)))
            j["budget"] = int(round(_log(rng, case["budget_lo"], case["budget_hi"])))
        else:
            j["vacancies"] = max(1, int(round(case["fraction"] * 2 * edge ** 3)))
        jobs.append(j)
    return jobs


def _pinned(a):
    return torch.from_numpy(a).pin_memory().numpy()


class _State:
    """What a program keeps: the context or server, pinned buffers, its own counters and draws."""

    def __init__(self, case):
        self.case = case
        self.passes = 0
        self.engine = None
        self.server = None

    def __del__(self):
        for h in (self.engine, self.server):
            try:
                if h is not None:
                    h.close()
            except Exception:
                pass


def prepare(case, seed):
    s = _State(case)
    kind = case["kind"]
    eam = ak.eam_johnson(POT_SEED)
    if kind == "serve":
        s.jobs = []
        for j in _many(case, seed):
            box, nb = (j["edge"],) * 3, (-(-j["edge"] // 24),) * 3
            occ = ak.create_lattice(box, _alloy(j["cu"], j["ni"], j["mn"]), j["vacancies"], j["seed"])
            s.jobs.append((_config(box, nb, case["model"], j["temperature"], j["seed"], eam, j["budget"]), occ))
        s.server = ak.Server()
        return s
    s.engine = ak.Engine()
    if kind == "replicas":
        lattices = []
        for j in _many(case, seed):
            box = (j["edge"],) * 3
            occ = ak.create_lattice(box, _alloy(j["cu"], j["ni"], j["mn"]), j["vacancies"], j["seed"])
            s.engine.add_job(_config(box, (_blocks(j["edge"], case["block"]),) * 3, case["model"], j["temperature"],
                                     j["seed"], eam), occ)
            lattices.append(occ)
        whole = np.concatenate(lattices)
        s.out = _pinned(np.empty_like(whole))
        s.lattice = _pinned(whole) if case["load"] else None
    else:
        occ = _lattice(case, seed)
        blocks = tuple(_blocks(e, case["block"]) for e in _box(case)) if kind == "run" else (
            tuple(_blocks(e, 16) for e in _box(case)) if kind == "clusters" else (1, 1, 1))
        s.engine.add_job(_config(_box(case), blocks, case.get("model", "pairbond"), case.get("temperature", 563.0), seed, eam),
                         occ)
        s.lattice = _pinned(occ) if kind == "rates" or case.get("load") else None
        if kind == "run":
            s.out = _pinned(np.empty_like(occ))
        elif kind == "hop":
            s.draws = np.random.default_rng(seed).random(4096).tolist()
    s.engine.prepare()
    return s


# --- one pass -------------------------------------------------------------------------------
def _run_hop(s):
    e = s.engine
    sector = ak.SECTOR_ORDER[s.passes % 8]
    u = s.draws[s.passes % len(s.draws)]
    s.passes += 1
    total = e.calculate(0, sector)
    event = np.full(5, -1, np.int64)
    if total > 0.0:
        ev = e.select_and_perform(0, sector, u)
        event[:] = (ev.from_site, ev.to_site, ev.species, ev.n_act, ev.n_dirty)
    return dict(total=total, event=event)


def _run_rates(s):
    e = s.engine
    e.load_occupancy(0, s.lattice)
    totals, sites, de, rates = np.zeros(8), [], [], []
    for k in range(8):
        totals[k] = e.calculate(0, k)
        a, b, c = e.calculated_rates()
        sites.append(a)
        de.append(b)
        rates.append(c)
    sites = np.concatenate(sites)
    by_site = np.argsort(sites)
    return dict(totals=totals, sites=sites[by_site], de=np.concatenate(de)[by_site], rates=np.concatenate(rates)[by_site])


def _run_rounds(s):
    e = s.engine
    if s.lattice is not None:
        e.load_occupancy(0, s.lattice)
    e.run_rounds(s.case["rounds"])
    lattice = e.occupancy(0, out=s.out)
    clocks, hops = e.block_clocks(0)
    return dict(lattice=lattice, clocks=clocks, hops=hops)


def _run_replicas(s):
    e = s.engine
    if s.lattice is not None:
        e.load_occupancies(s.lattice)
    e.run_rounds(s.case["rounds"])
    lattices = e.occupancies(out=s.out)
    states = e.job_states()
    return dict(lattices=lattices, hops=np.array([j["hops"] for j in states]), rounds=np.array([j["round"] for j in states]))


def _run_clusters(s):
    isolated, hist = s.engine.cluster_stats(0)
    return dict(isolated=isolated, hist=hist)


def _run_serve(s):
    tickets = [s.server.submit(cfg, occ) for cfg, occ in s.jobs]
    done = [s.server.wait(t, timeout=120.0) for t in tickets]
    for r, _ in done:
        if r["status"] != 0:
            raise RuntimeError("job failed: %s" % r["error"])
    return dict(lattices=np.concatenate([o for _, o in done]),
                hops=np.array([r["hops"] for r, _ in done]), rounds=np.array([r["rounds"] for r, _ in done]),
                clocks=np.array([r["clocks_fnv"] for r, _ in done], np.uint64).view(np.int64))


_RUN = dict(hop=_run_hop, rates=_run_rates, run=_run_rounds, replicas=_run_replicas, clusters=_run_clusters,
            serve=_run_serve)


def run(state):
    return _RUN[state.case["kind"]](state)


# --- what a pass cannot do without ----------------------------------------------------------
# A vacancy evaluation reads its footprint (EAM: 145 occupancy bytes and int32 densities; pair bond:
# 113 bytes) and writes 8 rates; a hop refreshes 78 densities, swaps two sites, writes its event and
# reads the rates it selects from.  EAM evaluation: 8 jumps x 77 sites x two cubics and the pair term.
def _eval_bytes(model):
    return 113 + 64 if model == "pairbond" else 145 * 5 + 64


def _hop_work(model):
    eam = model != "pairbond"
    return _eval_bytes(model) + (78 * 8 if eam else 0) + 2 + 16 + 64, (8 * 77 * 17 if eam else 8 * 2 * 26) + 200


def _hops(vacancies, rounds, temperature, block):
    """Hops of `rounds` sector rounds: a vacancy is in the active sector one round in eight, and hops
    there until its clock passes the window or it walks out of the sector."""
    per_window = 8.0 * NU * math.exp(-0.62 / (KB * temperature)) * WINDOW_S
    return vacancies * rounds / 8.0 * min(per_window, (block / 2.0) ** 2 / 6.5)


def work(case):
    kind = case["kind"]
    model = case.get("model", "pairbond")
    hb, hf = _hop_work(model)
    if kind == "hop":
        return dict(bytes=hb, flops=hf)
    if kind == "clusters":
        return dict(bytes=2 * case["nx"] * case["ny"] * case["nz"], flops=0)
    if kind == "rates":
        sites = 2 * case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=sites * 6 + case["vacancies"] * _eval_bytes(model), flops=sites * 58 + case["vacancies"] * hf)
    if kind == "run":
        sites = 2 * case["nx"] * case["ny"] * case["nz"]
        hops = _hops(case["vacancies"], case["rounds"], case["temperature"], min(case["block"], case["nx"]))
    else:
        jobs = _many(case, 1)
        sites = sum(2 * j["edge"] ** 3 for j in jobs)
        hops = sum(j["budget"] for j in jobs) if kind == "serve" else sum(
            _hops(j["vacancies"], case["rounds"], j["temperature"], min(case["block"], j["edge"])) for j in jobs)
    # the lattice is read back once (1 B a site); a new one is read, and its densities written
    load = kind == "serve" or case.get("load")
    per_site = 1 + (0 if not load else 1 if model == "pairbond" else 6)
    flops = hops * hf + (sites * 58 if load and model != "pairbond" else 0)
    return dict(bytes=hops * hb + sites * per_site, flops=flops)


# --- 64-bit values of the computed numbers --------------------------------------------------
_SHELL_D2 = (3, 4, 8, 11, 12)


def _energetics(case, seed):
    """{site: (dE[8], rates[8])} of every vacancy of the case's EAM lattice, and each one's sector,
    with plain numpy in double precision: dE = [F(rho_s - f_X) - F(rho_t)] + sum over the atoms j in
    the cutoff of s or t of [F(rho_j + f_X(sj) - f_X(tj)) - F(rho_j)] + phi_XY(sj) - phi_XY(tj),
    densities on the tables' 2^-24 grid, F by Catmull-Rom on its table."""
    nx, ny, nz = _box(case)
    occ = _lattice(case, seed).reshape(nz, ny, 2 * nx)
    t = ak.eam_johnson(POT_SEED)
    f = np.zeros((4, 7))
    f[:, 1:6] = np.round(np.array(t.f_shell) * 2.0 ** 24) / 2.0 ** 24
    phi = np.zeros((4, 4, 7))
    phi[:, :, 1:6] = np.array(t.phi_shell)
    table = np.array(t.F)
    species = {ak.FE: 0, ak.CU: 1, ak.NI: 2, ak.MN: 3}

    def F(rho):
        x = rho * 128.0
        k = int(math.floor(x))
        p = x - k
        m0, m1 = 0.5 * (table[k + 1] - table[k - 1]), 0.5 * (table[k + 2] - table[k])
        c2 = 3.0 * (table[k + 1] - table[k]) - 2.0 * m0 - m1
        c3 = 2.0 * (table[k] - table[k + 1]) + m0 + m1
        return table[k] + p * (m0 + p * (c2 + p * c3))

    def half(X, y, z):  # position in half lattice constants
        return X, 2 * y + (X & 1), 2 * z + (X & 1)

    def site(h):  # the site at a position, wrapped into the box
        X = h[0] % (2 * nx)
        return X, ((h[1] - (X & 1)) // 2) % ny, ((h[2] - (X & 1)) // 2) % nz

    near = [(a, b, c) for a in range(-4, 5) for b in range(-4, 5) for c in range(-4, 5)
            if a % 2 == b % 2 == c % 2 and a * a + b * b + c * c in _SHELL_D2]

    def shell(a, b):
        d2 = sum((p - q) ** 2 for p, q in zip(a, b))
        return _SHELL_D2.index(d2) + 1 if d2 in _SHELL_D2 else 0

    def code(h):
        X, y, z = site(h)
        return int(occ[z, y, X])

    memo = {}

    def rho(h):
        key = site(h)
        if key not in memo:
            r = 0.0
            for d in near:
                o = code((h[0] + d[0], h[1] + d[1], h[2] + d[2]))
                if o:
                    r += f[species[o], shell(d, (0, 0, 0))]
            memo[key] = r
        return memo[key]

    # first neighbours in the order (dx, dy, dz) of the site ids' own offsets
    jumps = [(dx, dy, dz) for dx in (-1, 1) for dy in (-1, 1) for dz in (-1, 1)]
    out = {}
    for z, y, X in zip(*np.nonzero(occ == ak.V)):
        s = half(int(X), int(y), int(z))
        de, rates = np.zeros(8), np.zeros(8)
        for b, d in enumerate(jumps):
            tt = (s[0] + d[0], s[1] + d[1], s[2] + d[2])
            o = code(tt)
            if not o:
                continue
            q = species[o]
            e = F(rho(s) - f[q, 1]) - F(rho(tt))
            around = {(s[0] + n[0], s[1] + n[1], s[2] + n[2]) for n in near}
            around |= {(tt[0] + n[0], tt[1] + n[1], tt[2] + n[2]) for n in near}
            for j in around - {s, tt}:
                oj = code(j)
                if not oj:
                    continue
                hs, ht = shell(j, s), shell(j, tt)
                r = rho(j)
                e += F(r + f[q, hs] - f[q, ht]) - F(r) + phi[q, species[oj], hs] - phi[q, species[oj], ht]
            de[b] = e
            rates[b] = NU * math.exp(-(E0[o] + e / 2.0) / (KB * case["temperature"]))
        n3 = (nx, ny, nz)
        c3 = (int(X) >> 1, int(y), int(z))
        sector = sum((1 << d) for d in range(3) if c3[d] >= n3[d] // 2)
        out[int(X) + 2 * nx * (int(y) + ny * int(z))] = (sector, de, rates)
    return out


def exact(case, seed):
    """The energy changes, rates and totals in 64 bits.  Trajectories (clocks of thousands of dependent
    hops) have no value here that plain numpy reaches in the time."""
    if case["kind"] not in ("hop", "rates") or case["model"] == "pairbond":
        return None
    v = _energetics(case, seed)
    totals = np.zeros(8)
    for k in sorted(v):
        totals[v[k][0]] += v[k][2].sum()
    if case["kind"] == "hop":
        return dict(total=float(totals[ak.SECTOR_ORDER[0]]), event=None)
    return dict(totals=totals, sites=None, de=np.stack([v[k][1] for k in sorted(v)]),
                rates=np.stack([v[k][2] for k in sorted(v)]))
