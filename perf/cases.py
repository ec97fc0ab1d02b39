"""The work that a user of this package has it do, as measurable cases.

A case is one whole call through the public Python interface -- a
parallel-tempering run, an annealing run, a batch of runs, a set of served
requests -- from what the caller has in hand (instances, ladders, seeds) to the
results the caller reads back (final replicas and energies, ground-state log,
acceptance counts, thermal samples).  `listed()` names the cases, `draw()` gives
others of the same ranges.

Every output of a chain depends on its random stream: no closed form or 64-bit
computation gives the value a seed leads to, only the distribution it is drawn
from, so `exact()` has no value for any of them.  A run is a deterministic
function of its inputs and seed, whatever kernels it takes: states, counts and
logs of the same seed stay equal.
"""
import math

import numpy as np

import tamc_b200 as tb
from tamc_b200 import instances as gi

_GPU = None


def _gpu():
    """The device context that a program opens once."""
    global _GPU
    if _GPU is None:
        _GPU = tb.Gpu(0)
    return _GPU


def listed():
    return [
        # -- single parallel-tempering runs, colour-ordered
        # the smallest call: a quick look at a 64-site plaquette, where creation,
        # launches and read-backs count as much as the rounds
        dict(name="pt_2d_l8_short", kind="pt", graph="lattice2", size=8, couplings="pm", nt=16, chains=2, sweeps=100,
             threads=1, icm=True, sample=0, level=0, mode="fast"),
        # the 2-D Edwards-Anderson benchmark run: 32 temperatures, thermal samples
        # and packed states every 32 sweeps
        dict(name="pt_2d_l16", kind="pt", graph="lattice2", size=16, couplings="pm", nt=32, chains=2, sweeps=2000,
             threads=1, icm=True, sample=32, level=2, mode="fast"),
        # the 3-D Gaussian benchmark run (its sweep count shortened): 64
        # temperatures, two Fourier weights, samples of every temperature
        dict(name="pt_3d_l16_gauss", kind="pt", graph="lattice3", size=16, couplings="gauss", nt=64, chains=2,
             sweeps=1000, threads=64, icm=True, sample=32, level=0, mode="fast"),
        # a large cubic lattice of a side that is no power of two (13824 sites)
        dict(name="pt_3d_l24_gauss", kind="pt", graph="lattice3", size=24, couplings="gauss", nt=24, chains=2,
             sweeps=300, threads=8, icm=True, sample=50, level=1, mode="fast"),
        # a QUBO of an odd size on a ladder of an odd length: rows of uneven
        # length, self-couplings
        dict(name="pt_qubo_2039", kind="pt", graph="qubo", size=2039, couplings="int", nt=21, chains=2, sweeps=400,
             threads=8, icm=True, sample=0, level=0, mode="fast"),
        # -- the reference's chain bit for bit: replay of a seed, per-slot streams
        # (threads > 1) and the serial loop (threads: 1)
        dict(name="pt_ref_threads", kind="pt", graph="lattice2", size=16, couplings="pm", nt=32, chains=2, sweeps=50,
             threads=16, icm=True, sample=10, level=0, mode="ref"),
        dict(name="pt_ref_serial", kind="pt", graph="rrg", size=100, couplings="gauss", nt=12, chains=2, sweeps=40,
             threads=1, icm=True, sample=5, level=0, mode="ref"),
        # -- annealing: few restarts of a small QUBO, the benchmark's 1024
        # restarts of a 3-regular instance, and many restarts of the largest size
        dict(name="sa_qubo_251", kind="sa", graph="qubo", size=251, couplings="int", restarts=100, nbeta=200),
        dict(name="sa_rrg_2000", kind="sa", graph="rrg", size=2000, couplings="gauss", restarts=1024, nbeta=1000),
        dict(name="sa_qubo_8192", kind="sa", graph="qubo", size=8192, couplings="int", restarts=512, nbeta=100),
        # -- many runs at once: the benchmark's batch of uneven 2-D +-J instances,
        # from host instances to every run's ground-state log and acceptance counts
        dict(name="batch_2d_256", kind="batch", jobs=256, sides="8,12,16,24,32", ladders="16,24,32", sweeps=5000),
        # -- the solve server: QUBO requests of log-uniform size, waiting together
        dict(name="serve_qubo_24", kind="serve", requests=24, nmin=64, nmax=8192, sweeps=400, chunk=125),
    ]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["pt", "pt", "pt", "pt", "ref", "sa", "sa", "batch", "serve"])
    if kind == "pt":
        graph = rng.choice(["lattice2", "lattice2", "lattice3", "lattice3", "rrg", "qubo"])
        size = {"lattice2": rng.randint(4, 48), "lattice3": rng.randint(3, 24), "rrg": 2 * logint(10, 2000),
                "qubo": logint(16, 6000)}[graph]
        n = _sites(graph, size)
        nt = rng.randint(4, 64) if n < 8192 else rng.randint(4, 32)
        chains = rng.choice([2, 2, 2, 4])
        if n * nt * chains > 600000:
            chains = 2
        sweeps = min(logint(20, 2000), max(20, int(3e8 / (n * nt * chains))))
        return dict(kind="pt", graph=graph, size=size,
                    couplings="int" if graph == "qubo" else "gauss" if graph == "rrg" else rng.choice(["pm", "gauss"]),
                    nt=nt, chains=chains, sweeps=sweeps, threads=rng.choice([1, 8]), icm=rng.random() < 0.85,
                    sample=rng.choice([0, 0, 16, 32, 50]), level=rng.randint(0, 2), mode="fast")
    if kind == "ref":
        graph = rng.choice(["lattice2", "rrg", "qubo"])
        size = {"lattice2": rng.randint(4, 12), "rrg": 2 * rng.randint(8, 75), "qubo": rng.randint(16, 150)}[graph]
        nt = rng.randint(4, 20)
        return dict(kind="pt", graph=graph, size=size,
                    couplings="int" if graph == "qubo" else "gauss" if graph == "rrg" else "pm", nt=nt, chains=2,
                    sweeps=max(5, min(50, int(1e5 / (_sites(graph, size) * nt * 2)))), threads=rng.choice([1, 4]),
                    icm=True, sample=rng.choice([0, 5]), level=rng.randint(0, 2), mode="ref")
    if kind == "sa":
        graph = rng.choice(["rrg", "qubo", "lattice2", "lattice3"])
        size = {"lattice2": rng.randint(4, 64), "lattice3": rng.randint(3, 16), "rrg": 2 * logint(16, 2048),
                "qubo": logint(32, 8192)}[graph]
        restarts = logint(32, 2048)
        return dict(kind="sa", graph=graph, size=size,
                    couplings="int" if graph == "qubo" else "gauss", restarts=restarts,
                    nbeta=max(50, min(logint(50, 1000), int(1.5e9 / (_sites(graph, size) * restarts)))))
    if kind == "batch":
        jobs = logint(4, 256)
        lo = rng.randint(0, 2)
        return dict(kind="batch", jobs=jobs, sides=",".join(str(x) for x in (8, 10, 12, 16, 20, 24, 32)[lo:lo + 5]),
                    ladders=rng.choice(["16,24,32", "8,13", "32", "20,40"]), sweeps=logint(100, 2000))
    return dict(kind="serve", requests=logint(2, 32), nmin=rng.choice([16, 64]), nmax=logint(256, 8192),
                sweeps=logint(50, 400), chunk=rng.choice([50, 100, 125]))


# ------------------------------------------------------------ inputs ----
def _sites(graph, size):
    return size ** 2 if graph == "lattice2" else size ** 3 if graph == "lattice3" else size


def _degree(graph):
    return {"lattice2": 4, "lattice3": 6, "rrg": 3, "qubo": 7}[graph]


def _instance(graph, size, couplings, seed):
    if graph == "lattice2":
        return tb.HostInstance.parse(gi.lattice(size, 2, couplings, seed))
    if graph == "lattice3":
        return tb.HostInstance.parse(gi.lattice(size, 3, couplings, seed))
    if graph == "rrg":
        return tb.HostInstance.parse(gi.sa_regular(size, 3, seed))
    return tb.HostInstance.parse(gi.qubo_er(size, 6.0, seed), qubo=True)


def _params(nt, sweeps, chains=2, threads=8, icm=True, sample=None, level=0):
    """The benchmark's ladder: geometric 0.2 -> 5.0, Houdayer moves from beta 1.0, half the run as warm-up."""
    b = tb.geometric_betas(0.2, 5.0, nt)
    lo = int(np.argmax(b >= np.float32(1.0)))
    return tb.PtParams(sweeps, b, lo, 0.5, icm, chains, threads, sample, sample, level)


def _batch_jobs(case):
    """(side, temperatures) of a batch's runs: the same shapes for every seed."""
    r = np.random.default_rng(0)
    sides = [int(x) for x in case["sides"].split(",")]
    ladders = [int(x) for x in case["ladders"].split(",")]
    return [(int(r.choice(sides)), int(r.choice(ladders))) for _ in range(case["jobs"])]


def _requests(case):
    """(sites, temperatures) of the served requests, the same for every seed."""
    r = np.random.default_rng(1)
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    return [(int(round(math.exp(r.uniform(lo, hi)))), int(r.integers(16, 33))) for _ in range(case["requests"])]


def prepare(case, seed):
    gpu, kind = _gpu(), case["kind"]
    if kind == "pt":
        host = _instance(case["graph"], case["size"], case["couplings"], seed)
        if case["graph"] == "lattice3" and case["sample"]:
            for axis in (0, 1):
                host.add_suscept(gi.fourier_weights(case["size"], 3, axis))
        p = _params(case["nt"], case["sweeps"], case["chains"], case["threads"], case["icm"], case["sample"] or None,
                    case["level"])
        return dict(kind=kind, inst=gpu.upload(host), params=p, seed=seed + 17,
                    mode=tb.MODE_REF if case["mode"] == "ref" else tb.MODE_FAST)
    if kind == "sa":
        host = _instance(case["graph"], case["size"], case["couplings"], seed)
        return dict(kind=kind, inst=gpu.upload(host), betas=np.linspace(0.1, 10.0, case["nbeta"]).astype(np.float32),
                    restarts=case["restarts"], seed=seed + 17)
    if kind == "batch":
        jobs = _batch_jobs(case)
        return dict(kind=kind, hosts=[_instance("lattice2", L, "pm", seed + k) for k, (L, _) in enumerate(jobs)],
                    params=[_params(nt, case["sweeps"]) for _, nt in jobs],
                    seeds=[seed + 7 + k for k in range(len(jobs))])
    reqs = _requests(case)
    return dict(kind=kind, hosts=[_instance("qubo", n, "int", seed + k) for k, (n, _) in enumerate(reqs)],
                params=[_params(nt, case["sweeps"]) for _, nt in reqs], chunk=case["chunk"],
                seeds=[seed + 7 + k for k in range(len(reqs))])


# ------------------------------------------------------------ one pass ----
def run(state):
    return {"pt": _run_pt, "sa": _run_sa, "batch": _run_batch, "serve": _run_serve}[state["kind"]](state)


def _table(a, rows):
    """A log, whose length depends on the chain, in a table of `rows` rows (zeros after its end)."""
    out = np.zeros((rows,) + a.shape[1:], a.dtype)
    out[:len(a)] = a
    return out


def _run_pt(s):
    p = s["params"]
    r = tb.PtRun(s["inst"], p, s["seed"], s["mode"]).run().sync()
    rows = p.num_sweeps - p.meas_init  # at most one new minimum per tracked sweep
    steps, energies, states = (_table(x, rows) for x in r.gs())
    spins, final = r.state()
    out = dict(gs_steps=steps, gs_energies=energies, gs_states=states, acceptance=r.acceptance(), spins=spins,
               final=final)
    if p.sample is not None:
        t = r.samples()
        out.update(e=np.array(t.e), q=np.array(t.q), samples=np.array(t.samples))
        if len(t.suscept[0]):
            out["suscept"] = np.array(t.suscept)
    return out


def _run_sa(s):
    energies, packed = tb.sa_run(s["inst"], s["betas"], s["restarts"], 1, s["seed"])
    return dict(energies=energies, packed=packed)


def _run_batch(s):
    gpu = _gpu()
    b = tb.Batch(gpu)
    for d, p, seed in zip(gpu.upload_many(s["hosts"]), s["params"], s["seeds"]):
        b.add(d, p, seed)
    b.run()
    logs, acceptance = b.gs_all(), b.acceptance_all()
    rows = 64 * len(logs)  # a +-J run's tracked minima are a few dozen energy levels at most
    return dict(gs_steps=_table(np.concatenate([x[0] for x in logs]), rows),
                gs_energies=_table(np.concatenate([x[1] for x in logs]), rows),
                gs_states=_table(np.concatenate([x[2].ravel() for x in logs]), 16 * rows),
                acceptance=np.concatenate(acceptance))


def _run_serve(s):
    srv = tb.Server(_gpu(), hbm_budget_bytes=64 << 30, max_active=512, chunk_sweeps=s["chunk"])
    ids = [srv.submit(h, p, seed) for h, p, seed in zip(s["hosts"], s["params"], s["seeds"])]
    while True:
        active, queued = srv.step()
        if not active and not queued:
            break
    best = np.array([srv.result(i)[1] for i in ids], np.float32)
    states = [srv.state(i) for i in ids]
    return dict(best=best, spins=np.concatenate([x.ravel() for x, _ in states]),
                final=np.concatenate([e.ravel() for _, e in states]))


# ------------------------------------------------------------ bounds ----
def _run_work(n, deg, nt, chains, sweeps, sample=0, level=0, nchi=0):
    """Bytes (instance in, replicas and samples out, bit-packed) and operations
    (per flip attempt: the local field's deg multiply-adds, the field, the
    energy change, the exponent and the comparison) of one run."""
    r = nt * chains
    rec = (sweeps // 2) // sample + 1 if sample else 0
    z = nt if level == 0 else nt // 2 if level == 1 else 1
    nbytes = n * (8 + 8 * deg) + r * n / 8 + r * 4 + rec * (r * 4 + nt * (chains // 2) * 4 * (1 + nchi)
                                                          + z * chains * n / 8)
    return nbytes, float(n) * r * sweeps * (2 * deg + 4)


def work(case):
    kind = case["kind"]
    if kind == "pt":
        nchi = 2 if case["graph"] == "lattice3" and case["sample"] else 0
        b, f = _run_work(_sites(case["graph"], case["size"]), _degree(case["graph"]), case["nt"], case["chains"],
                         case["sweeps"], case["sample"], case["level"], nchi)
    elif kind == "sa":
        n, d = _sites(case["graph"], case["size"]), _degree(case["graph"])
        b = n * (8 + 8 * d) + case["restarts"] * (n / 8 + 4) + 4 * case["nbeta"]
        f = float(n) * case["restarts"] * case["nbeta"] * (2 * d + 4)
    else:
        runs = _batch_jobs(case) if kind == "batch" else _requests(case)
        each = [_run_work(x * x if kind == "batch" else x, 4 if kind == "batch" else 7, nt, 2, case["sweeps"])
                for x, nt in runs]
        b, f = sum(x for x, _ in each), sum(x for _, x in each)
    return dict(bytes=b, flops=f)


def exact(case, seed):
    """No output of a Markov chain has a value in 64 bits (see the module's text)."""
    return None
