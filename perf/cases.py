"""Timing cases: what a user of the engine runs, through its public entry points.

A case is one call of a program that searches: a whole tabu search of a given
budget on a graph it has loaded (``tabu_search`` / a kept ``Solver``), a batch
of restarts replayed, a burst of requests to the server, building a lookup
structure and querying it, or one decision through the entry point that
allocates nothing.  Sizes, degrees, tenures and the six lookup structures are
those of the five benchmark workloads and of the reference's data sets
(ER n = 2,000; conflict-style bisection graph n = 100,000; Chung-Lu
n = 200,000; mixed batches and request streams; dense ``MDG`` instances), with
odd sizes between them.  Every output is an integer: searches are
deterministic, so results and final states repeat exactly.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "graph-data-structures-local-search_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ts_b200 as T  # noqa: E402

DEV = "cuda"
STRUCTS = ("csr", "hash", "wswap", "csr-bitset", "csr-bb", "csr-bitset-bb")


# ------------------------------------------------------------------ graphs
# The generators of ts_b200.gen, drawn on the GPU so that a prepared case takes
# milliseconds: the same families, degrees and weights.
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _finish(n, a, b, gen, wmul):
    keep = a != b
    a, b = a[keep], b[keep]
    key = torch.unique(torch.minimum(a, b) * n + torch.maximum(a, b))
    u, v = key // n, key % n
    nw = torch.randint(1, 1001, (n,), generator=gen, device=DEV) * wmul
    return u.to(torch.int32), v.to(torch.int32), (nw[u] + nw[v]).to(torch.int32)


def _erdos_renyi(n, degree, gen, wmul=1):
    e = max(1, int(n * degree / 2))
    a = torch.randint(0, n, (e,), generator=gen, device=DEV)
    b = torch.randint(0, n, (e,), generator=gen, device=DEV)
    return _finish(n, a, b, gen, wmul)


def _complete(n, gen):
    """Dense instance: every pair, weights 0.00-10.00 as exact hundredths (MDG-a)."""
    k = torch.triu_indices(n, n, 1, device=DEV)
    w = torch.randint(0, 1001, (k.shape[1],), generator=gen, device=DEV)
    return k[0].to(torch.int32), k[1].to(torch.int32), w.to(torch.int32)


def _chung_lu(n, mean_degree, max_degree, gen, wmul=1):
    d = (torch.arange(n, dtype=torch.float64, device=DEV) + 1.0) ** (-1.0 / 1.3)
    for _ in range(30):
        d = torch.clamp(d * (mean_degree / d.mean()), max=float(max_degree))
    cum = torch.cumsum(d, 0)
    perm = torch.randperm(n, generator=gen, device=DEV)
    e = int(n * mean_degree / 2 * 1.03) + 1000
    ends = [perm[torch.searchsorted(cum, torch.rand(e, generator=gen, device=DEV, dtype=torch.float64) * cum[-1])
                 .clamp_(max=n - 1)] for _ in range(2)]
    return _finish(n, ends[0], ends[1], gen, wmul)


def _conflict(n, degree, gen, wmul=1):
    """Unit-square points joined within a radius, plus n/50 cliques of 8-32 vertices."""
    x = torch.rand((n, 2), generator=gen, device=DEV, dtype=torch.float64)
    r = math.sqrt(degree / (math.pi * (n - 1)))
    g = max(1, int(1.0 / r))
    cell = (x * g).long().clamp_(max=g - 1)
    cid = cell[:, 0] * g + cell[:, 1]
    order = torch.argsort(cid, stable=True)
    bounds = torch.searchsorted(cid[order], torch.arange(g * g + 1, device=DEV))
    us, vs = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            nx, ny = cell[:, 0] + dx, cell[:, 1] + dy
            src = torch.nonzero((nx >= 0) & (nx < g) & (ny >= 0) & (ny < g)).flatten()
            nc = nx[src] * g + ny[src]
            cnt = bounds[nc + 1] - bounds[nc]
            first = torch.cumsum(cnt, 0) - cnt
            rep = torch.repeat_interleave(src, cnt)
            off = torch.repeat_interleave(bounds[nc] - first, cnt) + torch.arange(rep.numel(), device=DEV)
            dst = order[off]
            keep = rep < dst
            rep, dst = rep[keep], dst[keep]
            close = ((x[rep] - x[dst]) ** 2).sum(1) < r * r
            us.append(rep[close])
            vs.append(dst[close])
    cliques = max(1, n // 50)
    member = torch.randint(0, n, (cliques, 32), generator=gen, device=DEV)
    size = torch.randint(8, 33, (cliques,), generator=gen, device=DEV)
    i, j = torch.triu_indices(32, 32, 1, device=DEV)
    inside = (j.unsqueeze(0) < size.unsqueeze(1)).flatten()
    us.append(member[:, i].flatten()[inside])
    vs.append(member[:, j].flatten()[inside])
    return _finish(n, torch.cat(us), torch.cat(vs), gen, wmul)


def _edges(family, n, degree, seed, wmul=1):
    gen = _generator(seed)
    if family == "er":
        return _erdos_renyi(n, degree, gen, wmul)
    if family == "conflict":
        return _conflict(n, degree, gen, wmul)
    if family == "chung_lu":
        return _chung_lu(n, degree, min(5000, n // 4), gen, wmul)
    return _complete(n, gen)


def _mean_degree(family, n, degree):
    return n - 1 if family == "dense" else degree


# ------------------------------------------------------------------ cases
def _search(name, problem, family, n, degree, struct, iters, m=0, tenure=0, piter=500, wmul=1):
    """One tabu search of `iters` iterations; tenure 0: the reference's schedule."""
    return {"name": name, "form": "search", "problem": problem, "family": family, "n": n, "degree": degree,
            "struct": struct, "iters": iters, "m": m, "tenure": tenure, "piter": piter, "wmul": wmul}


def listed():
    return [
        # the smallest search a restart loop makes: all launch and call latency
        _search("mdp_tiny_hash", "mdp", "er", 200, 10, "hash", 100, m=20, tenure=10),
        # plain MDP of 2,000 vertices, the structure compared first
        _search("mdp_er2000_csr", "mdp", "er", 2000, 20, "csr", 2000, m=200, tenure=20),
        # a dense instance of the reference's MDG data set, its own tenure schedule
        _search("mdp_dense2000_bb", "mdp", "dense", 2000, 0, "csr-bb", 500, m=200),
        # the large sparse MDP graph with power-law degrees
        _search("mdp_powerlaw200k_hash", "mdp", "chung_lu", 200_000, 50, "hash", 500, m=2000, tenure=100),
        # the bisection benchmark: 2.5e9 pairs per iteration
        _search("maxbs_conflict100k_csr", "maxbs", "conflict", 100_000, 60, "csr", 1000, tenure=50),
        # the swap-weight matrix, the largest state a search holds
        _search("maxbs_conflict60k_wswap", "maxbs", "conflict", 60_001, 60, "wswap", 300, tenure=50),
        # odd size, reference tenures and frequent perturbations, bitmap rows
        _search("maxbs_perturb30k_bitset", "maxbs", "conflict", 30_011, 60, "csr-bitset", 400, piter=60),
        # large fixed-point weights: 64-bit contributions
        _search("maxbs_wide10k_bb", "maxbs", "conflict", 10_007, 40, "csr-bb", 300, tenure=30, wmul=20_000),
        # a batch of restarts of uneven instances, planned once and replayed
        {"name": "batch_64_mixed", "form": "batch", "jobs": 64, "n_lo": 200, "n_hi": 5000, "iters": 500},
        # a burst of requests to the server, small and large ones together
        {"name": "serve_16_mixed", "form": "serve", "jobs": 16, "n_lo": 1000, "n_hi": 40_000, "iters": 400},
        # loading: edge list on the host -> lookup structure on the GPU, then queries
        {"name": "build_lookup_100k_hash", "form": "build", "family": "conflict", "n": 100_000, "degree": 60,
         "struct": "hash", "queries": 1_000_000},
        # one decision from a caller-held state, nothing allocated
        {"name": "decide_noalloc_20k", "form": "decide", "problem": "mdp", "family": "chung_lu", "n": 20_001,
         "degree": 50, "m": 1000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    form = rng.choice(("search",) * 8 + ("batch", "serve", "build", "decide"))
    if form == "batch":
        return {"form": form, "jobs": rng.randint(8, 64), "n_lo": 200, "n_hi": _log_int(rng, 400, 5000),
                "iters": _log_int(rng, 100, 500)}
    if form == "serve":
        return {"form": form, "jobs": rng.randint(4, 16), "n_lo": 1000, "n_hi": _log_int(rng, 2000, 40_000),
                "iters": _log_int(rng, 100, 400)}
    if form == "build":
        return {"form": form, "family": rng.choice(("er", "conflict", "chung_lu")), "n": _log_int(rng, 500, 100_000),
                "degree": rng.randint(5, 60), "struct": rng.choice(STRUCTS), "queries": _log_int(rng, 1000, 1_000_000)}
    if form == "decide":
        n = _log_int(rng, 200, 20_000)
        return {"form": form, "problem": rng.choice(("mdp", "maxbs")), "family": rng.choice(("er", "chung_lu")), "n": n,
                "degree": rng.randint(5, 50), "m": max(1, n * rng.randint(5, 20) // 100)}
    problem = rng.choice(("mdp", "maxbs"))
    struct = rng.choice(STRUCTS)
    wmul = 20_000 if rng.random() < 0.1 else 1
    if problem == "mdp":
        family = rng.choice(("er", "chung_lu", "dense"))
        n = _log_int(rng, 200, 2000 if family == "dense" else 100_000)
        share = rng.uniform(0.05, 0.2) if n < 20_000 else rng.uniform(0.005, 0.02)
        m = max(2, int(n * share))
    else:
        family = rng.choice(("er", "conflict"))
        n, m = _log_int(rng, 200, 60_000), 0
    return {"form": form, "problem": problem, "family": family, "n": n,
            "degree": 0 if family == "dense" else rng.randint(5, 60), "struct": struct, "iters": _log_int(rng, 50, 300),
            "m": m, "tenure": rng.choice((0, 10, 20, 50, 100)) if n >= 1000 else rng.choice((0, 5, 10)),
            "piter": rng.choice((60, 500)), "wmul": 1 if family == "dense" else wmul}


# ------------------------------------------------------------------ states
def _problem(name):
    return T.PROBLEM_MDP if name == "mdp" else T.PROBLEM_MAXBS


def _graph(case, edges, problem):
    n = case["n"]
    g = T.Graph(n, *edges, case["struct"], drop_self_loops=problem == T.PROBLEM_MDP, device_arrays=True)
    torch.cuda.synchronize()  # the edge arrays may go now
    return g


def _mixed_job(case, k):
    """Solve k of a batch or burst: sizes spread over the range, problems in turn."""
    count = case["jobs"]
    rng = np.random.default_rng((count, k))
    lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
    n = int(round(math.exp(lo + (hi - lo) * (k + rng.random()) / count)))
    problem = T.PROBLEM_MDP if k % 2 == 0 else T.PROBLEM_MAXBS
    return n, problem, max(2, int(n * rng.uniform(0.05, 0.2))), float(rng.uniform(5, 50))


def prepare(case, seed):
    form = case["form"]
    if form == "search":
        problem = _problem(case["problem"])
        g = _graph(case, _edges(case["family"], case["n"], case["degree"], seed, case["wmul"]), problem)
        tenure = dict(tenure_policy=T.TENURE_FIXED, tenure=case["tenure"]) if case["tenure"] else {}
        s = T.Solver(g, problem, m=case["m"], max_iter=case["iters"], piter=case["piter"], seed=seed % 100_003 + 1, **tenure)
        start = T.random_start(problem, case["n"], case["m"], seed % 100_003 + 1)
        return {"form": form, "solver": s, "graph": g, "start": start, "iters": case["iters"]}
    if form == "batch":
        jobs = []
        for k in range(case["jobs"]):
            n, problem, m, degree = _mixed_job(case, k)
            # the structures in turn: the searches of one batch need not share one
            g = T.Graph(n, *_edges("er", n, degree, seed * 1000 + k), STRUCTS[(k // 2) % 6],
                        drop_self_loops=problem == T.PROBLEM_MDP, device_arrays=True)
            torch.cuda.synchronize()
            jobs.append(T.BatchJobSpec(g, problem, m=m if problem == T.PROBLEM_MDP else 0, max_iter=case["iters"],
                                       tenure_policy=T.TENURE_FIXED, tenure=10 + k % 20, piter=200, seed=k + 1))
        return {"form": form, "batch": T.Batch(jobs, max_bytes=8 << 30)}
    if form == "serve":
        reqs = []
        for k in range(case["jobs"]):
            n, problem, m, degree = _mixed_job(case, k)
            family = "chung_lu" if problem == T.PROBLEM_MDP else "conflict"
            u, v, w = (x.cpu().numpy() for x in _edges(family, n, degree, seed * 1000 + k))
            reqs.append(dict(n=n, u=u, v=v, w=w, problem=problem, kind=STRUCTS[k % 6],
                             m=max(2, n // 100) if problem == T.PROBLEM_MDP else 0, max_iter=case["iters"],
                             tenure_policy=T.TENURE_FIXED, tenure=10, seed=k + 1))
        order = np.random.default_rng(seed).permutation(len(reqs))
        return {"form": form, "server": T.Server(max_bytes=8 << 30), "reqs": [reqs[i] for i in order]}
    if form == "build":
        u, v, w = (x.cpu().numpy() for x in _edges(case["family"], case["n"], case["degree"], seed))
        rng = np.random.default_rng(seed)
        q = case["queries"]
        hit = rng.integers(0, len(u), q // 2)  # half of the queries are edges
        qu = np.concatenate([u[hit], rng.integers(0, case["n"], q - q // 2)]).astype(np.int32)
        qv = np.concatenate([v[hit], rng.integers(0, case["n"], q - q // 2)]).astype(np.int32)
        return {"form": form, "n": case["n"], "edges": (u, v, w), "struct": case["struct"], "qu": qu, "qv": qv}
    # decide: a state some moves into a search, held in the caller's own buffers
    problem = _problem(case["problem"])
    n = case["n"]
    m = case["m"] if problem == T.PROBLEM_MDP else n // 2
    u, v, w = _edges(case["family"], n, case["degree"], seed)
    g = T.Graph(n, u, v, w, "csr", drop_self_loops=problem == T.PROBLEM_MDP, device_arrays=True)
    torch.cuda.synchronize()
    s = T.Solver(g, problem, m=case["m"], max_iter=20, tenure_policy=T.TENURE_FIXED, tenure=15, seed=seed % 100_003 + 1)
    s.init(None)
    s.step(20)
    r = s.result()
    sol, _, tab, vg = s.state()
    s.close()
    g.close()
    a, b, ww = torch.cat([u, v]).long(), torch.cat([v, u]).long(), torch.cat([w, w])
    order = torch.argsort(a * n + b)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.cumsum(torch.bincount(a, minlength=n), 0)
    dev = lambda x, t: torch.from_numpy(np.ascontiguousarray(x)).to(DEV, t)  # noqa: E731
    return {"form": form, "problem": problem, "n": n, "m": m, "iter": r.iterations, "cur": r.cur, "best": r.best,
            "rowptr": rowptr, "col": b[order].to(torch.int32), "w": ww[order].contiguous(), "sol": dev(sol, torch.int32),
            "vg": dev(vg, torch.int64), "tab": dev(tab, torch.int32),
            "out": torch.zeros(2, dtype=torch.int64, device=DEV)}


# ------------------------------------------------------------------ runs
def _numbers(r):
    return np.array([r.iterations, r.evaluations, r.cur, r.best, r.best_true, r.perturbations, int(r.stopped)], np.int64)


def run(state):
    form = state["form"]
    if form == "search":
        s = state["solver"]
        s.init(state["start"])
        s.step(state["iters"])
        r = s.result()
        sol, pos, tab, vg = s.state()
        return {"numbers": _numbers(r), "best": r.best_sol, "sol": sol, "pos": pos, "tab": tab, "vg": vg}
    if form == "batch":
        res = state["batch"].run()
        return {"numbers": np.stack([_numbers(r) for r in res]), "best": np.concatenate([r.best_sol for r in res])}
    if form == "serve":
        server = state["server"]
        tickets = [server.submit(**q) for q in state["reqs"]]
        done = {}
        while len(done) < len(tickets):
            for d in server.poll(wait_ms=50):
                done[d.ticket] = d
        res = [done[t].result for t in tickets]
        return {"numbers": np.stack([_numbers(r) for r in res]), "best": np.concatenate([r.best_sol for r in res])}
    if form == "build":
        g = T.Graph(state["n"], *state["edges"], state["struct"], drop_self_loops=False)
        w = g.lookup(state["qu"], state["qv"])
        i = g.info()
        g.close()
        return {"w": w, "info": np.array([i.num_entries, i.max_weighted_degree], np.int64)}
    decide = T.lib().ts_best_swap_noalloc
    decide.argtypes = [ctypes.c_int32] * 3 + [ctypes.c_int64] * 3 + [ctypes.c_void_p] * 8
    st = decide(state["problem"], state["n"], state["m"], state["iter"], state["cur"], state["best"],
                *(state[k].data_ptr() for k in ("rowptr", "col", "w", "sol", "vg", "tab", "out")), None)
    if st != 0:
        raise RuntimeError(f"ts_best_swap_noalloc: status {st}")
    return state["out"]


# ------------------------------------------------------------------ work
def _search_work(n, entries, iters, key_bytes):
    """Graph, start and final state once; each iteration decides on every
    vertex's contribution and tabu stamp and walks the two moved vertices'
    rows (neighbour, weight, contribution updated)."""
    moved = 2.0 * entries / n * (8 + 2 * key_bytes)
    return 8.0 * (n + 1) + 8.0 * entries + 4.0 * n + n * (16.0 + 8.0) + iters * (n * (key_bytes + 4.0) + moved)


def work(case):
    form = case["form"]
    ops = 0.0
    if form == "search":
        n = case["n"]
        entries = n * _mean_degree(case["family"], n, case["degree"])
        b = _search_work(n, entries, case["iters"], 8 if case["wmul"] > 1 else 4)
    elif form in ("batch", "serve"):
        b = 0.0
        for k in range(case["jobs"]):
            n, _, _, degree = _mixed_job(case, k)
            b += _search_work(n, n * degree, case["iters"], 4)
    elif form == "build":
        entries = case["n"] * case["degree"]
        slots = 2.0 * entries if case["struct"] == "hash" else 0.0
        words = case["n"] ** 2 / 8.0 if "bitset" in case["struct"] else 0.0
        b = 6.0 * entries + 8.0 * entries + 8.0 * case["n"] + 8.0 * slots + words + 12.0 * case["queries"]
    else:
        n = case["n"]
        b = n * (4.0 + 8.0 + 4.0) + 16.0
    return {"bytes": b, "flops": ops}


def exact(case, seed):
    """Every output is a whole number, compared bit for bit."""
    return None
