"""Packed solves (batched form) of searches that the candidate pass leaves to the
sweeps: the same results as the oracle's on every cluster size, and no slower
than with the sweep pinned."""
import time

import numpy as np
import pytest

import ts_b200 as T
from oracle import oracle as O

pytestmark = pytest.mark.gpu
FIXED = T.TENURE_FIXED


def all_but_a_matching(n):
    """Every pair but (0, 1), (2, 3), ... joined by weight 1: ties everywhere."""
    u, v = np.triu_indices(n, 1)
    keep = (u // 2) != (v // 2)
    return u[keep].astype(np.int32), v[keep].astype(np.int32), np.ones(int(keep.sum()), np.int32)


@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
def test_tied_searches_on_every_cluster_size(gpu, problem, kind):
    n = 260
    drop = problem == T.PROBLEM_MDP
    u, v, w = all_but_a_matching(n)
    w[::97] = 3  # a few pairs stand out: the pass settles some iterations
    kw = dict(m=60 if drop else 0, max_iter=150, tenure_policy=FIXED, tenure=9, piter=20, gamma=12, seed=4)
    o = O.run(O.Graph(n, u, v, w, drop_self_loops=drop), O.MDP if drop else O.MAXBS, threads=0, **kw)
    g = T.Graph(n, u, v, w, kind, drop_self_loops=drop)
    got = T.batch_solve([T.BatchJobSpec(g, problem, cluster=cs, **kw) for cs in (0, 1, 2, 4, 8)])
    for r in got:
        assert (r.iterations, r.evaluations, r.cur, r.best, r.best_true, r.stopped, r.device_error) == \
               (o.iterations, o.evaluations, o.cur, o.best, o.best_true, o.stopped, 0)
        np.testing.assert_array_equal(r.best_sol, got[0].best_sol)
    g.close()


@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
def test_failed_tries_do_not_add_up(gpu, problem):
    """Where every iteration is left to the sweep, tries get rare (Max Bisection:
    a try at every iteration took 1.25 times the sweeps' time)."""
    n = 150
    u, v, w = all_but_a_matching(n)
    g = T.Graph(n, u, v, w, "csr", drop_self_loops=problem == T.PROBLEM_MDP)

    def batch_time(sweep):
        b = T.Batch([T.BatchJobSpec(g, problem, m=30, max_iter=2000, tenure_policy=FIXED, tenure=8, seed=k + 1, cluster=1,
                                    piter=10 ** 6, sweep=sweep) for k in range(40)])
        best = 1e9
        for _ in range(8):
            t = time.perf_counter()
            b.launch()
            b.sync()
            best = min(best, time.perf_counter() - t)
        out = [(r.cur, r.best) for r in b.results()]
        b.close()
        return best, out

    pinned, want = min((batch_time(s) for s in (T.PASS_TILE, T.PASS_ROWS)), key=lambda x: x[0])
    auto, got = batch_time(T.PASS_AUTO)
    g.close()
    assert got == want
    assert auto < 1.2 * pinned, (auto, pinned)


def complete(n):
    u, v = (x.astype(np.int32) for x in np.triu_indices(n, 1))
    return u, v, np.ones(len(u), np.int32)


def sparse(n, deg, seed):
    rng = np.random.default_rng(seed)
    a, b = rng.integers(0, n, (2, int(n * deg / 2)))
    key = np.unique(np.minimum(a, b)[a != b] * n + np.maximum(a, b)[a != b])
    return (key // n).astype(np.int32), (key % n).astype(np.int32), rng.integers(1, 1001, len(key)).astype(np.int32)


@pytest.mark.parametrize("case", ["complete", "complete, many", "sides tabu", "too large"])
def test_open_cluster_of_swept_solves(gpu, case):
    """A batch that leaves the cluster sizes open gives solves that sweep as many
    CTAs as the pinned sweep gets, so it is not slower."""
    problem, count, kw = T.PROBLEM_MAXBS, 4, dict(max_iter=60, tenure=10)
    if case == "complete":
        n, edges = 1000, complete(1000)
    elif case == "complete, many":
        problem, count, kw = T.PROBLEM_MDP, 200, dict(m=80, max_iter=60, tenure=8)
        n, edges = 500, complete(500)
    elif case == "sides tabu":
        n, edges, kw = 1500, sparse(1500, 12, 1), dict(max_iter=1200, tenure=1000, piter=10 ** 6)
    else:
        problem, count, kw = T.PROBLEM_MDP, 2, dict(m=300, max_iter=20, tenure=20)
        n, edges = 330_000, sparse(330_000, 8, 2)
    g = T.Graph(n, *edges, "hash", drop_self_loops=problem == T.PROBLEM_MDP)

    def batch_time(sweep):
        b = T.Batch([T.BatchJobSpec(g, problem, tenure_policy=FIXED, seed=k + 1, sweep=sweep, **kw) for k in range(count)])
        best = 1e9
        for _ in range(4):
            t = time.perf_counter()
            b.launch()
            b.sync()
            best = min(best, time.perf_counter() - t)
        out = [(r.cur, r.best, r.iterations) for r in b.results()]
        b.close()
        return best, out

    pinned, want = min((batch_time(s) for s in (T.PASS_TILE, T.PASS_ROWS)), key=lambda x: x[0])
    auto, got = batch_time(T.PASS_AUTO)
    g.close()
    assert got == want
    assert auto < 1.5 * pinned, (auto, pinned)  # 1.9 to 8 times by the number of vertices alone


def test_pinned_and_default_solves_run_in_kernels_of_their_own(gpu):
    """The sweeps' kernels are compiled without the candidate pass (64 MDP solves
    of n = 2,000 on the tile pass took 38.6 ms in one kernel with it, 23.1 in
    their own), so a batch of both has two groups."""
    n = 300
    u, v, w = sparse(n, 8, 5)
    g = T.Graph(n, u, v, w, "csr", drop_self_loops=True)
    b = T.Batch([T.BatchJobSpec(g, T.PROBLEM_MDP, m=30, max_iter=50, tenure_policy=FIXED, tenure=5, seed=9, cluster=1, sweep=sw)
                 for sw in (T.PASS_AUTO, T.PASS_TILE, T.PASS_AUTO, T.PASS_ROWS)])
    assert b.info().groups == 2
    got = b.run()
    b.close()
    g.close()
    for r in got[1:]:
        assert (r.iterations, r.cur, r.best, r.best_true) == (got[0].iterations, got[0].cur, got[0].best, got[0].best_true)
        np.testing.assert_array_equal(r.best_sol, got[0].best_sol)


@pytest.mark.parametrize("weights,groups", [("ones", 1), ("both signs", 2)])
def test_only_equal_weights_tie_everywhere(gpu, weights, groups):
    """A complete graph of weights 1 is left to the sweeps' kernels from the start;
    one of weights 1 and -1 is not: its contributions differ."""
    n = 200
    u, v, w = complete(n)
    if weights == "both signs":
        w = np.where(np.random.default_rng(2).random(len(u)) < 0.5, -1, 1).astype(np.int32)
    kw = dict(max_iter=100, tenure_policy=FIXED, tenure=8, piter=30, gamma=10, seed=3)
    o = O.run(O.Graph(n, u, v, w, drop_self_loops=False), O.MAXBS, threads=0, **kw)
    g = T.Graph(n, u, v, w, "hash", drop_self_loops=False)
    b = T.Batch([T.BatchJobSpec(g, T.PROBLEM_MAXBS, cluster=1, sweep=s, **kw) for s in (T.PASS_AUTO, T.PASS_TILE)])
    assert b.info().groups == groups
    for r in b.run():
        assert (r.iterations, r.cur, r.best, r.best_true) == (o.iterations, o.cur, o.best, o.best_true)
    b.close()
    g.close()


def tied(family, n):
    if family == "bipartite":
        u, v = (x.ravel() for x in np.meshgrid(np.arange(n // 2), np.arange(n // 2, n)))
    else:  # cliques of 20
        a, b = np.triu_indices(20, 1)
        first = np.arange(n // 20)[:, None] * 20
        u, v = (first + a).ravel(), (first + b).ravel()
    return u.astype(np.int32), v.astype(np.int32), np.ones(len(u), np.int32)


@pytest.mark.parametrize("family", ["bipartite", "cliques"])
@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
def test_solves_given_up_by_the_candidate_pass(gpu, problem, family):
    """Equal weights that tie for good: the solves are run again by the sweeps'
    kernel on its own clusters, beside others of their group that are not; twice,
    as a replay clears the list; with the sweep's clusters and explicit ones."""
    n, drop = 400, problem == T.PROBLEM_MDP
    kw = dict(m=40 if drop else 0, max_iter=200, tenure_policy=FIXED, tenure=8, piter=60, gamma=16)
    edges = [tied(family, n), sparse(n, 8, 3)]
    graphs = [T.Graph(n, *e, "csr", drop_self_loops=drop) for e in edges]
    want = [[O.run(O.Graph(n, *e, drop_self_loops=drop), O.MDP if drop else O.MAXBS, threads=0, seed=k + 1, **kw)
             for k in range(3)] for e in edges]
    specs = [(T.BatchJobSpec(g, problem, seed=k + 1, cluster=cs, **kw), w[k])
             for cs in (0, 1, 4) for g, w in zip(graphs, want) for k in range(3)]
    b = T.Batch([s for s, _ in specs])
    for _ in range(2):
        for r, (_, o) in zip(b.run(), specs):
            assert (r.iterations, r.evaluations, r.cur, r.best, r.best_true, r.stopped, r.device_error) == \
                   (o.iterations, o.evaluations, o.cur, o.best, o.best_true, o.stopped, 0)
    b.close()
    for g in graphs:
        g.close()


def test_given_up_solves_get_the_sweeps_clusters(gpu):
    """Eight bisections of 2,000 vertices in unit cliques: 7 times the sweeps' time
    on the candidate pass's one CTA each."""
    n = 2000
    g = T.Graph(n, *tied("cliques", n), "csr", drop_self_loops=False)

    def batch_time(sweep):
        b = T.Batch([T.BatchJobSpec(g, T.PROBLEM_MAXBS, max_iter=150, tenure_policy=FIXED, tenure=20, piter=100, seed=k + 1,
                                    sweep=sweep) for k in range(8)])
        best = 1e9
        for _ in range(4):
            t = time.perf_counter()
            b.launch()
            b.sync()
            best = min(best, time.perf_counter() - t)
        out = [(r.cur, r.best, r.iterations) for r in b.results()]
        b.close()
        return best, out

    pinned, want = min((batch_time(s) for s in (T.PASS_TILE, T.PASS_ROWS)), key=lambda x: x[0])
    auto, got = batch_time(T.PASS_AUTO)
    g.close()
    assert got == want
    assert auto < 3 * pinned, (auto, pinned)
