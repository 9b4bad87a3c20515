"""Forms of the candidate pass that its size tests do not reach, against the
CPU oracle: batched solves on every cluster size, 64-bit contributions in a
cluster of several CTAs, positions that stay in HBM, lists and queues that
overflow in one CTA of a cluster, more long rows than the whole-CTA walk takes.
"""
import numpy as np
import pytest

import ts_b200 as T
from oracle import oracle as O
from test_cand_gpu import er
from test_parity_gpu import compare_run, node_weight_graph

pytestmark = pytest.mark.gpu
FIXED = T.TENURE_FIXED


def same_as_oracle(r, o, n):
    assert (r.iterations, r.evaluations, r.cur, r.best, r.best_true, r.stopped, r.device_error) == \
           (o.iterations, o.evaluations, o.cur, o.best, o.best_true, o.stopped, 0)
    best = o.best_sol
    if len(r.best_sol) == n:  # Max Bisection: sides
        best = np.ones(n, np.int32)
        best[o.best_sol[: n // 2]] = 0
    np.testing.assert_array_equal(r.best_sol, best)


@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
@pytest.mark.parametrize("weights", ["positive", "both signs", "wide"])
def test_batched_on_every_cluster_size(gpu, problem, kind, weights):
    n = 1501
    drop = problem == T.PROBLEM_MDP
    lo, hi = {"positive": (1, 1000), "both signs": (-500, 500), "wide": (2 ** 27, 2 ** 28)}[weights]
    u, v, w = er(n, 12, 41, whi=hi, wlo=lo)
    kw = dict(m=150 if drop else 0, max_iter=200, tenure_policy=FIXED, tenure=15, piter=40, gamma=30, seed=6)
    o = O.run(O.Graph(n, u, v, w, drop_self_loops=drop), O.MDP if drop else O.MAXBS, threads=0, **kw)
    g = T.Graph(n, u, v, w, kind, drop_self_loops=drop)
    for r in T.batch_solve([T.BatchJobSpec(g, problem, cluster=cs, **kw) for cs in (0, 1, 2, 4, 8)]):
        same_as_oracle(r, o, n)
    g.close()


@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
def test_batched_bisections_that_get_four_ctas(gpu, kind):
    """2,048 < n <= 6,144 with an open cluster size in a batch that leaves SMs idle."""
    specs, want = [], []
    for n in (2049, 3333, 6143):
        u, v, w = node_weight_graph(n, 9.0, n)
        g = T.Graph(n, u, v, w, kind, drop_self_loops=False)
        kw = dict(max_iter=120, tenure_policy=FIXED, tenure=12, piter=25, gamma=20, seed=2)
        specs.append(T.BatchJobSpec(g, T.PROBLEM_MAXBS, **kw))
        want.append((n, O.run(O.Graph(n, u, v, w, drop_self_loops=False), O.MAXBS, threads=0, **kw)))
    for r, (n, o) in zip(T.batch_solve(specs), want):
        same_as_oracle(r, o, n)
    for s in specs:
        s.graph.close()


@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
@pytest.mark.parametrize("problem,n", [(T.PROBLEM_MDP, 9001), (T.PROBLEM_MAXBS, 2003), (T.PROBLEM_MAXBS, 13001)])
@pytest.mark.parametrize("signs", ["positive", "both signs"])
def test_wide_contributions_in_a_cluster(gpu, problem, n, kind, signs):
    u, v, w = er(n, 10, n, whi=2 ** 30, wlo=2 ** 27 if signs == "positive" else -2 ** 30)
    compare_run(problem, kind, n, u, v, w, m=n // 12 if problem == T.PROBLEM_MDP else 0, iters=50, tenure_policy=FIXED,
                tenure=6, piter=9, gamma=10, seed=5)


@pytest.mark.parametrize("kind", ["csr", "hash", "csr-bitset-bb"])
def test_positions_in_hbm(gpu, kind):
    """A bisection of 150,001 vertices: the cluster's shared memory has no room
    for the positions by vertex.  Near a local optimum, so that perturbations
    fall inside; against the tile pass (5.6e9 pairs an iteration)."""
    n = 150_001
    u, v, w = er(n, 6, 77)
    g = T.Graph(n, u, v, w, kind, drop_self_loops=False)

    def run(sweep, iters, piter, start, trace=True):
        s = T.Solver(g, T.PROBLEM_MAXBS, max_iter=iters, tenure_policy=FIXED, tenure=20, piter=piter, gamma=40, seed=8,
                     trace=trace, sweep=sweep)
        s.init(start)
        assert s.step(iters) == iters
        out = (s.result(), s.state(), s.trace() if trace else None)
        s.close()
        return out

    near = run(T.PASS_AUTO, 60_000, 10 ** 9, None, trace=False)[0].best_sol
    a, sa, ta = run(T.PASS_AUTO, 150, 40, near)
    b, sb, tb = run(T.PASS_TILE, 150, 40, near)
    g.close()
    assert a.perturbations >= 20  # at least one whole event
    np.testing.assert_array_equal(ta, tb)
    for x, y in zip(sa, sb):
        np.testing.assert_array_equal(x, y)
    assert (a.cur, a.best, a.best_true, a.perturbations) == (b.cur, b.best, b.best_true, b.perturbations)


def made_before_a_hand_over(kind, n, u, v, w, start, k, **kw):
    """Iterations of `k` that the candidate pass's launches make by themselves: it
    stops at the first that it leaves to a sweep, and one sweep follows."""
    g = T.Graph(n, u, v, w, kind, drop_self_loops=False)
    s = T.Solver(g, T.PROBLEM_MAXBS, max_iter=k, tenure_policy=FIXED, **kw)
    s.init(start)
    assert s.prepare(k) == k
    s.enqueue(k)
    made = s.result().iterations
    assert s.sync() == k
    s.close()
    g.close()
    return made


def matched(ids, w):
    return [(int(a), int(b), w) for a, b in zip(ids[::2], ids[1::2])]


@pytest.mark.parametrize("kind", ["csr", "hash", "wswap"])
def test_row_list_overflows_in_one_cta(gpu, kind):
    """40,000 vertices in 16 slices of 2,504 positions, lists of 2,048: the
    first CTA's positions hold pairs of a side (contribution 10, all of them
    candidates), everyone else is matched across the cut (-10)."""
    n, k = 40_000, 1252
    e = matched(np.arange(k), 10) + matched(np.arange(n // 2, n // 2 + k), 10)
    e += [(a, a + n // 2, 10) for a in range(k, n // 2)]
    u, v, w = (np.array(x, np.int32) for x in zip(*e))
    start = (np.arange(n) >= n // 2).astype(np.int32)
    assert made_before_a_hand_over(kind, n, u, v, w, start, 8, tenure=5) == 1
    compare_run(T.PROBLEM_MAXBS, kind, n, u, v, w, iters=8, tenure_policy=FIXED, tenure=5, seed=1, initial=start)


@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
def test_kept_entries_overflow_in_one_cta(gpu, kind):
    """5,000 vertices in 8 slices: those of the first CTA (300 of each side) have
    ten neighbours on each side among themselves (contribution 0), so that
    thousands of entries join candidates; the others lie three edges lower."""
    n, k, h = 5000, 300, 2500
    e = []
    for side in (0, h):
        e += [(side + a, side + (a + d) % k, 1) for a in range(k) for d in range(1, 6)]
    e += [(a, h + (a + d) % k, 1) for a in range(k) for d in range(10)]
    e += [(a, h + k + (a - k + d) % (h - k), 1) for a in range(k, h) for d in range(3)]
    u, v, w = (np.array(x, np.int32) for x in zip(*e))
    start = (np.arange(n) >= h).astype(np.int32)
    assert made_before_a_hand_over(kind, n, u, v, w, start, 8, tenure=4) == 1
    compare_run(T.PROBLEM_MAXBS, kind, n, u, v, w, iters=40, tenure_policy=FIXED, tenure=4, piter=9, gamma=6, seed=1,
                initial=start)


@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
def test_more_long_rows_than_the_whole_cta_walks(gpu, kind):
    """700 vertices matched within their sides by weights 1,000 to 1,500, else
    joined by weight 0 except at the two heaviest pairs: in the first iteration,
    which the pass settles, all of some 690 rows of 695 entries are walked."""
    n, h = 700, 350
    rng = np.random.default_rng(9)
    top = np.array([0, 1, h, h + 1])
    u, v = (x.astype(np.int32) for x in np.triu_indices(n, 1))
    mates = (u % 2 == 0) & (v == u + 1)
    keep = mates | ~(np.isin(u, top) | np.isin(v, top))
    u, v, mates = u[keep], v[keep], mates[keep]
    w = np.zeros(len(u), np.int32)
    w[mates] = rng.permutation(np.arange(1000, 1450))[: h]
    w[mates & np.isin(u, top)] = 1500
    start = (np.arange(n) >= h).astype(np.int32)
    assert made_before_a_hand_over(kind, n, u, v, w, start, 8, tenure=7) >= 2
    compare_run(T.PROBLEM_MAXBS, kind, n, u, v, w, iters=120, tenure_policy=FIXED, tenure=7, piter=15, gamma=12, seed=4,
                initial=start)
