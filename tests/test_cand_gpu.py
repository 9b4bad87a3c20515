"""The candidate pass (the default sweep choice) against the CPU oracle, bit for bit.

Sizes sit at the edges of its slices: one CTA to sixteen, slices that are not
a multiple of four, sides smaller than the cluster.  The graphs reach each of
its branches: seeds that decide alone, candidate pairs looked up, candidate
rows' entries (also rows walked by a whole CTA), both signs of weight, 64-bit
contributions, perturbations, ties that hand the iteration to the sweeps, and
searches that end or need the penalty rule.
"""
import numpy as np
import pytest

import ts_b200 as T
from test_parity_gpu import compare_run, rand_graph

pytestmark = pytest.mark.gpu
FIXED = T.TENURE_FIXED


def er(n, deg, seed, whi=1000, wlo=1):
    rng = np.random.default_rng(seed)
    a, b = rng.integers(0, n, (2, int(n * deg / 2)))
    key = np.unique(np.minimum(a, b)[a != b] * n + np.maximum(a, b)[a != b])
    w = rng.integers(wlo, whi + 1, len(key))
    return (key // n).astype(np.int32), (key % n).astype(np.int32), w.astype(np.int32)


@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
@pytest.mark.parametrize("n", [97, 4096, 4097, 8193, 16385, 66001])
def test_mdp_slice_edges(gpu, kind, n):
    u, v, w = er(n, 12, n)
    compare_run(T.PROBLEM_MDP, kind, n, u, v, w, m=max(3, n // 300), iters=60, tenure_policy=FIXED, tenure=7, seed=2)


@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
@pytest.mark.parametrize("n", [41, 4099, 8197])
def test_maxbs_slice_edges_and_perturbations(gpu, kind, n):
    u, v, w = er(n, 10, n + 1)
    compare_run(T.PROBLEM_MAXBS, kind, n, u, v, w, iters=60, tenure_policy=FIXED, tenure=5, piter=9, gamma=14, seed=3,
                initial=np.arange(n, dtype=np.int32) % 2 if n % 2 == 0 else (np.arange(n) >= n // 2).astype(np.int32))


@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
@pytest.mark.parametrize("case", ["negative", "unit", "wide", "dups", "dense"])
def test_weights_and_ties(gpu, kind, problem, case):
    n = 300
    m = 40 if problem == T.PROBLEM_MDP else 0
    drop = {}
    if case == "negative":
        u, v, w = er(n, 20, 5, whi=500, wlo=-500)
    elif case == "unit":
        u, v, w = er(n, 9, 6, whi=1)
    elif case == "wide":
        u, v, w = er(n, 20, 7, whi=2 ** 30, wlo=2 ** 28)
    elif case == "dups":
        u, v, w = rand_graph(n, 0.1, 8, dup=True, selfloops=problem == T.PROBLEM_MAXBS)
    else:
        u, v = (x.astype(np.int32) for x in np.triu_indices(n, 1))
        w = np.ones(len(u), np.int32)
    compare_run(problem, kind, n, u, v, w, m=m, iters=150, tenure_policy=T.TENURE_REF, maxt=24, piter=25, gamma=20,
                seed=9, step_chunks=(1, 7, None), **drop)


@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
def test_hub_rows(gpu, kind, problem):
    """Rows of more entries than a warp walks: degree-3,000 hubs on both sides."""
    n = 6000
    rng = np.random.default_rng(11)
    u, v, w = er(n, 6, 12)
    hubs = rng.choice(n, 24, replace=False)
    hu = np.repeat(hubs, 3000)
    hv = rng.integers(0, n, len(hu))
    key = np.unique(np.concatenate([np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v),
                                    np.minimum(hu, hv)[hu != hv] * n + np.maximum(hu, hv)[hu != hv]]))
    u, v = (key // n).astype(np.int32), (key % n).astype(np.int32)
    w = rng.integers(1, 1001, len(u)).astype(np.int32)
    compare_run(problem, kind, n, u, v, w, m=60 if problem == T.PROBLEM_MDP else 0, iters=60, tenure_policy=FIXED,
                tenure=6, seed=4)


@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
def test_enqueue_keeps_its_count(gpu, problem):
    """enqueue(j) advances j iterations at most, whatever the admitted target."""
    n = 500
    u, v, w = er(n, 10, 13)
    g = T.Graph(n, u, v, w, "csr", drop_self_loops=problem == T.PROBLEM_MDP)
    s = T.Solver(g, problem, m=30 if problem == T.PROBLEM_MDP else 0, max_iter=100, tenure_policy=FIXED, tenure=5)
    s.init(None)
    assert s.prepare(40) == 40
    s.enqueue(1)
    s.enqueue(3)
    assert s.result().iterations == 4
    assert s.sync() == 40
    s.close()
    g.close()


@pytest.mark.parametrize("sweep", [T.PASS_AUTO, T.PASS_TILE])
@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
def test_wswap_started_again(gpu, problem, sweep):
    """A solver started again (its matrix cleared along the old state's edges)
    searches as a new one does, with duplicated edges and self-loops too."""
    n = 400
    u, v, w = rand_graph(n, 0.05, 21, dup=True, selfloops=problem == T.PROBLEM_MAXBS)
    g = T.Graph(n, u, v, w, "wswap", drop_self_loops=problem == T.PROBLEM_MDP)
    kw = dict(m=40 if problem == T.PROBLEM_MDP else 0, max_iter=120, tenure_policy=FIXED, tenure=7, piter=11, gamma=9,
              sweep=sweep)
    again = T.Solver(g, problem, **kw)
    for seed in (1, 2, 3):
        start = T.random_start(problem, n, kw["m"], seed)
        new = T.Solver(g, problem, **kw)
        for s in (again, new):
            s.init(start)
            s.step(120)
        for a, b in zip(again.state(), new.state()):
            np.testing.assert_array_equal(a, b)
        assert again.result().best == new.result().best
        new.close()
    again.close()
    g.close()
