"""Inputs at the ends of their ranges, against the CPU oracle."""
import numpy as np
import pytest

import ts_b200 as T
from oracle import oracle as O
from test_parity_gpu import compare_run, rand_graph

pytestmark = pytest.mark.gpu
FIXED = T.TENURE_FIXED


def lowest_weight_graph():
    """A random graph of 60 vertices with five edges of weight -2^31."""
    u, v, w = rand_graph(60, 0.15, 31, wlo=-1000, whi=1000)
    w[np.random.default_rng(5).choice(len(w), 5, replace=False)] = -2 ** 31
    return 60, u, v, w


@pytest.mark.parametrize("sweep", [T.PASS_AUTO, T.PASS_TILE, T.PASS_ROWS], ids=["auto", "tile", "rows"])
@pytest.mark.parametrize("kind", T.STRUCT_NAMES)
@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
def test_lowest_weight(gpu, problem, kind, sweep):
    n, u, v, w = lowest_weight_graph()
    compare_run(problem, kind, n, u, v, w, m=12 if problem == T.PROBLEM_MDP else 0, iters=40, tenure_policy=FIXED,
                tenure=4, piter=9, gamma=8, seed=3, sweep=sweep)


@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
def test_lowest_weight_batched(gpu, problem):
    n, u, v, w = lowest_weight_graph()
    drop = problem == T.PROBLEM_MDP
    kw = dict(m=12 if drop else 0, max_iter=40, tenure_policy=FIXED, tenure=4, piter=9, gamma=8, seed=3)
    o = O.run(O.Graph(n, u, v, w, drop_self_loops=drop), O.MDP if drop else O.MAXBS, threads=0, **kw)
    graphs = [T.Graph(n, u, v, w, kind, drop_self_loops=drop) for kind in T.STRUCT_NAMES]
    for r in T.batch_solve([T.BatchJobSpec(g, problem, **kw) for g in graphs]):
        assert (r.iterations, r.cur, r.best, r.best_true, r.device_error) == (o.iterations, o.cur, o.best, o.best_true, 0)
    for g in graphs:
        g.close()
