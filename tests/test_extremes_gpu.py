"""Inputs at the ends of their ranges, against the CPU oracle: the lowest
32-bit weight, and a row of more entries than a packed queue word can number.
"""
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


def long_row_graph(problem):
    """2^22 + 9 parallel edges 0-1 of weight 0, so that vertex 0's other
    neighbours lie beyond the 2^22-th entry of its row, and weights for which
    the best swap is (0, 40), an adjacent pair that only row 0 leads to: column
    40 is further from its side's best than half of what the pair's weight
    makes up."""
    n, few = 64, 2 ** 22 + 9
    if problem == T.PROBLEM_MAXBS:  # part 0: vertices 0-31
        rest = [(0, k, 100) for k in range(2, 12)] + [(0, 40, 100), (50, 51, 50)]
    else:  # inside: 0-31; contributions are weighted degrees into the set
        rest = [(k, j, 100) for k in range(1, 32) for j in range(k + 1, 32)] + \
               [(50, k, 90) for k in range(1, 4)] + [(40, 1, 300), (0, 40, -100)]
    ru, rv, rw = (np.array(x, np.int32) for x in zip(*rest))
    u = np.concatenate([np.zeros(few, np.int32), ru])
    v = np.concatenate([np.ones(few, np.int32), rv])
    w = np.concatenate([np.zeros(few, np.int32), rw])
    initial = np.arange(32, dtype=np.int32) if problem == T.PROBLEM_MDP else (np.arange(n) >= 32).astype(np.int32)
    return n, u, v, w, initial


@pytest.mark.parametrize("kind", ["csr", "csr-bb", "hash", "wswap"])
@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
def test_row_of_more_than_2_to_22_entries(gpu, problem, kind):
    n, u, v, w, initial = long_row_graph(problem)
    compare_run(problem, kind, n, u, v, w, m=32 if problem == T.PROBLEM_MDP else 0, iters=6, tenure_policy=FIXED, tenure=3,
                initial=initial)
