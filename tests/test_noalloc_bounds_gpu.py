"""ts_best_swap_noalloc against every pair evaluated in numpy.

The entry point visits only rows and columns whose bounds reach a known pair;
these states reach each way it can go: seeds that decide, both signs of weight,
ties, duplicated pairs, aspiration, one side without a non-tabu position,
nothing allowed (every pair under the penalty rule), and sizes on both sides of
the bound on pairs below which all of them are visited.
"""
import numpy as np
import pytest

import ts_b200 as T
from test_zz_no_alloc import _csr, _entry

pytestmark = pytest.mark.gpu


def every_pair(problem, n, m, it, cur, best, rowptr, col, w, sol, vg, tab):
    W = np.zeros((n, n), np.int64)
    row = np.repeat(np.arange(n), np.diff(rowptr))
    _, first = np.unique(row * n + col, return_index=True)  # a duplicated pair's first entry
    W[row[first], col[first]] = w[first]
    a, b = sol[:m], sol[m:]
    wij = W[np.ix_(a, b)]
    x = vg[b][None, :] - vg[a][:, None] - wij if problem == T.PROBLEM_MDP else vg[a][:, None] + vg[b][None, :] + 2 * wij
    free = ((tab[a] <= it)[:, None] & (tab[b] <= it)[None, :]) | (x > best - cur)
    pen = -99999 if problem == T.PROBLEM_MDP else np.float32(x.astype(np.float64) - 9999999999.0).astype(np.int64)
    key = np.where(free, x, pen)
    i = int(np.argmax(key))  # the first of the largest
    return int(key.reshape(-1)[i]), i


@pytest.mark.parametrize("problem", [T.PROBLEM_MDP, T.PROBLEM_MAXBS])
@pytest.mark.parametrize("n,deg", [(2, 1), (257, 60), (2049, 90), (2200, 9)])
@pytest.mark.parametrize("weights", ["plain", "both signs", "unit"])
@pytest.mark.parametrize("tabu", ["none", "some", "aspire", "rows", "all"])
def test_decision_is_the_best_of_all_pairs(gpu, problem, n, deg, weights, tabu):
    import torch

    rng = np.random.default_rng([problem, n, deg, len(weights), len(tabu)])
    e = max(1, n * deg // 2)
    u, v = rng.integers(0, n, (2, e)).astype(np.int32)
    lo, hi = {"plain": (1, 1000), "both signs": (-1000, 1000), "unit": (1, 1)}[weights]
    wt = rng.integers(lo, hi + 1, e).astype(np.int32)
    rowptr, col, w = _csr(n, u, v, wt, True)
    m = max(1, 2 * n // 5) if problem == T.PROBLEM_MDP else n // 2
    sol = rng.permutation(n).astype(np.int32)
    vg = rng.integers(-3, 4, n).astype(np.int64) * (1 if weights == "unit" else 700)
    tab = np.zeros(n, np.int32)
    cur, best = 0, 10 ** 9
    if tabu in ("some", "aspire"):
        tab[rng.random(n) < 0.3] = 99
        best = 10 ** 9 if tabu == "some" else 0
    elif tabu == "rows":
        tab[sol[:m]] = 99
    elif tabu == "all":
        tab[:] = 99
    want = every_pair(problem, n, m, 50, cur, best, rowptr, col, w, sol, vg, tab)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (rowptr, col, w, sol, vg, tab)]
    if not len(col):
        d[1] = d[2] = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    st = _entry()(problem, n, m, 50, cur, best, *(x.data_ptr() for x in d), out.data_ptr(),
                  torch.cuda.current_stream().cuda_stream)
    assert st == 0
    assert tuple(out.tolist()) == want
