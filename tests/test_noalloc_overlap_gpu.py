"""ts_best_swap_noalloc after calls that overlapped on the GPU.

All calls share one scratch area.  Overlapping calls race on it (their own
decisions are undefined), but what they leave there must not reach the calls
that follow, one at a time: the launches' tickets count from 0 again.
"""
import numpy as np
import pytest

import ts_b200 as T
from test_noalloc_bounds_gpu import every_pair
from test_zz_no_alloc import _csr, _entry

pytestmark = pytest.mark.gpu


def case(problem, n, deg, seed):
    import torch

    rng = np.random.default_rng([problem, n, seed])
    u, v = rng.integers(0, n, (2, n * deg // 2)).astype(np.int32)
    rowptr, col, w = _csr(n, u, v, rng.integers(1, 1001, len(u)).astype(np.int32), True)
    m = 2 * n // 5 if problem == T.PROBLEM_MDP else n // 2
    sol = rng.permutation(n).astype(np.int32)
    vg = rng.integers(-3000, 3001, n).astype(np.int64)
    tab = np.where(rng.random(n) < 0.2, 99, 0).astype(np.int32)
    host = (rowptr, col, w, sol, vg, tab)
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in host]
    return problem, n, m, dev, every_pair(problem, n, m, 50, 0, 2500, *host)


def call(c, out, stream):
    problem, n, m, dev, _ = c
    assert _entry()(problem, n, m, 50, 0, 2500, *(x.data_ptr() for x in dev), out.data_ptr(), stream.cuda_stream) == 0


@pytest.mark.parametrize("sizes", [(2300, 2300), (2300, 2600), (2300, 300)])
def test_calls_after_overlapping_ones_decide_right(gpu, sizes):
    import torch

    cases = [case(p, n, 12, k) for k, (p, n) in enumerate(zip((T.PROBLEM_MDP, T.PROBLEM_MAXBS), sizes))]
    outs = [torch.zeros(2, dtype=torch.int64, device="cuda") for _ in cases]
    streams = [torch.cuda.Stream() for _ in cases]
    torch.cuda.synchronize()
    for _ in range(20):
        for _ in range(10):  # the two streams' calls overlap
            for c, out, st in zip(cases, outs, streams):
                call(c, out, st)
        torch.cuda.synchronize()
        for c, out, st in zip(cases, outs, streams):  # one at a time
            call(c, out, st)
            torch.cuda.synchronize()
            assert tuple(out.tolist()) == c[4]
