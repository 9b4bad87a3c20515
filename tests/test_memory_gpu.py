"""Device memory of graphs: a build that finds too little room for its
temporaries beside all of its arrays.
"""
import numpy as np
import pytest

import ts_b200 as T

pytestmark = pytest.mark.gpu


def edges(n, e, seed):
    rng = np.random.default_rng(seed)
    u, v = rng.integers(0, n, (2, e)).astype(np.int32)
    return u, v, rng.integers(1, 1001, e).astype(np.int32)


@pytest.mark.parametrize("kind,n,e", [("csr", 20_000, 32_000_000), ("csr-bitset", 100_000, 12_000_000),
                                      ("csr-bitset-bb", 100_000, 12_000_000), ("hash", 10_000, 16_000_000)])
def test_graph_that_fits_once_its_temporaries_are_gone(gpu, kind, n, e):
    """The keys to sort take 48 bytes an edge, the rows 16; the reverse index,
    the bitmap and the hash tables come on top.  With room for the temporaries
    and the rows (64 bytes an edge), or for the finished graph, whichever is
    more, and some slack, the graph is built, and answers as one built with
    room to spare does."""
    import torch

    u, v, w = edges(n, e, 7)
    rng = np.random.default_rng(8)
    q = rng.integers(0, e, 20_000)
    qu = np.concatenate([u[q], rng.integers(0, n, 20_000).astype(np.int32)])
    qv = np.concatenate([v[q], rng.integers(0, n, 20_000).astype(np.int32)])
    g = T.Graph(n, u, v, w, kind, drop_self_loops=False)
    want = g.lookup(qu, qv)
    finished = int(g.info().device_bytes)
    g.close()
    need = max(64 * e, finished) + (96 << 20)

    def fill(left):  # all of the device's memory but `left` bytes
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")

    try:
        hold = fill(2 << 20)
        with pytest.raises(T.TsError):  # far too large: what the pool kept unused is given back
            T.Graph(n, *(np.tile(x, 4) for x in (u, v, w)), kind, drop_self_loops=False)
        del hold
        hold = fill(need)
        g = T.Graph(n, u, v, w, kind, drop_self_loops=False)
        np.testing.assert_array_equal(g.lookup(qu, qv), want)
        g.close()
    finally:
        hold = None
        torch.cuda.empty_cache()
