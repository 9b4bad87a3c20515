"""A device context that goes away under the library: a program that resets the
device goes on with new graphs, and closes the old ones at any time."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes
import numpy as np
import ts_b200 as T

cuda = ctypes.CDLL("libcuda.so.1")
rng = np.random.default_rng(1)
n = 700
u, v = rng.integers(0, n, (2, 6000)).astype(np.int32)
w = rng.integers(1, 100, 6000).astype(np.int32)

def search():
    g = T.Graph(n, u, v, w, "hash", drop_self_loops=True)
    s = T.Solver(g, T.PROBLEM_MDP, m=50, max_iter=80, tenure_policy=T.TENURE_FIXED, tenure=5)
    s.init(None)
    s.step(80)
    assert g.lookup(u[:50], v[:50]).all()
    return s.result().best, s, g

best, s, g = search()
old = [(s, g)]
for _ in range(2):
    assert cuda.cuDevicePrimaryCtxReset_v2(0) == 0
    again, s, g = search()
    assert again == best, (again, best)
    old.append((s, g))
for s, g in old:  # of ended contexts and of this one
    s.close()
    g.close()
again, s, g = search()
assert again == best, (again, best)
s.close()
g.close()
print("same", best)
"""


def test_searches_after_a_device_reset(gpu):
    env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "graph-data-structures-local-search_b200"))
    r = subprocess.run([sys.executable, "-c", PROGRAM], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
