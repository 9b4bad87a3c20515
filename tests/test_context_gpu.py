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

DECIDE = r"""
import ctypes
import numpy as np
import ts_b200 as T
from test_noalloc_bounds_gpu import every_pair
from test_zz_no_alloc import _csr, _entry

cuda = ctypes.CDLL("libcuda.so.1")
P = ctypes.c_void_p

def on_device(x):
    d = ctypes.c_uint64()
    assert cuda.cuMemAlloc_v2(ctypes.byref(d), ctypes.c_size_t(x.nbytes)) == 0
    assert cuda.cuMemcpyHtoD_v2(d, x.ctypes.data_as(P), ctypes.c_size_t(x.nbytes)) == 0
    return d

def bind():
    c = P()
    assert cuda.cuInit(0) == 0 and cuda.cuDevicePrimaryCtxRetain(ctypes.byref(c), 0) == 0
    assert cuda.cuCtxSetCurrent(c) == 0

bind()
rng = np.random.default_rng(1)
n, m = 2200, 800
u, v = rng.integers(0, n, (2, 9000)).astype(np.int32)
state = (*_csr(n, u, v, rng.integers(1, 100, 9000).astype(np.int32), True), rng.permutation(n).astype(np.int32),
         rng.integers(-300, 301, n), np.where(rng.random(n) < 0.2, 99, 0).astype(np.int32))
want = every_pair(T.PROBLEM_MDP, n, m, 50, 0, 250, *state)
for turn in range(3):
    got = np.zeros(2, np.int64)
    d = [on_device(np.ascontiguousarray(x)) for x in state + (got,)]
    assert _entry()(T.PROBLEM_MDP, n, m, 50, 0, 250, *(x.value for x in d), None) == 0
    assert cuda.cuCtxSynchronize() == 0
    assert cuda.cuMemcpyDtoH_v2(got.ctypes.data_as(P), d[-1], ctypes.c_size_t(16)) == 0
    assert tuple(got.tolist()) == want, (turn, got, want)
    assert cuda.cuDevicePrimaryCtxReset_v2(0) == 0
    bind()
    spare = on_device(np.zeros(16 + 4 * turn, np.int8).repeat(1 << 20))  # the next context's memory lies elsewhere
print("same", want)
"""


@pytest.mark.parametrize("program", [PROGRAM, DECIDE], ids=["searches", "decisions"])
def test_goes_on_after_a_device_reset(gpu, program):
    paths = [ROOT, os.path.join(ROOT, "graph-data-structures-local-search_b200"), os.path.join(ROOT, "tests")]
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(paths))
    r = subprocess.run([sys.executable, "-c", program], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
