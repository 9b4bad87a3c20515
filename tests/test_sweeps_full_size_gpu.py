"""The sweeps at the benchmark configurations' full sizes, against the oracle.

The default pass settles these searches without them; they remain the path of
graphs beyond its shared memory and of the iterations that it leaves, with what
only large instances reach: rows above the staging budget, bitmap rows too
large to stage, many column chunks per row, multi-gigabyte WSwap matrices,
64-bit perturbation draws, hub rows of thousands of entries.
"""
import pytest

import ts_b200 as T
from test_parity_configs_gpu import (STRUCTS, assert_same, c1, c2, c2_graph, c2_perturbed, c3,  # noqa: F401
                                     gpu_run)

pytestmark = pytest.mark.gpu
SWEPT = [(kind, T.PASS_TILE) for kind in STRUCTS] + [("csr-bb", T.PASS_ROWS), ("csr-bitset", T.PASS_ROWS)]


@pytest.mark.parametrize("kind", STRUCTS)
def test_config1_by_the_default_pass(gpu, c1, kind):  # noqa: F811
    wl, ores = c1
    got = gpu_run(T.PROBLEM_MDP, kind, wl, m=wl["m"], iters=10_000, tenure=20)
    assert_same(kind, T.PROBLEM_MDP, wl["n"], got, ores)


@pytest.mark.parametrize("kind,sweep", SWEPT)
def test_config3_swept(gpu, c3, kind, sweep):  # noqa: F811
    wl, ores = c3
    got = gpu_run(T.PROBLEM_MDP, kind, wl, m=wl["m"], iters=500, tenure=100, sweep=sweep)
    assert_same(kind, T.PROBLEM_MDP, wl["n"], got, ores)


@pytest.mark.parametrize("kind,sweep", SWEPT)
def test_config2_swept(gpu, c2, kind, sweep):  # noqa: F811
    wl, ores = c2
    got = gpu_run(T.PROBLEM_MAXBS, kind, wl, m=0, iters=100, tenure=50, sweep=sweep)
    assert_same(kind, T.PROBLEM_MAXBS, wl["n"], got, ores)


@pytest.mark.parametrize("kind,sweep", SWEPT)
def test_config2_swept_past_perturbation_events(gpu, c2_perturbed, kind, sweep):  # noqa: F811
    wl, start, ores = c2_perturbed
    got = gpu_run(T.PROBLEM_MAXBS, kind, wl, m=0, iters=150, tenure=50, piter=50, seed=7, initial=start, sweep=sweep)
    assert_same(kind, T.PROBLEM_MAXBS, wl["n"], got, ores)
