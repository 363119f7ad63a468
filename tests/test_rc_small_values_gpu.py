"""Nets of at most 32 nodes with capacitances and resistances that are not
finite: which of the outputs are finite, infinite or undefined is as the
reference's sums have it."""
import numpy as np
import pytest

import oracle as O
import rcgen
from helpers import bfs_local
from test_rc_small_gpu import run

pytestmark = pytest.mark.gpu


def kind(x):
    return np.where(np.isnan(x), 3, np.where(x == np.inf, 1, np.where(x == -np.inf, 2, 0)))


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("where", ["root cap", "leaf cap", "any cap", "res"])
def test_not_finite(cuda, value, where):
    rng = np.random.default_rng(4)
    f = rcgen.forest(9, [1 + i % 32 for i in range(200)])
    ns = f.nodes_start
    for i in range(0, f.num_nets, 2):  # every other net
        n = ns[i + 1] - ns[i]
        if where == "res":
            if n > 1:
                f.res[ns[i] - i + rng.integers(0, n - 1)] = value
            continue
        v = f.roots[i] if where == "root cap" else rng.integers(0, n)
        if where == "leaf cap" and n > 1:
            e = f.edges[ns[i] - i:ns[i + 1] - i - 1].reshape(-1)
            deg = np.bincount(e, minlength=n)
            deg[f.roots[i]] = 2
            v = np.nonzero(deg == 1)[0][0]
        f.cap[ns[i] + v, rng.integers(0, 4)] = value
    got = run(cuda, f)
    st, ref = O.elmore_cpu_f32(f)
    assert st == 0
    for q, r in zip(["load", "delay", "ldelay", "impulse"], ref):
        x = bfs_local(ns, got["node2bfs"], got[q])
        assert np.array_equal(kind(x), kind(r)), q
