"""Nets of at most 32 nodes (eight to a warp): every size, packings that
fill a warp's slice exactly or overflow it, and the same bits whether the
call sorts its nets into size classes or not."""
import numpy as np
import pytest

import opentimer_b200 as otg
import oracle as O
import rcgen
from helpers import bfs_local, elmore_err

pytestmark = pytest.mark.gpu
OUT = ["node2bfs", "pid", "edges", "load", "delay", "ldelay", "impulse"]


def run(cuda, f, max_net_nodes=None):
    import torch
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)  # noqa: E731
    b = otg.RcBatch(t(f.nodes_start), t(f.edges.copy()), t(f.roots), t(f.res), t(f.cap),
                    max_net_nodes=max_net_nodes)
    b.run()
    b.check()
    return {k: getattr(b, k).cpu().numpy() for k in OUT}


@pytest.mark.parametrize("sizes", [
    [1, 2], [2], [32], [1] * 9 + [2], [32] * 9,  # few nets, single nodes, four to a slice
    [16] * 8, [17] * 8, [32, 32, 32, 31, 1, 1],  # a slice filled exactly, and overflowed
    list(range(1, 33)) * 3,
    [32, 1, 2, 3, 32, 32, 5, 32, 7] * 40,
], ids=lambda s: f"{len(s)}x{s[0]}..{s[-1]}")
@pytest.mark.parametrize("kind", ["rrt", "path", "star", "chain"])
def test_small_nets(cuda, sizes, kind):
    f = rcgen.forest(len(sizes) + sizes[0], sizes, [kind] * len(sizes))
    got = run(cuda, f)
    st, e, n2b, pid, _ = O.bfs(f)
    assert st == 0
    assert np.array_equal(got["node2bfs"], n2b) and np.array_equal(got["pid"], pid)
    assert np.array_equal(got["edges"], e)
    st, ref = O.elmore_cpu_f32(f)
    assert st == 0
    for q, r in zip(["load", "delay", "ldelay", "impulse"], ref):
        assert elmore_err(f.nodes_start, bfs_local(f.nodes_start, n2b, got[q]), r) <= 1.0, q
    # a larger bound sends the same nets through the size classes
    listed = run(cuda, f, max_net_nodes=200)
    for k in OUT:
        assert np.array_equal(got[k], listed[k]), k
