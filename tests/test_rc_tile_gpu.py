"""The one-CTA-per-net classes at the edges of their size ranges and of the
items a thread owns there, and one warp per net against two."""
import numpy as np
import pytest

import opentimer_b200 as otg
import oracle as O
import rcgen
from helpers import bfs_local, elmore_err
from test_rc_small_gpu import OUT, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [33, 95, 96, 97, 160, 161, 199, 200], [201, 320, 321, 419, 420], [421, 640, 641, 899, 900],
    [901, 1231, 1232], [1233, 1536, 1537, 2495, 2496], [2497, 3072, 3073, 4887, 4888, 4889],
], ids=lambda s: f"{s[0]}..{s[-1]}")
@pytest.mark.parametrize("kind", ["rrt", "path", "star", "chain"])
def test_class_edges(cuda, sizes, kind):
    f = rcgen.forest(sizes[0], sizes, [kind] * len(sizes))
    got = run(cuda, f)
    st, e, n2b, pid, _ = O.bfs(f)
    assert st == 0
    assert np.array_equal(got["node2bfs"], n2b) and np.array_equal(got["pid"], pid)
    assert np.array_equal(got["edges"], e)
    # the 64-bit oracle: along a path of 2,500 nodes the 32-bit one's own error
    # reaches the tolerance
    st, ref = O.elmore_f64(f)
    assert st == 0
    for q, r in zip(["load", "delay", "ldelay", "impulse"], ref):
        assert elmore_err(f.nodes_start, bfs_local(f.nodes_start, n2b, got[q]), r) <= 1.0, q


def test_warp_per_net_same_bits(cuda):
    f = rcgen.forest(5, list(range(33, 201)))
    one = run(cuda, f)
    otg.set_tuning({"class_max": [4888], "class_threads": [64], "class_items": [4]})
    try:
        two = run(cuda, f, max_net_nodes=201)
    finally:
        otg.set_tuning(None)
    for k in OUT:
        assert np.array_equal(one[k], two[k]), k


# the class table depends on the number of nets: one for up to 8 an SM, one
# for up to 20, one for more (1,184 and 2,960 nets on 148 SMs)
@pytest.mark.parametrize("nets", [40, 1500, 3100])
def test_class_tables(cuda, nets):
    edges = [33, 64, 128, 129, 256, 257, 512, 513, 1024, 1025, 1232, 1233, 2496, 2497, 4888, 4889]
    sizes = edges + [2 + i % 60 for i in range(nets - len(edges))]
    f = rcgen.forest(nets, sizes)
    got = run(cuda, f)
    st, e, n2b, pid, _ = O.bfs(f)
    assert st == 0
    assert np.array_equal(got["node2bfs"], n2b) and np.array_equal(got["pid"], pid)
    assert np.array_equal(got["edges"], e)
    st, ref = O.elmore_f64(f)
    assert st == 0
    for q, r in zip(["load", "delay", "ldelay", "impulse"], ref):
        assert elmore_err(f.nodes_start, bfs_local(f.nodes_start, n2b, got[q]), r) <= 1.0, q
