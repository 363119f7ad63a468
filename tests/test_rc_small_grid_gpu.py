"""The small-net kernel by the number of nets: one net, four or eight to a
warp, in one go or several, give the same bits."""
import numpy as np
import pytest

import oracle as O
import rcgen
from test_rc_small_gpu import OUT, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hi", [16, 17, 24, 32])
@pytest.mark.parametrize("copies", [1, 21, 30])  # 592 nets are the line on 148 SMs
def test_copies_of_a_forest(cuda, hi, copies):
    sizes = [2 + i % (hi - 1) for i in range(28)]
    f = rcgen.forest(hi, sizes * copies, ["rrt", "path", "star", "chain"] * (7 * copies))
    got = run(cuda, f)
    for a, b in ((0, 28 * (copies // 2) + 5), (28 * copies - 9, 28 * copies)):
        n0, n1 = int(f.nodes_start[a]), int(f.nodes_start[b])
        edges = slice(n0 - a, n1 - b)
        few = run(cuda, O.Forest(f.nodes_start[a:b + 1] - n0, f.edges[edges], f.roots[a:b],
                                 f.res[edges], f.cap[n0:n1]), max_net_nodes=hi)
        for k in OUT:
            assert np.array_equal(got[k][edges if k == "edges" else slice(n0, n1)], few[k]), k
