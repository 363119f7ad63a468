"""Nets beyond the shared-memory classes, by how many a pass has: clusters of
16 CTAs (few nets), of 8 with one CTA or two on an SM, in one round or two,
and one CTA per net.  The sums are exact, so all give the same bits."""
import numpy as np
import pytest

import oracle as O
import rcgen
from test_rc_small_gpu import OUT, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [4889], [4889, 5000, 16384, 16385], [4889] * 5, [4889, 8000] * 10, [4889, 8001] * 18,
    [4889] * 31, [5001, 4889, 20] * 30,
], ids=lambda s: f"{len(s)}x{s[0]}..{s[-1]}")
def test_by_number_of_nets(cuda, monkeypatch, sizes):
    kinds = [["rrt", "chain", "path", "star"][i % 4] for i in range(len(sizes))]
    f = rcgen.forest(len(sizes), sizes, kinds)
    got = run(cuda, f)
    monkeypatch.setenv("OTG_RC_HUGE_CLUSTER", "1")
    one = run(cuda, f)
    for k in OUT:
        assert np.array_equal(got[k], one[k]), k
    st, e, n2b, pid, _ = O.bfs(f)
    assert st == 0
    assert np.array_equal(got["node2bfs"], n2b) and np.array_equal(got["pid"], pid)
    assert np.array_equal(got["edges"], e)
