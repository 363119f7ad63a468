"""The launch shapes of the one-CTA-per-net classes: a tuning that was set
runs as it says whatever the number of nets, and one warp per net, over its
range of sizes, gives the bits of larger CTAs and the oracle's values."""
import re

import numpy as np
import pytest

import opentimer_b200 as otg
import oracle as O
import rcgen
from helpers import bfs_local, elmore_err
from test_rc_small_gpu import OUT, run

pytestmark = pytest.mark.gpu


@pytest.fixture
def restore_tuning():
    yield
    otg.set_tuning(None)


@pytest.fixture(scope="module")
def many(cuda):
    """Nets of 33..200 nodes, more than 20 per SM: the number from which the
    default table takes one warp per net."""
    import torch
    nets = 20 * torch.cuda.get_device_properties(cuda).multi_processor_count + 100
    return rcgen.forest(3, [33 + i % 168 for i in range(nets)])


def table(bounds, threads):
    return {"class_max": bounds, "class_threads": threads, "class_items": [4] * len(bounds)}


def launched(cuda, f):
    """Threads per CTA of the class kernels that one pass launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)  # noqa: E731
    b = otg.RcBatch(t(f.nodes_start), t(f.edges.copy()), t(f.roots), t(f.res), t(f.cap))
    b.run()
    b.check()
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
        b.run()
        torch.cuda.synchronize()
    names = [e.key for e in p.key_averages()]
    if not any("rc_" in x for x in names):
        pytest.skip("the profiler sees no kernels")
    return [int(m.group(1)) for x in names for m in [re.search(r"rc_block_kernel<(\d+)", x)] if m]


@pytest.mark.parametrize("threads", [32, 64, 128, 1024])
def test_set_tuning_runs_as_it_says(cuda, many, restore_tuning, threads):
    otg.set_tuning(table([200], [threads]))
    assert launched(cuda, many) == [threads]


def test_default_table(cuda, many):
    assert launched(cuda, many) == [32]
    assert otg.get_tuning()["class_threads"][0] == 32


def test_default_table_can_be_set(cuda, restore_tuning):
    t = otg.get_tuning()
    otg.set_tuning(t)
    assert otg.get_tuning() == t


def test_one_warp_by_default(cuda, many, restore_tuning):
    assert launched(cuda, many) == [32]
    one = run(cuda, many)
    otg.set_tuning(table([200], [64]))
    assert launched(cuda, many) == [64]
    two = run(cuda, many)
    for k in OUT:
        assert np.array_equal(one[k], two[k]), k
    st, e, n2b, pid, _ = O.bfs(many)
    assert st == 0
    assert np.array_equal(one["node2bfs"], n2b) and np.array_equal(one["pid"], pid)
    assert np.array_equal(one["edges"], e)
    st, ref = O.elmore_f64(many)
    assert st == 0
    for q, r in zip(["load", "delay", "ldelay", "impulse"], ref):
        assert elmore_err(many.nodes_start, bfs_local(many.nodes_start, n2b, one[q]), r) <= 1.0, q


@pytest.mark.parametrize("sizes", [[33, 63, 64, 65, 129, 160, 161, 199, 200, 201, 1023, 1024, 1025],
                                   [2495, 3071, 4887, 4888]], ids=["small", "large"])
@pytest.mark.parametrize("kind", ["rrt", "path", "star", "chain"])
def test_one_warp_at_every_size(cuda, restore_tuning, sizes, kind):
    f = rcgen.forest(len(sizes), sizes, [kind] * len(sizes))
    ref = run(cuda, f)
    otg.set_tuning(table([4888], [32]))
    got = run(cuda, f)
    for k in OUT:
        assert np.array_equal(got[k], ref[k]), k
