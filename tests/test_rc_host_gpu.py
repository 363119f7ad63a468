"""otg_rc_timing_host on pageable and pinned buffers, below and above the size
from which pageable copies go through the pinned ring: the same bits as the
device-resident pass."""
import threading

import numpy as np
import pytest

import opentimer_b200 as otg

pytestmark = pytest.mark.gpu
KEYS = ["nodes_start", "edges", "roots", "res", "cap", "sinks_start", "sink_nodes", "driver_slew"]
OUT = ["node2bfs", "pid", "load", "delay", "ldelay", "impulse", "sink_slew"]


def forest(cuda, nodes, seed, pinned=False):
    """Nets of nine nodes, the last one with what is left of `nodes`."""
    import torch
    ns = np.append(np.arange(0, nodes, 9), nodes).astype(np.int32)
    if ns[-1] - ns[-2] < 2:
        ns = np.delete(ns, -2)
    dev = otg.synth_forest(seed, torch.from_numpy(ns).to(cuda))
    b = otg.RcBatch(**{k: v.clone() for k, v in dev.items()}).run()
    b.check()
    ref = {k: getattr(b, k).cpu().numpy() for k in OUT + ["edges"]}
    host = {k: dev[k].cpu() for k in KEYS}
    if pinned:
        host = {k: v.pin_memory() for k, v in host.items()}
    return {k: v.numpy() for k, v in host.items()}, ref


def check(host, ref):
    out = otg.rc_timing_host(**host)
    for k in OUT:
        assert np.array_equal(out[k], ref[k]), k
    assert np.array_equal(host["edges"], ref["edges"])


# 16 bytes a node: 2^17 nodes fill a slot of the ring, 2^16 end on a slice of
# one; from 2^16 on what comes back is more than the size from which it is used
@pytest.mark.parametrize("nodes", [20, 1 << 14, (1 << 16) - 1, 1 << 16, (1 << 16) + 1,
                                   (1 << 17) - 1, 1 << 17, (1 << 18) + 5, 540_001])
@pytest.mark.parametrize("pinned", [False, True], ids=["pageable", "pinned-in"])
def test_host_pass(cuda, nodes, pinned):
    check(*forest(cuda, nodes, nodes, pinned))


def test_after_release_and_from_threads(cuda):
    jobs = [forest(cuda, 300_000 + 7 * k, k) for k in range(3)]
    otg.lib().otg_release_host_context()
    errors = []

    def work(job):
        try:
            check(*job)
        except BaseException as e:  # noqa: B036 -- reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
