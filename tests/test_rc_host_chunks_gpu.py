"""otg_rc_timing_host on more than one chunk of 2^25 nodes, whose copies
share the ring of pinned slots but not the stream: pageable and pinned inputs
and outputs in every combination, twice in a row, against the device-resident
pass."""
import ctypes

import numpy as np
import pytest

import opentimer_b200 as otg
from opentimer_b200._lib import RcForest, check

pytestmark = pytest.mark.gpu
OUT = {"node2bfs": 1, "pid": 1, "load": 4, "delay": 4, "ldelay": 4, "impulse": 4}


@pytest.fixture(scope="module")
def batch(cuda):
    import torch
    V = (1 << 25) + 600_007
    ns = np.append(np.arange(0, V - 8, 9), V).astype(np.int32)
    dev = otg.synth_forest(5, torch.from_numpy(ns).to(cuda), with_sinks=False)
    dev.pop("driver_slew")
    b = otg.RcBatch(**{k: v.clone() for k, v in dev.items()}).run()
    b.check()
    return dev, b


@pytest.mark.parametrize("pin_out", [False, True], ids=["pageable-out", "pinned-out"])
@pytest.mark.parametrize("pin_in", [False, True], ids=["pageable-in", "pinned-in"])
def test_chunks(cuda, batch, pin_in, pin_out):
    import torch
    dev, b = batch
    N, V = dev["roots"].numel(), dev["cap"].shape[0]
    host = {k: torch.empty(v.shape, dtype=v.dtype, pin_memory=pin_in) for k, v in dev.items()}
    # the edges are both
    host["edges"] = torch.empty(dev["edges"].shape, dtype=torch.int32, pin_memory=pin_out)
    out = {k: torch.empty(V, c, dtype=torch.int32 if c == 1 else torch.float32, pin_memory=pin_out)
           for k, c in OUT.items()}
    for _ in range(2):
        for k, v in dev.items():
            host[k].copy_(v)
        for v in out.values():
            v.zero_()
        p = lambda t: t.data_ptr()  # noqa: E731
        f = RcForest(N, V, p(host["nodes_start"]), p(host["edges"]), p(host["roots"]),
                     p(host["res"]), p(host["cap"]), *[p(out[k]) for k in OUT], None, None, None,
                     None)
        check("otg_rc_timing_host", otg.lib().otg_rc_timing_host(ctypes.byref(f)))
        assert torch.equal(host["edges"].to(cuda), b.edges)
        for k in OUT:
            assert torch.equal(out[k].to(cuda).view(-1), getattr(b, k).view(-1)), k
