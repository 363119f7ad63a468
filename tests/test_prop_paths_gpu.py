"""Propagation through every table form (prepared on chip or not, both axis
orders, single-entry axes, loads below, inside, on and above the load axis)
and every fanout count at which a driver's required time is gathered
another way, against the same arithmetic in 64 bits.

The design: one driver whose net has F sinks, each the input of a cell with
one output, a primary output."""
import numpy as np
import pytest

import opentimer_b200 as otg
from opentimer_b200.prop import TimingGraph

pytestmark = pytest.mark.gpu


def star(F, seed):
    """An RC net with F sinks at various distances from its driver (node 0)."""
    rng = np.random.default_rng(seed)
    n = F + 1
    edges = np.array([(0 if i < 3 else int(rng.integers(0, i)), i) for i in range(1, n)], np.int32)
    return (np.array([0, n], np.int32), edges.reshape(-1, 2), np.zeros(1, np.int32),
            rng.uniform(1e-4, 1e-2, F).astype(np.float32),
            rng.uniform(0.1, 0.4, (n, 4)).astype(np.float32))


def value(i1, i2, tab, x, y):
    """Bilinear in 64 bits, the outer segments extrapolated; (x, y) on (i1, i2)."""
    x, y = np.broadcast_arrays(np.atleast_1d(x), np.atleast_1d(y))
    tab = np.asarray(tab, np.float64)

    def seg(ax, q):  # the segment's ends, and how far along it q is
        ax = np.asarray(ax, np.float64)
        if len(ax) == 1:
            return np.zeros(len(q), int), np.zeros(len(q), int), np.zeros(len(q))
        k = np.clip(np.searchsorted(ax, q), 1, len(ax) - 1)
        return k - 1, k, (q - ax[k - 1]) / (ax[k] - ax[k - 1])
    a0, a1, fa = seg(i1, x)
    b0, b1, fb = seg(i2, y)
    lo = tab[a0, b0] + fa * (tab[a1, b0] - tab[a0, b0])
    hi = tab[a0, b1] + fa * (tab[a1, b1] - tab[a0, b1])
    return lo + fb * (hi - lo)


@pytest.mark.parametrize("F", [1, 4, 5, 33, 128, 129, 600])
@pytest.mark.parametrize("n1,n2,var,where,pad", [
    (7, 7, 0, "inside", 0), (7, 7, 0, "below", 0), (7, 7, 0, "above", 0), (7, 7, 0, "first", 0),
    (8, 2, 0, "last", 0), (2, 8, 0, "inside", 0), (7, 7, 1, "inside", 0), (9, 3, 0, "inside", 0),
    (3, 9, 0, "above", 0), (1, 5, 0, "inside", 0), (5, 1, 0, "inside", 0), (1, 1, 0, "inside", 0),
    (7, 7, 0, "inside", 12000)])
def test_tables_and_fanouts(cuda, F, n1, n2, var, where, pad):
    import torch
    rng = np.random.default_rng(F * 100 + n1 * 10 + n2)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)  # noqa: E731
    b = otg.RcBatch(*[t(a) for a in star(F, F)])
    b.run()
    b.check()
    slot = b.node2bfs.cpu().numpy()
    rc = {k: getattr(b, k).cpu().numpy().astype(np.float64) for k in ("load", "delay", "impulse")}
    load = rc["load"][0]  # per corner
    lo32 = b.load.cpu().numpy()[0]
    # a load axis (shared by the corners; their loads differ by a few percent)
    ln = n1 if var else n2
    step = {"inside": 0.4, "below": 0.1, "above": 0.01, "first": 0.1, "last": 0.3}[where]
    start = {"inside": lo32[0] * 0.5, "below": lo32.max() * 1.5, "above": lo32[0] * 0.1,
             "first": lo32[0], "last": lo32[0] * (1 - step * (ln - 1))}[where]
    lax = (start + lo32[0] * step * np.arange(ln)).astype(np.float32)
    if where == "last":
        lax[-1] = lo32[0]
    sn = n2 if var else n1
    sax = (0.02 + 0.03 * np.arange(sn)).astype(np.float32)
    ax1, ax2 = (lax, sax) if var else (sax, lax)
    tabs = [(rng.uniform(0.02, 0.05, (n1, n2)) + 0.01 * np.arange(n1)[:, None] +
             0.02 * np.arange(n2)).astype(np.float32) for _ in range(4)]
    data = np.concatenate([np.concatenate([ax1, ax2, x.reshape(-1)]) for x in tabs] +
                          [np.zeros(pad, np.float32)])
    size = n1 + n2 + n1 * n2
    P = 1 + 2 * F
    nan4 = lambda: np.full((P, 4), np.nan, np.float32)  # noqa: E731
    pi_at, pi_slew, po_rat = nan4(), nan4(), nan4()
    pi_at[0] = [0.1, 0.2, 0.3, 0.4]
    pi_slew[0] = [0.03, 0.05, 0.06, 0.08]
    po_rat[1 + F:] = rng.uniform(0.5, 1.5, (F, 4)).astype(np.float32)
    s, z = np.arange(1, 1 + F), np.arange(1 + F, P)
    g = TimingGraph({
        "num_pins": P, "arc_from": np.concatenate([np.zeros(F), s]),
        "arc_to": np.concatenate([s, z]), "arc_kind": np.repeat([0, 1], F),
        "arc_timing": np.repeat([[-1, -1], [0, 0]], F, axis=0),
        "arc_net": np.zeros(2 * F), "arc_node": np.concatenate([s, np.full(F, -1)]),
        "test_arc": [], "pi_at": pi_at, "pi_slew": pi_slew, "po_rat": po_rat,
        "timing": [[0, 0, 0, 0, 1, 2, 3, -1, -1]],  # positive unate
        "lut_meta": [(n1, n2, k * size, var) for k in range(4)], "lut_data": data,
        "period": 1.0}, device=cuda)
    got = g.propagate(b).result()
    # [sink][corner], corner = 2 * split + transition; tables by transition
    d, imp = rc["delay"][slot[s]], rc["impulse"][slot[s]]
    slew = np.sqrt(pi_slew[0].astype(np.float64) ** 2 + imp)
    q = (lambda tab, c: value(ax1, ax2, tab, load[c], slew[:, c])) if var else \
        (lambda tab, c: value(ax1, ax2, tab, slew[:, c], load[c]))
    delay = np.stack([np.broadcast_to(q(tabs[c & 1], c), (F,)) for c in range(4)], 1)
    out_slew = np.stack([np.broadcast_to(q(tabs[2 + (c & 1)], c), (F,)) for c in range(4)], 1)
    at_z = pi_at[0].astype(np.float64) + d + delay
    rat_s = po_rat[z].astype(np.float64) - delay
    r0 = rat_s - d
    rat_0 = np.array([r0[:, 0].max(), r0[:, 1].max(), r0[:, 2].min(), r0[:, 3].min()])
    # a few roundings of values up to `scale`, times the extrapolation's reach
    scale = max(1.0, np.abs(at_z).max(), np.abs(delay).max(), np.abs(out_slew).max())
    tol = 1e-5 * scale
    assert np.abs(got["slew"][s] - slew).max() <= tol
    assert np.abs(got["slew"][z] - out_slew).max() <= tol
    assert np.abs(got["at"][z] - at_z).max() <= tol
    assert np.abs(got["rat"][s] - rat_s).max() <= tol
    assert np.abs(got["rat"][0] - rat_0).max() <= tol
    assert np.abs(got["slack"][z][:, 2:] - (po_rat[z] - at_z)[:, 2:]).max() <= tol
