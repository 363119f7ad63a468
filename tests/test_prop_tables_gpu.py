"""Propagation through timing records that lack a table, and through tables
at the edges of the look-up rule (repeated axis entries, entries that are not
finite, axes out of order), against the rule itself in 64 bits.

The design is that of test_prop_paths_gpu.py: one driver whose net has F
sinks, each the input of a cell with one output, a primary output."""
import numpy as np
import pytest

import opentimer_b200 as otg
from opentimer_b200.prop import TimingGraph
from test_prop_paths_gpu import star

pytestmark = pytest.mark.gpu
F = 5
SLEW = np.array([0.03, 0.05, 0.06, 0.08], np.float32)


def graph(cuda, record, tables, pad):
    """tables: per LUT (axis 1, axis 2, values, variable order)."""
    size = lambda t: t[2].size + len(t[0]) + len(t[1])  # noqa: E731
    off = np.cumsum([0] + [size(t) for t in tables])
    data = np.concatenate([np.concatenate([t[0], t[1], t[2].reshape(-1)]) for t in tables] +
                          [np.zeros(pad)]).astype(np.float32)
    P = 1 + 2 * F
    nan4 = lambda: np.full((P, 4), np.nan, np.float32)  # noqa: E731
    pi_at, pi_slew, po_rat = nan4(), nan4(), nan4()
    pi_at[0] = [0.1, 0.2, 0.3, 0.4]
    pi_slew[0] = SLEW
    po_rat[1 + F:] = 1.0
    s, z = np.arange(1, 1 + F), np.arange(1 + F, P)
    return TimingGraph({
        "num_pins": P, "arc_from": np.concatenate([np.zeros(F), s]),
        "arc_to": np.concatenate([s, z]), "arc_kind": np.repeat([0, 1], F),
        "arc_timing": np.repeat([[-1, -1], [0, 0]], F, axis=0),
        "arc_net": np.zeros(2 * F), "arc_node": np.concatenate([s, np.full(F, -1)]),
        "test_arc": [], "pi_at": pi_at, "pi_slew": pi_slew, "po_rat": po_rat,
        "timing": [record],
        "lut_meta": [(len(t[0]), len(t[1]), o, t[3]) for t, o in zip(tables, off)],
        "lut_data": data, "period": 1.0}, device=cuda)


def lower_bound(ax, q):
    lo, hi = 0, len(ax)
    while lo < hi:
        mid = (lo + hi) >> 1
        if ax[mid] < q:
            lo = mid + 1
        else:
            hi = mid
    return lo


def line(q, x1, x2, y1, y2):
    if q == x1:
        return y1
    if q == x2:
        return y2
    slope = np.float64(y2 - y1) / np.float64(x2 - x1)
    return y1 - (x1 - q) * slope if q < x1 else y1 + (q - x1) * slope


def lookup(table, slew, load):
    """Lut::operator() on float32 queries, in 64 bits."""
    if table is None:
        return np.nan
    i1, i2, tab, var = table
    i1, i2, tab = i1.astype(np.float64), i2.astype(np.float64), tab.astype(np.float64)
    v1, v2 = (np.float64(slew), np.float64(load))[::1 if var == 0 else -1]
    a = max(1, min(lower_bound(i1, v1), len(i1) - 1))
    b = max(1, min(lower_bound(i2, v2), len(i2) - 1))
    lo = line(v1, i1[a - 1], i1[a], tab[a - 1, b - 1], tab[a, b - 1])
    hi = line(v1, i1[a - 1], i1[a], tab[a - 1, b], tab[a, b])
    return line(v2, i2[b - 1], i2[b], lo, hi)


def net(cuda):
    import torch
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)  # noqa: E731
    b = otg.RcBatch(*[t(a) for a in star(F, F)])
    b.run()
    b.check()
    return b


def expect_and_check(g, b, record, tables):
    got = g.propagate(b).result()
    s, z = np.arange(1, 1 + F), np.arange(1 + F, 1 + 2 * F)
    load = b.load.cpu().numpy()[0]
    slew, at = got["slew"][s], got["at"][s].astype(np.float64)
    pick = lambda k: tables[record[k]] if record[k] >= 0 else None  # noqa: E731
    with np.errstate(all="ignore"):
        d = np.array([[lookup(pick(3 + (c & 1)), slew[i, c], load[c]) for c in range(4)]
                      for i in range(F)])
        so = np.array([[lookup(pick(5 + (c & 1)), slew[i, c], load[c]) for c in range(4)]
                       for i in range(F)])
        want = {"slew": so, "at": at + d}
        rat = 1.0 - d
    for k, w in want.items():
        # a few roundings of values of the finite ones' size
        fin = np.isfinite(w)
        tol = 1e-5 * max(1.0, np.abs(w[fin]).max(initial=0.0))
        x = got[k][z]
        assert np.array_equal(np.isnan(x), np.isnan(w)), (k, x, w)
        assert np.array_equal(x[~fin & ~np.isnan(w)], w[~fin & ~np.isnan(w)]), (k, x, w)
        assert np.abs(x[fin] - w[fin]).max(initial=0.0) <= tol, (k, x, w)
    x = got["rat"][s]
    fin = np.isfinite(rat)
    assert np.array_equal(np.isnan(x), np.isnan(rat))
    assert np.abs(x[fin] - rat[fin]).max(initial=0.0) <= 1e-5 * max(
        1.0, np.abs(rat[fin]).max(initial=0.0))
    return got


def table(rng, sax, lax, var):
    i1, i2 = (sax, lax) if var == 0 else (lax, sax)
    v = rng.uniform(0.02, 0.05, (len(i1), len(i2))) + 0.01 * np.arange(len(i1))[:, None]
    return (np.asarray(i1, np.float32), np.asarray(i2, np.float32), v.astype(np.float32), var)


# LUT ids of cell_rise, cell_fall, rise_transition, fall_transition
@pytest.mark.parametrize("luts", [(0, 1, -1, -1), (0, 1, -1, 3), (0, 1, 2, -1), (-1, -1, 2, 3),
                                  (-1, 1, 2, 3), (0, -1, -1, 3), (-1, -1, -1, -1)])
@pytest.mark.parametrize("var", [0, 1])
@pytest.mark.parametrize("pad", [0, 12000], ids=["staged", "global"])
def test_missing_tables(cuda, luts, var, pad):
    rng = np.random.default_rng(7)
    b = net(cuda)
    lo = b.load.cpu().numpy()[0, 0]
    tables = [table(rng, 0.02 + 0.03 * np.arange(7), lo * (0.5 + 0.4 * np.arange(7)), var)
              for _ in range(4)]
    record = [0, 0, 0, *luts, -1, -1]
    expect_and_check(graph(cuda, record, tables, pad), b, record, tables)


@pytest.mark.parametrize("axis", ["slew", "load"])
@pytest.mark.parametrize("form", ["repeated first", "all repeated", "repeated, query above",
                                  "repeated, query below", "descending", "nan inside",
                                  "infinite beside", "infinite around"])
@pytest.mark.parametrize("pad", [0, 12000], ids=["staged", "global"])
def test_lookup_edges(cuda, axis, form, pad):
    rng = np.random.default_rng(3)
    b = net(cuda)
    load = b.load.cpu().numpy()[0]
    plain = [table(rng, 0.02 + 0.03 * np.arange(4), load[0] * (0.5 + 0.4 * np.arange(5)), 0)] * 4
    record = [0, 0, 0, 0, 1, 2, 3, -1, -1]
    # the first sink's own slew (as the device rounds it) and the net's load
    q = graph(cuda, record, plain, pad).propagate(b).result()["slew"][1, 2] \
        if axis == "slew" else load[2]
    ax = {"repeated first": [q, q, 2 * q, 3 * q], "all repeated": [q, q],
          "repeated, query above": [0.5 * q, 0.5 * q], "repeated, query below": [2 * q, 2 * q, 3 * q],
          "descending": [3 * q, 2 * q, 1.5 * q, 0.7 * q, 0.5 * q],
          "nan inside": [0.1 * q, 0.2 * q, np.nan, 0.4 * q, 0.5 * q, 0.9 * q, 2 * q],
          "infinite beside": [q, 2 * q, 4 * q],
          "infinite around": [0.2 * q, 1.1 * q, 2 * q]}[form]
    other = load[0] * (0.5 + 0.4 * np.arange(5)) if axis == "slew" else 0.02 + 0.03 * np.arange(5)
    sax, lax = (ax, other) if axis == "slew" else (other, ax)
    tables = [table(rng, sax, lax, k & 1) for k in range(4)]
    if form.startswith("infinite"):
        for t in tables:  # at entry 1 of the axis in question
            along = t[2] if (axis == "slew") == (t[3] == 0) else t[2].T
            along[1] = np.inf
    expect_and_check(graph(cuda, record, tables, pad), b, record, tables)
