"""Levelization where its lists and its sort change form: pins with more
fanins than a record, than a wide record, and parallel arcs; as many levels
as the sort's first digit holds, one more and one fewer; in both forms."""
import numpy as np
import pytest

import opentimer_b200 as otg
import oracle as O

pytestmark = pytest.mark.gpu


def check(cuda, fs, fi, od, f0):
    import torch
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.int32)).to(cuda)  # noqa: E731
    order, ends, level = otg.levelize(t(fs), t(fi), t(od), t(f0))
    o_order, o_ends, o_level = O.levelize(len(od), fs, fi, od, f0)
    assert np.array_equal(ends, o_ends)
    assert np.array_equal(order, o_order)
    assert np.array_equal(level, o_level)


def csr(n, src, dst):
    """Fanin CSR, fanout counts and seed of arcs src -> dst."""
    by = np.argsort(dst, kind="stable")
    fs = np.zeros(n + 1, np.int32)
    fs[1:] = np.cumsum(np.bincount(dst, minlength=n))
    od = np.bincount(src, minlength=n).astype(np.int32)
    return fs, src[by].astype(np.int32), od, np.nonzero(od == 0)[0].astype(np.int32)


@pytest.fixture(params=["0", "16", "1"], ids=["grid", "cluster16", "cluster1"])
def form(request, monkeypatch):
    monkeypatch.setenv("OTG_LEVELIZE_CLUSTER", request.param)


@pytest.mark.parametrize("deg", [3, 4, 5, 8, 63, 64, 65, 300])
def test_fanin_counts(cuda, form, deg):
    # eight layers of 500 pins; every pin has `deg` fanins in the layer before,
    # drawn with repeats (parallel arcs)
    rng = np.random.default_rng(deg)
    w, layers = 500, 8
    perm = rng.permutation(w * layers)
    dst = np.repeat(np.arange(w, w * layers), deg)
    src = (dst // w - 1) * w + rng.integers(0, w, len(dst))
    check(cuda, *csr(w * layers, perm[src], perm[dst]))


@pytest.mark.parametrize("levels", [1, 2, 1024, 1025, 1026, 2100])
def test_level_counts(cuda, form, levels):
    # a chain of that many levels, with side pins at random heights
    rng = np.random.default_rng(levels)
    side = 3 * levels + 50
    n = levels + side
    perm = rng.permutation(n)
    src = [np.arange(1, levels), np.arange(levels, n)]  # i -> i - 1; a side pin -> a chain pin
    dst = [np.arange(0, levels - 1), rng.integers(0, levels, side)]
    keep = src[1] >= levels + (5 if levels == 1 else 0)
    src, dst = np.concatenate([src[0], src[1][keep]]), np.concatenate([dst[0], dst[1][keep]])
    if levels == 1:
        src, dst = src[:0], dst[:0]
    fs, fi, od, f0 = csr(n, perm[src], perm[dst])
    check(cuda, fs, np.append(fi, 0)[:max(len(fi), 1)] if len(fi) == 0 else fi, od, f0)
