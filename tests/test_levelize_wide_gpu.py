"""Levelization of pins with very many fanins, at the edges of how their
records are cut: up to 64 fanins four to a record, beyond 32, beyond 512
records more; in both forms; more of them than a CTA's list holds; among many
other pins of the same level; in the seed."""
import numpy as np
import pytest

from test_levelize_paths_gpu import check, csr, form  # noqa: F401 -- form is a fixture

pytestmark = pytest.mark.gpu


def hubs(rng, degs, narrow, pool):
    """Seeds <- a level of pins with `degs` fanins, and `narrow` pins with one
    <- a pool of pins <- one pin each."""
    k = len(degs) + narrow
    deg = np.concatenate([degs, np.ones(narrow, int)]).astype(int)
    hub, mid, last = k + np.arange(k), 2 * k + np.arange(pool), 2 * k + pool + np.arange(pool)
    src = np.concatenate([hub, rng.choice(mid, deg.sum()), last])
    dst = np.concatenate([np.arange(k), np.repeat(hub, deg), mid])
    perm = rng.permutation(2 * k + 2 * pool)
    return len(perm), perm[src], perm[dst]


@pytest.mark.parametrize("deg", [64, 65, 95, 96, 97, 1024, 1025, 16384, 16385, 32769, 100_000])
def test_one_long_pin(cuda, form, deg):  # noqa: F811
    check(cuda, *csr(*hubs(np.random.default_rng(deg), [deg], 3, deg // 2 + 5)))


@pytest.mark.parametrize("degs", [[16384] * 12, [16385, 70, 4, 5, 64, 1025] * 5, [300] * 400],
                         ids=["12x16384", "mixed", "400x300"])
def test_many_long_pins(cuda, form, degs):  # noqa: F811
    check(cuda, *csr(*hubs(np.random.default_rng(2), degs, 30_000, 20_000)))


@pytest.mark.parametrize("deg", [65, 1025, 20_000])
def test_long_pins_in_the_seed(cuda, form, deg):  # noqa: F811
    rng = np.random.default_rng(deg)
    k, pool = 5, 3000
    src = k + rng.integers(0, pool, k * deg)
    perm = rng.permutation(k + pool)
    check(cuda, *csr(k + pool, perm[src], perm[np.repeat(np.arange(k), deg)]))
