"""Levelization of graphs with as many levels as two digits of the sort hold,
and more."""
import numpy as np
import pytest

from test_levelize_paths_gpu import check, csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [(1 << 20) + 1, (1 << 20) + 2, (1 << 20) + 300])
def test_two_digits_of_levels(cuda, levels):
    # a chain of that many levels, with side pins at random heights
    rng = np.random.default_rng(levels)
    side = 3000
    n = levels + side
    perm = rng.permutation(n)
    src = np.arange(1, n)  # i -> i - 1; a side pin -> a chain pin
    dst = np.concatenate([np.arange(0, levels - 1), rng.integers(0, levels - 1, side)])
    check(cuda, *csr(n, perm[src], perm[dst]))
