"""Levelization at the ends of its ranges: as many levels as two digits of the
sort hold, and more; so many pins in the seed that their fanins' numbers take
more than 31 bits."""
import numpy as np
import pytest

import opentimer_b200 as otg
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


@pytest.mark.parametrize("seeds", [(1 << 29) - 100, (1 << 29) + 32])
def test_half_a_billion_seeds(cuda, seeds):
    # the last 40 pins of the seed have one fanin each, the pins behind the seed
    import torch
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("60 GB of device memory")
    k = 40
    n = seeds + k
    i32 = dict(dtype=torch.int32, device=cuda)
    start = torch.zeros(n + 1, **i32)
    start[seeds - k + 1:] = k
    start[seeds - k:seeds + 1] = torch.arange(k + 1, **i32)
    fanin = torch.arange(seeds, n, **i32)
    deg = torch.zeros(n, **i32)
    deg[seeds:] = 1
    b = otg.LevelizeBatch(start, fanin, deg, torch.arange(seeds, **i32)).run()
    b.check()
    assert b.counts.tolist() == [2, n]
    assert b.level_ends[:3].tolist() == [0, seeds, n]
    assert torch.equal(b.order[:n], torch.arange(n, **i32))
    assert torch.equal(b.level[:n], deg)
