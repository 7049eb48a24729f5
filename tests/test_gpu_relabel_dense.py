"""The relabel operator's choice between one word per id and the hash table (by the largest key, from 2^19 keys on), on both
sides of the line and of the range of key numbers, and for keys that neither form takes, against numpy."""
import numpy as np
import pytest
import torch

from gpu_util import Words, unique_relabel
from test_gpu_relabel_paths import want

pytestmark = pytest.mark.gpu

ERR_RANGE = 6


def slots(n):
    s = 64
    while s < 2 * n:
        s *= 2
    return s


@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, 700_001, (1 << 20) + 5000, (1 << 21) - 1, 1 << 21])
@pytest.mark.parametrize("above", [-1, 0, 1])
@pytest.mark.parametrize("at", ["first", "last"])
def test_largest_key_at_the_line(n, above, at):
    """Keys below 2 * slots words are addressed directly."""
    words = Words()
    rng = np.random.default_rng(n)
    line = 2 * slots(n)
    keys = rng.integers(0, line, n)
    keys[0 if at == "first" else n - 1] = line + above
    ids = np.concatenate([keys[-5000:], keys[:5000], [0, line - 1, line, line + 1, -1, 2 ** 31 - 1], rng.integers(0, line, 50)])
    for dt in (np.int64, np.int32):
        t = torch.from_numpy(keys.astype(dt)).cuda()
        u, lab = unique_relabel([t[:1000], t[1000:]], [torch.from_numpy(ids.astype(dt)).cuda()], words)
        assert words.take_status() == 0
        wu, wl = want(keys, ids)
        assert np.array_equal(u, wu) and np.array_equal(lab, wl)


def test_wide_and_negative_keys():
    words = Words()
    keys = np.tile(np.array([5, 3, -2, 5, (1 << 40) + 5, 3]), 100_000)
    u, lab = unique_relabel([torch.from_numpy(keys).cuda()], [torch.from_numpy(keys).cuda()], words)
    assert words.take_status() == ERR_RANGE
    assert u.tolist() == [5, 3, (1 << 40) + 5] and np.array_equal(lab, np.tile([0, 1, -1, 0, 2, 1], 100_000))
