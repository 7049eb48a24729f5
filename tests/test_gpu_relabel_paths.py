"""The one-word table with keys beyond 32 bits and the numbering pass at the edges of its tiles (1024 keys) and of its
look-back window (256 tiles), against the oracle."""
import numpy as np
import pytest
import torch

from gpu_util import Words, unique_relabel

pytestmark = pytest.mark.gpu


@pytest.fixture
def words():
    return Words()


def want(keys, ids):
    """First-occurrence unique of keys, and the label of every id (-1 when absent)."""
    u, first, inverse = np.unique(keys, return_index=True, return_inverse=True)
    order = np.argsort(first, kind="stable")
    label = np.empty(u.size, dtype=np.int64)
    label[order] = np.arange(u.size)
    at = np.searchsorted(u, ids)
    at_ok = np.minimum(at, max(u.size - 1, 0))
    hit = (u[at_ok] == ids) if u.size else np.zeros(ids.size, bool)
    return u[order], np.where(hit, label[at_ok], -1)


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 4096, 256 * 1024, 257 * 1024 + 3, 1_100_001])
@pytest.mark.parametrize("spread", ["dense", "sparse"])
def test_numbering_at_tile_edges(words, n, spread):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, max(1, n // 3) if spread == "dense" else 1 << 31, n)
    ids = np.concatenate([keys[: n // 2 + 1], rng.integers(0, 1 << 31, 100)])
    for dt in (np.int64, np.int32):
        t = torch.from_numpy(keys.astype(dt)).cuda()
        u, lab = unique_relabel([t[: n // 2], t[n // 2:]], [torch.from_numpy(ids.astype(dt)).cuda()], words)
        assert words.take_status() == 0
        wu, wl = want(keys, ids)
        assert np.array_equal(u, wu) and np.array_equal(lab, wl)


def test_keys_that_share_their_low_32_bits(words):
    # 2^32 - 1 (all low bits set), multiples of 2^32 above one low half, the largest id, each beside its low half
    rng = np.random.default_rng(5)
    low = rng.integers(0, 1 << 32, 300)
    low[:4] = [0, 1, (1 << 32) - 1, (1 << 32) - 2]
    high = np.concatenate([[0, 1, 2, (1 << 31) - 1], rng.integers(0, 1 << 31, 20)])
    grid = (low[:, None] + (high[None, :] << 32)).reshape(-1)
    keys = np.concatenate([rng.permutation(grid), rng.choice(grid, 5000)]).astype(np.int64)
    absent = (rng.integers(0, 1 << 30, 3000) << 32) + rng.choice(low, 3000)
    ids = np.concatenate([rng.permutation(grid), absent, np.array([-1, -(1 << 40)])]).astype(np.int64)
    u, lab = unique_relabel([torch.from_numpy(keys).cuda()], [torch.from_numpy(ids).cuda()], words)
    assert words.take_status() == 0
    wu, wl = want(keys, ids)
    assert np.array_equal(u, wu) and np.array_equal(lab, wl)
