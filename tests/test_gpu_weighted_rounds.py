"""Weighted sampling without replacement at the edges of its windows (512 edges) and rounds (eight or four windows), with
windows that have more survivors than room, against keys computed in float64 from the same random numbers."""
import numpy as np
import pytest
import torch

from gpu_util import Words, plain_desc, sample

pytestmark = pytest.mark.gpu

DEGREES = [5, 33, 127, 128, 129, 511, 512, 513, 1024, 1025, 2561, 4096, 4097, 4608, 4609, 8705, 20_000]
M64 = (1 << 64) - 1


def mix64(z):
    z = (z + 0x9E3779B97F4A7C15) & M64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
    return z ^ (z >> 31)


def philox(key, c0, c1, c2, c3):
    """Philox4x32-10 over an array of third counter words."""
    c = [np.full(c2.shape, x, dtype=np.uint64) if np.isscalar(x) else x.astype(np.uint64) for x in (c0, c1, c2, c3)]
    k0, k1, low = key & 0xFFFFFFFF, key >> 32, np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def keys_of(i, w, rng):
    """log(u) / w of the edges of the row at position i."""
    key = mix64(rng[0]) ^ mix64(rng[1] ^ 0xA5A5A5A55A5A5A5A) ^ (0x41524553 << 32)
    e = np.arange(len(w))
    words = philox(key, i & 0xFFFFFFFF, i >> 32, (e // 128) * 32 + e % 32, 0)
    word = np.select([(e // 32) % 4 == j for j in range(4)], words)
    u = ((word >> np.uint64(8)).astype(np.float64) + 1.0) / 16777216.0
    return np.where(w > 0, np.log(u) / np.where(w > 0, w.astype(np.float64), 1.0), -np.inf)


@pytest.mark.parametrize("k", [1, 5, 10, 11, 20, 21, 25, 32])
@pytest.mark.parametrize("kind", ["even", "late"])
def test_rows_against_float64(k, kind):
    rng = np.random.default_rng(k)
    deg = np.array(DEGREES + [0, 700, 20_000, 3, 9000, 600, 40], dtype=np.int64)
    indptr = np.concatenate([[0], np.cumsum(deg)])
    w = (rng.random(indptr[-1]) + 0.05).astype(np.float32)
    if kind == "late":  # heavy stretches behind the first window: windows of 50 to 512 survivors
        for lo, d in zip(indptr[:-1], deg):
            for at, n in ((1000, 60), (1600, 300), (5200, 512), (9000, 40)):
                w[lo + min(at, d):lo + min(at + n, d)] *= 64
    words = Words()
    ip, ix, pr = torch.from_numpy(indptr).cuda(), torch.arange(int(indptr[-1])).cuda(), torch.from_numpy(w).cuda()
    seeds = np.arange(deg.size)
    draws = (17, 3)
    row, col, pos = sample(plain_desc(ip), plain_desc(ix), torch.from_numpy(seeds).cuda(), k, False, words,
                           probs_desc=plain_desc(pr), rng=draws)
    assert words.take_status() == 0
    for i in seeds:
        got = pos[row == i]
        assert np.array_equal(col[row == i], indptr[i] + got)
        if deg[i] <= k:
            assert np.array_equal(got, np.arange(deg[i]))
            continue
        assert got.size == k and np.unique(got).size == k
        wi = w[indptr[i]:indptr[i + 1]]
        key = keys_of(int(i), wi, draws)
        # __logf is off by 2^-21.4 at most on [0.5, 2] (2 ulp elsewhere), __fdividef by 2 ulp
        err = 2.0 ** -21.4 / wi + 1e-6 * np.abs(key)
        bar = np.sort(key)[-k]
        left_out = np.setdiff1d(np.arange(deg[i]), got)
        assert np.all(key[got] + err[got] >= bar) and (key[left_out] - err[left_out]).max() <= (key[got] + err[got]).min()
        assert np.all(np.diff(key[got]) <= err[got][1:] + err[got][:-1])  # best first


@pytest.mark.parametrize("k", [10, 25])
def test_a_row_does_not_depend_on_its_neighbours(k):
    rng = np.random.default_rng(3)
    deg = np.array(DEGREES[7:] + [0], dtype=np.int64)
    indptr = np.concatenate([[0], np.cumsum(deg)])
    w = (rng.random(indptr[-1]) + 0.05).astype(np.float32)
    words = Words()
    ip, ix, pr = torch.from_numpy(indptr).cuda(), torch.arange(int(indptr[-1])).cuda(), torch.from_numpy(w).cuda()
    run = lambda s: sample(plain_desc(ip), plain_desc(ix), torch.from_numpy(s).cuda(), k, False, words,
                           probs_desc=plain_desc(pr), rng=(5, 5))
    seeds = rng.integers(0, deg.size - 1, 24)
    row, col, pos = run(seeds)
    off = np.concatenate([[0], np.cumsum(np.minimum(deg[seeds], k))])
    for j in range(seeds.size):
        alone = np.full(seeds.size, deg.size - 1)
        alone[j] = seeds[j]
        assert np.array_equal(run(alone)[2], pos[off[j]:off[j + 1]])
