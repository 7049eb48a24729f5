"""Weighted sampling at the sizes where its paths meet: rows around 32, 128, 512 edges (one list, windows), 4096
(eight windows; one warp per row with replacement) and above, against the draws recomputed on the host."""
import numpy as np
import pytest
import torch

from gpu_util import Words, plain_desc, sample

pytestmark = pytest.mark.gpu

DEGREES = [1, 5, 31, 32, 33, 127, 128, 129, 511, 512, 513, 1023, 1025, 4095, 4096, 4097, 8193, 40001]


@pytest.fixture
def words():
    return Words()


def mix64(z):
    m = (1 << 64) - 1
    z = (z + 0x9E3779B97F4A7C15) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def philox(key, c0, c1, c2, c3):
    """Philox4x32-10 on arrays of counters: four uint32 arrays."""
    c = [np.broadcast_to(np.asarray(x, dtype=np.uint64), np.shape(c2)).copy() for x in (c0, c1, c2, c3)]
    k0, k1, low = key & 0xFFFFFFFF, key >> 32, np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def unit(word):
    return ((word >> np.uint64(8)).astype(np.float64) + 1.0) / 16777216.0


def graph(weights_of):
    """One row per degree, twice over, neighbours numbered; seeds in an order that mixes long and short rows."""
    deg = np.array(DEGREES + DEGREES[::-1], dtype=np.int64)
    indptr = np.concatenate([[0], np.cumsum(deg)])
    w = np.concatenate([weights_of(d, i) for i, d in enumerate(deg)]).astype(np.float32)
    order = np.random.default_rng(3).permutation(deg.size)
    t = [torch.from_numpy(x).cuda() for x in (indptr, np.arange(indptr[-1], dtype=np.int64), w, order.astype(np.int64))]
    return deg, w, indptr, order, t


@pytest.mark.parametrize("k", [1, 10, 17, 32])
@pytest.mark.parametrize("zeros", [False, True])
def test_without_replacement_follows_the_keys(words, k, zeros):
    # weights are 1 (or 0), so a key's order is that of its uniform; __logf is off by 2^-21.4 at most, so two keys can
    # change places only when their uniforms are closer than 2 * 2^-21.4 (7.2e-7 in the logarithm, hence in u <= 1)
    rng = np.random.default_rng(1)
    deg, w, indptr, order, (ip, ix, wt, seeds) = graph(
        lambda d, i: (rng.random(d) < 0.02 if zeros else np.ones(d)))
    key = mix64(7) ^ mix64(5 ^ 0xA5A5A5A55A5A5A5A) ^ (0x41524553 << 32)
    row, col, pos = sample(plain_desc(ip), plain_desc(ix), seeds, k, False, words, probs_desc=plain_desc(wt), rng=(7, 5))
    assert words.take_status() == 0
    at = 0
    for i, s in enumerate(order):
        d = int(deg[s])
        m = min(d, k)
        got, at = pos[at:at + m], at + m
        assert np.all(row[at - m:at] == s) and np.all(col[at - m:at] == indptr[s] + got)
        if d <= k:
            assert np.array_equal(got, np.arange(d))
            continue
        assert np.unique(got).size == k
        e = np.arange(d)
        block = philox(key, i & 0xFFFFFFFF, 0, (e // 128) * 32 + e % 32, np.zeros(d))
        u = unit(np.choose(e % 128 // 32, block))
        ws = w[indptr[s]:indptr[s + 1]]
        positive = int((ws > 0).sum())
        n_pos = min(k, positive)
        assert np.all(ws[got[:n_pos]] > 0) and not np.any(ws[got[n_pos:]] > 0)
        best = np.sort(u[ws > 0])[::-1][:n_pos]
        assert np.all(u[got[:n_pos]] >= best - 8e-7)
        if n_pos < k:  # the rest are zero weights, in scan order (above eight windows: by window modulo eight first)
            zero = e[ws == 0]
            place = zero if d <= 4096 else np.lexsort((zero, zero // 512 % 8))
            assert np.array_equal(got[n_pos:], (zero if d <= 4096 else zero[place])[:k - n_pos])


@pytest.mark.parametrize("k", [1, 10, 33, 70])
def test_with_replacement_follows_the_prefix_sums(words, k):
    # whole-number weights: every sum of them is exact in fp32, so the edge of a draw is known exactly
    rng = np.random.default_rng(2)
    deg, w, indptr, order, (ip, ix, wt, seeds) = graph(
        lambda d, i: np.where(rng.random(d) < 0.6, 0, rng.integers(1, 8, d)) if i % 3 else np.zeros(d) if i % 5 == 0
        else rng.integers(0, 3, d))
    key = mix64(7) ^ mix64(5 ^ 0xA5A5A5A55A5A5A5A)
    row, col, pos = sample(plain_desc(ip), plain_desc(ix), seeds, k, True, words, probs_desc=plain_desc(wt), rng=(7, 5))
    assert words.take_status() == 0
    pos = pos.reshape(-1, k)
    for i, s in enumerate(order):
        d = int(deg[s])
        cdf = np.cumsum(w[indptr[s]:indptr[s + 1]].astype(np.float64))
        u = unit(philox(key, i & 0xFFFFFFFF, 0, np.arange(k), np.full(k, 0x57524550))[0]).astype(np.float32)
        draw = u * np.float32(cdf[-1])
        want = np.minimum(np.searchsorted(cdf, draw.astype(np.float64), side="right"), d - 1)
        assert np.array_equal(pos[i], want), (i, d)


def one_row(words, w, k, offset=5, replace=False):
    """Positions picked from a single row with weights w, twice."""
    n = w.size
    ip, ix = torch.tensor([0, n], device="cuda"), torch.arange(n, device="cuda")
    wt, seeds = torch.from_numpy(w).cuda(), torch.zeros(1, dtype=torch.int64, device="cuda")
    got = [sample(plain_desc(ip), plain_desc(ix), seeds, k, replace, words, probs_desc=plain_desc(wt), rng=(7, offset))[2]
           for _ in range(2)]
    assert words.take_status() == 0 and np.array_equal(got[0], got[1])
    return got[0]


def test_ties_at_a_shared_bar(words):
    # equal keys are taken by share (window modulo eight) and then by place, whichever share found the bar first:
    # here window 2 fills a list early, and window 41 of an earlier share has the same keys
    w = np.zeros(48 * 512, dtype=np.float32)
    w[2 * 512:3 * 512] = w[41 * 512:42 * 512] = 1e-45  # the smallest positive weight: every key is the clamp
    assert np.array_equal(one_row(words, w, 10), 41 * 512 + np.arange(10))
    # a uniform of exactly 1 gives the key +0, infinite weights -0
    w[:] = 0
    w[1862] = 1.0  # its uniform at (7, 123) is 1
    w[41 * 512:42 * 512] = np.inf
    word = philox(mix64(7) ^ mix64(123 ^ 0xA5A5A5A55A5A5A5A) ^ (0x41524553 << 32), 0, 0, np.array([1862 // 128 * 32 + 1862 % 32]),
                  np.zeros(1))[1862 % 128 // 32]
    assert unit(word)[0] == 1.0
    assert np.array_equal(one_row(words, w, 1, offset=123), [41 * 512])


@pytest.mark.parametrize("k", [10, 70])
@pytest.mark.parametrize("spread", [0, 3, 12])
def test_with_replacement_fractional_weights(words, k, spread):
    # an edge lies within the rounding of its draw: sums of a row go through at most 64 roundings (32 edges walked, 5
    # folds of a group or 16 windows of a long one, 10 of the prefixes), each of 2^-24 of the row's total at most
    rng = np.random.default_rng(k + spread)
    deg, w, indptr, order, (ip, ix, wt, seeds) = graph(
        lambda d, i: rng.random(d) * 10.0 ** rng.uniform(-spread, spread, d) * (rng.random(d) < (0.5 if i % 2 else 1)))
    key = mix64(7) ^ mix64(5 ^ 0xA5A5A5A55A5A5A5A)
    row, col, pos = sample(plain_desc(ip), plain_desc(ix), seeds, k, True, words, probs_desc=plain_desc(wt), rng=(7, 5))
    assert words.take_status() == 0
    pos = pos.reshape(-1, k)
    for i, s in enumerate(order):
        ws = w[indptr[s]:indptr[s + 1]].astype(np.float64)
        cdf = np.concatenate([[0], np.cumsum(ws)])
        if cdf[-1] == 0:
            continue
        draw = unit(philox(key, i & 0xFFFFFFFF, 0, np.arange(k), np.full(k, 0x57524550))[0]) * cdf[-1]
        tol = 64 * 2.0 ** -24 * cdf[-1]
        inside = draw < cdf[-1] - tol  # a draw that rounds up to the total is the last edge's, whatever its weight
        assert np.all(cdf[pos[i]] <= draw + tol) and np.all(draw <= cdf[pos[i] + 1] + tol), (i, ws.size)
        assert np.all(ws[pos[i]][inside] > 0)


@pytest.mark.parametrize("k", [1, 10, 32])
@pytest.mark.parametrize("low,high", [(-30, 30), (-3, 3), (20, 30), (-30, -20)])
def test_without_replacement_spread_weights(words, k, low, high):
    # the picks are the k largest of log(u) / w but for what the fp32 key may be off by: __logf 2^-21.4 absolute on
    # [0.5, 2] and 3 ulp elsewhere, __fdividef 2 ulp, the subtraction-free rest nothing
    rng = np.random.default_rng(k)
    deg, w, indptr, order, (ip, ix, wt, seeds) = graph(lambda d, i: 10.0 ** rng.uniform(low, high, d))
    key = mix64(7) ^ mix64(5 ^ 0xA5A5A5A55A5A5A5A) ^ (0x41524553 << 32)
    row, col, pos = sample(plain_desc(ip), plain_desc(ix), seeds, k, False, words, probs_desc=plain_desc(wt), rng=(7, 5))
    assert words.take_status() == 0
    at = 0
    for i, s in enumerate(order):
        d = int(deg[s])
        m = min(d, k)
        got, at = pos[at:at + m], at + m
        if d <= k:
            assert np.array_equal(got, np.arange(d))
            continue
        assert np.unique(got).size == k
        e = np.arange(d)
        log_u = np.log(unit(np.choose(e % 128 // 32, philox(key, i & 0xFFFFFFFF, 0, (e // 128) * 32 + e % 32, np.zeros(d)))))
        ws = w[indptr[s]:indptr[s + 1]].astype(np.float64)
        keys = log_u / ws
        off = 2.0 ** -21.4 * np.maximum(1, -log_u) / ws + 2.0 ** -22 * -keys
        out = np.ones(d, bool)
        out[got] = False
        assert (keys + off)[got].min() >= (keys - off)[out].max()
        ranks = keys[got]  # and they come in the order of their keys
        assert np.all(ranks[:-1] + off[got][:-1] >= ranks[1:] - off[got][1:])


def test_without_replacement_weights_that_are_no_number(words):
    # infinite weights come first (their keys tie: by place), then the positive ones by key, then the rest in scan order;
    # a weight that is no number counts as none, as negative ones do
    for n in (100, 512, 3000):
        w = np.zeros(n, dtype=np.float32)
        w[5::7] = np.nan
        w[6::7] = -1.0
        w[[40, 77, n - 3]] = np.inf
        w[[11, 60, 90]] = [0.5, 2.0, 1e-3]
        got = one_row(words, w, 10)
        assert np.array_equal(got[:3], [40, 77, n - 3]) and set(got[3:6]) == {11, 60, 90}
        rest = np.flatnonzero(~(w > 0))
        assert np.array_equal(got[6:], rest[:4])
    w = np.full(9000, np.nan, dtype=np.float32)  # above eight windows: by window modulo eight, then by place
    w[[8 * 512 + 3, 100]] = np.inf
    assert np.array_equal(one_row(words, w, 5), [100, 8 * 512 + 3, 0, 1, 2])


def test_with_replacement_weights_that_are_no_number(words):
    w = np.ones(5000, dtype=np.float32)
    w[::2] = np.nan
    w[1::4] = -np.inf
    assert np.all(one_row(words, w, 200, replace=True) % 4 == 3)
    w[100] = np.inf  # no draw is below an infinite sum: the last edge
    assert np.all(one_row(words, w, 20, replace=True) == 4999)
    assert np.all(one_row(words, w[:300], 20, replace=True) == 299)
