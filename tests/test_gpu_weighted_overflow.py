"""Weighted sampling without replacement where the windows of a row keep more edges than there is room for, or nearly all
weights are zero: the picks, equal keys among them, and that such a row is still shared by the warps of its CTA."""
import numpy as np
import pytest
import torch

from gpu_util import Words, plain_desc, sample
from test_gpu_weighted_rounds import keys_of

pytestmark = pytest.mark.gpu

# one window, a few, and rows whose later rounds take stretches of two to sixteen windows
DEGREES = [40, 129, 300, 512, 513, 2600, 9000, 20_000, 70_001, 140_000]


def kinds(rng, d):
    """Weights of a row of d edges by name."""
    even, t = rng.random(d) + 0.05, np.arange(d)
    out = {"even": even, "few": even * (rng.random(d) < 0.01), "none": even * 0, "one": np.where(t == d - 1, 1.0, 0.0),
           "late": even * np.where((t >= 1600) & (t < 1950), 1000, 1), "last window": even * np.where(t >= d - 400, 1e6, 1),
           "rising": even * np.exp2(60 * t / d), "negative": even * np.where(rng.random(d) < 0.01, 1, -1)}
    return {name: w.astype(np.float32) for name, w in out.items()}


@pytest.mark.parametrize("k", [3, 10, 16, 17, 20, 21, 32])
def test_rows_whose_windows_have_no_room(k):
    rng = np.random.default_rng(k)
    rows = [w for d in DEGREES for w in kinds(rng, d).values()]
    order = rng.permutation(len(rows))
    deg = np.array([w.size for w in rows])
    indptr, w = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64), np.concatenate(rows)
    words, draws = Words(), (17, 3)
    ip, ix, pr = torch.from_numpy(indptr).cuda(), torch.arange(int(indptr[-1])).cuda(), torch.from_numpy(w).cuda()
    row, col, pos = sample(plain_desc(ip), plain_desc(ix), torch.from_numpy(order).cuda(), k, False, words,
                           probs_desc=plain_desc(pr), rng=draws)
    assert words.take_status() == 0 and np.array_equal(row, np.repeat(order, k)) and np.array_equal(col, indptr[row] + pos)
    for i, s in enumerate(order):
        got, wi = pos[i * k:(i + 1) * k], rows[s]
        assert np.unique(got).size == k
        key = keys_of(i, wi, draws)
        n_pos = min(k, int((wi > 0).sum()))
        assert np.all(wi[got[:n_pos]] > 0)
        # weights <= 0 share one key: the row's first of them, in order
        assert np.array_equal(got[n_pos:], np.flatnonzero(~(wi > 0))[:k - n_pos])
        if n_pos == 0:
            continue
        # __logf is off by 2^-21.4 at most on [0.5, 2] (2 ulp elsewhere), __fdividef by 2 ulp
        with np.errstate(divide="ignore", invalid="ignore"):
            err = np.where(wi > 0, 2.0 ** -21.4 / wi + 1e-6 * np.abs(key), 0.0)
        at = got[:n_pos]
        assert np.all(np.diff(key[at]) <= err[at][1:] + err[at][:-1])  # best first
        left_out = np.setdiff1d(np.flatnonzero(wi > 0), at)
        if left_out.size:
            assert (key[left_out] - err[left_out]).max() <= (key[at] + err[at]).min()


@pytest.mark.parametrize("k", [1, 10, 20, 32])
def test_equal_keys_keep_their_order(k):
    """Infinite weights have one key.  Windows (512 edges) belong to eight shares in turn; of equal keys the lower share wins,
    then the earlier edge."""
    d, words = 70_001, Words()
    w = np.ones(d, dtype=np.float32)
    rng = np.random.default_rng(k)
    at = np.sort(rng.permutation(np.arange(3 * 512, d))[:20_000])
    w[at] = np.inf
    ip, ix, pr = torch.tensor([0, d]).cuda(), torch.arange(d).cuda(), torch.from_numpy(w).cuda()
    pos = sample(plain_desc(ip), plain_desc(ix), torch.zeros(1, dtype=torch.int64).cuda(), k, False, words,
                 probs_desc=plain_desc(pr))[2]
    assert words.take_status() == 0
    assert np.array_equal(pos, at[np.argsort((at // 512) % 8, kind="stable")][:k])


def time_of(indptr, w, k):
    ops, n = torch.ops.dgs_ops, indptr.numel() - 1
    ix, seeds = torch.zeros(w.numel(), dtype=torch.int64, device="cuda"), torch.arange(n, device="cuda")
    best = float("inf")
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(5):
            ops._CAPI_sample_neighbors_with_probs(seeds, indptr, ix, w, k, False)
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


def test_no_row_is_left_to_one_warp(ops):
    """One warp instead of eight took 6 to 12 times as long as the row of even weights."""
    d = 100_000
    ip, t = torch.tensor([0, d]).cuda(), torch.arange(d, device="cuda")
    even = torch.rand(d, device="cuda") + 0.05
    base = time_of(ip, even, 10)
    for w in (even * 0, even * (torch.rand(d, device="cuda") < 0.01), even * torch.where((t >= 1600) & (t < 1950), 1000.0, 1.0)):
        assert time_of(ip, w, 10) < 4 * base


def test_the_fan_outs_where_two_forms_meet_take_alike(ops):
    """A first window that was given up took fan-out 20 to 1.6 times the time of fan-out 21."""
    n, d = 4000, 1500
    ip, w = torch.arange(n + 1, device="cuda") * d, torch.rand(n * d, device="cuda") + 0.05
    assert time_of(ip, w, 20) < 1.3 * time_of(ip, w, 21)
