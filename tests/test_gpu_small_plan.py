"""The plan of a seed list at the sizes where its form changes (one CTA with 1 to 4 seeds per thread, then one CTA per
256 seeds): counts, offsets and total against numpy, with bad seeds and broken row bounds among them."""
import ctypes

import numpy as np
import pytest
import torch

from gpu_util import Words, pkg, plain_desc, vp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("idt", [np.int64, np.int32])
@pytest.mark.parametrize("replace", [0, 1])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 1023, 1024, 1025, 2048, 3000, 4095, 4096, 4097, 9000])
def test_plan_offsets(n, replace, idt):
    words, abi, k = Words(), pkg.load_abi(), 7
    rng = np.random.default_rng(n)
    nodes = 500
    deg = rng.integers(0, 20, nodes)
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(idt)
    seeds = rng.integers(0, nodes, n).astype(idt)
    bad = n > 300
    if bad:
        seeds[[3, n - 1]] = [-1, nodes]
        indptr[41] = indptr[40] - 2  # row 40 ends before it begins, row 41 begins early
    good = (seeds >= 0) & (seeds < nodes)
    at = np.where(good, seeds, 0)
    d = np.where(good, indptr[at + 1].astype(np.int64) - indptr[at], 0)
    broken = d < 0
    if not bad:
        assert good.all() and not broken.any()
    d = np.where(broken, 0, d)
    rb = np.where(good & ~broken, indptr[at], 0)
    cnt = np.where(d > 0, k, 0) if replace else np.minimum(d, k)
    tiles = -(-n // 256)
    plan = torch.full((abi.dgs_sample_plan_bytes(n),), 0x5A, dtype=torch.uint8, device="cuda")
    ip = torch.from_numpy(indptr).cuda()
    desc = plain_desc(ip)
    st = torch.from_numpy(seeds).cuda()
    pkg.check(abi.dgs_sample_plan(ctypes.byref(desc), vp(st), int(idt == np.int64), n, k, replace, vp(plan), vp(words.sizes),
                                  vp(words.status), None))
    assert (words.take_status() != 0) == bad
    got = plan.cpu().numpy().view(np.int64)
    row_begin, degree, local, tile = got[:n], got[n:2 * n], got[2 * n:3 * n], got[3 * n:3 * n + tiles]
    assert np.array_equal(row_begin, rb) and np.array_equal(degree, d)
    assert np.array_equal(local + tile[np.arange(n) // 256], np.cumsum(cnt) - cnt)
    assert int(words.sizes[0]) == cnt.sum() == got[3 * n + tiles]


@pytest.mark.parametrize("idt", [np.int64, np.int32])
@pytest.mark.parametrize("replace", [0, 1])
@pytest.mark.parametrize("n", [2047, 2049])
def test_plan_offsets_at_the_line(n, replace, idt):
    test_plan_offsets(n, replace, idt)
