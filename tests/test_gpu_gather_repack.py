"""Rows of an odd number of words, which are repacked in shared memory: widths at the ends of the form's range, regions
whose last row cannot be covered by whole 16-byte blocks, rows that straddle regions, bad ids, counts off the group."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def words():
    from gpu_util import Words
    return Words()


@pytest.mark.parametrize("D", [39, 41, 75, 127, 255, 257, 499, 501])
@pytest.mark.parametrize("cap_rows,extra,world", [(10 ** 9, 0, 1), (100, 0, 3), (100, 5, 4), (0, 0, 1)])
@pytest.mark.parametrize("n", [1, 3, 97, 2500])
def test_odd_word_rows(words, D, cap_rows, extra, world, n):
    from gpu_util import EmulatedChunks, gather
    rng = np.random.default_rng(D + n)
    rows = 701
    table = rng.integers(0, 2 ** 32, (rows, D), dtype=np.uint32).view(np.float32)
    em = EmulatedChunks(table, D, (min(cap_rows, 10 ** 6) * D + extra) * 4, world)
    idx = np.array(list(rng.integers(0, rows, n)) + [rows - 1, 99, 100, 199, 299][: n - 1], dtype=np.int64)
    out = gather(em.desc, torch.from_numpy(idx).cuda(), D, torch.float32, words)
    assert words.take_status() == 0
    assert out.cpu().numpy().tobytes() == table[idx].tobytes()


def test_bad_ids_and_live_count(pkg, words):
    from gpu_util import gather, plain_desc, vp
    D, rows, n = 75, 300, 1000
    table = torch.randn(rows, D, device="cuda")
    idx = torch.randint(0, rows, (n,), device="cuda", dtype=torch.int32)
    idx[5], idx[77], idx[n - 1] = -1, rows, 1 << 30
    out = gather(plain_desc(table), idx, D, torch.float32, words)
    assert words.take_status() != 0
    good = (idx >= 0) & (idx < rows)
    assert torch.equal(out[good], table[idx[good].long()]) and not out[~good].any()
    # a row count on the device: rows past it stay as they are
    abi = pkg.load_abi()
    idx = idx.clamp(0, rows - 1)
    for live in (0, 1, 2, 3, 501, n, n + 50):
        count = torch.tensor([live], device="cuda")
        out = torch.full((n, D), -7.0, device="cuda")
        d = plain_desc(table)
        pkg.check(abi.dgs_gather_rows_counted(ctypes.byref(d), vp(idx), 0, n, vp(count), D, vp(out), vp(words.status), None))
        assert words.take_status() == 0
        m = min(live, n)
        assert torch.equal(out[:m], table[idx[:m].long()]) and torch.all(out[m:] == -7.0)


@pytest.mark.parametrize("D", [41, 75, 499])
def test_buffers_filled_both_ways_in_turn(words, D):
    # every warp goes through its buffers many times, with rows copied whole, zeroed and copied by words in all of them:
    # a buffer that a lane wrote by ordinary stores is filled by a bulk copy next, and the other way round
    from gpu_util import EmulatedChunks, gather
    rng = np.random.default_rng(D)
    rows, n = 4000, 400_000
    table = rng.integers(0, 2 ** 32, (rows, D), dtype=np.uint32).view(np.float32)
    em = EmulatedChunks(table, D, (500 * D + 7) * 4, 8)
    ends = np.array([p * em.each // D for p in range(1, 8)])
    idx = rng.integers(0, rows, n)
    kind = rng.integers(0, 4, n)
    idx[kind == 1] = -1 - idx[kind == 1]
    idx[kind == 2] = rng.choice(ends, int((kind == 2).sum()))
    out = gather(em.desc, torch.from_numpy(idx).cuda(), D, torch.float32, words).cpu().numpy()
    assert words.take_status() == 6  # DGS_ERR_RANGE
    want = table[np.maximum(idx, 0)]
    want[idx < 0] = 0
    assert out.tobytes() == want.tobytes()


@pytest.mark.parametrize("D,n", [(D, n) for D, group in ((41, 32), (75, 24), (149, 12), (179, 8), (181, 8), (301, 4), (499, 4))
                                 for n in [1, 15, 16, 17, 2499, 2500, 2501] +
                                 [148 * 8 * group * r + x for r in (1, 2) for x in (-1, 0, 1)] + [148 * 4 * group + 1]])
def test_number_of_rows(words, D, n):
    # where the form begins (16 rows, 2 500 of more than 720 bytes) and around whole rounds of groups over 148 SMs
    from gpu_util import gather, plain_desc
    table = torch.randn(5000, D, device="cuda")
    idx = torch.randint(0, 5000, (n,), device="cuda")
    out = gather(plain_desc(table), idx, D, torch.float32, words)
    assert words.take_status() == 0 and torch.equal(out, table[idx])
