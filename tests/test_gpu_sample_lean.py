"""The lean uniform sampler (one storage region) draws the same edges as the general one (chunked tensors), bit for
bit: rows around k, 2k, 32, 64 edges, the ends of the position bitmap, and beyond it."""
import numpy as np
import pytest
import torch

from gpu_util import EmulatedChunks, Words, plain_desc, sample

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("idt", [np.int64, np.int32])
@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 10, 15, 16, 17, 25, 31, 32])
def test_lean_and_general_draw_the_same(idt, k):
    words = Words()
    rng = np.random.default_rng(k)
    deg = np.concatenate([np.arange(0, 70), [k, k + 1, 2 * k - 1, 2 * k, 2 * k + 1], [511, 512, 513, 2047, 2048, 2049, 4096,
                          8191, 8192, 8193, 16383, 16384, 16385, 40000], rng.integers(0, 300, 400)])
    deg = rng.permutation(deg)
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(idt)
    indices = rng.integers(0, deg.size, indptr[-1]).astype(idt)
    seeds = torch.from_numpy(rng.permutation(np.concatenate([np.arange(deg.size)] * 2)).astype(idt)).cuda()
    ip, ix = torch.from_numpy(indptr).cuda(), torch.from_numpy(indices).cuda()
    chunks = EmulatedChunks(indices, 1, (indices.size // 3 + 1) * indices.itemsize, 3)
    assert chunks.desc.num_parts == 3

    def draw(desc, plan):
        # no picked positions: the lean form is for launches that do not ask for them
        import ctypes
        from gpu_util import pkg, vp
        abi, n = pkg.load_abi(), seeds.numel()
        row = torch.full((n * k,), -7, dtype=seeds.dtype, device="cuda")
        col = row.clone()
        pkg.check(abi.dgs_sample_uniform(ctypes.byref(desc), vp(seeds), int(idt == np.int64), n, k, 0, vp(plan), 5, 9, vp(row),
                                         vp(col), n * k, vp(words.sizes), None, vp(words.status), None))
        assert words.take_status() == 0
        return row.cpu().numpy(), col.cpu().numpy(), int(words.sizes[0])

    import ctypes
    from gpu_util import pkg, vp
    abi, n = pkg.load_abi(), seeds.numel()
    plan = torch.empty(abi.dgs_sample_plan_bytes(n), dtype=torch.uint8, device="cuda")
    d = plain_desc(ip)
    pkg.check(abi.dgs_sample_plan(ctypes.byref(d), vp(seeds), int(idt == np.int64), n, k, 0, vp(plan), None,
                                  vp(words.status), None))
    lean, general = draw(plain_desc(ix), plan), draw(chunks.desc, plan)
    assert lean[2] == general[2] == int(np.minimum(deg, k).sum()) * 2
    assert np.array_equal(lean[0], general[0]) and np.array_equal(lean[1], general[1])
    # and the general one is what it is with positions asked for
    row, col, _ = sample(d, chunks.desc, seeds, k, False, words, rng=(5, 9))
    assert np.array_equal(row, lean[0][:lean[2]]) and np.array_equal(col, lean[1][:lean[2]])


def test_more_than_2_32_outputs():
    # 2^32 outputs and some, of which a small buffer holds the first: cut to 32 bits, the offsets of the last seeds (another
    # node) would lie inside it again
    import ctypes
    from gpu_util import pkg, vp
    words, abi, k, n, cap = Words(), pkg.load_abi(), 32, (1 << 27) + 64, 2048
    ip = torch.tensor([0, 40, 80], dtype=torch.int32, device="cuda")
    ix = torch.arange(80, dtype=torch.int32, device="cuda")
    seeds = torch.zeros(n, dtype=torch.int32, device="cuda")
    seeds[1 << 27:] = 1
    plan = torch.empty(abi.dgs_sample_plan_bytes(n), dtype=torch.uint8, device="cuda")
    row = torch.full((cap,), -7, dtype=torch.int32, device="cuda")
    col = row.clone()
    d, dx = plain_desc(ip), plain_desc(ix)
    pkg.check(abi.dgs_sample_plan(ctypes.byref(d), vp(seeds), 0, n, k, 0, vp(plan), vp(words.sizes), vp(words.status), None))
    # no status word: one atomic for each output that is left out takes minutes
    pkg.check(abi.dgs_sample_uniform(ctypes.byref(dx), vp(seeds), 0, n, k, 0, vp(plan), 5, 9, vp(row), vp(col), cap, None, None,
                                     None, None))
    assert words.take_status() == 0 and int(words.sizes[0]) == n * k
    assert torch.all(row == 0) and torch.all((col >= 0) & (col < 40))


def test_no_capacity_at_all():
    # a capacity of 0 or below: nothing is written, the status says so
    import ctypes
    from gpu_util import pkg, vp
    words, abi, n, k = Words(), pkg.load_abi(), 50, 5
    ip, ix = torch.arange(0, 101 * 9, 9, device="cuda"), torch.arange(900, device="cuda")
    seeds = torch.arange(n, device="cuda")
    plan = torch.empty(abi.dgs_sample_plan_bytes(n), dtype=torch.uint8, device="cuda")
    d, dx = plain_desc(ip), plain_desc(ix)
    pkg.check(abi.dgs_sample_plan(ctypes.byref(d), vp(seeds), 1, n, k, 0, vp(plan), None, vp(words.status), None))
    for cap in (0, -1, -(1 << 40)):
        row = torch.full((n * k,), -7, device="cuda")
        col = row.clone()
        pkg.check(abi.dgs_sample_uniform(ctypes.byref(dx), vp(seeds), 1, n, k, 0, vp(plan), 5, 9, vp(row), vp(col), cap, None,
                                         None, vp(words.status), None))
        assert words.take_status() == 6 and torch.all(row == -7) and torch.all(col == -7)  # DGS_ERR_RANGE
