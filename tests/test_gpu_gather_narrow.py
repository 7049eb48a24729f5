"""Rows whose size is an odd number of 4-byte words but whose elements are 1 or 2 bytes, and their 4- and 8-byte
neighbours: the last row of a region that ends off the 16-byte grid, rows that straddle regions, a host tail, bad ids."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TORCH = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}


@pytest.fixture(scope="module")
def words():
    from gpu_util import Words
    return Words()


# widths in bytes; 8-byte elements have no row of an odd number of words
@pytest.mark.parametrize("row_bytes", [160, 164, 168, 172, 252, 300, 1004, 1996, 2004])
@pytest.mark.parametrize("esz", [1, 2, 4, 8])
# rows per region, bytes by which a region ends inside a row, regions (what does not fit is host memory)
@pytest.mark.parametrize("cap_rows,extra,world", [(2000, 0, 1), (100, 0, 3), (100, 84, 4), (77, 8, 8), (0, 0, 1)])
def test_rows_of_narrow_elements(words, row_bytes, esz, cap_rows, extra, world):
    from gpu_util import EmulatedChunks, gather
    if row_bytes % esz:
        pytest.skip("no such row")
    rng = np.random.default_rng(row_bytes * esz + cap_rows)
    rows = 701
    table = rng.integers(0, 256, (rows, row_bytes), dtype=np.uint8)
    flat = table.view({1: np.uint8, 2: np.int16, 4: np.int32, 8: np.int64}[esz])
    em = EmulatedChunks(flat, row_bytes // esz, cap_rows * row_bytes + extra, world)
    ends = [r for p in range(1, world + 1) for r in (p * em.each * esz // row_bytes - 1, p * em.each * esz // row_bytes)]
    idx = np.concatenate([rng.integers(0, rows, 1500), [rows - 1, 0], [r for r in ends if 0 <= r < rows], np.arange(rows)])
    out = gather(em.desc, torch.from_numpy(idx).cuda(), row_bytes // esz, TORCH[esz], words)
    assert words.take_status() == 0
    assert out.cpu().numpy().tobytes() == table[idx].tobytes()


@pytest.mark.parametrize("row_bytes", [164, 172, 252, 1996])
@pytest.mark.parametrize("esz", [1, 2, 4])
def test_bad_ids_give_zero_rows(words, row_bytes, esz):
    from gpu_util import gather, plain_desc
    rows, n = 301, 900  # 301 rows end off the 16-byte grid
    table = torch.randint(1, 120, (rows, row_bytes // esz), device="cuda").to(TORCH[esz])
    idx = torch.randint(0, rows, (n,), device="cuda")
    idx[torch.tensor([0, 5, 77, n - 1])] = torch.tensor([-1, rows, 1 << 40, rows - 1], device="cuda")
    out = gather(plain_desc(table), idx, row_bytes // esz, TORCH[esz], words)
    assert words.take_status() == 6  # DGS_ERR_RANGE
    good = (idx >= 0) & (idx < rows)
    assert torch.equal(out[good], table[idx[good]]) and not out[~good].any()


@pytest.mark.parametrize("width", [164, 172, 252, 1004])
def test_bool_chunk_tensor(ops, width):
    # through the operator layer: 1 001 rows of an odd number of words end off the 16-byte grid
    table = torch.rand(1001, width) < 0.5
    ct = torch.classes.dgs_classes.ChunkTensor([1001, width], torch.bool, table.numel())
    ct._CAPI_load_from_tensor(table)
    idx = torch.cat([torch.arange(1001), torch.randint(0, 1001, (5000,))])
    assert torch.equal(ct._CAPI_index(idx.cuda()).cpu(), table[idx])
