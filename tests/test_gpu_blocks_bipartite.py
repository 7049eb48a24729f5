"""sample_blocks through the operators on a CSC whose column ids go beyond its rows: the results, and what one hop costs."""
import numpy as np
import pytest
import torch

from test_gpu_blocks_dense import Request, graph, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("idt", [torch.int64, torch.int32])
@pytest.mark.parametrize("weighted", [False, True])
def test_the_last_hop_may_draw_ids_beyond_the_rows(pkg, ops, idt, weighted):
    """Rows 0 to 999 point at rows 1000 to 1999, those at ids from 2000 to 59 999, which have no rows."""
    rng = np.random.default_rng(5)
    indptr = np.arange(2001, dtype=np.int64) * 12
    indices = np.concatenate([rng.integers(1000, 2000, 12_000), rng.integers(2000, 60_000, 12_000)])
    probs = (rng.random(24_000) + 0.05).astype(np.float32) if weighted else None
    seeds = rng.permutation(1000)[:40]
    plain = Request(pkg, indptr, indices, seeds, [5, 4], idt, probs=probs).run(rng=(77, 0))
    assert plain[0] == 0 and plain[2][1][2].max().item() >= 2000 > plain[2][0][2].max().item()
    ip, ix, sd = to_dev(indptr, idt), to_dev(indices, idt), to_dev(seeds, idt)
    pr = torch.from_numpy(probs).cuda() if weighted else None
    for _ in range(2):
        torch.manual_seed(77)
        f, blocks, _ = pkg.sample_blocks(sd, [5, 4], ip, ix, probs=pr, fused=True)
        assert torch.equal(f, plain[2][1][2])
        for h in range(2):
            assert torch.equal(blocks[1 - h][0], plain[2][h][0]) and torch.equal(blocks[1 - h][1], plain[2][h][1])


def test_one_hop_costs_the_same_whatever_the_column_ids_are(pkg, ops):
    """Queued twice, the batch took 1.6 times as long as one whose ids are rows."""
    rng = np.random.default_rng(6)
    indptr, indices = graph(rng, 300_000, 30)
    ip, sd = to_dev(indptr), to_dev(rng.permutation(300_000)[:1024])

    def time_of(columns):
        ix, best = to_dev(columns), float("inf")
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                pkg.sample_blocks(sd, [10], ip, ix, fused=True)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    assert time_of(indices * 4) < 1.3 * time_of(indices)
