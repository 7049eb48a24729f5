"""sample_blocks and PipelinedSampler on a graph of more nodes than the form with one word per id takes: several hops
through the hash tables, as the operators and the pipeline (recordings, the gather behind a batch) queue them."""
import numpy as np
import pytest
import torch

from test_gpu_blocks import check_hops, to_dev
from test_gpu_pipeline import chunked

pytestmark = pytest.mark.gpu

NODES = (1 << 23) + 1


def graph(rng, rows, max_deg):
    """A CSC over NODES ids of which `rows`, the first and the last among them, have neighbours, all within these."""
    ids = np.unique(np.concatenate([[0, NODES - 1], rng.integers(0, NODES, rows)]))
    deg = np.zeros(NODES, dtype=np.int64)
    deg[ids] = rng.integers(1, max_deg, ids.size)
    indptr = np.concatenate([[0], np.cumsum(deg)])
    return ids, indptr, ids[rng.integers(0, ids.size, int(indptr[-1]))]


def hash_tables_are_used(pkg, fanouts, n):
    import ctypes
    abi, H = pkg.load_abi(), len(fanouts)
    hops = (pkg.Hop * H)()
    pkg.check(abi.dgs_sample_blocks_bounds(n, (ctypes.c_int64 * H)(*reversed(fanouts)), H, NODES, hops))
    return abi.dgs_sample_blocks_dense_wins(hops, H, NODES) == 0


@pytest.mark.parametrize("idt", [torch.int64, torch.int32])
@pytest.mark.parametrize("weighted", [False, True])
def test_operators_and_pipeline_equal_the_oracle(ops, oracle, pkg, idt, weighted):
    rng = np.random.default_rng(51)
    ids, indptr, indices = graph(rng, 6000, 6)              # no row is longer than a fan-out: one possible answer
    probs = (rng.random(indices.size) + 0.05).astype(np.float32)
    feats = rng.integers(-2 ** 31, 2 ** 31, (NODES, 2)).astype(np.int32)
    fanouts, npdt = [6, 7, 5], np.int64 if idt == torch.int64 else np.int32
    assert hash_tables_are_used(pkg, fanouts, 200)
    c_ip, c_ix, c_ft = chunked(indptr.astype(npdt)), chunked(indices.astype(npdt), 0.6), chunked(feats, 0.7)
    c_pr = chunked(probs, 0.6) if weighted else None
    batches = [np.concatenate([[NODES - 1, 0], rng.permutation(ids)[:n]]) for n in (150, 150, 150, 31, 150)]
    want = [oracle.sample_blocks(indptr, indices, s, fanouts) for s in batches]

    def same(f, blocks, ne, of, ob, oe):
        assert ne == oe and f.dtype == idt and np.array_equal(f.cpu().numpy(), of)
        for (r, c, ns, nd), (orow, ocol, ons, ond) in zip(blocks, ob):
            assert (ns, nd) == (ons, ond) and np.array_equal(r.cpu().numpy(), orow) and np.array_equal(c.cpu().numpy(), ocol)

    for s, w in zip(batches, want):
        same(*pkg.sample_blocks(to_dev(s, idt), fanouts, c_ip, c_ix, probs=c_pr, fused=True), *w)
    sampler = pkg.PipelinedSampler(c_ip, c_ix, fanouts, probs=c_pr, features=c_ft, max_seeds=152, depth=2)
    for (f, blocks, ne, x), w in zip(sampler(to_dev(s, idt) for s in batches), want):
        same(f, blocks, ne, *w)
        assert x.cpu().numpy().tobytes() == feats[w[0]].tobytes()
    del sampler


@pytest.mark.parametrize("weighted,replace", [(False, False), (True, False), (False, True), (True, True)])
def test_replayed_batches_equal_the_operator(ops, oracle, pkg, weighted, replace):
    rng = np.random.default_rng(52)
    ids, indptr, indices = graph(rng, 9000, 50)
    probs = (rng.random(indices.size) + 0.05).astype(np.float32)
    feats = rng.integers(-2 ** 31, 2 ** 31, (NODES, 1)).astype(np.int32)
    c_ip, c_ix, c_ft = chunked(indptr), chunked(indices, 0.8), chunked(feats)
    c_pr = chunked(probs, 0.8) if weighted else None
    fanouts = [10, 10, 5]
    assert hash_tables_are_used(pkg, fanouts, 300)
    host = [rng.permutation(ids)[:n] for n in (300, 300, 300, 300, 80, 80, 80, 300, 300)]
    batches = [to_dev(s) for s in host]
    sampler = pkg.PipelinedSampler(c_ip, c_ix, fanouts, probs=c_pr, features=c_ft, replace=replace, max_seeds=300, depth=2)
    torch.manual_seed(31)
    piped = [(f.clone(), [(r.clone(), c.clone(), a, b) for r, c, a, b in blocks], ne, x.clone())
             for f, blocks, ne, x in sampler(batches)]
    assert sampler.pipe.recorded_slots() == 2
    torch.manual_seed(31)
    for (f, blocks, ne, x), seeds, s in zip(piped, batches, host):
        f2, blocks2, ne2 = pkg.sample_blocks(seeds, fanouts, c_ip, c_ix, probs=c_pr, replace=replace, fused=True)
        assert ne == ne2 == check_hops(oracle, indptr, indices, s, fanouts, replace, f, blocks)
        assert torch.equal(f, f2) and x.cpu().numpy().tobytes() == feats[f.cpu().numpy()].tobytes()
        for (r, c, a, b), (r2, c2, a2, b2) in zip(blocks, blocks2):
            assert (a, b) == (a2, b2) and torch.equal(r, r2) and torch.equal(c, c2)
    del sampler
