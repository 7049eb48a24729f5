"""The multi-hop sequence with one word per id (dgs_sample_blocks_dense): the same results, bit for bit, as the form
with hash tables, at the edges of its tiles, for every kind of sampling, and with ids beyond the id space."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ERR_INVALID, ERR_ID_SPACE = 1, 9


def to_dev(a, dt=torch.int64):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dt).cuda()


def graph(rng, n, max_deg, hubs=(), n_src=None):
    deg = rng.integers(0, max_deg, size=n)
    for i, d in enumerate(hubs):
        deg[i] = d
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    return indptr, rng.integers(0, n_src or n, size=int(indptr[-1])).astype(np.int64)


class Request:
    """One request through the C ABI, in either form."""

    def __init__(self, pkg, indptr, indices, seeds, fanouts, idt=torch.int64, probs=None, replace=False):
        from gpu_util import plain_desc
        self.pkg, self.abi, self.idt, self.replace = pkg, pkg.load_abi(), idt, replace
        self.keep = [to_dev(indptr, idt), to_dev(indices, idt), to_dev(seeds, idt)]
        self.probs = torch.from_numpy(probs).cuda() if probs is not None else None
        self.d = [plain_desc(self.keep[0]), plain_desc(self.keep[1])]
        self.d_pr = plain_desc(self.probs) if probs is not None else None
        self.H, self.n, self.nodes = len(fanouts), len(seeds), len(indptr) - 1
        self.applied = (ctypes.c_int64 * self.H)(*reversed(fanouts))

    def run(self, id_space=None, record=False, rng=(5, 8)):
        from gpu_util import vp
        abi, H, pkg = self.abi, self.H, self.pkg
        hops = (pkg.Hop * H)()
        pkg.check(abi.dgs_sample_blocks_bounds(self.n, self.applied, H, max(self.nodes, id_space or 0), hops))
        bufs = []
        for h in range(H):
            cap = hops[h].seed_bound * hops[h].fanout
            r, c = (torch.full((cap,), -7, device="cuda", dtype=self.idt) for _ in range(2))
            fr = torch.full((hops[h].frontier_bound,), -7, device="cuda", dtype=self.idt)
            hops[h].coo_row, hops[h].coo_col, hops[h].frontier = vp(r), vp(c), vp(fr)
            bufs.append((r, c, fr))
        sizes = torch.zeros(2 * H, dtype=torch.int64).pin_memory()
        status = torch.zeros(1, dtype=torch.int32).pin_memory()
        head = [ctypes.byref(self.d[0]), ctypes.byref(self.d[1]), ctypes.byref(self.d_pr) if self.d_pr else None,
                vp(self.keep[2]), 1 if self.idt == torch.int64 else 0, hops, H, 1 if self.replace else 0]
        if id_space is None:
            wsb = abi.dgs_sample_blocks_workspace_bytes(hops, H)
            ws = torch.randint(0, 256, (wsb,), dtype=torch.uint8, device="cuda")  # contents are irrelevant
            pkg.check(abi.dgs_sample_blocks(*head, rng[0], rng[1], vp(ws), wsb, vp(sizes), vp(status), None))
            count = abi.dgs_sample_blocks_frontier_count(hops, H, vp(ws))
        else:
            wsb = abi.dgs_sample_blocks_dense_workspace_bytes(hops, H, id_space)
            ws = torch.randint(0, 256, (wsb,), dtype=torch.uint8, device="cuda")
            if record:
                words = torch.tensor(rng, dtype=torch.int64).pin_memory()
                stream, rec = torch.cuda.Stream(), ctypes.c_void_p()
                pkg.check(abi.dgs_sample_blocks_dense_record(*head, id_space, vp(words), vp(ws), wsb, vp(sizes), vp(status),
                                                             ctypes.c_void_p(stream.cuda_stream), ctypes.byref(rec)))
                torch.cuda.synchronize()
                for _ in range(2):  # a replay finds the words of the one before
                    pkg.check(abi.dgs_sample_blocks_replay(rec, ctypes.c_void_p(stream.cuda_stream)))
                torch.cuda.synchronize()
                abi.dgs_sample_blocks_recording_free(rec)
            else:
                pkg.check(abi.dgs_sample_blocks_dense(*head, id_space, rng[0], rng[1], vp(ws), wsb, vp(sizes), vp(status),
                                                      None))
            count = abi.dgs_sample_blocks_dense_frontier_count(hops, H, id_space, vp(ws))
        torch.cuda.synchronize()
        sz = sizes.tolist()
        at = count - ws.data_ptr()
        assert int(ws[at:at + 8].cpu().numpy().view(np.int64)[0]) == sz[2 * H - 1]
        out = [(b[0][:sz[2 * h]], b[1][:sz[2 * h]], b[2][:sz[2 * h + 1]]) for h, b in enumerate(bufs)]
        return status.item(), sz, out


def same(a, b):
    return a[0] == b[0] and a[1] == b[1] and all(torch.equal(x, y) for p, q in zip(a[2], b[2]) for x, y in zip(p, q))


@pytest.mark.parametrize("idt", [torch.int64, torch.int32])
@pytest.mark.parametrize("n_seeds,fanouts", [(1, [3]), (255, [4, 4]), (1023, [5, 5]), (1024, [15, 10]), (1025, [2, 40]),
                                             (2048, [1, 1, 1]), (2049, [3, 2]), (5000, [20, 30])])
def test_equals_the_hash_form(pkg, idt, n_seeds, fanouts):
    rng = np.random.default_rng(n_seeds)
    indptr, indices = graph(rng, 30_001, 30, hubs=(0, 1, 700, 5000))
    seeds = rng.permutation(30_001)[:n_seeds]
    seeds[:4] = [0, 1, 2, 3][:n_seeds]
    seeds[n_seeds // 2:n_seeds // 2 + n_seeds // 8] = seeds[:n_seeds // 8]   # repeated seeds
    q = Request(pkg, indptr, indices, seeds, fanouts, idt)
    plain = q.run()
    assert plain[0] == 0
    assert same(q.run(id_space=30_001), plain)
    assert same(q.run(id_space=30_001, record=True), plain)


@pytest.mark.parametrize("weighted,replace", [(False, True), (True, False), (True, True)])
def test_equals_the_hash_form_for_every_kind_of_sampling(pkg, weighted, replace):
    rng = np.random.default_rng(3)
    indptr, indices = graph(rng, 9000, 60, hubs=(0, 5000, 900))
    probs = (rng.random(indices.size) + 0.05).astype(np.float32) if weighted else None
    seeds = np.concatenate([[0, 1, 2], rng.permutation(9000)[:600]])
    q = Request(pkg, indptr, indices, seeds, [7, 12], probs=probs, replace=replace)
    assert same(q.run(id_space=9000), q.run())


def test_isolated_seeds_and_full_rows(pkg):
    indptr = np.zeros(101, dtype=np.int64)
    q = Request(pkg, indptr, np.zeros(1, dtype=np.int64), np.arange(100)[::-1], [4, 4])   # no edge anywhere
    st, sz, out = q.run(id_space=100)
    assert st == 0 and sz == [0, 100, 0, 100] and out[1][2].tolist() == list(range(100))[::-1]


def test_ids_beyond_the_id_space_are_reported_and_the_operators_take_them(pkg, ops):
    """A bipartite CSC: column ids of a larger space than its rows, but too few of them in one hop to outgrow a bound."""
    rng = np.random.default_rng(8)
    indptr, indices = graph(rng, 4000, 9, n_src=100_000)
    seeds = rng.permutation(4000)[:50]
    q = Request(pkg, indptr, indices, seeds, [5])
    plain = q.run(rng=(77, 0))
    assert plain[0] == 0 and plain[2][0][2].max().item() >= 4000
    assert q.run(id_space=4000, rng=(77, 0))[0] == ERR_ID_SPACE
    assert same(q.run(id_space=100_000, rng=(77, 0)), plain)
    ip, ix, sd = to_dev(indptr), to_dev(indices), to_dev(seeds)
    for _ in range(2):
        torch.manual_seed(77)
        f, blocks, _ = pkg.sample_blocks(sd, [5], ip, ix, fused=True)
        assert torch.equal(f, plain[2][0][2]) and torch.equal(blocks[0][1], plain[2][0][1])

    def chunked(a):
        ct = torch.classes.dgs_classes.ChunkTensor([a.size], torch.int64, a.size * 8)
        ct._CAPI_load_from_tensor(torch.from_numpy(a))
        return ct

    feats = torch.classes.dgs_classes.ChunkTensor([100_000, 4], torch.float32, 100_000 * 16)
    feats._CAPI_load_from_tensor(torch.arange(400_000, dtype=torch.float32).view(-1, 4))
    c_ip, c_ix = chunked(indptr), chunked(indices)
    sampler = pkg.PipelinedSampler(c_ip, c_ix, [5], features=feats, max_seeds=50, depth=3)
    for _ in range(3):                                  # batches in flight when the first one is found out
        torch.manual_seed(77)
        sampler.submit(sd)
    for i in range(6):
        f, blocks, _, x = sampler.next()
        assert torch.equal(f, plain[2][0][2]) and torch.equal(blocks[0][0], plain[2][0][0])
        assert torch.equal(blocks[0][1], plain[2][0][1]) and torch.equal(x[:, 0], (f * 4).float())
        if i < 3:
            torch.manual_seed(77)
            sampler.submit(sd)


def test_refused_arguments(pkg):
    from gpu_util import vp
    rng = np.random.default_rng(1)
    indptr, indices = graph(rng, 100, 5)
    q = Request(pkg, indptr, indices, np.arange(10), [3])
    hops = (pkg.Hop * 1)()
    pkg.check(q.abi.dgs_sample_blocks_bounds(10, q.applied, 1, 100, hops))
    buf = torch.zeros(1 << 16, dtype=torch.int64, device="cuda")
    hops[0].coo_row = hops[0].coo_col = hops[0].frontier = vp(buf)
    words = torch.zeros(4, dtype=torch.int64).pin_memory()
    need = q.abi.dgs_sample_blocks_dense_workspace_bytes(hops, 1, 100)

    def call(id_space, ws_bytes, status):
        return q.abi.dgs_sample_blocks_dense(ctypes.byref(q.d[0]), ctypes.byref(q.d[1]), None, vp(q.keep[2]), 1, hops, 1, 0,
                                             id_space, 1, 0, vp(buf), ws_bytes, vp(words), status, None)
    st = vp(torch.zeros(1, dtype=torch.int32).pin_memory())
    assert call(0, 1 << 18, st) == ERR_INVALID and call(1 << 33, 1 << 18, st) == ERR_INVALID
    assert call(100, need - 1, st) == ERR_INVALID and call(100, need, None) == ERR_INVALID
    assert q.abi.dgs_sample_blocks_dense_workspace_bytes(hops, 1, 0) == 0
