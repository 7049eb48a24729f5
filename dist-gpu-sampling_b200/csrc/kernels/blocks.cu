// Multi-hop sample -> relabel as ONE queued launch sequence.
//
// Replaces the loop of ChunkTensorSampler.sample_blocks (reference
// oppo_bench/single_node/utils/chunktensor_sampler.py:93-118), which for every
// hop calls the sampling operator (one blocking size read-back,
// src/cuda/rowwise_sampling.cu:147) and then the relabel operator (another one,
// src/cuda/tensor_reindex.cu:129) from Python, so the GPU idles between hops
// while the host learns each size and allocates the next output.
//
// Here the sizes never leave the device while the sequence runs: every kernel
// takes its item count as a device word written by its predecessor (Count),
// grids and buffers are sized by upper bounds the host can compute up front
// (hop h has at most seeds_h * (1 + fanout_h) frontier nodes, and never more
// than the graph has), and the actual sizes go to a caller-supplied (pinned)
// array that the host reads once, after everything is queued.
//
// Graphs of up to 2^23 ids take the form at dgs_sample_blocks_dense (one word per id); what follows is the form with a hash
// table per hop, which takes any id.
// Per hop: sample -> insert -> number.  The number launch of a hop also makes the
// plan of the next one (its unique list is the next seed list); only the first
// hop has a plan launch.  The sample launch carries, as extra CTAs, two jobs that
// depend on nothing it does: clearing the table this hop will fill and relabelling
// the COO of the hop before (whose numbering is complete by then).  The last hop's
// COO is relabelled by a launch of its own.  From the second hop on the seed list
// is a relabel's unique list, so a seed's relabelled id is its position and the
// sampler writes that directly; only the first hop (whose seeds the caller may
// repeat) looks its rows up.
#include <algorithm>
#include <cstdlib>
#include <new>

#include "common.cuh"
#include "launchers.h"
#include "philox.cuh"

namespace dgs {
namespace {

constexpr size_t WS_ALIGN = 256;
inline size_t ws_align(size_t x) { return (x + WS_ALIGN - 1) / WS_ALIGN * WS_ALIGN; }

__global__ void zero_sizes_kernel(int64_t* sizes, int n) {
  if (threadIdx.x < n) sizes[threadIdx.x] = 0;
}

int check_hops(const dgs_hop* hops, int32_t n_hops, const char* who) {
  DGS_REQUIRE(hops != nullptr && n_hops >= 1 && n_hops <= DGS_MAX_HOPS, DGS_ERR_INVALID,
              "%s: between 1 and %d hops", who, DGS_MAX_HOPS);
  for (int h = 0; h < n_hops; ++h) {
    DGS_REQUIRE(hops[h].fanout >= 1 && hops[h].seed_bound >= 0 && hops[h].frontier_bound >= 0, DGS_ERR_INVALID,
                "%s: hop %d: fanout %lld, bounds %lld / %lld", who, h, (long long)hops[h].fanout,
                (long long)hops[h].seed_bound, (long long)hops[h].frontier_bound);
    DGS_REQUIRE(hops[h].seed_bound * (1 + hops[h].fanout) < (1ll << 30), DGS_ERR_UNSUPPORTED,
                "%s: hop %d may produce %lld keys", who, h, (long long)(hops[h].seed_bound * (1 + hops[h].fanout)));
    DGS_REQUIRE(h == 0 || hops[h].seed_bound == hops[h - 1].frontier_bound, DGS_ERR_INVALID,
                "%s: hop %d: seed_bound must equal the previous hop's frontier_bound", who, h);
  }
  return DGS_OK;
}

}  // namespace
}  // namespace dgs

extern "C" int dgs_sample_blocks_bounds(int64_t n_seeds, const int64_t* fanouts, int32_t n_hops,
                                        int64_t num_nodes, dgs_hop* hops) {
  using namespace dgs;
  DGS_REQUIRE(fanouts != nullptr && hops != nullptr && n_hops >= 1 && n_hops <= DGS_MAX_HOPS && n_seeds >= 0 &&
                  num_nodes >= 0,
              DGS_ERR_INVALID, "dgs_sample_blocks_bounds: bad arguments");
  int64_t n = n_seeds;
  for (int h = 0; h < n_hops; ++h) {
    DGS_REQUIRE(fanouts[h] >= 1 && fanouts[h] < (1 << 20), DGS_ERR_INVALID, "dgs_sample_blocks_bounds: fanout %lld",
                (long long)fanouts[h]);
    hops[h].fanout = fanouts[h];
    hops[h].seed_bound = n;
    DGS_REQUIRE(n * (1 + fanouts[h]) < (1ll << 30), DGS_ERR_UNSUPPORTED,
                "dgs_sample_blocks_bounds: hop %d may produce %lld keys", h, (long long)(n * (1 + fanouts[h])));
    int64_t f = n * (1 + fanouts[h]);
    // a frontier of valid ids cannot be longer than the node list
    if (f > num_nodes) f = num_nodes > n ? num_nodes : n;
    hops[h].frontier_bound = f;
    n = f;
  }
  return DGS_OK;
}

extern "C" size_t dgs_sample_blocks_workspace_bytes(const dgs_hop* hops, int32_t n_hops) {
  using namespace dgs;
  if (hops == nullptr || n_hops < 1 || n_hops > DGS_MAX_HOPS) return 0;
  size_t total = WS_ALIGN;  // control words
  for (int h = 0; h < n_hops; ++h) {
    total += ws_align(dgs_sample_plan_bytes(hops[h].seed_bound));
    total += ws_align(dgs_relabel_table_bytes(hops[h].seed_bound * (1 + hops[h].fanout)));
  }
  return total;
}

extern "C" const int64_t* dgs_sample_blocks_frontier_count(const dgs_hop* hops, int32_t n_hops, void* workspace) {
  using namespace dgs;
  if (hops == nullptr || workspace == nullptr || n_hops < 1 || n_hops > DGS_MAX_HOPS) return nullptr;
  // same walk as the carving in dgs_sample_blocks: the word sits in the last hop's table
  char* p = static_cast<char*>(workspace) + WS_ALIGN;
  for (int h = 0; h < n_hops; ++h) {
    const int64_t key_bound = hops[h].seed_bound * (1 + hops[h].fanout);
    p += ws_align(dgs_sample_plan_bytes(hops[h].seed_bound));
    if (h == n_hops - 1) return unique_total(p, key_bound);
    p += ws_align(dgs_relabel_table_bytes(key_bound));
  }
  return nullptr;
}

namespace dgs {
namespace {

// ---- the form with one word per id -----------------------------------------------
// The hash tables cost an insert launch per hop (load, compare-and-swap and probes per key, 21 us for the 876 k keys of a
// last hop) and a table cleared per hop.  A fire-and-forget atomic in the sampling launch costs nothing that shows there
// (18.9 us with it, 18.5 without), and what numbers the nodes reads ids and words only.  Batches of 1 024 seeds [15, 10, 5]
// over 2.4 M nodes with 100 features, one at a time 191 -> 147 us, six in flight 806 -> 674; 64 seeds [10, 5] 77 -> 63.
// control words | plans | tickets and tile words of all hops | one word per id
struct DenseSpace {
  int64_t* n0;
  uint64_t* keys;
  int64_t* totals;            // [n_hops] length of each hop's frontier
  void* plan[DGS_MAX_HOPS];
  unsigned int* ticket[DGS_MAX_HOPS];
  unsigned long long* tiles[DGS_MAX_HOPS];
  uint32_t* first;
  uint32_t* beyond;           // a word beside the first hop's ticket
  FillJob fill;               // tickets, tile words and words of the ids
  size_t bytes;
};
static_assert(sizeof(int64_t) * (1 + 2 * DGS_MAX_HOPS) <= WS_ALIGN, "control words: n0, a key and a frontier length per hop");

// The line: clearing a word per id (the first launch does it beside the plan) against the probes it saves.  Recorded
// sequences, hash tables -> one word per id, us: 16 seeds [10, 5] over 0.5 M ids 39 -> 28, 2.4 M 39 -> 27, 8 M 40 -> 29,
// 20 M 37 -> 35, 111 M 37 -> 88; 1 024 seeds [15, 10, 5] over 2.4 M ids 141 -> 92, 8 M 141 -> 90, 20 M 131 -> 111, 111 M
// 134 -> 214.  With six batches in flight there are six tables, and past the L2 (126 MB) their words come from HBM:
// 8 M ids 730 -> 684 us, 16 M 711 -> 744.  (Before their words were kept in the L2 with a hint; with it 8.3 M ids 80 -> 77 a batch.)
// The hops do not move the line.  A batch through BlockPipeline, hash tables -> one word per id, us, one slot / six: 16 seeds
// [10, 5] over 0.5 M ids 59 -> 49 / 28 -> 29, 2.4 M 61 -> 49 / 30 -> 29, 8.3 M 59 -> 51 / 28 -> 28; 64 seeds 63 -> 52 / 29 -> 29,
// 63 -> 52 / 27 -> 28, 62 -> 53 / 28 -> 28; 256 seeds [15, 10, 5] 102 -> 79 / 39 -> 37, 112 -> 86 / 45 -> 38, 100 -> 80 / 39 -> 37 (with
// six slots about 24 us is the host's share of a batch).
constexpr int64_t DENSE_MAX_IDS = int64_t(1) << 23;
constexpr unsigned FILL_CTA_UNITS = 4096;  // 64 KB a CTA of 1 024 threads

DenseSpace dense_space(const dgs_hop* hops, int32_t n_hops, int64_t ids, void* workspace) {
  DenseSpace d{};
  char* const base = static_cast<char*>(workspace);
  size_t at = WS_ALIGN;
  d.n0 = reinterpret_cast<int64_t*>(base);
  d.keys = reinterpret_cast<uint64_t*>(d.n0 + 1);
  d.totals = d.n0 + 1 + DGS_MAX_HOPS;
  for (int h = 0; h < n_hops; ++h) {
    d.plan[h] = base + at;
    at += ws_align(dgs_sample_plan_bytes(hops[h].seed_bound));
  }
  const size_t cleared = at;
  for (int h = 0; h < n_hops; ++h) {
    d.ticket[h] = reinterpret_cast<unsigned int*>(base + at);
    d.tiles[h] = reinterpret_cast<unsigned long long*>(base + at + 16);
    at += 16 + 16 * static_cast<size_t>(dense_tiles(hops[h].seed_bound, hops[h].seed_bound * hops[h].fanout));
  }
  d.beyond = d.ticket[0] + 1;
  d.first = reinterpret_cast<uint32_t*>(base + at);
  at += (static_cast<size_t>(ids) * sizeof(uint32_t) + 15) / 16 * 16;
  d.fill.at = reinterpret_cast<ulonglong2*>(base + cleared);
  d.fill.units = static_cast<int64_t>((at - cleared) / 16);
  d.fill.ctas = static_cast<unsigned>(std::min<int64_t>((d.fill.units + FILL_CTA_UNITS - 1) / FILL_CTA_UNITS, 1 << 16));
  d.bytes = ws_align(at);
  return d;
}

// Per hop: sample (which marks what it draws) -> number (+ the next hop's plan); one lookup for all hops at the end.  The
// first launch, which makes the first hop's plan, also clears the words.
int queue_dense(const dgs_chunk_desc* indptr, const dgs_chunk_desc* indices, const dgs_chunk_desc* probs, const void* seeds,
                bool ids64, const dgs_hop* hops, int32_t n_hops, bool replace, int64_t id_space, uint64_t rng_seed,
                uint64_t rng_offset, const uint64_t* rng_words, void* workspace, int64_t* sizes, int32_t* status,
                cudaStream_t s) {
  const DenseSpace d = dense_space(hops, n_hops, id_space, workspace);
  const InitWords init{d.n0, hops[0].seed_bound, rng_words, d.keys, n_hops};
  int rc = launch_sample_plan(*indptr, seeds, ids64, hops[0].seed_bound, hops[0].fanout, replace, d.plan[0], nullptr, init,
                              d.fill, status, s);
  if (rc != DGS_OK) return rc;
  DenseLookup lookup{};
  lookup.first = d.first;
  lookup.ids = id_space;
  lookup.n_hops = n_hops;
  lookup.row0 = hops[0].coo_row;
  SizesReport report{};
  report.dst = sizes;
  const void* hop_seeds = seeds;
  const int64_t* n_dev = d.n0;
  for (int h = 0; h < n_hops; ++h) {
    const dgs_hop& hp = hops[h];
    const int64_t k = hp.fanout, edge_bound = hp.seed_bound * k;
    const Count n{hp.seed_bound, n_dev};
    const bool later = h > 0;  // the plan came with the numbering of these seeds, which are unique and labelled
    const RngKey key = rng_words != nullptr
                           ? RngKey{0, d.keys + h}
                           : host_key(sample_rng_key(rng_seed, rng_offset + static_cast<uint64_t>(h)));
    const IdMarks marks{d.first, id_space, !later, d.beyond};
    rc = probs != nullptr
             ? launch_sample_weighted(*indices, *probs, hop_seeds, ids64, n, k, replace, d.plan[h], later, key, hp.coo_row,
                                      hp.coo_col, edge_bound, nullptr, later, SideJobs{}, marks, status, s)
             : launch_sample_uniform(*indices, hop_seeds, ids64, n, k, replace, d.plan[h], later, key, hp.coo_row,
                                     hp.coo_col, edge_bound, nullptr, later, SideJobs{}, marks, status, s);
    if (rc != DGS_OK) return rc;
    const Count nnz{edge_bound, sample_plan_total(d.plan[h], hp.seed_bound)};
    report.src[2 * h] = nnz.dev;
    report.src[2 * h + 1] = d.totals + h;
    NextPlan next{};
    if (h + 1 < n_hops) next = make_next_plan(*indptr, hops[h + 1].seed_bound, hops[h + 1].fanout, replace, d.plan[h + 1]);
    else report.n = 2 * n_hops;  // the last hop's numbering sends all sizes to the host at once
    const DenseNumbering number{d.first, id_space, d.ticket[h], d.beyond, d.tiles[h], d.totals + h, later};
    rc = launch_dense_number(ids64, number, hop_seeds, n, hp.coo_col, nnz, hp.frontier, hp.frontier_bound, report, next,
                             status, s);
    if (rc != DGS_OK) return rc;
    lookup.col[h] = hp.coo_col;
    lookup.n[h] = nnz;
    lookup.end_cta[h] = (h > 0 ? lookup.end_cta[h - 1] : 0u) + static_cast<unsigned>((edge_bound + RL_TILE - 1) / RL_TILE);
    hop_seeds = hp.frontier;
    n_dev = d.totals + h;
  }
  return launch_dense_lookup(lookup, ids64, s);
}

// Queues the whole sequence on `stream`.  id_space > 0: with one word per id below it.  rng_words == nullptr: the keys come
// from (rng_seed, rng_offset) as launch parameters; otherwise the first kernel reads (seed, offset) from rng_words when it RUNS.
int queue_blocks(const dgs_chunk_desc* indptr, const dgs_chunk_desc* indices, const dgs_chunk_desc* probs,
                 const void* seeds, int32_t ids64, const dgs_hop* hops, int32_t n_hops, int32_t replace,
                 int64_t id_space, uint64_t rng_seed, uint64_t rng_offset, const uint64_t* rng_words, void* workspace,
                 size_t workspace_bytes, int64_t* sizes, int32_t* status, dgs_stream_t stream) {
  int rc = validate_desc(indptr, "dgs_sample_blocks(indptr)");
  if (rc != DGS_OK) return rc;
  rc = validate_desc(indices, "dgs_sample_blocks(indices)");
  if (rc != DGS_OK) return rc;
  if (probs != nullptr) {
    rc = validate_desc(probs, "dgs_sample_blocks(probs)");
    if (rc != DGS_OK) return rc;
    DGS_REQUIRE(probs->esz == 4, DGS_ERR_UNSUPPORTED, "dgs_sample_blocks: weights must be fp32");
  }
  rc = check_hops(hops, n_hops, "dgs_sample_blocks");
  if (rc != DGS_OK) return rc;
  const int esz = ids64 ? 8 : 4;
  DGS_REQUIRE(indptr->esz == esz && indices->esz == esz, DGS_ERR_INVALID,
              "dgs_sample_blocks: indptr / indices element size does not match the id type");
  DGS_REQUIRE(sizes != nullptr, DGS_ERR_INVALID, "dgs_sample_blocks: null sizes");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t n0 = hops[0].seed_bound;
  if (n0 == 0) {
    zero_sizes_kernel<<<1, 32, 0, s>>>(sizes, 2 * n_hops);
    DGS_LAUNCH_CHECK();
    return DGS_OK;
  }
  DGS_REQUIRE(seeds != nullptr, DGS_ERR_INVALID, "dgs_sample_blocks: null seeds");
  const size_t need = id_space > 0 ? dense_space(hops, n_hops, id_space, nullptr).bytes
                                   : dgs_sample_blocks_workspace_bytes(hops, n_hops);
  DGS_REQUIRE(workspace != nullptr && workspace_bytes >= need &&
                  (reinterpret_cast<uintptr_t>(workspace) & 15) == 0,
              DGS_ERR_INVALID, "dgs_sample_blocks: workspace too small or not 16-byte aligned");
  for (int h = 0; h < n_hops; ++h) {
    DGS_REQUIRE(hops[h].coo_row != nullptr && hops[h].coo_col != nullptr && hops[h].frontier != nullptr,
                DGS_ERR_INVALID, "dgs_sample_blocks: hop %d: null output", h);
    DGS_REQUIRE(probs == nullptr || replace || hops[h].fanout <= 32, DGS_ERR_UNSUPPORTED,
                "dgs_sample_blocks: weighted fan-out %lld > 32 without replacement is not supported",
                (long long)hops[h].fanout);
  }

  if (id_space > 0) return queue_dense(indptr, indices, probs, seeds, ids64 != 0, hops, n_hops, replace != 0, id_space, rng_seed,
                                       rng_offset, rng_words, workspace, sizes, status, s);

  // ---- carve the workspace ----
  char* p = static_cast<char*>(workspace);
  int64_t* n0_dev = reinterpret_cast<int64_t*>(p);
  p += WS_ALIGN;
  void* plan[DGS_MAX_HOPS];
  void* table[DGS_MAX_HOPS];
  static_assert(sizeof(int64_t) * (1 + DGS_MAX_HOPS) <= WS_ALIGN, "the control words hold n0 and one key per hop");
  uint64_t* keys_dev = reinterpret_cast<uint64_t*>(n0_dev + 1);
  for (int h = 0; h < n_hops; ++h) {
    const int64_t key_bound = hops[h].seed_bound * (1 + hops[h].fanout);
    plan[h] = p;
    p += ws_align(dgs_sample_plan_bytes(hops[h].seed_bound));
    table[h] = p;
    p += ws_align(dgs_relabel_table_bytes(key_bound));
  }

  // a graph with fewer nodes than 2^32 - 1 has no ids beyond
  const long long max_key = !ids64 || indptr->total - 1 < COMPACT_KEY_LIMIT ? COMPACT_KEY_LIMIT - 1 : INT64_MAX;

  // ---- queue every hop; no size is read back in between ----
  const void* hop_seeds = seeds;
  const int64_t* n_dev = n0_dev;
  LookupJob pending{};  // relabelling of the previous hop's COO, carried by the next sample launch
  SizesReport report{};
  report.dst = sizes;
  const InitWords init{n0_dev, n0, rng_words, keys_dev, n_hops};
  rc = launch_sample_plan(*indptr, seeds, ids64 != 0, n0, hops[0].fanout, replace != 0, plan[0], nullptr, init, FillJob{}, status, s);
  if (rc != DGS_OK) return rc;
  for (int h = 0; h < n_hops; ++h) {
    const dgs_hop& hp = hops[h];
    const int64_t k = hp.fanout;
    const int64_t edge_bound = hp.seed_bound * k;
    const int64_t key_bound = hp.seed_bound + edge_bound;
    const Count n{hp.seed_bound, n_dev};
    // the table is dimensioned before the neighbours are drawn: seeds * (1 + fanout) keys at most
    const TableSize size{n, 1 + k, max_key};
    const SideJobs jobs{make_clear_job(table[h], key_bound, size), pending, 0u};
    const int64_t* nnz_dev = sample_plan_total(plan[h], hp.seed_bound);
    const RngKey key = rng_words != nullptr
                           ? RngKey{0, keys_dev + h}
                           : host_key(sample_rng_key(rng_seed, rng_offset + static_cast<uint64_t>(h)));
    const bool later = h > 0;  // the plan came with the numbering of these seeds, which are unique
    rc = probs != nullptr
             ? launch_sample_weighted(*indices, *probs, hop_seeds, ids64 != 0, n, k, replace != 0, plan[h], later,
                                      key, hp.coo_row, hp.coo_col, edge_bound, nullptr, later, jobs, IdMarks{}, status, s)
             : launch_sample_uniform(*indices, hop_seeds, ids64 != 0, n, k, replace != 0, plan[h], later, key,
                                     hp.coo_row, hp.coo_col, edge_bound, nullptr, later, jobs, IdMarks{}, status, s);
    if (rc != DGS_OK) return rc;
    const Count nnz{edge_bound, nnz_dev};
    report.src[2 * h] = nnz_dev;
    report.src[2 * h + 1] = unique_total(table[h], key_bound);
    NextPlan next{};
    if (h + 1 < n_hops) next = make_next_plan(*indptr, hops[h + 1].seed_bound, hops[h + 1].fanout, replace != 0, plan[h + 1]);
    else report.n = 2 * n_hops;  // the last hop's numbering sends all sizes to the host at once
    rc = launch_unique_pair(ids64 != 0, hop_seeds, n, hp.coo_col, nnz, key_bound, size, table[h], hp.frontier,
                            hp.frontier_bound, nullptr, report, next, status, s);
    if (rc != DGS_OK) return rc;
    pending = make_lookup_job(table[h], key_bound, size, later ? nullptr : hp.coo_row, hp.coo_col, nnz, n);
    hop_seeds = hp.frontier;
    n_dev = unique_total(table[h], key_bound);
  }
  return launch_lookup(pending, ids64 != 0, s);
}

}  // namespace
}  // namespace dgs

extern "C" int dgs_sample_blocks(const dgs_chunk_desc* indptr, const dgs_chunk_desc* indices,
                                 const dgs_chunk_desc* probs, const void* seeds, int32_t ids64,
                                 const dgs_hop* hops, int32_t n_hops, int32_t replace, uint64_t rng_seed,
                                 uint64_t rng_offset, void* workspace, size_t workspace_bytes,
                                 int64_t* sizes, int32_t* status, dgs_stream_t stream) {
  return dgs::queue_blocks(indptr, indices, probs, seeds, ids64, hops, n_hops, replace, 0, rng_seed, rng_offset, nullptr,
                           workspace, workspace_bytes, sizes, status, stream);
}

extern "C" size_t dgs_sample_blocks_dense_workspace_bytes(const dgs_hop* hops, int32_t n_hops, int64_t id_space) {
  using namespace dgs;
  if (hops == nullptr || n_hops < 1 || n_hops > DGS_MAX_HOPS || id_space < 1 || id_space > COMPACT_KEY_LIMIT) return 0;
  return dense_space(hops, n_hops, id_space, nullptr).bytes;
}

extern "C" int32_t dgs_sample_blocks_dense_wins(const dgs_hop* hops, int32_t n_hops, int64_t id_space) {
  using namespace dgs;
  if (hops == nullptr || n_hops < 1 || n_hops > DGS_MAX_HOPS || id_space < 1 || id_space > COMPACT_KEY_LIMIT) return 0;
  return id_space <= DENSE_MAX_IDS;  // whatever the hops: see there
}

extern "C" const int64_t* dgs_sample_blocks_dense_frontier_count(const dgs_hop* hops, int32_t n_hops, int64_t id_space,
                                                                 void* workspace) {
  using namespace dgs;
  if (hops == nullptr || workspace == nullptr || n_hops < 1 || n_hops > DGS_MAX_HOPS || id_space < 1) return nullptr;
  return dense_space(hops, n_hops, id_space, workspace).totals + n_hops - 1;
}

extern "C" int dgs_sample_blocks_dense(const dgs_chunk_desc* indptr, const dgs_chunk_desc* indices,
                                       const dgs_chunk_desc* probs, const void* seeds, int32_t ids64,
                                       const dgs_hop* hops, int32_t n_hops, int32_t replace, int64_t id_space,
                                       uint64_t rng_seed, uint64_t rng_offset, void* workspace, size_t workspace_bytes,
                                       int64_t* sizes, int32_t* status, dgs_stream_t stream) {
  using namespace dgs;
  DGS_REQUIRE(id_space >= 1 && id_space <= COMPACT_KEY_LIMIT && status != nullptr, DGS_ERR_INVALID,
              "dgs_sample_blocks_dense: an id space of 1 to 2^32 - 1 ids and a status word, please (%lld)", (long long)id_space);
  return queue_blocks(indptr, indices, probs, seeds, ids64, hops, n_hops, replace, id_space, rng_seed, rng_offset, nullptr,
                      workspace, workspace_bytes, sizes, status, stream);
}

// ---- the sequence recorded once and replayed ------------------------------------
// Queuing a batch is a dozen kernel launches with the same parameters every time as long as the buffers, the
// bounds (the number of seeds) and the tables stay the same; only the random stream differs.  A recording
// holds those launches as one executable graph (stream capture keeps the programmatic edges between the
// kernels), and a replay is a single launch call.
struct dgs_blocks_recording {
  cudaGraphExec_t exec = nullptr;
};

namespace dgs {
namespace {
int record_blocks(const dgs_chunk_desc* indptr, const dgs_chunk_desc* indices, const dgs_chunk_desc* probs,
                  const void* seeds, int32_t ids64, const dgs_hop* hops, int32_t n_hops, int32_t replace, int64_t id_space,
                  const uint64_t* rng_words, void* workspace, size_t workspace_bytes, int64_t* sizes, int32_t* status,
                  dgs_stream_t capture_stream, dgs_blocks_recording** out) {
  DGS_REQUIRE(out != nullptr && rng_words != nullptr, DGS_ERR_INVALID, "dgs_sample_blocks_record: null argument");
  DGS_REQUIRE(capture_stream != nullptr, DGS_ERR_INVALID,
              "dgs_sample_blocks_record: the default stream cannot record; pass a stream of your own");
  *out = nullptr;
  cudaStream_t s = static_cast<cudaStream_t>(capture_stream);
  // thread-local mode: other host threads keep allocating and copying while this one records
  DGS_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  const int rc = queue_blocks(indptr, indices, probs, seeds, ids64, hops, n_hops, replace, id_space, 0, 0, rng_words,
                              workspace, workspace_bytes, sizes, status, capture_stream);
  cudaGraph_t graph = nullptr;
  const cudaError_t end = cudaStreamEndCapture(s, &graph);  // always closed, also after a refused argument
  if (rc != DGS_OK) {
    if (graph != nullptr) cudaGraphDestroy(graph);
    (void)cudaGetLastError();
    return rc;
  }
  if (end != cudaSuccess) return cuda_fail(end, "cudaStreamEndCapture", __FILE__, __LINE__);
  cudaGraphExec_t exec = nullptr;
  const cudaError_t inst = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (inst != cudaSuccess) return cuda_fail(inst, "cudaGraphInstantiate", __FILE__, __LINE__);
  dgs_blocks_recording* rec = new (std::nothrow) dgs_blocks_recording;
  if (rec == nullptr) {
    cudaGraphExecDestroy(exec);
    DGS_REQUIRE(false, DGS_ERR_CUDA, "dgs_sample_blocks_record: out of host memory");
  }
  rec->exec = exec;
  *out = rec;
  return DGS_OK;
}
}  // namespace
}  // namespace dgs

extern "C" int dgs_sample_blocks_record(const dgs_chunk_desc* indptr, const dgs_chunk_desc* indices,
                                        const dgs_chunk_desc* probs, const void* seeds, int32_t ids64,
                                        const dgs_hop* hops, int32_t n_hops, int32_t replace,
                                        const uint64_t* rng_words, void* workspace, size_t workspace_bytes,
                                        int64_t* sizes, int32_t* status, dgs_stream_t capture_stream,
                                        dgs_blocks_recording** out) {
  return dgs::record_blocks(indptr, indices, probs, seeds, ids64, hops, n_hops, replace, 0, rng_words, workspace,
                            workspace_bytes, sizes, status, capture_stream, out);
}

extern "C" int dgs_sample_blocks_dense_record(const dgs_chunk_desc* indptr, const dgs_chunk_desc* indices,
                                              const dgs_chunk_desc* probs, const void* seeds, int32_t ids64,
                                              const dgs_hop* hops, int32_t n_hops, int32_t replace, int64_t id_space,
                                              const uint64_t* rng_words, void* workspace, size_t workspace_bytes,
                                              int64_t* sizes, int32_t* status, dgs_stream_t capture_stream,
                                              dgs_blocks_recording** out) {
  using namespace dgs;
  DGS_REQUIRE(id_space >= 1 && id_space <= COMPACT_KEY_LIMIT && status != nullptr, DGS_ERR_INVALID,
              "dgs_sample_blocks_dense_record: an id space of 1 to 2^32 - 1 ids and a status word, please (%lld)",
              (long long)id_space);
  return record_blocks(indptr, indices, probs, seeds, ids64, hops, n_hops, replace, id_space, rng_words, workspace,
                       workspace_bytes, sizes, status, capture_stream, out);
}

extern "C" int dgs_sample_blocks_replay(dgs_blocks_recording* rec, dgs_stream_t stream) {
  using namespace dgs;
  DGS_REQUIRE(rec != nullptr && rec->exec != nullptr, DGS_ERR_INVALID, "dgs_sample_blocks_replay: null recording");
  DGS_CUDA_TRY(cudaGraphLaunch(rec->exec, static_cast<cudaStream_t>(stream)));
  return DGS_OK;
}

extern "C" void dgs_sample_blocks_recording_free(dgs_blocks_recording* rec) {
  if (rec == nullptr) return;
  if (rec->exec != nullptr) cudaGraphExecDestroy(rec->exec);
  delete rec;
}
