// Unique (first-occurrence order) + relabel through an open-addressing table.
//
// Replaces RelabelHashmap / Unique / Relabel / TensorRelabelCUDA
// (reference src/cuda/tensor_reindex.cu:11-205): three torch::full tables, two
// torch::cat copies, four thrust passes that each re-probe the table, a cub
// scan and a blocking read-back, with hash(key) = key & (cap-1) at a load
// factor of up to 100 %.
//
// Kept (the contract): the i-th distinct key in first-occurrence order gets
// label i; lookups return the label or -1.  The order is fixed by storing the
// MINIMUM input index per key (atomicMin) exactly as the reference does
// (:28,123), so the result does not depend on hash layout or thread timing.
//
// Different (the design):
//   * one 8-byte slot per entry, mixed hash, linear probing, load factor <= 50 %.
//   * inputs are read through a segment list instead of being concatenated.
//   * the insert pass remembers each input's slot, so later passes index the
//     table directly instead of probing again.
//   * first occurrences are counted and numbered in ONE pass (a look-back over
//     the tiles' sums); the label is stored into the slot with the top bit set,
//     which can never be mistaken for an input index by a concurrent reader, so
//     no third table.  In the multi-hop sequence the same pass reads the row
//     bounds of the nodes it numbers and places their outputs: the next hop's plan.
//   * the number of distinct keys goes to a caller-supplied (pinned) word.
#include "common.cuh"
#include "host_report.cuh"
#include "launchers.h"
#include "relabel_device.cuh"
#include "sample_device.cuh"
#include "tile_scan.cuh"

#include <type_traits>

namespace dgs {
namespace {

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// words | ticket, tile words, wide keys (within 8 bytes per slot: slots >= 2n) | slot_of | largest | total | dense
inline TableParts table_view(void* mem, int64_t n) {
  TableParts t;
  const uint64_t cap = slots_for(n);
  t.ntiles = (n + RL_TILE - 1) / RL_TILE;
  char* p = static_cast<char*>(mem);
  t.words = reinterpret_cast<unsigned long long*>(p);
  char* q = p + cap * sizeof(unsigned long long);
  t.ticket = reinterpret_cast<unsigned int*>(q);
  t.tiles = reinterpret_cast<unsigned long long*>(q + 16);
  t.tiles2 = t.tiles + t.ntiles;
  t.wide_keys = reinterpret_cast<long long*>(t.tiles2 + t.ntiles);
  p += 2 * cap * sizeof(unsigned long long);
  t.slot_of = reinterpret_cast<uint32_t*>(p);
  p += align_up(static_cast<size_t>(n) * sizeof(uint32_t), 16);
  t.largest = reinterpret_cast<unsigned long long*>(p);
  t.total = reinterpret_cast<int64_t*>(p) + t.ntiles;
  t.dense = t.total + 1;
  return t;
}
// the ticket and the tile words, in units of 16 bytes
inline int64_t ticket_units(const TableParts& t) { return 1 + t.ntiles; }

// ---- where the keys come from ---------------------------------------------------
// A host-known segment list (the per-operator entry points) ...
struct SegKeys {
  dgs_segments s;
  int64_t n;
  __device__ __forceinline__ int64_t size() const { return n; }
  __device__ __forceinline__ int64_t bound() const { return n; }
  template <typename IdT>
  __device__ __forceinline__ IdT load(int64_t i) const {
    return seg_load<IdT>(s, i);
  }
};
// ... or two arrays a[0:na) ++ b[0:nb) whose lengths are device words (the
// multi-hop sequence: a = this hop's seeds, b = the neighbours just sampled).
struct PairKeys {
  const void* a;
  const void* b;
  Count na, nb;
  __device__ __forceinline__ int64_t size() const { return count_of(na) + count_of(nb); }
  __device__ __forceinline__ int64_t bound() const { return na.bound + nb.bound; }
  template <typename IdT>
  __device__ __forceinline__ IdT load(int64_t i) const {
    const int64_t x = count_of(na);
    return i < x ? static_cast<const IdT*>(a)[i] : static_cast<const IdT*>(b)[i - x];
  }
};

// Insert key (input i), keeping the smallest input index per key: its slot, NO_SLOT for a key out of range or a full table.
template <typename IdT, typename Keys>
__device__ __forceinline__ uint32_t insert_key(const Keys& keys, const TableSize& size, unsigned long long* words, int64_t i,
                                               long long key, int32_t* status) {
  if (key < 0 || key > size.max_key) {
    raise_status(status, DGS_ERR_RANGE);
    return NO_SLOT;
  }
  const uint32_t mask32 = static_cast<uint32_t>(table_slots(size) - 1), key32 = static_cast<uint32_t>(key);
  const uint32_t flag = is_wide(key) ? WIDE_BIT32 : 0u;
  const unsigned long long mine =
      (static_cast<unsigned long long>(key32) << 32) | static_cast<unsigned long long>(flag | static_cast<uint32_t>(i));
  uint32_t found = NO_SLOT;
  uint32_t h = home_slot(key, mask32);
  for (uint32_t probes = 0; probes <= mask32; ++probes) {
    unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(&words[h]);
    if (cur == EMPTY_WORD) {
      cur = atomicCAS(&words[h], EMPTY_WORD, mine);
      if (cur == EMPTY_WORD) {  // claimed, and the first index is in place: nothing else to do
        found = h;
        break;
      }
    }
    const uint32_t low = static_cast<uint32_t>(cur);
    if (static_cast<uint32_t>(cur >> 32) == key32 && (low & WIDE_BIT32) == flag &&
        (flag == 0u || static_cast<long long>(keys.template load<IdT>(low & VALUE_MASK32)) == key)) {
      found = h;
      // same high half and flag, so the minimum of the words is the minimum of the indices; a stale read can only
      // cause a redundant atomic (indices only ever decrease)
      if (cur > mine) atomicMin(&words[h], mine);
      break;
    }
    h = (h + 1) & mask32;
  }
  if (found == NO_SLOT) raise_status(status, DGS_ERR_TABLE_FULL);
  return found;
}

// pass 1: insert every key
template <typename IdT, typename Keys>
__global__ void __launch_bounds__(RL_BLOCK)
relabel_insert_kernel(const __grid_constant__ Keys keys, const TableSize size, unsigned long long* words,
                      uint32_t* __restrict__ slot_of, int32_t* __restrict__ status) {
  pdl_enter();
  const int64_t n = keys.size();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * RL_BLOCK + threadIdx.x;
  if (i >= n) return;
  slot_of[i] = insert_key<IdT>(keys, size, words, i, static_cast<long long>(keys.template load<IdT>(i)), status);
}

// ---- the operator's passes over many keys --------------------------------------
// The operator's keys are node ids, and a large mini-batch holds a good part of a graph's: when every key is below the
// number of 32-bit words that the slots have, the words serve as one per id, addressed by the key (see IdMarks), and
// nothing is hashed, probed or remembered per input.  Which it is shows on the device: the pass that clears the table
// reads the keys too.  One hop of 60 000 seeds and fan-out 15, sampled and relabelled: 105.8 -> 94.7 us.
// Relabel calls, us, without -> with the look; keys that the words can address / too large and half of them distinct / too
// large and all distinct: 524 k 55 -> 42.5 / 49 -> 49 / 62 -> 61, 600 k 50 -> 37 / 42.7 -> 45.2 / 56 -> 55, 880 k 63 -> 43 / 54.7 -> 54.3 /
// 74 -> 72, 1.2 M 84 -> 62 / 75.6 -> 76.2 / 95 -> 93, 1.6 M 110 -> 76 / 90.9 -> 91.3 / 118 -> 117, 2.09 M 139 -> 97 / 114 -> 117.5 / 157 -> 158.
// Unique and lookup by themselves outside the range, with the look as it was at first: 180 k 26.5 -> 19.6 and 28 -> 31, 360 k
// 39 -> 27 and 41 -> 45, 3 M 180 -> 141 and 218 -> 233.  Hence the range: below, a graph is seldom small enough to make up for
// the others, above it the look costs them too much.
constexpr int64_t LOOK_MIN_KEYS = 1ll << 19, LOOK_MAX_KEYS = 1ll << 21;
inline bool looks_at_largest(int64_t n) { return n >= LOOK_MIN_KEYS && n < LOOK_MAX_KEYS; }
// CTAs that read the keys; no more than the range has tiles.  (With half as many, and the stores behind the reads, keys that are
// too large paid 2 us more from 1.6 M on.)
constexpr int LARGEST = 2 * RL_BLOCK;
static_assert(LARGEST <= LOOK_MIN_KEYS / RL_TILE, "a word per tile is their room");

template <typename IdT>
__global__ void __launch_bounds__(RL_BLOCK)
relabel_clear_kernel(const __grid_constant__ SegKeys keys, ulonglong2* __restrict__ units, const int64_t n_units,
                     unsigned long long* __restrict__ largest) {
  __shared__ unsigned long long s_max[RL_BLOCK / 32];
  pdl_enter();
  const ulonglong2 ones = make_ulonglong2(~0ull, ~0ull);
#pragma unroll 4
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * RL_BLOCK + threadIdx.x; i < n_units; i += static_cast<int64_t>(gridDim.x) * RL_BLOCK)
    units[i] = ones;
  if (blockIdx.x >= LARGEST) return;
  unsigned long long most = 0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * RL_TILE + threadIdx.x; i < keys.n; i += static_cast<int64_t>(LARGEST) * RL_TILE) {
    unsigned long long k[RL_ITEMS];
#pragma unroll
    for (int u = 0; u < RL_ITEMS; ++u)
      k[u] = i + u * RL_BLOCK < keys.n
                 ? static_cast<unsigned long long>(static_cast<long long>(keys.template load<IdT>(i + u * RL_BLOCK)))
                 : 0ull;
#pragma unroll
    for (int u = 0; u < RL_ITEMS; ++u) most = k[u] > most ? k[u] : most;  // a negative key is larger than any id
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(FULL_MASK, most, o);
    most = other > most ? other : most;
  }
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = most;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < RL_BLOCK / 32; ++w) most = s_max[w] > most ? s_max[w] : most;
    largest[blockIdx.x] = most;
  }
}

// mark every key in its word, or insert it in the hash table
template <typename IdT>
__global__ void __launch_bounds__(RL_BLOCK)
relabel_mark_kernel(const __grid_constant__ SegKeys keys, const TableSize size, const __grid_constant__ TableParts t,
                    int32_t* __restrict__ status) {
  pdl_enter();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * RL_BLOCK + threadIdx.x;
  const long long key = i < keys.n ? static_cast<long long>(keys.template load<IdT>(i)) : 0;
  const uint64_t words = 2 * table_slots(size);
  static_assert(LARGEST == 2 * RL_BLOCK, "two words a thread");
  const bool dense = !__syncthreads_or(t.largest[threadIdx.x] >= words || t.largest[threadIdx.x + RL_BLOCK] >= words);
  if (i == 0) *t.dense = dense;
  if (i >= keys.n) return;
  if (dense) atomicMin(reinterpret_cast<uint32_t*>(t.words) + key, static_cast<uint32_t>(i));
  else t.slot_of[i] = insert_key<IdT>(keys, size, t.words, i, key, status);
}

// count and number, as dense_number_kernel, over either form of the table
template <typename IdT>
__global__ void __launch_bounds__(RL_BLOCK, 6)
relabel_number_any_kernel(const __grid_constant__ SegKeys keys, const __grid_constant__ TableParts t, IdT* __restrict__ unique_out,
                          int64_t* n_unique_out, int32_t* __restrict__ status) {
  __shared__ TileScanShared<RL_BLOCK> s_tiles;
  __shared__ unsigned int s_tile;
  __shared__ int s_count[RL_BLOCK / 32];
  pdl_enter();
  if (threadIdx.x == 0) s_tile = atomicAdd(t.ticket, 1u) + 1u;
  const int64_t form = *t.dense;
  __syncthreads();
  const int64_t tile = s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = tile * RL_TILE + warp * 32 * RL_ITEMS + lane;
  long long key[RL_ITEMS];
  uint32_t slot[RL_ITEMS];
  // both are read while the word that says which counts is on its way
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    const int64_t i = base + 32 * u;
    key[u] = i < keys.n ? static_cast<long long>(keys.template load<IdT>(i)) : 0;
    slot[u] = i < keys.n ? t.slot_of[i] : NO_SLOT;  // nothing of meaning when dense
  }
  const bool dense = form != 0;
  uint32_t* at[RL_ITEMS];  // the word of each input's key
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u)
    at[u] = base + 32 * u >= keys.n ? nullptr
            : dense                 ? reinterpret_cast<uint32_t*>(t.words) + key[u]
            : slot[u] != NO_SLOT    ? reinterpret_cast<uint32_t*>(t.words + slot[u])
                                    : nullptr;
  uint32_t word[RL_ITEMS];
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) word[u] = at[u] != nullptr ? *static_cast<const volatile uint32_t*>(at[u]) : NOT_MET;
  unsigned votes[RL_ITEMS];
  int c = 0;
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    // a word that carries a label already (LABEL_BIT32) cannot equal an input
    votes[u] = __ballot_sync(FULL_MASK, at[u] != nullptr && (word[u] & ~WIDE_BIT32) == static_cast<uint32_t>(base + 32 * u));
    c += __popc(votes[u]);
  }
  if (lane == 0) s_count[warp] = c;
  __syncthreads();
  int ex = 0, total = 0;
#pragma unroll
  for (int w = 0; w < RL_BLOCK / 32; ++w) {
    if (w < warp) ex += s_count[w];
    total += s_count[w];
  }
  const int64_t before = sum_of_tiles_before<RL_BLOCK>(tile, total, t.tiles, s_tiles, status);
  if (tile == t.ntiles - 1 && threadIdx.x == 0) {
    *t.total = before + total;
    if (n_unique_out != nullptr) {
      *n_unique_out = before + total;
      __threadfence_system();
    }
  }
  int64_t next = before + ex;
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    const int64_t label = next + __popc(votes[u] & ((1u << lane) - 1u));
    next += __popc(votes[u]);
    if (((votes[u] >> lane) & 1u) == 0u) continue;
    unique_out[label] = static_cast<IdT>(key[u]);  // at most as many as inputs
    uint32_t flag = 0u;
    if (is_wide(key[u])) {
      flag = WIDE_BIT32;
      t.wide_keys[label] = key[u];
    }
    *at[u] = LABEL_BIT32 | flag | static_cast<uint32_t>(label);
  }
}

// label of each id over either form, -1 when absent
template <typename IdT>
__global__ void __launch_bounds__(RL_BLOCK)
relabel_lookup_any_kernel(const __grid_constant__ dgs_segments in, const int64_t n, const __grid_constant__ TableParts t,
                          const uint64_t mask, IdT* __restrict__ out) {
  pdl_enter();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * RL_BLOCK + threadIdx.x;
  if (i >= n) return;
  const int64_t dense = *t.dense;
  const long long id = static_cast<long long>(seg_load<IdT>(in, i));
  if (dense == 0) {
    out[i] = static_cast<IdT>(probe_label(t.words, t.wide_keys, mask, id));
    return;
  }
  const uint32_t word = static_cast<uint64_t>(id) < 2 * (mask + 1) ? reinterpret_cast<const uint32_t*>(t.words)[id] : NOT_MET;
  out[i] = word == NOT_MET ? static_cast<IdT>(-1) : static_cast<IdT>(word & VALUE_MASK32);
}

template <typename IdT>
int run_unique_any(const SegKeys& keys, const TableParts& t, void* unique_out, int64_t* n_unique, int32_t* status, cudaStream_t s) {
  const TableSize size{exact_count(keys.n), 1, INT64_MAX};
  // slots, ticket and tile words lie one behind the other
  const int64_t units = static_cast<int64_t>(slots_for(keys.n) / 2) + ticket_units(t);
  DGS_CUDA_TRY(launch_chained(SITE_INIT, relabel_clear_kernel<IdT>, 2u * LARGEST, RL_BLOCK, s, keys,
                              reinterpret_cast<ulonglong2*>(t.words), units, t.largest));
  DGS_CUDA_TRY(launch_chained(SITE_INSERT, relabel_mark_kernel<IdT>, static_cast<unsigned>((keys.n + RL_BLOCK - 1) / RL_BLOCK),
                              RL_BLOCK, s, keys, size, t, status));
  DGS_CUDA_TRY(launch_chained(SITE_NUMBER, relabel_number_any_kernel<IdT>, static_cast<unsigned>(t.ntiles), RL_BLOCK, s, keys, t,
                              static_cast<IdT*>(unique_out), n_unique, status));
  return DGS_OK;
}

// pass 2: input i is a first occurrence iff the stored minimum equals i.  A tile counts its first occurrences, learns
// from the tiles before it where its labels begin, emits the keys and stores the labels in the slots; the last tile
// publishes the number of distinct keys.
// With a plan (n_edges != nullptr; the multi-hop sequence), the tile then reads the row bounds of the nodes it has
// numbered -- they are the next hop's seeds -- and a second look-back places their outputs, so that the next hop needs
// no plan launch.
// Bound by dependent L2 round trips (slot, word, look-back, row bounds, second look-back), a tile's worth of keys per
// CTA so that a mini-batch's tiles are all in flight together.  Counting, numbering and planning in launches of their
// own (three per hop) a batch of 1 024 seeds and 826 k edges took 153 us of sampling sequence, this way 135 us; 880 k
// keys by themselves 26 us for count + number, now 21.
template <typename IdT, typename Keys, bool PLAN>
__global__ void __launch_bounds__(RL_BLOCK)
relabel_number_kernel(const __grid_constant__ Keys keys, const TableParts t, IdT* __restrict__ unique_out,
                      const int64_t unique_capacity, int64_t* n_unique_out, const SizesReport report,
                      const __grid_constant__ NextPlan plan, int32_t* __restrict__ status) {
  __shared__ int64_t smem[RL_BLOCK / 32 + 1];
  __shared__ TileScanShared<RL_BLOCK> s_tiles;
  __shared__ unsigned int s_tile;
  pdl_enter();
  if (threadIdx.x == 0) s_tile = atomicAdd(t.ticket, 1u) + 1u;
  __syncthreads();
  const int64_t tile = s_tile;
  const int64_t base = tile * RL_TILE + threadIdx.x * RL_ITEMS;
  const int64_t room = keys.bound();
  uint32_t slot[RL_ITEMS] = {NO_SLOT, NO_SLOT, NO_SLOT, NO_SLOT};
  if (base < room) {  // ahead of the count; the array is padded to 16 bytes
    const uint4 v = *reinterpret_cast<const uint4*>(t.slot_of + base);
    slot[0] = v.x;
    slot[1] = v.y;
    slot[2] = v.z;
    slot[3] = v.w;
  }
  const int64_t n = keys.size();
  if (tile > 0 && tile * RL_TILE >= n) return;  // past the live keys
  const bool last_tile = (tile + 1) * RL_TILE >= n;
  bool first[RL_ITEMS];
  int c = 0;
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    const int64_t i = base + u;
    // a slot already relabelled by another CTA carries LABEL_BIT32 and cannot equal i
    first[u] = i < n && slot[u] != NO_SLOT &&
               (*reinterpret_cast<const volatile uint32_t*>(reinterpret_cast<const uint2*>(t.words) + slot[u]) &
                ~WIDE_BIT32) == static_cast<uint32_t>(i);
    c += first[u] ? 1 : 0;
  }
  int64_t total;
  const int64_t ex = block_exclusive_scan<int64_t, RL_BLOCK>(c, smem, &total);
  const int64_t before = sum_of_tiles_before<RL_BLOCK>(tile, total, t.tiles, s_tiles, status);
  if (last_tile && threadIdx.x == 0) {
    *t.total = before + total;
    if (n_unique_out != nullptr) {
      *n_unique_out = before + total;
      __threadfence_system();
    }
    if (report.n > 0) report_sizes(report.dst, report.src, report.n, 0, status);  // the same thread that wrote *t.total
  }
  int64_t label = before + ex;
  int64_t id[RL_ITEMS];
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    id[u] = -1;
    if (first[u]) {
      const IdT key = keys.template load<IdT>(base + u);
      if (label < unique_capacity) {
        unique_out[label] = key;
        id[u] = static_cast<int64_t>(key);
      } else {
        raise_status(status, DGS_ERR_RANGE);
      }
      uint32_t flag = 0u;
      if (is_wide(static_cast<long long>(key))) {
        flag = WIDE_BIT32;
        t.wide_keys[label] = static_cast<long long>(key);
      }
      reinterpret_cast<uint2*>(t.words)[slot[u]].x = LABEL_BIT32 | flag | static_cast<uint32_t>(label);
      ++label;
    }
  }
  if (!PLAN) return;
  label = before + ex;
  int64_t rb[RL_ITEMS], deg[RL_ITEMS], cnt = 0;
  bool good[RL_ITEMS];
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    good[u] = id[u] >= 0 && id[u] + 1 < plan.indptr.total;
    if (id[u] >= 0 && !good[u]) raise_status(status, DGS_ERR_RANGE);
  }
  row_bounds<IdT, RL_ITEMS>(plan.indptr, id, good, rb, deg, status);
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) cnt += pick_count(deg[u], plan.k, plan.replace);
  int64_t tile_edges;
  int64_t at = block_exclusive_scan<int64_t, RL_BLOCK>(cnt, smem, &tile_edges);
  at += sum_of_tiles_before<RL_BLOCK>(tile, tile_edges, t.tiles2, s_tiles, status);
  if (last_tile && threadIdx.x == RL_BLOCK - 1) *plan.n_edges = at + cnt;
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    if (!first[u]) continue;
    if (id[u] >= 0) {  // the list has room for it
      plan.row_begin[label] = rb[u];
      plan.deg[label] = deg[u];
      plan.off[label] = at;
    }
    at += pick_count(deg[u], plan.k, plan.replace);
    ++label;
  }
}

// The numbering of a sequence that keeps one word per id (see IdMarks): input i -- the seeds, then the neighbours in the
// order they were drawn -- is a first occurrence iff the word of its id holds i.  The sampling launch has put the smallest
// index there, so nothing was probed, and a tile reads its ids, their words, and is where relabel_number_kernel is.
// Seeds and neighbours have tiles of their own; seeds that are labelled already (their label is their position) need
// no word and no look-back.  A warp owns 128 consecutive inputs, 32 at a time, so that ids are read in whole lines and ranks
// come out of votes.
template <typename IdT, bool PLAN>
__global__ void __launch_bounds__(RL_BLOCK)
dense_number_kernel(const DenseNumbering d, const IdT* __restrict__ seeds, const Count na, const IdT* __restrict__ cols,
                    const Count nb, IdT* __restrict__ unique_out, const int64_t unique_capacity, const SizesReport report,
                    const __grid_constant__ NextPlan plan, int32_t* __restrict__ status) {
  __shared__ int64_t smem[RL_BLOCK / 32 + 1];
  __shared__ TileScanShared<RL_BLOCK> s_tiles;
  __shared__ unsigned int s_tile;
  __shared__ int s_count[RL_BLOCK / 32];
  pdl_enter();
  if (threadIdx.x == 0) s_tile = atomicAdd(d.ticket, 1u) + 1u;
  const int64_t n_seeds = count_of(na), n_cols = count_of(nb);
  const bool beyond = report.n > 0 && threadIdx.x == 0 && *static_cast<const volatile uint32_t*>(d.beyond) != NOT_MET;
  __syncthreads();
  const int64_t tile = s_tile;
  const int64_t seed_tiles = (n_seeds + RL_TILE - 1) / RL_TILE, tiles = seed_tiles + (n_cols + RL_TILE - 1) / RL_TILE;
  const bool last_tile = tile == tiles - 1 || (tile == 0 && tiles == 0);
  if (tile >= tiles && !last_tile) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool of_seeds = tile < seed_tiles;
  const bool known = of_seeds && d.seeds_known;
  const IdT* list = of_seeds ? seeds : cols;
  const int64_t list_len = of_seeds ? n_seeds : n_cols, list_at = of_seeds ? 0 : n_seeds;
  const int64_t base = (of_seeds ? tile : tile - seed_tiles) * RL_TILE + warp * 32 * RL_ITEMS + lane;  // in the list
  int64_t id[RL_ITEMS];
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) id[u] = base + 32 * u < list_len ? static_cast<int64_t>(list[base + 32 * u]) : -1;
  uint32_t word[RL_ITEMS];
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    const bool in = static_cast<uint64_t>(id[u]) < static_cast<uint64_t>(d.ids);
    word[u] = !in ? NOT_MET : known ? static_cast<uint32_t>(base + 32 * u) : load_kept(d.first + id[u], l2_evict_last_policy());
  }
  unsigned votes[RL_ITEMS];
  int c = 0;
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    votes[u] = __ballot_sync(FULL_MASK, word[u] == static_cast<uint32_t>(list_at + base + 32 * u) && word[u] != NOT_MET);
    c += __popc(votes[u]);
  }
  if (lane == 0) s_count[warp] = c;
  __syncthreads();
  int ex = 0, total = 0;
#pragma unroll
  for (int w = 0; w < RL_BLOCK / 32; ++w) {
    if (w < warp) ex += s_count[w];
    total += s_count[w];
  }
  int64_t before;
  if (known) {
    before = tile * RL_TILE;
    if (threadIdx.x == 0) store_tile_word(d.tiles + tile, TILE_RUNNING | static_cast<unsigned long long>(before + total));
  } else {
    before = sum_of_tiles_before<RL_BLOCK>(tile, total, d.tiles, s_tiles, status);
  }
  if (last_tile && threadIdx.x == 0) {
    *d.total = before + total;
    // the same thread that wrote *d.total just above
    if (report.n > 0) report_sizes(report.dst, report.src, report.n, beyond ? DGS_ERR_ID_SPACE : 0, status);
  }
  int64_t label[RL_ITEMS];
  int64_t next = before + ex;
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    const bool first = (votes[u] >> lane) & 1u;
    label[u] = next + __popc(votes[u] & ((1u << lane) - 1u));
    next += __popc(votes[u]);
    if (first) {
      if (!known) store_kept(d.first + id[u], static_cast<uint32_t>(label[u]), l2_evict_last_policy());
      if (label[u] < unique_capacity) {
        unique_out[label[u]] = static_cast<IdT>(id[u]);
      } else {
        raise_status(status, DGS_ERR_RANGE);
        id[u] = -1;
      }
    } else {
      id[u] = -1;
    }
  }
  if (!PLAN) return;
  int64_t rb[RL_ITEMS], deg[RL_ITEMS], off[RL_ITEMS], warp_edges = 0;
  bool good[RL_ITEMS];
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    good[u] = id[u] >= 0 && id[u] + 1 < plan.indptr.total;
    if (id[u] >= 0 && !good[u]) raise_status(status, DGS_ERR_RANGE);
  }
  row_bounds<IdT, RL_ITEMS>(plan.indptr, id, good, rb, deg, status);
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    const int64_t n = pick_count(deg[u], plan.k, plan.replace);
    int64_t inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(FULL_MASK, inc, o);
      if (lane >= o) inc += t;
    }
    off[u] = warp_edges + inc - n;
    warp_edges += __shfl_sync(FULL_MASK, inc, 31);
  }
  if (lane == 0) smem[warp] = warp_edges;
  __syncthreads();
  int64_t at = 0, tile_edges = 0;
#pragma unroll
  for (int w = 0; w < RL_BLOCK / 32; ++w) {
    if (w < warp) at += smem[w];
    tile_edges += smem[w];
  }
  const int64_t edges_before = sum_of_tiles_before<RL_BLOCK>(tile, tile_edges, d.tiles + gridDim.x, s_tiles, status);
  if (last_tile && threadIdx.x == 0) *plan.n_edges = edges_before + tile_edges;
#pragma unroll
  for (int u = 0; u < RL_ITEMS; ++u) {
    if (id[u] < 0) continue;
    plan.row_begin[label[u]] = rb[u];
    plan.deg[label[u]] = deg[u];
    plan.off[label[u]] = edges_before + at + off[u];
  }
}

// The COO of all hops through that table, in place: an id that is not in it becomes -1.  Bound by the random reads of
// the words; four ids per thread in flight.
template <typename IdT>
__global__ void __launch_bounds__(RL_BLOCK) dense_lookup_kernel(const __grid_constant__ DenseLookup job) {
  pdl_enter();
  int h = 0;
  while (h + 1 < job.n_hops && blockIdx.x >= job.end_cta[h]) ++h;
  const int64_t base = static_cast<int64_t>(blockIdx.x - (h > 0 ? job.end_cta[h - 1] : 0u)) * RL_TILE + threadIdx.x;
  const int64_t n = count_of(job.n[h]);
  auto relabel = [&](IdT* ids) {
    int64_t id[RL_ITEMS];
    uint32_t word[RL_ITEMS];
#pragma unroll
    for (int u = 0; u < RL_ITEMS; ++u) id[u] = base + u * RL_BLOCK < n ? static_cast<int64_t>(ids[base + u * RL_BLOCK]) : -1;
#pragma unroll
    for (int u = 0; u < RL_ITEMS; ++u)
      word[u] = static_cast<uint64_t>(id[u]) < static_cast<uint64_t>(job.ids) ? load_kept(job.first + id[u], l2_evict_last_policy()) : NOT_MET;
#pragma unroll
    for (int u = 0; u < RL_ITEMS; ++u)
      if (base + u * RL_BLOCK < n) ids[base + u * RL_BLOCK] = word[u] == NOT_MET ? static_cast<IdT>(-1) : static_cast<IdT>(word[u]);
  };
  relabel(static_cast<IdT*>(job.col[h]));
  if (h == 0) relabel(static_cast<IdT*>(job.row0));
}

// lookup: label of each id, -1 when absent
template <typename IdT>
__global__ void __launch_bounds__(RL_BLOCK)
relabel_lookup_kernel(const __grid_constant__ dgs_segments in, const int64_t n,
                      const unsigned long long* __restrict__ words, const long long* __restrict__ wide_keys,
                      const uint64_t mask, IdT* __restrict__ out) {
  pdl_enter();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * RL_BLOCK + threadIdx.x;
  if (i >= n) return;
  out[i] = static_cast<IdT>(probe_label(words, wide_keys, mask, static_cast<long long>(seg_load<IdT>(in, i))));
}

// lookup of the sequence with device-side counts, when it does not ride on another launch
template <typename IdT>
__global__ void __launch_bounds__(RL_BLOCK) relabel_lookup_pair_kernel(const LookupJob job) {
  pdl_enter();
  run_lookup_cta<IdT>(job, blockIdx.x);
}

inline int64_t seg_total(const dgs_segments& s) {
  int64_t t = 0;
  for (int i = 0; i < s.count; ++i) t += s.len[i];
  return t;
}

int check_segments(const dgs_segments* s, const char* who) {
  DGS_REQUIRE(s != nullptr && s->count >= 0 && s->count <= DGS_MAX_SEGMENTS, DGS_ERR_INVALID,
              "%s: bad segment list", who);
  for (int i = 0; i < s->count; ++i)
    DGS_REQUIRE(s->len[i] >= 0 && (s->len[i] == 0 || s->ptr[i] != nullptr), DGS_ERR_INVALID,
                "%s: segment %d is null", who, i);
  return DGS_OK;
}

__global__ void zero_word_kernel(int64_t* w) { *w = 0; }

// insert -> number over a cleared table; the bounds size the grids
template <typename IdT, typename Keys>
int run_unique(const Keys& keys, int64_t n_bound, const TableSize& size, const TableParts& t, void* unique_out,
               int64_t unique_capacity, int64_t* n_unique, const SizesReport& report, const NextPlan& plan,
               int32_t* status, cudaStream_t s) {
  const unsigned per_key_grid = static_cast<unsigned>((n_bound + RL_BLOCK - 1) / RL_BLOCK);
  DGS_CUDA_TRY(launch_chained(SITE_INSERT, relabel_insert_kernel<IdT, Keys>, per_key_grid, RL_BLOCK, s, keys, size, t.words,
                              t.slot_of, status));
  if constexpr (std::is_same<Keys, PairKeys>::value) {
    if (plan.n_edges != nullptr) {
      DGS_CUDA_TRY(launch_chained(SITE_NUMBER, relabel_number_kernel<IdT, Keys, true>, static_cast<unsigned>(t.ntiles),
                                  RL_BLOCK, s, keys, t, static_cast<IdT*>(unique_out), unique_capacity, n_unique, report,
                                  plan, status));
      return DGS_OK;
    }
  }
  DGS_CUDA_TRY(launch_chained(SITE_NUMBER, relabel_number_kernel<IdT, Keys, false>, static_cast<unsigned>(t.ntiles), RL_BLOCK,
                              s, keys, t, static_cast<IdT*>(unique_out), unique_capacity, n_unique, report, plan, status));
  return DGS_OK;
}

}  // namespace

int64_t* unique_total(void* table, int64_t key_bound) { return table_view(table, key_bound).total; }

ClearJob make_clear_job(void* table, int64_t key_bound, const TableSize& size) {
  const TableParts t = table_view(table, key_bound);
  const int64_t units = static_cast<int64_t>(slots_for(key_bound) / 2) + ticket_units(t);
  return ClearJob{t.words, t.ticket, ticket_units(t), size,
                  static_cast<unsigned>((units + CLEAR_UNITS_PER_CTA - 1) / CLEAR_UNITS_PER_CTA)};
}

LookupJob make_lookup_job(void* table, int64_t key_bound, const TableSize& size, void* row, void* col, Count n,
                          Count n_seeds) {
  const TableParts t = table_view(table, key_bound);
  return LookupJob{row, col, n, n_seeds, t.words, t.slot_of, t.wide_keys, size,
                   static_cast<unsigned>((n.bound + RL_BLOCK - 1) / RL_BLOCK)};
}

int launch_unique_pair(bool ids64, const void* a, Count na, const void* b, Count nb, int64_t key_bound,
                       const TableSize& size, void* table, void* unique_out, int64_t unique_capacity,
                       int64_t* n_unique_out, const SizesReport& report, const NextPlan& plan, int32_t* status,
                       cudaStream_t s) {
  DGS_REQUIRE(key_bound > 0 && key_bound < (1ll << 30) && na.bound + nb.bound <= key_bound, DGS_ERR_UNSUPPORTED,
              "relabel: %lld keys", (long long)key_bound);
  DGS_REQUIRE(na.dev != nullptr && nb.dev != nullptr, DGS_ERR_INVALID, "relabel: the pair form takes a device word per length");
  const TableParts t = table_view(table, key_bound);
  const PairKeys keys{a, b, na, nb};
  return ids64 ? run_unique<int64_t, PairKeys>(keys, key_bound, size, t, unique_out, unique_capacity, n_unique_out,
                                               report, plan, status, s)
               : run_unique<int32_t, PairKeys>(keys, key_bound, size, t, unique_out, unique_capacity, n_unique_out,
                                               report, plan, status, s);
}

int launch_dense_number(bool ids64, const DenseNumbering& d, const void* seeds, Count n_seeds, const void* cols, Count n_cols,
                        void* unique_out, int64_t unique_capacity, const SizesReport& report, const NextPlan& plan,
                        int32_t* status, cudaStream_t s) {
  const int64_t tiles = dense_tiles(n_seeds.bound, n_cols.bound);
  DGS_REQUIRE(tiles > 0 && n_seeds.bound + n_cols.bound < (1ll << 30), DGS_ERR_UNSUPPORTED, "relabel: %lld keys",
              (long long)(n_seeds.bound + n_cols.bound));
  const unsigned grid = static_cast<unsigned>(tiles);
#define DGS_LAUNCH_DENSE(IdT, PLAN)                                                                                     \
  DGS_CUDA_TRY(launch_chained(SITE_NUMBER, (dense_number_kernel<IdT, PLAN>), grid, RL_BLOCK, s, d,                      \
                              static_cast<const IdT*>(seeds), n_seeds, static_cast<const IdT*>(cols), n_cols,           \
                              static_cast<IdT*>(unique_out), unique_capacity, report, plan, status))
  if (plan.n_edges != nullptr) {
    if (ids64) DGS_LAUNCH_DENSE(int64_t, true);
    else DGS_LAUNCH_DENSE(int32_t, true);
  } else {
    if (ids64) DGS_LAUNCH_DENSE(int64_t, false);
    else DGS_LAUNCH_DENSE(int32_t, false);
  }
#undef DGS_LAUNCH_DENSE
  return DGS_OK;
}

int launch_dense_lookup(const DenseLookup& job, bool ids64, cudaStream_t s) {
  const unsigned grid = job.end_cta[job.n_hops - 1];
  if (grid == 0) return DGS_OK;
  if (ids64) DGS_CUDA_TRY(launch_chained(SITE_LOOKUP, dense_lookup_kernel<int64_t>, grid, RL_BLOCK, s, job));
  else DGS_CUDA_TRY(launch_chained(SITE_LOOKUP, dense_lookup_kernel<int32_t>, grid, RL_BLOCK, s, job));
  return DGS_OK;
}

int launch_lookup(const LookupJob& job, bool ids64, cudaStream_t s) {
  if (job.ctas == 0) return DGS_OK;
  if (ids64) DGS_CUDA_TRY(launch_chained(SITE_LOOKUP, relabel_lookup_pair_kernel<int64_t>, job.ctas, RL_BLOCK, s, job));
  else DGS_CUDA_TRY(launch_chained(SITE_LOOKUP, relabel_lookup_pair_kernel<int32_t>, job.ctas, RL_BLOCK, s, job));
  return DGS_OK;
}

}  // namespace dgs

extern "C" size_t dgs_relabel_table_bytes(int64_t n) {
  using namespace dgs;
  if (n < 0) n = 0;
  const int64_t ntiles = (n + RL_TILE - 1) / RL_TILE;
  return 2 * slots_for(n) * sizeof(unsigned long long) + align_up(static_cast<size_t>(n) * sizeof(uint32_t), 16) +
         static_cast<size_t>(ntiles + 2) * sizeof(int64_t);
}

extern "C" int dgs_unique_first_occurrence(const dgs_segments* keys, int32_t ids64, void* table,
                                           size_t table_bytes, void* unique_out, int64_t* n_unique,
                                           int32_t* status, dgs_stream_t stream) {
  using namespace dgs;
  int rc = check_segments(keys, "dgs_unique_first_occurrence");
  if (rc != DGS_OK) return rc;
  const int64_t n = seg_total(*keys);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  DGS_REQUIRE(table != nullptr && table_bytes >= dgs_relabel_table_bytes(n), DGS_ERR_INVALID,
              "dgs_unique_first_occurrence: table scratch too small (%zu < %zu)", table_bytes,
              dgs_relabel_table_bytes(n));
  DGS_REQUIRE((reinterpret_cast<uintptr_t>(table) & 15) == 0, DGS_ERR_INVALID,
              "dgs_unique_first_occurrence: table must be 16-byte aligned");
  DGS_REQUIRE(n < (1ll << 30), DGS_ERR_UNSUPPORTED, "dgs_unique_first_occurrence: %lld keys", (long long)n);
  const TableParts t = table_view(table, n);
  if (looks_at_largest(n)) {
    DGS_REQUIRE(unique_out != nullptr, DGS_ERR_INVALID, "dgs_unique_first_occurrence: null output");
    const SegKeys many{*keys, n};
    return ids64 ? run_unique_any<int64_t>(many, t, unique_out, n_unique, status, s)
                 : run_unique_any<int32_t>(many, t, unique_out, n_unique, status, s);
  }
  // slots, ticket and tile words lie one behind the other
  DGS_CUDA_TRY(cudaMemsetAsync(table, 0xFF, slots_for(n) * sizeof(unsigned long long) + ticket_units(t) * 16, s));
  if (n == 0) {
    if (n_unique != nullptr) {
      zero_word_kernel<<<1, 1, 0, s>>>(n_unique);
      DGS_LAUNCH_CHECK();
    }
    return DGS_OK;
  }
  DGS_REQUIRE(unique_out != nullptr, DGS_ERR_INVALID, "dgs_unique_first_occurrence: null output");
  const SegKeys sk{*keys, n};
  const TableSize size{exact_count(n), 1, INT64_MAX};
  return ids64 ? run_unique<int64_t, SegKeys>(sk, n, size, t, unique_out, n, n_unique, SizesReport{}, NextPlan{}, status, s)
               : run_unique<int32_t, SegKeys>(sk, n, size, t, unique_out, n, n_unique, SizesReport{}, NextPlan{}, status, s);
}

extern "C" int dgs_relabel_lookup(const void* table, size_t table_bytes, int64_t n_keys_built,
                                  const dgs_segments* in, int32_t ids64, void* out,
                                  dgs_stream_t stream) {
  using namespace dgs;
  int rc = check_segments(in, "dgs_relabel_lookup");
  if (rc != DGS_OK) return rc;
  const int64_t n = seg_total(*in);
  if (n == 0) return DGS_OK;
  DGS_REQUIRE(table != nullptr && n_keys_built >= 0 && table_bytes >= dgs_relabel_table_bytes(n_keys_built),
              DGS_ERR_INVALID, "dgs_relabel_lookup: bad table");
  DGS_REQUIRE(out != nullptr, DGS_ERR_INVALID, "dgs_relabel_lookup: null output");
  DGS_REQUIRE((n + RL_BLOCK - 1) / RL_BLOCK <= 0x7fffffffLL, DGS_ERR_UNSUPPORTED, "dgs_relabel_lookup: too many ids");
  const TableParts t = table_view(const_cast<void*>(table), n_keys_built);
  const uint64_t mask = slots_for(n_keys_built) - 1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const unsigned grid = static_cast<unsigned>((n + RL_BLOCK - 1) / RL_BLOCK);
  if (looks_at_largest(n_keys_built)) {
    if (ids64)
      DGS_CUDA_TRY(launch_chained(SITE_LOOKUP, relabel_lookup_any_kernel<int64_t>, grid, RL_BLOCK, s, *in, n, t, mask,
                                  static_cast<int64_t*>(out)));
    else
      DGS_CUDA_TRY(launch_chained(SITE_LOOKUP, relabel_lookup_any_kernel<int32_t>, grid, RL_BLOCK, s, *in, n, t, mask,
                                  static_cast<int32_t*>(out)));
    return DGS_OK;
  }
  if (ids64)
    DGS_CUDA_TRY(launch_chained(SITE_LOOKUP, relabel_lookup_kernel<int64_t>, grid, RL_BLOCK, s, *in, n, t.words, t.wide_keys,
                                mask, static_cast<int64_t*>(out)));
  else
    DGS_CUDA_TRY(launch_chained(SITE_LOOKUP, relabel_lookup_kernel<int32_t>, grid, RL_BLOCK, s, *in, n, t.words, t.wide_keys,
                                mask, static_cast<int32_t*>(out)));
  return DGS_OK;
}
