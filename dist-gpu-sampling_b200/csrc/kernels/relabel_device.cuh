// Device-side pieces of the relabel table that more than one translation unit
// needs: the slot layout, the hash, and the two jobs (clearing a table, looking
// labels up) that the multi-hop sequence runs as extra CTAs of another kernel's
// launch instead of as launches of their own.
#pragma once
#include "common.cuh"

namespace dgs {

constexpr int RL_BLOCK = 256;
constexpr int RL_ITEMS = 4;
constexpr int RL_TILE = RL_BLOCK * RL_ITEMS;
constexpr uint32_t NO_SLOT = 0xFFFFFFFFu;
constexpr int CLEAR_UNITS_PER_CTA = RL_BLOCK * 4;  // of 16 bytes

// A slot is ONE 64-bit word: the low 32 bits of the key in the high half, the minimum input index (later the label)
// in the low half.  Claiming a slot and setting its first index is a single compare-and-swap, a repeated key costs
// one load and at most one atomicMin, and every later pass reads 8 bytes per key.  Input indices and labels stay
// below 2^30 (the key count is limited to that): bit 31 of the low half marks a label, bit 30 a key of 2^32 or more.
// Two keys below 2^32 are equal when their words agree in the high half and in bit 30; such wide keys are compared in
// full as well, with the input the index names or, once numbered, with the key kept beside the label (wide_keys).
// (64-bit ids used to have 16-byte {key, index} slots: 880 k keys took 27 + 18 + 25 + 27 us for insert, count,
// number and lookup where the one-word form of the multi-hop sequence took 21 + 16 + 26 + 22.)
constexpr unsigned long long EMPTY_WORD = ~0ull;
constexpr uint32_t LABEL_BIT32 = 0x80000000u;
constexpr uint32_t WIDE_BIT32 = 0x40000000u;
constexpr uint32_t VALUE_MASK32 = 0x3FFFFFFFu;
constexpr long long COMPACT_KEY_LIMIT = 0xFFFFFFFFll;  // ids of a graph with fewer nodes than this

// slots in use for a table built for n keys: the power of two >= max(2n, 64)
__host__ __device__ __forceinline__ uint64_t slots_for(int64_t n) {
  uint64_t want = 2 * static_cast<uint64_t>(n);
  if (want < 64) want = 64;
#ifdef __CUDA_ARCH__
  return 1ull << (64 - __clzll(static_cast<long long>(want - 1)));
#else
  uint64_t cap = 64;
  while (cap < want) cap <<= 1;
  return cap;
#endif
}

// How many keys a table is dimensioned for: count_of(n) * mult.  The per-operator
// path knows its key count (mult = 1).  The multi-hop sequence dimensions a hop's
// table before that hop's neighbours are drawn, for seeds * (1 + fanout) keys.
struct TableSize {
  Count n;
  int64_t mult;
  long long max_key;  // keys above are out of range
};

// The device arrays of one table.
struct TableParts {
  unsigned long long* words;    // [cap]
  unsigned int* ticket;         // [4]       all ones when cleared: the first draw is 0
  unsigned long long* tiles;    // [ntiles]  running count of distinct keys, see tile_scan.cuh
  unsigned long long* tiles2;   // [ntiles]  the same of the edges that the distinct keys will be given
  long long* wide_keys;         // [n]       by label: keys of 2^32 and more (64-bit ids only)
  uint32_t* slot_of;            // [n]       slot of every input
  unsigned long long* largest;  // [ntiles] where the largest key is looked at: those that the clearing CTAs have met
  int64_t* total;               // [1]
  int64_t* dense;               // [1]       and whether the words are addressed by the key
  int64_t ntiles;
};

// Sizes that only the host needs (how much of each output is valid): device words copied to a
// host-visible array by the kernel that computes the last of them, so that a sequence of kernels
// pays for one write over the host link instead of one per size.
struct SizesReport {
  int64_t* dst;  // [n], pinned
  int n;         // 0: nothing to report
  const int64_t* src[2 * DGS_MAX_HOPS];
};

// The other form of the table, for a sequence whose ids lie below a known bound: one 32-bit word per id of the id space,
// addressed by the id itself.  The word holds the smallest input index that an id was met at and, once numbered, its
// label; all ones is "not met".  ONE table serves all hops of a batch: a hop's frontier begins with its seeds, so a label
// given by one hop is the node's position among the next hop's inputs and stays the smallest there.
// A label never reads as another input's index: the label of the id first met at input e is at most e, and whoever
// meets that id again does so at an input behind e.
constexpr uint32_t NOT_MET = 0xFFFFFFFFu;

// Inputs that a sampling launch records in that table as it emits them (first == nullptr: none).
struct IdMarks {
  uint32_t* first;
  int64_t ids;  // words of the table
  bool seeds;   // the seeds are inputs too (first hop; from the second on they are labelled already)
  uint32_t* beyond;  // cleared with the table; anything but NOT_MET: an id at or beyond `ids` was met
};

// What relabels the COO of all hops of a sequence through that table, in one launch.
struct DenseLookup {
  const uint32_t* first;
  int64_t ids;
  int n_hops;
  void* row0;  // rows of the first hop (those of the others are positions already)
  void* col[DGS_MAX_HOPS];
  Count n[DGS_MAX_HOPS];
  unsigned end_cta[DGS_MAX_HOPS];  // RL_TILE ids a CTA; running
};

// Words to set to all ones, as extra CTAs of the first launch of a sequence (16-byte units; ctas == 0: none).
struct FillJob {
  ulonglong2* at;
  int64_t units;
  unsigned ctas;
};

#ifdef __CUDACC__

// The words are read and written at random by every launch of a batch while gathered rows stream through the L2: they are
// marked to be evicted last.  Six batches in flight, 2.4 M words each: 674 -> 662 us a pass, one at a time 146 -> 145;
// steadily one in, one out 102.5 -> 99.8 us a batch.  What runs beside them does not lose by it: ten passes over a buffer of
// 64 MB after each batch, 2.4 M ids, 283 us a batch with hash tables and 261 with these words (8.3 M: 261 and 251); behind the
// pipeline the same ten passes take 144 us in either case.
__device__ __forceinline__ uint64_t l2_evict_last_policy() {
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(policy));
  return policy;
}
__device__ __forceinline__ uint32_t load_kept(const uint32_t* p, uint64_t policy) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(policy) : "memory");
  return v;
}
__device__ __forceinline__ void store_kept(uint32_t* p, uint32_t v, uint64_t policy) {
  asm volatile("st.relaxed.gpu.global.L2::cache_hint.u32 [%0], %1, %2;" ::"l"(p), "r"(v), "l"(policy) : "memory");
}
__device__ __forceinline__ void min_kept(uint32_t* p, uint32_t v, uint64_t policy) {
  asm volatile("red.relaxed.gpu.global.min.L2::cache_hint.u32 [%0], %1, %2;" ::"l"(p), "r"(v), "l"(policy) : "memory");
}
__device__ __forceinline__ void mark_id(const IdMarks& m, int64_t id, uint32_t input, int32_t* status) {
  if (static_cast<uint64_t>(id) < static_cast<uint64_t>(m.ids)) min_kept(m.first + id, input, l2_evict_last_policy());
  else if (id < 0) raise_status(status, DGS_ERR_RANGE);
  else *static_cast<volatile uint32_t*>(m.beyond) = 0u;  // reported with the sizes
}

__device__ __forceinline__ void run_fill_cta(const FillJob& j, unsigned cta) {
  const int64_t stride = static_cast<int64_t>(j.ctas) * blockDim.x;
  const uint64_t policy = l2_evict_last_policy();
#pragma unroll 4
  for (int64_t i = static_cast<int64_t>(cta) * blockDim.x + threadIdx.x; i < j.units; i += stride)
    asm volatile("st.global.L2::cache_hint.v2.u64 [%0], {%1, %1}, %2;" ::"l"(j.at + i), "l"(~0ull), "l"(policy) : "memory");
}

__device__ __forceinline__ uint64_t table_slots(const TableSize& t) { return slots_for(count_of(t.n) * t.mult); }

__device__ __forceinline__ uint64_t hash_key(long long key) {
  uint64_t z = static_cast<uint64_t>(key);
  z = (z ^ (z >> 33)) * 0xFF51AFD7ED558CCDull;
  z = (z ^ (z >> 33)) * 0xC4CEB9FE1A85EC53ull;
  return z ^ (z >> 33);
}

// 32-bit finaliser for the one-word tables (their keys fit 32 bits and their slot counts stay below 2^31):
// a third of the instructions of the 64-bit mix, and these kernels are short of issue slots, not of bandwidth
__device__ __forceinline__ uint32_t hash_key32(uint32_t k) {
  k ^= k >> 16;
  k *= 0x85EBCA6Bu;
  k ^= k >> 13;
  k *= 0xC2B2AE35u;
  return k ^ (k >> 16);
}

__device__ __forceinline__ bool is_wide(long long key) { return (static_cast<unsigned long long>(key) >> 32) != 0; }
__device__ __forceinline__ uint32_t home_slot(long long key, uint32_t mask32) {
  return (is_wide(key) ? static_cast<uint32_t>(hash_key(key)) : hash_key32(static_cast<uint32_t>(key))) & mask32;
}

__device__ __forceinline__ long long probe_label(const unsigned long long* words, const long long* wide_keys,
                                                 uint64_t mask, long long key) {
  if (key < 0) return -1;
  const uint32_t mask32 = static_cast<uint32_t>(mask), key32 = static_cast<uint32_t>(key);
  const uint32_t flag = is_wide(key) ? WIDE_BIT32 : 0u;
  uint32_t h = home_slot(key, mask32);
  for (uint32_t probes = 0; probes <= mask32; ++probes) {
    const uint2 w = reinterpret_cast<const uint2*>(words)[h];  // one 8-byte load: x = index / label, y = key
    if ((w.x & w.y) == 0xFFFFFFFFu) break;                     // empty slot
    if (w.y == key32 && (w.x & WIDE_BIT32) == flag) {
      const uint32_t label = w.x & VALUE_MASK32;
      if (flag == 0u || wide_keys[label] == key) return static_cast<long long>(label);
    }
    h = (h + 1) & mask32;
  }
  return -1;
}

// ---- jobs that can ride on another kernel's launch -----------------------------
// Clear the slots a table will use, its ticket and its tile words.  Runs before anything touches the table.
struct ClearJob {
  unsigned long long* words;
  unsigned int* ticket;   // ticket and tile words are one run of 16-byte units
  int64_t ticket_units;
  TableSize size;
  unsigned ctas;  // CLEAR_UNITS_PER_CTA units each; 0: no job
};
__device__ __forceinline__ void run_clear_cta(const ClearJob& j, unsigned cta) {
  const int64_t slots = static_cast<int64_t>(table_slots(j.size) / 2);  // two to a unit
  const int64_t i = static_cast<int64_t>(cta) * CLEAR_UNITS_PER_CTA + threadIdx.x;
  const ulonglong2 empty = make_ulonglong2(~0ull, ~0ull);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int64_t at = i + static_cast<int64_t>(u) * RL_BLOCK;
    if (at < slots) reinterpret_cast<ulonglong2*>(j.words)[at] = empty;
    else if (at - slots < j.ticket_units) reinterpret_cast<ulonglong2*>(j.ticket)[at - slots] = empty;
  }
}

// Relabel a finished hop's COO in place: row[i] = label(row[i]) (skipped when row is null), and col[i] = the label
// in the slot that input n_seeds + i was inserted at, i < n.  Needs that hop's numbering.
struct LookupJob {
  void* row;
  void* col;
  Count n, n_seeds;
  const unsigned long long* words;
  const uint32_t* slot_of;
  const long long* wide_keys;
  TableSize size;
  unsigned ctas;  // RL_BLOCK ids each; 0: no job
};
template <typename IdT>
__device__ __forceinline__ void run_lookup_cta(const LookupJob& j, unsigned cta) {
  const int64_t i = static_cast<int64_t>(cta) * RL_BLOCK + threadIdx.x;
  // what does not depend on the live counts is read while they are on their way (room for n.bound ids)
  const long long kr = (i < j.n.bound && j.row != nullptr) ? static_cast<long long>(static_cast<const IdT*>(j.row)[i]) : -1;
  const int64_t n_seeds = count_of(j.n_seeds);
  if (i >= count_of(j.n)) return;
  const uint32_t slot = j.slot_of[n_seeds + i];
  if (j.row != nullptr)
    static_cast<IdT*>(j.row)[i] = static_cast<IdT>(probe_label(j.words, j.wide_keys, table_slots(j.size) - 1, kr));
  static_cast<IdT*>(j.col)[i] =
      slot == NO_SLOT ? static_cast<IdT>(-1)
                      : static_cast<IdT>(reinterpret_cast<const uint2*>(j.words)[slot].x & VALUE_MASK32);
}

#endif  // __CUDACC__
}  // namespace dgs
