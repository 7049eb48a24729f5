// Device-side pieces of neighbour sampling: writing one sampled edge, and drawing the edges of one row uniformly with
// a group of lanes.
#pragma once
#include "common.cuh"
#include "philox.cuh"
#include "relabel_device.cuh"

namespace dgs {

constexpr uint32_t TAG_UNIFORM = 0x554E4931u;
constexpr uint32_t TAG_REPLACE = 0x5245504Cu;
constexpr uint32_t TAG_FLOYD = 0x464C4F59u;

// 32-bit words of position bitmap per lane: a group of G lanes marks positions of rows of up to 512 * G edges
constexpr int TAKEN_WORDS_PER_LANE = 16;

#ifdef __CUDACC__

__device__ __forceinline__ int64_t pick_count(int64_t deg, int64_t k, bool replace) {
  return replace ? (deg > 0 ? k : 0) : (deg < k ? deg : k);
}

// Rows [rb[u], rb[u] + deg[u]) of the seeds s[u] (0, 0 when !good[u] or the bounds are broken).  All 32 lanes of a
// warp call this; the loads of all ITEMS seeds are in flight together.
// indptr[s] and indptr[s + 1] are fetched by TWO NEIGHBOURING LANES in one load instruction, half a warp's
// seeds at a time: the two addresses (almost always) lie in the same 128-byte line, so the pair costs one
// memory request instead of the two that two loads of one thread cost.  Inside one GPU that is noise; when
// the row of indptr lives on a peer, requests are what the link can deliver only so many of per second.
template <typename IdT, int ITEMS>
__device__ __forceinline__ void row_bounds(const dgs_chunk_desc& indptr, const int64_t (&s)[ITEMS],
                                           const bool (&good)[ITEMS], int64_t (&rb)[ITEMS], int64_t (&deg)[ITEMS],
                                           int32_t* status) {
  constexpr int sh = sizeof(IdT) == 8 ? 3 : 2;
  const int lane = threadIdx.x & 31;
  IdT v[ITEMS][2];  // what this lane fetched for the owners of either half
#pragma unroll
  for (int u = 0; u < ITEMS; ++u)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int owner = half * 16 + (lane >> 1);  // the lane whose seed this lane fetches an element for
      const int64_t so = __shfl_sync(FULL_MASK, good[u] ? s[u] : -1, owner);
      v[u][half] = so >= 0 ? load_at<IdT>(indptr, sh, so + (lane & 1)) : IdT(0);
    }
#pragma unroll
  for (int u = 0; u < ITEMS; ++u) {
    const int from = 2 * (lane & 15);
    const IdT lo0 = __shfl_sync(FULL_MASK, v[u][0], from), hi0 = __shfl_sync(FULL_MASK, v[u][0], from + 1);
    const IdT lo1 = __shfl_sync(FULL_MASK, v[u][1], from), hi1 = __shfl_sync(FULL_MASK, v[u][1], from + 1);
    const int64_t lo = static_cast<int64_t>(lane < 16 ? lo0 : lo1), hi = static_cast<int64_t>(lane < 16 ? hi0 : hi1);
    rb[u] = 0;
    deg[u] = 0;
    if (good[u]) {
      if (hi < lo || lo < 0) {
        raise_status(status, DGS_ERR_RANGE);
      } else {
        rb[u] = lo;
        deg[u] = hi - lo;
      }
    }
  }
}

template <typename IdT>
struct Emit {
  const dgs_chunk_desc& indices;
  IdT* coo_row;
  IdT* coo_col;
  int64_t* picked_pos;
  int64_t out_capacity;
  int32_t* status;
  const IdMarks& marks;
  const Count& n_seeds;

  // t-th output of a seed whose outputs start at o; `pos` = position in its row
  __device__ __forceinline__ void operator()(int64_t o, int64_t t, int64_t seed, int64_t rb,
                                             int64_t pos) const {
    constexpr int sh = sizeof(IdT) == 8 ? 3 : 2;
    const int64_t at = o + t;
    if (at >= out_capacity) {
      raise_status(status, DGS_ERR_RANGE);
      return;
    }
    const int64_t e = rb + pos;
    IdT c = static_cast<IdT>(-1);
    if (e >= 0 && e < indices.total) c = load_at<IdT>(indices, sh, e);
    else raise_status(status, DGS_ERR_RANGE);
    coo_row[at] = static_cast<IdT>(seed);
    coo_col[at] = c;
    if (picked_pos != nullptr) picked_pos[at] = pos;
    if (marks.first != nullptr) mark_id(marks, static_cast<int64_t>(c), static_cast<uint32_t>(count_of(n_seeds) + at), status);
  }
};

// Draws one row's edges with a group of G lanes (a power of two up to 32, aligned in the warp): emit(t, pos) is called
// for the t-th output of the row, `pos` its position in the row.  All 32 lanes of a warp come through here together,
// with deg = 0 in the groups that have no row.  `i` is the seed's position in its list (the address of its random
// numbers), `taken` the group's bitmap words, `slots` the row's outputs (room for k ids, used while k > G picks are
// drawn), slots_fit whether they lie inside the output.  False (in lane 0 of the group): they do not.
//
// The emit calls stand in two places only: with the address arithmetic of a chunked tensor inlined at seven of them
// the kernel was 50 KB of code (60 000 seeds, fan-out 15: 28 us; with 35 KB 26 us).
template <typename IdT, typename EmitF>
__device__ __forceinline__ bool sample_uniform_row(const uint64_t key, const int64_t i, const int64_t deg,
                                                   const int64_t k, const bool replace, const int G, uint32_t* taken,
                                                   IdT* slots_out, const bool slots_fit, int32_t* status,
                                                   const EmitF& emit) {
  const int lane = threadIdx.x & 31;
  const int l = lane & (G - 1);  // lane inside the group
  const int gw = lane / G;       // group inside the warp
  const unsigned gmask = (G == 32) ? FULL_MASK : (((1u << G) - 1u) << (gw * G));
  const uint32_t i_lo = static_cast<uint32_t>(i), i_hi = static_cast<uint32_t>(static_cast<uint64_t>(i) >> 32);

  if (!replace && k <= G) {  // uniform over the launch
    // -- distinct positions by parallel rejection (all 32 lanes take part) --
    // Every lane of a group draws a position and marks it in the group's bitmap
    // in shared memory; a lane that finds its bit already set draws again.  Only
    // equality of positions matters, so every k-subset is equally likely.
    const int64_t MAP_DEG = static_cast<int64_t>(G) * TAKEN_WORDS_PER_LANE * 32;
    const bool sampled = deg > k;
    const bool complement = sampled && 2 * k > deg;  // draw the deg-k positions to leave out
    const int64_t m = sampled ? (complement ? deg - k : k) : 0;
    const bool active = l < m;
    const bool in_map = deg <= MAP_DEG;              // longer rows compare candidates across the warp
    if (sampled && in_map)
      for (int wd = l; wd < static_cast<int>((deg + 31) >> 5); wd += G) taken[wd] = 0u;
    __syncwarp();
    bool need = active;
    int64_t c = 0;
    const bool small_row = deg <= 0xFFFFFFFFll;  // every real graph; longer rows take the general path
    const uint32_t deg32 = static_cast<uint32_t>(deg);
    Philox4 rnd{0u, 0u, 0u, 0u};
    for (uint32_t round = 0; __any_sync(FULL_MASK, need); ++round) {
      // one Philox block per lane feeds four rounds of (re)draws
      if ((round & 3u) == 0u && active && round < 64)
        rnd = philox4x32_10(key, i_lo, i_hi, ((round >> 2) << 8) | static_cast<uint32_t>(l), TAG_UNIFORM);
      bool usable = true;  // false: this attempt hit Lemire's rejection zone, draw again next round
      if (need) {
        if (round >= 64) {  // never reached in practice: step to a neighbour, keeps the loop bounded
          c = (c + 1 == deg) ? 0 : c + 1;
        } else if (small_row) {
          const uint32_t word = (round & 2u) ? ((round & 1u) ? rnd.w : rnd.z) : ((round & 1u) ? rnd.y : rnd.x);
          uint32_t pick;
          usable = bounded_try(word, deg32, &pick);
          c = pick;
        } else {
          const Philox4 r = philox4x32_10(key, i_lo, i_hi, (round << 8) | static_cast<uint32_t>(l), TAG_UNIFORM ^ 1u);
          c = static_cast<int64_t>(bounded(r, static_cast<uint64_t>(deg)));
        }
        if (in_map && usable) {
          const uint32_t bit = 1u << (static_cast<uint32_t>(c) & 31u);
          need = (atomicOr(&taken[c >> 5], bit) & bit) != 0u;
        }
      }
      if (__any_sync(FULL_MASK, active && !in_map)) {
        // lanes holding the same position inside one group see each other; the lowest keeps it
        const bool mine = active && !in_map;
        const unsigned long long tag =
            (mine && usable) ? (static_cast<unsigned long long>(c) | (static_cast<unsigned long long>(gw) << 58))
                             : (0x8000000000000000ull | static_cast<unsigned long long>(lane));
        const unsigned same = __match_any_sync(FULL_MASK, tag);
        if (mine) need = !usable || (__ffs(same) - 1 != lane);
      }
      if (round >= 64 + 1024) {
        if (need) raise_status(status, DGS_ERR_TABLE_FULL);
        break;
      }
    }
    __syncwarp();
    // what this lane emits: one edge, or (complement) up to two
    int t0 = l, t1 = 0, p1 = -1;
    int64_t p0 = -1;
    if (complement) {
      // the row has at most 2k-1 <= 63 positions, so its bitmap is one or two words:
      // every lane ranks its own two positions (a = l and b = l + G cover the row)
      // among the kept ones
      const unsigned long long out_mask =
          static_cast<unsigned long long>(taken[0]) |
          (deg > 32 ? static_cast<unsigned long long>(taken[1]) << 32 : 0ull);
      const unsigned long long row_mask = (1ull << deg) - 1ull;  // deg <= 63
      const unsigned long long kept = ~out_mask & row_mask;
      const int a = l, b = l + G;
      if ((kept >> a) & 1ull) {
        t0 = __popcll(kept & ((1ull << a) - 1ull));
        p0 = a;
      }
      if (b < 64 && ((kept >> b) & 1ull)) {
        t1 = __popcll(kept & ((1ull << b) - 1ull));
        p1 = b;
      }
    } else if (sampled) {
      if (active) p0 = c;
    } else if (l < deg) {
      p0 = l;  // whole row, CSC order (deg <= k <= G)
    }
#pragma unroll 1
    for (int u = 0; u < 2; ++u) {
      if (p0 >= 0) emit(t0, p0);
      if (!__any_sync(FULL_MASK, p1 >= 0)) break;
      t0 = t1;
      p0 = p1;
      p1 = -1;
    }
    return true;
  }

  // -- with replacement, or general k (> G is only possible with G == 32: the group is the warp) --
  volatile IdT* slots = slots_out;
  const bool whole = !replace && deg <= k;
  if (!replace && !whole) {
    if (!slots_fit) return l != 0;
    // Floyd's subset algorithm; the chosen positions are parked in the output
    int64_t have = 0;
    for (int64_t j = deg - k; j < deg; ++j, ++have) {
      const Philox4 r = philox4x32_10(key, i_lo, i_hi, static_cast<uint32_t>(have), TAG_FLOYD);
      const int64_t t = static_cast<int64_t>(bounded(r, static_cast<uint64_t>(j + 1)));
      bool found = false;
      for (int64_t q = l; q < have; q += G) found |= (static_cast<int64_t>(slots[q]) == t);
      found = __any_sync(gmask, found);
      if (l == 0) slots[have] = static_cast<IdT>(found ? j : t);
      __syncwarp(gmask);
    }
  }
  const int64_t count = pick_count(deg, k, replace);
#pragma unroll 1
  for (int64_t t = l; t < count; t += G) {
    int64_t pos = t;
    if (replace)
      pos = static_cast<int64_t>(bounded(philox4x32_10(key, i_lo, i_hi, static_cast<uint32_t>(t), TAG_REPLACE),
                                         static_cast<uint64_t>(deg)));
    else if (!whole)
      pos = static_cast<int64_t>(slots[t]);
    emit(t, pos);
  }
  return true;
}

#endif  // __CUDACC__
}  // namespace dgs
