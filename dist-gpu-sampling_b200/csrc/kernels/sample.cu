// Row-wise neighbour sampling on a CSC graph whose indptr / indices / weights
// live in ChunkTensors (or plain device tensors: num_parts == 1).
//
// Replaces, for both the plain-tensor and the ChunkTensor operators:
//   _GetSubIndptr + cub scan + blocking nnz read-back
//       (reference src/cuda/rowwise_sampling.cu:13-40,147),
//   _CSRRowWiseSampleUniformKernel / ...ReplaceKernel
//       (src/cuda/rowwise_sampling.cu:42-136,
//        src/cuda/rowwise_sampling_with_chunk_tensor.cu:15-111),
//   _CSRRowWiseSampleKernel / ...ReplaceKernel (weighted)
//       (src/cuda/rowwise_sampling_probs.cu:54-216) and the faiss-derived
//       WarpSelect it uses (src/cuda/warpselect/*.cuh).
//
// What is kept (the contract): per-seed counts min(deg,k) / (deg?k:0); COO
// grouped by seed position; rows with deg <= k copied whole in CSC order;
// uniform k-subsets / A-Res weighted subsets / proportional draws otherwise.
//
// What is different (the design):
//   * the reference spends one 128-thread block and one curand_init per seed
//     and draws O(deg) random numbers per row (Algorithm R).  Here a seed gets
//     a sub-warp group of G = 4..32 lanes (G >= k), the row is never scanned:
//     k candidate positions are drawn at once with counter-based Philox and
//     duplicates are re-drawn until the k positions are distinct
//     (__match_any_sync across the warp).  Equal treatment of positions makes
//     every k-subset equally likely.  When k > deg/2 the deg-k positions to
//     LEAVE OUT are drawn instead, so a draw collides with probability < 1/2.
//   * bounded integers use Lemire's multiply-shift with rejection instead of
//     `rand % n`.
//   * weighted sampling without replacement keeps the top-k keys in a sorted
//     per-warp register list (lane i = i-th largest); keys are compared in the
//     log domain, log(u)/w, which orders exactly like u^(1/w) but does not
//     underflow for small weights.  The first 512 edges of a row give one warp
//     a list and a bar; the 512-edge windows behind them (16 loads in flight
//     per lane) are dealt out to the eight warps of the CTA, which collect the
//     edges that may beat the bar, and one warp per row joins them with its list.
//   * weighted sampling with replacement builds no cumulative array in global
//     memory: the row is summed once into at most 128 groups, and every lane
//     finds its own draw's group by bisection and walks the edges in it.
//   * counts, offsets and the total come from a plan: one CTA for up to 2 048
//     seeds, a cluster of eight for up to 8 192; above, every CTA scans its 256 seeds and the one that finishes last
//     (an atomic ticket, nobody waits) scans the per-tile sums; from the second
//     hop of a multi-hop sequence on, the kernel that numbers the seeds.  The
//     total goes to a caller-supplied (pinned) word, so the host learns the
//     output size while the sampling kernel is still running.
//   * the sampling kernels give every seed its own group / warp and never loop
//     over seeds, so even a 1 024-seed hop fills the machine with independent
//     short chains instead of a few long ones.
#include "common.cuh"
#include "launchers.h"
#include "philox.cuh"
#include "sample_device.cuh"
#include "tile_scan.cuh"

#include <cooperative_groups.h>

namespace dgs {
namespace {

constexpr int SAMPLE_TILE = 256;   // seeds per CTA
constexpr int SAMPLE_BLOCK = 256;  // threads per CTA

constexpr uint32_t TAG_ARES = 0x41524553u;
constexpr uint32_t TAG_WREPL = 0x57524550u;

struct PlanView {
  int64_t* row_begin;  // [n]
  int64_t* deg;        // [n]
  int64_t* local_off;  // [n]       exclusive prefix of the counts inside the seed's 256-tile
  int64_t* tile_off;   // [ntiles]  per-tile sums, scanned in place by the last CTA
  int64_t* total;      // [1]
  unsigned int* ticket;  // [1]     CTAs that have published their tile sum
  int64_t ntiles;
};

inline PlanView plan_view(void* plan, int64_t n) {
  PlanView v;
  v.ntiles = (n + SAMPLE_TILE - 1) / SAMPLE_TILE;
  v.row_begin = static_cast<int64_t*>(plan);
  v.deg = v.row_begin + n;
  v.local_off = v.deg + n;
  v.tile_off = v.local_off + n;
  v.total = v.tile_off + v.ntiles;
  v.ticket = reinterpret_cast<unsigned int*>(v.total + 1);
  return v;
}

// The words a multi-hop sequence wants set before anything else runs (by 32 threads at least).
__device__ __forceinline__ void run_init(const InitWords& w) {
  if (threadIdx.x == 0 && w.n0 != nullptr) *w.n0 = w.n0_value;
  if (w.rng_src != nullptr && threadIdx.x < w.n_keys) {
    const volatile uint64_t* src = w.rng_src;  // host-written words: no cached copy
    w.keys[threadIdx.x] = fold_rng_key(src[0], src[1] + static_cast<uint64_t>(threadIdx.x));
  }
}
__global__ void init_kernel(const InitWords w, unsigned int* ticket, const FillJob fill) {
  pdl_enter();
  if (blockIdx.x > 0) {
    run_fill_cta(fill, blockIdx.x - 1);
    return;
  }
  if (threadIdx.x == 0) *ticket = 0u;
  run_init(w);
}

// ---------------------------------------------------------------------------
// plan: row range per seed + per-tile output counts
// ---------------------------------------------------------------------------
template <typename IdT>
__global__ void __launch_bounds__(SAMPLE_BLOCK)
sample_plan_kernel(const __grid_constant__ dgs_chunk_desc indptr, const IdT* __restrict__ seeds,
                   const Count nc, const int64_t k, const bool replace,
                   int64_t* __restrict__ row_begin, int64_t* __restrict__ deg_out,
                   int64_t* __restrict__ local_off, int64_t* tile_sums, int64_t* total_out,
                   unsigned int* ticket, int64_t* nnz_out, int32_t* __restrict__ status) {
  __shared__ int64_t smem[SAMPLE_BLOCK / 32 + 1];
  pdl_enter();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * SAMPLE_TILE + threadIdx.x;
  // the seed is read before the live count arrives (the list has room for nc.bound entries), so that
  // the two round trips overlap; an entry past the count is never used
  const IdT seed_raw = i < nc.bound ? seeds[i] : IdT(0);
  const int64_t n = count_of(nc);
  const int64_t s = static_cast<int64_t>(seed_raw);
  const bool good = i < n && s >= 0 && s + 1 < indptr.total;
  if (i < n && !good) raise_status(status, DGS_ERR_RANGE);
  const int64_t seed[1] = {s};
  const bool ok[1] = {good};
  int64_t rb[1], deg[1];
  row_bounds<IdT, 1>(indptr, seed, ok, rb, deg, status);
  int64_t cnt = 0;
  if (i < n) {
    row_begin[i] = rb[0];
    deg_out[i] = deg[0];
    cnt = pick_count(deg[0], k, replace);
  }
  int64_t total;
  const int64_t ex = block_exclusive_scan<int64_t, SAMPLE_BLOCK>(cnt, smem, &total);
  if (i < n) local_off[i] = ex;

  // publish the tile sum; the CTA that draws the last ticket scans all of them
  publish_and_scan_tiles<SAMPLE_BLOCK>(total, tile_sums, ticket, total_out, nnz_out, smem);
}

// The plan of up to SMALL_PLAN seeds by one CTA: no ticket, hence nothing that has to be cleared before it, and in the
// multi-hop sequence it sets the words that a launch of its own sets otherwise.  Bound by latency (seed, row bounds,
// scan); two seeds per thread with their loads in flight together.
// The line, against a CTA per 256 seeds behind a clearing launch (us; indptr of 2.4 M nodes on the GPU, then of 20 M in
// host memory): 64 seeds 2.1 against 3.9 and 3.3 against 5.5, 1 024 seeds 3.0 against 4.2 and 6.7 against 9.3, 2 048
// seeds 4.4 against 5.0 and 10.6 against 11.6.  With four seeds per thread: 3 072 seeds 6.1 against 5.0 and 14.7 against
// 14.6, 4 096 seeds 7.5 against 5.0 and 18.6 against 18.3.
constexpr int SMALL_PLAN_BLOCK = 1024;
constexpr int SMALL_PLAN_ITEMS = 2;
constexpr int SMALL_PLAN = SMALL_PLAN_BLOCK * SMALL_PLAN_ITEMS;

template <typename IdT>
__global__ void __launch_bounds__(SMALL_PLAN_BLOCK)
sample_small_plan_kernel(const __grid_constant__ dgs_chunk_desc indptr, const IdT* __restrict__ seeds, const int n,
                         const int64_t k, const bool replace, const PlanView plan, int64_t* nnz_out,
                         const __grid_constant__ InitWords init, const FillJob fill, int32_t* __restrict__ status) {
  __shared__ int64_t smem[SMALL_PLAN_BLOCK / 32 + 1];
  pdl_enter();
  if (blockIdx.x > 0) {
    run_fill_cta(fill, blockIdx.x - 1);
    return;
  }
  run_init(init);
  int64_t s[SMALL_PLAN_ITEMS], rb[SMALL_PLAN_ITEMS], deg[SMALL_PLAN_ITEMS];
  bool good[SMALL_PLAN_ITEMS];
#pragma unroll
  for (int u = 0; u < SMALL_PLAN_ITEMS; ++u) {
    const int i = u * SMALL_PLAN_BLOCK + threadIdx.x;
    s[u] = i < n ? static_cast<int64_t>(seeds[i]) : -1;
  }
#pragma unroll
  for (int u = 0; u < SMALL_PLAN_ITEMS; ++u) {
    good[u] = s[u] >= 0 && s[u] + 1 < indptr.total;
    if (u * SMALL_PLAN_BLOCK + static_cast<int>(threadIdx.x) < n && !good[u]) raise_status(status, DGS_ERR_RANGE);
  }
  row_bounds<IdT, SMALL_PLAN_ITEMS>(indptr, s, good, rb, deg, status);
  int64_t carry = 0;
#pragma unroll
  for (int u = 0; u < SMALL_PLAN_ITEMS; ++u) {
    if (u * SMALL_PLAN_BLOCK >= n) break;  // uniform
    const int i = u * SMALL_PLAN_BLOCK + threadIdx.x;
    int64_t total;
    const int64_t ex = block_exclusive_scan<int64_t, SMALL_PLAN_BLOCK>(i < n ? pick_count(deg[u], k, replace) : 0, smem, &total);
    if (i < n) {
      plan.row_begin[i] = rb[u];
      plan.deg[i] = deg[u];
      plan.local_off[i] = carry + ex;
    }
    carry += total;
  }
  // offsets are those in the whole output, whichever way the sampling launch adds them up
  if (static_cast<int64_t>(threadIdx.x) < plan.ntiles) plan.tile_off[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    *plan.total = carry;
    if (nnz_out != nullptr) {
      *nnz_out = carry;
      __threadfence_system();
    }
  }
}

// The plan of an operator call's up to CLUSTER_PLAN seeds by one cluster of eight CTAs: each takes an eighth of the seeds, and
// the CTAs' sums are read over distributed shared memory -- nothing to clear before it, and no round trip through L2 for
// the offsets.  (The multi-hop sequence keeps to the forms before and behind: its batches run beside others, and a
// cluster waits for room on eight SMs at once.)
// Against the clearing launch and a CTA per 256 seeds, whole operator calls: 4 096 weighted draws with replacement 45.7 ->
// 42.4 us, 3 000 of them 45.9 -> 42.6, 8 000 without replacement (fan-out 5) 45.8 -> 43.7.  With four seeds per thread, for
// 11 000 seeds, level or slower (91.2 -> 92.2).
constexpr int CLUSTER_PLAN_CTAS = 8;
constexpr int CLUSTER_PLAN_BLOCK = 512;
constexpr int CLUSTER_PLAN_ITEMS = 2;
constexpr int CLUSTER_PLAN = CLUSTER_PLAN_CTAS * CLUSTER_PLAN_BLOCK * CLUSTER_PLAN_ITEMS;

template <typename IdT>
__global__ void __cluster_dims__(CLUSTER_PLAN_CTAS, 1, 1) __launch_bounds__(CLUSTER_PLAN_BLOCK)
sample_cluster_plan_kernel(const __grid_constant__ dgs_chunk_desc indptr, const IdT* __restrict__ seeds, const int n,
                           const int64_t k, const bool replace, const PlanView plan, int64_t* nnz_out,
                           int32_t* __restrict__ status) {
  __shared__ int64_t smem[CLUSTER_PLAN_BLOCK / 32 + 1];
  __shared__ int64_t s_sum;
  auto cluster = cooperative_groups::this_cluster();
  pdl_enter();
  const int rank = blockIdx.x;
  const int per = (n + CLUSTER_PLAN_CTAS - 1) / CLUSTER_PLAN_CTAS, lo = rank * per, end = min(lo + per, n);
  int64_t s[CLUSTER_PLAN_ITEMS], rb[CLUSTER_PLAN_ITEMS], deg[CLUSTER_PLAN_ITEMS], off[CLUSTER_PLAN_ITEMS];
  bool good[CLUSTER_PLAN_ITEMS];
#pragma unroll
  for (int u = 0; u < CLUSTER_PLAN_ITEMS; ++u) {
    const int i = lo + u * CLUSTER_PLAN_BLOCK + threadIdx.x;
    s[u] = i < end ? static_cast<int64_t>(seeds[i]) : -1;
  }
#pragma unroll
  for (int u = 0; u < CLUSTER_PLAN_ITEMS; ++u) {
    good[u] = s[u] >= 0 && s[u] + 1 < indptr.total;
    if (lo + u * CLUSTER_PLAN_BLOCK + static_cast<int>(threadIdx.x) < end && !good[u]) raise_status(status, DGS_ERR_RANGE);
  }
  row_bounds<IdT, CLUSTER_PLAN_ITEMS>(indptr, s, good, rb, deg, status);
  int64_t carry = 0;
#pragma unroll
  for (int u = 0; u < CLUSTER_PLAN_ITEMS; ++u) {
    off[u] = 0;
    if (lo + u * CLUSTER_PLAN_BLOCK >= end) continue;  // uniform
    const int i = lo + u * CLUSTER_PLAN_BLOCK + threadIdx.x;
    int64_t total;
    off[u] = carry + block_exclusive_scan<int64_t, CLUSTER_PLAN_BLOCK>(i < end ? pick_count(deg[u], k, replace) : 0, smem, &total);
    carry += total;
  }
  if (threadIdx.x == 0) s_sum = carry;
  cluster.sync();
  int64_t before = 0, all = 0;
#pragma unroll
  for (int r = 0; r < CLUSTER_PLAN_CTAS; ++r) {
    const int64_t v = *cluster.map_shared_rank(&s_sum, r);
    if (r < rank) before += v;
    all += v;
  }
#pragma unroll
  for (int u = 0; u < CLUSTER_PLAN_ITEMS; ++u) {
    const int i = lo + u * CLUSTER_PLAN_BLOCK + threadIdx.x;
    if (i < end) {
      plan.row_begin[i] = rb[u];
      plan.deg[i] = deg[u];
      plan.local_off[i] = before + off[u];
    }
  }
  if (rank == 0) {
    // offsets are those in the whole output, whichever way the sampling launch adds them up
    if (static_cast<int64_t>(threadIdx.x) < plan.ntiles) plan.tile_off[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
      *plan.total = all;
      if (nnz_out != nullptr) {
        *nnz_out = all;
        __threadfence_system();
      }
    }
  }
  cluster.sync();  // the sums stay until all CTAs have read them
}
static_assert(CLUSTER_PLAN / SAMPLE_TILE <= CLUSTER_PLAN_BLOCK, "a thread per tile offset");

// CTAs of a sampling launch beyond the main ones carry two jobs of the multi-hop sequence that depend on nothing the
// launch does: clearing the table this hop will fill, relabelling the COO of the hop before.
template <typename IdT>
__device__ __forceinline__ bool run_side_job(const SideJobs& jobs) {
  if (blockIdx.x < jobs.main_ctas) return false;
  const unsigned int extra = blockIdx.x - jobs.main_ctas;
  if (extra < jobs.clear.ctas) run_clear_cta(jobs.clear, extra);
  else run_lookup_cta<IdT>(jobs.lookup, extra - jobs.clear.ctas);
  return true;
}

// What a group / warp needs to know about its seed.
struct SeedPlan {
  int64_t rb, deg, o;
};
__device__ __forceinline__ SeedPlan seed_plan(const int64_t* __restrict__ plan_rb,
                                              const int64_t* __restrict__ plan_deg,
                                              const int64_t* __restrict__ local_off,
                                              const int64_t* __restrict__ tile_off, int64_t i, bool valid) {
  SeedPlan p{0, 0, 0};
  if (valid) {
    p.rb = plan_rb[i];
    p.deg = plan_deg[i];
    p.o = (tile_off != nullptr ? tile_off[i / SAMPLE_TILE] : 0) + local_off[i];
  }
  return p;
}

// ---------------------------------------------------------------------------
// uniform sampling: G lanes per seed
// ---------------------------------------------------------------------------
template <typename IdT, int G>
__global__ void __launch_bounds__(SAMPLE_BLOCK, 6)
sample_uniform_kernel(const __grid_constant__ dgs_chunk_desc indices, const IdT* __restrict__ seeds,
                      const Count nc, const int64_t k, const bool replace,
                      const int64_t* __restrict__ plan_rb, const int64_t* __restrict__ plan_deg,
                      const int64_t* __restrict__ local_off, const int64_t* __restrict__ tile_off,
                      const RngKey rng, IdT* coo_row, IdT* coo_col,
                      const int64_t out_capacity, int64_t* __restrict__ picked_pos,
                      const bool row_is_position, const __grid_constant__ SideJobs jobs, const IdMarks marks,
                      int32_t* __restrict__ status) {
  const Emit<IdT> emit{indices, coo_row, coo_col, picked_pos, out_capacity, status, marks, nc};
  pdl_enter();
  if (run_side_job<IdT>(jobs)) return;
  const uint64_t key = key_of(rng);
  constexpr int GROUPS = SAMPLE_BLOCK / G;  // seeds per CTA
  __shared__ uint32_t s_taken[SAMPLE_BLOCK * TAKEN_WORDS_PER_LANE];
  const int group = threadIdx.x / G;  // group inside the CTA
  const int64_t i = static_cast<int64_t>(blockIdx.x) * GROUPS + group;  // the seed this group serves
  // everything that only needs the slot is read before the live count arrives (all arrays have room for
  // nc.bound entries); what belongs to a slot past the count is dropped below
  const bool in_bound = i < nc.bound;
  const SeedPlan sp = seed_plan(plan_rb, plan_deg, local_off, tile_off, i, in_bound);
  const int64_t seed_raw = !in_bound ? 0 : (row_is_position ? i : static_cast<int64_t>(seeds[i]));
  const bool valid = i < count_of(nc);
  const int64_t o = valid ? sp.o : 0;
  if (valid && marks.seeds && (threadIdx.x & (G - 1)) == 0) mark_id(marks, seed_raw, static_cast<uint32_t>(i), status);
  if (!sample_uniform_row(key, i, valid ? sp.deg : 0, k, replace, G, s_taken + group * (G * TAKEN_WORDS_PER_LANE),
                          coo_col + o, o + k <= out_capacity, status,
                          [&](int64_t t, int64_t pos) { emit(o, t, seed_raw, sp.rb, pos); }))
    raise_status(status, DGS_ERR_RANGE);
}

// The same for the common launch: without replacement, k <= G, `indices` in one piece on this GPU and rows and outputs
// that 32-bit arithmetic can hold (see uniform_typed).  Same random numbers, same picks.
// Bound by issue slots: 449 warp instructions per two seeds at 32 registers (76 % of the warps), where the general kernel
// has 544 at 40 (57 %): the address arithmetic of chunked tensors, 64-bit positions and the branches around both.
// 60 000 seeds, fan-out 15: 26 -> 17.7 us.
template <typename IdT, int G, bool MARK>
__global__ void __launch_bounds__(SAMPLE_BLOCK)
sample_uniform_lean_kernel(const IdT* __restrict__ indices, const int64_t n_edges, const IdT* __restrict__ seeds,
                           const Count nc, const uint32_t k, const int64_t* __restrict__ plan_rb,
                           const int64_t* __restrict__ plan_deg, const int64_t* __restrict__ local_off,
                           const int64_t* __restrict__ tile_off, const RngKey rng, IdT* coo_row, IdT* coo_col,
                           const uint32_t out_capacity, const bool row_is_position, const __grid_constant__ SideJobs jobs,
                           const IdMarks marks, int32_t* __restrict__ status) {
  pdl_enter();
  if (!MARK && run_side_job<IdT>(jobs)) return;  // the sequence with marks has no side jobs
  const uint64_t key = key_of(rng);
  constexpr uint32_t GROUPS = SAMPLE_BLOCK / G;  // seeds per CTA
  constexpr uint32_t WORDS = G * TAKEN_WORDS_PER_LANE;
  __shared__ uint32_t s_taken[SAMPLE_BLOCK * TAKEN_WORDS_PER_LANE];
  const uint32_t group = threadIdx.x / G, l = threadIdx.x & (G - 1), lane = threadIdx.x & 31;
  uint32_t* taken = s_taken + group * WORDS;
  const uint32_t i = blockIdx.x * GROUPS + group;  // the seed this group serves
  const bool in_bound = i < nc.bound;              // ahead of the live count: the arrays have room for nc.bound
  const int64_t rb = in_bound ? plan_rb[i] : 0;
  const int64_t deg_plan = in_bound ? plan_deg[i] : 0;
  const uint32_t o = in_bound ? static_cast<uint32_t>(local_off[i] + (tile_off != nullptr ? tile_off[i / SAMPLE_TILE] : 0)) : 0u;
  const IdT seed = row_is_position ? static_cast<IdT>(i) : in_bound ? seeds[i] : IdT(0);
  const bool live = in_bound && (nc.dev == nullptr || i < *nc.dev);
  const uint32_t n_seeds = MARK ? static_cast<uint32_t>(count_of(nc)) : 0u;
  const uint32_t deg = !live ? 0u : deg_plan > 0xFFFFFFFFll ? 0xFFFFFFFFu : static_cast<uint32_t>(deg_plan);
  if (live && deg_plan > 0xFFFFFFFFll) raise_status(status, DGS_ERR_RANGE);  // longer than `indices`: broken row bounds
  if (MARK && marks.seeds && live && l == 0) mark_id(marks, static_cast<int64_t>(seed), i, status);

  const bool sampled = deg > k;
  const bool complement = sampled && deg < 2 * k;  // draw the deg - k positions to leave out
  const uint32_t m = complement ? deg - k : k;     // positions to draw
  const bool active = sampled && l < m;
  const bool in_map = deg <= WORDS * 32;           // longer rows compare candidates across the warp
  if (sampled && in_map)
    for (uint32_t wd = l; wd < (deg + 31) >> 5; wd += G) taken[wd] = 0u;
  __syncwarp();
  bool need = active;
  uint32_t c = l;  // a row that is copied whole: position l
  Philox4 rnd{0u, 0u, 0u, 0u};
#pragma unroll 1
  for (uint32_t round = 0; __any_sync(FULL_MASK, need); ++round) {
    // one Philox block per lane feeds four rounds of (re)draws
    if ((round & 3u) == 0u && active && round < 64) rnd = philox4x32_10(key, i, 0u, ((round >> 2) << 8) | l, TAG_UNIFORM);
    bool usable = true;  // false: this attempt hit Lemire's rejection zone, draw again next round
    if (need) {
      if (round < 64) {
        usable = bounded_try(rnd.x, deg, &c);
        const uint32_t x = rnd.x;  // the next round's word
        rnd.x = rnd.y;
        rnd.y = rnd.z;
        rnd.z = rnd.w;
        rnd.w = x;
      } else {  // never reached in practice: step to a neighbour, keeps the loop bounded
        c = (c + 1 == deg) ? 0 : c + 1;
      }
      if (in_map && usable) {
        const uint32_t bit = 1u << (c & 31u);
        need = (atomicOr(&taken[c >> 5], bit) & bit) != 0u;
      }
    } else {
      const uint32_t x = rnd.x;
      rnd.x = rnd.y;
      rnd.y = rnd.z;
      rnd.z = rnd.w;
      rnd.w = x;
    }
    if (__any_sync(FULL_MASK, active && !in_map)) {
      // lanes holding the same position inside one group see each other; the lowest keeps it
      const bool mine = active && !in_map;
      const unsigned long long tag =
          (mine && usable) ? (static_cast<unsigned long long>(c) | (static_cast<unsigned long long>(lane / G) << 58))
                           : (0x8000000000000000ull | static_cast<unsigned long long>(lane));
      const unsigned same = __match_any_sync(FULL_MASK, tag);
      if (mine) need = !usable || static_cast<uint32_t>(__ffs(same) - 1) != lane;
    }
    if (round >= 64 + 1024) {
      if (need) raise_status(status, DGS_ERR_TABLE_FULL);
      break;
    }
  }
  __syncwarp();

  // what this lane emits: the edge at position c as the row's t-th, or (complement) up to two
  uint32_t t = l, c2 = 0, t2 = 0;
  bool emits = sampled ? active : l < deg, second = false;
  if (complement) {
    // the row has at most 2k-1 <= 63 positions, so its bitmap is one or two words: every lane ranks its own two
    // positions (l and l + G cover the row) among the kept ones
    const unsigned long long out_mask =
        static_cast<unsigned long long>(taken[0]) | (deg > 32 ? static_cast<unsigned long long>(taken[1]) << 32 : 0ull);
    const unsigned long long kept = ~out_mask & ((1ull << deg) - 1ull);
    c = l;
    c2 = l + G;
    emits = (kept >> c) & 1ull;
    second = (kept >> c2) & 1ull;
    t = __popcll(kept & ((1ull << c) - 1ull));
    t2 = __popcll(kept & ((1ull << c2) - 1ull));
  }
  auto emit = [&](uint32_t at, uint32_t pos) {
    if (at >= out_capacity) {
      raise_status(status, DGS_ERR_RANGE);
      return;
    }
    const int64_t e = rb + pos;
    IdT col = static_cast<IdT>(-1);
    if (e < n_edges) col = indices[e];  // row bounds are never negative (the plan)
    else raise_status(status, DGS_ERR_RANGE);
    coo_row[at] = seed;
    coo_col[at] = col;
    if (MARK) mark_id(marks, static_cast<int64_t>(col), n_seeds + at, status);
  };
  if (emits) emit(o + t, c);
  if (second) emit(o + t2, c2);
}

// ---------------------------------------------------------------------------
// weighted sampling: one warp per seed for the first 512 edges of its row; what is
// left of longer rows is dealt out to the eight warps of the CTA
// ---------------------------------------------------------------------------
// a weight of a row that straddles storage regions (at most one row per boundary); out of line, because its
// address arithmetic, inlined at every load, made the sampling kernel 300 KB of code
__device__ __noinline__ float straddling_weight(const dgs_chunk_desc* probs, int64_t e) {
  return load_at<float>(*probs, 2, e);
}

struct RowWeights {
  const dgs_chunk_desc& probs;
  const float* direct;  // non-null when the whole row lies in one storage region
  int64_t rb;
  __device__ __forceinline__ float operator()(int64_t e) const {
    return direct != nullptr ? direct[e] : straddling_weight(&probs, rb + e);
  }
  // COUNT weights at base + 32 j + lane, all loads in flight together; 0 past the row's end
  template <int COUNT>
  __device__ __forceinline__ void load(float (&v)[COUNT], int64_t base, int64_t deg, int l) const {
    if (direct != nullptr) {
      const float* p = direct + base + l;
      if (deg - base >= 32 * COUNT) {
#pragma unroll
        for (int j = 0; j < COUNT; ++j) v[j] = p[j * 32];
      } else {
        const int left = static_cast<int>(deg - base) - l;  // <= 0: none
#pragma unroll
        for (int j = 0; j < COUNT; ++j) v[j] = j * 32 < left ? p[j * 32] : 0.f;
      }
    } else {
#pragma unroll
      for (int j = 0; j < COUNT; ++j) v[j] = base + j * 32 + l < deg ? straddling_weight(&probs, rb + base + j * 32 + l) : 0.f;
    }
  }
};
__device__ __forceinline__ RowWeights row_weights(const dgs_chunk_desc& probs, int64_t rb, int64_t deg) {
  int64_t run;
  const char* wp = resolve(probs, 2, rb, &run);
  return RowWeights{probs, run >= deg ? reinterpret_cast<const float*>(wp) : nullptr, rb};
}

constexpr int64_t HUB_DEG = 4096;  // with replacement: rows above this are left to the whole CTA
constexpr int WEIGHTED_WARPS = SAMPLE_BLOCK / 32;

// One entry of a list of candidates, as an integer whose order is the list's: the key in the high half (both zeros are one
// key), the complement of the edge's place in the low half, so that of equal keys the earlier place comes first.
using Entry = unsigned long long;
constexpr Entry NO_ENTRY = 0x007FFFFF00000000ull;  // key -inf, behind every edge
__device__ __forceinline__ Entry make_entry(float key, uint32_t place) {
  const uint32_t u = __float_as_uint(key + 0.f);
  const uint32_t up = (u & 0x80000000u) ? ~u : u | 0x80000000u;
  return (static_cast<Entry>(up) << 32) | static_cast<uint32_t>(~place);
}
__device__ __forceinline__ float entry_key(Entry e) {
  const uint32_t up = static_cast<uint32_t>(e >> 32);
  return __uint_as_float((up & 0x80000000u) ? up ^ 0x80000000u : ~up);
}
__device__ __forceinline__ uint32_t entry_place(Entry e) { return ~static_cast<uint32_t>(e); }

// Sorts 32 entries, one per lane, the best to lane 0.  Out of line: 15 exchange steps, called from several places.
__device__ __noinline__ Entry sort32(Entry e) {
  const int l = threadIdx.x & 31;
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
    for (int d = size >> 1; d > 0; d >>= 1) {
      const Entry o = __shfl_xor_sync(FULL_MASK, e, d);
      const bool want_larger = ((l & d) == 0) == ((l & size) == 0);
      if ((o > e) == want_larger) e = o;
    }
  }
  return e;
}

// The k-th largest of 32 values, one per lane.
__device__ __forceinline__ float kth_of_32(float v, int l, int k) {
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
    for (int d = size >> 1; d > 0; d >>= 1) {
      const float o = __shfl_xor_sync(FULL_MASK, v, d);
      v = ((l & d) == 0) == ((l & size) == 0) ? fmaxf(v, o) : fminf(v, o);
    }
  }
  return __shfl_sync(FULL_MASK, v, k - 1);
}

// The best edges of a row so far: lane j holds the j-th; `thresh` is the key held by lane k-1 (the bar to beat).
struct ShareList {
  Entry e;
  float thresh;
  __device__ __forceinline__ void set(Entry sorted, int k) {
    e = sorted;
    thresh = entry_key(__shfl_sync(FULL_MASK, e, k - 1));
  }
  // 32 more entries, one per lane, in any order
  __device__ __forceinline__ void merge(Entry more, int l, int k) {
    const Entry c = __shfl_sync(FULL_MASK, sort32(more), 31 - l);
    Entry m = c > e ? c : e;  // the 32 best of both, in bitonic order
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const Entry o = __shfl_xor_sync(FULL_MASK, m, d);
      if ((o > m) == ((l & d) == 0)) m = o;
    }
    set(m, k);
  }
};

// The same with positions of 64 bits, one insertion at a time.
struct RowList {
  float key;
  int64_t pos;
  float thresh;
  __device__ __forceinline__ void insert(float nk, int64_t np, int l, int k) {
    // warp-uniform call with nk > thresh; the keys >= nk form a prefix of the lanes
    const int p = __popc(__ballot_sync(FULL_MASK, key >= nk));  // <= k-1
    const float up_key = __shfl_up_sync(FULL_MASK, key, 1);
    const int64_t up_pos = __shfl_up_sync(FULL_MASK, pos, 1);
    if (l > p) {
      key = up_key;
      pos = up_pos;
    } else if (l == p) {
      key = nk;
      pos = np;
    }
    thresh = __shfl_sync(FULL_MASK, key, k - 1);
  }
};

// Floats in an order-preserving integer form; its own inverse.
__device__ __forceinline__ int ordered_float(float f) {
  const int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float float_of_ordered(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

constexpr float FLOOR_ZERO_W = -3.402823466e+38f;  // key of a weight <= 0: behind every positive weight
constexpr float FLOOR_POS_W = -3.0e+38f;           // clamp for positive weights
constexpr float LEAST_POS_W = -3.2e+38f;           // between the two

__device__ __forceinline__ float ares_key(uint32_t word, float w) {
  float ck = fmaxf(__fdividef(__logf(unit_float(word)), w), FLOOR_POS_W);
  asm volatile("" : "+f"(ck));  // computed by every lane: a branch around it costs more than the few it would spare
  return (w > 0.f) ? ck : FLOOR_ZERO_W;
}

// The next key below: "at or above x" as "above key_below(x)".  Both zeros are one key (log(1) / w is +0, the key of an
// infinite weight -0).
__device__ __forceinline__ float key_below(float x) {
  return x == __int_as_float(0xff800000) ? x : float_of_ordered((x == 0.f ? -1 : ordered_float(x)) - 1);
}

__device__ __forceinline__ Philox4 ares_words(uint64_t key, uint32_t i_lo, uint32_t i_hi, int64_t e0, int l) {
  // one Philox block per four edges, addressed by (seed position, edge index): the result does not depend on
  // which warp scans the window
  const uint64_t ctr = static_cast<uint64_t>(e0 >> 2) + static_cast<uint64_t>(l);
  return philox4x32_10(key, i_lo, i_hi, static_cast<uint32_t>(ctr), static_cast<uint32_t>(ctr >> 32));
}

constexpr int ARES_EDGES = 512;  // edges per window
constexpr int ARES_GROUP = 128;  // edges per step: four per lane, one Philox block

// Edges that passed the filter below and whose keys are still to be computed: of a row's windows of one round, a stretch
// of `room` entries each, with their offsets in the stretch.
struct Survivors {
  static constexpr int ROOM = 256;
  uint2 word_weight[ROOM];
  uint16_t at[ROOM];
  __device__ __forceinline__ Entry* entries() { return reinterpret_cast<Entry*>(word_weight); }
};

// The first 512 edges of a row: every lane computes its 16 keys; the k-th largest of the 32 lane maxima is a bar that at
// least k keys reach and not many more (expected -32 ln(1 - k/32) of them: 12 at k = 10, 22 at k = 16, 31 at k = 20, 49 at
// k = 25, 130 at k = 32), so those are packed and sorted 32 at a time.
// With fewer than k lanes that have a positive weight the bar is the key of zero weights.  Of those only the ones among the
// first 32 edges count, which with the positive ones are k already.  False: more reach the bar than there is room for
// (keys that are equal).
__device__ __forceinline__ bool ares_first_window(ShareList& top, const RowWeights& W, int64_t deg, uint64_t key, uint32_t i_lo,
                                                  uint32_t i_hi, int l, int k, Entry* pack) {
  constexpr int ITEMS = ARES_EDGES / 32;
  const float NEG_INF = __int_as_float(0xff800000);
  float ck[ITEMS];
  W.load(ck, 0, deg, l);
  float best = NEG_INF;
  const int left = deg < ARES_EDGES ? static_cast<int>(deg) - l : ARES_EDGES;
#pragma unroll
  for (int q = 0; q < ITEMS / 4; ++q) {
    if (q * ARES_GROUP < deg) {  // warp-uniform
      const Philox4 r = ares_words(key, i_lo, i_hi, q * ARES_GROUP, l);
      const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
      for (int j = 4 * q; j < 4 * q + 4; ++j) {
        ck[j] = j * 32 < left ? ares_key(rw[j - 4 * q], ck[j]) : NEG_INF;
        best = fmaxf(best, ck[j]);
      }
    } else {
#pragma unroll
      for (int j = 4 * q; j < 4 * q + 4; ++j) ck[j] = NEG_INF;
    }
  }
  if (deg <= 32) {
    top.set(sort32(ck[0] > NEG_INF ? make_entry(ck[0], l) : NO_ENTRY), k);
    return true;
  }
  const float bar = kth_of_32(best, l, k);
  const float rest = fmaxf(bar, LEAST_POS_W);  // what the edges behind the first 32 have to reach
  int have = 0;
#pragma unroll
  for (int q = 0; q < ITEMS / 4; ++q) {
    if (q * ARES_GROUP >= deg) break;  // warp-uniform
#pragma unroll
    for (int j = 4 * q; j < 4 * q + 4; ++j) {
      const bool in = ck[j] >= (j == 0 ? bar : rest);
      const unsigned m = __ballot_sync(FULL_MASK, in);
      const int at = have + __popc(m & ((1u << l) - 1u));
      if (in && at < Survivors::ROOM) pack[at] = make_entry(ck[j], j * 32 + l);
      have += __popc(m);
    }
  }
  __syncwarp();
  const bool fits = have <= Survivors::ROOM;
  if (fits) {
    top.set(sort32(l < have ? pack[l] : NO_ENTRY), k);
#pragma unroll 1
    for (int i0 = 32; i0 < have; i0 += 32) {
      const Entry e = i0 + l < have ? pack[i0 + l] : NO_ENTRY;
      if (__any_sync(FULL_MASK, entry_key(e) > top.thresh)) top.merge(e, l, k);  // of equal keys the earlier win
    }
  }
  __syncwarp();  // the room is used again
  return fits;
}

// The order of equal keys (zero weights, equal weights): window w of 512 edges belongs to share w % 8; equal keys are
// ordered by share and then position, which up to eight windows is by position.  The tag of an edge holds that in 32
// bits for rows below 2^32 edges.
constexpr int ARES_SHARES = 8;
__device__ __forceinline__ uint32_t window_tag(int64_t window) {
  return (static_cast<uint32_t>(window & (ARES_SHARES - 1)) << 29) | (static_cast<uint32_t>(window / ARES_SHARES) * ARES_EDGES);
}
// position in the row of a place (512 per window) in share r
__device__ __forceinline__ int64_t position_of(int r, uint32_t place) {
  return static_cast<int64_t>(place & ~(ARES_EDGES - 1u)) * ARES_SHARES + r * ARES_EDGES + (place & (ARES_EDGES - 1u));
}
__device__ __forceinline__ int64_t tag_position(uint32_t tag) { return position_of(static_cast<int>(tag >> 29), tag & 0x1FFFFFFFu); }

// Of a row's n edges only about k (1 + ln(n/k)) ever enter its list, so the logarithm and the division are spent only on
// edges that a bound lets through: log(u) <= u - 1, so an edge whose u - 1 <= bar * w cannot beat the bar.  The test is
// that inequality with the slack that the errors of __logf (2^-21.4 absolute on [0.5, 2]), __fdividef (2 ulp) and of the 23
// random bits it looks at need, so every edge that the exact key lets in passes, and the exact key decides.  A bar above
// -2.5e-38 is taken as that: keys nearer to zero than 2^-126 may come out as zero, those of weights from 2^126 on do.  (With
// -1e-30 in its place a row of weights around 1e32 passed as a whole.)  At or below the clamp of positive weights the
// inequality says nothing about keys that were clamped, and every positive weight passes.  Weights <= 0 (or no number) do
// not: a list that is full has had them from the row's first edges, which come before all others of that key.  (For a
// list that is not full yet: `zeros`.)
constexpr float ARES_PASS = 2.0f - 0x1p-18f;
__device__ __forceinline__ float filter_bar(float above) {  // for keys above `above`
  return above <= FLOOR_POS_W ? __int_as_float(0xff800000) : fminf(above * 1.00001f, -2.5e-38f);
}
__device__ __forceinline__ bool may_beat(float bar, uint32_t word, float w) {
  return __uint_as_float((word >> 9) | 0x3f800000u) > fmaf(bar, fmaxf(w, 0.f), ARES_PASS);  // not above NaN: -inf * 0
}

// The edges of a window (`base`: its first edge) that may beat `bar`, behind the `have` that are in s[from, from + room)
// already, their offsets counted from `off`; their number, which may exceed the room: what has none is dropped.  (Past the
// row's end weights are 0; what passes there is left out when the keys are computed.)
__device__ __forceinline__ int ares_collect(const RowWeights& W, int64_t deg, int64_t base, uint64_t key, uint32_t i_lo,
                                            uint32_t i_hi, int l, float bar, Survivors& s, int from, int room, int have,
                                            int off) {
  float w[16];
  W.load(w, base, deg, l);
  const uint64_t ctr = static_cast<uint64_t>(base >> 2);  // the low seven bits are clear
  const uint32_t c_lo = static_cast<uint32_t>(ctr) | l, c_hi = static_cast<uint32_t>(ctr >> 32);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (base + q * ARES_GROUP >= deg) break;  // warp-uniform
    const Philox4 rnd = philox4x32_10(key, i_lo, i_hi, c_lo + q * 32, c_hi);
    const uint32_t rw[4] = {rnd.x, rnd.y, rnd.z, rnd.w};
    bool pass[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) pass[j] = may_beat(bar, rw[j], w[q * 4 + j]);
    if (!__any_sync(FULL_MASK, pass[0] || pass[1] || pass[2] || pass[3])) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const unsigned m = __ballot_sync(FULL_MASK, pass[j]);
      const int at = have + __popc(m & ((1u << l) - 1u));
      if (pass[j] && at < room) {
        s.word_weight[from + at] = make_uint2(rw[j], __float_as_uint(w[q * 4 + j]));
        s.at[from + at] = static_cast<uint16_t>(off + q * ARES_GROUP + j * 32 + l);
      }
      have += __popc(m);
    }
  }
  return have;
}

// A list, and the edges [lo, hi) of one window: the best of both, whatever the weights are.  For what ares_collect has no room
// for.  Keys above `above` that may enter are put aside (waiting[63]), and whenever 32 are waiting they are sorted and merged.
// place0: of edge lo.
__device__ __noinline__ Entry ares_window(Entry list, const dgs_chunk_desc* probs, int64_t rb, int64_t deg, int64_t lo, int64_t hi,
                                          uint64_t key, uint32_t i_lo, uint32_t i_hi, uint32_t place0, float above, bool zeros,
                                          int l, int k, Entry* waiting) {
  const RowWeights W = row_weights(*probs, rb, deg);
  ShareList top;
  top.set(list, k);
  float bar = filter_bar(fmaxf(above, key_below(top.thresh)));
  int have = 0;
#pragma unroll 1
  for (int64_t e0 = lo; e0 < hi && e0 < deg; e0 += ARES_GROUP) {
    float w[4];
    W.load(w, e0, deg, l);
    const Philox4 r = ares_words(key, i_lo, i_hi, e0, l);
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      const uint32_t word = j == 0 ? r.x : j == 1 ? r.y : j == 2 ? r.z : r.w;
      const float weight = j == 0 ? w[0] : j == 1 ? w[1] : j == 2 ? w[2] : w[3];
      const bool pass = e0 + j * 32 + l < deg && (may_beat(bar, word, weight) || (zeros && bar == __int_as_float(0xff800000)));
      if (!__any_sync(FULL_MASK, pass)) continue;
      const float ck = ares_key(word, weight);
      const Entry e = make_entry(ck, place0 + static_cast<uint32_t>(e0 - lo) + j * 32 + l);
      const Entry last = __shfl_sync(FULL_MASK, top.e, k - 1);
      const bool in = pass && ck > above && e > last;
      const unsigned m = __ballot_sync(FULL_MASK, in);
      if (in) waiting[have + __popc(m & ((1u << l) - 1u))] = e;
      have += __popc(m);
      if (have < 32) continue;
      __syncwarp();
      const Entry one = waiting[l], two = l + 32 < have ? waiting[l + 32] : NO_ENTRY;
      __syncwarp();
      if (l + 32 < have) waiting[l] = two;
      have -= 32;
      top.merge(one, l, k);
      bar = filter_bar(fmaxf(above, key_below(top.thresh)));
    }
  }
  __syncwarp();
  if (have > 0) top.merge(l < have ? waiting[l] : NO_ENTRY, l, k);
  __syncwarp();
  return top.e;
}

// Joins a row's list with what its windows from w0 on have collected: stretch b, of `room` entries and `windows` windows, holds
// as many as lane b says.
// With more than 32 the k-th largest of the lanes' best keys is a bar that few more than k reach (for k well below 32),
// so that one sort and one merge do.
__device__ __forceinline__ void ares_join(ShareList& top, Survivors& s, int count, int room, int64_t w0, int windows, int64_t deg,
                                          int l, int k) {
  int upto = count;  // entries of the stretches up to this lane's
#pragma unroll
  for (int o = 1; o < ARES_SHARES; o <<= 1) {
    const int t = __shfl_up_sync(FULL_MASK, upto, o);
    if (l >= o) upto += t;
  }
  const int total = __shfl_sync(FULL_MASK, upto, ARES_SHARES - 1);
  if (total == 0) return;
  // the i-th entry of all: its stretch, and its slot
  auto slot_of = [&](int i, int* stretch) {
    int b = 0, before = 0;
#pragma unroll
    for (int x = 0; x < ARES_SHARES - 1; ++x) {
      const int end = __shfl_sync(FULL_MASK, upto, x);
      if (i >= end) {
        b = x + 1;
        before = end;
      }
    }
    *stretch = b;
    return b * room + i - before;
  };
  Entry* out = s.entries();
  Entry first = NO_ENTRY, best = NO_ENTRY;
  __syncwarp();
#pragma unroll 1
  for (int i0 = 0; i0 < total; i0 += 32) {
    int b;
    const int slot = slot_of(i0 + l, &b);
    Entry e = NO_ENTRY;
    if (i0 + l < total) {
      const uint2 x = s.word_weight[slot];
      const uint32_t off = s.at[slot];
      const int64_t w = w0 + b * windows + off / ARES_EDGES;
      if (w * ARES_EDGES + off % ARES_EDGES < deg)
        e = make_entry(ares_key(x.x, __uint_as_float(x.y)), window_tag(w) + off % ARES_EDGES);
      out[slot] = e;
      best = e > best ? e : best;
    }
    if (i0 == 0) first = e;
  }
  if (total <= 32) {
    if (__any_sync(FULL_MASK, entry_key(first) >= top.thresh)) top.merge(first, l, k);
    return;
  }
  float bar = top.thresh;
  bar = fmaxf(bar, kth_of_32(entry_key(best), l, k));
  __syncwarp();
  // those that reach the bar, 32 at a time.  Packed in place: what is written lies in front of what is still to be read
  int have = 0;
#pragma unroll 1
  for (int i0 = 0; i0 < total; i0 += 32) {
    int b;
    const int slot = slot_of(i0 + l, &b);
    const Entry e = i0 + l < total ? out[slot] : NO_ENTRY;
    const bool in = e != NO_ENTRY && entry_key(e) >= bar;
    const unsigned m = __ballot_sync(FULL_MASK, in);
    __syncwarp();
    if (in) out[have + __popc(m & ((1u << l) - 1u))] = e;  // at most 31 + 32 of them
    have += __popc(m);
    __syncwarp();
    const bool last = i0 + 32 >= total;
    if (have >= 32 || last) {
      const Entry one = l < have ? out[l] : NO_ENTRY, two = l + 32 < have ? out[l + 32] : NO_ENTRY;
      __syncwarp();
      if (have > 0) top.merge(one, l, k);
      if (have > 32) {
        if (last) top.merge(two, l, k);
        else if (l + 32 < have) out[l] = two;
      }
      have = have > 32 ? have - 32 : 0;
      __syncwarp();
    }
  }
}

// A row's list with its windows [first, last), which had more survivors than room: once more, window by window, with the bar that
// there is now and all of the row's room.
__device__ __forceinline__ Entry ares_again(Entry list, const dgs_chunk_desc* probs, int64_t rb, int64_t deg, int64_t first, int64_t last,
                                         uint64_t key, uint32_t i_lo, uint32_t i_hi, int l, int k, Survivors* s) {
  ShareList top;
  top.set(list, k);
#pragma unroll 1
  for (int64_t w = first; w < last && w * ARES_EDGES < deg; ++w) {
    const float above = key_below(top.thresh);
    __syncwarp();
    const int have = ares_collect(row_weights(*probs, rb, deg), deg, w * ARES_EDGES, key, i_lo, i_hi, l, filter_bar(above), *s, 0,
                                  Survivors::ROOM, 0, 0);
    if (have <= Survivors::ROOM) {
      ares_join(top, *s, l == 0 ? have : 0, Survivors::ROOM, w, 1, deg, l, k);
    } else {
      __syncwarp();
      top.set(ares_window(top.e, probs, rb, deg, w * ARES_EDGES, (w + 1) * ARES_EDGES, key, i_lo, i_hi, window_tag(w), above, false, l,
                          k, s->entries()), k);
    }
  }
  return top.e;
}

// A whole row by one warp, share after share, for rows whose tags do not fit 32 bits; lane t's position of rank t.
__device__ __noinline__ int64_t ares_row(const dgs_chunk_desc* probs, int64_t rb, int64_t deg, uint64_t key, uint32_t i_lo,
                                         uint32_t i_hi, int l, int k, Entry* waiting) {
  RowList row{__int_as_float(0xff800000), 0, __int_as_float(0xff800000)};
#pragma unroll 1
  for (int r = 0; r < ARES_SHARES; ++r) {
    uint32_t place = 0;
#pragma unroll 1
    do {
      const int64_t lo = position_of(r, place);
      if (lo >= deg) break;
      const Entry list = ares_window(NO_ENTRY, probs, rb, deg, lo, lo + ARES_EDGES, key, i_lo, i_hi, 0u, row.thresh, lo == 0, l, k,
                                     waiting);
#pragma unroll 1
      for (int t = 0; t < k; ++t) {
        const Entry next = __shfl_sync(FULL_MASK, list, t);
        if (!(entry_key(next) > row.thresh)) break;  // the list is sorted: the rest of it is behind the bar too
        row.insert(entry_key(next), lo + entry_place(next), l, k);
      }
      place += ARES_EDGES;
    } while (place != 0);  // 0: past 2^32 places
  }
  return row.pos;
}

// What the warps of a CTA share of its eight rows.
struct AresRows {
  int how[WEIGHTED_WARPS];
  float bar[WEIGHTED_WARPS];
  int64_t rb[WEIGHTED_WARPS], deg[WEIGHTED_WARPS], off[WEIGHTED_WARPS], seed[WEIGHTED_WARPS];
  int64_t left[WEIGHTED_WARPS];  // deg where there are windows to scan, else 0
  int count[WEIGHTED_WARPS][ARES_SHARES];
  __align__(16) Survivors scratch[WEIGHTED_WARPS];
};

// One round: the windows from w0 on of all rows, in stretches of up to `most` (1 unless LONG), of which a row has room for so
// many, are dealt out to the warps, which only collect the edges that may beat the row's bar; each row's own warp joins what was
// collected with its list.  False: no row has windows left.  *crowded: some stretch took more than half of its room (LONG).
template <bool LONG>
__device__ __forceinline__ bool ares_round(AresRows& c, ShareList& top, const dgs_chunk_desc& probs, uint64_t key, int64_t i0, int l,
                                           int warp, int k, int64_t w0, int room, int most, bool* crowded) {
  const int stretches = Survivors::ROOM / room;
  // lane r: the stretches of row r in this round, their windows, and how many tasks the rows up to it make
  const int64_t rest = (l < WEIGHTED_WARPS ? c.left[l] : 0) - w0 * ARES_EDGES;
  const int left = rest <= 0 ? 0 : static_cast<int>((rest + ARES_EDGES - 1) / ARES_EDGES);
  if (__ballot_sync(FULL_MASK, left > 0) == 0u) return false;  // the same for all warps
  const int even = (left + stretches - 1) / stretches, windows = !LONG || even < 1 ? 1 : even < most ? even : most;
  const int parts = LONG ? (left + windows - 1) / windows : left;
  int upto = parts < stretches ? parts : stretches;
#pragma unroll
  for (int o = 1; o < WEIGHTED_WARPS; o <<= 1) {
    const int t = __shfl_up_sync(FULL_MASK, upto, o);
    if (l >= o) upto += t;
  }
  const int tasks = __shfl_sync(FULL_MASK, upto, WEIGHTED_WARPS - 1);
  bool dense = false;
#pragma unroll 1
  for (int t = warp; t < tasks; t += WEIGHTED_WARPS) {
    const int row = __popc(__ballot_sync(FULL_MASK, l < WEIGHTED_WARPS && upto <= t));
    const int b = t - (row > 0 ? __shfl_sync(FULL_MASK, upto, row - 1) : 0);  // row: the same in all lanes
    const int count = LONG ? __shfl_sync(FULL_MASK, windows, row) : 1;
    const int64_t deg = c.deg[row], first = w0 + static_cast<int64_t>(b) * count;
    // a key equal to the bar may still win: its share may come before the one that holds the bar
    const float bar = filter_bar(key_below(c.bar[row]));
    int have = 0;
#pragma unroll 1
    for (int w = 0; w < count && (!LONG || (first + w) * ARES_EDGES < deg); ++w)
      have = ares_collect(row_weights(probs, c.rb[row], deg), deg, (first + w) * ARES_EDGES, key, static_cast<uint32_t>(i0 + row),
                          static_cast<uint32_t>((i0 + row) >> 32), l, bar, c.scratch[row], b * room, room, have, w * ARES_EDGES);
    dense = dense || have > room / 2;
    if (l == 0) c.count[row][b] = have;
  }
  if (LONG) *crowded = __syncthreads_or(dense);
  else __syncthreads();
  const int own = __shfl_sync(FULL_MASK, upto, warp) - (warp > 0 ? __shfl_sync(FULL_MASK, upto, warp - 1) : 0);
  const int own_windows = LONG ? __shfl_sync(FULL_MASK, windows, warp) : 1;
  if (own > 0) {
    const int count = l < own ? c.count[warp][l] : 0;
    ares_join(top, c.scratch[warp], count > room ? 0 : count, room, w0, own_windows, c.deg[warp], l, k);
    for (unsigned again = __ballot_sync(FULL_MASK, count > room); again != 0u; again &= again - 1) {
      const int64_t first = w0 + static_cast<int64_t>(__ffs(again) - 1) * own_windows;
      top.set(ares_again(top.e, &probs, c.rb[warp], c.deg[warp], first, first + own_windows, key, static_cast<uint32_t>(i0 + warp),
                         static_cast<uint32_t>((i0 + warp) >> 32), l, k, &c.scratch[warp]), k);
    }
    if (l == 0) c.bar[warp] = top.thresh;
  }
  __syncthreads();
  return true;
}

// The rounds from window ARES_SHORT on.  A window has about k / w survivors of the bar of w windows, so that those of eight
// stretches of w / 8 windows are few beside the room; the rounds double, and a row of 10^5 edges takes 8 of them instead of 24.
// Where a stretch takes more than half of its room -- weights that rise along the row -- they stay half as long from there on.
// One such row alone in its CTA, whole calls, fan-out 10 and 25: 73.9 and 127 us with eight (four) windows a round throughout,
// 56 and 61 now; 64 of them 297 and 352 -> 273 and 280.  Out of line, and not before window 33: rows of a hub-heavy graph are
// shorter and paid for it (11 000 rows, fan-out 10: 60.8 without, 62.6 from window 17 on, 60.5 from 33 on, 61.0 from 65 on).
constexpr int ARES_SHORT = 33;
__device__ __noinline__ Entry ares_long_rounds(Entry list, AresRows* c, const dgs_chunk_desc* probs, uint64_t key, int64_t i0, int l,
                                               int warp, int k, int64_t w0) {
  ShareList top;
  top.set(list, k);
  constexpr int room = 32;
  bool crowded = false;
  for (int most = 2, cap = 64; ares_round<true>(*c, top, *probs, key, i0, l, warp, k, w0, room, most, &crowded);) {
    w0 += Survivors::ROOM / room * most;
    if (!crowded) most = min(min(2 * most, static_cast<int>(w0 >> 3)), cap);
    else if (most > 1) cap = most >>= 1;
  }
  return top.e;
}

// (The exponential-jump form of the sampler -- keys only for the edges that enter, a
// streamed prefix sum for the rest -- was built and measured here: with fan-outs of
// 10-32 and rows of 10^3-10^4 edges an entry costs ~250 instructions at a rate of k/n
// per edge, and the kernel ran 1.6-2.3x slower than with per-edge keys, so it is not used.)

// A-Res without replacement.  Bound by issue slots and the CTA's barriers, not by the bytes of the weights.  Eight seeds per CTA
// of eight warps.  Each warp takes the first 512 edges of its own row, which gives the row a list and a bar to beat; then, in
// rounds, the windows behind them are dealt out to the CTA's warps, which only collect the edges that may beat the bar, and each
// row's own warp joins what was collected with the list: one sort and one merge a round.
// 11 000 rows of a hub-heavy graph (9.1 M weights), whole calls, a list per share of the row kept by its warp -> this:
// fan-out 10 69.6 -> 60.6, 20 90.9 -> 69, 25 109 -> 70.6; 2 000 rows, fan-out 15 57.5 -> 33.9; 2 000 rows of 4 096 edges, fan-out 10
// 61.4 -> 37.5.  Rows of which few weights are positive are as fast: one in a hundred, fan-out 10, 94.7 -> 61.  (Four CTAs per
// SM at 64 registers: level; two at 128: 66.7 for 60.6.)
template <typename IdT>
__global__ void __launch_bounds__(SAMPLE_BLOCK, 3)
sample_weighted_kernel(const __grid_constant__ dgs_chunk_desc indices,
                       const __grid_constant__ dgs_chunk_desc probs, const IdT* __restrict__ seeds,
                       const Count nc, const int64_t k,
                       const int64_t* __restrict__ plan_rb, const int64_t* __restrict__ plan_deg,
                       const int64_t* __restrict__ local_off, const int64_t* __restrict__ tile_off,
                       const RngKey rng, IdT* coo_row, IdT* coo_col,
                       const int64_t out_capacity, int64_t* __restrict__ picked_pos,
                       const bool row_is_position, const __grid_constant__ SideJobs jobs, const IdMarks marks,
                       int32_t* __restrict__ status) {
  const Emit<IdT> emit{indices, coo_row, coo_col, picked_pos, out_capacity, status, marks, nc};
  pdl_enter();
  if (run_side_job<IdT>(jobs)) return;
  const uint64_t key = uniform_word(key_of(rng) ^ (static_cast<uint64_t>(TAG_ARES) << 32));
  const int64_t n = count_of(nc);
  const int l = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int kk = static_cast<int>(k);
  enum : int { NOTHING, WHOLE, LIST, ALONE };  // how a warp's row is sampled; ALONE: by the warp, behind everything else
  __shared__ AresRows c;

  const int64_t i0 = static_cast<int64_t>(blockIdx.x) * WEIGHTED_WARPS;
  ShareList top{NO_ENTRY, __int_as_float(0xff800000)};
  {
    SeedPlan sp{0, 0, 0};
    int64_t seed = 0;
    int how = NOTHING;
    if (i0 + warp < n) {
      sp = seed_plan(plan_rb, plan_deg, local_off, tile_off, i0 + warp, true);
      seed = row_is_position ? i0 + warp : static_cast<int64_t>(seeds[i0 + warp]);
      if (marks.seeds && l == 0) mark_id(marks, seed, static_cast<uint32_t>(i0 + warp), status);
      if (sp.deg <= k) {
        how = WHOLE;
      } else if (sp.rb + sp.deg > probs.total || sp.deg >> 35 != 0) {  // places within a share fit 32 bits below 2^35
        if (l == 0) raise_status(status, DGS_ERR_RANGE);
      } else if (sp.deg >> 32 != 0) {
        how = ALONE;
      } else {
        how = LIST;
        const uint32_t i_lo = static_cast<uint32_t>(i0 + warp), i_hi = static_cast<uint32_t>((i0 + warp) >> 32);
        const RowWeights W = row_weights(probs, sp.rb, sp.deg);
        Survivors& s = c.scratch[warp];
        if (!ares_first_window(top, W, sp.deg, key, i_lo, i_hi, l, kk, s.entries()))
          top.set(ares_window(NO_ENTRY, &probs, sp.rb, sp.deg, 0, ARES_EDGES, key, i_lo, i_hi, 0u, __int_as_float(0xff800000), true,
                              l, kk, s.entries()), kk);
      }
    }
    if (l == 0) {
      c.how[warp] = how;
      c.rb[warp] = sp.rb;
      c.deg[warp] = sp.deg;
      c.off[warp] = sp.o;
      c.seed[warp] = seed;
      c.left[warp] = how == LIST && sp.deg > ARES_EDGES ? sp.deg : 0;
      c.bar[warp] = top.thresh;
    }
  }
  __syncthreads();
  // with the bar of one window a window has about k survivors, give or take sqrt(2k)
  int64_t w0 = 1;
  bool more = true;
  while (more && w0 < ARES_SHORT) {
    const int room = w0 == 1 && kk > 10 ? 64 : 32;
    more = ares_round<false>(c, top, probs, key, i0, l, warp, kk, w0, room, 1, nullptr);
    w0 += Survivors::ROOM / room;
  }
  if (more) top.set(ares_long_rounds(top.e, &c, &probs, key, i0, l, warp, kk, w0), kk);
  const int how = c.how[warp];
  if (how == NOTHING) return;
  int64_t pick = -1;  // lane l emits the edge at `pick` as the seed's l-th
  if (how == WHOLE) {
    if (l < c.deg[warp]) pick = l;
  } else if (how == LIST) {
    if (l < k) pick = tag_position(entry_place(top.e));
  } else {
    const uint64_t i = static_cast<uint64_t>(i0 + warp);
    const int64_t at = ares_row(&probs, c.rb[warp], c.deg[warp], key, static_cast<uint32_t>(i), static_cast<uint32_t>(i >> 32), l,
                                kk, c.scratch[warp].entries());
    if (l < k) pick = at;
  }
  if (pick >= 0) emit(c.off[warp], l, c.seed[warp], c.rb[warp], pick);
}

// ---- proportional draws with replacement --------------------------------------
// A row is kept as the sums of stretches of 2^m * 32 edges, at most 128 of them, in shared memory: groups of 32 for
// rows of up to 4096 edges.  The sums of a 512-edge window (16 loads per lane in flight) are folded across the warp
// with 16 shuffles in all, where a scan of every 32 edges takes 80, and their prefixes are formed once per row; each
// lane then looks its own draw up by bisection and walks the 32 edges that it falls into.
struct CtaSeeds {  // what phase 1 read about the CTA's seeds
  int64_t rb[WEIGHTED_WARPS], deg[WEIGHTED_WARPS], o[WEIGHTED_WARPS], seed[WEIGHTED_WARPS];
};

constexpr int MAX_GROUPS = 128;
constexpr int WINDOW_ITEMS = 16;

// 16 sums of 32 edges from `base`, sum j in lanes 2j and 2j + 1
__device__ __forceinline__ float group_sums(const RowWeights& W, int64_t base, int64_t deg, int l) {
  float v[WINDOW_ITEMS];
  W.load(v, base, deg, l);
#pragma unroll
  for (int j = 0; j < WINDOW_ITEMS; ++j) v[j] = fmaxf(v[j], 0.f);
#pragma unroll
  for (int half = 8, d = 16; half >= 1; half >>= 1, d >>= 1) {
    const bool upper = (l & d) != 0;
#pragma unroll
    for (int j = 0; j < half; ++j) {
      const float give = upper ? v[j] : v[j + half];
      v[j] = (upper ? v[j + half] : v[j]) + __shfl_xor_sync(FULL_MASK, give, d);
    }
  }
  return v[0] + __shfl_xor_sync(FULL_MASK, v[0], 1);
}

__device__ __forceinline__ float warp_inclusive_sum(float s, int l) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const float t = __shfl_up_sync(FULL_MASK, s, d);
    if (l >= d) s += t;
  }
  return s;
}

// The edge of the 32 from `base` that r (a distance into their sum) falls on: the first with a weight whose prefix
// is above r, the last with a weight where rounding leaves none.  -1: no edge of them has a weight, or r is not
// below their sum and !stop_here (r is then what is left behind them).
__device__ __forceinline__ int64_t edge_of_32(const RowWeights& W, int64_t base, int64_t deg, float* r, bool stop_here,
                                              int l) {
  const int64_t e = base + l;
  const float w = (e < deg) ? fmaxf(W(e), 0.f) : 0.f;
  const float s = warp_inclusive_sum(w, l);
  const unsigned some = __ballot_sync(FULL_MASK, w > 0.f);
  const unsigned hit = __ballot_sync(FULL_MASK, w > 0.f && s > *r);
  if (hit) return base + __ffs(hit) - 1;
  if (stop_here) return some ? base + 31 - __clz(static_cast<int>(some)) : -1;
  *r -= __shfl_sync(FULL_MASK, s, 31);
  return -1;
}

struct RowGroups {
  float sum[MAX_GROUPS];   // of each group
  float incl[MAX_GROUPS];  // inclusive prefix
};

// groups g0, g0 + step, ... of the row (in units of one window when shift == 0)
__device__ __forceinline__ void sum_groups(const RowWeights& W, int64_t deg, int shift, int first, int step, int l,
                                           float* sum) {
  if (shift == 0) {
    for (int64_t w = first; w * 512 < deg; w += step) {
      const float s = group_sums(W, w * 512, deg, l);
      if ((l & 1) == 0 && w * 512 + (l >> 1) * 32 < deg) sum[w * 16 + (l >> 1)] = s;
    }
  } else {
    const int64_t len = static_cast<int64_t>(32) << shift;
    for (int64_t g = first; g * len < deg; g += step) {
      const int64_t end = (g + 1) * len < deg ? (g + 1) * len : deg;
      float acc = 0.f;
      for (int64_t b = g * len; b < end; b += 512) acc += group_sums(W, b, end, l);
      // lanes 2j and 2j + 1 hold the same sum: fold over j
#pragma unroll
      for (int d = 2; d < 32; d <<= 1) acc += __shfl_xor_sync(FULL_MASK, acc, d);
      if (l == 0) sum[g] = acc;
    }
  }
}

__device__ __forceinline__ int group_shift(int64_t deg) {
  int shift = 0;
  while ((static_cast<int64_t>(32 * MAX_GROUPS) << shift) < deg) ++shift;
  return shift;
}

// prefixes of the row's group sums; returns the row's total.  sum[] past the last group is 0.
__device__ __forceinline__ float prefix_groups(RowGroups& g, int l) {
  float4 v = reinterpret_cast<const float4*>(g.sum)[l];
  v.y += v.x;
  v.z += v.y;
  v.w += v.z;
  // the sums of a scan are rounded each in its own way: the largest so far, so that prefixes never step back
  float last = warp_inclusive_sum(v.w, l);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const float t = __shfl_up_sync(FULL_MASK, last, d);
    if (l >= d) last = fmaxf(last, t);
  }
  const float up = __shfl_up_sync(FULL_MASK, last, 1);
  const float base = l == 0 ? 0.f : up;
  reinterpret_cast<float4*>(g.incl)[l] =
      make_float4(fminf(base + v.x, last), fminf(base + v.y, last), fminf(base + v.z, last), last);
  return __shfl_sync(FULL_MASK, last, 31);
}

// This lane's draw (0 <= draw < total): the group it falls into, and what is left of it there.
__device__ __forceinline__ int group_of(const RowGroups& g, float draw, float* rest) {
  int lo = 0, hi = MAX_GROUPS - 1;  // first group whose inclusive prefix is above the draw
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (g.incl[mid] > draw) hi = mid;
    else lo = mid + 1;
  }
  while (lo < MAX_GROUPS - 1 && !(g.sum[lo] > 0.f)) ++lo;  // rounding can lift a group that adds nothing
  while (lo > 0 && !(g.sum[lo] > 0.f)) --lo;
  *rest = lo > 0 ? draw - g.incl[lo - 1] : draw;
  return lo;
}

// Bound by the latency of dependent loads and shuffles, not by bytes.  One warp per row of up to HUB_DEG edges;
// longer rows are summed by all warps of the CTA.  4 096 rows, 1.4 M weights, fan-out 10: 13 us, against 68 us when a
// warp scanned every 32 edges of its row twice.
template <typename IdT>
__global__ void __launch_bounds__(SAMPLE_BLOCK)
sample_weighted_replace_kernel(const __grid_constant__ dgs_chunk_desc indices,
                               const __grid_constant__ dgs_chunk_desc probs, const IdT* __restrict__ seeds,
                               const Count nc, const int64_t k,
                               const int64_t* __restrict__ plan_rb, const int64_t* __restrict__ plan_deg,
                               const int64_t* __restrict__ local_off, const int64_t* __restrict__ tile_off,
                               const RngKey rng, IdT* coo_row, IdT* coo_col,
                               const int64_t out_capacity, int64_t* __restrict__ picked_pos,
                               const bool row_is_position, const __grid_constant__ SideJobs jobs, const IdMarks marks,
                               int32_t* __restrict__ status) {
  const Emit<IdT> emit{indices, coo_row, coo_col, picked_pos, out_capacity, status, marks, nc};
  pdl_enter();
  if (run_side_job<IdT>(jobs)) return;
  const uint64_t key = key_of(rng);
  const int64_t n = count_of(nc);
  const int l = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  __shared__ __align__(16) RowGroups s_row[WEIGHTED_WARPS];
  __shared__ int s_long[WEIGHTED_WARPS];
  __shared__ int s_nlong;
  __shared__ CtaSeeds s_seed;
  if (threadIdx.x == 0) s_nlong = 0;
  for (int x = l; x < MAX_GROUPS; x += 32) s_row[warp].sum[x] = 0.f;
  __syncthreads();

  // draws t0 .. t0 + 31 of a row, one per lane; the calling warp resolves them all
  auto draws = [&](const RowGroups& g, float total, const RowWeights& W, int64_t deg, int64_t i, int64_t seed,
                   int64_t rb, int64_t o, int64_t t0) {
    const int64_t t = t0 + l;
    const uint32_t i_lo = static_cast<uint32_t>(i), i_hi = static_cast<uint32_t>(static_cast<uint64_t>(i) >> 32);
    const Philox4 r = philox4x32_10(key, i_lo, i_hi, static_cast<uint32_t>(t), TAG_WREPL);
    const float draw = unit_float(r.x) * total;
    const int shift = group_shift(deg);
    int64_t pos = deg - 1;  // a draw not below the final sum maps to the last edge
    float rest = 0.f;
    int group = -1;
    if (t < k && draw < total) group = group_of(g, draw, &rest);
    if (shift == 0) {
      // 32 edges, just read: every lane walks those of its own draw (a scan by the whole warp per draw takes ~60
      // instructions a draw; this takes ~160 for all 32)
      if (group >= 0) {
        const int lo = group * 32, end = lo + 32 < deg ? lo + 32 : static_cast<int>(deg);
        float s = 0.f;
        int last = -1, at = -1;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
          const int e = lo + j;
          const float w = e < end ? W(e) : 0.f;
          if (w > 0.f) {
            s += w;
            last = e;
            if (at < 0 && s > rest) at = e;
          }
        }
        if (last >= 0) pos = at >= 0 ? at : last;  // a rounding short of the group's sum: its last edge with a weight
      }
    } else {
      for (unsigned m = __ballot_sync(FULL_MASK, group >= 0); m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        float left = __shfl_sync(FULL_MASK, rest, src);
        const int64_t lo = static_cast<int64_t>(__shfl_sync(FULL_MASK, group, src)) * (static_cast<int64_t>(32) << shift);
        const int64_t end = lo + (static_cast<int64_t>(32) << shift) < deg ? lo + (static_cast<int64_t>(32) << shift) : deg;
        int64_t at = -1;
        for (int64_t b = lo; b < end && at < 0; b += 32) at = edge_of_32(W, b, deg, &left, false, l);
        // a rounding short of the group's sum: its last edge with a weight
        for (int64_t b = (end - 1 - lo) / 32 * 32 + lo; b >= lo && at < 0; b -= 32) at = edge_of_32(W, b, deg, &left, true, l);
        if (l == src && at >= 0) pos = at;
      }
    }
    if (t < k) emit(o, t, seed, rb, pos);
  };

  // ---- phase 1: one seed per warp ----
  const int64_t i0 = static_cast<int64_t>(blockIdx.x) * WEIGHTED_WARPS;
  if (i0 + warp < n) {
    const SeedPlan sp = seed_plan(plan_rb, plan_deg, local_off, tile_off, i0 + warp, true);
    const int64_t seed = row_is_position ? i0 + warp : static_cast<int64_t>(seeds[i0 + warp]);
    if (marks.seeds && l == 0) mark_id(marks, seed, static_cast<uint32_t>(i0 + warp), status);
    if (sp.deg > 0 && sp.rb + sp.deg > probs.total) {
      if (l == 0) raise_status(status, DGS_ERR_RANGE);
    } else if (sp.deg > HUB_DEG) {
      if (l == 0) {
        s_long[atomicAdd(&s_nlong, 1)] = warp;
        s_seed.rb[warp] = sp.rb;
        s_seed.deg[warp] = sp.deg;
        s_seed.o[warp] = sp.o;
        s_seed.seed[warp] = seed;
      }
    } else if (sp.deg > 0) {
      const RowWeights W = row_weights(probs, sp.rb, sp.deg);
      sum_groups(W, sp.deg, 0, 0, 1, l, s_row[warp].sum);
      __syncwarp();
      const float total = prefix_groups(s_row[warp], l);
      __syncwarp();
      for (int64_t t0 = 0; t0 < k; t0 += 32) draws(s_row[warp], total, W, sp.deg, i0 + warp, seed, sp.rb, sp.o, t0);
    }
  }

  // ---- phase 2: rows above HUB_DEG ----
  __syncthreads();
  const int nlong = s_nlong;
  for (int h = 0; h < nlong; ++h) {
    RowGroups& g = s_row[s_long[h]];  // the seed's own: phase 1 left it at 0
    const int64_t deg = s_seed.deg[s_long[h]];
    sum_groups(row_weights(probs, s_seed.rb[s_long[h]], deg), deg, group_shift(deg), warp, WEIGHTED_WARPS, l, g.sum);
  }
  __syncthreads();
  if (warp < nlong) {
    const int src = s_long[warp];
    const float total = prefix_groups(s_row[src], l);
    __syncwarp();
    const RowWeights W = row_weights(probs, s_seed.rb[src], s_seed.deg[src]);
    for (int64_t t0 = 0; t0 < k; t0 += 32)
      draws(s_row[src], total, W, s_seed.deg[src], i0 + src, s_seed.seed[src], s_seed.rb[src], s_seed.o[src], t0);
  }
}

__global__ void copy_total_kernel(const int64_t* total, int64_t* nnz) { *nnz = *total; }
__global__ void zero_total_kernel(int64_t* nnz) { *nnz = 0; }

int check_sample_args(const char* who, const void* seeds, int64_t n, int64_t k, const void* plan) {
  DGS_REQUIRE(n >= 0 && k >= 0, DGS_ERR_INVALID, "%s: n=%lld k=%lld", who, (long long)n, (long long)k);
  DGS_REQUIRE(n == 0 || (seeds != nullptr && plan != nullptr), DGS_ERR_INVALID, "%s: null buffer", who);
  DGS_REQUIRE(n / (SAMPLE_BLOCK / 32) < 0x7fffffffLL, DGS_ERR_UNSUPPORTED, "%s: too many seeds", who);
  return DGS_OK;
}

template <typename IdT>
int plan_typed(const dgs_chunk_desc& indptr, const void* seeds, Count n, int64_t k, bool replace,
               const PlanView& pv, int64_t* nnz, const InitWords& init, const FillJob& fill, int32_t* status, cudaStream_t s) {
  if (n.bound <= SMALL_PLAN) {
    DGS_CUDA_TRY(launch_chained(SITE_PLAN, sample_small_plan_kernel<IdT>, 1u + fill.ctas, SMALL_PLAN_BLOCK, s, indptr,
                                static_cast<const IdT*>(seeds), static_cast<int>(n.bound), k, replace, pv, nnz, init, fill,
                                status));
    return DGS_OK;
  }
  if (n.bound <= CLUSTER_PLAN && init.n0 == nullptr && fill.ctas == 0) {
    DGS_CUDA_TRY(launch_chained(SITE_PLAN, sample_cluster_plan_kernel<IdT>, CLUSTER_PLAN_CTAS, CLUSTER_PLAN_BLOCK, s, indptr,
                                static_cast<const IdT*>(seeds), static_cast<int>(n.bound), k, replace, pv, nnz, status));
    return DGS_OK;
  }
  DGS_CUDA_TRY(launch_chained(SITE_INIT, init_kernel, 1u + fill.ctas, fill.ctas > 0 ? 1024u : 32u, s, init, pv.ticket, fill));
  DGS_CUDA_TRY(launch_chained(SITE_PLAN, sample_plan_kernel<IdT>, static_cast<unsigned>(pv.ntiles), SAMPLE_BLOCK, s, indptr,
                              static_cast<const IdT*>(seeds), n, k, replace, pv.row_begin, pv.deg, pv.local_off,
                              pv.tile_off, pv.total, pv.ticket, nnz, status));
  return DGS_OK;
}

template <typename IdT>
int uniform_typed(const dgs_chunk_desc& indices, const void* seeds, Count n, int64_t k, bool replace,
                  const PlanView& pv, RngKey key, void* coo_row, void* coo_col,
                  int64_t cap, int64_t* pos, bool rowpos, SideJobs jobs, const IdMarks& marks, int32_t* status, cudaStream_t s) {
#define DGS_LAUNCH_U(G)                                                                                       \
  do {                                                                                                        \
    jobs.main_ctas = static_cast<unsigned>((n.bound + SAMPLE_BLOCK / G - 1) / (SAMPLE_BLOCK / G));            \
    DGS_CUDA_TRY(launch_chained(SITE_SAMPLE, sample_uniform_kernel<IdT, G>,                                   \
                                jobs.main_ctas + jobs.clear.ctas + jobs.lookup.ctas, SAMPLE_BLOCK, s,         \
                                indices, static_cast<const IdT*>(seeds), n, k, replace, pv.row_begin, pv.deg, \
                                pv.local_off, pv.tile_off, key, static_cast<IdT*>(coo_row),                   \
                                static_cast<IdT*>(coo_col), cap, pos, rowpos, jobs, marks, status));          \
  } while (0)
#define DGS_LAUNCH_LEAN(G, MARK)                                                                              \
  do {                                                                                                        \
    jobs.main_ctas = static_cast<unsigned>((n.bound + SAMPLE_BLOCK / G - 1) / (SAMPLE_BLOCK / G));            \
    DGS_CUDA_TRY(launch_chained(SITE_SAMPLE, (sample_uniform_lean_kernel<IdT, G, MARK>),                       \
                                jobs.main_ctas + jobs.clear.ctas + jobs.lookup.ctas, SAMPLE_BLOCK, s,         \
                                static_cast<const IdT*>(indices.dev[0]), indices.total,                       \
                                static_cast<const IdT*>(seeds), n, static_cast<uint32_t>(k), pv.row_begin,    \
                                pv.deg, pv.local_off, pv.tile_off, key, static_cast<IdT*>(coo_row),           \
                                static_cast<IdT*>(coo_col), static_cast<uint32_t>(cap), rowpos, jobs, marks, status)); \
  } while (0)
  // one storage region, and everything that is counted fits 32 bits: rows (they lie in indices), seeds, and the offsets of
  // all outputs that a plan may hold, also of those past the capacity
  const bool lean = !replace && k <= 32 && pos == nullptr && indices.num_parts == 1 && indices.threshold == indices.total &&
                    indices.total <= 0xFFFFFFFFll && cap >= 0 && cap < (1ll << 31) && n.bound < (1ll << 31) &&
                    n.bound * k < (1ll << 32) - 64;
  if (lean && marks.first != nullptr) {
    if (k <= 4) DGS_LAUNCH_LEAN(4, true);
    else if (k <= 8) DGS_LAUNCH_LEAN(8, true);
    else if (k <= 16) DGS_LAUNCH_LEAN(16, true);
    else DGS_LAUNCH_LEAN(32, true);
    return DGS_OK;
  }
  if (lean) {
    if (k <= 4) DGS_LAUNCH_LEAN(4, false);
    else if (k <= 8) DGS_LAUNCH_LEAN(8, false);
    else if (k <= 16) DGS_LAUNCH_LEAN(16, false);
    else DGS_LAUNCH_LEAN(32, false);
    return DGS_OK;
  }
  if (k <= 4) DGS_LAUNCH_U(4);
  else if (k <= 8) DGS_LAUNCH_U(8);
  else if (k <= 16) DGS_LAUNCH_U(16);
  else DGS_LAUNCH_U(32);
#undef DGS_LAUNCH_LEAN
#undef DGS_LAUNCH_U
  return DGS_OK;
}

template <typename IdT>
int weighted_typed(const dgs_chunk_desc& indices, const dgs_chunk_desc& probs, const void* seeds, Count n,
                   int64_t k, bool replace, const PlanView& pv, RngKey key,
                   void* coo_row, void* coo_col, int64_t cap, int64_t* pos, bool rowpos, SideJobs jobs, const IdMarks& marks,
                   int32_t* status, cudaStream_t s) {
  jobs.main_ctas = static_cast<unsigned>((n.bound + WEIGHTED_WARPS - 1) / WEIGHTED_WARPS);
  auto kernel = replace ? sample_weighted_replace_kernel<IdT> : sample_weighted_kernel<IdT>;
  DGS_CUDA_TRY(launch_chained(SITE_SAMPLE, kernel, jobs.main_ctas + jobs.clear.ctas + jobs.lookup.ctas, SAMPLE_BLOCK, s,
                              indices, probs, static_cast<const IdT*>(seeds), n, k, pv.row_begin, pv.deg, pv.local_off,
                              pv.tile_off, key, static_cast<IdT*>(coo_row), static_cast<IdT*>(coo_col), cap,
                              pos, rowpos, jobs, marks, status));
  return DGS_OK;
}

}  // namespace

int64_t* sample_plan_total(void* plan, int64_t n_bound) { return plan_view(plan, n_bound).total; }

uint64_t sample_rng_key(uint64_t rng_seed, uint64_t rng_offset) {
  return fold_rng_key(rng_seed, rng_offset);
}

int launch_sample_plan(const dgs_chunk_desc& indptr, const void* seeds, bool ids64, int64_t n, int64_t k,
                       bool replace, void* plan, int64_t* nnz_out, const InitWords& init, const FillJob& fill, int32_t* status,
                       cudaStream_t s) {
  const PlanView pv = plan_view(plan, n);
  const Count nc = exact_count(n);
  return ids64 ? plan_typed<int64_t>(indptr, seeds, nc, k, replace, pv, nnz_out, init, fill, status, s)
               : plan_typed<int32_t>(indptr, seeds, nc, k, replace, pv, nnz_out, init, fill, status, s);
}

NextPlan make_next_plan(const dgs_chunk_desc& indptr, int64_t n_bound, int64_t k, bool replace, void* plan) {
  const PlanView pv = plan_view(plan, n_bound);
  return NextPlan{indptr, k, replace, pv.row_begin, pv.deg, pv.local_off, pv.total};
}

int launch_sample_uniform(const dgs_chunk_desc& indices, const void* seeds, bool ids64, Count n, int64_t k,
                          bool replace, void* plan, bool whole_offsets, RngKey key, void* coo_row,
                          void* coo_col, int64_t out_capacity, int64_t* picked_pos, bool row_is_position,
                          const SideJobs& jobs, const IdMarks& marks, int32_t* status, cudaStream_t s) {
  static_assert(SAMPLE_BLOCK == RL_BLOCK, "the jobs riding on the sampling launch assume its CTA size");
  PlanView pv = plan_view(plan, n.bound);
  if (whole_offsets) pv.tile_off = nullptr;
  return ids64 ? uniform_typed<int64_t>(indices, seeds, n, k, replace, pv, key, coo_row, coo_col,
                                        out_capacity, picked_pos, row_is_position, jobs, marks, status, s)
               : uniform_typed<int32_t>(indices, seeds, n, k, replace, pv, key, coo_row, coo_col,
                                        out_capacity, picked_pos, row_is_position, jobs, marks, status, s);
}

int launch_sample_weighted(const dgs_chunk_desc& indices, const dgs_chunk_desc& probs, const void* seeds,
                           bool ids64, Count n, int64_t k, bool replace, void* plan, bool whole_offsets,
                           RngKey key, void* coo_row, void* coo_col, int64_t out_capacity,
                           int64_t* picked_pos, bool row_is_position, const SideJobs& jobs, const IdMarks& marks,
                           int32_t* status, cudaStream_t s) {
  PlanView pv = plan_view(plan, n.bound);
  if (whole_offsets) pv.tile_off = nullptr;
  return ids64 ? weighted_typed<int64_t>(indices, probs, seeds, n, k, replace, pv, key, coo_row, coo_col,
                                         out_capacity, picked_pos, row_is_position, jobs, marks, status, s)
               : weighted_typed<int32_t>(indices, probs, seeds, n, k, replace, pv, key, coo_row, coo_col,
                                         out_capacity, picked_pos, row_is_position, jobs, marks, status, s);
}

}  // namespace dgs

extern "C" size_t dgs_sample_plan_bytes(int64_t n) {
  if (n < 0) n = 0;
  const int64_t ntiles = (n + dgs::SAMPLE_TILE - 1) / dgs::SAMPLE_TILE;
  return static_cast<size_t>(3 * n + ntiles + 2) * sizeof(int64_t);
}

extern "C" int dgs_sample_plan(const dgs_chunk_desc* indptr, const void* seeds, int32_t ids64,
                               int64_t n, int64_t k, int32_t replace, void* plan, int64_t* nnz,
                               int32_t* status, dgs_stream_t stream) {
  using namespace dgs;
  int rc = validate_desc(indptr, "dgs_sample_plan");
  if (rc != DGS_OK) return rc;
  rc = check_sample_args("dgs_sample_plan", seeds, n, k, plan);
  if (rc != DGS_OK) return rc;
  DGS_REQUIRE(indptr->esz == (ids64 ? 8 : 4), DGS_ERR_INVALID,
              "dgs_sample_plan: indptr element size %d does not match the id type", indptr->esz);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (n == 0) {
    if (nnz != nullptr) {
      zero_total_kernel<<<1, 1, 0, s>>>(nnz);
      DGS_LAUNCH_CHECK();
    }
    return DGS_OK;
  }
  return launch_sample_plan(*indptr, seeds, ids64 != 0, n, k, replace != 0, plan, nnz, InitWords{}, FillJob{}, status, s);
}

extern "C" int dgs_sample_uniform(const dgs_chunk_desc* indices, const void* seeds, int32_t ids64,
                                  int64_t n, int64_t k, int32_t replace, const void* plan,
                                  uint64_t rng_seed, uint64_t rng_offset,
                                  void* coo_row, void* coo_col, int64_t out_capacity, int64_t* nnz,
                                  int64_t* picked_pos, int32_t* status, dgs_stream_t stream) {
  using namespace dgs;
  int rc = validate_desc(indices, "dgs_sample_uniform");
  if (rc != DGS_OK) return rc;
  rc = check_sample_args("dgs_sample_uniform", seeds, n, k, plan);
  if (rc != DGS_OK) return rc;
  DGS_REQUIRE(indices->esz == (ids64 ? 8 : 4), DGS_ERR_INVALID,
              "dgs_sample_uniform: indices element size %d does not match the id type", indices->esz);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (n == 0 || k == 0) {
    if (nnz != nullptr) {
      zero_total_kernel<<<1, 1, 0, s>>>(nnz);
      DGS_LAUNCH_CHECK();
    }
    return DGS_OK;
  }
  DGS_REQUIRE(out_capacity == 0 || (coo_row != nullptr && coo_col != nullptr), DGS_ERR_INVALID,
              "dgs_sample_uniform: null output");
  rc = launch_sample_uniform(*indices, seeds, ids64 != 0, exact_count(n), k, replace != 0, const_cast<void*>(plan),
                             false, host_key(sample_rng_key(rng_seed, rng_offset)), coo_row, coo_col, out_capacity,
                             picked_pos, false, SideJobs{}, IdMarks{}, status, s);
  if (rc != DGS_OK) return rc;
  if (nnz != nullptr) {
    copy_total_kernel<<<1, 1, 0, s>>>(sample_plan_total(const_cast<void*>(plan), n), nnz);
    DGS_LAUNCH_CHECK();
  }
  return DGS_OK;
}

extern "C" int dgs_sample_weighted(const dgs_chunk_desc* indices, const dgs_chunk_desc* probs,
                                   const void* seeds, int32_t ids64, int64_t n, int64_t k,
                                   int32_t replace, const void* plan,
                                   uint64_t rng_seed, uint64_t rng_offset, void* coo_row, void* coo_col,
                                   int64_t out_capacity, int64_t* nnz, int64_t* picked_pos,
                                   int32_t* status, dgs_stream_t stream) {
  using namespace dgs;
  int rc = validate_desc(indices, "dgs_sample_weighted");
  if (rc != DGS_OK) return rc;
  rc = validate_desc(probs, "dgs_sample_weighted(probs)");
  if (rc != DGS_OK) return rc;
  rc = check_sample_args("dgs_sample_weighted", seeds, n, k, plan);
  if (rc != DGS_OK) return rc;
  DGS_REQUIRE(indices->esz == (ids64 ? 8 : 4), DGS_ERR_INVALID,
              "dgs_sample_weighted: indices element size %d does not match the id type", indices->esz);
  DGS_REQUIRE(probs->esz == 4, DGS_ERR_UNSUPPORTED, "dgs_sample_weighted: weights must be fp32");
  // the reference asserts the same bound on the device (rowwise_sampling_probs.cu:65)
  DGS_REQUIRE(replace || k <= 32, DGS_ERR_UNSUPPORTED,
              "dgs_sample_weighted: k=%lld > 32 without replacement is not supported", (long long)k);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (n == 0 || k == 0) {
    if (nnz != nullptr) {
      zero_total_kernel<<<1, 1, 0, s>>>(nnz);
      DGS_LAUNCH_CHECK();
    }
    return DGS_OK;
  }
  DGS_REQUIRE(out_capacity == 0 || (coo_row != nullptr && coo_col != nullptr), DGS_ERR_INVALID,
              "dgs_sample_weighted: null output");
  rc = launch_sample_weighted(*indices, *probs, seeds, ids64 != 0, exact_count(n), k, replace != 0,
                              const_cast<void*>(plan), false, host_key(sample_rng_key(rng_seed, rng_offset)), coo_row,
                              coo_col, out_capacity, picked_pos, false, SideJobs{}, IdMarks{}, status, s);
  if (rc != DGS_OK) return rc;
  if (nnz != nullptr) {
    copy_total_kernel<<<1, 1, 0, s>>>(sample_plan_total(const_cast<void*>(plan), n), nnz);
    DGS_LAUNCH_CHECK();
  }
  return DGS_OK;
}
