// Exclusive scan of per-tile sums: the middle step of every "count per tile ->
// scan tile sums -> write with known offsets" sequence in this library (sample
// offsets, first-occurrence numbering, split-index classes).  Replaces the
// reference's cub::DeviceScan wrapper (src/cuda/cub_function.h:10-22) plus its
// blocking read-back of the last element (src/cuda/rowwise_sampling.cu:147,
// src/cuda/tensor_reindex.cu:129): the totals go straight to a caller-supplied
// (normally pinned) location, so the host reads them whenever it next
// synchronises instead of stalling mid-sequence.
#pragma once
#include "common.cuh"

namespace dgs {

constexpr int TILE_SCAN_BLOCK = 1024;

// sums: [ntiles][C] tile-major.  In place: sums[t][c] becomes the exclusive
// prefix over tiles; totals_dev[c] (device scratch, optional) and
// totals_out[c] (optional) receive the grand totals.  One CTA.
template <int C>
__global__ void __launch_bounds__(TILE_SCAN_BLOCK)
tile_scan_kernel(int64_t* __restrict__ sums, const int64_t ntiles, int64_t* __restrict__ totals_dev,
                 int64_t* __restrict__ totals_out) {
  __shared__ int64_t smem[TILE_SCAN_BLOCK / 32 + 1];
  int64_t carry[C];
#pragma unroll
  for (int c = 0; c < C; ++c) carry[c] = 0;
  for (int64_t t0 = 0; t0 < ntiles; t0 += TILE_SCAN_BLOCK) {
    const int64_t t = t0 + threadIdx.x;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int64_t v = (t < ntiles) ? sums[t * C + c] : 0;
      int64_t total;
      const int64_t ex = block_exclusive_scan<int64_t, TILE_SCAN_BLOCK>(v, smem, &total);
      if (t < ntiles) sums[t * C + c] = carry[c] + ex;
      carry[c] += total;
    }
  }
  if (threadIdx.x == 0) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (totals_dev != nullptr) totals_dev[c] = carry[c];
      if (totals_out != nullptr) totals_out[c] = carry[c];
    }
  }
}


// The same scan without a second launch: every CTA of a counting kernel calls
// this after computing its tile sum.  The CTA that draws the last ticket (an
// atomic counter that must be zero at launch; nobody waits on anybody) scans
// all tile sums in place and publishes the total.  `smem` needs BLOCK/32 + 1
// entries; must be called by all threads of the CTA.  The tiles are the CTAs of the launch.
template <int BLOCK>
__device__ __forceinline__ void publish_and_scan_tiles(int64_t my_tile_sum, int64_t* tile_sums,
                                                       unsigned int* ticket, int64_t* total_dev,
                                                       int64_t* total_out, int64_t* smem) {
  __shared__ bool s_last;
  if (threadIdx.x == 0) {
    tile_sums[blockIdx.x] = my_tile_sum;
    __threadfence();
    s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // Every thread takes a contiguous run of `per` tiles: all loads of the CTA are issued together (one round
  // trip to L2 whatever the number of tiles, instead of one per BLOCK tiles), one block scan over the threads'
  // sums gives each run its offset, and a second walk over the run (now in L1/L2) writes the prefixes.  This
  // CTA works alone at the end of its kernel, so every microsecond here is latency of the whole sequence.
  const int64_t ntiles = gridDim.x;
  const int64_t per = (ntiles + BLOCK - 1) / BLOCK;
  const int64_t lo = static_cast<int64_t>(threadIdx.x) * per;
  const int64_t hi = lo + per < ntiles ? lo + per : ntiles;
  int64_t mine = 0;
  for (int64_t t = lo; t < hi; ++t) mine += __ldcg(tile_sums + t);
  int64_t carry;
  int64_t run = block_exclusive_scan<int64_t, BLOCK>(mine, smem, &carry);
  for (int64_t t = lo; t < hi; ++t) {
    const int64_t v = __ldcg(tile_sums + t);
    tile_sums[t] = run;
    run += v;
  }
  if (threadIdx.x == 0) {
    if (total_dev != nullptr) *total_dev = carry;
    *ticket = 0;
    if (total_out != nullptr) {
      *total_out = carry;
      __threadfence_system();
    }
  }
}

// ---- offsets in one pass -------------------------------------------------------
// A kernel that counts per tile and then writes with known offsets can do both in one launch: every tile publishes
// its sum, adds up what the tiles before it have published, and publishes the running sum for those behind it
// (Merrill and Garland, "Single-pass parallel prefix scan with decoupled look-back", 2016).  Here a tile looks back
// over BLOCK predecessors at a time, one per thread: with the few hundred to few thousand tiles of a mini-batch, all
// of them in flight at once, hardly any running sum exists yet when a tile looks, and a walk of 32 at a time is a
// chain of as many L2 round trips as there are tiles / 32.
// A tile word is 2 bits of state and a 62-bit sum; all ones (the cleared table) is "nothing yet".  Tiles are numbered
// by an atomic ticket, so every tile that one waits for has started.  Waits are bounded: a tile that gives up raises
// DGS_ERR_CUDA and goes on with what it has.
constexpr unsigned long long TILE_SUM = 1ull << 62;      // the tile's own sum
constexpr unsigned long long TILE_RUNNING = 2ull << 62;  // sum of this tile and all before it
constexpr unsigned long long TILE_STATE = 3ull << 62;    // nothing yet
constexpr uint32_t TILE_WAIT_LIMIT = 1u << 22;

template <int BLOCK>
struct TileScanShared {
  int64_t sum[BLOCK / 32];
  int done[BLOCK / 32];
};

__device__ __forceinline__ unsigned long long load_tile_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_tile_word(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Sum of all tiles before `tile`; every thread of the CTA calls this with the tile's own sum and gets the result.
template <int BLOCK>
__device__ __forceinline__ int64_t sum_of_tiles_before(int64_t tile, int64_t own, unsigned long long* words,
                                                       TileScanShared<BLOCK>& sm, int32_t* status) {
  if (threadIdx.x == 0)
    store_tile_word(words + tile, (tile == 0 ? TILE_RUNNING : TILE_SUM) | static_cast<unsigned long long>(own));
  if (tile == 0) return 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t before = 0;
  for (int64_t end = tile; end > 0; end -= BLOCK) {
    const int64_t at = end - 1 - threadIdx.x;  // thread 0: the nearest
    unsigned long long w = TILE_RUNNING;       // before the first tile: nothing to add, nothing further back
    if (at >= 0) {
      w = load_tile_word(words + at);
      for (uint32_t polls = 0; (w & TILE_STATE) == TILE_STATE; ++polls) {
        if (polls == TILE_WAIT_LIMIT) {
          raise_status(status, DGS_ERR_CUDA);
          w = TILE_RUNNING;
          break;
        }
        w = load_tile_word(words + at);
      }
    }
    // of a warp's 32 tiles, the ones up to the nearest running sum count
    const unsigned running = __ballot_sync(FULL_MASK, (w & TILE_STATE) == TILE_RUNNING);
    const int last = running ? __ffs(running) - 1 : 31;
    int64_t v = lane <= last ? static_cast<int64_t>(w & ~TILE_STATE) : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL_MASK, v, o);
    if (lane == 0) {
      sm.sum[warp] = v;
      sm.done[warp] = running != 0u;
    }
    __syncthreads();
    bool done = false;
#pragma unroll
    for (int q = 0; q < BLOCK / 32; ++q) {
      if (done) break;
      before += sm.sum[q];
      done = sm.done[q] != 0;
    }
    __syncthreads();  // the shared words are written again
    if (done) break;
  }
  if (threadIdx.x == 0) store_tile_word(words + tile, TILE_RUNNING | static_cast<unsigned long long>(before + own));
  return before;
}

}  // namespace dgs
