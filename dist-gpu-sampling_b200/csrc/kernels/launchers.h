// Internal launchers shared between the per-operator entry points (sample.cu,
// relabel.cu) and the multi-hop sequence (blocks.cu).  Not part of the C ABI.
#pragma once
#include "common.cuh"
#include "relabel_device.cuh"

namespace dgs {

// ---- sample.cu ---------------------------------------------------------------
// `plan` is laid out for n seeds.  nnz_out (optional, normally pinned)
// receives the number of sampled edges; the same number stays in the plan at
// sample_plan_total().
// init: words to set before anything behind it runs (n0 == nullptr, rng_src == nullptr: none).
struct InitWords {
  int64_t* n0;
  int64_t n0_value;
  // a recorded sequence takes its random stream from memory: (seed, offset) at rng_src, read on every replay and
  // folded into one Philox key per hop for the sampling kernels
  const uint64_t* rng_src;
  uint64_t* keys;
  int n_keys;
};
int launch_sample_plan(const dgs_chunk_desc& indptr, const void* seeds, bool ids64, int64_t n, int64_t k,
                       bool replace, void* plan, int64_t* nnz_out, const InitWords& init, const FillJob& fill, int32_t* status,
                       cudaStream_t s);
// The plan of a hop whose seeds are being numbered (launch_unique_pair writes it): offsets are those in the whole
// output, so sampling takes whole_offsets = true.  n_edges == nullptr: no plan wanted.
struct NextPlan {
  dgs_chunk_desc indptr;
  int64_t k;
  bool replace;
  int64_t *row_begin, *deg, *off;
  int64_t* n_edges;
};
NextPlan make_next_plan(const dgs_chunk_desc& indptr, int64_t n_bound, int64_t k, bool replace, void* plan);
int64_t* sample_plan_total(void* plan, int64_t n_bound);

// Independent jobs run by extra CTAs of a sampling launch (either may have ctas == 0).
struct SideJobs {
  ClearJob clear;
  LookupJob lookup;
  unsigned main_ctas;  // set by the launcher
};

// marks: record what is emitted in the table of a sequence that numbers its nodes through one word per id.
// row_is_position: write the seed's position in the seed list to coo_row instead
// of the seed id (valid as a relabelled id when the seed list has no duplicates).
int launch_sample_uniform(const dgs_chunk_desc& indices, const void* seeds, bool ids64, Count n, int64_t k,
                          bool replace, void* plan, bool whole_offsets, RngKey key, void* coo_row,
                          void* coo_col, int64_t out_capacity, int64_t* picked_pos, bool row_is_position,
                          const SideJobs& jobs, const IdMarks& marks, int32_t* status, cudaStream_t s);
int launch_sample_weighted(const dgs_chunk_desc& indices, const dgs_chunk_desc& probs, const void* seeds,
                           bool ids64, Count n, int64_t k, bool replace, void* plan, bool whole_offsets,
                           RngKey key, void* coo_row, void* coo_col, int64_t out_capacity,
                           int64_t* picked_pos, bool row_is_position, const SideJobs& jobs, const IdMarks& marks,
                           int32_t* status, cudaStream_t s);
uint64_t sample_rng_key(uint64_t rng_seed, uint64_t rng_offset);

// ---- relabel.cu ----------------------------------------------------------------
// `table` is laid out for key_bound keys (dgs_relabel_table_bytes(key_bound)); `size`
// says how much of it is in use (cleared, probed); every kernel of one table gets
// the same TableSize.
ClearJob make_clear_job(void* table, int64_t key_bound, const TableSize& size);
LookupJob make_lookup_job(void* table, int64_t key_bound, const TableSize& size, void* row, void* col, Count n,
                          Count n_seeds);
int launch_lookup(const LookupJob& job, bool ids64, cudaStream_t s);  // as a launch of its own

// First-occurrence unique of the logical concatenation a[0:na) ++ b[0:nb) whose
// lengths are device words, into a table that has been cleared.  unique_out holds
// unique_capacity ids; a larger result raises DGS_ERR_RANGE in the status word and
// is cut off.  `report` (n may be 0) is carried out by the kernel that knows the number of distinct keys; `plan` is
// filled for the distinct keys as the next hop's seeds.
int launch_unique_pair(bool ids64, const void* a, Count na, const void* b, Count nb, int64_t key_bound,
                       const TableSize& size, void* table, void* unique_out, int64_t unique_capacity,
                       int64_t* n_unique_out, const SizesReport& report, const NextPlan& plan, int32_t* status,
                       cudaStream_t s);
int64_t* unique_total(void* table, int64_t key_bound);

// The same numbering through a table of one word per id (IdMarks), which the sampling launch before it has marked.
// seeds_known: the seeds carry their labels already (they are the unique list of the hop before).
struct DenseNumbering {
  uint32_t* first;
  int64_t ids;
  unsigned int* ticket;       // [4]  cleared with the table
  const uint32_t* beyond;     // IdMarks::beyond
  unsigned long long* tiles;  // [2 * dense_tiles(bounds)], cleared with the table
  int64_t* total;
  bool seeds_known;
};
inline int64_t dense_tiles(int64_t seed_bound, int64_t edge_bound) {
  return (seed_bound + RL_TILE - 1) / RL_TILE + (edge_bound + RL_TILE - 1) / RL_TILE;
}
int launch_dense_number(bool ids64, const DenseNumbering& d, const void* seeds, Count n_seeds, const void* cols, Count n_cols,
                        void* unique_out, int64_t unique_capacity, const SizesReport& report, const NextPlan& plan,
                        int32_t* status, cudaStream_t s);
int launch_dense_lookup(const DenseLookup& job, bool ids64, cudaStream_t s);

}  // namespace dgs
