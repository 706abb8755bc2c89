// What the one-call layer (layer.cu) needs of the single entry points' files, and how their kernels
// are launched.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/anemoi_sm100.h"

namespace layer {

// Attention results written straight to their tokens: `out` [S][H][D] in the caller's type, the slot
// tables of the layout.  Rows of query blocks with empty lists become +0.
struct TokenRows {
  void* out;
  const int32_t* indices;
  const int32_t* counts;
};

int video_rows(const anemoi_sm100_shape& s, const anemoi_sm100_operands& ops, const int32_t* row_offset,
               const int32_t* row_counts, const int32_t* stage_ids, const int32_t* pair_counts,
               const int32_t* pair_ids, int64_t capacity, const int32_t* valid_k, const TokenRows& rows,
               int32_t* status, cudaStream_t st, const int32_t* pair_table);
int prefix_rows(const anemoi_sm100_shape& s, const anemoi_sm100_operands& ops, const int32_t* valid_k,
                const TokenRows& rows, int32_t* status, cudaStream_t st);
// Whether the draft map is formed by the routing kernel, and both in one launch (pair_counts: for pairs).
bool drafts_in_routing(const anemoi_sm100_shape& s);
int draft_and_route(const anemoi_sm100_shape& s, const anemoi_sm100_operands& ops, float maxpool_weight,
                    void* probability, int64_t n16, int64_t n8, int64_t n4, int prefix_phase, int32_t* row_offset,
                    int32_t* row_counts, int32_t* stage_ids, int32_t* pair_counts, int32_t* pair_ids, int64_t capacity,
                    cudaStream_t st);
// What the routing leaves for the choice of the Q64 pairs: bit j of a row = column j is in its list, per phase with a
// budget, [H][phases][R][pair_bit_words(R)] words; `slot`: place of the NVFP4, INT8, FP16 phase among them, or -1.
struct PairBits {
  uint32_t* words;
  int phases, slot[3];
};
// (rows are whole 16-byte pieces: 128 columns)
__host__ __device__ inline int pair_bit_words(int R) { return (R + 127) / 128 * 4; }
int route_bits(const anemoi_sm100_shape& s, const void* probability, int64_t n16, int64_t n8, int64_t n4,
               int prefix_phase, void* scratch, int32_t* row_offset, int32_t* row_counts, const PairBits& bits,
               int64_t capacity, cudaStream_t st);
// The pairs and their lists.  `table` [H][ceil(R/2)][8] in launch order: first block, second (-1: none), where the
// list starts, its stages, and those of each phase.
int match_pairs(const anemoi_sm100_shape& s, const PairBits& bits, int prefix_phase, const int32_t* row_offset,
                const int32_t* row_counts, int32_t* table, int32_t* pair_ids, int64_t capacity, int32_t* status,
                cudaStream_t st);
// Limit of the bounded waits of kernels launched now.
uint64_t wait_limit_ns();
// Whether a Q64 call's pair lists come out of the routing kernel itself.
bool routes_pairs(const anemoi_sm100_shape& s);
// The prefix rows alone, from [H][rows][D] (fp16, or already in the caller's type).
int assemble_prefix(const anemoi_sm100_shape& s, const void* prefix_out, int64_t prefix_rows, int prefix_is_caller,
                    void* out, cudaStream_t st);

// Programmatic dependent launch: a kernel of the chain may be set up, and its first CTAs become
// resident, while the one before it drains; every kernel launched this way begins with
// grid_dependency_wait(), which returns when the kernels before it in the stream are complete and
// their writes visible.  Between the short kernels of a small call that takes the 2-4 us gap of an
// ordinary launch to about 1.
template <typename... P, typename... A>
cudaError_t launch_cluster(void (*kernel)(P...), dim3 grid, dim3 cluster, dim3 block, size_t smem, cudaStream_t st,
                           A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster.x;
  attr[1].val.clusterDim.y = cluster.y;
  attr[1].val.clusterDim.z = cluster.z;
  cfg.attrs = attr;
  cfg.numAttrs = cluster.x * cluster.y * cluster.z > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}
template <typename... P, typename... A>
cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  return launch_cluster(kernel, grid, dim3(1), block, smem, st, std::forward<A>(args)...);
}

__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel of the chain be set up as soon as every CTA of this one has started.
__device__ __forceinline__ void grid_dependency_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace layer
