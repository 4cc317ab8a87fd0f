// What the forward's tile kernels for tabular input (ht_forest_tiled.cu) and for inner positions (ht_forest_tiled_inner.cu) share.
#pragma once

#include "ht_forest_tiled.cuh"
#include "ht_tile_common.cuh"
#include "ht_tma.cuh"

namespace ht {
namespace tile {

struct TilePlan {
  bool weights;    // the records carry the leaf weights (one output per leaf)
  int S;           // samples per tile
  int G;           // trees per parameter group
  int per_warp;    // trees a warp walks at once: G / slots
  int ord_bytes;   // 1 or 2
  RecordLayout rec;
  size_t smem;
};

struct TiledArgs {
  CUtensorMap out_map;  // the output [B, T] in boxes of 32 rows x G trees (when tma_store is set)
  const float *x;
  const unsigned char *records;
  const float *w;  // leaf weights in global memory, read when there are several outputs per leaf
  float *out;
  uint32_t *status_word;
  int64_t B, T, K;
  int C, S, G, per_warp, M;
  uint32_t record_bytes;
  int width;                 // several outputs per leaf: numbers per load and store
  Divisor by_M, by_pieces;   // ... and what a place in a warp's outputs is divided by
  Divisor by_K;              // inner positions
  int tma_store;  // results of full groups leave through the TMA engine (G is 16 or 32)
  // a forward that saves its traversal for the backward (SAVE kernels): threshold - feature at the deciding
  // vertex, and the packed vertex / leaf key, in the evaluation-record layout
  float *save_margin;
  void *save_where;
};

template <typename Kernel>
inline int launch_one(Kernel kernel, const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream) {
  HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
  kernel<<<grid, kThreads, plan.smem, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

// ht_forest_tiled_inner.cu: the plan for a problem with inner positions (false: not taken), and its launch.
bool make_inner_plan(const ht_forest_problem *p, TilePlan &plan);
// ... of ferns, compiled in a file of their own
int launch_inner_ferns(int depth, const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream);
int launch_inner(int kind, int depth, const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream);

}  // namespace tile
}  // namespace ht
