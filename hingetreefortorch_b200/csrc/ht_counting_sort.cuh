// Pieces of the kernels that sort a slice of evaluations by counting in shared memory, so that what belongs to one leaf or one
// vertex lies together and is summed before it meets memory.
#pragma once

#include "ht_common.cuh"

namespace ht {

// Turns counts[0 .. 4 * quads) into the sums of what is before each.  All threads of the block; partial: a number per warp.
template <int THREADS>
__device__ __forceinline__ void exclusive_sums(uint4 *counts, int quads, uint32_t *partial) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (quads + THREADS - 1) / THREADS;  // 16 bytes each: one up to 1024 numbers
  const int first = min(tid * per, quads), last = min(first + per, quads);
  uint32_t mine = 0;
  for (int b = first; b < last; ++b) {
    const uint4 c = counts[b];
    mine += c.x + c.y + c.z + c.w;
  }
  uint32_t sum = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t below = __shfl_up_sync(0xffffffffu, sum, d);
    if (lane >= d) sum += below;
  }
  if (lane == 31) partial[warp] = sum;
  __syncthreads();
  uint32_t base = sum - mine;
#pragma unroll
  for (int k = 0; k < THREADS / 32 - 1; ++k) base += k < warp ? partial[k] : 0u;
  for (int b = first; b < last; ++b) {
    uint4 c = counts[b], before;
    before.x = base;
    before.y = before.x + c.x;
    before.z = before.y + c.y;
    before.w = before.z + c.z;
    base = before.w + c.w;
    counts[b] = before;
  }
  __syncthreads();
}

// A warp's numbers, neighbours with the same key summed: true for the first lane of a run, which is left with the run's sums.
// All 32 lanes; equal keys are neighbours.
template <typename Real, int NUMBERS>
__device__ __forceinline__ bool sums_of_runs(uint32_t key, Real (&sum)[NUMBERS], int lane) {
  const uint32_t before = __shfl_up_sync(0xffffffffu, key, 1);
  const bool leads = lane == 0 || before != key;
  const uint32_t leaders = __ballot_sync(0xffffffffu, leads) & ~((2u << lane) - 1u);  // of the runs above this lane's
  const int last = (leaders != 0u ? __ffs((int)leaders) - 1 : 32) - lane;             // lanes to the end of the run
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
    for (int u = 0; u < NUMBERS; ++u) {
      const Real other = __shfl_down_sync(0xffffffffu, sum[u], d);
      if (d < last) sum[u] += other;
    }
  }
  return leads;
}

}  // namespace ht
