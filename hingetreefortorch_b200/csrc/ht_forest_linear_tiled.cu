// Forest with its linear layer on tabular data: forward and backward over the paths of all evaluations.
//
// The paths (margin; deciding vertex and leaf) lie [block of 256 samples][tree][256]: a thread that stays with its sample
// reads them in runs, whatever order it takes the trees in.
#include "ht_forest_linear_tiled.cuh"
#include "ht_forest_multi.cuh"
#include "ht_forest_rows.cuh"
#include "ht_forest_tiled.cuh"
#include "ht_tile_common.cuh"

#include <algorithm>

namespace ht {

namespace {

constexpr int kForwardBlock = 64;    // a divisor of the record block; small, so that few samples still fill the machine
constexpr int kBackwardBlock = 256;  // the record block
constexpr int kMostOutputs = 16;

struct LinearArgs {
  const float *w, *lin, *bias, *g;
  float *out, *glin;
  EvalRecords r;
  int64_t B, T, L, O;
  int write_terms;
};

// Linear weights as [tree][OP], outputs past the last zero: a tree's come in 16-byte broadcasts.
template <int OP>
__device__ __forceinline__ void stage_linear(const LinearArgs &a, float *lt) {
  for (int e = threadIdx.x; e < (int)a.T * OP; e += blockDim.x) {
    const int j = e / OP, o = e - j * OP;
    lt[e] = o < a.O ? __ldg(a.lin + o * a.T + j) : 0.0f;
  }
}

// Thread per sample: out[i, o] = bias[o] + sum over j ascending of (|margin| * lin[o, j]) * w[j, leaf], the reference's order
// and roundings.  A thread per output read every path again for each of them, 32 rows at a time: 262144 samples, 100 trees,
// 10 outputs 321 us there, 97 here (eight trees' paths under way: 110 with four).
template <int OP, typename WhereT>
__global__ void __launch_bounds__(kForwardBlock) linear_rows_forward_kernel(const __grid_constant__ LinearArgs a) {
  extern __shared__ __align__(16) float lt[];
  __shared__ float results[kForwardBlock * OP];
  stage_linear<OP>(a, lt);
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * kForwardBlock + threadIdx.x;
  const int64_t at0 = record_index(min(i, a.B - 1), 0, a.T);
  float acc[OP];
#pragma unroll
  for (int o = 0; o < OP; ++o) acc[o] = o < a.O ? __ldg(a.bias + o) : 0.0f;
  constexpr int kAhead = 8;
  for (int64_t j0 = 0; j0 < a.T; j0 += kAhead) {
    float size[kAhead], weight[kAhead];
    uint32_t key[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int64_t at = at0 + min(j0 + u, a.T - 1) * kRecordBlock;
      size[u] = fabsf(__ldg(a.r.dx + at));
      key[u] = load_where<WhereT>(a.r.where, at) >> 16;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) weight[u] = __ldg(a.w + min(j0 + u, a.T - 1) * a.L + key[u]);
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (j0 + u < a.T) {
#pragma unroll
        for (int o = 0; o < OP; o += 4) {
          const float4 l = *reinterpret_cast<const float4 *>(lt + (j0 + u) * OP + o);
          acc[o + 0] = add_rn(acc[o + 0], mul_rn(mul_rn(size[u], l.x), weight[u]));
          acc[o + 1] = add_rn(acc[o + 1], mul_rn(mul_rn(size[u], l.y), weight[u]));
          acc[o + 2] = add_rn(acc[o + 2], mul_rn(mul_rn(size[u], l.z), weight[u]));
          acc[o + 3] = add_rn(acc[o + 3], mul_rn(mul_rn(size[u], l.w), weight[u]));
        }
      }
  }
  // the block's results are one run of the output
#pragma unroll
  for (int o = 0; o < OP; ++o)
    if (o < a.O) results[threadIdx.x * a.O + o] = acc[o];
  __syncthreads();
  const int64_t first = (int64_t)blockIdx.x * kForwardBlock * a.O;
  const int count = (int)(min((int64_t)kForwardBlock, a.B - (int64_t)blockIdx.x * kForwardBlock) * a.O);
  for (int e = threadIdx.x; e < count; e += kForwardBlock) a.out[first + e] = results[e];
}

// CTA = a record block of 256 samples at a time (several, one after another), with its upstream gradients [output][sample]
// in shared memory; a warp takes a tree, its lanes samples.  Per evaluation: what arrives at the tree's output,
// through = sum over o of lin[o, j] * g[o]; from it the two terms of the records, which the forest's reductions turn into the
// other gradients; and |margin| * w * g[o] for the linear weights' gradient, summed in registers over the block's samples
// and in shared memory over the blocks.
// Bound by reading and writing the records (14 bytes per evaluation).  262144 samples, 100 trees, 10 outputs: 131 us.
template <int OP, typename WhereT>
__global__ void __launch_bounds__(kBackwardBlock) linear_rows_backward_kernel(const __grid_constant__ LinearArgs a) {
  extern __shared__ __align__(16) float smem[];
  constexpr int kPitch = kBackwardBlock + 1;
  float *lt = smem;                    // [T][OP]
  float *sums = lt + a.T * OP;         // [T][OP]: of the linear weights' gradient
  float *gt = sums + a.T * OP;         // [OP][kPitch]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  stage_linear<OP>(a, lt);
  for (int e = tid; e < (int)a.T * OP; e += kBackwardBlock) sums[e] = 0.0f;
  for (int e = tid; e < OP * kPitch; e += kBackwardBlock) gt[e] = 0.0f;
  const int64_t blocks = (a.B + kBackwardBlock - 1) / kBackwardBlock;
  const int share = ((int)a.T + (int)gridDim.y - 1) / (int)gridDim.y;  // few record blocks: their trees are split over gridDim.y
  const int tree0 = (int)blockIdx.y * share, tree_end = min(tree0 + share, (int)a.T);
  const int O = (int)a.O;
  for (int64_t block = blockIdx.x; block < blocks; block += gridDim.x) {
    __syncthreads();
    const int64_t i0 = block * kBackwardBlock;
    const int here = (int)min((int64_t)kBackwardBlock, a.B - i0);
    for (int e = tid; e < kBackwardBlock * O; e += kBackwardBlock) {
      const int s = e / O, o = e - s * O;
      gt[o * kPitch + s] = s < here ? __ldg(a.g + i0 * O + e) : 0.0f;
    }
    __syncthreads();
    for (int j = tree0 + warp; j < tree_end; j += kBackwardBlock / 32) {
      const int64_t at0 = (block * a.T + j) * kRecordBlock + lane;
      const float *leaves = a.w + j * a.L;
      float l[OP], gl[OP];
#pragma unroll
      for (int o = 0; o < OP; ++o) {
        l[o] = lt[j * OP + o];
        gl[o] = 0.0f;
      }
      constexpr int kAhead = 8;
      for (int c0 = 0; c0 < here; c0 += 32 * kAhead) {
        float nm[kAhead], weight[kAhead];
        uint32_t where[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          nm[u] = stream_f32(a.r.dx + at0 + c0 + 32 * u);
          where[u] = stream_raw_where<WhereT>(a.r.where, at0 + c0 + 32 * u);
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u)  // (positions past the last sample hold anything: they are masked, their leaf is in range)
          weight[u] = __ldg(leaves + min((uint32_t)(a.L - 1), unpack_where<WhereT>(where[u]) >> 16));
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const int s = c0 + 32 * u + lane;
          const bool on = s < here;
          const float size = fabsf(nm[u]), f = on ? size * weight[u] : 0.0f;
          float through = 0.0f;
#pragma unroll
          for (int o = 0; o < OP; ++o) {
            const float go = gt[o * kPitch + (on ? s : lane)];
            through += l[o] * go;
            gl[o] += f * go;
          }
          if (a.write_terms && on) {
            __stcs(a.r.dx + at0 + c0 + 32 * u, tile::signed_term(nm[u], weight[u] * through));
            __stcs(a.r.dw + at0 + c0 + 32 * u, size * through);
          }
        }
      }
      if (a.glin != nullptr) {
        // every exchange halves the number of sums that a lane holds: lane o ends up with output o's (OP <= 16)
#pragma unroll
        for (int o = 0; o < OP; ++o) gl[o] += __shfl_xor_sync(0xffffffffu, gl[o], 16);
        float mine = 0.0f;
#pragma unroll
        for (int o = 0; o < OP; ++o) {
          float v = gl[o];
          v += __shfl_xor_sync(0xffffffffu, v, 8);
          v += __shfl_xor_sync(0xffffffffu, v, 4);
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          mine = lane == o ? v : mine;
        }
        if (lane < O) sums[j * OP + lane] += mine;
      }
    }
  }
  if (a.glin == nullptr) return;
  __syncthreads();
  for (int e = tid; e < (int)a.T * OP; e += kBackwardBlock) {
    const int j = e / OP, o = e - j * OP;
    if (o < O && sums[e] != 0.0f) atomicAdd(a.glin + o * a.T + j, sums[e]);
  }
}

inline int padded_outputs(int64_t outputs) { return (int)((outputs + 3) / 4 * 4); }
inline size_t backward_smem(int64_t T, int op) { return (size_t)(2 * T * op + op * (kBackwardBlock + 1)) * 4; }

template <int OP, typename WhereT>
int launch_forward(const LinearArgs &a, cudaStream_t stream) {
  auto kernel = linear_rows_forward_kernel<OP, WhereT>;
  const size_t smem = (size_t)a.T * OP * 4;
  if (smem > 40 * 1024) HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kernel<<<(unsigned)((a.B + kForwardBlock - 1) / kForwardBlock), kForwardBlock, smem, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

template <int OP, typename WhereT>
int launch_backward(const LinearArgs &a, cudaStream_t stream) {
  auto kernel = linear_rows_backward_kernel<OP, WhereT>;
  const size_t smem = backward_smem(a.T, OP);
  if (smem > 48 * 1024) HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t blocks = (a.B + kBackwardBlock - 1) / kBackwardBlock;
  // four CTAs per SM, and a tree for every warp
  const int64_t splits = std::max<int64_t>(1, std::min<int64_t>(148 * 4 / blocks, (a.T + 7) / 8));
  kernel<<<dim3((unsigned)std::min<int64_t>(blocks, 148 * 4), (unsigned)splits), kBackwardBlock, smem, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

template <typename F>
int with_outputs(int64_t outputs, F &&f) {
  switch (padded_outputs(outputs)) {
    case 4: return f(std::integral_constant<int, 4>{});
    case 8: return f(std::integral_constant<int, 8>{});
    case 12: return f(std::integral_constant<int, 12>{});
    case 16: return f(std::integral_constant<int, 16>{});
    default: return HT_ERR_UNSUPPORTED;
  }
}

// The paths: row by row, or with a thread per evaluation where x is not aligned for the row copies.
int walk_paths(const ht_forest_problem *p, const float *x, const float *thr, const int32_t *ord, const float *w, const EvalRecords &r,
               uint32_t *status_word, cudaStream_t stream) {
  const int rc = rows_forward(p, x, thr, ord, w, nullptr, r.dx, r.where, status_word, stream);
  if (rc != HT_ERR_UNSUPPORTED) return rc;
  return multi_forward<float>(p, x, thr, ord, w, nullptr, PathRecordsOf<float>{r.dx, r.where}, stream);
}

}  // namespace

bool linear_tiled_takes(const ht_forest_problem *p, int64_t outputs) {
  return p->M == 1 && outputs >= 1 && outputs <= kMostOutputs && rows_forward_takes(p) && rows_x_gradient_takes(p) &&
         backward_smem(p->T, padded_outputs(outputs)) <= tile::kSmemBudget;
}

size_t linear_tiled_bytes(const ht_forest_problem *p) {
  return 2 * record_array_bytes(p, 4) + record_array_bytes(p, where_bytes(p->depth));
}

int linear_tiled_forward(const ht_forest_problem *p, int64_t outputs, const float *x, const float *thr, const int32_t *ord,
                         const float *w, const float *lin, const float *bias, float *out, void *area, uint32_t *status_word,
                         cudaStream_t stream) {
  if (!linear_tiled_takes(p, outputs)) return HT_ERR_UNSUPPORTED;
  LinearArgs a = {};
  a.r = eval_record_arrays(p, area);
  const int rc = walk_paths(p, x, thr, ord, w, a.r, status_word, stream);
  if (rc != HT_OK) return rc;
  a.w = w;
  a.lin = lin;
  a.bias = bias;
  a.out = out;
  a.B = p->B;
  a.T = p->T;
  a.L = ((int64_t)1) << p->depth;
  a.O = outputs;
  if (where_bytes(p->depth) == 2)
    return with_outputs(outputs, [&](auto op) { return launch_forward<decltype(op)::value, unsigned short>(a, stream); });
  return with_outputs(outputs, [&](auto op) { return launch_forward<decltype(op)::value, uint32_t>(a, stream); });
}

int linear_tiled_backward(const ht_forest_problem *p, int64_t outputs, const float *x, const float *thr, const int32_t *ord,
                          const float *w, const float *lin, const float *g, float *gx, float *gthr, float *gw, float *glin,
                          void *area, bool kept, uint32_t *status_word, cudaStream_t stream) {
  if (!linear_tiled_takes(p, outputs)) return HT_ERR_UNSUPPORTED;
  LinearArgs a = {};
  a.r = eval_record_arrays(p, area);
  if (!kept) {
    const int rc = walk_paths(p, x, thr, ord, w, a.r, status_word, stream);
    if (rc != HT_OK) return rc;
  }
  a.w = w;
  a.lin = lin;
  a.g = g;
  a.glin = glin;
  a.B = p->B;
  a.T = p->T;
  a.L = ((int64_t)1) << p->depth;
  a.O = outputs;
  a.write_terms = gx != nullptr || gthr != nullptr || gw != nullptr;
  const bool narrow = where_bytes(p->depth) == 2;
  const int rc = narrow ? with_outputs(outputs, [&](auto op) { return launch_backward<decltype(op)::value, unsigned short>(a, stream); })
                        : with_outputs(outputs, [&](auto op) { return launch_backward<decltype(op)::value, uint32_t>(a, stream); });
  if (rc != HT_OK) return rc;
  if (gthr != nullptr || gw != nullptr) {
    const int prc = reduce_parameter_terms(p, a.r, gthr, gw, stream);
    if (prc != HT_OK) return prc;
  }
  return gx == nullptr ? HT_OK : rows_x_gradient(p, ord, a.r.dx, a.r.where, gx, stream);
}

}  // namespace ht
