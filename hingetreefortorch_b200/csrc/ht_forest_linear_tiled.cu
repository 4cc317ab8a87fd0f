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
#include <type_traits>

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
  float minus_zero;
};

// Two numbers in a register pair: one instruction multiplies, adds or fuses both, each rounded as by itself.
using Pair = unsigned long long;
__device__ __forceinline__ Pair pair_of(float low, float high) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(low), "f"(high));
  return r;
}
__device__ __forceinline__ float2 numbers_of(Pair p) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ Pair add_rn(Pair a, Pair b) {
  Pair r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ Pair fma_rn(Pair a, Pair b, Pair c) {
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// a * b, rounded, with a minus zero from the kernel's arguments, which the assembler does not know for one: a product of pairs that
// is added next was seen to be fused with the addition in spite of its rounding mode.  (x + -0 is x, whatever x.)
__device__ __forceinline__ Pair mul_rn(Pair a, Pair b, Pair minus_zero) { return fma_rn(a, b, minus_zero); }

// NP: pairs of outputs; the row of a tree's linear weights holds an even number of them, for loads of 16 bytes.
__host__ __device__ constexpr int row_pairs(int np) { return (np + 1) & ~1; }

// Linear weights as [tree][output], outputs past the last zero: a tree's come in 16-byte broadcasts.
template <int NP>
__device__ __forceinline__ void stage_linear(const LinearArgs &a, float *lt) {
  constexpr int kRow = 2 * row_pairs(NP);
  for (int e = threadIdx.x; e < (int)a.T * kRow; e += blockDim.x) {
    const int j = e / kRow, o = e - j * kRow;
    lt[e] = o < a.O ? __ldg(a.lin + o * a.T + j) : 0.0f;
  }
}
template <int NP>
__device__ __forceinline__ void load_linear(const float *row, Pair (&l)[NP]) {
#pragma unroll
  for (int q = 0; q < NP; q += 2) {
    if (q + 1 < NP) {
      const ulonglong2 two = *reinterpret_cast<const ulonglong2 *>(row + 2 * q);
      l[q] = two.x;
      l[q + 1 < NP ? q + 1 : q] = two.y;
    } else {
      l[q] = *reinterpret_cast<const Pair *>(row + 2 * q);
    }
  }
}

// Thread per sample: out[i, o] = bias[o] + sum over j ascending of (|margin| * lin[o, j]) * w[j, leaf], the reference's order
// and roundings, two outputs per instruction.  A thread per output read every path again for each of them, 32 rows at a time:
// 262144 samples, 100 trees, 10 outputs 321 us there, 73 here (97 with an output per instruction, of a multiple of four; eight
// trees' paths under way: 110 with four).
template <int NP, typename WhereT>
__global__ void __launch_bounds__(kForwardBlock) linear_rows_forward_kernel(const __grid_constant__ LinearArgs a) {
  extern __shared__ __align__(16) float lt[];
  __shared__ float results[kForwardBlock * 2 * NP];
  constexpr int kRow = 2 * row_pairs(NP);
  stage_linear<NP>(a, lt);
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * kForwardBlock + threadIdx.x;
  const int64_t at0 = record_index(min(i, a.B - 1), 0, a.T);
  Pair acc[NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) acc[q] = pair_of(__ldg(a.bias + 2 * q), 2 * q + 1 < a.O ? __ldg(a.bias + 2 * q + 1) : 0.0f);
  const Pair minus_zero = pair_of(a.minus_zero, a.minus_zero);
  constexpr int kAhead = 8;
  const float *margins = a.r.dx + at0;
  const WhereT *wheres = static_cast<const WhereT *>(a.r.where) + at0;
  auto trees = [&](int j0, auto all) {
    constexpr bool ALL = decltype(all)::value;  // eight trees are left
    const int left = (int)a.T - j0;
    float size[kAhead], weight[kAhead];
    uint32_t key[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int from = (ALL ? u : min(u, left - 1)) * kRecordBlock;
      size[u] = fabsf(__ldg(margins + from));
      key[u] = load_where<WhereT>(wheres, from) >> 16;
    }
    const float *leaves = a.w + j0 * a.L;
#pragma unroll
    for (int u = 0; u < kAhead; ++u) weight[u] = __ldg(leaves + (ALL ? u : min(u, left - 1)) * (int)a.L + key[u]);
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (ALL || u < left) {
        Pair l[NP];
        load_linear<NP>(lt + (j0 + u) * kRow, l);
        const Pair size2 = pair_of(size[u], size[u]), weight2 = pair_of(weight[u], weight[u]);
#pragma unroll
        for (int q = 0; q < NP; ++q) acc[q] = add_rn(acc[q], mul_rn(mul_rn(size2, l[q], minus_zero), weight2, minus_zero));
      }
    margins += kAhead * kRecordBlock;
    wheres += kAhead * kRecordBlock;
  };
  int j0 = 0;
  for (; j0 + kAhead <= (int)a.T; j0 += kAhead) trees(j0, std::true_type());
  if (j0 < (int)a.T) trees(j0, std::false_type());
  // the block's results are one run of the output
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const float2 two = numbers_of(acc[q]);
    results[threadIdx.x * a.O + 2 * q] = two.x;
    if (2 * q + 1 < a.O) results[threadIdx.x * a.O + 2 * q + 1] = two.y;
  }
  __syncthreads();
  const int64_t first = (int64_t)blockIdx.x * kForwardBlock * a.O;
  const int count = (int)(min((int64_t)kForwardBlock, a.B - (int64_t)blockIdx.x * kForwardBlock) * a.O);
  for (int e = threadIdx.x; e < count; e += kForwardBlock) a.out[first + e] = results[e];
}

// The sum over the warp's lanes of each of the numbers in `v`: lane l gets that of number l / (32 / W), W the power of two
// that holds them.  Every exchange halves the numbers that a lane holds: 16 shuffles for 16 numbers.
template <int N>
__device__ __forceinline__ float sums_over_lanes(float (&v)[N], int lane) {
  int d = 16;
#pragma unroll
  for (int half = N / 2; half >= 1; half /= 2, d /= 2) {
    const bool upper = (lane & d) != 0;
#pragma unroll
    for (int k = 0; k < half; ++k) {
      const float mine = upper ? v[k + half] : v[k], theirs = upper ? v[k] : v[k + half];
      v[k] = mine + __shfl_xor_sync(0xffffffffu, theirs, d);
    }
  }
#pragma unroll
  for (; d >= 1; d /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], d);
  return v[0];
}

// CTA = a record block of 256 samples at a time (several, one after another), with its upstream gradients [pair of outputs]
// [sample] in shared memory; a warp takes a tree, its lanes samples.  Per evaluation: what arrives at the tree's output,
// through = sum over o of lin[o, j] * g[o]; from it the two terms of the records, which the forest's reductions turn into the
// other gradients; and |margin| * w * g[o] for the linear weights' gradient, summed in registers over the block's samples
// and in shared memory over the blocks.
// Bound by issue slots and the records (14 bytes per evaluation read and written).  262144 samples, 100 trees, 10 outputs: 101 us
// (135 with an output per instruction and 60 shuffles per tree and block).
template <int NP, typename WhereT>
__global__ void __launch_bounds__(kBackwardBlock, 4) linear_rows_backward_kernel(const __grid_constant__ LinearArgs a) {
  extern __shared__ __align__(16) float smem[];
  constexpr int kPitch = kBackwardBlock + 1, kRow = 2 * row_pairs(NP);
  constexpr int kNumbers = NP <= 1 ? 2 : NP <= 2 ? 4 : NP <= 4 ? 8 : 16;
  float *lt = smem;                                         // [T][kRow]
  float *sums = lt + a.T * kRow;                            // [T][kRow]: of the linear weights' gradient
  Pair *gt = reinterpret_cast<Pair *>(sums + a.T * kRow);   // [NP][kPitch]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  stage_linear<NP>(a, lt);
  for (int e = tid; e < (int)a.T * kRow; e += kBackwardBlock) sums[e] = 0.0f;
  for (int e = tid; e < NP * kPitch; e += kBackwardBlock) gt[e] = 0ull;
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
      reinterpret_cast<float *>(gt + (o >> 1) * kPitch + s)[o & 1] = s < here ? __ldg(a.g + i0 * O + e) : 0.0f;
    }
    __syncthreads();
    for (int j = tree0 + warp; j < tree_end; j += kBackwardBlock / 32) {
      const int64_t at0 = (block * a.T + j) * kRecordBlock + lane;
      const float *leaves = a.w + j * a.L;
      Pair l[NP], gl[NP];
      load_linear<NP>(lt + j * kRow, l);
#pragma unroll
      for (int q = 0; q < NP; ++q) gl[q] = 0ull;
      constexpr int kAhead = 8;
      float nm[kAhead], weight[kAhead];  // (kAhead * 32 samples: the block)
      uint32_t where[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        nm[u] = stream_f32(a.r.dx + at0 + 32 * u);
        where[u] = stream_raw_where<WhereT>(a.r.where, at0 + 32 * u);
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u)  // (positions past the last sample hold anything: they are masked, their leaf is in range)
        weight[u] = __ldg(leaves + min((uint32_t)(a.L - 1), unpack_where<WhereT>(where[u]) >> 16));
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int s = 32 * u + lane;
        const bool on = s < here;
        const float size = fabsf(nm[u]), f = on ? size * weight[u] : 0.0f;
        const Pair f2 = pair_of(f, f);
        Pair through2 = 0ull;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const Pair go = gt[q * kPitch + s];  // (zero past the last sample)
          through2 = fma_rn(l[q], go, through2);
          gl[q] = fma_rn(f2, go, gl[q]);
        }
        const float2 halves = numbers_of(through2);
        const float through = halves.x + halves.y;
        if (a.write_terms && on) {
          __stcs(a.r.dx + at0 + 32 * u, tile::signed_term(nm[u], weight[u] * through));
          __stcs(a.r.dw + at0 + 32 * u, size * through);
        }
      }
      if (a.glin != nullptr) {
        float v[kNumbers];
#pragma unroll
        for (int q = 0; q < kNumbers / 2; ++q) {
          const float2 two = q < NP ? numbers_of(gl[q < NP ? q : 0]) : make_float2(0.f, 0.f);
          v[2 * q] = two.x;
          v[2 * q + 1] = two.y;
        }
        const float mine = sums_over_lanes(v, lane);
        constexpr int kSame = 32 / kNumbers;  // lanes with the same sum
        if (lane % kSame == 0 && lane / kSame < O) sums[j * kRow + lane / kSame] += mine;
      }
    }
  }
  if (a.glin == nullptr) return;
  __syncthreads();
  for (int e = tid; e < (int)a.T * kRow; e += kBackwardBlock) {
    const int j = e / kRow, o = e - j * kRow;
    if (o < O && sums[e] != 0.0f) atomicAdd(a.glin + o * a.T + j, sums[e]);
  }
}

inline int output_pairs(int64_t outputs) { return (int)((outputs + 1) / 2); }
inline size_t backward_smem(int64_t T, int np) { return (size_t)(2 * T * 2 * row_pairs(np)) * 4 + (size_t)np * (kBackwardBlock + 1) * 8; }

template <int NP, typename WhereT>
int launch_forward(const LinearArgs &a, cudaStream_t stream) {
  auto kernel = linear_rows_forward_kernel<NP, WhereT>;
  const size_t smem = (size_t)a.T * 2 * row_pairs(NP) * 4;
  if (smem > 40 * 1024) HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kernel<<<(unsigned)((a.B + kForwardBlock - 1) / kForwardBlock), kForwardBlock, smem, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

template <int NP, typename WhereT>
int launch_backward(const LinearArgs &a, cudaStream_t stream) {
  auto kernel = linear_rows_backward_kernel<NP, WhereT>;
  const size_t smem = backward_smem(a.T, NP);
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
  switch (output_pairs(outputs)) {
    case 1: return f(std::integral_constant<int, 1>{});
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    case 4: return f(std::integral_constant<int, 4>{});
    case 5: return f(std::integral_constant<int, 5>{});
    case 6: return f(std::integral_constant<int, 6>{});
    case 7: return f(std::integral_constant<int, 7>{});
    case 8: return f(std::integral_constant<int, 8>{});
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
         backward_smem(p->T, 2 * (int)((outputs + 3) / 4)) <= tile::kSmemBudget;
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
  a.minus_zero = -0.0f;
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
