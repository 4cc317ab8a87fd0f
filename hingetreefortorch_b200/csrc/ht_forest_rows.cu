// Row-stationary kernels for tabular data with many features.
//
// The tile kernels (ht_forest_tiled.cu) keep a feature-major tile of samples in shared memory and stream the trees past it,
// which is right while a sample's features are few against its decisions.  With C = 784 a tile is 64 samples, and staging it
// takes longer than walking 100 trees over it.  Here the trees' thresholds and feature indices stay in shared memory and
// rows of x stream past them as they lie in memory, by bulk async copies.
#include "ht_forest_rows.cuh"
#include "ht_tile_common.cuh"

#include <algorithm>

namespace ht {

using namespace tile;

namespace {

constexpr int kRowWarps = 16;
constexpr int kRowThreads = kRowWarps * 32;

struct RowPlan {
  int rows;    // per step: 16, 8 or 4
  int trees;   // per CTA
  size_t smem;
};

__host__ __device__ inline size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }
// thresholds and feature indices of the CTA's trees, two buffers of rows, two of results, two barriers
inline size_t row_smem(int64_t N, int64_t C, int rows, int trees) {
  return align16((size_t)trees * N * 4) + align16((size_t)trees * N * 2) + 2 * align16((size_t)rows * C * 4) +
         2 * (size_t)trees * rows * 8 + 64;
}

bool make_row_plan(const ht_forest_problem *p, RowPlan &plan) {
  if (p->K != 1 || p->M < 1 || p->M > 64 || p->C > 65536 || p->depth > 12 || p->T < 1 || p->B < 1 || p->B > 0x7fffffff || p->T > 0x7fffff) return false;
  const int64_t N = threshold_count(p->kind, p->depth);
  for (int rows = 16; rows >= 4; rows /= 2) {
    // as many trees as fit, but groups of the same size; a warp walks 32 trees at a time
    int64_t fit = 0;
    for (int64_t groups = 1; groups <= p->T; ++groups) {
      fit = (p->T + groups - 1) / groups;
      if (row_smem(N, p->C, rows, (int)std::min<int64_t>(fit, 4096)) <= kSmemBudget && fit <= 4096) break;
      fit = 0;
      if ((p->T + groups - 1) / groups < 16) break;
    }
    if (fit >= std::min<int64_t>(p->T, 16)) {
      plan.rows = rows;
      plan.trees = (int)fit;
      plan.smem = row_smem(N, p->C, rows, (int)fit);
      return true;
    }
  }
  return false;
}

struct RowArgs {
  const float *x, *thr, *w;
  float *out;
  Divisor by_M;
  int64_t L;
  int M, width;
  const int32_t *ord;
  float *margin;
  void *where;
  uint32_t *status_word;
  int64_t B, T;
  int C, N, depth, rows, trees, groups, slices;
};

// CTA (one per SM) = a group of trees and a slice of the rows.  A step is `rows` rows: 16 / rows warps share one, a lane walks
// up to four trees at once.  A row is copied as it lies, so features are gathered at random banks (3.4 wavefronts for 32
// lanes on average, as many for the thresholds, which start at an odd pitch per tree): 10 wavefronts per level against 3.4 in
// the tile kernels, but nothing is transposed and the copies run under the walk.  The paths leave through a staging area in
// runs of consecutive samples.
// Bound by shared-memory wavefronts.  262144 x 784, 100 trees of depth 7: 358 us (383 without the heads in registers, 608 with
// a thread per evaluation gathering through L1).
// HEADS: a lane meets the same (up to four) trees in every row, so their roots' and the roots' children's decisions, two of
// the levels, stay in registers.
template <int KIND, typename WhereT, bool HEADS>
__global__ void __launch_bounds__(kRowThreads, 1) rows_forward_kernel(const __grid_constant__ RowArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int R = a.rows, G = a.trees, C = a.C, N = a.N;
  float *thr = reinterpret_cast<float *>(smem);
  unsigned short *ord = reinterpret_cast<unsigned short *>(smem + align16((size_t)G * N * 4));
  unsigned char *row_base = smem + align16((size_t)G * N * 4) + align16((size_t)G * N * 2);
  const uint32_t row_bytes = (uint32_t)align16((size_t)R * C * 4);
  uint2 *stage = reinterpret_cast<uint2 *>(row_base + 2 * (size_t)row_bytes);  // [2][G][R]: margin bits, where
  uint64_t *full = reinterpret_cast<uint64_t *>(stage + 2 * (size_t)G * R);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = blockIdx.x % a.groups, slice = blockIdx.x / a.groups;
  const int64_t j0 = (int64_t)group * G;
  const int trees = (int)min((int64_t)G, a.T - j0);
  const int64_t all_steps = (a.B + R - 1) / R;
  const int64_t per = (all_steps + a.slices - 1) / a.slices;
  const int64_t step0 = slice * per, steps = min(per, all_steps - step0);  // <= 0: nothing to do

  // a full step is one bulk copy; the last rows of x, whose bytes need not be a multiple of 16, are copied by the threads
  auto rows_of = [&](int64_t s) { return (int)min((int64_t)R, a.B - (step0 + s) * R); };
  auto issue = [&](int64_t s) {
    if (s >= steps || rows_of(s) < R) return;
    mbar_expect_tx(&full[s & 1], (uint32_t)R * C * 4);
    bulk_load(smem_addr(row_base + (s & 1) * row_bytes), a.x + (step0 + s) * R * C, (uint32_t)R * C * 4, &full[s & 1]);
  };
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    issue(0);
    issue(1);
  }
  for (int e = tid; e < trees * N; e += kRowThreads) {
    const float t = __ldg(a.thr + j0 * N + e);
    thr[e] = t == 0.0f ? 0.0f : t;  // -0 becomes +0: then threshold - feature is -0 for no feature
    ord[e] = (unsigned short)__ldg(a.ord + j0 * N + e);
  }
  __syncthreads();

  const int per_row = kRowWarps / R, my_row = warp / per_row, part = warp % per_row;
  constexpr int kAtOnce = 4;
  float head_thr[HEADS ? kAtOnce : 1][3];
  int head_ord[HEADS ? kAtOnce : 1][3];
  if constexpr (HEADS) {
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) {
      const int base = min(part * 32 + lane + u * per_row * 32, trees - 1) * N;
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        head_thr[u][h] = thr[base + min(h, N - 1)];
        head_ord[u][h] = ord[base + min(h, N - 1)];
      }
    }
  }
  // the outputs of the group's trees are one run in every row: V numbers per thread, consecutive threads along the run
  auto write_outputs = [&](int64_t s, int here, const uint2 *staged, auto vector) {
    constexpr int V = decltype(vector)::value;
    const int pieces = trees * a.M / V;
    float *to = a.out + ((step0 + s) * R * a.T + j0) * a.M;
    for (int r = my_row; r < here; r += R)
#pragma unroll 4
      for (int q = part * 32 + lane; q < pieces; q += per_row * 32) {
        const uint32_t element = (uint32_t)q * V, t = a.by_M.quotient(element);
        const uint2 path = staged[t * R + r];
        const float size = fabsf(__uint_as_float(path.x));
        const uint32_t key = sizeof(WhereT) == 2 ? path.y >> 8 : path.y >> 16;
        Vec<float, V> v = load_vec<float, V>(a.w + ((j0 + t) * a.L + key) * a.M + (element - t * (uint32_t)a.M));
#pragma unroll
        for (int u = 0; u < V; ++u) v.v[u] = mul_rn(size, v.v[u]);
        *reinterpret_cast<Vec<float, V> *>(to + (int64_t)r * a.T * a.M + element) = v;
      }
  };
  bool poisoned = false;
  for (int64_t s = 0; s < steps; ++s) {
    const int here = rows_of(s);
    float *rows = reinterpret_cast<float *>(row_base + (s & 1) * row_bytes);
    if (here < R) {  // (the buffer's last reader has passed the barrier of the step before)
      for (int e = tid; e < here * C; e += kRowThreads) rows[e] = __ldg(a.x + (step0 + s) * R * C + e);
      __syncthreads();
    } else if (!poisoned && !mbar_wait(&full[s & 1], (uint32_t)((s >> 1) & 1))) {
      poisoned = true;
      if (a.status_word != nullptr) atomicOr(a.status_word, HT_FLAG_PIPELINE_TIMEOUT);
    }
    uint2 *out = stage + (size_t)(s & 1) * G * R;
    const float *x = rows + my_row * C;
    if (my_row < here) {
      for (int t0 = part * 32 + lane; t0 - lane < trees; t0 += per_row * 128) {
        int base[kAtOnce];
        uint32_t v[kAtOnce], at[kAtOnce];
        float best[kAtOnce];
#pragma unroll
        for (int u = 0; u < kAtOnce; ++u) {
          base[u] = min(t0 + u * per_row * 32, trees - 1) * N - 1;  // vertices count from 1
          v[u] = 1;
          at[u] = 1;
          best[u] = 0.0f;
        }
        if (!poisoned) {  // a buffer that never arrived is not read: the paths are those of a zero margin at the root
          auto level = [&](int l) {
#pragma unroll
            for (int u = 0; u < kAtOnce; ++u) {
              const int vertex = KIND == FERN ? l + 1 : (int)v[u];
              float t;
              int feature;
              if (HEADS && l == 0) {
                t = head_thr[u][0];
                feature = head_ord[u][0];
              } else if (HEADS && l == 1) {
                t = vertex == 3 ? head_thr[u][2] : head_thr[u][1];
                feature = vertex == 3 ? head_ord[u][2] : head_ord[u][1];
              } else {
                t = thr[base[u] + vertex];
                feature = ord[base[u] + vertex];
              }
              const float nm = t - x[feature];
              if (l == 0 || fabsf(nm) < fabsf(best[u])) {
                best[u] = nm;
                at[u] = (uint32_t)vertex;
              }
              v[u] = 2 * v[u] + (nm < 0.0f ? 1u : 0u);
            }
          };
          level(0);
          if (a.depth > 1) level(1);
          for (int l = 2; l < a.depth; ++l) level(l);
        }
#pragma unroll
        for (int u = 0; u < kAtOnce; ++u) {
          const int t = t0 + u * per_row * 32;
          const uint32_t key = poisoned ? 0u : bit_reverse(v[u] - (1u << a.depth), a.depth);
          if (t < trees)
            out[t * R + my_row] = make_uint2(__float_as_uint(best[u]), sizeof(WhereT) == 2 ? (at[u] | key << 8) : (at[u] | key << 16));
        }
      }
    }
    __syncthreads();  // rows read, results staged
    if (tid == 0) issue(s + 2);
    if (a.out != nullptr) {
      if (a.width == 4) write_outputs(s, here, out, std::integral_constant<int, 4>{});
      else if (a.width == 2) write_outputs(s, here, out, std::integral_constant<int, 2>{});
      else write_outputs(s, here, out, std::integral_constant<int, 1>{});
    }
    if (a.margin == nullptr) continue;
    // four rows of a tree per thread: they are consecutive samples of one record block
    const int64_t sample = (step0 + s) * R;
    const int64_t at0 = record_index(sample, j0, a.T);
    for (int e = tid; e < trees * R / 4; e += kRowThreads) {
      const int t = e / (R / 4), r = (e - t * (R / 4)) * 4;
      const int64_t at = at0 + (int64_t)t * kRecordBlock + r;
      uint2 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = out[t * R + r + u];
      // (samples past the last are padding of the record block)
      *reinterpret_cast<uint4 *>(a.margin + at) = make_uint4(q[0].x, q[1].x, q[2].x, q[3].x);
      if (sizeof(WhereT) == 2)
        *reinterpret_cast<uint2 *>(static_cast<unsigned short *>(a.where) + at) = make_uint2(q[0].y | q[1].y << 16, q[2].y | q[3].y << 16);
      else
        *reinterpret_cast<uint4 *>(static_cast<uint32_t *>(a.where) + at) = make_uint4(q[0].y, q[1].y, q[2].y, q[3].y);
    }
  }
}

template <typename WhereT>
int launch_rows(const RowArgs &a, int kind, size_t smem, cudaStream_t stream) {
  const bool heads = a.trees <= 128 * (kRowWarps / a.rows);
  auto kernel = kind == TREE ? (heads ? rows_forward_kernel<TREE, WhereT, true> : rows_forward_kernel<TREE, WhereT, false>)
                             : (heads ? rows_forward_kernel<FERN, WhereT, true> : rows_forward_kernel<FERN, WhereT, false>);
  HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
  kernel<<<(unsigned)(a.groups * a.slices), kRowThreads, smem, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

// ---- x gradient ------------------------------------------------------------------------------------------------------

constexpr int kXRows = 32;
constexpr int kXThreads = 512;

struct RowXArgs {
  const float *dx;
  const void *where;
  const int32_t *ord;
  float *gx;
  int64_t B, T;
  int C, N, pitch;
};

// CTA = 32 rows of gx in shared memory (lane = row, so that records are read in runs), a warp per tree.  Two warps may add
// into an element at the same time, hence atomics; on different rows they do not meet.  Every element of gx is written once,
// where scattering into cleared global memory touches it twice and half of it in 32-byte pieces.
// Bound by writing gx: two CTAs per SM for rows of up to 880 features, so that one adds while the other writes.
// 262144 x 784, 100 trees: 234 us, 3.5 TB/s (clearing and scattering took over 500).
template <typename WhereT>
__global__ void __launch_bounds__(kXThreads) rows_x_gradient_kernel(const __grid_constant__ RowXArgs a) {
  extern __shared__ __align__(16) float tile_rows[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * kXRows;
  const int rows = (int)min((int64_t)kXRows, a.B - row0);
  for (int e = tid; e < kXRows * a.pitch; e += kXThreads) tile_rows[e] = 0.0f;
  __syncthreads();
  constexpr int kAhead = 4, kWarps = kXThreads / 32;
  const int64_t at0 = record_index(row0, 0, a.T) + lane;
  float *mine = tile_rows + lane * a.pitch;
  for (int64_t j0 = warp; j0 < a.T; j0 += kWarps * kAhead) {
    float d[kAhead];
    uint32_t vertex[kAhead];
    int feature[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int64_t j = j0 + u * kWarps;
      const bool on = j < a.T && lane < rows;
      d[u] = on ? __ldcs(a.dx + at0 + j * kRecordBlock) : 0.0f;
      vertex[u] = on ? load_where<WhereT>(a.where, at0 + j * kRecordBlock) & 0xffffu : 1u;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int64_t j = min(j0 + u * kWarps, a.T - 1);
      feature[u] = __ldg(a.ord + j * a.N + vertex[u] - 1);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (d[u] != 0.0f) atomicAdd(mine + feature[u], d[u]);  // (a NaN is not equal to 0)
  }
  __syncthreads();
  float *out = a.gx + row0 * a.C;
  // (a number per lane: 16 bytes per lane would take every row of four banks four times)
  for (int r = warp; r < rows; r += kWarps)
    for (int c = lane; c < a.C; c += 32) __stcs(out + (int64_t)r * a.C + c, tile_rows[r * a.pitch + c]);
}

inline size_t row_x_smem(int64_t C) { return (size_t)kXRows * (C | 1) * 4; }

}  // namespace

// One CTA per SM, and a CTA fetches its parameters once: groups x slices as close below 148 as it gets.
static int row_slices(const ht_forest_problem *p, const RowPlan &plan) {
  const int64_t steps = (p->B + plan.rows - 1) / plan.rows, groups = (p->T + plan.trees - 1) / plan.trees;
  return (int)std::max<int64_t>(1, std::min<int64_t>(148 / std::min<int64_t>(groups, 148), steps));
}

// Rounds of CTAs, each of them steps x (levels of the walks that a warp does one after another, outputs, row copies) behind
// the fetch of its parameters.  The coefficients are a least-squares fit to forwards in a loop (B 1000 .. 65536, C 32 .. 1500, T 40
// .. 800, depth 5 .. 10, M 1 .. 10).  Single calls on cold caches (profiles/forward_kernel_choice.csv) take 1.3 times the estimate,
// give or take 28 %; the choice between the kernels needs the ratio of two estimates, and forward_tiled_cost() is off likewise.
double rows_forward_cost(const ht_forest_problem *p) {
  RowPlan plan;
  if (!make_row_plan(p, plan)) return -1.0;
  const int64_t groups = (p->T + plan.trees - 1) / plan.trees, slices = row_slices(p, plan);
  const double waves = (double)((groups * slices + 147) / 148);
  const double steps = (double)(((p->B + plan.rows - 1) / plan.rows + slices - 1) / slices);
  const int at_once = 128 * (kRowWarps / plan.rows), rounds = (plan.trees + at_once - 1) / at_once;
  return 6.1 + waves * (steps * (0.34 * rounds * p->depth + 0.22e-3 * plan.rows * plan.trees * (double)p->M + 0.008e-3 * plan.rows * (double)p->C) +
                        0.13e-3 * plan.trees * (double)threshold_count(p->kind, p->depth));
}

bool rows_forward_takes(const ht_forest_problem *p) {
  RowPlan plan;
  return make_row_plan(p, plan);
}

int rows_forward(const ht_forest_problem *p, const float *x, const float *thr, const int32_t *ord, const float *w, float *out,
                 float *margin, void *where, uint32_t *status_word, cudaStream_t stream) {
  RowPlan plan;
  if (!make_row_plan(p, plan) || (reinterpret_cast<uintptr_t>(x) & 15u) != 0) return HT_ERR_UNSUPPORTED;
  RowArgs a = {};
  a.x = x;
  a.thr = thr;
  a.ord = ord;
  a.margin = margin;
  a.where = where;
  a.w = w;
  a.out = out;
  a.M = (int)p->M;
  a.L = ((int64_t)1) << p->depth;
  a.by_M = Divisor((uint32_t)std::max<int64_t>(p->M, 1));
  a.width = out != nullptr ? vector_width(p->M, sizeof(float), {w, out}) : 1;
  a.status_word = status_word;
  a.B = p->B;
  a.T = p->T;
  a.C = (int)p->C;
  a.N = (int)threshold_count(p->kind, p->depth);
  a.depth = p->depth;
  a.rows = plan.rows;
  a.trees = plan.trees;
  a.groups = (int)((p->T + plan.trees - 1) / plan.trees);
  a.slices = row_slices(p, plan);
  return where_bytes(p->depth) == 2 ? launch_rows<unsigned short>(a, p->kind, plan.smem, stream)
                                    : launch_rows<uint32_t>(a, p->kind, plan.smem, stream);
}

bool rows_x_gradient_takes(const ht_forest_problem *p) {
  return p->K == 1 && row_x_smem(p->C) <= kSmemBudget && p->depth <= 15 && p->B <= 0x7fffffff && p->B > 0;
}

int rows_x_gradient(const ht_forest_problem *p, const int32_t *ord, const float *dx, const void *where, float *gx, cudaStream_t stream) {
  if (!rows_x_gradient_takes(p)) return HT_ERR_UNSUPPORTED;
  RowXArgs a = {dx, where, ord, gx, p->B, p->T, (int)p->C, (int)threshold_count(p->kind, p->depth), (int)(p->C | 1)};
  auto kernel = where_bytes(p->depth) == 2 ? rows_x_gradient_kernel<unsigned short> : rows_x_gradient_kernel<uint32_t>;
  HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
  kernel<<<(unsigned)((p->B + kXRows - 1) / kXRows), kXThreads, row_x_smem(p->C), stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

}  // namespace ht
