// Row-stationary kernels for tabular data with many features.
//
// The tile kernels (ht_forest_tiled.cu) keep a feature-major tile of samples in shared memory and stream the trees past it,
// which is right while a sample's features are few against its decisions.  With C = 784 a tile is 64 samples, and staging it
// takes longer than walking 100 trees over it.  Here the trees' thresholds and feature indices stay in shared memory and
// rows of x stream past them as they lie in memory, by bulk async copies.
#include "ht_forest_rows.cuh"
#include "ht_tile_common.cuh"
#include "ht_tma.cuh"

#include <algorithm>
#include <type_traits>

namespace ht {

using namespace tile;

namespace {

constexpr int kMostWalkers = 28;  // warps that walk; one more keeps the rows coming
constexpr int kAtOnce = 2;        // sets of trees that a warp walks at once

struct RowPlan {
  int rows;     // per step: 16, 8 or 4
  int trees;    // per CTA
  int buffers;  // of rows: 2 or more
  int walkers;  // warps
  size_t smem;
};

// Between the rows of a step in shared memory, in numbers.  The lanes of a warp look at up to 16 rows, all at the same feature in
// the root and at few different ones below: rows that start 4 banks apart or an odd or even number of banks meet in two ways at
// most, where 8, 16 or 32 apart (C a multiple of 8) they would in four to sixteen.
__host__ __device__ inline int64_t row_pitch(int64_t C) { return (C & 7) == 0 ? C + 4 : C; }

__host__ __device__ inline size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }
// thresholds and feature indices of the CTA's trees, buffers of rows, two of results (for outputs), two barriers per buffer
constexpr int kMostBuffers = 8;
inline size_t row_smem(int64_t N, int64_t C, int rows, int trees, int buffers, bool outputs) {
  return align16((size_t)trees * N * 4) + align16((size_t)trees * N * 2) + buffers * align16((size_t)rows * row_pitch(C) * 4) +
         (outputs ? 2 * (size_t)trees * rows * 8 : 0) + 2 * kMostBuffers * 8;
}

// `outputs`: of the leaves, not only paths.
bool make_row_plan(const ht_forest_problem *p, RowPlan &plan, bool outputs = true) {
  if (p->K != 1 || p->M < 1 || p->M > 64 || p->C > 65536 || p->depth > 12 || p->T < 1 || p->B < 1 || p->B > 0x7fffffff || p->T > 0x7fffff) return false;
  const int64_t N = threshold_count(p->kind, p->depth);
  for (int rows = 16; rows >= 4; rows /= 2) {
    // as many trees as fit, but groups of the same size
    int64_t fit = 0;
    for (int64_t groups = 1; groups <= p->T; ++groups) {
      fit = (p->T + groups - 1) / groups;
      if (row_smem(N, p->C, rows, (int)std::min<int64_t>(fit, 4096), 2, true) <= kSmemBudget && fit <= 4096) break;
      fit = 0;
      if ((p->T + groups - 1) / groups < 16) break;
    }
    if (fit >= std::min<int64_t>(p->T, 16)) {
      plan.rows = rows;
      plan.trees = (int)fit;
      plan.buffers = 2;
      // A copy takes longer to arrive than a step takes to walk: what room is left goes to more copies under way.
      while (plan.buffers < kMostBuffers && row_smem(N, p->C, rows, (int)fit, plan.buffers + 1, outputs) <= kSmemBudget) ++plan.buffers;
      plan.smem = row_smem(N, p->C, rows, (int)fit, plan.buffers, outputs);
      // A step lasts as long as its busiest warp: as few warps as give all the same number of sets of trees.  262144 x 784, 100
      // trees, 50 sets: 25 warps walk two each, 204 us; 263 with 20 and 284 with 24 (some walk three), 217 with 28.  Over 16 sizes and
      // every count from 12 to 28 the rule takes at most 5 % more than the best count, 2 % on average (profiles/conv_rows_codes_ncu.md).
      const int sets = (int)((fit + 32 / rows - 1) / (32 / rows)), rounds = (sets + kAtOnce * kMostWalkers - 1) / (kAtOnce * kMostWalkers);
      plan.walkers = sets <= kMostWalkers ? std::max(sets, 16) : (sets + kAtOnce * rounds - 1) / (kAtOnce * rounds);
      return true;
    }
  }
  return false;
}

struct RowArgs {
  const float *x, *thr, *w;
  float *out;
  Divisor by_M, by_pieces;  // a place among a row's outputs by M, one among the step's pieces of outputs by those of a row
  int64_t L;
  int M, width;
  const int32_t *ord;
  float *margin;
  void *where;
  uint32_t *status_word;
  int64_t B, T;
  int C, N, depth, rows, trees, groups, slices, buffers, walkers;
};

// CTA (one per SM) = a group of trees and a slice of the rows.  A step is `rows` rows; a warp's lanes are those rows on 32 / rows
// trees, and it walks up to two such sets of trees at once.  Rows are copied as they lie, so features are gathered at random
// banks (3.4 wavefronts for 32 lanes on average where the vertices differ), but lanes on one tree share its thresholds and
// feature indices, nothing is transposed and the copies run under the walk.  The paths leave from registers, runs of consecutive
// samples; outputs through a staging area.
// Bound by shared-memory wavefronts and the rows' arrival.  262144 x 784, 100 trees of depth 7, paths only: 204 us, 4.8 TB/s (358 with
// 32 trees on one row per warp, whose thresholds and indices lay at random banks as well; 608 with a thread per evaluation gathering
// through L1).
// HEADS: a lane meets the same (one or two) trees in every step, so their roots' and the roots' children's decisions, two of
// the levels, stay in registers.
// DEPTH: of the trees, 0 for any.
template <int KIND, int DEPTH, typename WhereT, bool HEADS>
__global__ void __launch_bounds__(32 * kMostWalkers + 32, 1) rows_forward_kernel(const __grid_constant__ RowArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int R = a.rows, G = a.trees, C = a.C, N = a.N, depth = DEPTH > 0 ? DEPTH : a.depth;
  const int walkers = a.walkers, walking = 32 * walkers;  // warps, threads
  float *thr = reinterpret_cast<float *>(smem);
  unsigned short *ord = reinterpret_cast<unsigned short *>(smem + align16((size_t)G * N * 4));
  unsigned char *row_base = smem + align16((size_t)G * N * 4) + align16((size_t)G * N * 2);
  const int pitch = (int)row_pitch(C);
  const uint32_t row_bytes = (uint32_t)align16((size_t)R * pitch * 4);
  uint64_t *full = reinterpret_cast<uint64_t *>(row_base + a.buffers * (size_t)row_bytes);  // rows arrived
  uint64_t *left = full + kMostBuffers;                                                     // rows read by every walking warp
  uint2 *stage = reinterpret_cast<uint2 *>(left + kMostBuffers);  // [2][G][R]: margin bits, where (with outputs only)

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = blockIdx.x % a.groups, slice = blockIdx.x / a.groups;
  const int64_t j0 = (int64_t)group * G;
  const int trees = (int)min((int64_t)G, a.T - j0);
  const int64_t all_steps = (a.B + R - 1) / R;
  const int64_t per = (all_steps + a.slices - 1) / a.slices;
  const int64_t step0 = slice * per, steps = min(per, all_steps - step0);  // <= 0: nothing to do

  // a full step is one bulk copy, or one per row; the last rows of x, whose bytes need not be a multiple of 16, are copied by the
  // threads
  auto rows_of = [&](int64_t s) { return (int)min((int64_t)R, a.B - (step0 + s) * R); };
  auto issue = [&](int64_t s, int buffer) {
    if (rows_of(s) < R) return;
    mbar_expect_tx(&full[buffer], (uint32_t)R * C * 4);
    const uint32_t to = smem_addr(row_base + buffer * (size_t)row_bytes);
    const float *from = a.x + (step0 + s) * R * C;
    if (pitch == C)
      bulk_load(to, from, (uint32_t)R * C * 4, &full[buffer]);
    else
      for (int r = 0; r < R; ++r) bulk_load(to + (uint32_t)(r * pitch) * 4u, from + (int64_t)r * C, (uint32_t)C * 4, &full[buffer]);
  };
  if (tid == walking) {  // the warp that keeps the rows coming: the first ones before anything else
    for (int k = 0; k < a.buffers; ++k) {
      mbar_init(&full[k], 1);
      mbar_init(&left[k], walkers);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int s = 0; s < a.buffers && s < steps; ++s) issue(s, s);
  }
  for (int e = tid; e < trees * N; e += walking + 32) {
    const float t = __ldg(a.thr + j0 * N + e);
    thr[e] = t == 0.0f ? 0.0f : t;  // -0 becomes +0: then threshold - feature is -0 for no feature
    ord[e] = (unsigned short)__ldg(a.ord + j0 * N + e);
  }
  __syncthreads();
  if (warp == walkers) {  // refills a buffer when every walking warp has left it
    if (lane == 0) {
      int buffer = 0;
      uint32_t phase = 0;
      for (int64_t s = a.buffers; s < steps; ++s) {
        if (!mbar_wait(&left[buffer], phase)) break;  // (the walking warps flag the rows that fail to come)
        issue(s, buffer);
        if (++buffer == a.buffers) {
          buffer = 0;
          phase ^= 1u;
        }
      }
    }
    return;
  }

  const int my_row = lane & (R - 1), per_set = 32 / R, my_tree = lane / R;
  const int sets = (trees + per_set - 1) / per_set;
  float head_thr[HEADS ? kAtOnce : 1][3];
  uint32_t head_ord[HEADS ? kAtOnce : 1][3];
  const uint32_t thr_addr = smem_addr(thr), ord_addr = smem_addr(ord);
  if constexpr (HEADS) {
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) {
      const int base = min((warp + u * walkers) * per_set + my_tree, trees - 1) * N;
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
    const bool whole = trees == G;
#pragma unroll 4
    for (uint32_t e = (uint32_t)tid; e < (uint32_t)(here * pieces); e += (uint32_t)walking) {
      const uint32_t r = whole ? a.by_pieces.quotient(e) : e / (uint32_t)pieces;
      const uint32_t element = (e - r * (uint32_t)pieces) * V, t = a.by_M.quotient(element);
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
  int buffer = 0;
  uint32_t phase = 0;
  for (int64_t s = 0; s < steps; ++s) {
    const int here = rows_of(s);
    float *rows = reinterpret_cast<float *>(row_base + buffer * (size_t)row_bytes);
    if (here < R) {  // once all have left the buffer
      named_barrier(1, walking);
      for (int e = tid; e < here * C; e += walking) {
        const int r = e / C;
        rows[r * pitch + e - r * C] = __ldg(a.x + (step0 + s) * R * C + e);
      }
      named_barrier(1, walking);
    } else if (!poisoned && !mbar_wait(&full[buffer], phase)) {
      poisoned = true;
      if (a.status_word != nullptr) atomicOr(a.status_word, HT_FLAG_PIPELINE_TIMEOUT);
    }
    uint2 *out = stage + (size_t)(s & 1) * G * R;
    const uint32_t x = smem_addr(rows + min(my_row, here - 1) * pitch);  // lanes past the last row repeat it and leave nothing
    const int64_t at0 = record_index((step0 + s) * R + my_row, j0, a.T);
    auto walk_sets = [&](int first_set, auto count) {
      constexpr int n = decltype(count)::value;
      uint32_t thr_at[n], ord_at[n], v[n], at[n];
      float best[n];
#pragma unroll
      for (int u = 0; u < n; ++u) {
        const uint32_t base = (uint32_t)(min((first_set + u * walkers) * per_set + my_tree, trees - 1) * N);
        thr_at[u] = thr_addr + 4u * base;
        ord_at[u] = ord_addr + 2u * base;
        v[u] = 1;
        at[u] = 1;
        best[u] = 0.0f;
      }
      if (!poisoned) {  // a buffer that never arrived is not read: the paths are those of a zero margin at the root
        auto level = [&](int l) {
#pragma unroll
          for (int u = 0; u < n; ++u) {
            const uint32_t vertex = KIND == FERN ? (uint32_t)l + 1u : v[u];
            float t;
            uint32_t feature;
            if (HEADS && l == 0) {
              t = head_thr[u][0];
              feature = head_ord[u][0];
            } else if (HEADS && l == 1) {
              t = vertex == 3u ? head_thr[u][2] : head_thr[u][1];
              feature = vertex == 3u ? head_ord[u][2] : head_ord[u][1];
            } else {
              t = lds_f32(thr_at[u] + 4u * vertex - 4u);  // vertices count from 1
              feature = lds_ord<uint16_t>(ord_at[u] + 2u * vertex - 2u);
            }
            const float nm = t - lds_f32(x + 4u * feature);
            if (l == 0 || fabsf(nm) < fabsf(best[u])) {
              best[u] = nm;
              at[u] = vertex;
            }
            v[u] = __funnelshift_l(__float_as_uint(nm), v[u], 1);  // (set where nm < 0: a sum that is no number is positive)
          }
        };
        if constexpr (DEPTH > 0) {
          static_for<0, DEPTH>([&](auto l) { level(decltype(l)::value); });
        } else {
          level(0);
          if (depth > 1) level(1);
          for (int l = 2; l < depth; ++l) level(l);
        }
      }
#pragma unroll
      for (int u = 0; u < n; ++u) {
        const int t = (first_set + u * walkers) * per_set + my_tree;
        const uint32_t key = poisoned ? 0u : bit_reverse(v[u] - (1u << depth), depth);
        if (t >= trees || my_row >= here) continue;
        if (a.out != nullptr)
          out[t * R + my_row] = make_uint2(__float_as_uint(best[u]), sizeof(WhereT) == 2 ? (at[u] | key << 8) : (at[u] | key << 16));
        if (a.margin != nullptr) {  // the samples of a tree are consecutive in a record block
          __stcs(a.margin + at0 + (int64_t)t * kRecordBlock, best[u]);
          store_where<WhereT>(a.where, at0 + (int64_t)t * kRecordBlock, at[u], key);
        }
      }
    };
    for (int set = warp; set < sets; set += kAtOnce * walkers) {
      const int n = min(kAtOnce, (sets - set + walkers - 1) / walkers);
      if (n == kAtOnce) walk_sets(set, std::integral_constant<int, kAtOnce>{});
      else walk_sets(set, std::integral_constant<int, 1>{});
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&left[buffer]);
    if (++buffer == a.buffers) {
      buffer = 0;
      phase ^= 1u;
    }
    if (a.out != nullptr) {
      named_barrier(1, walking);  // results staged (and those of two steps before written)
      if (a.width == 4) write_outputs(s, here, out, std::integral_constant<int, 4>{});
      else if (a.width == 2) write_outputs(s, here, out, std::integral_constant<int, 2>{});
      else write_outputs(s, here, out, std::integral_constant<int, 1>{});
    }
  }
  if (poisoned)  // copies still under way end, or are given up on, before the CTA's shared memory goes
    for (int64_t s = max((int64_t)0, steps - a.buffers); s < steps; ++s)
      if (rows_of(s) == R) mbar_wait(&full[s % a.buffers], (uint32_t)((s / a.buffers) & 1), 64);
}

template <int KIND, int DEPTH>
auto rows_kernel(bool heads) {
  using WhereT = typename std::conditional<(DEPTH <= 8), unsigned short, uint32_t>::type;
  return heads ? rows_forward_kernel<KIND, DEPTH, WhereT, true> : rows_forward_kernel<KIND, 0, WhereT, false>;
}
template <int KIND>
auto rows_kernel_of(int depth, bool heads) {
  switch (depth) {
#define HT_DEPTH_CASE(D) \
  case D:                \
    return rows_kernel<KIND, D>(heads);
    HT_DEPTH_CASE(3)
    HT_DEPTH_CASE(4)
    HT_DEPTH_CASE(5)
    HT_DEPTH_CASE(6)
    HT_DEPTH_CASE(7)
    HT_DEPTH_CASE(8)
    HT_DEPTH_CASE(9)
    HT_DEPTH_CASE(10)
#undef HT_DEPTH_CASE
    default:
      if (depth <= 8) return heads ? rows_forward_kernel<KIND, 0, unsigned short, true> : rows_forward_kernel<KIND, 0, unsigned short, false>;
      return heads ? rows_forward_kernel<KIND, 0, uint32_t, true> : rows_forward_kernel<KIND, 0, uint32_t, false>;
  }
}

int launch_rows(const RowArgs &a, int kind, size_t smem, cudaStream_t stream) {
  const bool heads = a.trees <= kAtOnce * a.walkers * (32 / a.rows);  // a lane's trees in one go
  auto kernel = kind == TREE ? rows_kernel_of<TREE>(a.depth, heads) : rows_kernel_of<FERN>(a.depth, heads);
  HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
  kernel<<<(unsigned)(a.groups * a.slices), 32 * a.walkers + 32, smem, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

// ---- x gradient ------------------------------------------------------------------------------------------------------

constexpr int kXRows = 16;
constexpr int kXTrees = 32 / kXRows;  // of a warp at a time
constexpr int kXThreads = 512;

struct RowXArgs {
  const float *dx;
  const void *where;
  const int32_t *ord;
  float *gx;
  int64_t B, T;
  int C, N, pitch;
};

// CTA = 16 rows of gx in shared memory (a warp is 16 rows on two trees, so that records are read in runs).  Two warps may add
// into an element at the same time, hence atomics; on different rows they do not meet.  Every element of gx is written once,
// where scattering into cleared global memory touches it twice and half of it in 32-byte pieces.  The records of a warp's first
// sets of trees are under way while the rows are cleared.
// BULK: rows leave by bulk copies (they lie on 16-byte boundaries here and there).
// Bound by writing gx: four CTAs per SM for rows of up to 880 features, so that some add while others write.
// 262144 x 784, 100 trees: 203 us, 4.8 TB/s (237 with 32 rows, four trees at a time after the clearing, and rows written by the threads;
// clearing and scattering took over 500).
template <typename WhereT, bool BULK>
__global__ void __launch_bounds__(kXThreads) rows_x_gradient_kernel(const __grid_constant__ RowXArgs a) {
  extern __shared__ __align__(16) float tile_rows[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * kXRows;
  const int rows = (int)min((int64_t)kXRows, a.B - row0);
  constexpr int kAhead = 4, kApart = kXThreads / 32 * kXTrees;  // trees between a lane's
  const int my_row = lane % kXRows, first = warp * kXTrees + lane / kXRows;
  const int64_t at0 = record_index(row0, 0, a.T) + my_row;
  const int T = (int)a.T;
  float d[kAhead];
  uint32_t vertex[kAhead];
  auto fetch = [&](int j0) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int j = j0 + u * kApart;
      d[u] = 0.0f;
      vertex[u] = 1u;
      if (j < T && my_row < rows) {
        d[u] = stream_f32(a.dx + at0 + (int64_t)j * kRecordBlock);
        vertex[u] = stream_raw_where<WhereT>(a.where, at0 + (int64_t)j * kRecordBlock);
      }
    }
  };
  fetch(first);
  for (int e = tid; e < kXRows * a.pitch / 4; e += kXThreads) reinterpret_cast<float4 *>(tile_rows)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  float *mine = tile_rows + my_row * a.pitch;
  for (int j0 = first; j0 - lane / kXRows < T; j0 += kApart * kAhead) {
    if (j0 != first) fetch(j0);
    int feature[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int j = min(j0 + u * kApart, T - 1);
      feature[u] = __ldg(a.ord + (int64_t)j * a.N + (unpack_where<WhereT>(vertex[u]) & 0xffffu) - 1);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (d[u] != 0.0f) atomicAdd(mine + feature[u], d[u]);  // (a NaN is not equal to 0)
  }
  float *out = a.gx + row0 * a.C;
  if constexpr (BULK) {
    tma::fence_async_shared();
    __syncthreads();
    if (warp == 0) {
      if (lane < rows) tma::store_rows(out + (int64_t)lane * a.C, smem_addr(mine), (uint32_t)a.C * 4u);  // (lane < 16: its own row)
      tma::commit_group();
      tma::wait_stores_read();
    }
  } else {
    __syncthreads();
    // (a number per lane: 16 bytes per lane would take every row of four banks four times)
    for (int r = warp; r < rows; r += kXThreads / 32)
      for (int c = lane; c < a.C; c += 32) __stcs(out + (int64_t)r * a.C + c, tile_rows[r * a.pitch + c]);
  }
}

// Rows that leave by bulk copies start on 16-byte boundaries, four banks apart or a multiple of that; others at an odd distance.
inline int64_t row_x_pitch(int64_t C, bool bulk) { return bulk ? row_pitch(C) : C | 1; }
inline size_t row_x_smem(int64_t C) { return (size_t)kXRows * std::max(row_x_pitch(C, (C & 3) == 0), C | 1) * 4; }

}  // namespace

// One CTA per SM, and a CTA fetches its parameters once: groups x slices as close below 148 as it gets.
static int row_slices(const ht_forest_problem *p, const RowPlan &plan) {
  const int64_t steps = (p->B + plan.rows - 1) / plan.rows, groups = (p->T + plan.trees - 1) / plan.trees;
  return (int)std::max<int64_t>(1, std::min<int64_t>(148 / std::min<int64_t>(groups, 148), steps));
}

// Microseconds of a single call on cold caches: rounds of CTAs, each of them steps x (levels of the sets of trees walked, paths and
// outputs, the latter by bytes and by the stores they go in (a third more for these where the leaf weights exceed 10 MB), row copies by bytes and by what of them comes from memory rather than
// from L2, where groups of trees share the rows) behind the fetch of its parameters.  A fit to profiles/forward_kernel_choice.csv (the
// logarithm of estimate over time has a spread of 0.12), as are forward_tiled_cost() (0.09) and the estimate for a thread per evaluation
// (0.13); rows_are_better() says how good the choice between them is.
double rows_forward_cost(const ht_forest_problem *p) {
  RowPlan plan;
  if (!make_row_plan(p, plan)) return -1.0;
  const int64_t groups = (p->T + plan.trees - 1) / plan.trees, slices = row_slices(p, plan);
  const double waves = (double)((groups * slices + 147) / 148);
  const double steps = (double)(((p->B + plan.rows - 1) / plan.rows + slices - 1) / slices);
  const int per_set = 32 / plan.rows, sets = (plan.trees + per_set - 1) / per_set;
  const int rounds = (sets + kAtOnce * kMostWalkers - 1) / (kAtOnce * kMostWalkers);
  const double paths = (double)plan.rows * plan.trees, outputs = paths * (double)p->M;
  const bool far_leaves = (double)p->T * (double)(((int64_t)1) << p->depth) * (double)p->M > 2.5e6;
  return 13.7 + waves * (steps * (0.446 + (2.34e-3 * sets + 0.0675 * rounds) * p->depth + 0.369e-3 * paths +
                                  (0.0356e-3 + (far_leaves ? 0.444e-3 : 0.329e-3) / vector_width(p->M, sizeof(float), {})) * outputs +
                                  (0.0112e-3 + 0.0276e-3 * slices / 148.0) * plan.rows * (double)p->C) +
                         0.71e-3 * plan.trees * (double)threshold_count(p->kind, p->depth));
}

bool rows_forward_takes(const ht_forest_problem *p) {
  RowPlan plan;
  return make_row_plan(p, plan);
}

int rows_forward(const ht_forest_problem *p, const float *x, const float *thr, const int32_t *ord, const float *w, float *out,
                 float *margin, void *where, uint32_t *status_word, cudaStream_t stream) {
  RowPlan plan;
  if (!make_row_plan(p, plan, out != nullptr) || (reinterpret_cast<uintptr_t>(x) & 15u) != 0) return HT_ERR_UNSUPPORTED;
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
  a.by_pieces = Divisor((uint32_t)std::max<int64_t>(plan.trees * p->M / a.width, 1));
  a.status_word = status_word;
  a.B = p->B;
  a.T = p->T;
  a.C = (int)p->C;
  a.N = (int)threshold_count(p->kind, p->depth);
  a.depth = p->depth;
  a.rows = plan.rows;
  a.buffers = plan.buffers;
  a.walkers = plan.walkers;
  a.trees = plan.trees;
  a.groups = (int)((p->T + plan.trees - 1) / plan.trees);
  a.slices = row_slices(p, plan);
  return launch_rows(a, p->kind, plan.smem, stream);
}

bool rows_x_gradient_takes(const ht_forest_problem *p) {
  return p->K == 1 && row_x_smem(p->C) <= kSmemBudget && p->depth <= 15 && p->B <= 0x7fffffff && p->B > 0;
}

int rows_x_gradient(const ht_forest_problem *p, const int32_t *ord, const float *dx, const void *where, float *gx, cudaStream_t stream) {
  if (!rows_x_gradient_takes(p)) return HT_ERR_UNSUPPORTED;
  const bool bulk = (p->C & 3) == 0 && (reinterpret_cast<uintptr_t>(gx) & 15u) == 0;
  RowXArgs a = {dx, where, ord, gx, p->B, p->T, (int)p->C, (int)threshold_count(p->kind, p->depth), (int)row_x_pitch(p->C, bulk)};
  auto kernel = where_bytes(p->depth) == 2
                    ? (bulk ? rows_x_gradient_kernel<unsigned short, true> : rows_x_gradient_kernel<unsigned short, false>)
                    : (bulk ? rows_x_gradient_kernel<uint32_t, true> : rows_x_gradient_kernel<uint32_t, false>);
  HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
  kernel<<<(unsigned)((p->B + kXRows - 1) / kXRows), kXThreads, row_x_smem(p->C), stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

}  // namespace ht
