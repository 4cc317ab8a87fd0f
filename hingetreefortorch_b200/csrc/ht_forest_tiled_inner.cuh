// Shared-memory tile kernel for the forest forward on inputs with inner positions (x [B, C, K...]): the decomposition of
// ht_forest_tiled.cu, with samples that are (row, position) pairs.  Trees and ferns are compiled in files of their own.
#pragma once

#include "ht_eval_records.cuh"
#include "ht_forest_tile_plan.cuh"

#include <type_traits>

namespace ht {
namespace tile {

// One output per leaf, its weights in the records, four trees per warp.  (The kernel below in its place took 4 to 10 % longer.)
template <int KIND, int DEPTH, typename OrdT>
__global__ void __launch_bounds__(kThreads, 1) forest_forward_tiled_inner_one_kernel(const __grid_constant__ TiledArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr RecordLayout lay =
      record_layout(KIND, DEPTH, (uint32_t)sizeof(OrdT), true, paired_ordinals(KIND, DEPTH, (uint32_t)sizeof(OrdT)));
  const int S = a.S, G = a.G, C = a.C;
  float *xs = reinterpret_cast<float *>(smem);
  unsigned char *params = smem + (size_t)C * S * 4;
  uint64_t *full = reinterpret_cast<uint64_t *>(params + 2 * (size_t)G * lay.bytes);
  uint32_t *finished = reinterpret_cast<uint32_t *>(full + 2);

  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int groups_of_samples = S >> 5;
  const int sample_group = warp % groups_of_samples;
  const int slot = warp / groups_of_samples;
  const int64_t samples = a.B * a.K;
  const int64_t sample0 = (int64_t)blockIdx.x * S;
  const int all_groups = (int)((a.T + G - 1) / G);
  const int groups_per_cta = (all_groups + (int)gridDim.y - 1) / (int)gridDim.y;
  const int group0 = (int)blockIdx.y * groups_per_cta;
  const int num_groups = max(0, min(groups_per_cta, all_groups - group0));
  const uint32_t params_addr = smem_addr(params);

  auto issue = [&](int it) {
    const int64_t first_tree = (int64_t)(group0 + it) * G;
    const int64_t count = min((int64_t)G, a.T - first_tree);
    const uint32_t bytes = (uint32_t)(count * lay.bytes);
    uint64_t *bar = &full[it & 1];
    mbar_expect_tx(bar, bytes);
    bulk_load(params_addr + (uint32_t)(it & 1) * (uint32_t)G * lay.bytes, a.records + first_tree * lay.bytes, bytes, bar);
  };
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    finished[0] = 0;
    finished[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (num_groups > 0) issue(0);
    if (num_groups > 1) issue(1);
  }

  // features of the tile's samples, feature-major; consecutive samples are consecutive positions.
  // A thread stages the features c0, c0 + step, ... of one sample, or of 4 consecutive positions
  // at a time when the rows allow 16-byte loads (S divides the thread count; a tile starts on a
  // multiple of S, so 4 positions never straddle a row when 4 divides K)
  if ((a.K & 3) == 0) {
    const int quads = S >> 2, t = (tid % quads) * 4, c_step = kThreads / quads;
    const int64_t sample = sample0 + t;
    const bool inside = sample < samples;  // then sample + 3 < samples as well
    const int64_t row = inside ? sample / a.K : 0, k = inside ? sample - row * a.K : 0;
    const float *src = a.x + row * C * a.K + k;
#pragma unroll 4
    for (int c = tid / quads; c < C; c += c_step) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (inside) v = __ldg(reinterpret_cast<const float4 *>(src + (int64_t)c * a.K));
      *reinterpret_cast<float4 *>(xs + c * S + t) = v;
    }
  } else {
    const int t = tid % S, c_step = kThreads / S;
    const int64_t sample = sample0 + t;
    const bool inside = sample < samples;
    const int64_t row = inside ? sample / a.K : 0, k = inside ? sample - row * a.K : 0;
    const float *src = a.x + row * C * a.K + k;
#pragma unroll 8
    for (int c = tid / S; c < C; c += c_step) xs[c * S + t] = inside ? __ldg(src + (int64_t)c * a.K) : 0.0f;
  }
  __syncthreads();

  const int64_t my_sample = sample0 + sample_group * 32 + lane;
  const bool valid = my_sample < samples;
  const int64_t my_row = valid ? my_sample / a.K : 0, my_k = valid ? my_sample - my_row * a.K : 0;
  float *my_out = a.out + my_row * a.T * a.K + my_k;  // tree j of this sample: + j * K
  const uint32_t xl_addr = smem_addr(xs + sample_group * 32 + lane);
  const uint32_t x_stride = (uint32_t)S * 4u;
  const int t_first = slot * 4;
  bool poisoned = false;

  for (int it = 0; it < num_groups; ++it) {
    const int group = group0 + it;
    if (!poisoned && !mbar_wait(&full[it & 1], (uint32_t)((it >> 1) & 1))) {
      poisoned = true;
      if (a.status_word != nullptr) atomicOr(a.status_word, HT_FLAG_PIPELINE_TIMEOUT);
    }
    const int in_group = (int)min((int64_t)G, a.T - (int64_t)group * G);
    const uint32_t base_addr = params_addr + (uint32_t)(it & 1) * (uint32_t)G * lay.bytes;
    float result[4] = {0.f, 0.f, 0.f, 0.f};
    if (t_first < in_group && !poisoned) {
      uint32_t rec[4], unused[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) rec[u] = base_addr + (uint32_t)min(t_first + u, in_group - 1) * lay.bytes;
      walk<KIND, DEPTH, OrdT, 4, true>(rec, xl_addr, x_stride, result, unused);
    }
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();
      const uint32_t before = atomicAdd(&finished[it & 1], 1u);
      if (before == kWarps - 1) {
        atomicExch(&finished[it & 1], 0u);
        __threadfence_block();
        if (it + 2 < num_groups) issue(it + 2);
      }
    }
    if (valid) {
      float *dst = my_out + ((int64_t)group * G + t_first) * a.K;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (t_first + u < in_group) dst[(int64_t)u * a.K] = result[u];
    }
  }
}

// Everything else.  The weights are in the records (of a.record_bytes), or are read from global
// memory.  Up to four outputs per leaf are written by their evaluation's lane; more, which are 32 * M consecutive numbers for the
// warp's 32 evaluations of a tree where the positions stay in one row, are dealt out to the lanes, `width` at a time.  SAVE: the traversal goes to the evaluation records, or to the paths of
// several outputs per leaf, and with out == nullptr nothing else.
// Bound by the walk (issue slots and the shared memory's wavefronts, as in ht_forest_tiled.cu) and, from five outputs on, by dealing
// them out.  Several outputs per leaf took a thread per evaluation before, whose warps wait for gathers on as many cache lines as
// a level has vertices: 135 x 152 x 2500, 527 trees of depth 3, 3 outputs 1952 -> 643 us; 455 x 70 x 2025, 291 of depth 10, 2
// outputs 5024 -> 2197.  With the weights in global memory, and outputs of two to four dealt out as well, the first took 1389.
template <int KIND, int DEPTH, typename OrdT, bool WREC, bool SAVE>
__global__ void __launch_bounds__(kThreads, 1) forest_forward_tiled_inner_kernel(const __grid_constant__ TiledArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr RecordLayout lay =
      record_layout(KIND, DEPTH, (uint32_t)sizeof(OrdT), false, paired_ordinals(KIND, DEPTH, (uint32_t)sizeof(OrdT)));
  constexpr uint32_t kL = 1u << DEPTH;
  const int S = a.S, G = a.G, C = a.C, per_warp = a.per_warp;
  const uint32_t record_bytes = a.record_bytes;
  float *xs = reinterpret_cast<float *>(smem);
  unsigned char *params = smem + (size_t)C * S * 4;
  uint64_t *full = reinterpret_cast<uint64_t *>(params + 2 * (size_t)G * record_bytes);
  uint32_t *finished = reinterpret_cast<uint32_t *>(full + 2);

  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int groups_of_samples = S >> 5;
  const int sample_group = warp % groups_of_samples;
  const int slot = warp / groups_of_samples;
  const int64_t samples = a.B * a.K;
  const int64_t sample0 = (int64_t)blockIdx.x * S;
  const int all_groups = (int)((a.T + G - 1) / G);
  const int groups_per_cta = (all_groups + (int)gridDim.y - 1) / (int)gridDim.y;
  const int group0 = (int)blockIdx.y * groups_per_cta;
  const int num_groups = max(0, min(groups_per_cta, all_groups - group0));
  const uint32_t params_addr = smem_addr(params);

  auto issue = [&](int it) {
    const int64_t first_tree = (int64_t)(group0 + it) * G;
    const int64_t count = min((int64_t)G, a.T - first_tree);
    const uint32_t bytes = (uint32_t)(count * record_bytes);
    uint64_t *bar = &full[it & 1];
    mbar_expect_tx(bar, bytes);
    bulk_load(params_addr + (uint32_t)(it & 1) * (uint32_t)G * record_bytes, a.records + first_tree * record_bytes, bytes, bar);
  };
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    finished[0] = 0;
    finished[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (num_groups > 0) issue(0);
    if (num_groups > 1) issue(1);
  }

  // features of the tile's samples, feature-major; consecutive samples are consecutive positions.
  // A thread stages the features c0, c0 + step, ... of one sample, or of 4 consecutive positions
  // at a time when the rows allow 16-byte loads (S divides the thread count; a tile starts on a
  // multiple of S, so 4 positions never straddle a row when 4 divides K)
  if ((a.K & 3) == 0) {
    const int quads = S >> 2, t = (tid % quads) * 4, c_step = kThreads / quads;
    const int64_t sample = sample0 + t;
    const bool inside = sample < samples;  // then sample + 3 < samples as well
    const int64_t row = inside ? sample / a.K : 0, k = inside ? sample - row * a.K : 0;
    const float *src = a.x + row * C * a.K + k;
#pragma unroll 4
    for (int c = tid / quads; c < C; c += c_step) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (inside) v = __ldg(reinterpret_cast<const float4 *>(src + (int64_t)c * a.K));
      *reinterpret_cast<float4 *>(xs + c * S + t) = v;
    }
  } else {
    const int t = tid % S, c_step = kThreads / S;
    const int64_t sample = sample0 + t;
    const bool inside = sample < samples;
    const int64_t row = inside ? sample / a.K : 0, k = inside ? sample - row * a.K : 0;
    const float *src = a.x + row * C * a.K + k;
#pragma unroll 8
    for (int c = tid / S; c < C; c += c_step) xs[c * S + t] = inside ? __ldg(src + (int64_t)c * a.K) : 0.0f;
  }
  __syncthreads();

  const int64_t first_sample = sample0 + sample_group * 32, my_sample = first_sample + lane;
  const bool valid = my_sample < samples;
  const int64_t my_row = valid ? my_sample / a.K : 0, my_k = valid ? my_sample - my_row * a.K : 0;
  const uint32_t xl_addr = smem_addr(xs + sample_group * 32 + lane);
  const uint32_t x_stride = (uint32_t)S * 4u;
  const int t_first = slot * per_warp;
  bool poisoned = false;
  // outputs of tree j of this sample: my_out[j * K * M]
  float *my_out = a.out + (my_row * a.T * a.K + my_k) * a.M;
  // several: the warp's run of outputs starts with its first sample's; what lies behind the end of a row is (T - 1) * K samples on
  const int here = (int)max((int64_t)0, min((int64_t)32, samples - first_sample));
  const uint32_t k0 = (uint32_t)__shfl_sync(0xffffffffu, (long long)my_k, 0);
  float *warp_out = a.out + (__shfl_sync(0xffffffffu, (long long)my_row, 0) * a.T * a.K + k0) * a.M;
  const bool one_row = k0 + 32u <= (uint32_t)a.K;
  const int64_t row_step = (a.T - 1) * a.K * a.M;

  // This warp no longer reads parameter buffer (it & 1).  The last warp to say so refills it.
  auto done_with_buffer = [&](int it) {
    __syncwarp();
    if (lane == 0) {
      uint32_t before;  // wraps to zero with the last warp: acquire / release order the warps' reads before the refill
      asm volatile("atom.acq_rel.cta.shared::cta.inc.u32 %0, [%1], %2;"
                   : "=r"(before)
                   : "r"(smem_addr(&finished[it & 1])), "r"((uint32_t)kWarps - 1u)
                   : "memory");
      if (before == (uint32_t)kWarps - 1u && it + 2 < num_groups) issue(it + 2);
    }
  };
  // V weights of the leaf at the end of `path` (of output `first` on) of the warp's u-th tree
  auto weights_at = [&](auto vector, int64_t tree, uint32_t record, uint32_t path, uint32_t first) {
    constexpr int V = decltype(vector)::value;
    Vec<float, V> r = {};
    if constexpr (WREC) {
      if (poisoned) return r;  // a buffer that never arrived is not read
      const uint32_t at = record + lay.w + 4u * ((path - kL) * (uint32_t)a.M + first);
      if constexpr (V == 4) {
        const uint4 q = lds_b128(at);
        r = *reinterpret_cast<const Vec<float, 4> *>(&q);
      } else {
#pragma unroll
        for (int v = 0; v < V; ++v) r.v[v] = lds_f32(at + 4u * v);
      }
    } else {
      r = load_vec<float, V>(a.w + ((tree << DEPTH) + (__brev(path - kL) >> (32 - DEPTH))) * (int64_t)a.M + first);
    }
    return r;
  };
  auto write_own = [&](auto outputs, int64_t tree0, int in_group, const float (&size)[4], const uint32_t (&path)[4], uint32_t records) {
    constexpr int M = decltype(outputs)::value, V = M == 3 ? 1 : M;
    float *dst = my_out + tree0 * a.K * M;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (u >= per_warp || t_first + u >= in_group) break;
      if (valid) {
#pragma unroll
        for (int m = 0; m < M; m += V) {
          Vec<float, V> r = weights_at(std::integral_constant<int, V>{}, tree0 + u, records + (uint32_t)(t_first + u) * record_bytes, path[u], m);
#pragma unroll
          for (int v = 0; v < V; ++v) r.v[v] = __fmul_rn(size[u], r.v[v]);
          *reinterpret_cast<Vec<float, V> *>(dst + (int64_t)u * a.K * M + m) = r;
        }
      }
    }
  };
  auto deal_out = [&](auto vector, int64_t tree0, int in_group, const float (&size)[4], const uint32_t (&path)[4], uint32_t records) {
    constexpr int V = decltype(vector)::value;
    const uint32_t M = (uint32_t)a.M, pieces = (uint32_t)here * M / V;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (u >= per_warp || t_first + u >= in_group) break;
      float *dst = warp_out + (tree0 + u) * a.K * M;
#pragma unroll 4
      for (uint32_t t = (uint32_t)lane; t - (uint32_t)lane < pieces; t += 32) {
        const uint32_t element = t * V, owner = min(a.by_M.quotient(element), 31u);
        const float scale = __shfl_sync(0xffffffffu, size[u], (int)owner);
        const uint32_t whose = __shfl_sync(0xffffffffu, path[u], (int)owner);
        if (t < pieces) {
          Vec<float, V> r = weights_at(vector, tree0 + u, records + (uint32_t)(t_first + u) * record_bytes, whose, element - owner * M);
#pragma unroll
          for (int v = 0; v < V; ++v) r.v[v] = __fmul_rn(scale, r.v[v]);
          float *to = dst + element;
          if (!one_row) to += (int64_t)a.by_K.quotient(k0 + owner) * row_step;
          *reinterpret_cast<Vec<float, V> *>(to) = r;
        }
      }
    }
  };

  for (int it = 0; it < num_groups; ++it) {
    const int group = group0 + it;
    if (!poisoned && !mbar_wait(&full[it & 1], (uint32_t)((it >> 1) & 1))) {
      poisoned = true;
      if (a.status_word != nullptr) atomicOr(a.status_word, HT_FLAG_PIPELINE_TIMEOUT);
    }
    const int in_group = (int)min((int64_t)G, a.T - (int64_t)group * G);
    const uint32_t base_addr = params_addr + (uint32_t)(it & 1) * (uint32_t)G * record_bytes;
    float result[4] = {0.f, 0.f, 0.f, 0.f};  // after a lost copy: zeros, and the paths of a zero margin at the root
    uint32_t path[4] = {kL, kL, kL, kL};
    [[maybe_unused]] float margin[4] = {0.f, 0.f, 0.f, 0.f};
    [[maybe_unused]] uint32_t vertex[4] = {1u, 1u, 1u, 1u};
    if (t_first < in_group && !poisoned) {
      // trees beyond the end of a short last group repeat the last valid one (results unused)
      auto walk_trees = [&](auto trees) {
        constexpr int n = decltype(trees)::value;
        uint32_t rec[n], p[n];
        float r[n];
#pragma unroll
        for (int u = 0; u < n; ++u) rec[u] = base_addr + (uint32_t)min(t_first + u, in_group - 1) * record_bytes;
        if constexpr (SAVE) {
          Walked found[n];
          walk_full<KIND, DEPTH, OrdT, n, lay.paired>(rec, xl_addr, x_stride, found);
#pragma unroll
          for (int u = 0; u < n; ++u) {
            margin[u] = found[u].nm;
            vertex[u] = found[u].v;
            r[u] = fabsf(found[u].nm);
            p[u] = found[u].path;
          }
        } else {
          walk<KIND, DEPTH, OrdT, n, false>(rec, xl_addr, x_stride, r, p);
        }
#pragma unroll
        for (int u = 0; u < n; ++u) {
          result[u] = r[u];
          path[u] = p[u];
        }
      };
      if (per_warp == 4)
        walk_trees(std::integral_constant<int, 4>{});
      else if (per_warp == 2)
        walk_trees(std::integral_constant<int, 2>{});
      else
        walk_trees(std::integral_constant<int, 1>{});
    }
    const int64_t tree0 = (int64_t)group * G + t_first;
    if constexpr (SAVE) {
      using WhereT = typename std::conditional<(DEPTH <= 8), unsigned short, uint32_t>::type;
      const int64_t at = record_index(my_sample, tree0, a.T);
      if (valid) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u < per_warp && t_first + u < in_group) {
            __stcs(a.save_margin + at + u * kRecordBlock, margin[u]);
            store_where<WhereT>(a.save_where, at + u * kRecordBlock, vertex[u], __brev(path[u] - kL) >> (32 - DEPTH));
          }
      }
    }
    if (!SAVE || a.out != nullptr) {
      if (a.M == 1) {
        write_own(std::integral_constant<int, 1>{}, tree0, in_group, result, path, base_addr);
      } else if (a.M == 2 && a.width == 2)
        write_own(std::integral_constant<int, 2>{}, tree0, in_group, result, path, base_addr);
      else if (a.M == 3)
        write_own(std::integral_constant<int, 3>{}, tree0, in_group, result, path, base_addr);
      else if (a.M == 4 && a.width == 4)
        write_own(std::integral_constant<int, 4>{}, tree0, in_group, result, path, base_addr);
      else if (a.width == 4)
        deal_out(std::integral_constant<int, 4>{}, tree0, in_group, result, path, base_addr);
      else if (a.width == 2)
        deal_out(std::integral_constant<int, 2>{}, tree0, in_group, result, path, base_addr);
      else
        deal_out(std::integral_constant<int, 1>{}, tree0, in_group, result, path, base_addr);
    }
    done_with_buffer(it);
  }
}

template <int KIND, int DEPTH, typename OrdT>
int launch_inner_form(const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream) {
  if (plan.weights && a.M == 1) return launch_one(forest_forward_tiled_inner_one_kernel<KIND, DEPTH, OrdT>, plan, a, grid, stream);
  if (a.save_margin != nullptr)
    return plan.weights ? launch_one(forest_forward_tiled_inner_kernel<KIND, DEPTH, OrdT, true, true>, plan, a, grid, stream)
                        : launch_one(forest_forward_tiled_inner_kernel<KIND, DEPTH, OrdT, false, true>, plan, a, grid, stream);
  return plan.weights ? launch_one(forest_forward_tiled_inner_kernel<KIND, DEPTH, OrdT, true, false>, plan, a, grid, stream)
                      : launch_one(forest_forward_tiled_inner_kernel<KIND, DEPTH, OrdT, false, false>, plan, a, grid, stream);
}

template <int KIND, typename OrdT>
int launch_inner_depth(int depth, const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream) {
  switch (depth) {
#define HT_DEPTH_CASE(D) \
  case D:                \
    return launch_inner_form<KIND, D, OrdT>(plan, a, grid, stream);
    HT_DEPTH_CASE(1)
    HT_DEPTH_CASE(2)
    HT_DEPTH_CASE(3)
    HT_DEPTH_CASE(4)
    HT_DEPTH_CASE(5)
    HT_DEPTH_CASE(6)
    HT_DEPTH_CASE(7)
    HT_DEPTH_CASE(8)
    HT_DEPTH_CASE(9)
    HT_DEPTH_CASE(10)
    HT_DEPTH_CASE(11)
    HT_DEPTH_CASE(12)
#undef HT_DEPTH_CASE
    default:
      return HT_ERR_UNSUPPORTED;
  }
}

template <int KIND>
int launch_inner_kind(int depth, const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream) {
  return plan.ord_bytes == 1 ? launch_inner_depth<KIND, uint8_t>(depth, plan, a, grid, stream)
                             : launch_inner_depth<KIND, uint16_t>(depth, plan, a, grid, stream);
}

}  // namespace tile
}  // namespace ht
