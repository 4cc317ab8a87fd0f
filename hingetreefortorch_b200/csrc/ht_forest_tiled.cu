// Shared-memory tile kernels for the forest forward.
//
// forest_forward_tiled_kernel: tabular input (K == 1), one or several outputs per leaf.  Inputs with inner positions:
// ht_forest_tiled_inner.cu.
//
// Work decomposition (one CTA of 1024 threads per tile, sized for one CTA per SM):
//   * a CTA owns S consecutive samples and walks ALL trees (or, when the batch alone gives too
//     few tiles for the machine, its share of the tree groups), so every input element is read
//     from HBM once;
//   * the samples' features sit in shared memory feature-major, xs[c][s]: lane l of a warp
//     always reads bank l whatever feature its current vertex tests, so the data gather never
//     conflicts although the 32 lanes are at 32 different vertices;
//   * a warp is (sample group, slot): S/32 sample groups of 32 samples, 32/(S/32) slots.  Trees
//     are processed in groups of G; inside a group slot q owns G/slots consecutive trees and
//     walks them all at once (independent dependent-load chains hide shared-memory latency);
//   * tree parameters arrive as per-tree records {root and its two children for a single
//     broadcast load, thresholds, feature indices, leaf weights in path order}, written once per
//     call by a small repack kernel, and are streamed into shared memory with 1-D bulk async
//     copies (cp.async.bulk, the TMA engine) completing on an mbarrier.  Two buffers; the last
//     warp to finish a group issues the copy that refills its buffer, so no warp ever waits for
//     another in order to keep the pipeline fed.  One-byte feature indices are stored as words
//     {own, left child's, right child's} of the even-level vertices, one load for two levels;
//   * tabular results of a group are transposed through a per-sample-group staging area (named
//     barriers over the 4..32 warps of the sample group only) and leave as row segments; with
//     inner positions consecutive samples are consecutive positions of the same output row, so
//     the results leave straight from registers.
//
// Only the smallest |margin| matters in the forward, so the minimum is tracked on absolute
// values.  CUDA's fminf ignores a NaN operand; the reference keeps a NaN only when the root
// margin is NaN, which is patched after the loop.
//
// The vertex index is kept 1-based (root 1, children 2v and 2v+1) so that one funnel shift
// appends the branch bit.  The bit is the sign of (threshold - feature): it is set exactly
// when the margin (feature - threshold) is positive, given that records hold +0 for a -0
// threshold and that an add producing NaN produces the canonical positive NaN (so NaN margins
// go left, as `margin > 0` does in the reference).  |threshold - feature| equals
// |feature - threshold| bit for bit.
#include "ht_eval_records.cuh"
#include "ht_forest_multi.cuh"
#include "ht_forest_tile_plan.cuh"
#include "ht_forest_tiled.cuh"
#include "ht_tile_common.cuh"
#include "ht_tma.cuh"

#include <algorithm>
#include <type_traits>

namespace ht {

using namespace tile;

namespace {


// Shared-memory layout of forest_forward_tiled_kernel, from a 1024-byte boundary: the results area (a
// staging row per sample with one output per leaf — boxes the TMA engine can store —, or the warps'
// (margin, leaf) pairs), the feature tile, two parameter buffers, the barriers.
__host__ __device__ inline size_t results_bytes(bool one_output, int S, int G) {
  const size_t bytes = one_output ? (size_t)S * (G + 1) * 4 : (size_t)kWarps * 32 * 4 * 8;
  return (bytes + 1023) & ~(size_t)1023;
}

bool make_plan(const ht_forest_problem *p, TilePlan &plan) {
  if (p->K != 1 || p->M < 1 || p->M > 64) return false;
  if (p->C > 65536 || p->depth > 12) return false;
  if (p->B * p->T < 32 * 1024) return false;  // too small to fill the machine with sample tiles
  plan.ord_bytes = p->C <= 256 ? 1 : 2;
  // One output per leaf: weights in the records first; where those do not fit beside a tile (ferns of depth 10 on 579 features:
  // 121336 x 241 forwards 297 us, 444 with a thread per evaluation) they are read from global memory like several outputs'.
  for (int weights = p->M == 1 ? 1 : 0; weights >= 0; --weights) {
    plan.weights = weights != 0;
    plan.rec = record_layout(p->kind, p->depth, (uint32_t)plan.ord_bytes, plan.weights,
                             paired_ordinals(p->kind, p->depth, (uint32_t)plan.ord_bytes));
    for (int S = 256; S >= 32; S >>= 1) {
      const int slots = kWarps / (S / 32);
      for (int per_warp = 4; per_warp >= 1; per_warp >>= 1) {
        const int G = slots * per_warp;
        plan.S = S;
        plan.G = G;
        plan.per_warp = per_warp;
        // results: a staging row per sample (one output per leaf), or the warps' (margin, leaf) pairs
        plan.smem = 1024 + results_bytes(plan.weights, S, G) + (size_t)p->C * S * 4 + 2 * (size_t)G * plan.rec.bytes + 64;
        // without the weights only for batches that fill the machine with whole tiles: 3262 x 684 forwards took 55 us with 51
        // tiles shared out, 44 with a thread per evaluation
        if (plan.smem <= kSmemBudget) return plan.weights || p->M > 1 || p->B >= (int64_t)148 * S;
      }
    }
  }
  return false;
}

template <int KIND, int DEPTH, typename OrdT, bool WREC, bool SAVE = false>
__global__ void __launch_bounds__(kThreads, 1) forest_forward_tiled_kernel(const __grid_constant__ TiledArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr RecordLayout lay =
      record_layout(KIND, DEPTH, (uint32_t)sizeof(OrdT), WREC, paired_ordinals(KIND, DEPTH, (uint32_t)sizeof(OrdT)));
  const int S = a.S, G = a.G, C = a.C;
  const int M = WREC ? 1 : a.M;
  // staging row of one sample (one output per leaf): G trees, padded against bank conflicts; dense when
  // the area holds the TMA boxes, so that a sample group's rows stay inside its own box
  const int row_floats = a.tma_store != 0 ? G : G + 1;
  unsigned char *base = smem + ((1024u - (smem_addr(smem) & 1023u)) & 1023u);
  float *outs = reinterpret_cast<float *>(base);
  float *xs = reinterpret_cast<float *>(base + results_bytes(WREC, S, G));
  unsigned char *params = reinterpret_cast<unsigned char *>(xs + (size_t)C * S);
  uint64_t *full = reinterpret_cast<uint64_t *>(params + 2 * (size_t)G * lay.bytes);  // [2] copy landed
  uint32_t *finished = reinterpret_cast<uint32_t *>(full + 2);                         // [2] warps done with a buffer

  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int groups_of_samples = S >> 5;
  const int slots = kWarps / groups_of_samples;
  const int sample_group = warp % groups_of_samples;
  const int slot = warp / groups_of_samples;
  const int64_t row0 = (int64_t)blockIdx.x * S;
  // blockIdx.y splits the tree groups among CTAs when there are too few sample tiles to fill the
  // machine; this CTA walks groups [group0, group0 + num_groups), `it` counts them from 0
  const int all_groups = (int)((a.T + G - 1) / G);
  const int groups_per_cta = (all_groups + (int)gridDim.y - 1) / (int)gridDim.y;
  const int group0 = (int)blockIdx.y * groups_per_cta;
  const int num_groups = max(0, min(groups_per_cta, all_groups - group0));
  const uint32_t params_addr = smem_addr(params);

  const int per_warp = a.per_warp;
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

  stage_rows(xs, a.x, row0, a.B, C, S, tid);
  __syncthreads();  // features staged; barrier initialisation visible

  const uint32_t xl_addr = smem_addr(xs + sample_group * 32 + lane);
  const uint32_t x_stride = (uint32_t)S * 4u;
  float *stage = outs + (size_t)sample_group * 32 * row_floats;  // this sample group's [32][G*M + 1] staging rows
  const int group_threads = slots * 32;
  const int tid_in_group = slot * 32 + lane;
  constexpr uint32_t kL = 1u << DEPTH;
  bool poisoned = false;  // a bounded wait ran out: keep the barriers matched, stop waiting
  // Output of a full group when its 32 x (G*M/4) 16-byte pieces are one per thread of the sample
  // group (the usual case): which piece is this thread's, worked out once
  const int full_groups = (int)(a.T / G), tail_trees = (int)(a.T - (int64_t)full_groups * G);  // a.T < 2^31 * G
  const int full_quads = (G * M) >> 2;
  const int64_t row_pitch = a.T * M;
  const bool one_piece = ((G * M) & 3) == 0 && (row_pitch & 3) == 0 && 32 * full_quads == group_threads;
  const int piece_row = one_piece ? tid_in_group / full_quads : 0;
  const int piece_quad = one_piece ? tid_in_group - piece_row * full_quads : 0;
  const int64_t piece_sample = row0 + sample_group * 32 + piece_row;
  float *piece_dst = a.out + piece_sample * row_pitch + 4 * piece_quad;
  const float *piece_src = stage + piece_row * row_floats + 4 * piece_quad;
  // Full groups with 4 trees per warp and the weights in the records take a body without the
  // bookkeeping of short groups, other tree counts and several outputs per leaf.
  const bool streamlined = WREC && one_piece && per_warp == 4;
  const uint32_t warp_records = (uint32_t)(slot * per_warp) * lay.bytes;
  float *stage_mine = stage + lane * row_floats + slot * per_warp;
  // TMA form of the streamlined body: this sample group's box of 32 rows x G floats, and where this
  // lane's 4 results (chunk `slot` of row `lane`) sit in it
  const bool tma_store = streamlined && a.tma_store != 0;
  const bool store_issuer = tma_store && slot == 0 && lane == 0;
  const uint32_t box_addr = smem_addr(outs) + (uint32_t)sample_group * 32u * (uint32_t)G * 4u;
  const uint32_t box_mine = box_addr + (G == 16 ? tma::swizzled_offset<16>((uint32_t)lane, (uint32_t)slot)
                                                : tma::swizzled_offset<32>((uint32_t)lane, (uint32_t)slot));

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

  int it = 0;
  if (tma_store) {
    // The loop of the benchmark shapes, with nothing in it that the full groups of a forest with the
    // weights in its records do not need: one register addresses the warp's four consecutive records,
    // and the buffer goes back with one atomic (it wraps to zero with the last warp, which refills).
    const int fast = max(0, min(num_groups, full_groups - group0));
    for (; it < fast; ++it) {
      const uint32_t buffer = (uint32_t)(it & 1);
      if (!poisoned && !mbar_wait(&full[buffer], (uint32_t)((it >> 1) & 1))) {
        poisoned = true;
        if (a.status_word != nullptr) atomicOr(a.status_word, HT_FLAG_PIPELINE_TIMEOUT);
      }
      const uint32_t first_record = params_addr + buffer * (uint32_t)G * lay.bytes + warp_records;
      float result[4] = {0.f, 0.f, 0.f, 0.f};
      if constexpr (SAVE) {
        // the walk of the backward (signed margin, deciding vertex, path): the same |margin| * leaf weight leaves as
        // the result, and the traversal itself goes to the evaluation records, from registers (consecutive lanes
        // are consecutive samples: 128 and 64 contiguous bytes per tree)
        using WhereT = typename std::conditional<(DEPTH <= 8), unsigned short, uint32_t>::type;
        const int64_t sample = row0 + sample_group * 32 + lane;
        const int64_t at = record_index(sample, (int64_t)(group0 + it) * G + slot * 4, a.T);
        uint32_t rec[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) rec[u] = first_record + (uint32_t)u * lay.bytes;
        Walked wk[4];
        if (!poisoned) {
          walk_full<KIND, DEPTH, OrdT, 4, lay.paired>(rec, xl_addr, x_stride, wk);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            result[u] = __fmul_rn(fabsf(wk[u].nm), lds_f32(rec[u] + 4u * wk[u].path + (lay.w - 4u * (1u << DEPTH))));
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) wk[u] = Walked{0.0f, 1u, 1u << DEPTH};
        }
        if (sample < a.B) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            __stcs(a.save_margin + at + u * kRecordBlock, wk[u].nm);
            store_where<WhereT>(a.save_where, at + u * kRecordBlock, wk[u].v, __brev(wk[u].path - (1u << DEPTH)) >> (32 - DEPTH));
          }
        }
      } else {
        const uint32_t rec[4] = {first_record, 0u, 0u, 0u};
        uint32_t unused[4];
        if (!poisoned) walk<KIND, DEPTH, OrdT, 4, WREC, true>(rec, xl_addr, x_stride, result, unused);
      }
      done_with_buffer(it);
      if (store_issuer) tma::wait_stores_read();  // the previous box has been read out of the staging area
      named_barrier(1 + sample_group, group_threads);
      sts_b128(box_mine, result[0], result[1], result[2], result[3]);
      tma::fence_async_shared();
      named_barrier(1 + sample_group, group_threads);  // box complete and visible to the TMA engine
      if (store_issuer) {
        tma::store_2d(&a.out_map, box_addr, (group0 + it) * G, (int)(row0 + sample_group * 32));
        tma::commit_group();
      }
    }
  }
  for (; it < num_groups; ++it) {
    const int group = group0 + it;
    if (!poisoned && !mbar_wait(&full[it & 1], (uint32_t)((it >> 1) & 1))) {
      poisoned = true;
      if (a.status_word != nullptr) atomicOr(a.status_word, HT_FLAG_PIPELINE_TIMEOUT);
    }
    const int in_group = group < full_groups ? G : tail_trees;
    const uint32_t base_addr = params_addr + (uint32_t)(it & 1) * (uint32_t)G * lay.bytes;
    if (streamlined && in_group == G) {
      uint32_t rec[4], unused[4];
      float result[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int u = 0; u < 4; ++u) rec[u] = base_addr + warp_records + (uint32_t)u * lay.bytes;
      if (SAVE) {
        // the walk of the backward (signed margin, deciding vertex, path): the same |margin| * leaf weight
        // leaves as the result, and the traversal itself goes to the evaluation records, from registers
        // (consecutive lanes are consecutive samples: 128 and 64 contiguous bytes per tree)
        using WhereT = typename std::conditional<(DEPTH <= 8), unsigned short, uint32_t>::type;
        const int64_t sample = row0 + sample_group * 32 + lane;
        const int64_t at = record_index(sample, (int64_t)group * G + slot * 4, a.T);
        Walked wk[4];
        if (!poisoned) {
          walk_full<KIND, DEPTH, OrdT, 4, lay.paired>(rec, xl_addr, x_stride, wk);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            result[u] = __fmul_rn(fabsf(wk[u].nm), lds_f32(rec[u] + 4u * wk[u].path + (lay.w - 4u * (1u << DEPTH))));
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) wk[u] = Walked{0.0f, 1u, 1u << DEPTH};
        }
        if (sample < a.B) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            __stcs(a.save_margin + at + u * kRecordBlock, wk[u].nm);
            store_where<WhereT>(a.save_where, at + u * kRecordBlock, wk[u].v, __brev(wk[u].path - (1u << DEPTH)) >> (32 - DEPTH));
          }
        }
      } else if (!poisoned) {
        walk<KIND, DEPTH, OrdT, 4, WREC>(rec, xl_addr, x_stride, result, unused);  // a buffer that never arrived is not read
      }
      done_with_buffer(it);
      if (tma_store) {
        // The sample group's [32 samples x G trees] block goes to shared memory in the swizzled box layout
        // (a lane writes the 16 bytes of its own row: conflict free) and leaves as ONE tiled TMA store.
        if (store_issuer) tma::wait_stores_read();  // the previous box has been read out of the staging area
        named_barrier(1 + sample_group, group_threads);
        sts_b128(box_mine, result[0], result[1], result[2], result[3]);
        tma::fence_async_shared();
        named_barrier(1 + sample_group, group_threads);  // box complete and visible to the TMA engine
        if (store_issuer) {
          tma::store_2d(&a.out_map, box_addr, group * G, (int)(row0 + sample_group * 32));
          tma::commit_group();
        }
        continue;
      }
      named_barrier(1 + sample_group, group_threads);  // previous group's rows have left the staging area
#pragma unroll
      for (int u = 0; u < 4; ++u) stage_mine[u] = result[u];
      named_barrier(1 + sample_group, group_threads);  // staging area complete
      if (piece_sample < a.B)
        *reinterpret_cast<float4 *>(piece_dst + (int64_t)group * G) =
            make_float4(piece_src[0], piece_src[1], piece_src[2], piece_src[3]);
      continue;
    }
    if (store_issuer) tma::wait_stores_read();  // the body below writes the staging area with plain stores
    const int t_first = slot * per_warp;  // this warp's consecutive trees inside the group
    float result[4] = {0.f, 0.f, 0.f, 0.f};
    uint32_t path[4] = {kL, kL, kL, kL};
    // SAVE with several outputs per leaf; after a lost copy the paths are those of a zero margin at the root
    [[maybe_unused]] Walked wk[4] = {{0.f, 1u, kL}, {0.f, 1u, kL}, {0.f, 1u, kL}, {0.f, 1u, kL}};
    if (t_first < in_group && !poisoned) {  // after a lost copy the buffer is not read: zeros leave instead
      // trees beyond the end of a short last group repeat the last valid one (results unused)
      auto walk_trees = [&](auto trees) {
        constexpr int n = decltype(trees)::value;
        uint32_t rec[n], p[n];
        float r[n];
#pragma unroll
        for (int u = 0; u < n; ++u)
          rec[u] = base_addr + (uint32_t)(in_group == G ? t_first + u : min(t_first + u, in_group - 1)) * lay.bytes;
        if constexpr (SAVE && !WREC) {
          Walked found[n];
          walk_full<KIND, DEPTH, OrdT, n, lay.paired>(rec, xl_addr, x_stride, found);
#pragma unroll
          for (int u = 0; u < n; ++u) {
            wk[u] = found[u];
            r[u] = fabsf(found[u].nm);
            p[u] = found[u].path;
          }
        } else {
          walk<KIND, DEPTH, OrdT, n, WREC>(rec, xl_addr, x_stride, r, p);
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
    done_with_buffer(it);
    if constexpr (SAVE && !WREC) {
      using WhereT = typename std::conditional<(DEPTH <= 8), unsigned short, uint32_t>::type;
      const int64_t sample = row0 + sample_group * 32 + lane;
      const int64_t at = record_index(sample, (int64_t)group * G + t_first, a.T);
      if (sample < a.B) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u < per_warp && t_first + u < in_group) {
            a.save_margin[at + u * kRecordBlock] = wk[u].nm;
            store_where<WhereT>(a.save_where, at + u * kRecordBlock, wk[u].v, __brev(wk[u].path - kL) >> (32 - DEPTH));
          }
      }
    }

    const int64_t col0 = (int64_t)group * G;
    if (!WREC) {
      // Several outputs per leaf: out[i, j, :] = |margin| * w[j, leaf, :], and the warp's trees
      // j .. j + n - 1 of one sample are n * M consecutive outputs.  Every lane leaves its (|margin|, leaf)
      // pairs in the warp's corner of shared memory; then the warp writes the 32 samples' runs one after
      // another, lane by lane along a run, reading the weight rows from global memory (L2 resident)
      // the same way: loads and stores are contiguous whatever leaves the samples reached.
      const int trees_here = min(per_warp, in_group - t_first);  // <= 0: nothing for this warp in a short group
      float2 *pairs = reinterpret_cast<float2 *>(outs) + (size_t)warp * 32 * 4;
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 4; ++u)
        pairs[lane * 4 + u] = make_float2(result[u], __uint_as_float(__brev(path[u] - kL) >> (32 - DEPTH)));
      __syncwarp();
      if (trees_here > 0 && (!SAVE || a.out != nullptr)) {
        const int64_t first_row = row0 + sample_group * 32;
        const int rows_here = (int)max((int64_t)0, min((int64_t)32, a.B - first_row));
        const float *w_first = a.w + (col0 + t_first) * (int64_t)kL * M;
        float *dst = a.out + first_row * row_pitch + (col0 + t_first) * M;
        // The outputs of all 32 samples, V at a time, are dealt out to the lanes one after another: a run of one or two trees
        // with few outputs would leave most lanes idle (10007 x 257 trees, 3 outputs, one tree per warp: 1055 instructions per
        // evaluation of 32 samples with a pass per sample: 118 us, dealt out 77).
        auto write_out = [&](auto vector) {
          constexpr int V = decltype(vector)::value;
          const uint32_t pieces = (uint32_t)(trees_here * M) / V, total = (uint32_t)rows_here * pieces;
          const bool whole = trees_here == per_warp;
#pragma unroll 4
          for (uint32_t e = (uint32_t)lane; e < total; e += 32) {
            const uint32_t sample = whole ? a.by_pieces.quotient(e) : e / pieces, element = (e - sample * pieces) * V;
            const uint32_t u = a.by_M.quotient(element);
            const float2 pr = pairs[sample * 4 + u];
            Vec<float, V> v = load_vec<float, V>(w_first + ((u << DEPTH) + __float_as_uint(pr.y)) * (uint32_t)M + (element - u * (uint32_t)M));
#pragma unroll
            for (int k = 0; k < V; ++k) v.v[k] = pr.x * v.v[k];
            *reinterpret_cast<Vec<float, V> *>(dst + (int64_t)sample * row_pitch + element) = v;
          }
        };
        if (a.width == 4) write_out(std::integral_constant<int, 4>{});
        else if (a.width == 2) write_out(std::integral_constant<int, 2>{});
        else write_out(std::integral_constant<int, 1>{});
      }
      continue;
    }
    named_barrier(1 + sample_group, group_threads);  // previous group's rows have left the staging area
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (u < per_warp && t_first + u < in_group) stage[lane * row_floats + t_first + u] = result[u];
    named_barrier(1 + sample_group, group_threads);  // staging area complete

    // the sample group's warps write its [32 x in_group*M] block of results as row segments
    const int64_t row_base = row0 + sample_group * 32;
    const int width = in_group * M;
    const int64_t first_col = col0 * M;
    if (one_piece && in_group == G) {
      if (piece_sample < a.B)
        *reinterpret_cast<float4 *>(piece_dst + first_col) = make_float4(piece_src[0], piece_src[1], piece_src[2], piece_src[3]);
    } else if ((row_pitch & 3) == 0 && (first_col & 3) == 0 && (width & 3) == 0) {
      const int quads = width >> 2;
      for (int idx = tid_in_group; idx < 32 * quads; idx += group_threads) {
        const int s = idx / quads, q = idx - s * quads;
        if (row_base + s < a.B) {
          const float *src = stage + s * row_floats + 4 * q;
          *reinterpret_cast<float4 *>(a.out + (row_base + s) * row_pitch + first_col + 4 * q) =
              make_float4(src[0], src[1], src[2], src[3]);
        }
      }
    } else {
      for (int idx = tid_in_group; idx < 32 * width; idx += group_threads) {
        const int s = idx / width, t = idx - s * width;
        if (row_base + s < a.B) a.out[(row_base + s) * row_pitch + first_col + t] = stage[s * row_floats + t];
      }
    }
  }
  if (store_issuer) tma::wait_stores_read();  // shared memory stays valid until the last box has been read
}

template <int KIND, int DEPTH>
int launch_depth(const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream) {
  const bool wrec = plan.weights;
  if (a.save_margin != nullptr) {
    if (plan.ord_bytes == 1)
      return wrec ? launch_one(forest_forward_tiled_kernel<KIND, DEPTH, uint8_t, true, true>, plan, a, grid, stream)
                  : launch_one(forest_forward_tiled_kernel<KIND, DEPTH, uint8_t, false, true>, plan, a, grid, stream);
    return wrec ? launch_one(forest_forward_tiled_kernel<KIND, DEPTH, uint16_t, true, true>, plan, a, grid, stream)
                : launch_one(forest_forward_tiled_kernel<KIND, DEPTH, uint16_t, false, true>, plan, a, grid, stream);
  }
  if (plan.ord_bytes == 1)
    return wrec ? launch_one(forest_forward_tiled_kernel<KIND, DEPTH, uint8_t, true>, plan, a, grid, stream)
                : launch_one(forest_forward_tiled_kernel<KIND, DEPTH, uint8_t, false>, plan, a, grid, stream);
  return wrec ? launch_one(forest_forward_tiled_kernel<KIND, DEPTH, uint16_t, true>, plan, a, grid, stream)
              : launch_one(forest_forward_tiled_kernel<KIND, DEPTH, uint16_t, false>, plan, a, grid, stream);
}

template <int KIND>
int launch_kind(int depth, const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream) {
  switch (depth) {
#define HT_DEPTH_CASE(D) \
  case D:                \
    return launch_depth<KIND, D>(plan, a, grid, stream);
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

}  // namespace

size_t forward_tiled_workspace_bytes(const ht_forest_problem *p) {
  TilePlan plan;
  if (p->K > 1) {
    if (p->M != 1 || !make_inner_plan(p, plan) || !plan.weights) return 0;
  } else if (!make_plan(p, plan)) {
    return 0;
  }
  // one output per leaf: the backward's records carry the leaf weights whatever the forward's do
  const size_t with_weights =
      p->M == 1 ? record_layout(p->kind, p->depth, (uint32_t)plan.ord_bytes, true, plan.rec.paired).bytes : 0;
  return align_up((size_t)p->T * std::max<size_t>(plan.rec.bytes, with_weights), 256);
}

size_t inner_spare_records_bytes(const ht_forest_problem *p) {
  TilePlan plan;
  if (p->K <= 1 || forward_tiled_workspace_bytes(p) > 0 || !make_inner_plan(p, plan)) return 0;
  return align_up((size_t)p->T * plan.rec.bytes, 256);
}

// Rounds of CTAs, each staging its tile and walking its share of the tree groups; one, two or four trees per warp at once
// differ in what a group costs (few in flight leave the shared memory's latency in the open).  Fitted like
// rows_forward_cost(): single calls on cold caches, spread 0.09.
double forward_tiled_cost(const ht_forest_problem *p) {
  TilePlan plan;
  if (!make_plan(p, plan)) return -1.0;
  const int64_t tiles = (p->B + plan.S - 1) / plan.S, groups = (p->T + plan.G - 1) / plan.G;
  const int splits = choose_splits(tiles, groups);
  const double waves = (double)((tiles * splits + 147) / 148), per_cta = (double)((groups + splits - 1) / splits);
  const double level = plan.per_warp == 1 ? 0.0167 : plan.per_warp == 2 ? 0.0681 : 0.141;
  const double output = plan.weights ? 0.0 : 0.0293e-3 + 0.181e-3 / vector_width(p->M, sizeof(float), {});
  return 11.1 + waves * (1.45 + 0.177e-3 * plan.S * (double)p->C +
                         per_cta * (1.37 + level * p->depth + output * plan.G * plan.S * (double)p->M));
}

bool forward_saves(const ht_forest_problem *p) {
  TilePlan plan;
  if (p->K != 1 || p->M != 1 || !make_plan(p, plan)) return false;
  // every tree group takes the kernel's streamlined body: 4 trees per warp, no short last group
  // ... and the kernel that expands the records fits its tables into shared memory
  return plan.weights && plan.per_warp == 4 && p->T % plan.G == 0 && p->B <= 0x7fffffff && backward_records_bytes(p) > 0 &&
         saved_samples_per_cta(p) != 0;
}

int forward_tiled(const ht_forest_problem *p, const float *x, const float *thr, int32_t *ord, const float *w,
                  float *out, void *records, void *eval_records, uint32_t *status_word, cudaStream_t stream, const WideOrdinals *wide) {
  TilePlan plan;
  if (!(p->K > 1 ? make_inner_plan(p, plan) : make_plan(p, plan))) return HT_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(x) & 15u) != 0 || (reinterpret_cast<uintptr_t>(out) & 15u) != 0)
    return HT_ERR_UNSUPPORTED;
  const int64_t N = threshold_count(p->kind, p->depth);
  const int64_t L = ((int64_t)1) << p->depth;
  const int outputs = plan.weights ? (int)p->M : 1;  // of a leaf, in the records
  const int64_t elements = p->T * (N + L * outputs);
  const unsigned pack_grid = (unsigned)((elements + 255) / 256);
  unsigned char *rec = static_cast<unsigned char *>(records);
  PackOnTheWay pack;
  if (wide != nullptr) pack = PackOnTheWay{wide->at, wide->channels, ord, status_word};
  if (plan.ord_bytes == 1)
    repack_records_kernel<uint8_t><<<pack_grid, 256, 0, stream>>>(thr, ord, w, rec, p->kind, p->depth, p->T, plan.rec, RecordMap(), pack, outputs);
  else
    repack_records_kernel<uint16_t><<<pack_grid, 256, 0, stream>>>(thr, ord, w, rec, p->kind, p->depth, p->T, plan.rec, RecordMap(), pack, outputs);
  HT_CHECK_LAUNCH();

  TiledArgs a = {};
  a.x = x;
  a.records = rec;
  a.w = w;
  a.M = (int)p->M;
  a.width = vector_width(p->M, sizeof(float), {w, out});
  a.by_M = Divisor((uint32_t)p->M);
  a.by_K = Divisor((uint32_t)p->K);
  a.by_pieces = Divisor((uint32_t)std::max<int64_t>(1, plan.per_warp * p->M / a.width));
  a.out = out;
  a.status_word = status_word;
  a.B = p->B;
  a.T = p->T;
  a.K = p->K;
  a.C = (int)p->C;
  a.S = plan.S;
  a.G = plan.G;
  a.per_warp = plan.per_warp;
  a.record_bytes = plan.rec.bytes;
  a.save_margin = nullptr;
  a.save_where = nullptr;
  if (eval_records != nullptr && p->M > 1) {
    const PathRecordsOf<float> paths = multi_paths<float>(p, eval_records);
    a.save_margin = paths.margin;
    a.save_where = paths.where;
  } else if (eval_records != nullptr && forward_saves(p)) {
    const EvalRecords saved = eval_record_arrays(p, eval_records);
    a.save_margin = saved.dx;
    a.save_where = saved.where;
  }
  // Full groups of 16 or 32 trees leave as tiled TMA stores when the output admits a tensor map
  // (rows of a multiple of 16 bytes); otherwise, and for a short last group, as row segments.
  a.tma_store = 0;
  if (p->K == 1 && plan.weights && plan.per_warp == 4 && (plan.G == 16 || plan.G == 32) && (p->T & 3) == 0 &&
      p->T >= plan.G && tma::encode_matrix_f32(&a.out_map, out, p->B, p->T, 32, plan.G))
    a.tma_store = 1;
  // With few sample tiles the tree groups are split among CTAs (grid.y) so that the SMs are busy in
  // every round; every split re-stages the feature tile, which is cheap next to the walk.
  const int64_t tiles = (p->B * p->K + plan.S - 1) / plan.S;
  if (tiles > 0x7fffffff) return HT_ERR_UNSUPPORTED;
  const int64_t groups = (p->T + plan.G - 1) / plan.G;
  const dim3 grid((unsigned)tiles, (unsigned)choose_splits(tiles, groups));
  if (p->K > 1) return launch_inner(p->kind, p->depth, plan, a, grid, stream);
  return p->kind == TREE ? launch_kind<TREE>(p->depth, plan, a, grid, stream)
                         : launch_kind<FERN>(p->depth, plan, a, grid, stream);
}

}  // namespace ht

// ---- self test of the bounded wait ---------------------------------------------------------
namespace ht {
namespace {
// One warp waits on a barrier that nothing ever arrives on, with a limit of a few tries: the wait has to
// run out, the kernel has to set the flag and return with its context intact.  This is the path a lost
// parameter copy takes in the tile kernels, exercised without losing a copy.
__global__ void bounded_wait_selftest_kernel(uint32_t *status_word) {
  __shared__ uint64_t never;
  if (threadIdx.x == 0) {
    tile::mbar_init(&never, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (!tile::mbar_wait(&never, 0u, 8u) && threadIdx.x == 0) atomicOr(status_word, HT_FLAG_PIPELINE_TIMEOUT);
}
}  // namespace
}  // namespace ht

extern "C" int ht_selftest_bounded_wait(uint32_t *status_word, ht_stream_t stream) {
  if (status_word == nullptr) return HT_ERR_INVALID_ARGUMENT;
  ht::bounded_wait_selftest_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(status_word);
  HT_CHECK_LAUNCH();
  return HT_OK;
}
