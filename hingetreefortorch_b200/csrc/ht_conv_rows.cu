// Forward of 1-D / 2-D convolutional hinge trees and ferns (one output per leaf), four rows of outputs at a time.
//
// out[b, j, p] = sum over input channels c (ascending) of tree (j, c) evaluated on the kernel window of channel c at output
// position p.  A CTA owns a tile of output positions of one sample and holds the pixels under it in shared memory, for as many
// input channels at a time as fit.  A warp is (four or eight rows, one output channel) and walks ONE tree at four rows x 32
// columns at a time: the root's entry serves all four, and its children's where no codes are left; where the backward wants the
// paths, four rows' codes make one 8-byte store.  Every warp has a ring of records of its own, filled by bulk copies, and waits for no other
// warp but where pixels are staged.  The sums of an output go to memory and back between two lots of input channels.  Outputs
// of a single row are taken as rows of 32 columns.
//
// Bound by the shared-memory pipe (80 % of its cycles, 12.9 wavefronts per 32 evaluations of depth 5 and no conflicts) and, with the
// codes, by issue slots (76 %; 61 instructions).  x [64, 64, 64, 64], 3 x 3, 128 trees of depth 5 (2.1e9 evaluations): 3.58 ms where
// four trees at a time on one row of a patch took 4.59 (16.4 wavefronts, 3.3 of them conflicts), 4.78 with the codes, which save the
// backward 4.7 (ht_conv_codes.cu).  With buffers of records shared by all warps 4.24, with copies instead of a patch but these buffers
// 4.43 (two records at a time, and every warp at every barrier), with a ring per warp 3.87, with the row step known to the compiler
// 3.58.
#include "ht_conv_rows.cuh"

#include <type_traits>

namespace ht {

using namespace tile;
using namespace conv_tile;
using namespace conv_rows;

namespace {

constexpr int kStages = 2;  // of a warp's ring of records

struct RowsPlan {
  int row_groups, quads;  // a tile has row_groups warps' rows, 4 * quads each
  int staged;             // input channels whose pixels are staged together
  int CC;                 // records per stage of the ring
  int splits;             // of the output channels, among CTAs
  bool flat;
  Geometry geometry;
  uint32_t record_bytes;
  size_t smem;
  int rows() const { return 4 * quads * row_groups; }
};

bool find_plan(const ConvTileProblem &p, RowsPlan &plan) {
  if (p.depth < 2 || p.depth > kMaxDepth || p.Ci < 1 || p.Co < 1 || p.B < 1 || p.Ho < 1 || p.Wo < 1) return false;
  if ((double)p.B * p.Ho * p.Wo * (double)p.Co * p.Ci < 1048576.0) return false;  // not worth a 1024-thread CTA
  plan.flat = p.Ho == 1 && p.H == 1 && p.kh == 1;
  plan.record_bytes = rows_layout(p.kind, p.depth).bytes;
  const int rows = plan.flat ? (p.Wo + kTileColumns - 1) / kTileColumns : p.Ho;
  const int columns = plan.flat ? 1 : (p.Wo + kTileColumns - 1) / kTileColumns;
  // The plan that needs the least time on the 148 SMs, in walks of 4 x 32 windows by a warp: one per output and input channel and
  // four rows.  A stage of the ring costs about a tenth of a walk, staging a channel about as much; windows read from a patch
  // instead of copies a quarter more for bank conflicts.
  double best = 0.0;
  for (int copies = 1; copies >= 0; --copies)
    for (int row_groups = 1; row_groups <= 8; row_groups *= 2)
      for (int quads = 2; quads >= 1; --quads) {
        const int R = 4 * quads * row_groups;
        if (R > 4 && R / 2 >= rows) continue;  // no taller than the output needs
        Geometry g = plan.flat ? stage_geometry(p, 1, R * kTileColumns, copies != 0) : stage_geometry(p, R, kTileColumns, copies != 0);
        if (plan.flat) g.out_step = kTileColumns * g.lane_step;
        if (g.far > kMaxOffset) continue;
        const int JB = kWarps / row_groups;
        const int64_t tiles = p.B * columns * ((rows + R - 1) / R), blocks = (p.Co + JB - 1) / JB;
        for (int CC = 4; CC >= 1; CC /= 2) {
          if (CC > 1 && CC / 2 >= p.Ci) continue;
          const size_t rings = (size_t)kWarps * kStages * CC * plan.record_bytes + kWarps * kStages * 8;
          if (rings >= kSmemBudget) continue;
          const int64_t staged = std::min<int64_t>(p.Ci, (int64_t)((kSmemBudget - rings - 128) / ((size_t)g.elements * 4)));
          if (staged < 1) continue;
          const double lots = (double)((p.Ci + staged - 1) / staged);
          for (int64_t splits = 1; splits <= std::min<int64_t>(blocks, 16); ++splits) {
            const double walks = (double)((blocks + splits - 1) / splits) * (double)p.Ci * (quads + 0.1 / CC) * (copies ? 1.0 : 1.25);
            const double cost = (double)((tiles * splits + 147) / 148) * (walks + 0.1 * (double)p.Ci + 2.0 * lots);
            if (best != 0.0 && cost >= best * 0.999) continue;
            best = cost;
            plan.row_groups = row_groups;
            plan.quads = quads;
            plan.staged = (int)staged;
            plan.CC = CC;
            plan.splits = (int)splits;
            plan.geometry = g;
            plan.smem = rings + align_up((size_t)staged * g.elements * 4, 128);
          }
        }
      }
  return best != 0.0 && plan.smem <= kSmemBudget;
}

bool make_plan(const ConvTileProblem &p, RowsPlan &plan) { return plan_at_hand(p, plan, find_plan); }

struct RowsArgs {
  const float *x;
  const unsigned char *records;  // (output channel, input channel) order
  float *out;
  uint2 *codes;  // [sample][input channel][output channel][group of four rows][column], or null
  uint32_t *status_word;
  int Ci, Co, H, W, Ho, Wo, sy, sx, py, px, dx;
  int row_groups, staged, CC, tiles_x, tiles_y, flat;
  int code_groups, code_columns;
  Geometry geometry;
};

// ROW_BYTES: between the staged rows of outputs, 0 for any.
template <int KIND, int DEPTH, int QUADS, bool CODES, uint32_t ROW_BYTES>
__global__ void __launch_bounds__(kThreads, 1) conv_forward_rows_kernel(const __grid_constant__ RowsArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr Layout lay = rows_layout(KIND, DEPTH);
  const int JB = kWarps / a.row_groups;  // output channels at a time
  const uint32_t stage_bytes = (uint32_t)a.CC * lay.bytes;
  unsigned char *rings = smem;
  uint64_t *full = reinterpret_cast<uint64_t *>(rings + (size_t)kWarps * kStages * stage_bytes);
  float *pixels = reinterpret_cast<float *>(smem + (((size_t)kWarps * kStages * (stage_bytes + 8) + 127) & ~(size_t)127));

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row0 = 4 * QUADS * (warp % a.row_groups), slot = warp / a.row_groups;
  const int tiles = a.tiles_x * a.tiles_y, rows = 4 * QUADS * a.row_groups;
  const int64_t b = blockIdx.x / tiles;
  const int tile = (int)(blockIdx.x - b * tiles);
  const int oy0 = a.flat ? 0 : (tile / a.tiles_x) * rows, ox0 = (tile % a.tiles_x) * kTileColumns * (a.flat ? rows : 1);

  // this warp's output channels: first_j, first_j + JB .. below end_j
  const int all_blocks = (a.Co + JB - 1) / JB;
  const int share = (all_blocks + (int)gridDim.y - 1) / (int)gridDim.y;
  const int first_j = (int)blockIdx.y * share * JB + slot;
  const int end_j = min(a.Co, ((int)blockIdx.y + 1) * share * JB);

  uint64_t *my_full = full + warp * kStages;
  const uint32_t ring = smem_addr(rings) + (uint32_t)(warp * kStages) * stage_bytes;
  // the ring's next fill: records of output channel fill_j and input channels fill_c .. of the lot that ends at fill_lot
  int fill_j = first_j, fill_c = 0, fill_lot0 = 0, fill_stage = 0;
  auto fill = [&]() {
    if (fill_lot0 >= a.Ci || first_j >= end_j) return;
    const int lot_end = min(fill_lot0 + a.staged, a.Ci), count = min(a.CC, lot_end - fill_c);
    const uint32_t bytes = (uint32_t)count * lay.bytes;
    mbar_expect_tx(&my_full[fill_stage], bytes);
    bulk_load(ring + (uint32_t)fill_stage * stage_bytes, a.records + ((int64_t)fill_j * a.Ci + fill_c) * lay.bytes, bytes,
              &my_full[fill_stage]);
    fill_stage = fill_stage + 1 == kStages ? 0 : fill_stage + 1;
    fill_c += count;
    if (fill_c == lot_end) {
      fill_j += JB;
      if (fill_j >= end_j) {
        fill_j = first_j;
        fill_lot0 = lot_end;
      }
      fill_c = fill_lot0;
    }
  };
  if (lane == 0) {
    for (int k = 0; k < kStages; ++k) mbar_init(&my_full[k], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int k = 0; k < kStages; ++k) fill();
  }
  __syncwarp();

  // this lane's window origin among the staged pixels; a window cell is origin + the offset held in the record
  const uint32_t row_bytes = (uint32_t)a.geometry.out_step * 4u, channel_bytes = (uint32_t)a.geometry.elements * 4u;
  const uint32_t origin = smem_addr(pixels) + (uint32_t)(lane * a.geometry.lane_step) * 4u + (uint32_t)row0 * row_bytes;
  // output of row r: at out0 + r * out_pitch; `valid_rows` of them are on the output
  const int ox = ox0 + lane + (a.flat ? row0 * kTileColumns : 0), oy = a.flat ? 0 : oy0 + row0;
  const int out_pitch = a.flat ? kTileColumns : a.Wo;
  const int valid_rows = ox >= a.Wo ? 0 : a.flat ? (a.Wo - ox + kTileColumns - 1) / kTileColumns : a.Ho - oy;
  const int code_group = a.flat ? (ox0 >> 7) + (row0 >> 2) : oy >> 2;
  const int64_t code_quads = (int64_t)a.code_groups * a.code_columns;
  const int64_t code_at = (int64_t)code_group * a.code_columns + (a.flat ? lane : ox);
  const int code_rows = a.flat || ox < a.Wo ? a.code_groups - code_group : 0;  // of this lane's, how many groups are on the output
  const int64_t code_step = a.Co * code_quads;                                 // between input channels
  const float *image = a.x + b * a.Ci * (int64_t)a.H * a.W;
  const int iy0 = oy0 * a.sy - a.py, ix0 = ox0 * a.sx - a.px;
  const int lines_per_channel = a.geometry.copies * a.geometry.rows;

  const uint32_t eight = opaque(8u);
  int stage = 0;
  uint32_t phase = 0;
  bool poisoned = false;  // a bounded wait ran out: fill and wait no more, but keep meeting the other warps
  for (int lot0 = 0; lot0 < a.Ci; lot0 += a.staged) {
    const int lot = min(a.staged, a.Ci - lot0);
    if (lot0 > 0) __syncthreads();
#pragma unroll 4
    for (int line = warp; line < lot * lines_per_channel; line += kWarps) {  // 0 outside the image (ImageToMatrix.h:138)
      const int c = (int)a.geometry.by_lines.quotient((uint32_t)line), r = line - c * lines_per_channel;
      const int copy = (int)a.geometry.by_rows.quotient((uint32_t)r), iy = iy0 + r - copy * a.geometry.rows;
      const bool inside = iy >= 0 && iy < a.H;
      const float *from = image + ((int64_t)(lot0 + c) * a.H + (inside ? iy : 0)) * a.W;
      float *to = pixels + (int64_t)line * a.geometry.width;
      for (int k = lane; k < a.geometry.width; k += 32) {
        const int ix = ix0 + k * a.geometry.pixel_step + copy * a.dx;
        to[k] = inside && ix >= 0 && ix < a.W ? __ldg(from + ix) : 0.0f;
      }
    }
    __syncthreads();
    for (int j = first_j; j < end_j; j += JB) {
      float *out = a.out + ((b * a.Co + j) * a.Ho + oy) * (int64_t)a.Wo + ox;
      float acc[4 * QUADS];
#pragma unroll
      for (int r = 0; r < 4 * QUADS; ++r) acc[r] = lot0 > 0 && r < valid_rows ? out[r * out_pitch] : 0.0f;
      uint2 *codes = nullptr;
      if constexpr (CODES) codes = a.codes + ((b * a.Ci + lot0) * a.Co + j) * code_quads + code_at;
      for (int c = 0; c < lot && !poisoned; c += a.CC) {
        if (!__all_sync(0xffffffffu, mbar_wait(&my_full[stage], phase))) {  // (the lanes leave together or not at all)
          poisoned = true;
          if (lane == 0 && a.status_word != nullptr) atomicOr(a.status_word, HT_FLAG_PIPELINE_TIMEOUT);
          break;
        }
        const int count = min(a.CC, lot - c);
        uint32_t rec = ring + (uint32_t)stage * stage_bytes, x_addr = origin + (uint32_t)c * channel_bytes;
        for (int ci = 0; ci < count; ++ci) {
#pragma unroll
          for (int q = 0; q < QUADS; ++q) {
            float value[4];
            uint32_t code[4];
            walk_rows<KIND, DEPTH, CODES, ROW_BYTES>(rec, x_addr + (uint32_t)(4 * q) * row_bytes, row_bytes, eight, value, code);
            if constexpr (CODES) {
              if (q < code_rows) __stcs(codes + q * a.code_columns, make_uint2(prmt(code[0], code[1], 0x5410u), prmt(code[2], code[3], 0x5410u)));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[4 * q + u] = __fadd_rn(acc[4 * q + u], value[u]);
          }
          if constexpr (CODES) codes += code_step;
          x_addr += channel_bytes;
          rec += lay.bytes;
        }
        __syncwarp();
        if (lane == 0) fill();
        stage = stage + 1 == kStages ? 0 : stage + 1;
        phase ^= stage == 0 ? 1u : 0u;
      }
#pragma unroll
      for (int r = 0; r < 4 * QUADS; ++r)
        if (r < valid_rows) out[r * out_pitch] = acc[r];
    }
  }
  if (poisoned) {  // copies still under way end, or are given up on, before the CTA's shared memory goes
    for (int k = 1; k < kStages; ++k) {
      stage = stage + 1 == kStages ? 0 : stage + 1;
      phase ^= stage == 0 ? 1u : 0u;
      mbar_wait(&my_full[stage], phase, 64);
    }
  }
}

template <int KIND, int DEPTH, bool CODES>
int launch_rows(const RowsPlan &plan, const RowsArgs &a, dim3 grid, cudaStream_t stream) {
  auto kernel = plan.geometry.out_step == 32
                    ? (plan.quads == 2 ? conv_forward_rows_kernel<KIND, DEPTH, 2, CODES, 128> : conv_forward_rows_kernel<KIND, DEPTH, 1, CODES, 128>)
                    : (plan.quads == 2 ? conv_forward_rows_kernel<KIND, DEPTH, 2, CODES, 0> : conv_forward_rows_kernel<KIND, DEPTH, 1, CODES, 0>);
  HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
  kernel<<<grid, kThreads, plan.smem, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

template <int KIND, bool CODES>
int launch_kind(int depth, const RowsPlan &plan, const RowsArgs &a, dim3 grid, cudaStream_t stream) {
  switch (depth) {
#define HT_DEPTH_CASE(D) \
  case D:                \
    return launch_rows<KIND, D, CODES>(plan, a, grid, stream);
    HT_DEPTH_CASE(2)
    HT_DEPTH_CASE(3)
    HT_DEPTH_CASE(4)
    HT_DEPTH_CASE(5)
    HT_DEPTH_CASE(6)
    HT_DEPTH_CASE(7)
#undef HT_DEPTH_CASE
    default:
      return HT_ERR_UNSUPPORTED;
  }
}

// One thread per record element.
__global__ void repack_rows_kernel(const float *__restrict__ thr, const int32_t *__restrict__ ord, const float *__restrict__ w,
                                   unsigned char *__restrict__ records, int kind, int depth, int64_t T, Layout lay, RecordMap map,
                                   CodeFormat format) {
  const int64_t N = threshold_count(kind, depth), L = ((int64_t)1) << depth, per_tree = N + L;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= T * per_tree) return;
  const int64_t j = e / per_tree, r = e - j * per_tree;
  unsigned char *rec = records + map.slot(j) * lay.bytes;
  if (r < N) {
    const float t = thr[j * N + r];
    const uint32_t cell = (uint32_t)ord[j * N + r];
    const uint32_t level = kind == FERN ? (uint32_t)r : 31u - (uint32_t)__clz((int)r + 1);
    reinterpret_cast<uint2 *>(rec)[r + 1] = make_uint2(__float_as_uint(t == 0.0f ? 0.0f : t), 4u * map.feature(cell));  // -0: +0
    reinterpret_cast<unsigned short *>(rec + lay.codes)[r + 1] =  // wraps: the path's leading one goes
        (unsigned short)((cell << kCodeCellShift) + format.height_code((uint32_t)depth - level) - (uint32_t)L);
    if (r == 0) reinterpret_cast<uint2 *>(rec)[0] = make_uint2(0u, 0u);
  } else {
    const int64_t h = r - N;
    reinterpret_cast<float *>(rec + lay.w)[h] = w[j * L + (int64_t)bit_reverse((uint32_t)h, depth)];
  }
}

}  // namespace

namespace conv_rows {

int repack_rows(const ConvTileProblem &p, const float *thr, const int32_t *ord, const float *w, void *records, RecordMap map,
                cudaStream_t stream) {
  const int64_t trees = p.Co * p.Ci;
  const int64_t elements = trees * (threshold_count(p.kind, p.depth) + (((int64_t)1) << p.depth));
  repack_rows_kernel<<<(unsigned)((elements + 255) / 256), 256, 0, stream>>>(
      thr, ord, w, static_cast<unsigned char *>(records), p.kind, p.depth, trees, rows_layout(p.kind, p.depth), map,
      code_format(p.depth, (int64_t)p.kh * p.kw));
  HT_CHECK_LAUNCH();
  return HT_OK;
}

}  // namespace conv_rows

size_t conv_rows_workspace_bytes(const ConvTileProblem &p) {
  RowsPlan plan;
  return make_plan(p, plan) ? align_up((size_t)(p.Co * p.Ci) * plan.record_bytes, 256) : 0;
}

int conv_forward_rows(const ConvTileProblem &p, const float *x, const float *thr, const int32_t *ord, const float *w, float *out,
                      void *records, void *codes, uint32_t *status_word, cudaStream_t stream) {
  RowsPlan plan;
  if (!make_plan(p, plan)) return HT_ERR_UNSUPPORTED;
  const CodeFormat format = code_format(p.depth, (int64_t)p.kh * p.kw);
  if (codes != nullptr && !format.fits) return HT_ERR_UNSUPPORTED;
  const int R = plan.rows(), tile_columns = kTileColumns * (plan.flat ? R : 1);
  const int tiles_x = (p.Wo + tile_columns - 1) / tile_columns, tiles_y = plan.flat ? 1 : (p.Ho + R - 1) / R;
  const int64_t ctas = p.B * tiles_x * tiles_y;
  if (ctas > 0x7fffffff) return HT_ERR_UNSUPPORTED;
  RecordMap map;
  map.columns = p.kw;
  map.row_step = plan.geometry.row_step;
  map.column_step = plan.geometry.column_step;
  const int rc = repack_rows(p, thr, ord, w, records, map, stream);
  if (rc != HT_OK) return rc;
  RowsArgs a = {};
  a.x = x;
  a.records = static_cast<const unsigned char *>(records);
  a.out = out;
  a.codes = static_cast<uint2 *>(codes);
  a.status_word = status_word;
  a.Ci = (int)p.Ci;
  a.Co = (int)p.Co;
  a.H = p.H;
  a.W = p.W;
  a.Ho = p.Ho;
  a.Wo = p.Wo;
  a.sy = p.sy;
  a.sx = p.sx;
  a.py = p.py;
  a.px = p.px;
  a.dx = p.dx;
  a.row_groups = plan.row_groups;
  a.staged = plan.staged;
  a.CC = plan.CC;
  a.tiles_x = tiles_x;
  a.tiles_y = tiles_y;
  a.flat = plan.flat ? 1 : 0;
  a.code_groups = plan.flat ? (p.Wo + 4 * kTileColumns - 1) / (4 * kTileColumns) : (p.Ho + 3) / 4;
  a.code_columns = plan.flat ? kTileColumns : p.Wo;
  a.geometry = plan.geometry;
  const dim3 grid((unsigned)ctas, (unsigned)plan.splits);
  if (codes != nullptr)
    return p.kind == TREE ? launch_kind<TREE, true>(p.depth, plan, a, grid, stream) : launch_kind<FERN, true>(p.depth, plan, a, grid, stream);
  return p.kind == TREE ? launch_kind<TREE, false>(p.depth, plan, a, grid, stream) : launch_kind<FERN, false>(p.depth, plan, a, grid, stream);
}

}  // namespace ht
