// Threshold and leaf-weight gradients of 1-D / 2-D convolutional hinge trees and ferns (one output per leaf) from the codes that
// the forward left (ht_conv_rows.cuh): no walk.
//
// A CTA owns one input channel, the trees of up to 32 output channels on it, and a run of the batch's bands (some rows of a
// sample's outputs); a warp owns one tree, or with fewer trees a share of a band's windows too.  The pixels under a band are
// staged for all warps while they work on the band before.  A code gives the leaf and the deciding vertex, whose threshold and
// pixel give the margin as the walk had it; the terms go into bins in shared memory that the warp's lanes own by columns, as in
// ht_conv_tiled_bwd.cu, and leave after the CTA's last band, one global reduction per touched bin.
//
// Bound by issue slots (78 %; 59 instructions and 10.4 shared-memory wavefronts per 32 evaluations).  x [64, 64, 64, 64], 3 x 3, 128
// trees of depth 5 (2.1e9 evaluations): 4.37 ms where the kernel that walks takes 9.03 (its bins leave per tree and tile, and it
// writes the codes for the image gradient itself).  Divisions per staged pixel, 64-bit addresses per load and pixels held in
// registers until the next band had made it 7.5.
#include "ht_conv_rows.cuh"

#include <type_traits>

namespace ht {

using namespace tile;
using namespace conv_tile;
using namespace conv_rows;

namespace {

constexpr int kMostPixels = 8;  // of a band per thread

// Columns of a warp's bins, 4 KB of them: lanes that share one take turns.
__host__ __device__ constexpr int bin_columns(int depth) { return depth <= 5 ? 16 : depth == 6 ? 8 : 4; }

struct CodesPlan {
  int trees, parts;   // of a CTA at a time: trees * parts warps
  int columns;        // lanes' columns per bin: 16, 8 or 4
  int quads, blocks;  // of a band: groups of four rows, and blocks of 32 columns
  int bands_y, bands_x;
  bool flat;
  Geometry geometry;
  Layout record;
  size_t smem;
};

bool find_plan(const ConvTileProblem &p, CodesPlan &plan) {
  plan.flat = p.Ho == 1 && p.H == 1 && p.kh == 1;
  plan.record = rows_layout(p.kind, p.depth);
  plan.trees = 1;
  while (plan.trees < kWarps && plan.trees < p.Co) plan.trees *= 2;
  plan.parts = kWarps / plan.trees;
  plan.columns = bin_columns(p.depth);
  const size_t fixed = (size_t)plan.trees * plan.record.bytes + (size_t)kWarps * (2 << p.depth) * plan.columns * 4 + 128 + 16;
  if (fixed >= kSmemBudget) return false;
  // The largest band: its pixels fit twice beside the bins.
  const size_t most = std::min<size_t>((kSmemBudget - fixed) / 8, (size_t)kMostPixels * kThreads);
  const int all_quads = plan.flat ? (p.Wo + 4 * kTileColumns - 1) / (4 * kTileColumns) : (p.Ho + 3) / 4;
  const int all_blocks = plan.flat ? 1 : (p.Wo + kTileColumns - 1) / kTileColumns;
  int64_t largest = 0;
  for (int copies = 1; copies >= 0 && largest == 0; --copies)
    for (int blocks = std::min(all_blocks, 4); blocks >= 1; --blocks)
      for (int quads = std::min(all_quads, 16); quads >= 1; --quads) {
        Geometry g = plan.flat ? stage_geometry(p, 1, 4 * kTileColumns * quads, copies != 0)
                               : stage_geometry(p, 4 * quads, kTileColumns * blocks, copies != 0);
        if (plan.flat) g.out_step = kTileColumns * g.lane_step;
        if (g.far > kMaxOffset || (size_t)g.elements > most) continue;
        // by the windows of the band's share of the whole, even bands first
        const int bands_y = (all_quads + quads - 1) / quads, bands_x = (all_blocks + blocks - 1) / blocks;
        const int64_t value = (int64_t)1000000 / ((int64_t)bands_y * quads * bands_x * blocks) * 64 + quads * blocks;
        if (value <= largest) continue;
        largest = value;
        plan.quads = quads;
        plan.blocks = blocks;
        plan.bands_y = bands_y;
        plan.bands_x = bands_x;
        plan.geometry = g;
        plan.smem = fixed + 8 * align_up((size_t)g.elements, 32);
      }
  return largest != 0 && plan.smem <= kSmemBudget;
}

bool make_plan(const ConvTileProblem &p, CodesPlan &plan) { return plan_at_hand(p, plan, find_plan); }

struct CodesArgs {
  const float *x, *g;
  const unsigned char *records;  // (input channel, output channel) order
  const uint2 *codes;
  float *gthr, *gw;
  int64_t bands, code_quads;
  int Ci, Co, H, W, Ho, Wo, sy, sx, py, px, dx;
  int trees, parts, quads, blocks, bands_y, bands_x, flat, code_columns;
  CodeFormat format;
  Geometry geometry;
};

// A number from global to shared memory without a register on its way, or zero.
__device__ __forceinline__ void copy_or_zero(uint32_t to, const float *from, bool copy) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(from), "r"(copy ? 4 : 0) : "memory");
}
__device__ __forceinline__ void wait_for_copies() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// SPLIT: the heights stand in two places of the codes.
template <int KIND, int DEPTH, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1) conv_params_from_codes_kernel(const __grid_constant__ CodesArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr Layout lay = rows_layout(KIND, DEPTH);
  constexpr uint32_t kN = KIND == FERN ? DEPTH : (1u << DEPTH) - 1u, kL = 1u << DEPTH;
  constexpr int kColumns = bin_columns(DEPTH);
  const int pixels = (a.geometry.elements + 31) & ~31;
  float *stage = reinterpret_cast<float *>(smem);  // two bands' pixels
  float *bins = stage + 2 * pixels;                // [warp][2^DEPTH][threshold bin | leaf bin][columns]
  unsigned char *records = reinterpret_cast<unsigned char *>(bins + (size_t)kWarps * 2 * kL * kColumns);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c = blockIdx.x, j = blockIdx.y * a.trees + warp % a.trees, part = warp / a.trees;
  const int64_t share = (a.bands + gridDim.z - 1) / gridDim.z, band0 = blockIdx.z * share, band_end = min(band0 + share, a.bands);
  if (band0 >= band_end) return;
  const int per_sample = a.bands_y * a.bands_x;

  for (int i = tid; i < kWarps * 2 * (int)kL * kColumns; i += kThreads) bins[i] = 0.0f;
  for (int t = warp; t < a.trees && blockIdx.y * a.trees + t < a.Co; t += kWarps) {
    const uint4 *from = reinterpret_cast<const uint4 *>(a.records + ((int64_t)c * a.Co + blockIdx.y * a.trees + t) * lay.bytes);
    for (int i = lane; i < (int)(lay.bytes / 16); i += 32) reinterpret_cast<uint4 *>(records + t * lay.bytes)[i] = __ldg(from + i);
  }

  auto place = [&](int64_t band, int64_t &b, int &oy0, int &ox0) {
    b = band / per_sample;
    const int r = (int)(band - b * per_sample), by = r / a.bands_x;
    oy0 = a.flat ? 0 : by * 4 * a.quads;
    ox0 = a.flat ? by * 4 * kTileColumns * a.quads : (r - by * a.bands_x) * kTileColumns * a.blocks;
  };
  auto stage_pixels = [&](int64_t band) {  // under way when it returns; 0 outside the image (ImageToMatrix.h:138)
    int64_t b;
    int oy0, ox0;
    place(band, b, oy0, ox0);
    const float *image = a.x + (b * a.Ci + c) * (int64_t)a.H * a.W;
    const uint32_t to = smem_addr(stage) + (uint32_t)((int)((band - band0) & 1) * pixels) * 4u;
    for (int at = tid; at < a.geometry.elements; at += kThreads) {
      int iy, ix;
      staged_pixel(a.geometry, a.dx, at, iy, ix);
      iy += oy0 * a.sy - a.py;
      ix += ox0 * a.sx - a.px;
      const bool inside = iy >= 0 && iy < a.H && ix >= 0 && ix < a.W;
      copy_or_zero(to + (uint32_t)at * 4u, image + (inside ? (int64_t)iy * a.W + ix : 0), inside);
    }
  };
  stage_pixels(band0);
  wait_for_copies();
  __syncthreads();

  const bool working = j < a.Co;
  const uint32_t record = smem_addr(records) + (uint32_t)(warp % a.trees) * lay.bytes;
  constexpr uint32_t kBinBytes = 4u * kColumns, kRowBytes = 2u * kBinBytes;
  constexpr int kTurns = 32 / kColumns;
  const int group = lane / kColumns;
  const uint32_t my_bins = smem_addr(bins) + (uint32_t)(warp * 2 * (int)kL * kColumns + lane % kColumns) * 4u;
  const uint32_t eight = opaque(8u), four = opaque(4u), row_bytes = opaque(kRowBytes);
  const uint32_t x_row = (uint32_t)a.geometry.out_step * 4u, x_block = (uint32_t)(kTileColumns * a.geometry.lane_step) * 4u;
  const int pitch = a.flat ? kTileColumns : a.Wo;  // between a lane's four windows, in outputs
  // the next group of windows of this warp: `parts` further, as rows and blocks
  const int step_q = a.parts / a.blocks, step_b = a.parts - step_q * a.blocks;
  const int step_up = step_q * 4 * pitch + step_b * kTileColumns, wrap_up = 4 * pitch - a.blocks * kTileColumns;
  const int step_code = step_q * a.code_columns + step_b * kTileColumns, wrap_code = a.code_columns - a.blocks * kTileColumns;
  const uint32_t step_x = (uint32_t)(4 * step_q) * x_row + (uint32_t)step_b * x_block, wrap_x = 4u * x_row - (uint32_t)a.blocks * x_block;

  for (int64_t band = band0; band < band_end; ++band) {
    if (band + 1 < band_end) stage_pixels(band + 1);  // into the buffer that all warps left before the last barrier
    if (working) {
      int64_t b;
      int oy0, ox0;
      place(band, b, oy0, ox0);
      const int q0 = part / a.blocks, block0 = part - q0 * a.blocks;  // this warp's first group of windows: rows, columns
      const int first = q0 * 4 * pitch + block0 * kTileColumns;
      const float *up_at = a.g + (b * a.Co + j) * a.Ho * (int64_t)a.Wo + (a.flat ? ox0 : oy0 * a.Wo + ox0) + lane + first;
      const uint2 *code_at = a.codes + ((b * a.Ci + c) * a.Co + j) * a.code_quads +
                             (a.flat ? (ox0 >> 7) * kTileColumns : (oy0 >> 2) * a.code_columns + ox0) + lane +
                             q0 * a.code_columns + block0 * kTileColumns;
      uint32_t x_next = smem_addr(stage) + (uint32_t)((int)((band - band0) & 1) * pixels + lane * a.geometry.lane_step) * 4u +
                        (uint32_t)(4 * q0) * x_row + (uint32_t)block0 * x_block;
      // WHOLE: all windows of the band are on the output
      auto run = [&](auto whole) {
        constexpr bool WHOLE = decltype(whole)::value;
        uint2 code_next = make_uint2(0u, 0u);
        float up_next[4] = {0.f, 0.f, 0.f, 0.f};
        int rows_next = 4;  // of this lane's four windows, how many (the first ones) are on the output
        int block = block0, q = q0;
        auto fetch = [&]() {
          if constexpr (!WHOLE) {
            const int ox = ox0 + (a.flat ? 128 * q : 32 * block) + lane, oy = oy0 + 4 * q;
            rows_next = ox >= a.Wo ? 0 : a.flat ? (a.Wo - ox + 31) >> 5 : max(a.Ho - oy, 0);
            if (rows_next == 0) return;
          }
          code_next = __ldcs(code_at);
#pragma unroll
          for (int u = 0; u < 4; ++u) up_next[u] = __ldg(up_at + (WHOLE ? u : min(u, rows_next - 1)) * pitch);
        };
        if (q < a.quads) fetch();
        while (q < a.quads) {
          const uint32_t raw[2] = {code_next.x, code_next.y};
          float up[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) up[u] = up_next[u];
          const int rows = rows_next;
          const uint32_t x_at = x_next;
          q += step_q;
          block += step_b;
          up_at += step_up;
          code_at += step_code;
          x_next += step_x;
          if (block >= a.blocks) {  // on to the next rows
            block -= a.blocks;
            ++q;
            up_at += wrap_up;
            code_at += wrap_code;
            x_next += wrap_x;
          }
          if (q < a.quads) fetch();
          float term_thr[4], term_w[4];
          uint32_t at_thr[4], at_w[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t code = u & 1 ? raw[u >> 1] >> 16 : raw[u >> 1];
            const uint32_t leaf = code & (kL - 1u);
            uint32_t height;
            if constexpr (SPLIT)
              height = ((code >> DEPTH) & ((1u << (7 - DEPTH)) - 1u)) | ((code >> a.format.high_shift) << (7 - DEPTH) & 7u);
            else
              height = (code >> a.format.low_shift) & 7u;
            // (masked: codes that a forward left unwritten, or of lanes without windows, must lead to some vertex too; entry 0 is empty)
            const uint32_t v = KIND == FERN ? min(((uint32_t)DEPTH + 1u - height) & 7u, (uint32_t)DEPTH) : ((leaf | kL) >> height) & (kL - 1u);
            const uint2 entry = lds_b64<0>(record + eight * v);
            const float nm = __uint_as_float(entry.x) - lds_f32(x_at + (uint32_t)u * x_row + entry.y);
            const float wv = lds_f32_at<lay.w>(record + four * leaf);
            // the threshold term is -sign(margin) * w * g, the factor twice the sign
            const float factor = __uint_as_float((u & 1 ? raw[u >> 1] : raw[u >> 1] << 16) & 0xc0000000u);
            term_thr[u] = __fmul_rn(-factor, __fmul_rn(wv, 0.5f * up[u]));
            term_w[u] = __fmul_rn(fabsf(nm), up[u]);
            if constexpr (!WHOLE)
              if (u >= rows) term_thr[u] = term_w[u] = 0.0f;
            at_thr[u] = my_bins + v * row_bytes;
            at_w[u] = my_bins + leaf * row_bytes + kBinBytes;
          }
          // Lanes that share a column (32 / columns of them) do not update it together: while one group adds its threshold terms
          // its neighbour adds its leaf terms, then they swap.  The four bins of one kind may coincide, so they stay in order.
          auto add_one_kind = [&](bool thr_now) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const uint32_t at = thr_now ? at_thr[u] : at_w[u];
              sts_f32(at, __fadd_rn(thr_now ? term_thr[u] : term_w[u], lds_f32(at)));
            }
          };
          if constexpr (kTurns == 2) {
            add_one_kind(group == 0);
            __syncwarp();
            add_one_kind(group != 0);
            __syncwarp();
          } else {
#pragma unroll
            for (int turn = 0; turn < kTurns; ++turn) {
              if ((group >> 1) == (turn >> 1)) add_one_kind(((group ^ turn) & 1) == 0);
              __syncwarp();
            }
          }
        }
      };
      const bool whole = a.flat ? ox0 + 4 * kTileColumns * a.quads <= a.Wo
                                : oy0 + 4 * a.quads <= a.Ho && ox0 + kTileColumns * a.blocks <= a.Wo;
      if (whole) run(std::true_type());
      else run(std::false_type());
    }
    wait_for_copies();
    __syncthreads();
  }
  if (!working) return;
  // sum the columns of every bin, send the touched bins out
  const int64_t tree = (int64_t)j * a.Ci + c;
  const uint32_t warp_bins = smem_addr(bins) + (uint32_t)(warp * 2 * (int)kL * kColumns) * 4u;
  for (int bin = lane; bin < (int)(kN + kL); bin += 32) {
    const bool of_thr = bin < (int)kN;
    if ((of_thr ? a.gthr : a.gw) == nullptr) continue;
    const int piece = of_thr ? 2 * (bin + 1) : 2 * (bin - (int)kN) + 1;  // a row: vertex and leaf of its number
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < kColumns; k += 4) {
      const uint4 v = lds_b128(warp_bins + (uint32_t)(piece * kColumns + k) * 4u);
      sum += (__uint_as_float(v.x) + __uint_as_float(v.y)) + (__uint_as_float(v.z) + __uint_as_float(v.w));
    }
    if (sum != 0.0f) {
      if (of_thr)
        atomicAdd(a.gthr + tree * kN + bin, sum);
      else  // bins are in path order; the reference's leaf key has the root decision as bit 0
        atomicAdd(a.gw + tree * kL + (__brev((uint32_t)(bin - (int)kN)) >> (32 - DEPTH)), sum);
    }
  }
}

template <int KIND, int DEPTH>
int launch_codes(const CodesPlan &plan, const CodesArgs &a, dim3 grid, cudaStream_t stream) {
  auto kernel = conv_params_from_codes_kernel<KIND, DEPTH, false>;
  if (a.format.low_bits < 3) {
    if constexpr (DEPTH == 5 || DEPTH == 6) kernel = conv_params_from_codes_kernel<KIND, DEPTH, true>;
    else return HT_ERR_UNSUPPORTED;
  }
  HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
  kernel<<<grid, kThreads, plan.smem, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

template <int KIND>
int launch_kind(int depth, const CodesPlan &plan, const CodesArgs &a, dim3 grid, cudaStream_t stream) {
  switch (depth) {
#define HT_DEPTH_CASE(D) \
  case D:                \
    return launch_codes<KIND, D>(plan, a, grid, stream);
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

}  // namespace

size_t conv_saved_code_bytes(const ConvTileProblem &p) {
  CodesPlan plan;
  if (conv_rows_workspace_bytes(p) == 0 || !code_format(p.depth, (int64_t)p.kh * p.kw).fits || !make_plan(p, plan)) return 0;
  if (p.Ci > 0x7fffffff || (p.Co + plan.trees - 1) / plan.trees > 65535) return 0;
  const int64_t quads = plan.flat ? (int64_t)((p.Wo + 4 * kTileColumns - 1) / (4 * kTileColumns)) * kTileColumns : (int64_t)((p.Ho + 3) / 4) * p.Wo;
  if ((double)((quads + 31) / 32) * (double)((p.Ci + 1) / 2) * (double)p.B * 16.0 > 2147483647.0) return 0;  // blocks of the image kernel
  return (size_t)(p.B * p.Ci * p.Co) * (size_t)quads * sizeof(uint2);
}

int conv_params_from_codes(const ConvTileProblem &p, const float *x, const float *thr, const int32_t *ord, const float *w,
                           const float *g, float *gthr, float *gw, void *records, const void *codes, cudaStream_t stream) {
  CodesPlan plan;
  if (conv_saved_code_bytes(p) == 0 || !make_plan(p, plan)) return HT_ERR_UNSUPPORTED;
  RecordMap map;
  map.columns = p.kw;
  map.row_step = plan.geometry.row_step;
  map.column_step = plan.geometry.column_step;
  map.inner = p.Ci;  // tree (j, c) goes to record c * Co + j
  map.outer_count = p.Co;
  const int rc = repack_rows(p, thr, ord, w, records, map, stream);
  if (rc != HT_OK) return rc;
  if (gthr == nullptr && gw == nullptr) return HT_OK;
  CodesArgs a = {};
  a.x = x;
  a.g = g;
  a.records = static_cast<const unsigned char *>(records);
  a.codes = static_cast<const uint2 *>(codes);
  a.gthr = gthr;
  a.gw = gw;
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
  a.trees = plan.trees;
  a.parts = plan.parts;
  a.quads = plan.quads;
  a.blocks = plan.blocks;
  a.bands_y = plan.bands_y;
  a.bands_x = plan.bands_x;
  a.bands = p.B * plan.bands_y * plan.bands_x;
  a.flat = plan.flat ? 1 : 0;
  a.format = code_format(p.depth, (int64_t)p.kh * p.kw);
  a.code_columns = plan.flat ? kTileColumns : p.Wo;
  a.code_quads = (int64_t)(plan.flat ? (p.Wo + 4 * kTileColumns - 1) / (4 * kTileColumns) : (p.Ho + 3) / 4) * a.code_columns;
  a.geometry = plan.geometry;
  // enough CTAs for some seven rounds of the machine, so that the last round's idle SMs cost little, of two bands at least
  const int64_t owners = p.Ci * ((p.Co + plan.trees - 1) / plan.trees);
  const int64_t splits = std::max<int64_t>(1, std::min<int64_t>({(7 * 148 + owners - 1) / owners, (a.bands + 1) / 2, 65535}));
  const dim3 grid((unsigned)p.Ci, (unsigned)((p.Co + plan.trees - 1) / plan.trees), (unsigned)splits);
  return p.kind == TREE ? launch_kind<TREE>(p.depth, plan, a, grid, stream) : launch_kind<FERN>(p.depth, plan, a, grid, stream);
}

}  // namespace ht
