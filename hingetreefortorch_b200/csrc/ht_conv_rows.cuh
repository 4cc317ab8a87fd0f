// Records, traversal and codes of the convolution kernels that take four rows of outputs at a time (ht_conv_rows.cu,
// ht_conv_codes.cu).
#pragma once

#include "ht_conv_tiled.cuh"
#include "ht_tile_common.cuh"

#include <algorithm>
#include <cstring>
#include <type_traits>

namespace ht {
namespace conv_rows {

constexpr int kMaxDepth = 7;
constexpr int64_t kMaxOffset = 16383;  // of a window cell from the window origin, in staged numbers

// What the backward needs of an evaluation, in 16 bits: the leaf in path order (bits 0 .. depth - 1), the window cell of the
// deciding vertex (from bit 7), the factor sign(margin) as the first two bits of a float on top (2, -2, or 0 for a margin of zero
// or none), and the deciding vertex's height (depth - level, 1 .. depth, three bits) where bits are left: from bit 11 (cells of
// four bits), below bit 7, or the lower ones there and the higher ones above the cell.
constexpr uint32_t kCodeCellShift = 7;
struct CodeFormat {
  bool fits;
  int cell_bits;
  int low_bits, low_shift, high_shift;  // the height: low_bits bits at low_shift, the others at high_shift
  __host__ __device__ uint32_t height_code(uint32_t height) const {
    return (height & ((1u << low_bits) - 1u)) << low_shift | (height >> low_bits) << high_shift;
  }
};
inline CodeFormat code_format(int depth, int64_t cells) {
  CodeFormat f = {false, 0, 3, 0, 0};
  while ((((int64_t)1) << f.cell_bits) < cells) ++f.cell_bits;
  const int above = 7 - f.cell_bits, below = 7 - depth;
  f.high_shift = (int)kCodeCellShift + f.cell_bits;
  f.low_shift = above >= 3 ? (int)kCodeCellShift + 4 : depth;
  if (above < 3 && below < 3) f.low_bits = below;
  f.fits = depth >= 2 && depth <= kMaxDepth && above >= 0 && below >= 0 && (above >= 3 || below >= 3 || above + below >= 3);
  return f;
}

// Vertex v (1-based; ferns: level + 1) has the entry {threshold, byte offset of its window cell among the staged numbers} at byte
// 8 v (bytes 0..7 are zero); the leaf weights follow in path order, root decision first, then for every vertex (16 bits at 2 v)
// its part of a code.
struct Layout {
  uint32_t w, codes, bytes;
};
__host__ __device__ constexpr Layout rows_layout(int kind, int depth) {
  const uint32_t n = kind == FERN ? (uint32_t)depth : (1u << depth) - 1u;
  const uint32_t w = tile::round16(8u * (n + 1u)), codes = w + 4u * (1u << depth);
  return Layout{w, codes, tile::round16(codes + 2u * (n + 1u))};
}

// How the image under `rows` x `columns` outputs lies in shared memory, per input channel.  As a patch: its rows, one after
// another.  As copies: for every window column the pixels that it meets under the output columns, [window column][image row]
// [output column], so that the 32 lanes read 32 banks whatever cells they look at, and whatever the stride; kw / stride times
// the patch.
struct Geometry {
  int rows, width;            // image rows; numbers per row
  int copies, pixel_step;     // 1, or as many as window columns; between the pixels of neighbouring numbers of a row
  int row_step, column_step;  // between window rows and window columns
  int lane_step, out_step;    // between output columns and output rows
  int elements;
  int64_t far;  // the largest offset of a cell
  Divisor by_width, by_rows, by_lines;  // quotients by width, rows and copies * rows
};
inline Geometry stage_geometry(const ConvTileProblem &p, int rows, int columns, bool copies) {
  Geometry g;
  g.rows = (rows - 1) * p.sy + (p.kh - 1) * p.dy + 1;
  g.width = copies ? columns : (columns - 1) * p.sx + (p.kw - 1) * p.dx + 1;
  g.copies = copies ? p.kw : 1;
  g.pixel_step = copies ? p.sx : 1;
  g.row_step = p.dy * g.width;
  g.column_step = copies ? g.rows * g.width : p.dx;
  g.lane_step = copies ? 1 : p.sx;
  g.out_step = p.sy * g.width;
  g.elements = (int)std::min<int64_t>((int64_t)g.copies * g.rows * g.width, 1 << 24);
  g.far = (int64_t)(p.kh - 1) * g.row_step + (int64_t)(p.kw - 1) * g.column_step;
  g.by_width = Divisor((uint32_t)g.width);
  g.by_rows = Divisor((uint32_t)g.rows);
  g.by_lines = Divisor((uint32_t)(g.copies * g.rows));
  return g;
}

// A call asks for its plans several times (scratch, what is kept, the launch): each thread has the last one of each kind at hand.
// Finding one takes 3 us (the forward's) or 0.7 to 1.4 us (the parameter kernel's, asked for twice in a saving forward and four times
// in a backward), a comparison some 0.02.
template <typename Plan>
bool plan_at_hand(const ConvTileProblem &p, Plan &plan, bool (*find)(const ConvTileProblem &, Plan &)) {
  static_assert(std::has_unique_object_representations<ConvTileProblem>::value, "compared byte by byte");
  thread_local ConvTileProblem last = {};
  thread_local Plan found = {};
  thread_local bool known = false, takes = false;
  if (!known || std::memcmp(&last, &p, sizeof p) != 0) {
    takes = find(p, found);
    last = p;
    known = true;
  }
  plan = found;
  return takes;
}

// The records of all trees; `map`: from window cells to offsets, and from trees (j * Ci + c) to records.
int repack_rows(const ConvTileProblem &p, const float *thr, const int32_t *ord, const float *w, void *records, tile::RecordMap map,
                cudaStream_t stream);

#ifdef __CUDACC__
// Where staged number `at` of a channel comes from, relative to the window origin of the first output.
__device__ __forceinline__ void staged_pixel(const Geometry &g, int dx, int at, int &y, int &x) {
  const int line = (int)g.by_width.quotient((uint32_t)at);
  const int copy = (int)g.by_rows.quotient((uint32_t)line);
  y = line - copy * g.rows;
  x = (at - line * g.width) * g.pixel_step + copy * dx;
}

template <uint32_t OFFSET>
__device__ __forceinline__ uint2 lds_b64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(addr), "n"(OFFSET));
  return v;
}

template <uint32_t OFFSET>
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u16 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(OFFSET));
  return v;
}

// A number that the compiler does not know: products with it run on the FMA pipe (IMAD), which these kernels leave half idle,
// where shifts and additions of known numbers would join the compares and selects on the ALU pipe.
__device__ __forceinline__ uint32_t opaque(uint32_t known) {
  uint32_t v;
  asm volatile("mov.u32 %0, %1;" : "=r"(v) : "r"(known));
  return v;
}

// Walks the tree at `rec` on four windows: value[u] = |least margin| * leaf weight, and with CODES the evaluation's code.
// The root's entry, the same for all windows, is loaded once for the four, and without CODES its children's are; another vertex's
// threshold and offset come in one load from the address that the path makes.
// Window u's origin is x_addr + u * row_bytes; ROW_BYTES, if not 0, says how many those are and joins the loads' immediates.
template <int KIND, int DEPTH, bool CODES, uint32_t ROW_BYTES>
__device__ __forceinline__ void walk_rows(uint32_t rec, uint32_t x_addr, uint32_t row_bytes, uint32_t eight, float (&value)[4],
                                          uint32_t (&code)[4]) {
  constexpr Layout lay = rows_layout(KIND, DEPTH);
  constexpr uint32_t kWeightAt = lay.w, kLeaves = 1u << DEPTH, kCodesAt = lay.codes;
  uint32_t v[4], decided[4];
  float best[4], first[4], held[4];
  const uint2 root = lds_b64<8>(rec);
  uint4 children = make_uint4(0u, 0u, 0u, 0u);
  if constexpr (KIND != FERN && !CODES) children = tile::lds_b128_at<16>(rec);
  static_for<0, DEPTH>([&](auto level) {
    constexpr int l = decltype(level)::value;
    uint2 same = root;
    if constexpr (KIND == FERN && l > 0) same = lds_b64<8u * (l + 1)>(rec);
    static_for<0, 4>([&](auto row) {
      constexpr int u = decltype(row)::value;
      uint2 entry = same;
      if constexpr (KIND != FERN && l == 1 && !CODES) {
        const bool right = v[u] == 3u;
        entry = make_uint2(right ? children.z : children.x, right ? children.w : children.y);
      } else if constexpr (KIND != FERN && l >= 1) {
        entry = lds_b64<0>(CODES ? rec + eight * v[u] : rec + 8u * v[u]);
      }
      float x;
      if constexpr (ROW_BYTES != 0) x = tile::lds_f32_at<u * ROW_BYTES>(x_addr + entry.y);
      else x = tile::lds_f32(x_addr + u * row_bytes + entry.y);
      const float nm = __uint_as_float(entry.x) - x;
      if constexpr (l == 0) v[u] = 1u;
      if constexpr (CODES) {  // the shallowest least margin, signed
        if (l == 0 || fabsf(nm) < fabsf(best[u])) {
          best[u] = nm;
          decided[u] = KIND == FERN ? (uint32_t)(l + 1) : v[u];
        }
      } else {
        const float am = fabsf(nm);
        if constexpr (l == 0) best[u] = first[u] = am;
        else if constexpr (l % 2 == 1) held[u] = am;  // joins the minimum together with the next level's
        else best[u] = tile::min3(best[u], held[u], am);
      }
      v[u] = __funnelshift_l(__float_as_uint(nm), v[u], 1);
    });
  });
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    float am;
    if constexpr (CODES) {
      am = fabsf(best[u]);
      const uint32_t factor = am > 0.0f ? ((__float_as_uint(best[u]) >> 16) & 0x8000u) ^ 0xc000u : 0u;
      // (the low 16 bits; the vertex's part makes up for the path's leading one)
      code[u] = lds_u16<kCodesAt>(rec + 2u * decided[u]) + v[u] + factor;
    } else {
      if (DEPTH % 2 == 0) best[u] = fminf(best[u], held[u]);  // the last level was an odd one
      am = first[u] != first[u] ? first[u] : best[u];
    }
    if constexpr (kWeightAt >= 4u * kLeaves)
      value[u] = __fmul_rn(am, tile::lds_f32_at<kWeightAt - 4u * kLeaves>(rec + 4u * v[u]));
    else  // short records (ferns): the constant is negative
      value[u] = __fmul_rn(am, tile::lds_f32(rec + 4u * v[u] + (kWeightAt - 4u * kLeaves)));
  }
}
#endif

}  // namespace conv_rows
}  // namespace ht
