// Convolutional hinge trees / ferns (1-D, 2-D, 3-D) and contract / expand.
//
// Output channel j sums, over the input channels c in ascending order, the value of the
// single-channel tree (j, c) evaluated on the kernel window of channel c at every output
// position.  The reference launches one im2col gather and one tree kernel per (sample, input
// channel) and materialises index and feature matrices (hingetree_conv_gpu.cu:368-380);
// here one launch covers the whole call: a thread owns one output position of one (sample,
// output channel), reads window cells straight from the image (padding cells read as 0) and
// walks the input channels itself, adding in the reference's order, so the forward is
// deterministic and equal to the reference CPU loop bit for bit.
#include "ht_common.cuh"
#include "ht_conv_tiled.cuh"
#include "ht_counting_sort.cuh"

#include <algorithm>
#include <cmath>

namespace ht {

namespace {

constexpr int kBlock = 256;
constexpr int kMaxCells = 2048;  // window cells whose offsets are tabulated in shared memory

struct ConvShape {
  int64_t B, Ci, Co, M, N, L;
  int64_t in_count, out_count;
  int dims, depth, cells;
  int size[3], osize[3], kernel[3], stride[3], pad[3], dil[3];
};

template <typename Real>
struct ConvArgsOf : ConvShape {
  const Real *x;
  const Real *thr;
  const int32_t *ord;
  const Real *w;
};
using ConvArgs = ConvArgsOf<float>;

// Offsets (in elements along z, y, x; dilation applied) of a window cell, 10 bits each.
__device__ __forceinline__ uint32_t packed_cell(const ConvShape &a, int cell) {
  uint32_t packed = 0;
  for (int d = a.dims - 1; d >= 0; --d) {
    const int qd = cell % a.kernel[d];
    cell /= a.kernel[d];
    packed |= (uint32_t)(qd * a.dil[d]) << (10 * (a.dims - 1 - d));
  }
  return packed;
}
__device__ __forceinline__ void fill_cell_table(const ConvShape &a, uint32_t *table) {
  for (int q = threadIdx.x; q < a.cells; q += blockDim.x) table[q] = packed_cell(a, q);
}

// Image coordinates of the first window cell of output position p (may be negative: padding).
__device__ __forceinline__ void window_origin(const ConvShape &a, int64_t p, int (&origin)[3]) {
#pragma unroll
  for (int d = 2; d >= 0; --d) {
    if (d < a.dims) {
      const int od = (int)(p % a.osize[d]);
      p /= a.osize[d];
      origin[d] = od * a.stride[d] - a.pad[d];
    } else {
      origin[d] = 0;
    }
  }
}

// The same with quotients by multiplication (positions below 2^31).
struct PositionDivisors {
  Divisor size[3];
};
__device__ __forceinline__ void window_origin(const ConvShape &a, const PositionDivisors &by, uint32_t p, int (&origin)[3]) {
#pragma unroll
  for (int d = 2; d >= 0; --d) {
    origin[d] = 0;
    if (d < a.dims) {
      const uint32_t rest = by.size[d].quotient(p);
      origin[d] = (int)(p - rest * by.size[d].number) * a.stride[d] - a.pad[d];
      p = rest;
    }
  }
}

// Flat index of window cell `packed` inside one channel image, or -1 when it lies in the padding.
__device__ __forceinline__ int cell_index(const ConvShape &a, const int (&origin)[3], uint32_t packed) {
  int index = 0;
  bool inside = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (d < a.dims) {
      const int at = origin[d] + (int)((packed >> (10 * (a.dims - 1 - d))) & 1023u);
      inside = inside && at >= 0 && at < a.size[d];
      index = index * a.size[d] + at;
    }
  }
  return inside ? index : -1;
}

template <typename Real>
struct WindowFeatureOf {
  typedef Real value_type;
  const ConvShape &a;
  const Real *chan;
  const int (&origin)[3];
  const uint32_t *table;
  __device__ __forceinline__ Real operator()(int q) const {
    const int idx = cell_index(a, origin, table[q]);
    return idx < 0 ? (Real)0 : __ldg(chan + idx);
  }
};

template <int KIND, typename Real>
__global__ void __launch_bounds__(kBlock) conv_forward_kernel(ConvArgsOf<Real> a, Real *__restrict__ out) {
  __shared__ uint32_t table[kMaxCells];
  fill_cell_table(a, table);
  __syncthreads();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // (i, j, p), p fastest
  if (e >= a.B * a.Co * a.out_count) return;
  const int64_t p = e % a.out_count;
  const int64_t j = (e / a.out_count) % a.Co;
  const int64_t i = e / (a.out_count * a.Co);
  int origin[3];
  window_origin(a, p, origin);
  Real *o = out + e * a.M;
  Real acc[8] = {};
  const bool in_registers = a.M <= 8;
  if (!in_registers)
    for (int64_t m = 0; m < a.M; ++m) o[m] = (Real)0;
  for (int64_t c = 0; c < a.Ci; ++c) {
    const int64_t tree = j * a.Ci + c;
    const WindowFeatureOf<Real> feat{a, a.x + (i * a.Ci + c) * a.in_count, origin, table};
    const PathOf<Real> path = traverse<KIND>(feat, a.thr + tree * a.N, a.ord + tree * a.N, a.depth);
    const Real am = abs_of(path.margin);
    const Real *wl = a.w + (tree * a.L + path.key) * a.M;
    if (in_registers) {
#pragma unroll
      for (int m = 0; m < 8; ++m)
        if (m < a.M) acc[m] = add_rn(acc[m], mul_rn(__ldg(wl + m), am));
    } else {
      for (int64_t m = 0; m < a.M; ++m) o[m] = add_rn(o[m], mul_rn(__ldg(wl + m), am));
    }
  }
  if (in_registers) {
#pragma unroll
    for (int m = 0; m < 8; ++m)
      if (m < a.M) o[m] = acc[m];
  }
}

// The same sums for calls with too few outputs to fill the machine: a warp per input channel walks, eight at a time, and leaves
// |margin| and the leaf's place; then a thread per output adds the eight in ascending order.  What bounds the kernel above there is
// the chain of Ci walks of a thread (1458 outputs of 30 channels, depth 7: 92 us, 19 here).
constexpr int kSharing = 8;       // channels under way
constexpr int kSharedOutputs = 8;  // outputs that a thread adds up: M <= kSharing * kSharedOutputs
template <int KIND, typename Real>
__global__ void __launch_bounds__(32 * kSharing) conv_forward_shared_kernel(ConvArgsOf<Real> a, Real *__restrict__ out) {
  __shared__ uint32_t table[kMaxCells];
  __shared__ Real sizes[2][kSharing][32];
  __shared__ uint32_t leaves[2][kSharing][32];
  fill_cell_table(a, table);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t outputs = a.B * a.Co * a.out_count, mine = (int64_t)blockIdx.x * 32 + lane;
  const int64_t e = min(mine, outputs - 1);  // (i, j, p), p fastest
  const int64_t p = e % a.out_count;
  const int64_t j = (e / a.out_count) % a.Co;
  const int64_t i = e / (a.out_count * a.Co);
  int origin[3];
  window_origin(a, p, origin);
  Real acc[kSharedOutputs] = {};
  int buffer = 0;
  for (int64_t c0 = 0; c0 < a.Ci; c0 += kSharing, buffer ^= 1) {
    const int64_t c = c0 + warp;
    if (c < a.Ci) {
      const int64_t tree = j * a.Ci + c;
      const WindowFeatureOf<Real> feat{a, a.x + (i * a.Ci + c) * a.in_count, origin, table};
      const PathOf<Real> path = traverse<KIND>(feat, a.thr + tree * a.N, a.ord + tree * a.N, a.depth);
      sizes[buffer][warp][lane] = abs_of(path.margin);
      leaves[buffer][warp][lane] = (uint32_t)(tree * a.L) + path.key;  // Co * Ci * L < 2^32 (host)
    }
    __syncthreads();  // one per round: the next round writes the other buffer
    const int here = (int)min((int64_t)kSharing, a.Ci - c0);
#pragma unroll
    for (int r = 0; r < kSharedOutputs; ++r) {
      const int m = warp + r * kSharing;
      if (m >= a.M) break;
      Real weight[kSharing];
#pragma unroll
      for (int u = 0; u < kSharing; ++u) weight[u] = u < here ? __ldg(a.w + (int64_t)leaves[buffer][u][lane] * a.M + m) : (Real)0;
#pragma unroll
      for (int u = 0; u < kSharing; ++u)
        if (u < here) acc[r] = add_rn(acc[r], mul_rn(weight[u], sizes[buffer][u][lane]));
    }
  }
  if (mine >= outputs) return;
#pragma unroll
  for (int r = 0; r < kSharedOutputs; ++r)
    if (warp + r * kSharing < a.M) out[e * a.M + warp + r * kSharing] = acc[r];
}

// One thread per (i, j, p) walking the input channels; the three gradients are scattered with atomics.
// sorting_is_better() says when.
template <int KIND, typename Real>
__global__ void __launch_bounds__(kBlock) conv_backward_kernel(ConvArgsOf<Real> a, const Real *__restrict__ g, Real *gx,
                                                               Real *gthr, Real *gw) {
  __shared__ uint32_t table[kMaxCells];
  fill_cell_table(a, table);
  __syncthreads();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.B * a.Co * a.out_count) return;
  const int64_t p = e % a.out_count;
  const int64_t j = (e / a.out_count) % a.Co;
  const int64_t i = e / (a.out_count * a.Co);
  int origin[3];
  window_origin(a, p, origin);
  const Real *gl = g + e * a.M;
  for (int64_t c = 0; c < a.Ci; ++c) {
    const int64_t tree = j * a.Ci + c;
    const WindowFeatureOf<Real> feat{a, a.x + (i * a.Ci + c) * a.in_count, origin, table};
    const PathOf<Real> path = traverse<KIND>(feat, a.thr + tree * a.N, a.ord + tree * a.N, a.depth);
    const Real s = sign_of(path.margin), am = abs_of(path.margin);
    const Real *wl = a.w + (tree * a.L + path.key) * a.M;
    Real acc = (Real)0;
    for (int64_t m = 0; m < a.M; ++m) {
      const Real gm = __ldg(gl + m);
      acc = add_rn(acc, mul_rn(mul_rn(s, __ldg(wl + m)), gm));
      if (gw != nullptr) atomicAdd(gw + (tree * a.L + path.key) * a.M + m, mul_rn(am, gm));
    }
    if (gx != nullptr) {
      const int idx = cell_index(a, origin, table[a.ord[tree * a.N + path.vertex]]);
      if (idx >= 0) atomicAdd(gx + (i * a.Ci + c) * a.in_count + idx, acc);  // a padding cell has no gradient
    }
    if (gthr != nullptr) atomicAdd(gthr + tree * a.N + path.vertex, -acc);
  }
}

// CTA per (tree, slice of its evaluations): the slice's walks are sorted by leaf and by deciding vertex by counting in shared
// memory, so that the terms of a bin lie together, and a warp hands in one sum per run of 32 of them.
// What bounds the kernel above is where its reductions meet: the trees of a convolution see every position of every sample, so
// that a handful of thresholds and leaves take all terms one after the other.  It also walks the input channels of a position in
// one thread.  159744 positions of 135 ferns of depth 3 (3-D): 3923 us there, 532 here; 30375 of 24 trees of depth 3 242 and 24;
// 9947 of 420 trees of depth 4 with 4 outputs 468 and 137.  Issue slots bound it (78 % used): 772 instructions per 32
// evaluations at depth 4 with 4 outputs.
// Slices of a tree next to each other instead of trees of a slice: 728 us for the first, 532 here (its tree's sums meet).
constexpr int kSortedBins = 2048;  // leaves + decisions, at most: depth 10
template <typename Real>
__host__ __device__ constexpr int sorted_terms() { return 16 / (int)sizeof(Real); }  // outputs of a leaf at a time

// Where its arrays lie in shared memory: terms by bin [outputs at a time][slice], the tree's thresholds, bins, the tree's cells,
// partial sums, and the bin of every term.
struct ConvSortedPlaces {
  uint32_t thresholds, bins, cells, partial, keys, bytes;
};
template <typename Real>
__host__ __device__ inline ConvSortedPlaces conv_sorted_places(const ConvShape &a, uint32_t slice) {
  const uint32_t N = (uint32_t)a.N, outputs = a.M < sorted_terms<Real>() ? (uint32_t)a.M : (uint32_t)sorted_terms<Real>();
  ConvSortedPlaces at;
  at.thresholds = outputs * slice * (uint32_t)sizeof(Real);
  at.bins = (at.thresholds + N * (uint32_t)sizeof(Real) + 15u) & ~15u;
  at.cells = at.bins + 16u * (((uint32_t)a.L + N + 4u) / 4u);
  at.partial = at.cells + 4u * N;
  at.keys = at.partial + 4u * (kBlock / 32);
  at.bytes = at.keys + 2u * slice;
  return at;
}

template <int KIND, typename Real, int PER>
__global__ void __launch_bounds__(kBlock, sizeof(Real) == 4 ? 4 : 2) conv_backward_sorted_kernel(ConvArgsOf<Real> a, Divisor positions, PositionDivisors by,
                                                                      uint32_t evals, uint32_t trees, int quad_sums, const Real *__restrict__ g, Real *gx, Real *gthr, Real *gw) {
  constexpr int S = kBlock * PER, W = sorted_terms<Real>();
  extern __shared__ __align__(16) unsigned char smem[];
  const ConvSortedPlaces at = conv_sorted_places<Real>(a, S);
  Real *terms = reinterpret_cast<Real *>(smem), *thresholds = reinterpret_cast<Real *>(smem + at.thresholds);
  uint32_t *bins = reinterpret_cast<uint32_t *>(smem + at.bins);  // leaves, then vertices: counts, then first places
  uint32_t *cells = reinterpret_cast<uint32_t *>(smem + at.cells), *partial = reinterpret_cast<uint32_t *>(smem + at.partial);
  unsigned short *keys = reinterpret_cast<unsigned short *>(smem + at.keys);
  const int L = (int)a.L, N = (int)a.N, quads = (L + N + 4) / 4;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t tree = blockIdx.x % trees, first = blockIdx.x / trees * S;
  const int n = (int)min((uint32_t)S, evals - first);
  const int64_t j = tree / (uint32_t)a.Ci, c = tree - j * a.Ci;
  for (int b = tid; b < quads; b += kBlock) reinterpret_cast<uint4 *>(bins)[b] = make_uint4(0u, 0u, 0u, 0u);
  for (int v = tid; v < N; v += kBlock) {
    thresholds[v] = __ldg(a.thr + (int64_t)tree * N + v);
    cells[v] = packed_cell(a, __ldg(a.ord + (int64_t)tree * N + v));
  }
  __syncthreads();
  // the walks, all of a thread's at once; threads without an evaluation walk the slice's first
  int origin[PER][3];
  uint32_t sample[PER], position[PER], key[PER], vertex[PER], v[PER];
  Real margin[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int t = tid + u * kBlock;
    const uint32_t q = first + (uint32_t)(t < n ? t : 0);
    sample[u] = positions.quotient(q);
    position[u] = q - sample[u] * positions.number;
    window_origin(a, by, position[u], origin[u]);
    key[u] = vertex[u] = v[u] = 0;
    margin[u] = (Real)0;
  }
  for (int l = 0; l < a.depth; ++l) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const uint32_t here = KIND == FERN ? (uint32_t)l : v[u];
      const int idx = cell_index(a, origin[u], cells[here]);
      const Real m = (idx < 0 ? (Real)0 : __ldg(a.x + ((int64_t)sample[u] * a.Ci + c) * a.in_count + idx)) - thresholds[here];
      const uint32_t bit = m > (Real)0 ? 1u : 0u;
      if (l == 0 || abs_of(m) < abs_of(margin[u])) {
        margin[u] = m;
        vertex[u] = here;
      }
      key[u] |= bit << l;
      v[u] = 2 * v[u] + 1 + bit;
    }
  }
  uint32_t by_leaf[PER], by_vertex[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    by_leaf[u] = by_vertex[u] = 0;
    if (tid + u * kBlock < n) {
      by_leaf[u] = atomicAdd(&bins[key[u]], 1u);
      by_vertex[u] = atomicAdd(&bins[L + vertex[u]], 1u);
    }
  }
  __syncthreads();
  exclusive_sums<kBlock>(reinterpret_cast<uint4 *>(bins), quads, partial);
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    by_leaf[u] += bins[key[u]];
    by_vertex[u] += bins[L + vertex[u]] - (uint32_t)n;
    if (tid + u * kBlock < n) keys[by_leaf[u]] = (unsigned short)key[u];
  }

  // sums of runs: `to(bin, sums)` takes those of one
  auto hand_in = [&](auto numbers, auto to) {
    constexpr int count = decltype(numbers)::value;
    for (int e0 = warp * 32; e0 < n; e0 += kBlock) {
      const int e = e0 + lane;
      Real sum[count];
#pragma unroll
      for (int k = 0; k < count; ++k) sum[k] = e < n && (k == 0 || k < a.M) ? terms[k * S + e] : (Real)0;
      const uint32_t bin = e < n ? keys[e] : 0xffffu;
      if (sums_of_runs(bin, sum, lane) && e < n) to(bin, sum);
    }
  };
  const Real *w = a.w + (int64_t)tree * L * a.M;
  Real through[PER];  // the gradient that arrives at the margin
#pragma unroll
  for (int u = 0; u < PER; ++u) through[u] = (Real)0;
  for (int64_t m0 = 0; m0 < a.M; m0 += W) {
    const int here = (int)min((int64_t)W, a.M - m0);
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      if (tid + u * kBlock >= n) continue;
      const Real s = sign_of(margin[u]), am = abs_of(margin[u]);
      const Real *gl = g + (((int64_t)sample[u] * a.Co + j) * a.out_count + position[u]) * a.M + m0, *wl = w + (int64_t)key[u] * a.M + m0;
#pragma unroll
      for (int k = 0; k < W; ++k) {
        if (k >= here) break;
        const Real gm = __ldg(gl + k);
        through[u] = add_rn(through[u], mul_rn(mul_rn(s, __ldg(wl + k)), gm));
        if (gw != nullptr) terms[k * S + by_leaf[u]] = mul_rn(am, gm);
      }
    }
    if (gw == nullptr) continue;
    __syncthreads();
    Real *dst = gw + (int64_t)tree * L * a.M + m0;
    if (here == 1) {
      hand_in(std::integral_constant<int, 1>{}, [&](uint32_t bin, Real(&sum)[1]) { atomicAdd(dst + (int64_t)bin * a.M, sum[0]); });
    } else {
      hand_in(std::integral_constant<int, W>{}, [&](uint32_t bin, Real(&sum)[W]) {
        Real *to = dst + (int64_t)bin * a.M;
        if constexpr (W == 4) {
          if (quad_sums) return red_add_quad(to, sum[0], sum[1], sum[2], sum[3]);
        }
#pragma unroll
        for (int k = 0; k < W; ++k)
          if (k < here) atomicAdd(to + k, sum[k]);
      });
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    if (tid + u * kBlock >= n) continue;
    if (gx != nullptr) {
      const int idx = cell_index(a, origin[u], cells[vertex[u]]);
      if (idx >= 0) atomicAdd(gx + ((int64_t)sample[u] * a.Ci + c) * a.in_count + idx, through[u]);  // a padding cell has no gradient
    }
  }
  if (gthr == nullptr) return;
  __syncthreads();  // every thread has read its place among the leaves, and the leaves' sums have been read
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    if (tid + u * kBlock >= n) continue;
    terms[by_vertex[u]] = -through[u];
    keys[by_vertex[u]] = (unsigned short)vertex[u];
  }
  __syncthreads();
  hand_in(std::integral_constant<int, 1>{}, [&](uint32_t bin, Real(&sum)[1]) { atomicAdd(gthr + (int64_t)tree * N + bin, sum[0]); });
}

// ---- contract / expand: non-overlapping windows <-> image, any element size ----------------

struct PatchArgs {
  int dims;
  int64_t BC, image_count, window_count, cells;
  int64_t size[3], osize[3], win[3], pad[3];
};

// One thread per patch element (b, window p, cell q): its image coordinate, or -1 outside.
__device__ __forceinline__ int64_t patch_image_index(const PatchArgs &a, int64_t p, int64_t q) {
  int64_t index = 0, scale = 1;
  for (int d = a.dims - 1; d >= 0; --d) {
    const int64_t at = (p % a.osize[d]) * a.win[d] - a.pad[d] + (q % a.win[d]);
    p /= a.osize[d];
    q /= a.win[d];
    if (at < 0 || at >= a.size[d]) return -1;
    index += at * scale;
    scale *= a.size[d];
  }
  return index;
}

template <typename Word>
__global__ void __launch_bounds__(kBlock) contract_kernel(PatchArgs a, const Word *__restrict__ image,
                                                          Word *__restrict__ patches) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t per_image = a.window_count * a.cells;
  if (e >= a.BC * per_image) return;
  const int64_t b = e / per_image, r = e - b * per_image;
  const int64_t idx = patch_image_index(a, r / a.cells, r % a.cells);
  patches[e] = idx < 0 ? Word(0) : image[b * a.image_count + idx];
}

// One thread per image element: every pixel belongs to exactly one window cell (or to none, when
// the windows do not reach it), so expand is a gather as well and needs no clearing pass.
template <typename Word>
__global__ void __launch_bounds__(kBlock) expand_kernel(PatchArgs a, const Word *__restrict__ patches,
                                                        Word *__restrict__ image) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.BC * a.image_count) return;
  const int64_t b = e / a.image_count;
  int64_t rest = e - b * a.image_count;
  int64_t p = 0, q = 0, pscale = 1, qscale = 1;
  bool covered = true;
  for (int d = a.dims - 1; d >= 0; --d) {
    const int64_t at = rest % a.size[d] + a.pad[d];
    rest /= a.size[d];
    const int64_t od = at / a.win[d];
    covered = covered && od < a.osize[d];
    p += od * pscale;
    q += (at % a.win[d]) * qscale;
    pscale *= a.osize[d];
    qscale *= a.win[d];
  }
  image[e] = covered ? patches[(b * a.window_count + p) * a.cells + q] : Word(0);
}

// The same two gathers with 32-bit index arithmetic and divisions by multiplication (every divisor is a
// launch constant), for images and patch sets of fewer than 2^31 elements each: the 64-bit division chains
// above cost several hundred instructions per element and kept these pure copies at an eighth of the
// memory bandwidth.  blockIdx.y walks the (batch x channel) images.
struct FastDivisor {
  uint32_t divisor, multiplier, shift;
  __device__ __forceinline__ uint32_t quotient(uint32_t n) const {  // n < 2^31
    return divisor == 1u ? n : __umulhi(n, multiplier) >> shift;
  }
  __device__ __forceinline__ void split(uint32_t n, uint32_t &q, uint32_t &r) const {  // q may be the variable n came from
    const uint32_t whole = quotient(n);
    r = n - whole * divisor;
    q = whole;
  }
};

inline FastDivisor make_divisor(int64_t d) {
  FastDivisor f;
  f.divisor = (uint32_t)d;
  f.multiplier = 0;
  f.shift = 0;
  if (d > 1) {
    uint32_t log2 = 0;
    while ((((uint64_t)1) << log2) < (uint64_t)d) ++log2;  // ceil(log2 d)
    const uint32_t p = 31 + log2;
    f.multiplier = (uint32_t)(((((uint64_t)1) << p) + (uint64_t)d - 1) / (uint64_t)d);
    f.shift = p - 32;
  }
  return f;
}

struct PatchArgs32 {
  int dims;
  uint32_t image_count, per_image;  // elements of one image, of one image's patches
  int64_t BC;
  FastDivisor cells, osize[3], win[3], size[3];
  uint32_t pad[3], window_count;
};

template <typename Word>
__global__ void __launch_bounds__(kBlock) contract32_kernel(PatchArgs32 a, const Word *__restrict__ image,
                                                            Word *__restrict__ patches) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= a.per_image) return;
  uint32_t p, q;
  a.cells.split(r, p, q);
  uint32_t index = 0, scale = 1;
  bool inside = true;
  for (int d = a.dims - 1; d >= 0; --d) {
    uint32_t pd, qd;
    a.osize[d].split(p, p, pd);
    a.win[d].split(q, q, qd);
    const uint32_t at = pd * a.win[d].divisor + qd - a.pad[d];  // wraps below zero: caught by the comparison
    inside = inside && at < a.size[d].divisor;
    index += at * scale;
    scale *= a.size[d].divisor;
  }
  // the same place in every image: the index arithmetic above is paid once per thread, four copies in flight
  const int64_t step = gridDim.y;
  int64_t b = blockIdx.y;
  for (; b + 3 * step < a.BC; b += 4 * step) {
    Word v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = inside ? image[(b + u * step) * a.image_count + index] : Word(0);
#pragma unroll
    for (int u = 0; u < 4; ++u) patches[(b + u * step) * a.per_image + r] = v[u];
  }
  for (; b < a.BC; b += step) patches[b * a.per_image + r] = inside ? image[b * a.image_count + index] : Word(0);
}

template <typename Word>
__global__ void __launch_bounds__(kBlock) expand32_kernel(PatchArgs32 a, const Word *__restrict__ patches,
                                                          Word *__restrict__ image) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.image_count) return;
  uint32_t rest = e, p = 0, q = 0, pscale = 1, qscale = 1;
  bool covered = true;
  for (int d = a.dims - 1; d >= 0; --d) {
    uint32_t at, od, cell;
    a.size[d].split(rest, rest, at);
    at += a.pad[d];
    a.win[d].split(at, od, cell);
    covered = covered && od < a.osize[d].divisor;
    p += od * pscale;
    q += cell * qscale;
    pscale *= a.osize[d].divisor;
    qscale *= a.win[d].divisor;
  }
  const uint32_t from = p * a.cells.divisor + q;
  const int64_t step = gridDim.y;
  int64_t b = blockIdx.y;
  for (; b + 3 * step < a.BC; b += 4 * step) {
    Word v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = covered ? patches[(b + u * step) * a.per_image + from] : Word(0);
#pragma unroll
    for (int u = 0; u < 4; ++u) image[(b + u * step) * a.image_count + e] = v[u];
  }
  for (; b < a.BC; b += step) image[b * a.image_count + e] = covered ? patches[b * a.per_image + from] : Word(0);
}

inline unsigned blocks_for(int64_t n) { return (unsigned)((n + kBlock - 1) / kBlock); }

int check_conv(const ht_conv_problem *p, ConvShape &a) {
  if (p == nullptr) return HT_ERR_INVALID_ARGUMENT;
  if (p->kind != TREE && p->kind != FERN) return HT_ERR_INVALID_ARGUMENT;
  if (p->depth < 1 || p->depth > 31) return HT_ERR_DEPTH;
  if (p->dims < 1 || p->dims > 3 || p->B < 0 || p->Ci < 1 || p->Co < 0 || p->M < 0) return HT_ERR_INVALID_ARGUMENT;
  a.dims = p->dims;
  a.depth = p->depth;
  a.B = p->B;
  a.Ci = p->Ci;
  a.Co = p->Co;
  a.M = p->M;
  a.N = threshold_count(p->kind, p->depth);
  a.L = ((int64_t)1) << p->depth;
  a.in_count = a.out_count = 1;
  int64_t cells = 1;
  for (int d = 0; d < 3; ++d) {
    a.size[d] = a.osize[d] = a.kernel[d] = a.stride[d] = a.dil[d] = 1;
    a.pad[d] = 0;
  }
  for (int d = 0; d < p->dims; ++d) {
    if (p->kernel[d] <= 0 || p->stride[d] <= 0 || p->padding[d] < 0 || p->dilation[d] <= 0 || p->size[d] < 1)
      return HT_ERR_INVALID_ARGUMENT;
    const int64_t window = p->kernel[d] + (p->kernel[d] - 1) * (p->dilation[d] - 1);
    if (p->size[d] + 2 * p->padding[d] < window) return HT_ERR_INVALID_ARGUMENT;
    if ((p->kernel[d] - 1) * p->dilation[d] >= 1024 || p->size[d] > 0x3fffffff) return HT_ERR_UNSUPPORTED;
    a.size[d] = (int)p->size[d];
    a.kernel[d] = (int)p->kernel[d];
    a.stride[d] = (int)p->stride[d];
    a.pad[d] = (int)p->padding[d];
    a.dil[d] = (int)p->dilation[d];
    a.osize[d] = (int)((p->size[d] + 2 * p->padding[d] - window) / p->stride[d] + 1);
    a.in_count *= p->size[d];
    a.out_count *= a.osize[d];
    cells *= p->kernel[d];
  }
  if (cells > kMaxCells || a.in_count > 0x7fffffff) return HT_ERR_UNSUPPORTED;
  a.cells = (int)cells;
  return HT_OK;
}

size_t conv_ordinal_bytes(const ConvShape &a) { return align_up((size_t)(a.Co * a.Ci * a.N) * sizeof(int32_t), 256); }

// The problem as the shared-memory tile kernels see it (1-D and 2-D, one output per leaf).
bool tile_problem(const ht_conv_problem *p, const ConvShape &a, ConvTileProblem &t) {
  if (p->dims > 2 || a.M != 1) return false;
  const int row = p->dims == 2 ? 0 : -1, col = p->dims - 1;  // a 1-D signal is one image row
  t.kind = p->kind;
  t.depth = p->depth;
  t.B = a.B;
  t.Ci = a.Ci;
  t.Co = a.Co;
  t.H = row < 0 ? 1 : a.size[row];
  t.W = a.size[col];
  t.Ho = row < 0 ? 1 : a.osize[row];
  t.Wo = a.osize[col];
  t.kh = row < 0 ? 1 : a.kernel[row];
  t.kw = a.kernel[col];
  t.sy = row < 0 ? 1 : a.stride[row];
  t.sx = a.stride[col];
  t.py = row < 0 ? 0 : a.pad[row];
  t.px = a.pad[col];
  t.dy = row < 0 ? 1 : a.dil[row];
  t.dx = a.dil[col];
  return true;
}

size_t conv_records_bytes(const ht_conv_problem *p, const ConvShape &a) {
  ConvTileProblem t;
  if (!tile_problem(p, a, t)) return 0;
  return std::max({conv_tiled_workspace_bytes(t), conv_rows_workspace_bytes(t), conv_backward_tiled_workspace_bytes(t)});
}

template <typename Real>
int prepare_conv(const ht_conv_problem *p, const Real *x, const Real *thr, const int64_t *ord, const Real *w,
                 void *workspace, size_t workspace_bytes, uint32_t *status_word, cudaStream_t stream, ConvArgsOf<Real> &a,
                 Real *gx = nullptr, Real *gthr = nullptr, Real *gw = nullptr) {
  const int rc = check_conv(p, a);
  if (rc != HT_OK) return rc;
  const int64_t decisions = a.Co * a.Ci * a.N;
  if ((x == nullptr && a.B * a.Ci * a.in_count > 0) || ((thr == nullptr || ord == nullptr) && decisions > 0) ||
      (w == nullptr && a.Co * a.M > 0))
    return HT_ERR_INVALID_ARGUMENT;
  if (workspace == nullptr || workspace_bytes < conv_ordinal_bytes(a) + 256 ||
      (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
    return HT_ERR_WORKSPACE;
  a.x = x;
  a.thr = thr;
  a.w = w;
  a.ord = static_cast<const int32_t *>(workspace);
  ClearList clear;
  clear.add(gx, sizeof(Real) * (size_t)(a.B * a.Ci * a.in_count));
  clear.add(gthr, sizeof(Real) * (size_t)decisions);
  clear.add(gw, sizeof(Real) * (size_t)(a.Co * a.Ci * a.L * a.M));
  return pack_and_clear(ord, decisions, a.cells, static_cast<int32_t *>(workspace), status_word, clear, stream);
}

template <typename Word>
int launch_patches(bool contract, const PatchArgs &a, const void *in, void *out, cudaStream_t stream) {
  const int64_t per_image = a.window_count * a.cells;
  bool narrow = a.image_count < 0x40000000 && per_image < 0x40000000 && a.BC > 0;
  for (int d = 0; d < a.dims; ++d) narrow = narrow && a.pad[d] < 0x40000000 && a.size[d] + a.pad[d] < 0x40000000;
  if (narrow) {
    PatchArgs32 n;
    n.dims = a.dims;
    n.image_count = (uint32_t)a.image_count;
    n.per_image = (uint32_t)per_image;
    n.window_count = (uint32_t)a.window_count;
    n.BC = a.BC;
    n.cells = make_divisor(a.cells);
    for (int d = 0; d < 3; ++d) {
      n.osize[d] = make_divisor(d < a.dims ? a.osize[d] : 1);
      n.win[d] = make_divisor(d < a.dims ? a.win[d] : 1);
      n.size[d] = make_divisor(d < a.dims ? a.size[d] : 1);
      n.pad[d] = d < a.dims ? (uint32_t)a.pad[d] : 0u;
    }
    // enough blocks to fill the machine several times over, and as many images per thread as that leaves
    const unsigned across = blocks_for(contract ? per_image : a.image_count);
    const int64_t wanted = std::max<int64_t>(1, (148 * 32 + across - 1) / across);
    const dim3 grid(across, (unsigned)std::min<int64_t>(std::min<int64_t>(a.BC, wanted), 65535));
    if (contract)
      contract32_kernel<Word><<<grid, kBlock, 0, stream>>>(n, static_cast<const Word *>(in), static_cast<Word *>(out));
    else
      expand32_kernel<Word><<<grid, kBlock, 0, stream>>>(n, static_cast<const Word *>(in), static_cast<Word *>(out));
    HT_CHECK_LAUNCH();
    return HT_OK;
  }
  if (contract) {
    const int64_t n = a.BC * a.window_count * a.cells;
    if (n > 0) contract_kernel<Word><<<blocks_for(n), kBlock, 0, stream>>>(a, static_cast<const Word *>(in), static_cast<Word *>(out));
  } else {
    const int64_t n = a.BC * a.image_count;
    if (n > 0) expand_kernel<Word><<<blocks_for(n), kBlock, 0, stream>>>(a, static_cast<const Word *>(in), static_cast<Word *>(out));
  }
  HT_CHECK_LAUNCH();
  return HT_OK;
}

int run_patches(bool contract, int dims, int elem_bytes, const void *in, void *out, int64_t BC, const int64_t *size,
                const int64_t *osize, const int64_t *window, const int64_t *padding, cudaStream_t stream) {
  if (dims < 2 || dims > 3 || BC < 0 || size == nullptr || osize == nullptr || window == nullptr || padding == nullptr)
    return HT_ERR_INVALID_ARGUMENT;
  PatchArgs a;
  a.dims = dims;
  a.BC = BC;
  a.image_count = a.window_count = a.cells = 1;
  for (int d = 0; d < dims; ++d) {
    if (size[d] < 1 || osize[d] < 1 || window[d] < 1 || padding[d] < 0) return HT_ERR_INVALID_ARGUMENT;
    a.size[d] = size[d];
    a.osize[d] = osize[d];
    a.win[d] = window[d];
    a.pad[d] = padding[d];
    a.image_count *= size[d];
    a.window_count *= osize[d];
    a.cells *= window[d];
  }
  if ((in == nullptr || out == nullptr) && BC > 0) return HT_ERR_INVALID_ARGUMENT;
  switch (elem_bytes) {
    case 1: return launch_patches<uint8_t>(contract, a, in, out, stream);
    case 2: return launch_patches<uint16_t>(contract, a, in, out, stream);
    case 4: return launch_patches<uint32_t>(contract, a, in, out, stream);
    case 8: return launch_patches<uint64_t>(contract, a, in, out, stream);
    default: return HT_ERR_UNSUPPORTED;
  }
}

// Whether a call's outputs are too few for a thread each to fill the machine (and the leaves' places fit 32 bits).  Up to some 85 000
// of them a warp per channel, eight under way, is better, fewer outputs where there are fewer channels than warps: 60000 outputs of 24 channels 62 us with
// a thread each, 38 shared; 20776 of 7 21 and 8; 81000 of 52 198 and 127; but 144342 of 29 71 and 85, 69984 of 6 14.6 and 16.6, 25984
// of 2 8.6 and 10.5.
bool shares_channels(const ConvShape &a) {
  return a.Ci > 2 && a.M <= kSharing * kSharedOutputs && a.Co * a.Ci * a.L <= 0xffffffffll &&
         a.B * a.Co * a.out_count * kSharing <= 148 * 576 * std::min<int64_t>(a.Ci, kSharing);
}

// Forward / backward for either precision; the shared-memory tile kernels are single precision only.
template <typename Real>
int conv_forward(const ht_conv_problem *p, const Real *x, const Real *thr, const int64_t *ord, const Real *w, Real *out,
                 void *workspace, size_t workspace_bytes, uint32_t *status_word, ht_stream_t stream, void *codes = nullptr) {
  ConvArgsOf<Real> a;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int rc = prepare_conv<Real>(p, x, thr, ord, w, workspace, workspace_bytes, status_word, s, a);
  if (rc != HT_OK) return rc;
  const int64_t threads = a.B * a.Co * a.out_count;
  if (threads * a.M == 0) return HT_OK;
  if (out == nullptr) return HT_ERR_INVALID_ARGUMENT;
  if constexpr (std::is_same<Real, float>::value) {
    ConvTileProblem t;
    if (tile_problem(p, a, t)) {
      unsigned char *records_at = static_cast<unsigned char *>(workspace) + conv_ordinal_bytes(a);
      const size_t rows_records = conv_rows_workspace_bytes(t);
      if (rows_records != 0 && workspace_bytes >= conv_ordinal_bytes(a) + rows_records + 256) {
        const int by_rows = conv_forward_rows(t, x, thr, a.ord, w, out, records_at, codes, status_word, s);
        if (by_rows != HT_ERR_UNSUPPORTED || codes != nullptr) return by_rows;
      }
      const size_t records = conv_tiled_workspace_bytes(t);
      if (records != 0 && workspace_bytes >= conv_ordinal_bytes(a) + records + 256) {
        const int tiled = conv_forward_tiled(t, x, thr, a.ord, w, out, records_at, status_word, s);
        if (tiled != HT_ERR_UNSUPPORTED) return tiled;
      }
    }
  }
  if (shares_channels(a)) {
    auto kernel = p->kind == TREE ? conv_forward_shared_kernel<TREE, Real> : conv_forward_shared_kernel<FERN, Real>;
    kernel<<<(unsigned)((threads + 31) / 32), 32 * kSharing, 0, s>>>(a, out);
  } else {
    auto kernel = p->kind == TREE ? conv_forward_kernel<TREE, Real> : conv_forward_kernel<FERN, Real>;
    kernel<<<blocks_for(threads), kBlock, 0, s>>>(a, out);
  }
  HT_CHECK_LAUNCH();
  return HT_OK;
}

// Evaluations per thread of the sorted backward: four where the last slices are not too empty and there are CTAs enough.  6000
// evaluations of 363 trees 83 us with one per thread, 72 with four; 28090 of 575 633 and 531; but 390 of 1254 22 and 30, 10658 of 9 6 and 11.
int evaluations_per_thread(const ConvShape &a) {
  const int64_t evals = a.B * a.out_count, slices = (evals + 4 * kBlock - 1) / (4 * kBlock);
  return slices * a.Co * a.Ci >= 4 * 148 && slices * 4 * kBlock * 3 <= evals * 4 ? 4 : 1;
}

// Whether a backward sorts (conv_backward_sorted_kernel) rather than scatters (conv_backward_kernel): where its estimate is the lower
// one, in microseconds.  Sorting pays for its evaluations and for its CTAs, which clear and sum their bins.  A scatter is bound by its
// reductions, by those that meet in one threshold (a vertex that decides often) or one leaf, which are the fewer the more trees are
// under way (some 300 000 threads on consecutive positions, at different channels), or, with few outputs, by the chain of Ci walks
// of a thread; no two of them hide one another entirely, hence the norm of order 3/2.  Fits to 780 of the 1040 backwards of random
// sizes in profiles/conv_backward_choice.csv, timed both ways in one session; on the 260 others, all calls together, the chosen kernels
// take 1.013 (single precision; always sorted 1.013, always scattered 3.27) and 1.016 (double; 1.058, 2.83) of the better ones'
// time, on those of the fit 1.006 (1.021, 3.15) and 1.003 (1.076, 2.25).  [35, 30, 7, 7, 7], 75 x 30 trees of depth 3, 2 x 2 x 2, padding 1:
// sorted 982 us, scattered 695; in double precision [24, 20, 1900], 72 x 20 of depth 5: 1983 and 1247.
struct ConvBackwardRates {
  double sort, eval, level, output, piece, cta, cta_piece, cta_bin;
  double scatter, walk, line, reduction, tree_vertex, fern_vertex, leaf, chain_level, chain_output;
};
constexpr ConvBackwardRates kSingleRates = {7.38, 12.8, 1.40, 0.805, 6.69, 6.79e-4, 1.77e-4, 3.82e-6, 6.64, 0.0, 0.166, 11.6, 14600, 13500, 3710, 0.436, 0.121};
constexpr ConvBackwardRates kDoubleRates = {7.56, 17.4, 1.12, 3.10, 2.91, 17.4e-4, 20.6e-4, 6.68e-6, 6.89, 0.449, 0.183, 11.3, 10600, 10500, 2130, 0.432, 0.266};

template <typename Real>
bool sorting_is_better(const ConvShape &a, int kind) {
  const int64_t evals = a.B * a.out_count, trees = a.Co * a.Ci;
  if (a.L + a.N > kSortedBins || evals >= ((int64_t)1 << 31) || trees >= ((int64_t)1 << 31)) return false;
  const int64_t slice = evaluations_per_thread(a) * kBlock, ctas = (evals + slice - 1) / slice * trees;
  if (ctas > 0x7fffffff) return false;
  const ConvBackwardRates &r = sizeof(Real) == 4 ? kSingleRates : kDoubleRates;
  const double E = 1e-6 * (double)evals * (double)trees, M = (double)a.M, levels = (double)a.depth;
  const double pieces = (double)((a.M + sorted_terms<Real>() - 1) / sorted_terms<Real>());
  const double sorted = r.sort + E * (r.eval + r.level * levels + r.output * M + r.piece * pieces) +
                        (double)ctas * (r.cta + r.cta_piece * pieces + r.cta_bin * (double)(a.L + a.N));
  double lines = 0.0;  // cache lines that a warp's levels are on
  for (int l = 0; l < a.depth; ++l) lines += kind == FERN ? 1.0 : std::min(24.0, (double)(1u << l));
  const double under_way = std::pow(std::min((double)a.Co, std::max(1.0, 148 * 2048.0 / (double)a.out_count)), 0.8) * std::pow((double)a.Ci, 0.6);
  const double work = E * (r.walk + r.line * lines + r.reduction * M);
  const double vertices = E / under_way * (kind == FERN ? r.fern_vertex / levels : r.tree_vertex / (levels * std::sqrt(levels)));
  const double leaves = E * M / under_way * r.leaf / std::sqrt((double)a.L);
  const double chain = (double)a.Ci * (r.chain_level * levels + r.chain_output * M);
  const double sum = work * std::sqrt(work) + vertices * std::sqrt(vertices) + leaves * std::sqrt(leaves) + chain * std::sqrt(chain);
  return sorted <= r.scatter + std::cbrt(sum * sum);
}

// HT_ERR_UNSUPPORTED: sizes that sorting is not for, or not the better way for.
template <typename Real>
int launch_backward_sorted(const ConvArgsOf<Real> &a, int kind, const Real *g, Real *gx, Real *gthr, Real *gw, cudaStream_t stream) {
  if (!sorting_is_better<Real>(a, kind)) return HT_ERR_UNSUPPORTED;
  const int64_t evals = a.B * a.out_count, trees = a.Co * a.Ci;
  const int per = evaluations_per_thread(a);
  const int64_t grid = (evals + per * kBlock - 1) / (per * kBlock) * trees;
  const int quad_sums = sorted_terms<Real>() == 4 && a.M % 4 == 0 && (reinterpret_cast<uintptr_t>(gw) & 15u) == 0;
  auto kernel = kind == TREE ? (per == 4 ? conv_backward_sorted_kernel<TREE, Real, 4> : conv_backward_sorted_kernel<TREE, Real, 1>)
                             : (per == 4 ? conv_backward_sorted_kernel<FERN, Real, 4> : conv_backward_sorted_kernel<FERN, Real, 1>);
  PositionDivisors by;
  for (int d = 0; d < 3; ++d) by.size[d] = Divisor((uint32_t)a.osize[d]);
  kernel<<<(unsigned)grid, kBlock, conv_sorted_places<Real>(a, (uint32_t)(per * kBlock)).bytes, stream>>>(a, Divisor((uint32_t)a.out_count), by, (uint32_t)evals,
                                                                            (uint32_t)trees, quad_sums, g, gx, gthr, gw);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

template <typename Real>
int conv_backward(const ht_conv_problem *p, const Real *x, const Real *thr, const int64_t *ord, const Real *w, const Real *g,
                  Real *gx, Real *gthr, Real *gw, void *workspace, size_t workspace_bytes, uint32_t *status_word,
                  ht_stream_t stream, const void *saved_codes = nullptr) {
  ConvArgsOf<Real> a;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int rc = prepare_conv<Real>(p, x, thr, ord, w, workspace, workspace_bytes, status_word, s, a, gx, gthr, gw);
  if (rc != HT_OK) return rc;
  const int64_t threads = a.B * a.Co * a.out_count;
  if (threads * a.M == 0 || (gx == nullptr && gthr == nullptr && gw == nullptr)) return HT_OK;
  if (g == nullptr) return HT_ERR_INVALID_ARGUMENT;
  if constexpr (std::is_same<Real, float>::value) {
    ConvTileProblem t;
    if (saved_codes != nullptr) {
      unsigned char *records_at = static_cast<unsigned char *>(workspace) + conv_ordinal_bytes(a);
      if (!tile_problem(p, a, t) || conv_saved_code_bytes(t) == 0) return HT_ERR_INVALID_ARGUMENT;
      if (workspace_bytes < conv_ordinal_bytes(a) + conv_rows_workspace_bytes(t) + 256) return HT_ERR_WORKSPACE;
      const int params = conv_params_from_codes(t, x, thr, a.ord, w, g, gthr, gw, records_at, saved_codes, s);
      if (params != HT_OK || gx == nullptr) return params;
      return conv_image_from_saved_codes(t, g, gx, records_at, saved_codes, s);
    }
    if (tile_problem(p, a, t)) {
      const size_t records = conv_backward_tiled_workspace_bytes(t);
      if (records != 0 && workspace_bytes >= conv_ordinal_bytes(a) + records + 256) {
        unsigned char *ws = static_cast<unsigned char *>(workspace);
        const size_t codes_at = conv_ordinal_bytes(a) + conv_records_bytes(p, a) + 256;
        const size_t code_bytes = workspace_bytes > codes_at ? workspace_bytes - codes_at : 0;
        const int tiled = conv_backward_tiled(t, x, thr, a.ord, w, g, gx, gthr, gw, ws + conv_ordinal_bytes(a),
                                              code_bytes > 0 ? ws + codes_at : nullptr, code_bytes, status_word, s);
        if (tiled != HT_ERR_UNSUPPORTED) return tiled;
      }
    }
  }
  const int sorted = launch_backward_sorted<Real>(a, p->kind, g, gx, gthr, gw, s);
  if (sorted != HT_ERR_UNSUPPORTED) return sorted;
  auto kernel = p->kind == TREE ? conv_backward_kernel<TREE, Real> : conv_backward_kernel<FERN, Real>;
  kernel<<<blocks_for(threads), kBlock, 0, s>>>(a, g, gx, gthr, gw);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

}  // namespace
}  // namespace ht

using namespace ht;

extern "C" {

int ht_conv_output_size(const ht_conv_problem *p, int64_t *osize) {
  ConvArgs a;
  const int rc = check_conv(p, a);
  if (rc != HT_OK) return rc;
  if (osize == nullptr) return HT_ERR_INVALID_ARGUMENT;
  for (int d = 0; d < p->dims; ++d) osize[d] = a.osize[d];
  return HT_OK;
}

int ht_conv_backward_kernel(const ht_conv_problem *p, int real_bytes) {
  ConvArgs a;
  const int rc = check_conv(p, a);
  if (rc != HT_OK) return rc;
  if (real_bytes != 4 && real_bytes != 8) return HT_ERR_INVALID_ARGUMENT;
  ConvTileProblem t;
  if (real_bytes == 4 && tile_problem(p, a, t) && conv_backward_tiled_workspace_bytes(t) != 0) return HT_CONV_BACKWARD_TILES;
  const bool sorts = real_bytes == 4 ? sorting_is_better<float>(a, p->kind) : sorting_is_better<double>(a, p->kind);
  return sorts ? HT_CONV_BACKWARD_SORTED : HT_CONV_BACKWARD_SCATTERED;
}

size_t ht_conv_workspace_bytes(const ht_conv_problem *p) {
  ConvArgs a;
  if (check_conv(p, a) != HT_OK) return 0;
  return conv_ordinal_bytes(a) + conv_records_bytes(p, a) + 256;
}

size_t ht_conv_backward_workspace_bytes(const ht_conv_problem *p) {
  ConvArgs a;
  ConvTileProblem t;
  const size_t base = ht_conv_workspace_bytes(p);
  if (base == 0 || check_conv(p, a) != HT_OK || !tile_problem(p, a, t)) return base;
  const size_t per_sample = conv_code_bytes(t);
  if (per_sample == 0) return base;
  // Whole batches up to 8 GiB of codes, then a part of the batch at a time: parts of that size fill the machine many times over
  // (64 samples of 64 channels of 64 x 64 under 128 trees, 4.3 GB, are 16 ms of work), so more memory would buy nothing.
  const size_t samples = std::min<size_t>((size_t)p->B, std::max<size_t>(1, ((size_t)8 << 30) / per_sample));
  return base + samples * per_sample;
}

int ht_conv_forward_f32(const ht_conv_problem *p, const float *x, const float *thr, const int64_t *ord, const float *w,
                        float *out, void *workspace, size_t workspace_bytes, uint32_t *status_word, ht_stream_t stream) {
  return conv_forward<float>(p, x, thr, ord, w, out, workspace, workspace_bytes, status_word, stream);
}
size_t ht_conv_saved_bytes(const ht_conv_problem *p) {
  ConvShape a;
  ConvTileProblem t;
  if (check_conv(p, a) != HT_OK || !tile_problem(p, a, t)) return 0;
  return conv_saved_code_bytes(t);
}
int ht_conv_forward_saving_f32(const ht_conv_problem *p, const float *x, const float *thr, const int64_t *ord, const float *w,
                               float *out, void *kept, void *workspace, size_t workspace_bytes, uint32_t *status_word,
                               ht_stream_t stream) {
  if (kept == nullptr || (reinterpret_cast<uintptr_t>(kept) & 15u) != 0 || ht_conv_saved_bytes(p) == 0) return HT_ERR_INVALID_ARGUMENT;
  if (workspace_bytes < ht_conv_workspace_bytes(p)) return HT_ERR_WORKSPACE;
  return conv_forward<float>(p, x, thr, ord, w, out, workspace, workspace_bytes, status_word, stream, kept);
}
int ht_conv_backward_saved_f32(const ht_conv_problem *p, const float *x, const float *thr, const int64_t *ord, const float *w,
                               const float *g, float *gx, float *gthr, float *gw, const void *kept, void *workspace,
                               size_t workspace_bytes, uint32_t *status_word, ht_stream_t stream) {
  if (kept == nullptr || (reinterpret_cast<uintptr_t>(kept) & 15u) != 0 || ht_conv_saved_bytes(p) == 0) return HT_ERR_INVALID_ARGUMENT;
  return conv_backward<float>(p, x, thr, ord, w, g, gx, gthr, gw, workspace, workspace_bytes, status_word, stream, kept);
}
int ht_conv_forward_f64(const ht_conv_problem *p, const double *x, const double *thr, const int64_t *ord, const double *w,
                        double *out, void *workspace, size_t workspace_bytes, uint32_t *status_word, ht_stream_t stream) {
  return conv_forward<double>(p, x, thr, ord, w, out, workspace, workspace_bytes, status_word, stream);
}

int ht_conv_backward_f32(const ht_conv_problem *p, const float *x, const float *thr, const int64_t *ord, const float *w,
                         const float *g, float *gx, float *gthr, float *gw, void *workspace, size_t workspace_bytes,
                         uint32_t *status_word, ht_stream_t stream) {
  return conv_backward<float>(p, x, thr, ord, w, g, gx, gthr, gw, workspace, workspace_bytes, status_word, stream);
}
int ht_conv_backward_f64(const ht_conv_problem *p, const double *x, const double *thr, const int64_t *ord, const double *w,
                         const double *g, double *gx, double *gthr, double *gw, void *workspace, size_t workspace_bytes,
                         uint32_t *status_word, ht_stream_t stream) {
  return conv_backward<double>(p, x, thr, ord, w, g, gx, gthr, gw, workspace, workspace_bytes, status_word, stream);
}

int ht_contract(int dims, int elem_bytes, const void *image, void *patches, int64_t batch_times_channels,
                const int64_t *size, const int64_t *window, const int64_t *padding, ht_stream_t stream) {
  if (dims < 2 || dims > 3 || size == nullptr || window == nullptr || padding == nullptr) return HT_ERR_INVALID_ARGUMENT;
  int64_t osize[3];
  for (int d = 0; d < dims; ++d) {
    if (window[d] < 1 || padding[d] < 0 || window[d] > size[d] + 2 * padding[d]) return HT_ERR_INVALID_ARGUMENT;
    osize[d] = (size[d] + 2 * padding[d] - window[d]) / window[d] + 1;
  }
  return run_patches(true, dims, elem_bytes, image, patches, batch_times_channels, size, osize, window, padding,
                     reinterpret_cast<cudaStream_t>(stream));
}

int ht_expand(int dims, int elem_bytes, const void *patches, void *image, int64_t batch_times_channels,
              const int64_t *osize, const int64_t *window, const int64_t *padding, ht_stream_t stream) {
  if (dims < 2 || dims > 3 || osize == nullptr || window == nullptr || padding == nullptr) return HT_ERR_INVALID_ARGUMENT;
  int64_t size[3];
  for (int d = 0; d < dims; ++d) {
    if (window[d] < 1 || padding[d] < 0 || osize[d] < 1) return HT_ERR_INVALID_ARGUMENT;
    size[d] = osize[d] * window[d] - ((2 * padding[d]) / window[d]) * window[d];
    if (size[d] < 1) return HT_ERR_INVALID_ARGUMENT;
  }
  return run_patches(false, dims, elem_bytes, patches, image, batch_times_channels, size, osize, window, padding,
                     reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"
