// Fixed-order parameter gradients of the forest backward from the paths of all evaluations.
//
// The reference adds one term per (sample, position, output) into every threshold and leaf weight in that order, so each
// gradient element is a chain of dependent additions that no split of the samples may break.  What can be split is
// everything else: ordered_sort_kernel lists every tree's evaluations by leaf and by deciding vertex, keeping their order,
// and ordered_sum_kernel forms the terms with many threads and adds them with one lane per chain.
#include "ht_forest_multi.cuh"
#include "ht_tile_common.cuh"

#include <algorithm>

namespace ht {

namespace {

constexpr int kSortBlock = 512;
constexpr int kSumBlock = 256;
constexpr int kMaxOrderedDepth = 12;
constexpr size_t kTermBytes = 16 * 1024;  // of one of the two buffers of terms

// What a sort leaves: for each tree the positions by leaf (kind 0) or deciding vertex (kind 1), and where a bin's begin.
struct OrderedLists {
  uint32_t *list[2];   // [T][P]
  void *value[2];      // [T][P]: of the listed position |margin| (kind 0), or leaf key << 2 | -sign(margin) + 1 (kind 1)
  uint32_t *first[2];  // [T][bins + 1]
};

template <typename Real>
struct OrderedArgs {
  const Real *margin;
  const void *where;
  const Real *w, *g;
  Real *gthr, *gw;
  OrderedLists lists;
  int64_t T, K, P, N, L, M;
  int depth, narrow, warps, parts;
};

template <typename Real>
__device__ __forceinline__ uint32_t where_at(const OrderedArgs<Real> &a, int64_t at) {
  return a.narrow ? unpack_where<unsigned short>(__ldg(static_cast<const unsigned short *>(a.where) + at))
                  : __ldg(static_cast<const uint32_t *>(a.where) + at);
}

// CTA per (tree, kind): counting sort that keeps the order.  A warp owns consecutive positions and has counts of its own,
// so that the place of a position is its warp's first place in the bin plus how many of the warp's positions came before.
template <typename Real>
__global__ void __launch_bounds__(kSortBlock) ordered_sort_kernel(const __grid_constant__ OrderedArgs<Real> a) {
  extern __shared__ uint32_t counts[];  // [warps][bins]
  __shared__ uint32_t partial[kSortBlock / 32];
  const int kind = blockIdx.y;
  if ((kind == 0 ? a.gw : a.gthr) == nullptr) return;
  const int bins = (int)(kind == 0 ? a.L : a.N);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x;
  const int64_t j = blockIdx.x;
  uint32_t *list = a.lists.list[kind] + j * a.P, *first = a.lists.first[kind] + j * (bins + 1);
  for (int b = tid; b < a.warps * bins; b += threads) counts[b] = 0;
  __syncthreads();
  const int64_t share = ((a.P + a.warps - 1) / a.warps + 31) / 32 * 32;
  const int64_t begin = min((int64_t)warp * share, a.P), end = min(begin + share, a.P);
  uint32_t *mine = counts + warp * bins;
  constexpr uint32_t kNone = 0xffffffffu;
  // use(position, bin, lanes of the same bin) for 32 positions at a time; the bins of four rounds are loaded ahead
  auto for_each_round = [&](auto &&use) {
    constexpr int kAhead = 4;
    for (int64_t p0 = begin; p0 < end; p0 += 32 * kAhead) {
      uint32_t bin[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int64_t p = p0 + 32 * u + lane;
        bin[u] = kNone;
        if (p < end) {
          const uint32_t where = where_at(a, record_index(p, j, a.T));
          bin[u] = kind == 0 ? where >> 16 : (where & 0xffffu) - 1u;
        }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        use(p0 + 32 * u + lane, bin[u], __match_any_sync(0xffffffffu, bin[u]));
        __syncwarp();
      }
    }
  };
  for_each_round([&](int64_t, uint32_t bin, unsigned peers) {
    if (bin != kNone && lane == __ffs((int)peers) - 1) mine[bin] += __popc(peers);
  });
  __syncthreads();
  // counts become first places: over the warps of a bin, then over the bins
  uint32_t base = 0;
  for (int b0 = 0; b0 < bins; b0 += threads) {
    const int b = b0 + tid;
    uint32_t total = 0;
    if (b < bins)
      for (int k = 0; k < a.warps; ++k) total += counts[k * bins + b];
    uint32_t sum = total;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t below = __shfl_up_sync(0xffffffffu, sum, d);
      if (lane >= d) sum += below;
    }
    if (lane == 31) partial[warp] = sum;
    __syncthreads();
    uint32_t all = 0, place = base + sum - total;
    for (int k = 0; k < threads / 32; ++k) {
      if (k < warp) place += partial[k];
      all += partial[k];
    }
    if (b < bins) {
      first[b] = place;
      for (int k = 0; k < a.warps; ++k) {
        const uint32_t count = counts[k * bins + b];
        counts[k * bins + b] = place;
        place += count;
      }
    }
    base += all;
    __syncthreads();
  }
  if (tid == 0) first[bins] = (uint32_t)a.P;
  for_each_round([&](int64_t p, uint32_t bin, unsigned peers) {
    const uint32_t at = bin != kNone ? mine[bin] : 0u;
    __syncwarp();
    if (bin != kNone) {
      const uint32_t to = at + __popc(peers & ((1u << lane) - 1u));
      const int64_t record = record_index(p, j, a.T);
      const Real behind = __ldg(a.margin + record);  // threshold - feature
      list[to] = (uint32_t)p;
      if (kind == 0)
        static_cast<Real *>(a.lists.value[0])[j * a.P + to] = abs_of(behind);
      else
        static_cast<uint32_t *>(a.lists.value[1])[j * a.P + to] = (where_at(a, record) >> 16) << 2 | (uint32_t)((int)sign_of(behind) + 1);
      if (lane == __ffs((int)peers) - 1) mine[bin] = at + __popc(peers);
    }
  });
}

// acc + t[0] + t[stride] + .. in this order, the next sixteen numbers always under way (16 additions take 64 clocks, a
// load from shared memory about 30); neighbouring numbers (STRIDE 1; else `stride` apart) come 16 bytes at a time.
template <int STRIDE, typename Real>
__device__ __forceinline__ void load_links(const Real *t, Real (&to)[16], int stride) {
  if constexpr (STRIDE == 1) {
    constexpr int kPerLoad = 16 / (int)sizeof(Real);
#pragma unroll
    for (int u = 0; u < 16; u += kPerLoad) {
      const uint4 q = *reinterpret_cast<const uint4 *>(t + u);
#pragma unroll
      for (int v = 0; v < kPerLoad; ++v) to[u + v] = reinterpret_cast<const Real *>(&q)[v];
    }
  } else {
#pragma unroll
    for (int u = 0; u < 16; ++u) to[u] = t[u * stride];
  }
}
template <int STRIDE, typename Real>
__device__ __forceinline__ Real chain(const Real *t, int n, Real acc, int stride) {
  constexpr int kAhead = 16;
  int e = 0;
  if (STRIDE == 1)
    for (; e < n && (reinterpret_cast<uintptr_t>(t + e) & 15u) != 0; ++e) acc = add_rn(acc, t[e]);
  if (n - e >= kAhead) {
    Real now[kAhead], next[kAhead];
    load_links<STRIDE>(t + e * stride, now, stride);
    for (; e + 3 * kAhead <= n; e += 2 * kAhead) {
      load_links<STRIDE>(t + (e + kAhead) * stride, next, stride);
#pragma unroll
      for (int u = 0; u < kAhead; ++u) acc = add_rn(acc, now[u]);
      load_links<STRIDE>(t + (e + 2 * kAhead) * stride, now, stride);
#pragma unroll
      for (int u = 0; u < kAhead; ++u) acc = add_rn(acc, next[u]);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) acc = add_rn(acc, now[u]);
    e += kAhead;
  }
  while (e < n) {  // the rest: loads together, none past the end
    Real rest[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) rest[u] = t[min(e + u, n - 1) * stride];
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (e + u < n) acc = add_rn(acc, rest[u]);
    e += kAhead;
  }
  return acc;
}

// CTA per (tree, part of its bins, kind).  All warps but the first turn rows of the list into terms in shared memory, one
// buffer ahead of the first warp, which adds them in order.  Leaf weights (kind 0): a lane per output, one addition per
// position, 32 outputs per CTA.  Thresholds (kind 1): a position's M terms follow one another in the same chain.  A bin is
// in one part only: the part that its first position falls into when the list is cut evenly.
// Bound by the chain of the fullest bin, 4 clocks per addition (data in [0, 1] under thresholds in [-3, 3]: many samples
// decide at one vertex).  8192 x 784, 100 trees of depth 7, 10 outputs: 248 us, of which the longest
// chain (81920 terms at one vertex) is 172 (266 with seven producing warps and the adding one always the first); one warp per
// tree that walked and added in turn took 7476.  Measured and not faster: three CTAs per SM instead of two (284), one (313), the outcomes
// of pieces of a chain worked out ahead for the binade that the sum is in (270 to 460).
template <typename Real>
__global__ void __launch_bounds__(kSumBlock) ordered_sum_kernel(const __grid_constant__ OrderedArgs<Real> a) {
  __shared__ __align__(16) unsigned char buffers[2][kTermBytes];
  const int kind = blockIdx.z == 0 ? 1 : 0;  // the thresholds' longer chains start first
  if ((kind == 0 ? a.gw : a.gthr) == nullptr) return;
  const int m0 = kind == 0 ? 32 * ((int)blockIdx.z - 1) : 0;
  const int width = kind == 0 ? (int)min((int64_t)32, a.M - m0) : (int)a.M;  // terms per position
  const int bins = (int)(kind == 0 ? a.L : a.N);
  const int tid = threadIdx.x, lane = tid & 31;
  // Which warp does what: 0 adds, kIdle would share its scheduler (a warp's number modulo 4) and with it the issue slots that the
  // chain of additions asks for every fourth clock, the others produce.  CTAs that are likely to share an SM (148 are launched at
  // a time) add on different schedulers.
  constexpr int kIdle = 4;
  const uint32_t cta = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  const int warp = ((tid >> 5) + (int)((cta / 148) & 3u)) & (kSumBlock / 32 - 1);
  const bool produces = warp != 0 && warp != kIdle;
  const int64_t j = blockIdx.x;
  const uint32_t *list = a.lists.list[kind] + j * a.P, *first = a.lists.first[kind] + j * (bins + 1);
  // the first bin that begins at or after part / parts of the list: as many as begin before it
  auto bin_at = [&](int64_t part) {
    int before = 0;
    for (int b0 = 0; b0 < bins; b0 += kSumBlock) {
      const int b = b0 + tid;
      before += __syncthreads_count(b < bins && (int64_t)__ldg(first + b) * a.parts < part * a.P);
    }
    return before;
  };
  const Real *sizes = static_cast<const Real *>(a.lists.value[0]) + j * a.P;
  const uint32_t *keys = static_cast<const uint32_t *>(a.lists.value[1]) + j * a.P;
  int bin = bin_at(blockIdx.y);
  const int last_bin = bin_at((int64_t)blockIdx.y + 1);
  if (bin >= last_bin) return;
  const int64_t begin = __ldg(first + bin), end = __ldg(first + last_bin);
  constexpr int kTerms = (int)(kTermBytes / sizeof(Real));
  // A warp produces terms of 32 / lanes positions at a time.  A position with more terms than a buffer holds is cut into
  // pieces (kind 1).
  const int piece = min(width, kTerms), pieces = (width + piece - 1) / piece;
  int lanes = 1;
  while (lanes < 32 && lanes < piece) lanes *= 2;
  // (whole loads and whole turns of the adding loop, where a bin goes on)
  const int pitch = kind == 0 ? lanes : piece, room = max(1, kTerms / pitch), rows = room >= 32 ? room & ~31 : room;
  const int64_t steps = ((end - begin + rows - 1) / rows) * pieces;

  auto produce = [&](int64_t step) {
    Real *to = reinterpret_cast<Real *>(buffers[step & 1]);
    const int64_t row0 = begin + step / pieces * rows;
    const int count = (int)min((int64_t)rows, end - row0);
    const int from = (int)(step % pieces) * piece, here = min(piece, width - from);
    constexpr int kAhead = 8, kWarps = kSumBlock / 32 - 2;
    const int per_warp = 32 / lanes;
    const int m_lane = lane % lanes, first_row = (warp < kIdle ? warp - 1 : warp - 2) * per_warp + lane / lanes;
    for (int m = m_lane; m - m_lane < here; m += lanes) {
      const bool on = m < here;
      const int mc = min(m, here - 1);  // lanes and rows past the end load what their neighbours load, and store nothing
      for (int r0 = first_row; r0 - first_row < count; r0 += kWarps * per_warp * kAhead) {
        int64_t at[kAhead];
        Real weight[kAhead], up[kAhead];
        uint32_t value[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const int64_t row = row0 + min(r0 + u * kWarps * per_warp, count - 1);
          at[u] = __ldg(list + row);
          if (kind == 0) weight[u] = __ldg(sizes + row);
          else value[u] = __ldg(keys + row);
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const int64_t i = a.K == 1 ? at[u] : (int64_t)((uint32_t)at[u] / (uint32_t)a.K);
          at[u] = ((i * a.T + j) * a.K + (at[u] - i * a.K)) * a.M + m0 + from + mc;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          up[u] = __ldg(a.g + at[u]);
          if (kind == 1) weight[u] = mul_rn((Real)((int)(value[u] & 3u) - 1), __ldg(a.w + (j * a.L + (value[u] >> 2)) * a.M + from + mc));
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const int r = r0 + u * kWarps * per_warp;
          if (r < count && on) to[r * pitch + m] = mul_rn(weight[u], up[u]);
        }
      }
    }
  };

  if (produces) produce(0);
  __syncthreads();
  Real acc = (Real)0;
  int64_t row = begin, bin_end = __ldg(first + bin + 1);  // the adding warp's place in the list
  auto next_bin = [&]() {  // hands in full bins and passes empty ones
    while (bin < last_bin && row >= bin_end) {
      if (bin_end > (int64_t)__ldg(first + bin)) {
        if (kind == 0) {
          if (lane < width) a.gw[(j * a.L + bin) * a.M + m0 + lane] = acc;
        } else if (lane == 0) {
          a.gthr[j * a.N + bin] = acc;
        }
      }
      acc = (Real)0;
      if (++bin < last_bin) bin_end = __ldg(first + bin + 1);
    }
  };
  if (warp == 0) next_bin();
  for (int64_t step = 0; step < steps; ++step) {
    if (warp != 0) {
      if (produces && step + 1 < steps) produce(step + 1);
    } else {
      const Real *from = reinterpret_cast<const Real *>(buffers[step & 1]);
      const int64_t row0 = begin + step / pieces * rows;
      const int64_t row_end = min(row0 + rows, end);
      const int here = kind == 0 ? pitch : min(piece, width - (int)(step % pieces) * piece);
      while (row < row_end) {
        const int n = (int)(min(bin_end, row_end) - row);
        const Real *term = from + (row - row0) * here;
        if (kind == 0) {
          acc = chain<0>(term + lane % lanes, n, acc, pitch);
        } else {
          acc = chain<1>(term, n * here, acc, 1);
          if (step % pieces + 1 < pieces) break;  // the position goes on in the next buffer
        }
        row += n;
        next_bin();
      }
    }
    __syncthreads();
  }
}

}  // namespace

size_t ordered_list_bytes(const ht_forest_problem *p, size_t real_bytes) {
  const int64_t P = p->B * p->K;
  if (p->depth > kMaxOrderedDepth || P > 0x7fffffff || P < 1 || p->T < 1 || p->T > 0x7fffffff || p->M < 1) return 0;
  const int64_t N = threshold_count(p->kind, p->depth), L = ((int64_t)1) << p->depth;
  return 3 * align_up((size_t)(p->T * P) * 4, 256) + align_up((size_t)(p->T * P) * real_bytes, 256) +
         align_up((size_t)(p->T * (L + 1)) * 4, 256) + align_up((size_t)(p->T * (N + 1)) * 4, 256);
}

template <typename Real>
int ordered_parameters(const ht_forest_problem *p, const Real *w, const Real *g, Real *gthr, Real *gw, PathRecordsOf<Real> paths,
                       void *lists, cudaStream_t stream) {
  if (gthr == nullptr && gw == nullptr) return HT_OK;
  OrderedArgs<Real> a = {};
  a.margin = paths.margin;
  a.where = paths.where;
  a.w = w;
  a.g = g;
  a.gthr = gthr;
  a.gw = gw;
  a.T = p->T;
  a.K = p->K;
  a.P = p->B * p->K;
  a.N = threshold_count(p->kind, p->depth);
  a.L = ((int64_t)1) << p->depth;
  a.M = p->M;
  a.depth = p->depth;
  a.narrow = where_bytes(p->depth) == 2;
  unsigned char *at = static_cast<unsigned char *>(lists);
  const size_t list = align_up((size_t)(p->T * a.P) * 4, 256);
  a.lists.list[0] = reinterpret_cast<uint32_t *>(at);
  a.lists.list[1] = reinterpret_cast<uint32_t *>(at + list);
  a.lists.value[1] = at + 2 * list;
  a.lists.value[0] = at + 3 * list;
  at += 3 * list + align_up((size_t)(p->T * a.P) * sizeof(Real), 256);
  a.lists.first[0] = reinterpret_cast<uint32_t *>(at);
  a.lists.first[1] = reinterpret_cast<uint32_t *>(at + align_up((size_t)(p->T * (a.L + 1)) * 4, 256));
  // as many warps as have 128 positions each, and counts that leave room for two CTAs per SM
  a.warps = kSortBlock / 32;
  while (a.warps > 1 && ((a.P + a.warps - 1) / a.warps < 128 || (size_t)a.warps * (size_t)a.L * 4 > 100 * 1024)) a.warps /= 2;
  const size_t counts = (size_t)a.warps * (size_t)a.L * 4;
  auto sort = ordered_sort_kernel<Real>;
  if (counts > 48 * 1024) HT_CUDA_TRY(cudaFuncSetAttribute(sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)counts));
  sort<<<dim3((unsigned)p->T, 2), a.warps * 32, counts, stream>>>(a);
  HT_CHECK_LAUNCH();
  // parts: six CTAs on every SM, as long as a part has rows for its warps
  const int64_t slices = (p->M + 31) / 32 + 1;
  if (slices > 65535) return HT_ERR_UNSUPPORTED;
  const int64_t fill = std::max<int64_t>(1, 6 * 148 / (p->T * slices));
  a.parts = (int)std::min<int64_t>({fill, 64, std::max<int64_t>(1, a.P / 64)});
  ordered_sum_kernel<Real><<<dim3((unsigned)p->T, (unsigned)a.parts, (unsigned)slices), kSumBlock, 0, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

template int ordered_parameters<float>(const ht_forest_problem *, const float *, const float *, float *, float *,
                                       PathRecordsOf<float>, void *, cudaStream_t);
template int ordered_parameters<double>(const ht_forest_problem *, const double *, const double *, double *, double *,
                                        PathRecordsOf<double>, void *, cudaStream_t);

}  // namespace ht
