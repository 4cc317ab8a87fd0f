// Forest and fern with several outputs per leaf: forward for any shape and the backward of every shape.
//
// multi_forward_kernel: thread per evaluation for the traversal, then the warp writes the outputs of its 32 evaluations
// together.
// sorted_backward_kernel: the paths of one tree and a slice of the samples are sorted by leaf in shared memory, after which
// the leaf-weight gradient of a leaf is a sum in registers.
#include "ht_forest_multi.cuh"
#include "ht_tile_common.cuh"

#include <algorithm>

namespace ht {

namespace {

constexpr int kForwardThreads = 256;
constexpr int kSortThreads = 256;
constexpr uint32_t kSlice = 1024;  // evaluations per CTA
constexpr int kMaxSortDepth = 12;
constexpr int64_t kMaxDivisor = 4096;

template <int V>
__device__ __forceinline__ void red_add(float *p, const float (&v)[V]) {
  if constexpr (V == 4) red_add_quad(p, v[0], v[1], v[2], v[3]);
  else if constexpr (V == 2) red_add_pair(p, v[0], v[1]);
  else atomicAdd(p, v[0]);
}
template <int V>
__device__ __forceinline__ void red_add(double *p, const double (&v)[V]) {
#pragma unroll
  for (int k = 0; k < V; ++k) atomicAdd(p + k, v[k]);
}

template <typename Real>
struct MultiForwardArgs {
  const Real *x, *thr, *w;
  const int32_t *ord;
  WideOrdinals wide;  // WIDE kernels
  uint32_t *status_word;
  Real *out;
  Real *margin;
  void *where;
  int64_t evals, T, C, K, N, L;
  int M, depth, narrow;
  uint32_t divide_M;  // ceil(2^32 / M): quotients of numbers below 32 M (0: M is too large for it)
};

// Bound by the traversal's gathers for few outputs per leaf and by writing them for many.  A thread that writes the M
// outputs of its own evaluation makes every store of the warp touch 32 rows; here the warp's outputs, which are 32 * M
// consecutive numbers, leave in 16-byte pieces that consecutive lanes own, each lane asking the evaluation's owner for
// |margin| and the leaf.  x [8, 100, 32, 32], 100 trees of depth 7, 8 x 8 outputs (210 MB): 287 -> 41 us.
template <int KIND, int V, bool WIDE, typename Real>
__global__ void __launch_bounds__(kForwardThreads) multi_forward_kernel(const __grid_constant__ MultiForwardArgs<Real> a) {
  const int64_t e = (int64_t)blockIdx.x * kForwardThreads + threadIdx.x;
  const int lane = threadIdx.x & 31;
  Real am = (Real)0;
  uint32_t leaf = 0;
  if (e < a.evals) {
    int64_t i, j, k = 0;
    if (a.K == 1) {
      i = e / a.T;
      j = e - i * a.T;
    } else {
      const int64_t ij = e / a.K;
      k = e - ij * a.K;
      i = ij / a.T;
      j = ij - i * a.T;
    }
    const PlainFeatureOf<Real> feat{a.x + i * a.C * a.K + k, a.K};
    PathOf<Real> p;
    if constexpr (WIDE) {
      // small calls: this launch checks the ordinals too, which a packing kernel would have done
      for (int64_t o = e; o < a.T * a.N; o += a.evals)
        if (!a.wide.valid(o) && a.status_word != nullptr) atomicOr(a.status_word, HT_FLAG_ORDINAL_RANGE);
      p = traverse<KIND>(feat, a.thr + j * a.N, WideOrdinals{a.wide.at + j * a.N, a.wide.channels}, a.depth);
    } else {
      p = traverse<KIND>(feat, a.thr + j * a.N, a.ord + j * a.N, a.depth);
    }
    am = abs_of(p.margin);
    leaf = (uint32_t)(j * a.L) + p.key;  // T * L < 2^32 (host)
    if (a.margin != nullptr) {
      const int64_t at = record_index(i * a.K + k, j, a.T);
      a.margin[at] = -p.margin;
      if (a.narrow)
        store_where<unsigned short>(a.where, at, p.vertex + 1, p.key);
      else
        store_where<uint32_t>(a.where, at, p.vertex + 1, p.key);
    }
  }
  if (a.out == nullptr) return;
  const int64_t first = e - lane;
  const int here = (int)max((int64_t)0, min((int64_t)32, a.evals - first));
  const int pieces = here * a.M / V;
  Real *out = a.out + first * a.M;
#pragma unroll 4
  for (int t = lane; t - lane < pieces; t += 32) {
    const uint32_t element = (uint32_t)t * V;
    const uint32_t owner = min(a.divide_M != 0 ? __umulhi(element, a.divide_M) : element / (uint32_t)a.M, 31u);
    const Real scale = __shfl_sync(0xffffffffu, am, (int)owner);
    const uint32_t row = __shfl_sync(0xffffffffu, leaf, (int)owner);
    if (t < pieces) {
      Vec<Real, V> r = load_vec<Real, V>(a.w + (int64_t)row * a.M + (element - owner * a.M));
#pragma unroll
      for (int v = 0; v < V; ++v) r.v[v] = mul_rn(scale, r.v[v]);
      *reinterpret_cast<Vec<Real, V> *>(out + element) = r;
    }
  }
}

// ---- backward, default mode ------------------------------------------------------------------------------------------

template <typename Real>
struct SortedArgs {
  const Real *margin;
  const void *where;
  const int32_t *ord;
  const Real *w, *g;
  Real *gx, *gthr, *gw;
  int64_t T, C, N, L;
  Divisor K;           // positions per sample
  uint32_t P;          // evaluations per tree
  int M, depth, fern, narrow;
  int exclusive;       // a CTA has all the evaluations of its tree
};

// g rows (and rows of weights) in flight per group of lanes, as far as registers go
template <typename Real>
__host__ __device__ constexpr int sort_ahead(int numbers) {
  return numbers * (int)sizeof(Real) > 16 ? 2 : 4;
}

// Turns counts[0 .. size) into the sums of what is before each (a run of them per thread).  All threads of the block.
template <int THREADS>
__device__ __forceinline__ void exclusive_sums(uint32_t *counts, int size, uint32_t *partial) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (size + THREADS - 1) / THREADS;
  const int first = min(tid * per, size), last = min(first + per, size);
  uint32_t mine = 0;
  for (int b = first; b < last; ++b) mine += counts[b];
  uint32_t sum = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t below = __shfl_up_sync(0xffffffffu, sum, d);
    if (lane >= d) sum += below;
  }
  if (lane == 31) partial[warp] = sum;
  __syncthreads();
  uint32_t base = sum - mine;
  for (int k = 0; k < warp; ++k) base += partial[k];
  for (int b = first; b < last; ++b) {
    const uint32_t count = counts[b];
    counts[b] = base;
    base += count;
  }
  __syncthreads();
}

// CTA per (tree, slice of its evaluations).
//
// The slice's paths are sorted by leaf, root decision first, by counting in shared memory.  `lanes` lanes share an
// evaluation (R pieces of V of its M outputs each), and every such group of lanes walks a contiguous part of the list:
//   * an evaluation of the same leaf as the one before adds |margin| * g to the leaf's sums in registers; only where the
//     leaf changes do they go to memory, so the leaf-weight gradient costs one reduction per leaf and group instead of
//     one per evaluation, and a plain store where nobody else can have a part of that leaf;
//   * the leaf's weights stay in registers as long as the leaf does, and D = sum over m of w * g needs no gather.
// D replaces the margin in the list.  Then a thread per evaluation adds it to the x gradient, and a second sort, by
// deciding vertex, gives every threshold gradient as a sum over a run of the list (scatters would meet at the root and its
// neighbours: 28 us of reductions into 257 x 511 thresholds for 2.6 million evaluations, CAS loops in shared memory 30).
//
// What bounds it: for long rows the latency of the g rows (x [8, 100, 32, 32], 100 trees, 64 outputs: 68 us for 210 MB,
// 228 us with a reduction per weight term), for short ones the issue slots (4096 x 500 ferns of depth 10, 10 outputs: 83 us
// against 95; 10007 x 257 trees of depth 9, 3 outputs: 68 against 164) and the L1's rate of one row per cycle: three
// pieces per lane instead of five lanes with one each cost 73 us for the first pass of the ferns, not 45.
// Slices of 1024 evaluations: the counts and the lists take 16 KB and the evaluations of a thread stay in registers;
// 4096 (16 evaluations per thread: 121 registers) run the ferns in 137 us.
template <typename Real, int V, int LANES, int R, int PER>
__global__ void __launch_bounds__(kSortThreads) sorted_backward_kernel(const __grid_constant__ SortedArgs<Real> a) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr uint32_t S = PER * kSortThreads;
  Real *values = reinterpret_cast<Real *>(smem);                 // by leaf: |margin|, later D
  uint32_t *offsets = reinterpret_cast<uint32_t *>(values + S);  // by leaf: g row, in numbers from the slice's first
  uint32_t *tags = offsets + S;                                  // by leaf: sign | level << 24 | path << 12 | place in the slice
  uint32_t *bins = tags + S;                                     // [L]: counts, then first places
  uint32_t *partial = bins + a.L;                                // [kSortThreads / 32]

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t j = blockIdx.x % (uint32_t)a.T;  // neighbouring trees run together: their g rows share sectors
  const uint32_t p0 = (uint32_t)(blockIdx.x / (uint32_t)a.T) * S;
  const int n = (int)min(S, a.P - p0);
  const int depth = a.depth, L = 1 << depth;
  const uint32_t i0 = a.K.quotient(p0), k0 = p0 - i0 * a.K.number;
  constexpr uint32_t kPositive = 1u << 28, kNegative = 1u << 29;

  // every thread's evaluations tid, tid + 256, ... are loaded at once and stay in registers while they are counted
  uint32_t where[PER];
  Real margin[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int t = tid + u * kSortThreads;
    const int64_t at = record_index((int64_t)p0 + t, j, a.T);
    where[u] = 0;
    margin[u] = (Real)0;
    if (t < n) {
      where[u] = a.narrow ? __ldg(static_cast<const unsigned short *>(a.where) + at) : __ldg(static_cast<const uint32_t *>(a.where) + at);
      margin[u] = -__ldg(a.margin + at);
    }
  }
  for (int b = tid; b < L; b += kSortThreads) bins[b] = 0;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    if (tid + u * kSortThreads < n) {
      const uint32_t packed = a.narrow ? unpack_where<unsigned short>(where[u]) : where[u];
      const uint32_t path = tile::bit_reverse(packed >> 16, depth), vertex = packed & 0xffffu;
      const uint32_t level = a.fern ? vertex - 1 : 31 - __clz((int)vertex);
      where[u] = level << 24 | path << 12 | atomicAdd(&bins[path], 1u);
    }
  }
  __syncthreads();
  exclusive_sums<kSortThreads>(bins, L, partial);
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int t = tid + u * kSortThreads;
    if (t < n) {
      const uint32_t to = bins[(where[u] >> 12) & 0xfffu] + (where[u] & 0xfffu);
      const uint32_t sign = margin[u] > (Real)0 ? kPositive : margin[u] < (Real)0 ? kNegative : 0u;
      const uint32_t i = a.K.quotient(p0 + t), k = p0 + t - i * a.K.number;
      values[to] = abs_of(margin[u]);
      offsets[to] = ((i - i0) * (uint32_t)a.T * a.K.number + k - k0) * (uint32_t)a.M;
      tags[to] = sign | (where[u] & 0xffff000u) | (uint32_t)t;
    }
  }
  __syncthreads();

  {
    constexpr int kAhead = sort_ahead<Real>(R * V), kGroupsPerWarp = 32 / LANES, groups = kGroupsPerWarp * (kSortThreads / 32);
    const int group_in_warp = lane / LANES, q = lane % LANES;
    const int share = ((n + groups - 1) / groups + kAhead - 1) / kAhead * kAhead;
    const bool idle = group_in_warp >= kGroupsPerWarp;  // lanes left over
    const int begin = idle ? n : min((warp * kGroupsPerWarp + group_in_warp) * share, n);
    const int end = min(begin + share, n);
    const Real *g_first = a.g + (((int64_t)i0 * a.T + j) * a.K.number + k0) * a.M + q * V;
    Real sums[R][V], weight[R][V];
    bool on[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      on[r] = (q + r * LANES) * V < a.M;
#pragma unroll
      for (int v = 0; v < V; ++v) sums[r][v] = weight[r][v] = (Real)0;
    }
    constexpr uint32_t kNone = 0xffffffffu;
    uint32_t current = kNone;  // the leaf (path) whose sums are in the registers
    bool whole = false;        // all of its evaluations are in this group's part

    auto leave = [&]() {
      if (a.gw == nullptr || current == kNone) return;
      Real *row = a.gw + (j * L + tile::bit_reverse(current, depth)) * a.M + q * V;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (on[r]) {
          Real *to = row + r * LANES * V;
          if (whole) {
            Vec<Real, V> out;
#pragma unroll
            for (int v = 0; v < V; ++v) out.v[v] = sums[r][v];
            *reinterpret_cast<Vec<Real, V> *>(to) = out;
          } else {
            red_add<V>(to, sums[r]);
          }
        }
    };
    auto walk_list = [&](int t0, auto no_bounds) {
      constexpr bool full = decltype(no_bounds)::value;
      Vec<Real, V> rows[kAhead][R], entered[kAhead][R];  // g rows, and the weights of the leaves that this round enters
      uint32_t path[kAhead];
      Real dot[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int t = t0 + u;
        path[u] = full || t < end ? (tags[t] >> 12) & 0xfffu : kNone;
        if (full || t < end) {
          const Real *row = g_first + (int32_t)offsets[t];
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (on[r]) rows[u][r] = load_vec<Real, V>(row + r * LANES * V);
          if (path[u] != (u == 0 ? current : path[u == 0 ? 0 : u - 1])) {
            const Real *leaf = a.w + (j * L + tile::bit_reverse(path[u], depth)) * a.M + q * V;
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (on[r]) entered[u][r] = load_vec<Real, V>(leaf + r * LANES * V);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int t = t0 + u;
        dot[u] = (Real)0;
        if (full || t < end) {
          if (path[u] != current) {
            leave();
            current = path[u];
            if (a.exclusive) {
              const int run_end = current + 1 < (uint32_t)L ? (int)bins[current + 1] : n;
              whole = run_end <= end && (int)bins[current] >= begin;
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int v = 0; v < V; ++v) {
                sums[r][v] = (Real)0;
                weight[r][v] = entered[u][r].v[v];
              }
          }
          const Real size = values[t];
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (on[r]) {
#pragma unroll
              for (int v = 0; v < V; ++v) {
                sums[r][v] += size * rows[u][r].v[v];
                dot[u] += weight[r][v] * rows[u][r].v[v];
              }
            }
        }
      }
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) {
        if (d >= LANES) continue;
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const Real other = __shfl_down_sync(0xffffffffu, dot[u], d);
          if (q + d < LANES || (LANES & (LANES - 1)) == 0) dot[u] += other;  // (powers of two: only lane q = 0 is read)
        }
      }
      __syncwarp();  // the margins of this round have been read
      if (q == 0) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          if (full || t0 + u < end) values[t0 + u] = dot[u];
      }
    };
    // the groups of a warp go through their parts together; only a warp that holds the list's end, or lanes left over,
    // has short parts
    if (__all_sync(0xffffffffu, begin + share == end))
      for (int t0 = begin; t0 < begin + share; t0 += kAhead) walk_list(t0, std::true_type{});
    else
      for (int t0 = begin; t0 < begin + share; t0 += kAhead) walk_list(t0, std::false_type{});
    // groups of the warp that end in the same leaf hand in one sum (23 million evaluations of 22 trees of depth 4, 2 outputs:
    // 495 us; 1293 when all 256 groups of a slice met in 16 leaves)
    if constexpr (kGroupsPerWarp > 1) {
#pragma unroll
      for (int d = 1; d < kGroupsPerWarp; d <<= 1) {
        const bool join = __shfl_down_sync(0xffffffffu, current, d * LANES) == current && group_in_warp + d < kGroupsPerWarp;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const Real other = __shfl_down_sync(0xffffffffu, sums[r][v], d * LANES);
            if (join) sums[r][v] += other;
          }
      }
      const uint32_t before = __shfl_up_sync(0xffffffffu, current, LANES);
      if (group_in_warp > 0 && before == current) current = kNone;
    }
    leave();
  }
  if (a.gx == nullptr && a.gthr == nullptr) return;
  __syncthreads();

  // thread per evaluation: x gradient, and the evaluations of every vertex are counted
  for (int b = tid; b < L; b += kSortThreads) bins[b] = 0;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int t = tid + u * kSortThreads;
    if (t < n) {
      const uint32_t tag = tags[t];
      const Real d = values[t];
      margin[u] = (tag & kPositive) ? d : (tag & kNegative) ? -d : (Real)0 * d;  // sign(margin) * D
      const int level = (int)(tag >> 24) & 0xf;
      const uint32_t vertex = a.fern ? (uint32_t)level : (1u << level | ((tag >> 12) & 0xfffu) >> (depth - level)) - 1u;
      if (a.gx != nullptr) {
        const uint32_t p = p0 + (tag & 0xfffu);
        const uint32_t i = a.K.quotient(p), k = p - i * a.K.number;
        atomicAdd(a.gx + ((int64_t)i * a.C + __ldg(a.ord + j * a.N + vertex)) * a.K.number + k, margin[u]);
      }
      if (a.gthr != nullptr) where[u] = vertex << 12 | atomicAdd(&bins[vertex], 1u);
    }
  }
  if (a.gthr == nullptr) return;
  __syncthreads();
  const int N = (int)a.N;
  exclusive_sums<kSortThreads>(bins, N, partial);
#pragma unroll
  for (int u = 0; u < PER; ++u)
    if (tid + u * kSortThreads < n) {
      const uint32_t to = bins[where[u] >> 12] + (where[u] & 0xfffu);
      values[to] = margin[u];  // every D and tag is in registers by now
      tags[to] = where[u] >> 12;
    }
  __syncthreads();
  // warps sum runs of 32: a lane adds what is d lanes above while that is the same vertex
  for (int e0 = warp * 32; e0 < n; e0 += kSortThreads) {
    const int e = e0 + lane;
    Real sum = e < n ? values[e] : (Real)0;
    const uint32_t vertex = e < n ? tags[e] : 0xffffu;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const Real other = __shfl_down_sync(0xffffffffu, sum, d);
      const uint32_t whose = __shfl_down_sync(0xffffffffu, vertex, d);
      if (lane + d < 32 && whose == vertex) sum += other;
    }
    const uint32_t before = __shfl_up_sync(0xffffffffu, vertex, 1);
    if (e < n && (lane == 0 || before != vertex)) atomicAdd(a.gthr + j * N + vertex, -sum);
  }
}

template <typename Real, int V, int LANES, int R>
int launch_sorted(const SortedArgs<Real> &a, unsigned grid, size_t smem, cudaStream_t stream) {
  auto kernel = sorted_backward_kernel<Real, V, LANES, R, kSlice / kSortThreads>;
  if (smem > 48 * 1024) HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kernel<<<grid, kSortThreads, smem, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

template <typename Real, int V>
int launch_sorted_width(const SortedArgs<Real> &a, unsigned grid, size_t smem, cudaStream_t stream) {
  // one load per lane and row up to half a warp per row (64 outputs: 68 us, with two loads and 8 lanes 78)
  const int pieces = (a.M + V - 1) / V;
  const bool one = pieces <= 16;
#define HT_SORTED(LANES, R) \
  if (pieces <= LANES * R && one == (R == 1)) return launch_sorted<Real, V, LANES, R>(a, grid, smem, stream);
  HT_SORTED(1, 1)
  HT_SORTED(2, 1)
  HT_SORTED(3, 1)
  HT_SORTED(4, 1)
  HT_SORTED(5, 1)
  HT_SORTED(8, 1)
  HT_SORTED(16, 1)
  HT_SORTED(16, 2)
  HT_SORTED(32, 2)
#undef HT_SORTED
  return HT_ERR_UNSUPPORTED;
}

template <int KIND, bool WIDE, typename Real>
int launch_forward(const MultiForwardArgs<Real> &a, int width, cudaStream_t stream) {
  const unsigned grid = (unsigned)((a.evals + kForwardThreads - 1) / kForwardThreads);
  if (width == 1)
    multi_forward_kernel<KIND, 1, WIDE, Real><<<grid, kForwardThreads, 0, stream>>>(a);
  else if (width == 2)
    multi_forward_kernel<KIND, 2, WIDE, Real><<<grid, kForwardThreads, 0, stream>>>(a);
  else if constexpr (sizeof(Real) == 4)
    multi_forward_kernel<KIND, 4, WIDE, Real><<<grid, kForwardThreads, 0, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

}  // namespace

bool multi_takes(const ht_forest_problem *p, size_t real_bytes) {
  if (p->M < 2 || p->M > 64 || p->depth > kMaxSortDepth || p->B * p->K > 0x7fffffff) return false;
  if (p->T * (((int64_t)1) << p->depth) > 0xffffffffll || p->T < 1) return false;
  // below, the kernels that sort wait longer for their launches than the scatters take
  return p->B * p->K * p->T >= 32768;
}

// Up to 32 GiB, like the records of one output per leaf: the forward keeps the paths until the backward, and in between the
// program needs its memory for what it computes from the outputs.  Larger problems scatter; a caller's limit may be lower.
size_t multi_area_bytes(const ht_forest_problem *p, size_t real_bytes) {
  if (!multi_takes(p, real_bytes)) return 0;
  const size_t bytes = path_bytes(p, real_bytes);
  return bytes <= ((size_t)32 << 30) ? bytes : 0;
}

template <typename Real>
int multi_forward(const ht_forest_problem *p, const Real *x, const Real *thr, const int32_t *ord, const Real *w, Real *out,
                  PathRecordsOf<Real> paths, cudaStream_t stream, const WideOrdinals *wide, uint32_t *status_word) {
  MultiForwardArgs<Real> a = {};
  a.evals = p->B * p->T * p->K;
  a.T = p->T;
  a.C = p->C;
  a.K = p->K;
  a.N = threshold_count(p->kind, p->depth);
  a.L = ((int64_t)1) << p->depth;
  if (p->M < 1 || p->M > (1 << 26) || a.T * a.L > 0xffffffffll || a.evals > ((int64_t)kForwardThreads << 31) - kForwardThreads)
    return HT_ERR_UNSUPPORTED;
  a.x = x;
  a.thr = thr;
  a.w = w;
  a.ord = ord;
  a.out = out;
  a.M = (int)p->M;
  a.depth = p->depth;
  a.narrow = where_bytes(p->depth) == 2;
  a.divide_M = p->M > kMaxDivisor ? 0 : (uint32_t)(((1ull << 32) + p->M - 1) / (uint64_t)p->M);
  a.margin = paths.margin;
  a.where = paths.where;
  const int width = vector_width(p->M, sizeof(Real), {w, out});
  if (wide != nullptr) {
    a.wide = *wide;
    a.status_word = status_word;
    return p->kind == TREE ? launch_forward<TREE, true>(a, width, stream) : launch_forward<FERN, true>(a, width, stream);
  }
  return p->kind == TREE ? launch_forward<TREE, false>(a, width, stream) : launch_forward<FERN, false>(a, width, stream);
}

template <typename Real>
int backward_multi(const ht_forest_problem *p, const int32_t *ord, const Real *w, const Real *g, Real *gx, Real *gthr,
                   Real *gw, void *area, cudaStream_t stream) {
  if (!multi_takes(p, sizeof(Real)) || (p->flags & HT_DETERMINISTIC) != 0) return HT_ERR_UNSUPPORTED;
  const PathRecordsOf<Real> paths = multi_paths<Real>(p, area);
  SortedArgs<Real> a = {};
  a.margin = paths.margin;
  a.where = paths.where;
  a.ord = ord;
  a.w = w;
  a.g = g;
  a.gx = gx;
  a.gthr = gthr;
  a.gw = gw;
  a.T = p->T;
  a.C = p->C;
  a.N = threshold_count(p->kind, p->depth);
  a.L = ((int64_t)1) << p->depth;
  a.P = (uint32_t)(p->B * p->K);
  a.K = Divisor((uint32_t)p->K);
  a.M = (int)p->M;
  a.depth = p->depth;
  a.fern = p->kind == FERN;
  a.narrow = where_bytes(p->depth) == 2;
  constexpr uint32_t slice = kSlice;
  a.exclusive = a.P <= slice;
  const int64_t grid = (int64_t)((a.P + slice - 1) / slice) * p->T;
  if (grid > 0x7fffffff) return HT_ERR_UNSUPPORTED;
  if ((int64_t)slice * p->T * p->M + (int64_t)p->T * p->K * p->M > 0x7fffffff) return HT_ERR_UNSUPPORTED;  // g row offsets
  const size_t smem = (size_t)slice * (sizeof(Real) + 8) + 4 * (size_t)(a.L + kSortThreads / 32);
  const int width = vector_width(p->M, sizeof(Real), {w, g, gw});
  if (width == 1) return launch_sorted_width<Real, 1>(a, (unsigned)grid, smem, stream);
  if (width == 2) return launch_sorted_width<Real, 2>(a, (unsigned)grid, smem, stream);
  if constexpr (sizeof(Real) == 4) return launch_sorted_width<Real, 4>(a, (unsigned)grid, smem, stream);
  return HT_ERR_UNSUPPORTED;
}

template int multi_forward<float>(const ht_forest_problem *, const float *, const float *, const int32_t *, const float *,
                                  float *, PathRecordsOf<float>, cudaStream_t, const WideOrdinals *, uint32_t *);
template int multi_forward<double>(const ht_forest_problem *, const double *, const double *, const int32_t *, const double *,
                                   double *, PathRecordsOf<double>, cudaStream_t, const WideOrdinals *, uint32_t *);
template int backward_multi<float>(const ht_forest_problem *, const int32_t *, const float *, const float *, float *, float *,
                                   float *, void *, cudaStream_t);
template int backward_multi<double>(const ht_forest_problem *, const int32_t *, const double *, const double *, double *,
                                    double *, double *, void *, cudaStream_t);

}  // namespace ht
