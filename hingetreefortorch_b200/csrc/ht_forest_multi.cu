// Forest and fern with several outputs per leaf: forward for any shape and the backward of every shape.
//
// multi_forward_kernel: thread per evaluation for the traversal, then the warp writes the outputs of its 32 evaluations
// together.
// sorted_backward_kernel: the paths of one tree and a slice of the samples are sorted by leaf in shared memory, after which
// the leaf-weight gradient of a leaf is a sum in registers.
#include "ht_counting_sort.cuh"
#include "ht_forest_multi.cuh"
#include "ht_tile_common.cuh"

#include <algorithm>

namespace ht {

namespace {

constexpr int kForwardThreads = 256;
constexpr int kSortThreads = 256;
constexpr int kMaxSortDepth = 12;
constexpr int64_t kMaxDivisor = 4096;

// p[0 .. V) += v where `now` is set, without a branch.
template <int V>
__device__ __forceinline__ void red_add_if(float *p, const float (&v)[V], bool now) {
  if constexpr (V == 4)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(p), "f"(v[0]),
                 "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"((int)now)
                 : "memory");
  else if constexpr (V == 2)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p red.global.add.v2.f32 [%0], {%1, %2};\n\t}" ::"l"(p), "f"(v[0]),
                 "f"(v[1]), "r"((int)now)
                 : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p red.global.add.f32 [%0], %1;\n\t}" ::"l"(p), "f"(v[0]), "r"((int)now)
                 : "memory");
}
// base + index without the second instruction that a 64-bit sum of two registers takes
__device__ __forceinline__ const float *element(const float *base, uint32_t index) {
  uint64_t at;
  asm("mad.wide.u32 %0, %1, 4, %2;" : "=l"(at) : "r"(index), "l"(base));
  return reinterpret_cast<const float *>(at);
}
// r = p[0 .. V) where `now` is set, without a branch
template <int V>
__device__ __forceinline__ void load_if(Vec<float, V> &r, const float *p, bool now) {
  if constexpr (V == 4)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "+f"(r.v[0]), "+f"(r.v[1]), "+f"(r.v[2]), "+f"(r.v[3])
                 : "l"(p), "r"((int)now));
  else if constexpr (V == 2)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p ld.global.nc.v2.f32 {%0, %1}, [%2];\n\t}"
                 : "+f"(r.v[0]), "+f"(r.v[1])
                 : "l"(p), "r"((int)now));
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p ld.global.nc.f32 %0, [%1];\n\t}" : "+f"(r.v[0]) : "l"(p), "r"((int)now));
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
  EvalDivisors by;
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
    int64_t i, j, k;
    a.by.split(e, a.T, a.K, i, j, k);
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

struct SortedArgs {
  const float *margin;
  const void *where;
  const int32_t *ord;
  const float *w, *g;
  float *gx, *gthr, *gw;
  int64_t T, C, N, L;
  Divisor K;           // positions per sample
  uint32_t P;          // evaluations per tree
  int M, depth, fern, narrow;
};

// CTAs per SM that the registers are shared out for
__host__ __device__ constexpr int sort_blocks(int numbers) { return numbers > 2 ? 3 : 4; }
// g rows (and rows of weights) in flight per group of lanes, as far as registers go
__host__ __device__ constexpr int sort_ahead(int numbers) { return numbers > 4 ? 2 : 4; }

// Evaluations per CTA: whole rounds for every group of lanes (three and five lanes per evaluation leave 80 and 48 groups).
__host__ __device__ constexpr uint32_t sort_slice(int lanes) { return lanes == 3 || lanes == 5 ? 960u : 1024u; }

// Place of the list entries without an evaluation, which fill up the last parts: they read the slice's first g row.
constexpr uint32_t kNobody = 1024;

// Lanes of three and five leave their parts of D to the evaluation's own thread; others add them up.
__host__ __device__ constexpr int sort_dots(int lanes) { return (lanes & (lanes - 1)) == 0 ? 1 : lanes; }

// Rows of eight lanes and more: the list holds the places of the g row and of the weights, so that no lane works them out
// (64 outputs: 56 -> 53 us).  Shorter rows are bound by the shared memory's wavefronts, to which a list of 16-byte entries adds
// (3 and 10 outputs: 56 us each, 60 with it).
__host__ __device__ constexpr bool sort_rows_listed(int lanes) { return lanes >= 8; }

// Where the arrays of sorted_backward_kernel lie in its shared memory; the counts, whose number varies, come last.
struct SortedPlaces {
  uint32_t dots, partial, bins;
};
__host__ __device__ constexpr SortedPlaces sorted_places(int lanes) {
  SortedPlaces at = {};
  const uint32_t slice = sort_slice(lanes), entries = slice + (uint32_t)(32 / lanes * (kSortThreads / 32));
  const uint32_t columns = kMaxSortDepth * kSortThreads * 4u;  // of the ferns' thresholds, in the list's place after the walk
  at.dots = entries * (sort_rows_listed(lanes) ? 16u : 8u);
  at.dots = at.dots < slice * 8u ? slice * 8u : at.dots;  // terms and vertices, after the walk as well
  at.dots = at.dots < columns ? columns : at.dots;
  at.partial = at.dots + (((kNobody + 1u) * (uint32_t)sort_dots(lanes) * 4u + 15u) & ~15u);
  at.bins = at.partial + ((4u * (kSortThreads / 32) + 15u) & ~15u);
  return at;
}
__host__ __device__ inline int sorted_bin_quads(int L, int N, bool fern) { return (L + (fern ? 0 : N) + 1 + 3) / 4; }

// Sums of dot[0 .. LEFT) over groups of 2 D lanes, D a power of two: lanes hand each other the halves of the list that they drop,
// as long as there is more than one number, so that sum u ends in the lanes whose upper bits (of the lane in its group) say u.
// Those bits are appended to `mine`; the lane is left with dot[0 .. LEFT / 2 D), at least one.
template <int D, int LEFT, int A>
__device__ __forceinline__ void sums_over_lanes(float (&dot)[A], int q, int &mine) {
  if constexpr (D >= 1) {
    if constexpr (LEFT > 1) {
      const bool upper = (q & D) != 0;
#pragma unroll
      for (int u = 0; u < LEFT / 2; ++u) {
        const float away = upper ? dot[u] : dot[u + LEFT / 2], kept = upper ? dot[u + LEFT / 2] : dot[u];
        dot[u] = kept + __shfl_xor_sync(0xffffffffu, away, D);
      }
      mine = mine * 2 + (upper ? 1 : 0);
    } else {
      dot[0] += __shfl_xor_sync(0xffffffffu, dot[0], D);
    }
    sums_over_lanes<D / 2, (LEFT > 1 ? LEFT / 2 : 1)>(dot, q, mine);
  }
}

// CTA per (tree, slice of its evaluations).
//
// The slice's paths are sorted by leaf by counting in shared memory.  LANES lanes share an evaluation (R pieces of V of its M
// outputs each), and every such group of lanes walks a contiguous part of the list: the evaluations of a leaf follow one
// another, so their |margin| * g are summed in registers and the leaf-weight gradient costs one reduction per leaf and group;
// the leaf's weights are loaded with the first of them, and D = sum over m of w * g comes from the same registers.  Where a
// leaf begins and ends is marked in the list when it is written, so that a step is straight code: two list loads, the g row,
// two products per output and a predicated reduction.
// D goes back to the evaluation's own thread, which adds it to the x gradient (neighbouring threads are neighbouring positions)
// and to the threshold sums: for trees through a second list, by deciding vertex, whose places were counted together with the
// leaves' (scatters would meet at the root and its neighbours); for ferns, whose few thresholds everybody meets in, through a
// column of shared memory per thread.
//
// What bounds it: issue slots (60 % used by 32 warps per SM) and the shared memory's wavefronts for short rows, the latency of
// the g rows for long ones.  4096 x 500 ferns of depth 10, 10 outputs: 83 -> 57 us; 10007 x 257 trees of depth 9, 3 outputs:
// 74 -> 57; x [8, 100, 32, 32], 100 trees of depth 7, 64 outputs (210 MB of g): 62 -> 53.  What had cost that: a test and a
// branch at every change of leaf, which with five or ten groups in a warp is every step (a predicated load and a predicated
// reduction instead; 24 -> 17.5 warp instructions per evaluation for the ferns), parts of the list that begin in the same bank,
// a batch of g rows that is waited for before the next is asked for (a ring instead), a second count for the vertices.
// Slices of 2048 and 4096 evaluations: ferns 98 and 137 us against 83 in the earlier form (registers).  Asking for the rows
// ahead of the sort (prefetches into L2): 65 -> 73 us.  Two rows in flight instead of four, in exchange for five or six CTAs per
// SM: ferns 57 and 73 us, 64 outputs 71 and 61.
template <int V, int LANES, int R>
__global__ void __launch_bounds__(kSortThreads, sort_blocks(R * V)) sorted_backward_kernel(const __grid_constant__ SortedArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kAhead = sort_ahead(R * V), kGroupsPerWarp = 32 / LANES, kGroups = kGroupsPerWarp * (kSortThreads / 32);
  constexpr uint32_t S = sort_slice(LANES);
  constexpr int PER = (int)((S + kSortThreads - 1) / kSortThreads);
  constexpr int kParts = sort_dots(LANES);
  static_assert(S % (kGroups * kAhead) == 0, "whole rounds");
  constexpr SortedPlaces at = sorted_places(LANES);
  constexpr bool kListed = sort_rows_listed(LANES);
  using Entry = typename std::conditional<kListed, uint4, uint2>::type;
  Entry *list = reinterpret_cast<Entry *>(smem);              // by leaf: {tag, |margin|}, and where listed {g row, weight row}
  float *dots = reinterpret_cast<float *>(smem + at.dots);      // by place in the slice: D, or its parts
  uint32_t *partial = reinterpret_cast<uint32_t *>(smem + at.partial);
  uint32_t *bins = reinterpret_cast<uint32_t *>(smem + at.bins);  // leaves, then vertices: counts, then first places
  float *by_vertex = reinterpret_cast<float *>(smem);               // after the walk: signed D by vertex, or the ferns' columns
  uint32_t *vertices = reinterpret_cast<uint32_t *>(by_vertex + S);  // ... and the vertices

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t j = blockIdx.x % (uint32_t)a.T;  // neighbouring trees run together: their g rows share sectors
  const uint32_t p0 = (uint32_t)(blockIdx.x / (uint32_t)a.T) * S;
  const int n = (int)min(S, a.P - p0);
  const int L = (int)a.L, N = a.fern ? 0 : (int)a.N;  // N: vertices that are counted
  const uint32_t K = a.K.number, M = (uint32_t)a.M;
  const uint32_t i0 = K == 1 ? p0 : a.K.quotient_above_one(p0);
  // tag: place in the slice | leaf << 12, whether there is an evaluation, and whether it is the first or the last of its leaf
  constexpr uint32_t kHere = 1u << 29, kFirst = 1u << 30, kLast = 1u << 31;
  // what a thread keeps of each of its evaluations: vertex (1-based) | place by vertex << 13 | sign of the margin
  constexpr uint32_t kPositive = 1u << 28, kNegative = 1u << 29;

  // every thread's evaluations tid, tid + 256, ... are loaded at once and stay in registers; `whole`: a full slice, all of them there
  uint32_t where[PER], keep[PER];
  float margin[PER];
  const int quads = sorted_bin_quads(L, N, a.fern != 0);
  const int share = ((n + kGroups - 1) / kGroups + kAhead - 1) / kAhead * kAhead;
  auto here = [&](int u, bool whole) {
    if (whole && (uint32_t)(u + 1) * kSortThreads <= S) return true;
    return tid + u * kSortThreads < (whole ? (int)S : n);
  };
  // g rows, from the one of sample i0's first position: evaluation p of the tree is row p + (samples before it) * (T - 1) * K
  const uint32_t from_first = p0 - i0 * K, skipped = ((uint32_t)a.T - 1u) * K;
  auto g_row = [&](uint32_t p) { return (p + (K == 1 ? p : a.K.quotient_above_one(p)) * skipped) * M; };
  auto make_list = [&](auto whole_slice) {
    constexpr bool whole = decltype(whole_slice)::value;
    const uint32_t sample = p0 + (uint32_t)tid, blocks = (uint32_t)a.T * kRecordBlock;
    const int64_t from = (int64_t)(sample / kRecordBlock) * blocks + j * kRecordBlock + sample % kRecordBlock;
    static_assert(kSortThreads == kRecordBlock, "a thread's evaluations are one record block apart");
    const float *margins = a.margin + from;
#pragma unroll
    for (int u = 0; u < PER; ++u) margin[u] = here(u, whole) ? -__ldg(margins + (int64_t)u * blocks) : 0.0f;
    if (a.narrow) {
      const unsigned short *wheres = static_cast<const unsigned short *>(a.where) + from;
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        where[u] = here(u, whole) ? __ldg(wheres + (int64_t)u * blocks) : 0u;
        where[u] = (where[u] & 0xffu) | (where[u] >> 8) << 16;
      }
    } else {
      const uint32_t *wheres = static_cast<const uint32_t *>(a.where) + from;
#pragma unroll
      for (int u = 0; u < PER; ++u) where[u] = here(u, whole) ? __ldg(wheres + (int64_t)u * blocks) : 0u;
    }
    for (int b = tid; b < quads; b += kSortThreads) reinterpret_cast<uint4 *>(bins)[b] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const uint32_t leaf = where[u] >> 16, vertex = where[u] & 0xffffu;
      keep[u] = vertex | (margin[u] > 0.0f ? kPositive : 0u) | (margin[u] < 0.0f ? kNegative : 0u);
      if (here(u, whole)) {
        if (N > 0) keep[u] |= atomicAdd(&bins[L - 1 + vertex], 1u) << 13;
        where[u] = leaf << 12 | atomicAdd(&bins[leaf], 1u);
      }
    }
    __syncthreads();
    exclusive_sums<kSortThreads>(reinterpret_cast<uint4 *>(bins), quads, partial);  // bins[L] = n, the first vertex's place + n
    const float per_share = 1.0f / (float)share;
    // the groups' parts lie one entry further apart than they are long: their reads fall into different banks
    auto slot_of = [&](uint32_t to) { return to + (uint32_t)(((float)to + 0.5f) * per_share); };
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      if (here(u, whole)) {
        const int t = tid + u * kSortThreads;
        const uint32_t leaf = where[u] >> 12, rank = where[u] & 0xfffu, next = bins[leaf + 1];
        const uint32_t to = bins[leaf] + rank;
        Entry entry = {};
        entry.x = (uint32_t)t | leaf << 12 | kHere | (rank == 0 ? kFirst : 0u) | (to + 1 == next ? kLast : 0u);
        if constexpr (kListed) {
          entry.z = g_row(from_first + (uint32_t)t);
          entry.w = leaf * M;
        }
        entry.y = __float_as_uint(fabsf(margin[u]));
        list[slot_of(to)] = entry;
        if (N > 0) keep[u] += (bins[L - 1 + (keep[u] & 0x1fffu)] - (uint32_t)n) << 13;
      }
    }
    if constexpr (!whole) {  // entries without an evaluation fill the last parts
      for (uint32_t to = (uint32_t)(n + tid); to < (uint32_t)(share * kGroups); to += kSortThreads) {
        Entry nobody = {};
        nobody.x = kNobody;
        if constexpr (kListed) nobody.z = g_row(from_first);
        list[slot_of(to)] = nobody;
      }
    }
  };
  if (n == (int)S)
    make_list(std::true_type{});
  else
    make_list(std::false_type{});
  __syncthreads();

  {
    // lanes left over (32 is no multiple of LANES) accompany the last group, and lanes beyond a row's end its first; neither
    // hands anything in
    const int group_in_warp = min(lane / LANES, kGroupsPerWarp - 1), q = lane - group_in_warp * LANES;
    const int part = warp * kGroupsPerWarp + group_in_warp;
    const Entry *my_list = list + part * (share + 1);
    bool on[R];
    uint32_t piece[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      on[r] = q < LANES && (q + r * LANES) * V < a.M;
      piece[r] = on[r] ? (uint32_t)((q + r * LANES) * V) : 0u;
    }
    const float *g_first = a.g + ((int64_t)i0 * a.T + j) * K * M;
    const float *w_first = a.w + j * L * M;
    const float *gw_first = a.gw + j * L * M;
    const bool want_w = a.gw != nullptr;
    float sums[R][V], weight[R][V];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int v = 0; v < V; ++v) sums[r][v] = weight[r][v] = 0.0f;
    auto hand_in = [&](uint32_t leaf_row, bool now) {
#pragma unroll
      for (int r = 0; r < R; ++r) red_add_if<V>(const_cast<float *>(element(gw_first, leaf_row + piece[r])), sums[r], now && on[r]);
    };
    // a ring of kAhead evaluations: their list entries, g rows, and the weights of the leaves that they enter
    Vec<float, V> rows[kAhead][R], entered[kAhead][R] = {};
    uint32_t tag[kAhead], leaf_row[kAhead];
    float size[kAhead];
    auto fetch = [&](int u, int t, bool enters) {
      const Entry entry = my_list[t];
      tag[u] = entry.x | (enters ? kFirst : 0u);
      size[u] = __uint_as_float(entry.y);
      uint32_t row;
      if constexpr (kListed) {
        row = entry.z;
        leaf_row[u] = entry.w;
      } else {
        row = g_row(from_first + (entry.x & (kNobody - 1u)));
        leaf_row[u] = ((entry.x >> 12) & 0xfffu) * M;
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        rows[u][r] = load_vec<float, V>(element(g_first, row + piece[r]));
        load_if<V>(entered[u][r], element(w_first, leaf_row[u] + piece[r]), (tag[u] & kFirst) != 0);
      }
    };
    auto round = [&](int t0, auto more) {
      uint32_t place[kAhead];
      float dot[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        place[u] = tag[u];
        dot[u] = 0.0f;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float mine = 0.0f;
#pragma unroll
          for (int v = 0; v < V; ++v) {
            weight[r][v] = (tag[u] & kFirst) ? entered[u][r].v[v] : weight[r][v];
            sums[r][v] += size[u] * rows[u][r].v[v];
            mine += weight[r][v] * rows[u][r].v[v];
          }
          dot[u] += kParts > 1 || on[r] ? mine : 0.0f;
        }
        hand_in(leaf_row[u], want_w && (tag[u] & kLast) != 0);
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int v = 0; v < V; ++v) sums[r][v] = (tag[u] & kLast) ? 0.0f : sums[r][v];
        if constexpr (decltype(more)::value) fetch(u, t0 + u + kAhead, false);
      }
      if constexpr (kParts > 1) {
        if (q < LANES) {
#pragma unroll
          for (int u = 0; u < kAhead; ++u) dots[(place[u] & (2u * kNobody - 1u)) * kParts + q] = dot[u];
        }
      } else {
        constexpr int kLists = LANES < kAhead ? LANES : kAhead, kEach = kAhead / kLists;  // sums that a lane is left with
        int mine = 0;
        sums_over_lanes<LANES / 2, kAhead>(dot, q, mine);
        if ((q & (LANES / kLists - 1)) == 0) {
#pragma unroll
          for (int e = 0; e < kEach; ++e) {
            uint32_t whose = place[e];
#pragma unroll
            for (int l = 1; l < kLists; ++l) whose = mine == l ? place[l * kEach + e] : whose;
            dots[whose & (2u * kNobody - 1u)] = dot[e];
          }
        }
      }
    };
#pragma unroll
    for (int u = 0; u < kAhead; ++u) fetch(u, u, u == 0);
    int t0 = 0;
    for (; t0 + kAhead < share; t0 += kAhead) round(t0, std::true_type{});
    round(t0, std::false_type{});
    if (want_w) {
      constexpr uint32_t kNone = 0xffffffffu;
      const uint32_t final = my_list[share - 1].x;
      // the leaf (its row) whose evaluations go on behind this group's part
      uint32_t current = (final & (kHere | kLast)) == kHere ? ((final >> 12) & 0xfffu) * M : kNone;
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
              const float other = __shfl_down_sync(0xffffffffu, sums[r][v], d * LANES);
              sums[r][v] += join ? other : 0.0f;
            }
        }
        const uint32_t before = __shfl_up_sync(0xffffffffu, current, LANES);
        if (group_in_warp > 0 && before == current) current = kNone;
      }
      hand_in(current, current != kNone);
    }
  }
  if (a.gx == nullptr && a.gthr == nullptr) return;
  __syncthreads();

  // thread per evaluation again
  if (a.fern && a.gthr != nullptr)
    for (int l = 0; l < (int)a.N; ++l) by_vertex[l * kSortThreads + tid] = 0.0f;
  auto finish = [&](auto whole_slice) {
    constexpr bool whole = decltype(whole_slice)::value;
    const int32_t *features = a.ord + j * a.N - 1;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      if (here(u, whole)) {
        const int t = tid + u * kSortThreads;
        float d = dots[t * kParts];
#pragma unroll
        for (int part = 1; part < kParts; ++part) d += dots[t * kParts + part];
        const uint32_t vertex = keep[u] & 0x1fffu;
        float term = (keep[u] & kPositive) ? d : -d;  // sign(margin) * D
        if ((keep[u] & (kPositive | kNegative)) == 0) term = 0.0f * d;
        if (a.gx != nullptr) {
          const uint32_t f = (uint32_t)__ldg(features + vertex);
          if (K == 1) {
            atomicAdd(a.gx + (int64_t)(p0 + (uint32_t)t) * a.C + f, term);
          } else {
            const uint32_t i = a.K.quotient_above_one(p0 + t), k = p0 + t - i * K;
            atomicAdd(a.gx + ((int64_t)i * a.C + f) * K + k, term);
          }
        }
        if (a.gthr != nullptr) {
          if (a.fern) {
            by_vertex[(vertex - 1) * kSortThreads + tid] += term;
          } else {
            const uint32_t to = (keep[u] >> 13) & 0x7fffu;
            by_vertex[to] = term;
            vertices[to] = vertex - 1;
          }
        }
      }
    }
  };
  if (n == (int)S)
    finish(std::true_type{});
  else
    finish(std::false_type{});
  if (a.gthr == nullptr) return;
  __syncthreads();
  if (a.fern) {
    for (int l = warp; l < (int)a.N; l += kSortThreads / 32) {
      float sum = 0.0f;
#pragma unroll
      for (int e = 0; e < kSortThreads; e += 32) sum += by_vertex[l * kSortThreads + e + lane];
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
      if (lane == 0) atomicAdd(a.gthr + j * a.N + l, -sum);
    }
    return;
  }
  // warps sum runs of 32
  for (int e0 = warp * 32; e0 < n; e0 += kSortThreads) {
    const int e = e0 + lane;
    float sum[1] = {e < n ? by_vertex[e] : 0.0f};
    const uint32_t vertex = e < n ? vertices[e] : 0xffffu;
    if (sums_of_runs(vertex, sum, lane) && e < n) atomicAdd(a.gthr + j * a.N + vertex, -sum[0]);
  }
}

template <int V, int LANES, int R>
int launch_sorted(const SortedArgs &a, cudaStream_t stream) {
  constexpr uint32_t slice = sort_slice(LANES);
  const int64_t grid = (int64_t)((a.P + slice - 1) / slice) * a.T;
  if (grid > 0x7fffffff) return HT_ERR_UNSUPPORTED;
  auto kernel = sorted_backward_kernel<V, LANES, R>;
  const size_t smem = sorted_places(LANES).bins + 16 * (size_t)sorted_bin_quads((int)a.L, (int)a.N, a.fern != 0);
  if (smem > 48 * 1024) HT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kernel<<<(unsigned)grid, kSortThreads, smem, stream>>>(a);
  HT_CHECK_LAUNCH();
  return HT_OK;
}

template <int V>
int launch_sorted_width(const SortedArgs &a, cudaStream_t stream) {
  // one load per lane and row up to half a warp per row (64 outputs: 68 us, with two loads and 8 lanes 78)
  const int pieces = (a.M + V - 1) / V;
  const bool one = pieces <= 16;
#define HT_SORTED(LANES, R) \
  if (pieces <= LANES * R && one == (R == 1)) return launch_sorted<V, LANES, R>(a, stream);
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
  a.by = EvalDivisors(a.evals, a.T, a.K);
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

int backward_multi(const ht_forest_problem *p, const int32_t *ord, const float *w, const float *g, float *gx, float *gthr,
                   float *gw, void *area, cudaStream_t stream) {
  if (!multi_takes(p, sizeof(float)) || (p->flags & HT_DETERMINISTIC) != 0) return HT_ERR_UNSUPPORTED;
  const PathRecordsOf<float> paths = multi_paths<float>(p, area);
  SortedArgs a = {};
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
  if ((int64_t)1024 * p->T * p->M + (int64_t)p->T * p->K * p->M > 0x7fffffff) return HT_ERR_UNSUPPORTED;  // g row offsets
  const int width = vector_width(p->M, sizeof(float), {w, g, gw});
  if (width == 1) return launch_sorted_width<1>(a, stream);
  if (width == 2) return launch_sorted_width<2>(a, stream);
  return launch_sorted_width<4>(a, stream);
}

template int multi_forward<float>(const ht_forest_problem *, const float *, const float *, const int32_t *, const float *,
                                  float *, PathRecordsOf<float>, cudaStream_t, const WideOrdinals *, uint32_t *);
template int multi_forward<double>(const ht_forest_problem *, const double *, const double *, const int32_t *, const double *,
                                   double *, PathRecordsOf<double>, cudaStream_t, const WideOrdinals *, uint32_t *);

}  // namespace ht
