// Several outputs per leaf: forward that leaves its paths, and the backward that sorts them (ht_forest_multi.cu).
#pragma once

#include "ht_common.cuh"
#include "ht_eval_records.cuh"

namespace ht {

// Whether the kernels of ht_forest_multi.cu take the backward of this problem (any number of inner positions, several
// outputs per leaf), given a scratch area of multi_area_bytes() bytes for the paths.
bool multi_takes(const ht_forest_problem *p, size_t real_bytes);
size_t multi_area_bytes(const ht_forest_problem *p, size_t real_bytes);

// Bytes of the paths of all evaluations.
inline size_t path_bytes(const ht_forest_problem *p, size_t real_bytes) {
  return record_array_bytes(p, real_bytes) + record_array_bytes(p, where_bytes(p->depth));
}

// The paths of all evaluations inside that area: threshold - feature at the deciding vertex, and the deciding vertex
// with the leaf key, in the layout of the evaluation records.
template <typename Real>
struct PathRecordsOf {
  Real *margin;
  void *where;  // 8 + 8 bits up to depth 8, 16 + 16 beyond
};
template <typename Real>
PathRecordsOf<Real> multi_paths(const ht_forest_problem *p, void *area) {
  unsigned char *base = static_cast<unsigned char *>(area);
  return PathRecordsOf<Real>{reinterpret_cast<Real *>(base), base + record_array_bytes(p, sizeof(Real))};
}

// Forward of any shape with the results of a warp written together; where `paths` has a place for them it also leaves the
// paths, and with out == nullptr nothing else.  With `wide` the ordinals are read from there, not from `ord`, and all of them
// are checked on the way.  HT_ERR_UNSUPPORTED: nothing was launched.
template <typename Real>
int multi_forward(const ht_forest_problem *p, const Real *x, const Real *thr, const int32_t *ord, const Real *w, Real *out,
                  PathRecordsOf<Real> paths, cudaStream_t stream, const WideOrdinals *wide = nullptr, uint32_t *status_word = nullptr);

// Gradients from the paths in `area`, single precision (double precision scatters: ht_forest_backward_f64).  The gradients that are
// asked for (the others are null) must have been cleared.
int backward_multi(const ht_forest_problem *p, const int32_t *ord, const float *w, const float *g, float *gx, float *gthr,
                   float *gw, void *area, cudaStream_t stream);

// Fixed-order mode (ht_forest_ordered.cu), any number of outputs per leaf: bytes of the lists that the paths are sorted
// into (0: not for this problem), and the threshold and leaf-weight gradients from the paths.
size_t ordered_list_bytes(const ht_forest_problem *p, size_t real_bytes);
template <typename Real>
int ordered_parameters(const ht_forest_problem *p, const Real *w, const Real *g, Real *gthr, Real *gw, PathRecordsOf<Real> paths,
                       void *lists, cudaStream_t stream);

}  // namespace ht
