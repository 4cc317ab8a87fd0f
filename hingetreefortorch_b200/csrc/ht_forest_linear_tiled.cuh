// Forest with its linear layer on tabular data, from kept paths (ht_forest_linear_tiled.cu): single precision, one output
// per leaf, up to 16 linear outputs.
#pragma once

#include "ht_common.cuh"
#include "ht_eval_records.cuh"

namespace ht {

bool linear_tiled_takes(const ht_forest_problem *p, int64_t outputs);
size_t linear_tiled_bytes(const ht_forest_problem *p);  // scratch: the evaluation records

// out [B, outputs]; leaves the paths of all evaluations in `area` for the backward.  `ord`: packed ordinals.
int linear_tiled_forward(const ht_forest_problem *p, int64_t outputs, const float *x, const float *thr, const int32_t *ord,
                         const float *w, const float *lin, const float *bias, float *out, void *area, uint32_t *status_word,
                         cudaStream_t stream);

// The gradients from the paths in `area`, which `kept` says are there already.  gthr, gw and glin (null where not asked for)
// have been cleared; every element of gx is written.
int linear_tiled_backward(const ht_forest_problem *p, int64_t outputs, const float *x, const float *thr, const int32_t *ord,
                          const float *w, const float *lin, const float *g, float *gx, float *gthr, float *gw, float *glin,
                          void *area, bool kept, uint32_t *status_word, cudaStream_t stream);

}  // namespace ht
