// Row-stationary kernels for tabular data with many features (ht_forest_rows.cu): whole rows of x or of its gradient in
// shared memory, the trees around them.
#pragma once

#include "ht_common.cuh"
#include "ht_eval_records.cuh"

namespace ht {

// The walk with the tree parameters in shared memory and the rows streaming past them.  What it leaves: the paths of all
// evaluations (threshold - feature at the deciding vertex; vertex and leaf key in the packing of the evaluation records)
// where `margin` and `where` are given, and the forest's output [B, T, M] where `out` is.
bool rows_forward_takes(const ht_forest_problem *p);
double rows_forward_cost(const ht_forest_problem *p);  // estimated microseconds; negative: not taken
int rows_forward(const ht_forest_problem *p, const float *x, const float *thr, const int32_t *ord, const float *w, float *out,
                 float *margin, void *where, uint32_t *status_word, cudaStream_t stream);

// gx [B, C] from records that hold the x-gradient terms (EvalRecords::dx), every element written; sums in free order.
bool rows_x_gradient_takes(const ht_forest_problem *p);
int rows_x_gradient(const ht_forest_problem *p, const int32_t *ord, const float *dx, const void *where, float *gx, cudaStream_t stream);

}  // namespace ht
