// Row-stationary kernels for tabular data with many features (ht_forest_rows.cu): whole rows of x or of its gradient in
// shared memory, the trees around them.
#pragma once

#include "ht_common.cuh"
#include "ht_eval_records.cuh"

namespace ht {

// The paths of all evaluations (threshold - feature at the deciding vertex; vertex and leaf key in the packing of the
// evaluation records) with the tree parameters in shared memory and the rows streaming past them.
bool rows_paths_takes(const ht_forest_problem *p);
int rows_paths(const ht_forest_problem *p, const float *x, const float *thr, const int32_t *ord, float *margin, void *where,
               uint32_t *status_word, cudaStream_t stream);

// gx [B, C] from records that hold the x-gradient terms (EvalRecords::dx), every element written; sums in free order.
bool rows_x_gradient_takes(const ht_forest_problem *p);
int rows_x_gradient(const ht_forest_problem *p, const int32_t *ord, const float *dx, const void *where, float *gx, cudaStream_t stream);

}  // namespace ht
