// Shared-memory tile kernel for the forest forward (see ht_forest_tiled.cu).
#pragma once

#include "ht_common.cuh"

namespace ht {

// Bytes of per-tree records the tile kernel needs in the workspace (0 when the shape does not qualify).
// Without them the calls of such a shape are refused.
size_t forward_tiled_workspace_bytes(const ht_forest_problem *p);
// ... of inputs with inner positions that are served without tiles, too: several outputs per leaf, or one whose weights stay in
// global memory.  They lie behind everything else in the workspace, and a call that has no room for them takes another kernel.
size_t inner_spare_records_bytes(const ht_forest_problem *p);

// Estimated microseconds of the tile kernel on tabular data; negative: not taken.
double forward_tiled_cost(const ht_forest_problem *p);
// ... and on inputs with inner positions; `keep`: the paths of several outputs per leaf are left, too.
double inner_tiled_cost(const ht_forest_problem *p, bool keep);

// Runs the forward with the tile kernel when the shape qualifies; returns HT_ERR_UNSUPPORTED
// (and launches nothing) when it does not, so that the caller can use the any-shape kernel.
// `ord` are the compact (validated, clamped) int32 ordinals; `records` is 256-byte aligned
// scratch of forward_tiled_workspace_bytes() bytes, or of inner_spare_records_bytes().
// With `eval_records` (backward_records_bytes() bytes) and a problem for which forward_saves() holds, the forward
// also leaves its traversal there: the signed margin and the deciding vertex / leaf of every evaluation, from which
// backward_saved() computes the gradients without walking the trees again.  Several outputs per leaf: `eval_records` is
// the paths' area of ht_forest_multi.cuh (every shape), and with out == nullptr nothing but the paths is written.
bool forward_saves(const ht_forest_problem *p);
int saved_samples_per_cta(const ht_forest_problem *p);  // 0: the backward from saved records does not take the shape
// With `wide` the ordinals are packed into `ord` on the way to the records.
int forward_tiled(const ht_forest_problem *p, const float *x, const float *thr, int32_t *ord, const float *w,
                  float *out, void *records, void *eval_records, uint32_t *status_word, cudaStream_t stream,
                  const WideOrdinals *wide = nullptr);

// The backward from the records a saving forward left (either mode; forward_saves(p) must hold and the inputs must
// be the forward's).  `ord` are the compact ordinals.  Any of gx / gthr / gw may be null; the others must have been
// cleared.
int backward_saved(const ht_forest_problem *p, const int32_t *ord, const float *w, const float *g, float *gx, float *gthr,
                   float *gw, void *eval_records, cudaStream_t stream);

// Threshold and leaf-weight gradients (added to; null where not asked for) from records that hold the x-gradient and
// leaf-weight terms.
struct EvalRecords;
int reduce_parameter_terms(const ht_forest_problem *p, const EvalRecords &records, float *gthr, float *gw, cudaStream_t stream);

// Backward with the tile kernels of ht_forest_tiled_bwd.cu; same contract as forward_tiled.  With
// `eval_records` (backward_records_bytes() bytes of 256-byte aligned scratch; 0 = shape not
// supported) the traversal kernel writes per-evaluation records and two reduction kernels add
// them in the reference's order: deterministic, and the only tile path taken in HT_DETERMINISTIC
// mode.  Without it the traversal kernel scatters with global reductions (default mode only).
// Any of gx / gthr / gw may be null; the others must have been cleared.
size_t backward_records_bytes(const ht_forest_problem *p);
int backward_tiled(const ht_forest_problem *p, const float *x, const float *thr, const int32_t *ord, const float *w,
                   const float *g, float *gx, float *gthr, float *gw, void *records, void *eval_records,
                   uint32_t *status_word, cudaStream_t stream);

}  // namespace ht
