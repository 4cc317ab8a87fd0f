// Helpers shared by the translation units of the `hingetree_cpp` torch extension.
#pragma once

#include <torch/extension.h>

#include <string>
#include <vector>

#include "hingetree_b200.h"

namespace htx {

[[noreturn]] void bad_argument(const std::string &what);  // std::invalid_argument -> ValueError
[[noreturn]] void bad_runtime(const std::string &what);   // std::runtime_error -> RuntimeError
void raise_status(int rc, const char *op);

ht_stream_t current_stream(const torch::Tensor &t);
int64_t inner_count(const torch::Tensor &t, int64_t from);
int depth_of(int64_t leaves);
int64_t threshold_count(int kind, int depth);
void require_cuda(const torch::Tensor &t);
void require_float32(const torch::Tensor &t);
torch::Tensor make_workspace(size_t bytes, const torch::Tensor &like);
// Uninitialised contiguous memory on `like`'s device.  Straight from the allocator: torch.empty costs 2.5 us of dispatch, and
// in deterministic mode a launch that fills it (with what every operator here overwrites).
torch::Tensor fresh(c10::IntArrayRef sizes, const torch::Tensor &like, c10::ScalarType type);
inline torch::Tensor fresh(c10::IntArrayRef sizes, const torch::Tensor &like) { return fresh(sizes, like, like.scalar_type()); }
inline torch::Tensor fresh_like(const torch::Tensor &like) { return fresh(like.sizes(), like); }
int64_t backward_scratch_limit();              // set by the caller; see hingetree_cpp.cpp
bool may_keep(int64_t bytes);                  // from a forward to its backward, by the caller's settings
bool may_keep(const torch::Tensor &scratch);
void set_ordinal_check(const std::string &mode);
int64_t pipeline_status();

// Owns the device status word of one call and turns a flagged ordinal into the reference's
// RuntimeError.  When this ordinals tensor is already known to be valid nothing is read back and word() is the
// device's long-lived status word, which keeps a kernel's timeout flag for the next call that synchronises.
class OrdinalGuard {
 public:
  OrdinalGuard(const torch::Tensor &ord, int64_t channels);
  uint32_t *word();
  void finish();

 private:
  torch::Tensor ord_, word_, sticky_;
  int64_t channels_;
  bool check_;
};

// Argument checks and shape bookkeeping of the plain forest operators.
struct ForestCall {
  // allow_double: torch.float64 tensors are taken too (the plain operators have double precision kernels)
  ForestCall(int kind, const torch::Tensor &x, const torch::Tensor &thr, const torch::Tensor &ord,
             const torch::Tensor &w, const torch::Tensor *g, bool allow_double = false);
  ht_forest_problem problem;
  bool is_double = false;
  std::vector<int64_t> out_sizes;  // [B, T, inner data dims..., inner weight dims...]
  std::vector<int64_t> map_sizes;  // [B, T, inner data dims...]
};

// The operators that the autograd nodes are made of (hingetree_cpp.cpp, hingetree_cpp_more.cpp).
torch::Tensor forest_forward(int kind, torch::Tensor x, torch::Tensor thr, torch::Tensor ord, torch::Tensor w);
std::vector<torch::Tensor> forest_forward_saving(int kind, torch::Tensor x, torch::Tensor thr, torch::Tensor ord, torch::Tensor w);
std::vector<torch::Tensor> forest_backward(int kind, bool deterministic, torch::Tensor x, bool need_x, torch::Tensor thr, bool need_thr,
                                           torch::Tensor ord, bool need_ord, torch::Tensor w, bool need_w, torch::Tensor g);
std::vector<torch::Tensor> forest_backward_saved(int kind, bool deterministic, torch::Tensor x, bool need_x, torch::Tensor thr,
                                                 bool need_thr, torch::Tensor ord, bool need_ord, torch::Tensor w, bool need_w,
                                                 torch::Tensor g, torch::Tensor saved);
// `scratch`: receives the forward's workspace, which holds the paths of all evaluations, where it may be kept; given to the
// backward it saves it another walk.
torch::Tensor linear_forward(int kind, torch::Tensor data, const torch::Tensor *vec, torch::Tensor thr, torch::Tensor ord,
                             torch::Tensor w, torch::Tensor lin, torch::Tensor bias, torch::Tensor *scratch = nullptr);
std::vector<torch::Tensor> linear_backward(int kind, torch::Tensor data, bool need_data, const torch::Tensor *vec, bool need_vec,
                                           torch::Tensor thr, bool need_thr, torch::Tensor ord, bool need_ord, torch::Tensor w,
                                           bool need_w, torch::Tensor lin, bool need_lin, torch::Tensor bias, bool need_bias,
                                           torch::Tensor g, const torch::Tensor *scratch = nullptr);
// `kept`: receives the codes of all evaluations where the library and the caller's settings provide for that; a backward that is
// given them does not walk, and leaves them as they are.
torch::Tensor conv_forward(int kind, int dims, torch::Tensor x, torch::Tensor thr, torch::Tensor ord, torch::Tensor w,
                           std::vector<int64_t> kernel, std::vector<int64_t> stride, std::vector<int64_t> padding,
                           std::vector<int64_t> dilation, torch::Tensor *kept = nullptr);
std::vector<torch::Tensor> conv_backward(int kind, int dims, torch::Tensor x, bool need_x, torch::Tensor thr, bool need_thr,
                                         torch::Tensor ord, bool need_ord, torch::Tensor w, bool need_w, torch::Tensor g,
                                         std::vector<int64_t> kernel, std::vector<int64_t> stride, std::vector<int64_t> padding,
                                         std::vector<int64_t> dilation, const torch::Tensor *kept = nullptr);
std::vector<torch::Tensor> linear_tf32_stats(torch::Tensor x, torch::Tensor w);
std::vector<torch::Tensor> batchnorm_statistics(torch::Tensor sum, torch::Tensor sumsq, int64_t rows, double eps);
void batchnorm_running(torch::Tensor mean, torch::Tensor var, int64_t rows, double momentum, torch::Tensor running_mean,
                       torch::Tensor running_var, torch::Tensor batches);
std::vector<torch::Tensor> forest_normalised_forward(int kind, torch::Tensor z, torch::Tensor mean, torch::Tensor invstd,
                                                     torch::Tensor thr, torch::Tensor ord, torch::Tensor w, bool keep);
std::vector<torch::Tensor> forest_normalised_backward(int kind, torch::Tensor z, torch::Tensor mean, torch::Tensor invstd,
                                                      torch::Tensor thr, bool need_thr, torch::Tensor ord, torch::Tensor w,
                                                      bool need_w, torch::Tensor g, torch::Tensor margin, torch::Tensor where);

// Registers the autograd nodes (hingetree_cpp_autograd.cpp).
void bind_autograd(pybind11::module_ &m);

// Registers the convolution, fused-linear, fusion, sparse, trie and contract/expand operators.
void bind_more_ops(pybind11::module_ &m);

// Median initialisation of the thresholds (CPU tensors, in place); false when the shapes or the
// feature indices do not describe a forest over the data.
enum class InitFamily { Tree, Fern, Trie };
bool init_medians(InitFamily family, torch::Tensor x, torch::Tensor thr, torch::Tensor ord, torch::Tensor w);

// Greedy initialisation of a forest's thresholds and feature indices from class labels (CPU tensors, in
// place), drawing from a process-wide generator that seed_init() resets.
bool init_greedy(torch::Tensor x, torch::Tensor labels, torch::Tensor thr, torch::Tensor ord, torch::Tensor w);
void seed_init(uint64_t seed);

}  // namespace htx
