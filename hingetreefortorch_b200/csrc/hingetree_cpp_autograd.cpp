// Autograd nodes of the operators that training steps are made of: plain forest / fern, fused linear, convolution, and the
// Linear -> BatchNorm1d -> forest step.  They do what the Function classes of HingeTree/_HingeTree.py describe, in C++: a
// small training step is host time, and a Python Function costs about 40 us of it (the backward's trip through the
// interpreter included).  A call that will not be differentiated runs the plain forward and builds no node.
#include <torch/extension.h>

#include <ATen/Context.h>
#include <c10/core/DeviceGuard.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include "hingetree_cpp_ops.h"

namespace htx {

namespace {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// Forward-mode derivatives count, with or without grad mode: the nodes refuse them, the plain forward would drop the tangents.
bool differentiated(std::initializer_list<const torch::Tensor *> tensors) {
  if (at::GradMode::is_enabled())
    for (const torch::Tensor *t : tensors)
      if (t->requires_grad()) return true;
  if (torch::autograd::ForwardADLevel::try_get_by_idx(0) != nullptr)  // a dual level is open
    for (const torch::Tensor *t : tensors)
      if (t->_fw_grad(/*level=*/0).defined()) return true;
  return false;
}

bool deterministic_mode() { return at::globalContext().deterministicAlgorithms(); }

void refuse_deterministic(const torch::Tensor &t, const std::string &what) {
  if (deterministic_mode() && !t.is_cpu()) bad_runtime("No deterministic implementation of " + what + " on GPUs.");
}

std::string name_of(int64_t kind) { return kind == HT_KIND_FERN ? "fern" : "tree"; }

// The forward keeps its traversal where the library offers that; the backward uses it once (it rewrites the scratch) and
// walks the trees again in a second backward through the same node.
struct PlainNode : public torch::autograd::Function<PlainNode> {
  static torch::Tensor forward(AutogradContext *ctx, const torch::Tensor &x, const torch::Tensor &thr, const torch::Tensor &ord,
                               const torch::Tensor &w, int64_t kind) {
    std::vector<torch::Tensor> result = forest_forward_saving((int)kind, x, thr, ord, w);
    ctx->save_for_backward({x, thr, ord, w});
    ctx->saved_data["kind"] = kind;
    if (result[1].numel() > 0) ctx->saved_data["kept"] = result[1];
    return result[0];
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const int kind = (int)ctx->saved_data["kind"].toInt();
    const bool need_x = ctx->needs_input_grad(0), need_thr = ctx->needs_input_grad(1), need_w = ctx->needs_input_grad(3);
    const torch::Tensor g = grads[0].contiguous();
    const auto kept = ctx->saved_data.find("kept");
    std::vector<torch::Tensor> r;
    if (kept != ctx->saved_data.end()) {
      const torch::Tensor scratch = kept->second.toTensor();
      ctx->saved_data.erase(kept);
      r = forest_backward_saved(kind, deterministic_mode(), saved[0], need_x, saved[1], need_thr, saved[2], false, saved[3], need_w, g,
                                scratch);
    } else {
      r = forest_backward(kind, deterministic_mode(), saved[0], need_x, saved[1], need_thr, saved[2], false, saved[3], need_w, g);
    }
    return {r[0], r[1], torch::Tensor(), r[3], torch::Tensor()};
  }
};

torch::Tensor plain_apply(int kind, const torch::Tensor &x, const torch::Tensor &thr, const torch::Tensor &ord, const torch::Tensor &w) {
  if (!differentiated({&x, &thr, &w})) return forest_forward(kind, x, thr, ord, w);
  return PlainNode::apply(x, thr, ord, w, (int64_t)kind);
}

struct LinearNode : public torch::autograd::Function<LinearNode> {
  static torch::Tensor forward(AutogradContext *ctx, const torch::Tensor &x, const torch::Tensor &thr, const torch::Tensor &ord,
                               const torch::Tensor &w, const torch::Tensor &lin, const torch::Tensor &bias, int64_t kind) {
    ctx->save_for_backward({x, thr, ord, w, lin, bias});
    ctx->saved_data["kind"] = kind;
    torch::Tensor scratch;
    const torch::Tensor out = linear_forward((int)kind, x, nullptr, thr, ord, w, lin, bias, &scratch);
    if (scratch.defined()) ctx->saved_data["kept"] = scratch;
    return out;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const int64_t kind = ctx->saved_data["kind"].toInt();
    refuse_deterministic(grads[0], "backpropagation for hinge " + name_of(kind) + " + linear");
    torch::Tensor scratch;  // used once: the backward rewrites it
    const auto kept = ctx->saved_data.find("kept");
    if (kept != ctx->saved_data.end()) {
      scratch = kept->second.toTensor();
      ctx->saved_data.erase(kept);
    }
    std::vector<torch::Tensor> r =
        linear_backward((int)kind, s[0], ctx->needs_input_grad(0), nullptr, false, s[1], ctx->needs_input_grad(1), s[2], false, s[3],
                        ctx->needs_input_grad(3), s[4], ctx->needs_input_grad(4), s[5], ctx->needs_input_grad(5), grads[0].contiguous(),
                        scratch.defined() ? &scratch : nullptr);
    r.push_back(torch::Tensor());
    return r;
  }
};

torch::Tensor linear_apply(int kind, const torch::Tensor &x, const torch::Tensor &thr, const torch::Tensor &ord, const torch::Tensor &w,
                           const torch::Tensor &lin, const torch::Tensor &bias) {
  refuse_deterministic(x, "forward for hinge " + name_of(kind) + " + linear");
  if (!differentiated({&x, &thr, &w, &lin, &bias})) return linear_forward(kind, x, nullptr, thr, ord, w, lin, bias);
  return LinearNode::apply(x, thr, ord, w, lin, bias, (int64_t)kind);
}

struct ConvNode : public torch::autograd::Function<ConvNode> {
  static torch::Tensor forward(AutogradContext *ctx, const torch::Tensor &x, const torch::Tensor &thr, const torch::Tensor &ord,
                               const torch::Tensor &w, const std::vector<int64_t> &geometry, int64_t kind) {
    ctx->save_for_backward({x, thr, ord, w});
    ctx->saved_data["kind"] = kind;
    ctx->saved_data["geometry"] = geometry;
    const Geometry g(geometry);
    torch::Tensor kept;
    const torch::Tensor out = conv_forward((int)kind, g.dims, x, thr, ord, w, g.part(0), g.part(1), g.part(2), g.part(3), &kept);
    if (kept.defined()) ctx->saved_data["kept"] = kept;
    return out;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const int64_t kind = ctx->saved_data["kind"].toInt();
    refuse_deterministic(grads[0], "backpropagation for hinge " + name_of(kind) + " convolution");
    const Geometry g(ctx->saved_data["geometry"].toIntVector());
    // The codes serve every backward through this node.  They go with the graph's buffers: saved_data lives as long as the output
    // is referenced, which in a training loop is until the next step's forward has taken as much again.
    const auto at = ctx->saved_data.find("kept");
    torch::Tensor kept;
    if (at != ctx->saved_data.end()) {
      kept = at->second.toTensor();
      if (!torch::autograd::get_current_graph_task_keep_graph()) ctx->saved_data.erase(at);
    }
    auto from = [&](const torch::Tensor *codes) {
      return conv_backward((int)kind, g.dims, s[0], ctx->needs_input_grad(0), s[1], ctx->needs_input_grad(1), s[2], false, s[3],
                           ctx->needs_input_grad(3), grads[0].contiguous(), g.part(0), g.part(1), g.part(2), g.part(3), codes);
    };
    std::vector<torch::Tensor> r;
    try {
      r = from(&kept);
    } catch (const c10::OutOfMemoryError &) {  // the codes may be in the way of what the backward cannot do without
      if (!kept.defined()) throw;
      kept.reset();
      ctx->saved_data.erase("kept");
    }
    if (r.empty()) r = from(nullptr);
    return {r[0], r[1], torch::Tensor(), r[3], torch::Tensor(), torch::Tensor()};
  }
  struct Geometry {  // kernel size, stride, padding and dilation one after another
    std::vector<int64_t> all;
    int dims;
    explicit Geometry(std::vector<int64_t> values) : all(std::move(values)), dims((int)all.size() / 4) {}
    std::vector<int64_t> part(int n) const { return {all.begin() + n * dims, all.begin() + (n + 1) * dims}; }
  };
};

torch::Tensor conv_apply(int kind, int dims, const torch::Tensor &x, const torch::Tensor &thr, const torch::Tensor &ord,
                         const torch::Tensor &w, const std::vector<int64_t> &kernel, const std::vector<int64_t> &stride,
                         const std::vector<int64_t> &padding, const std::vector<int64_t> &dilation) {
  const bool regular = kernel.size() == (size_t)dims && stride.size() == (size_t)dims && padding.size() == (size_t)dims &&
                       dilation.size() == (size_t)dims;
  if (!differentiated({&x, &thr, &w}) || !regular)  // (a geometry of the wrong length raises in the forward)
    return conv_forward(kind, dims, x, thr, ord, w, kernel, stride, padding, dilation);
  std::vector<int64_t> geometry;
  for (const std::vector<int64_t> *v : {&kernel, &stride, &padding, &dilation}) geometry.insert(geometry.end(), v->begin(), v->end());
  return ConvNode::apply(x, thr, ord, w, geometry, (int64_t)kind);
}

// torch.backends.cuda.matmul.allow_tf32 for the scope: the dense gradients of the projection are taken like its forward.
class AllowTf32 {
 public:
  AllowTf32() : before_(at::globalContext().allowTF32CuBLAS()) { at::globalContext().setAllowTF32CuBLAS(true); }
  ~AllowTf32() { at::globalContext().setAllowTF32CuBLAS(before_); }

 private:
  bool before_;
};

// forest((z - mean) * invstd) with z = x @ w.T and batch statistics, the normalised activations never written: the forest
// normalises the features it visits, and its backward hands the normalisation's backward one entry per (sample, tree) and
// the two column sums that it needs.
struct PipelineNode : public torch::autograd::Function<PipelineNode> {
  static variable_list forward(AutogradContext *ctx, const torch::Tensor &x_in, const torch::Tensor &w_in, const torch::Tensor &thr,
                               const torch::Tensor &ord, const torch::Tensor &leaves, double eps, int64_t kind) {
    const torch::Tensor x = x_in.contiguous(), w = w_in.contiguous();
    const std::vector<torch::Tensor> z = linear_tf32_stats(x, w), stats = batchnorm_statistics(z[1], z[2], x.size(0), eps);
    const std::vector<torch::Tensor> r = forest_normalised_forward((int)kind, z[0], stats[0], stats[2], thr, ord, leaves, true);
    ctx->save_for_backward({x, w, z[0], stats[0], stats[2], thr, ord, leaves, r[1], r[2]});
    ctx->saved_data["kind"] = kind;
    ctx->mark_non_differentiable({stats[0], stats[1]});
    ctx->set_materialize_grads(false);  // no zeros for the gradients of mean and variance
    return {r[0], stats[0], stats[1]};
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const std::vector<torch::Tensor> r =
        forest_normalised_backward((int)ctx->saved_data["kind"].toInt(), s[2], s[3], s[4], s[5], ctx->needs_input_grad(2), s[6], s[7],
                                   ctx->needs_input_grad(4), grads[0].contiguous(), s[8], s[9]);
    torch::Tensor gx, gw;
    {
      AllowTf32 allow;
      if (ctx->needs_input_grad(0)) gx = at::mm(r[0], s[1]);
      if (ctx->needs_input_grad(1)) gw = at::mm(r[0].t(), s[0]);
    }
    return {gx, gw, r[1], torch::Tensor(), r[2], torch::Tensor(), torch::Tensor()};
  }
};

torch::Tensor pipeline_apply(const torch::Tensor &x, const torch::Tensor &w, const torch::Tensor &thr, const torch::Tensor &ord,
                             const torch::Tensor &leaves, double eps, bool fern, torch::Tensor running_mean, torch::Tensor running_var,
                             torch::Tensor batches, double momentum) {
  const int64_t kind = fern ? HT_KIND_FERN : HT_KIND_TREE;
  variable_list out;
  if (differentiated({&x, &w, &thr, &leaves})) {
    out = PipelineNode::apply(x, w, thr, ord, leaves, eps, kind);
  } else {
    const torch::Tensor xc = x.contiguous(), wc = w.contiguous();
    const std::vector<torch::Tensor> z = linear_tf32_stats(xc, wc), stats = batchnorm_statistics(z[1], z[2], xc.size(0), eps);
    out = {forest_normalised_forward((int)kind, z[0], stats[0], stats[2], thr, ord, leaves, false)[0], stats[0], stats[1]};
  }
  batchnorm_running(out[1], out[2], x.size(0), momentum, running_mean, running_var, batches);
  return out[0];
}

// While torch.jit.trace records, what the extension computes by itself would end up in the trace as a constant.  A Python
// Function is recorded as an operation, so the call is made through one (_HingeTree.py, _Traced), which calls `name` again: then,
// and whenever the trace runs, straight through.
thread_local bool recording = false;
template <typename Compute, typename... Args>
torch::Tensor traceable(const std::string &name, Compute &&compute, const Args &...args) {
  if (!torch::jit::tracer::isTracing()) return compute(args...);
  if (recording) {  // the result stands for something the recorder has seen made
    const torch::Tensor out = compute(args...);
    torch::jit::tracer::setValueTrace(out, torch::jit::tracer::getValueTrace(at::empty({0}, out.options())));
    return out;
  }
  struct Recording {
    Recording() { recording = true; }
    ~Recording() { recording = false; }
  } scope;
  return pybind11::module_::import("hingetreefortorch_b200.HingeTree._HingeTree")
      .attr("_Traced")
      .attr("apply")(name, args...)
      .template cast<torch::Tensor>();
}

}  // namespace

void bind_autograd(pybind11::module_ &m) {
  for (const int kind : {HT_KIND_TREE, HT_KIND_FERN}) {
    const std::string prefix = name_of(kind), plain = prefix + "_apply", linear = prefix + "_fused_linear_apply";
    m.def(plain.c_str(), [kind, plain](const torch::Tensor &x, const torch::Tensor &t, const torch::Tensor &o, const torch::Tensor &w) {
      return traceable(plain, [kind](auto &...a) { return plain_apply(kind, a...); }, x, t, o, w);
    });
    m.def(linear.c_str(), [kind, linear](const torch::Tensor &x, const torch::Tensor &t, const torch::Tensor &o, const torch::Tensor &w,
                                         const torch::Tensor &l, const torch::Tensor &b) {
      return traceable(linear, [kind](auto &...a) { return linear_apply(kind, a...); }, x, t, o, w, l, b);
    });
    for (int dims = 1; dims <= 3; ++dims) {
      const std::string conv = prefix + "_conv" + std::to_string(dims) + "d_apply";
      m.def(conv.c_str(), [kind, dims, conv](const torch::Tensor &x, const torch::Tensor &t, const torch::Tensor &o,
                                             const torch::Tensor &w, const std::vector<int64_t> &k, const std::vector<int64_t> &s,
                                             const std::vector<int64_t> &p, const std::vector<int64_t> &d) {
        return traceable(conv, [kind, dims](auto &...a) { return conv_apply(kind, dims, a...); }, x, t, o, w, k, s, p, d);
      });
    }
  }
  m.def("linear_batchnorm_forest", &pipeline_apply,
        "One training-mode step forward of Linear -> BatchNorm1d(affine=False) -> forest / fern, differentiable; advances the "
        "running statistics in place.");
  m.def("batchnorm_running", &batchnorm_running,
        "Advances running mean, running (unbiased) variance and batch count in place by one batch's mean and biased variance.");
}

}  // namespace htx
