// PyTorch side of the package: autograd nodes and argument handling of the ops, in C++ on top of the C ABI of
// libd2conv3d.so (which knows nothing about torch).  Built into d2conv3d_b200/_C.so.
//
// Why native: one pass of a small layer is a dozen kernels of a few microseconds each, and the same front-end written in
// Python (checks, descriptor, output allocation, a Python autograd function that the engine calls back under the
// interpreter lock) took 280 us of host time per forward + backward, four times what the GPU needs.  Here the engine runs
// the backward without the interpreter.
//
// Interfaces it stands in for: csrc/ops/dconv3d.h:70-226 (DeformConv3dFunction, deform_conv3d), csrc/ops/dconv1d.h:69-186,
// fast-depthwise-conv3d/csrc/grouped_conv3d.h:29-106, and the half-precision up-cast of deform_conv.py:54-59.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/cuda/Event.h>
#include <torch/extension.h>

#include <array>
#include <atomic>
#include <mutex>
#include <optional>
#include <vector>

#include "d2conv3d.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using Triple = std::array<int64_t, 3>;
using OptTensor = std::optional<Tensor>;

// ---- helpers --------------------------------------------------------------------------------------------

// TORCH_CHECK(expr) of the reference reads "Expected <expr> to be true ..."
#define D2C_REQUIRE(cond, text) TORCH_CHECK(cond, "Expected " text " to be true, but got false.")

void check(int status, const char* what) {
  TORCH_CHECK(status == 0, what, ": ", d2c_status_string(status), status > 0 ? ": " : "",
              status > 0 ? d2c_last_cuda_error() : "", " (status ", status, ")");
}

Tensor get(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
Tensor contiguous(const Tensor& t) { return t.defined() ? t.contiguous() : t; }
Tensor like(const Tensor& t) { return t.defined() ? at::empty_like(t, at::MemoryFormat::Contiguous) : t; }
Tensor bytes_on(size_t n, const Tensor& t) {
  return n ? at::empty({(int64_t)n}, t.options().dtype(at::kByte).requires_grad(false)) : Tensor();
}
void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// deform_conv.py:15-16,54-59: if any tensor is fp16, every tensor is converted to fp32 and the result stays fp32
void upcast_if_any_half(std::initializer_list<Tensor*> tensors) {
  bool half = false;
  for (Tensor* t : tensors) half |= t->defined() && t->scalar_type() == at::kHalf;
  if (!half) return;
  for (Tensor* t : tensors)
    if (t->defined()) *t = t->to(at::kFloat);
}

int dtype_code(const Tensor& t, const char* op, bool half_ok) {
  switch (t.scalar_type()) {
    case at::kFloat: return D2C_F32;
    case at::kDouble: return D2C_F64;
    case at::kHalf:
      if (half_ok) return D2C_F16;
      [[fallthrough]];
    default: TORCH_CHECK(false, "\"", op, "\" not implemented for '", t.scalar_type(), "'");
  }
}

d2c_conv_desc make_desc(const Tensor& x, const Tensor& w, int dtype, const Triple& s, const Triple& p, const Triple& d,
                        int64_t groups, int64_t offset_groups) {
  d2c_conv_desc c{};
  c.dtype = dtype;
  c.batch = (int32_t)x.size(0); c.in_channels = (int32_t)x.size(1); c.out_channels = (int32_t)w.size(0);
  c.in_d = (int32_t)x.size(2); c.in_h = (int32_t)x.size(3); c.in_w = (int32_t)x.size(4);
  c.kd = (int32_t)w.size(2); c.kh = (int32_t)w.size(3); c.kw = (int32_t)w.size(4);
  c.stride_d = (int32_t)s[0]; c.stride_h = (int32_t)s[1]; c.stride_w = (int32_t)s[2];
  c.pad_d = (int32_t)p[0]; c.pad_h = (int32_t)p[1]; c.pad_w = (int32_t)p[2];
  c.dil_d = (int32_t)d[0]; c.dil_h = (int32_t)d[1]; c.dil_w = (int32_t)d[2];
  c.groups = (int32_t)groups; c.offset_groups = (int32_t)offset_groups;
  return c;
}

// Whether a forward that will be differentiated keeps its blended samples for the weight gradient.
std::atomic<bool> g_keep_samples{true};

// Events that deformable backwards record as soon as their parameter gradients are final.  A backward records one that nobody
// else holds; the last one recorded waits here until params_ready_event() hands it out for good (a later backward then records
// another), the one before it is recorded again.
struct ReadyEvents {
  std::mutex mutex;
  std::optional<at::cuda::CUDAEvent> latest;
  std::vector<at::cuda::CUDAEvent> spare;      // as many as backwards ran at the same time

  at::cuda::CUDAEvent borrow(const at::cuda::CUDAStream& stream) {
    {
      const std::lock_guard<std::mutex> lock(mutex);
      for (auto it = spare.begin(); it != spare.end(); ++it)
        if (it->device_index() == stream.device_index()) {
          at::cuda::CUDAEvent ev = std::move(*it);
          spare.erase(it);
          return ev;
        }
    }
    at::cuda::CUDAEvent ev;
    ev.record(stream);                          // creates it
    return ev;
  }
  void publish(at::cuda::CUDAEvent&& ev) {
    const std::lock_guard<std::mutex> lock(mutex);
    if (latest) spare.push_back(std::move(*latest));
    latest = std::move(ev);
  }
};
ReadyEvents& ready_events() {
  static auto* const events = new ReadyEvents();     // outlives the CUDA context
  return *events;
}

// Results of a backward node: gradients are computed outside the graph, so a second derivative has to fail loudly.
variable_list once_differentiable(variable_list&& grads) {
  if (!at::GradMode::is_enabled()) return std::move(grads);
  auto error = std::make_shared<torch::autograd::DelayedError>(
      "trying to differentiate twice a function that was marked with @once_differentiable", (int64_t)grads.size());
  error->set_next_edges(torch::autograd::edge_list(1));
  for (Tensor& t : grads)
    if (t.defined()) t.set_requires_grad(true);
  return (*error)(std::move(grads));
}

// ---- deformable / dynamic-dilated / fused-head / 1-D op ---------------------------------------------------

enum class Kind { offsets, field, head_offsets, head_field, conv1d };

struct DeformNode : public Node {
  Kind kind;
  d2c_conv_desc desc;
  d2c_head_desc head;
  int field_mode;
  bool has_bias;
  SavedVariable x, geo, mask, weight;
  Tensor cache_buf;
  d2c_sample_cache cache{};

  std::string name() const override { return "D2CDeformConvBackward"; }

  // Two threads may run backward over a shared graph: what a node holds is unpacked and released under its mutex, as PyTorch's
  // own nodes do; the pass itself works on its own references.
  void release_variables() override {
    const std::lock_guard<std::mutex> lock(mutex_);
    x.reset_data(); geo.reset_data(); mask.reset_data(); weight.reset_data();
    cache_buf = Tensor();
    cache = d2c_sample_cache{};
  }

  variable_list apply(variable_list&& grads) override {
    const bool is_head = kind == Kind::head_offsets || kind == Kind::head_field;
    const size_t n_out = is_head ? 4 : 5;
    if (!grads[0].defined()) return variable_list(n_out);
    Tensor xv, gv, mv, wv, kept_buf;
    d2c_sample_cache kept;
    {
      const std::lock_guard<std::mutex> lock(mutex_);
      xv = x.unpack(); gv = geo.unpack(); mv = mask.unpack(); wv = weight.unpack();
      kept_buf = cache_buf;
      kept = cache;
    }
    Tensor gx, ggeo, gmask, gw, gbias;
    {
      at::AutoGradMode no_grad(false);
      c10::cuda::CUDAGuard guard(xv.device());
      const Tensor gy = grads[0].contiguous();
      gx = like(xv); ggeo = like(gv); gmask = like(mv); gw = like(wv);
      if (has_bias) gbias = at::empty({wv.size(0)}, wv.options());
      const int op = (kind == Kind::field || kind == Kind::head_field) ? D2C_OP_DYNDIL_BWD : D2C_OP_DEFORM_BWD;
      const size_t n = is_head ? d2c_head_workspace_bytes(op, &desc, &head, field_mode) : d2c_workspace_bytes(op, &desc);
      const Tensor ws = bytes_on(n, xv);
      const at::cuda::CUDAStream stream = at::cuda::getCurrentCUDAStream(xv.device().index());
      void* st = stream.stream();
      std::optional<at::cuda::CUDAEvent> ready;
      if (kind != Kind::conv1d) ready = ready_events().borrow(stream);
      cudaEvent_t ev = ready ? ready->event() : nullptr;
      if (kept.format) check(d2c_bind_sample_cache(&kept), "bind_sample_cache");
      int rc = 0;
      switch (kind) {
        case Kind::offsets:
          rc = d2c_deform_conv3d_bwd_ev(&desc, ptr(gy), ptr(xv), ptr(gv), ptr(mv), ptr(wv), ptr(gx), ptr(ggeo), ptr(gmask),
                                        ptr(gw), ptr(gbias), ptr(ws), n, st, ev);
          break;
        case Kind::field:
          rc = d2c_dyn_dilated_conv3d_bwd_ev(&desc, field_mode, ptr(gy), ptr(xv), ptr(gv), ptr(mv), ptr(wv), ptr(gx),
                                             ptr(ggeo), ptr(gmask), ptr(gw), ptr(gbias), ptr(ws), n, st, ev);
          break;
        case Kind::head_offsets:
          rc = d2c_deform_conv3d_head_bwd(&desc, &head, ptr(gy), ptr(xv), ptr(gv), ptr(wv), ptr(gx), ptr(ggeo), ptr(gw),
                                          ptr(gbias), ptr(ws), n, st, ev);
          break;
        case Kind::head_field:
          rc = d2c_dyn_dilated_conv3d_head_bwd(&desc, &head, field_mode, ptr(gy), ptr(xv), ptr(gv), ptr(wv), ptr(gx),
                                               ptr(ggeo), ptr(gw), ptr(gbias), ptr(ws), n, st, ev);
          break;
        case Kind::conv1d:
          rc = d2c_deform_conv1d_bwd(&desc, ptr(gy), ptr(xv), ptr(gv), ptr(mv), ptr(wv), ptr(gx), ptr(ggeo), ptr(gmask),
                                     ptr(gw), ptr(gbias), ptr(ws), n, st);
          break;
      }
      check(rc, "deformable convolution backward");
      if (ready) ready_events().publish(std::move(*ready));
    }
    if (is_head) return once_differentiable({gx, ggeo, gw, gbias});
    return once_differentiable({gx, ggeo, gmask, gw, gbias});
  }
};

// Runs the forward of `kind` on contiguous tensors and, when autograd is recording, hangs a DeformNode on the result.
// cache_buf: buffer for the forward's samples chosen by the caller; otherwise allocated here for a call that will be
// differentiated (never for one that will not: an evaluation pass over trainable weights must keep nothing).
Tensor run_deform(Kind kind, const d2c_conv_desc& desc, const d2c_head_desc& head, int field_mode, const Tensor& input,
                  const Tensor& geo, const Tensor& mask, const Tensor& weight, const Tensor& bias, at::IntArrayRef out_dims,
                  bool own_cache, Tensor cache_buf) {
  const bool is_head = kind == Kind::head_offsets || kind == Kind::head_field;
  const bool record = torch::autograd::compute_requires_grad(input, geo, mask, weight, bias);
  Tensor y, x, g, m, w, b;
  d2c_sample_cache cache{};
  {
    at::AutoGradMode no_grad(false);
    c10::cuda::CUDAGuard guard(input.device());
    x = contiguous(input); g = contiguous(geo); m = contiguous(mask); w = contiguous(weight); b = contiguous(bias);
    std::vector<int64_t> shape{x.size(0), w.size(0)};
    shape.insert(shape.end(), out_dims.begin(), out_dims.end());
    y = at::empty(shape, x.options().requires_grad(false));
    void* st = stream_of(x);
    if (kind == Kind::conv1d) {
      check(d2c_deform_conv1d_fwd(&desc, ptr(x), ptr(g), ptr(m), ptr(w), ptr(b), ptr(y), st), "deform_conv1d forward");
    } else {
      const int op = (kind == Kind::field || kind == Kind::head_field) ? D2C_OP_DYNDIL_FWD : D2C_OP_DEFORM_FWD;
      const size_t n = is_head ? d2c_head_workspace_bytes(op, &desc, &head, field_mode) : d2c_workspace_bytes(op, &desc);
      const Tensor ws = bytes_on(n, x);
      if (own_cache && record && g_keep_samples.load(std::memory_order_relaxed))
        cache_buf = bytes_on(d2c_sample_cache_bytes(&desc), x);
      if (cache_buf.defined()) {
        cache.data = cache_buf.data_ptr();
        cache.bytes = (size_t)cache_buf.numel();
        check(d2c_bind_sample_cache(&cache), "bind_sample_cache");
      }
      int rc = 0;
      switch (kind) {
        case Kind::offsets:
          rc = d2c_deform_conv3d_fwd(&desc, ptr(x), ptr(g), ptr(m), ptr(w), ptr(b), ptr(y), ptr(ws), n, st);
          break;
        case Kind::field:
          rc = d2c_dyn_dilated_conv3d_fwd(&desc, field_mode, ptr(x), ptr(g), ptr(m), ptr(w), ptr(b), ptr(y), ptr(ws), n, st);
          break;
        case Kind::head_offsets:
          rc = d2c_deform_conv3d_head_fwd(&desc, &head, ptr(x), ptr(g), ptr(w), ptr(b), ptr(y), ptr(ws), n, st);
          break;
        default:
          rc = d2c_dyn_dilated_conv3d_head_fwd(&desc, &head, field_mode, ptr(x), ptr(g), ptr(w), ptr(b), ptr(y), ptr(ws), n, st);
          break;
      }
      check(rc, "deformable convolution forward");
    }
  }
  if (record) {
    auto node = std::shared_ptr<DeformNode>(new DeformNode(), torch::autograd::deleteNode);
    if (is_head)
      node->set_next_edges(torch::autograd::collect_next_edges(input, geo, weight, bias));
    else
      node->set_next_edges(torch::autograd::collect_next_edges(input, geo, mask, weight, bias));
    node->kind = kind; node->desc = desc; node->head = head; node->field_mode = field_mode;
    node->has_bias = bias.defined();
    node->x = SavedVariable(x, false);
    node->geo = SavedVariable(g, false);
    if (m.defined()) node->mask = SavedVariable(m, false);
    node->weight = SavedVariable(w, false);
    if (cache.format) {           // nothing kept: the buffer is released here
      node->cache = cache;
      node->cache_buf = cache_buf;
    }
    torch::autograd::set_history(y, node);
  }
  return y;
}

// SANITY_CHECK_DCONV_INPUTS / _GROUPS, csrc/ops/dconv_gpu_common.h:17-51
void sanity_check(const Tensor& input, const Tensor& offset, const Tensor& alpha, const Tensor& weight, const Tensor& bias) {
  D2C_REQUIRE(input.dim() == 5, "input.ndimension() == ((3) + 2)");
  D2C_REQUIRE(offset.dim() == 5, "offset.ndimension() == ((3) + 2)");
  D2C_REQUIRE(!alpha.defined() || alpha.dim() == 5, "alpha.ndimension() == ((3) + 2)");
  D2C_REQUIRE(weight.dim() == 5, "weight.ndimension() == ((3) + 2)");
  D2C_REQUIRE(!bias.defined() || bias.dim() == 1, "bias.ndimension() == 1");
  D2C_REQUIRE(input.is_cuda(), "input.device().is_cuda()");
  D2C_REQUIRE(offset.is_cuda(), "offset.device().is_cuda()");
  D2C_REQUIRE(!alpha.defined() || alpha.is_cuda(), "alpha.device().is_cuda()");
  D2C_REQUIRE(weight.is_cuda(), "weight.device().is_cuda()");
  D2C_REQUIRE(!bias.defined() || bias.is_cuda(), "bias.device().is_cuda()");
  D2C_REQUIRE(offset.size(0) == input.size(0), "offset.size(0) == input.size(0)");
  D2C_REQUIRE(!alpha.defined() || alpha.size(0) == input.size(0), "alpha.size(0) == input.size(0)");
}

void same_dtype(const Tensor& input, std::initializer_list<const Tensor*> others) {
  for (const Tensor* t : others)
    TORCH_CHECK(!t->defined() || t->scalar_type() == input.scalar_type(), "expected scalar type ", input.scalar_type(),
                " but found ", t->scalar_type());
}

void check_groups(const Tensor& input, const Tensor& weight, const Tensor& bias, int64_t groups) {
  D2C_REQUIRE(weight.size(1) * groups == input.size(1), "weight.size(1) * (n_weight_groups) == input.size(1)");
  D2C_REQUIRE(!bias.defined() || bias.size(0) == weight.size(0), "bias.size(0) == weight.size(0)");
}

std::array<int64_t, 3> output_dims(const d2c_conv_desc& desc, const char* what) {
  int32_t o[3];
  check(d2c_output_dims(&desc, o), what);
  return {o[0], o[1], o[2]};
}

Tensor deform_conv3d(Tensor input, Tensor offset, const OptTensor& alpha_, Tensor weight, const OptTensor& bias_,
                     const Triple& stride, const Triple& padding, const Triple& dilation, int64_t groups,
                     int64_t offset_groups, bool upcast) {
  Tensor alpha = get(alpha_), bias = get(bias_);
  if (upcast) upcast_if_any_half({&input, &offset, &alpha, &weight, &bias});
  sanity_check(input, offset, alpha, weight, bias);
  same_dtype(input, {&offset, &alpha, &weight, &bias});
  const int dtype = dtype_code(input, "deform_conv3d", false);
  check_groups(input, weight, bias, groups);
  const d2c_conv_desc desc = make_desc(input, weight, dtype, stride, padding, dilation, groups, offset_groups);
  const int64_t od[4] = {offset.size(1), offset.size(2), offset.size(3), offset.size(4)};
  int64_t md[4] = {0, 0, 0, 0};
  if (alpha.defined())
    for (int i = 0; i < 4; ++i) md[i] = alpha.size(i + 1);
  check(d2c_deform_conv3d_check(&desc, od, alpha.defined() ? md : nullptr), "deform_conv3d");
  const auto out = output_dims(desc, "deform_conv3d");
  return run_deform(Kind::offsets, desc, d2c_head_desc{}, 0, input, offset, alpha, weight, bias, out, true, Tensor());
}

int64_t field_channels(int64_t mode) { return mode == D2C_FIELD_X ? 1 : (mode == D2C_FIELD_XYZ ? 3 : 2); }

Tensor dyn_dilated_conv3d(Tensor input, Tensor size_map, const OptTensor& alpha_, Tensor weight, const OptTensor& bias_,
                          int64_t field_mode, const Triple& stride, const Triple& padding, const Triple& dilation,
                          int64_t groups, int64_t offset_groups, bool upcast) {
  Tensor alpha = get(alpha_), bias = get(bias_);
  if (upcast) upcast_if_any_half({&input, &size_map, &alpha, &weight, &bias});
  sanity_check(input, size_map, alpha, weight, bias);
  same_dtype(input, {&size_map, &alpha, &weight, &bias});
  const int dtype = dtype_code(input, "deform_conv3d", false);
  check_groups(input, weight, bias, groups);
  const d2c_conv_desc desc = make_desc(input, weight, dtype, stride, padding, dilation, groups, offset_groups);
  const auto out = output_dims(desc, "dyn_dilated_conv3d");
  const int64_t nch = field_channels(field_mode);
  TORCH_CHECK(size_map.size(1) == nch && size_map.size(2) == out[0] && size_map.size(3) == out[1] && size_map.size(4) == out[2],
              "size_map must be [B, ", nch, ", (", out[0], ", ", out[1], ", ", out[2], ")], got ", size_map.sizes());
  const int64_t K = weight.size(2) * weight.size(3) * weight.size(4);
  if (alpha.defined() && !(alpha.size(1) == offset_groups * K && alpha.size(2) == out[0] && alpha.size(3) == out[1] &&
                           alpha.size(4) == out[2]))
    TORCH_CHECK(false, d2c_status_string(D2C_ERR_MASK_SHAPE));
  return run_deform(Kind::field, desc, d2c_head_desc{}, (int)field_mode, input, size_map, alpha, weight, bias, out, true,
                    Tensor());
}

// field_mode < 0: `raw` holds offsets.  mask_channel0 < 0: no modulation.
Tensor deform_conv3d_head(const Tensor& input, const Tensor& raw, const Tensor& weight, const OptTensor& bias_,
                          int64_t field_mode, int64_t mask_channel0, int64_t mask_act, int64_t size_act, const Triple& stride,
                          const Triple& padding, const Triple& dilation, int64_t groups, int64_t offset_groups,
                          const OptTensor& cache_buf) {
  const Tensor bias = get(bias_);
  D2C_REQUIRE(input.dim() == 5, "input.ndimension() == 5");
  D2C_REQUIRE(input.is_cuda(), "input.device().is_cuda()");
  D2C_REQUIRE(raw.dim() == 5, "deformation.ndimension() == 5");
  D2C_REQUIRE(raw.is_cuda(), "deformation.device().is_cuda()");
  D2C_REQUIRE(weight.dim() == 5, "weight.ndimension() == 5");
  D2C_REQUIRE(weight.is_cuda(), "weight.device().is_cuda()");
  D2C_REQUIRE(!bias.defined() || bias.dim() == 1, "bias.ndimension() == 1");
  D2C_REQUIRE(!bias.defined() || bias.is_cuda(), "bias.device().is_cuda()");
  same_dtype(input, {&raw, &weight, &bias});
  const int dtype = dtype_code(input, "deform_conv3d", false);
  D2C_REQUIRE(raw.size(0) == input.size(0), "offset.size(0) == input.size(0)");
  check_groups(input, weight, bias, groups);
  const d2c_conv_desc desc = make_desc(input, weight, dtype, stride, padding, dilation, groups, offset_groups);
  const auto out = output_dims(desc, "deform_conv3d");
  if (!(raw.size(2) == out[0] && raw.size(3) == out[1] && raw.size(4) == out[2]))
    TORCH_CHECK(false, d2c_status_string(D2C_ERR_OFFSET_SHAPE));
  const d2c_head_desc head{(int32_t)raw.size(1), 0, (int32_t)mask_channel0, (int32_t)mask_act, (int32_t)size_act};
  return run_deform(field_mode < 0 ? Kind::head_offsets : Kind::head_field, desc, head, (int)(field_mode < 0 ? 0 : field_mode),
                    input, raw, Tensor(), weight, bias, out, false, get(cache_buf));
}

Tensor deform_conv1d(Tensor input, Tensor offset, const OptTensor& alpha_, Tensor weight, const OptTensor& bias_,
                     int64_t stride, int64_t padding, int64_t dilation, int64_t groups, int64_t offset_groups, bool upcast) {
  Tensor alpha = get(alpha_), bias = get(bias_);
  if (upcast) upcast_if_any_half({&input, &offset, &alpha, &weight, &bias});
  D2C_REQUIRE(input.dim() == 3, "input.ndimension() == 3");
  D2C_REQUIRE(input.is_cuda(), "input.device().is_cuda()");
  D2C_REQUIRE(offset.dim() == 3, "offset.ndimension() == 3");
  D2C_REQUIRE(offset.is_cuda(), "offset.device().is_cuda()");
  D2C_REQUIRE(!alpha.defined() || alpha.dim() == 3, "alpha.ndimension() == 3");
  D2C_REQUIRE(!alpha.defined() || alpha.is_cuda(), "alpha.device().is_cuda()");
  D2C_REQUIRE(weight.dim() == 3, "weight.ndimension() == 3");
  D2C_REQUIRE(weight.is_cuda(), "weight.device().is_cuda()");
  D2C_REQUIRE(!bias.defined() || bias.dim() == 1, "bias.ndimension() == 1");
  D2C_REQUIRE(!bias.defined() || bias.is_cuda(), "bias.device().is_cuda()");
  same_dtype(input, {&offset, &alpha, &weight, &bias});
  const int dtype = dtype_code(input, "deform_conv1d", false);
  check_groups(input, weight, bias, groups);
  const int64_t K = weight.size(2);
  d2c_conv_desc desc{};            // the [B, C, 1, 1, L] view of the problem
  desc.dtype = dtype;
  desc.batch = (int32_t)input.size(0); desc.in_channels = (int32_t)input.size(1); desc.out_channels = (int32_t)weight.size(0);
  desc.in_d = desc.in_h = 1; desc.in_w = (int32_t)input.size(2);
  desc.kd = desc.kh = 1; desc.kw = (int32_t)K;
  desc.stride_d = desc.stride_h = 1; desc.stride_w = (int32_t)stride;
  desc.pad_d = desc.pad_h = 0; desc.pad_w = (int32_t)padding;
  desc.dil_d = desc.dil_h = 1; desc.dil_w = (int32_t)dilation;
  desc.groups = (int32_t)groups; desc.offset_groups = (int32_t)offset_groups;
  const int64_t Lo = output_dims(desc, "deform_conv1d")[2];
  TORCH_CHECK(offset.size(0) == input.size(0) && offset.size(1) == offset_groups * K && offset.size(2) == Lo,
              "offset output dims do not match computed dims. Got: ", offset.sizes(), " but expected: [", input.size(0), ", ",
              offset_groups * K, ", ", Lo, "]");
  TORCH_CHECK(!alpha.defined() || alpha.sizes() == offset.sizes(),
              "mask output dims do not match computed dims. Got: ", alpha.defined() ? alpha.sizes() : at::IntArrayRef(),
              " but expected: ", offset.sizes());
  const std::array<int64_t, 1> out{Lo};
  return run_deform(Kind::conv1d, desc, d2c_head_desc{}, 0, input, offset, alpha, weight, bias, out, false, Tensor());
}

// ---- depthwise conv3d ---------------------------------------------------------------------------------------

struct DepthwiseNode : public Node {
  d2c_conv_desc desc;
  bool has_bias, unbatched;
  SavedVariable x, weight;

  std::string name() const override { return "D2CDepthwiseConv3dBackward"; }
  void release_variables() override {
    const std::lock_guard<std::mutex> lock(mutex_);
    x.reset_data(); weight.reset_data();
  }

  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return variable_list(3);
    Tensor xv, wv;
    {
      const std::lock_guard<std::mutex> lock(mutex_);
      xv = x.unpack(); wv = weight.unpack();
    }
    Tensor gx, gw, gb;
    {
      at::AutoGradMode no_grad(false);
      c10::cuda::CUDAGuard guard(xv.device());
      const Tensor gy = (unbatched ? grads[0].unsqueeze(0) : grads[0]).contiguous();
      if (task_should_compute_output(0)) gx = like(xv);
      Tensor ws;
      size_t n = 0;
      if (task_should_compute_output(1)) {
        gw = like(wv);
        n = d2c_workspace_bytes(D2C_OP_DEPTHWISE_BWD, &desc);
        ws = bytes_on(n, xv);
      }
      if (has_bias && task_should_compute_output(2)) gb = at::empty({wv.size(0)}, wv.options());
      check(d2c_depthwise_conv3d_bwd(&desc, ptr(gy), ptr(xv), ptr(wv), ptr(gx), ptr(gw), ptr(gb), ptr(ws), n, stream_of(xv)),
            "depthwise_separable_conv3d backward");
      if (unbatched && gx.defined()) gx = gx.squeeze(0);
    }
    return once_differentiable({gx, gw, gb});
  }
};

Tensor depthwise_conv3d(const Tensor& input, const Tensor& weight, const OptTensor& bias_, const Triple& stride,
                        const Triple& padding, const Triple& dilation) {
  const Tensor bias = get(bias_);
  TORCH_CHECK(input.is_cuda() && weight.is_cuda(), "depthwise_separable_conv3d expects CUDA tensors");
  TORCH_CHECK(input.device() == weight.device() && (!bias.defined() || bias.device() == input.device()),
              "expects input and weight tensors to be on the same device.");
  const bool unbatched = input.dim() == 4;
  TORCH_CHECK(unbatched || input.dim() == 5, "Input dimension should be 4D or 5D, got ", input.dim(), "D");
  TORCH_CHECK(weight.dim() == 5, "Weight dimension should be 5D, got ", weight.dim(), "D");
  TORCH_CHECK(weight.size(1) == 1, "Depthwise weight should have in_channels=1, got ", weight.size(1));
  const int64_t cin = input.size(unbatched ? 0 : 1);
  TORCH_CHECK(cin > 0 && weight.size(0) % cin == 0, "Depthwise out channels should be a multiple of in channels, got ",
              weight.size(0), " and ", cin);
  TORCH_CHECK(!bias.defined() || (bias.dim() == 1 && bias.size(0) == weight.size(0)),
              "Bias length should be equal to out_channels, got ", bias.defined() ? bias.sizes() : at::IntArrayRef(), " and ",
              weight.size(0));
  TORCH_CHECK(weight.scalar_type() == input.scalar_type() &&
                  (!bias.defined() || bias.scalar_type() == input.scalar_type()),
              "input, weight and bias must have the same dtype");
  const int dtype = dtype_code(input, "depthwise_separable_conv3d", true);
  const bool record = torch::autograd::compute_requires_grad(input, weight, bias);
  Tensor y, x, w, b;
  d2c_conv_desc desc;
  {
    at::AutoGradMode no_grad(false);
    c10::cuda::CUDAGuard guard(input.device());
    x = (unbatched ? input.unsqueeze(0) : input).contiguous();
    w = weight.contiguous();
    b = contiguous(bias);
    desc = make_desc(x, w, dtype, stride, padding, dilation, cin, 1);
    const auto out = output_dims(desc, "depthwise_separable_conv3d");
    y = at::empty({x.size(0), w.size(0), out[0], out[1], out[2]}, x.options().requires_grad(false));
    check(d2c_depthwise_conv3d_fwd(&desc, ptr(x), ptr(w), ptr(b), ptr(y), stream_of(x)), "depthwise_separable_conv3d forward");
    if (unbatched) y = y.squeeze(0);
  }
  if (record) {
    auto node = std::shared_ptr<DepthwiseNode>(new DepthwiseNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(input, weight, bias));
    node->desc = desc; node->has_bias = bias.defined(); node->unbatched = unbatched;
    node->x = SavedVariable(x, false);
    node->weight = SavedVariable(w, false);
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ---- state ------------------------------------------------------------------------------------------------------

void set_keep_samples(bool on) { g_keep_samples.store(on); }
bool get_keep_samples() { return g_keep_samples.load(); }

// The event of the most recent backward as a torch.cuda.Event, once; None where there is none that was not handed out.
py::object take_params_ready_event() {
  ReadyEvents& events = ready_events();
  {
    const std::lock_guard<std::mutex> lock(events.mutex);
    if (!events.latest) return py::none();
  }
  py::object event = py::module_::import("torch.cuda").attr("Event")();
  const std::lock_guard<std::mutex> lock(events.mutex);
  if (!events.latest) return py::none();
  reinterpret_cast<THCPEvent*>(event.ptr())->cuda_event = std::move(*events.latest);
  events.latest.reset();
  return event;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  // the interpreter lock is not needed below this line, and errors keep their plain text
  m.def("deform_conv3d", torch::wrap_pybind_function_no_gil(deform_conv3d));
  m.def("dyn_dilated_conv3d", torch::wrap_pybind_function_no_gil(dyn_dilated_conv3d));
  m.def("deform_conv3d_head", torch::wrap_pybind_function_no_gil(deform_conv3d_head));
  m.def("deform_conv1d", torch::wrap_pybind_function_no_gil(deform_conv1d));
  m.def("depthwise_conv3d", torch::wrap_pybind_function_no_gil(depthwise_conv3d));
  m.def("set_keep_samples", set_keep_samples);
  m.def("get_keep_samples", get_keep_samples);
  m.def("take_params_ready_event", take_params_ready_event);
}
