// The PyTorch side of the operators: argument checks, output allocation and the autograd nodes, in C++.
//
// The C-ABI library (include/dk_b200.h) does the work; this extension only binds it to torch.  The same steps written as
// Python autograd functions cost 123 us of host time per forward + backward call, whatever the tensors' size (the
// C-ABI calls through ctypes about a third of that), so every call whose kernels take less was bound by it.
//
// The library's entry points are handed over once, by address (`bind`), from the Python module that loaded it: the
// extension links neither the library nor CUDA, and DK_B200_LIB keeps deciding which build is used.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/DeviceGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/python_numbers.h>
#include <torch/torch.h>

#include <limits>

#include "dk_b200.h"

namespace {

using at::Tensor;
using torch::autograd::collect_next_edges;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

#define DK_BOUND(X)                                \
  X(dk_sample_depthwise_forward)                   \
  X(dk_sample_depthwise_backward_workspace_bytes)  \
  X(dk_sample_depthwise_backward)                  \
  X(dk_deform_sample_depthwise_forward_workspace_bytes) \
  X(dk_deform_sample_depthwise_forward_ws)         \
  X(dk_deform_sample_depthwise_backward_workspace_bytes) \
  X(dk_deform_sample_depthwise_backward)           \
  X(dk_nd_linear_sample_forward)                   \
  X(dk_nd_linear_sample_backward_data)             \
  X(dk_nd_linear_sample_backward_coord_sum)        \
  X(dk_plane_scale_forward)                        \
  X(dk_plane_scale_backward)                       \
  X(dk_global_dk_forward)                          \
  X(dk_global_dk_backward_workspace_bytes)         \
  X(dk_global_dk_backward)                         \
  X(dk_offset_clip_forward)                        \
  X(dk_offset_clip_backward)                       \
  X(dk_status_string)                              \
  X(dk_last_cuda_error)

struct Library {
#define DK_MEMBER(name) decltype(&::name) name = nullptr;
  DK_BOUND(DK_MEMBER)
#undef DK_MEMBER
} lib;

PyObject* g_dk_error = nullptr;  // deformable_kernels._cabi.DkError

// ------------------------------------------------------------------ errors and small helpers

// A failed library call, as DkError.  The backward runs on an autograd thread that does not hold the GIL.
[[noreturn]] void throw_status(int status, const char* what) {
  std::string msg = std::string(what) + ": " + lib.dk_status_string(status);
  if (status == DK_ERR_CUDA) msg += " (cudaError " + std::to_string(lib.dk_last_cuda_error()) + ")";
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(g_dk_error ? g_dk_error : PyExc_RuntimeError, msg.c_str());
  python_error err;
  err.persist();
  throw err;
}
inline void check(int status, const char* what) {
  if (C10_UNLIKELY(status != DK_OK)) throw_status(status, what);
}

inline int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return DK_F32;
    case at::kHalf: return DK_F16;
    case at::kDouble: return DK_F64;
    default: break;
  }
  TORCH_CHECK_TYPE(false, "deformable kernels support float16, float32 and float64 tensors, got ", t.scalar_type());
  return -1;
}

// CPU tensors are refused the way the reference refuses them
inline void require_cuda(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || t->is_cuda(), "deformable kernels run on CUDA tensors only");
}
inline void same_dtype(const Tensor& first, std::initializer_list<const Tensor*> rest) {
  for (const Tensor* t : rest)
    TORCH_CHECK_TYPE(!t->defined() || t->scalar_type() == first.scalar_type(), "all tensors of one call must share a dtype (",
                     t->scalar_type(), " vs ", first.scalar_type(), ")");
}
inline void same_device(const Tensor& first, std::initializer_list<const Tensor*> rest) {
  for (const Tensor* t : rest)
    TORCH_CHECK(!t->defined() || t->device() == first.device(), "all tensors of one call must be on the same device (",
                t->device(), " vs ", first.device(), ")");
}

inline Tensor empty_as(const Tensor& like, at::IntArrayRef sizes) {
  return Tensor(at::detail::empty_cuda(sizes, like.scalar_type(), like.device(), std::nullopt));
}
inline Tensor empty_of(const Tensor& like, at::IntArrayRef sizes, at::ScalarType type) {
  return Tensor(at::detail::empty_cuda(sizes, type, like.device(), std::nullopt));
}
inline Tensor workspace(size_t bytes, const Tensor& like) {
  if (bytes == 0) return Tensor();
  return empty_of(like, {(int64_t)bytes}, at::kByte);
}
inline const void* cptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
inline void* mptr(Tensor& t) { return t.defined() ? t.mutable_data_ptr() : nullptr; }
inline void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

inline bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}
// the operators have no forward-mode derivative
inline void no_forward_ad(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(0).defined(),
                                "deformable kernels have no forward-mode derivative");
}

// what every backward does to the gradient that arrives: zeros for an absent one, the operator's dtype, dense
inline Tensor arrived(const variable_list& grads, at::IntArrayRef sizes, const Tensor& like) {
  if (!grads[0].defined()) return at::zeros(sizes, like.options());
  Tensor g = grads[0];
  TORCH_CHECK_NOT_IMPLEMENTED(g.is_cuda(), "deformable kernels run on CUDA tensors only");
  if (g.scalar_type() != like.scalar_type()) g = g.to(like.scalar_type());
  return g.contiguous();
}

inline int as_int(int64_t v) {
  TORCH_CHECK_VALUE(v >= std::numeric_limits<int>::min() && v <= std::numeric_limits<int>::max(), "size out of range: ", v);
  return (int)v;
}

// ------------------------------------------------------------------ local DK and DK + DCN

struct ConvArgs {
  int kernel[2], stride[2], padding[2], dilation[2], groups;
};

// Output extent and shape checks (reference functions/filter_sample_depthwise.py:90-101).
dk_geom make_geom(const Tensor& x, const Tensor& off, const Tensor& rot, const Tensor& w, const ConvArgs& a, int64_t* out4) {
  const int64_t dims = x.dim();
  int64_t out[2] = {1, 1};
  bool ok = true;
  for (int64_t d = 0; d + 2 < dims && d < 2; ++d) {
    const int64_t num = x.size(d + 2) + 2 * (int64_t)a.padding[d] - ((int64_t)a.dilation[d] * (a.kernel[d] - 1) + 1);
    out[d] = num < 0 || a.stride[d] <= 0 ? 0 : num / a.stride[d] + 1;
    ok = ok && out[d] > 0;
  }
  TORCH_CHECK_VALUE(ok, "convolution input is too small (output would be ", out[0], "x", out[1], ")");
  TORCH_CHECK_VALUE(dims == 4 && w.dim() == 4 && w.size(0) == x.size(1) && w.size(1) == 1,
                    "expected input [N,C,H,W] and a depthwise weight bank [C,1,sH,sW]");
  TORCH_CHECK_VALUE(a.groups > 0 && x.size(1) % a.groups == 0, "channels must be divisible by rotation_groups");
  const int64_t taps2 = (int64_t)a.kernel[0] * a.kernel[1] * 2;
  const std::array<int64_t, 4> want_rot = {x.size(0), a.groups * taps2, out[0], out[1]};
  TORCH_CHECK_VALUE(!rot.defined() || rot.sizes() == at::IntArrayRef(want_rot), "rotation must have shape ",
                    at::IntArrayRef(want_rot), ", got ", rot.sizes());
  const std::array<int64_t, 4> want_off = {x.size(0), taps2, out[0], out[1]};
  TORCH_CHECK_VALUE(!off.defined() || off.sizes() == at::IntArrayRef(want_off), "offset must have shape ",
                    at::IntArrayRef(want_off), ", got ", off.sizes());
  out4[0] = x.size(0), out4[1] = x.size(1), out4[2] = out[0], out4[3] = out[1];
  dk_geom g;
  g.batch = as_int(x.size(0)), g.channels = as_int(x.size(1)), g.in_h = as_int(x.size(2)), g.in_w = as_int(x.size(3));
  g.kernel_h = a.kernel[0], g.kernel_w = a.kernel[1], g.stride_h = a.stride[0], g.stride_w = a.stride[1];
  g.pad_h = a.padding[0], g.pad_w = a.padding[1], g.dil_h = a.dilation[0], g.dil_w = a.dilation[1];
  g.scope_h = as_int(w.size(2)), g.scope_w = as_int(w.size(3)), g.rotation_groups = a.groups;
  return g;
}

struct SampleDepthwiseBackward : public Node {
  SavedVariable input, rotation, weight;
  dk_geom g;
  std::array<int64_t, 4> out_size;

  variable_list apply(variable_list&& grads) override {
    at::NoGradGuard no_grad;
    const Tensor x = input.unpack(), r = rotation.unpack(), w = weight.unpack();
    const c10::DeviceGuard guard(x.device());
    const Tensor dy = arrived(grads, out_size, x);
    Tensor dx, dr, dw;
    if (task_should_compute_output(0)) dx = empty_as(x, x.sizes());
    if (task_should_compute_output(1)) dr = empty_as(r, r.sizes());
    if (task_should_compute_output(2)) dw = empty_as(w, w.sizes());
    const int code = dtype_code(x);
    const size_t bytes = lib.dk_sample_depthwise_backward_workspace_bytes(&g, code);
    Tensor ws = workspace(bytes, x);
    check(lib.dk_sample_depthwise_backward(cptr(dy), cptr(x), cptr(r), cptr(w), mptr(dx), mptr(dr), mptr(dw), &g, code,
                                           mptr(ws), bytes, stream_of(x)),
          "sample_depthwise backward");
    return {dx, dr, dw};
  }
  std::string name() const override { return "SampleDepthwiseFunctionBackward"; }
  void release_variables() override {
    input.reset_data(), rotation.reset_data(), weight.reset_data();
  }
};

Tensor sample_depthwise(const Tensor& input, const Tensor& rotation, const Tensor& weight, const ConvArgs& a) {
  require_cuda({&input, &rotation, &weight});
  same_dtype(input, {&rotation, &weight});
  same_device(input, {&rotation, &weight});
  no_forward_ad({&input, &rotation, &weight});
  const int code = dtype_code(input);
  std::array<int64_t, 4> out_size;
  const dk_geom g = make_geom(input, Tensor(), rotation, weight, a, out_size.data());
  const bool grad = wants_grad({&input, &rotation, &weight});
  Tensor out, x, r, w;
  {
    at::NoGradGuard no_grad;
    const c10::DeviceGuard guard(input.device());
    x = input.contiguous(), r = rotation.contiguous(), w = weight.contiguous();
    out = empty_as(x, out_size);
    check(lib.dk_sample_depthwise_forward(cptr(x), cptr(r), cptr(w), mptr(out), &g, code, stream_of(x)),
          "sample_depthwise forward");
  }
  if (grad) {
    auto node = std::make_shared<SampleDepthwiseBackward>();
    node->set_next_edges(collect_next_edges(input, rotation, weight));
    node->input = SavedVariable(x, false), node->rotation = SavedVariable(r, false), node->weight = SavedVariable(w, false);
    node->g = g;
    node->out_size = out_size;
    torch::autograd::set_history(out, node);
  }
  return out;
}

struct DeformableSampleDepthwiseBackward : public Node {
  SavedVariable input, offset, rotation, weight;
  bool has_rotation = false;
  dk_geom g;
  std::array<int64_t, 4> out_size;

  variable_list apply(variable_list&& grads) override {
    at::NoGradGuard no_grad;
    const Tensor x = input.unpack(), o = offset.unpack(), w = weight.unpack();
    Tensor r = has_rotation ? rotation.unpack() : Tensor();
    const c10::DeviceGuard guard(x.device());
    const Tensor dy = arrived(grads, out_size, x);
    Tensor dx, doff, dr, dw;
    if (task_should_compute_output(0)) dx = empty_as(x, x.sizes());
    if (task_should_compute_output(1)) doff = empty_as(o, o.sizes());
    if (has_rotation && task_should_compute_output(2)) dr = empty_as(r, r.sizes());
    if (task_should_compute_output(3)) dw = empty_as(w, w.sizes());
    const int code = dtype_code(x);
    const size_t bytes = lib.dk_deform_sample_depthwise_backward_workspace_bytes(&g, code);
    Tensor ws = workspace(bytes, x);
    auto call = [&] {
      return lib.dk_deform_sample_depthwise_backward(cptr(dy), cptr(x), cptr(o), cptr(r), cptr(w), mptr(dx), mptr(doff),
                                                     mptr(dr), mptr(dw), &g, code, mptr(ws), bytes, stream_of(x));
    };
    int status = call();
    if (status == DK_ERR_UNSUPPORTED && !has_rotation) {
      // a shape whose kernels do not take an absent rotation
      r = at::zeros({x.size(0), (int64_t)g.rotation_groups * g.kernel_h * g.kernel_w * 2, out_size[2], out_size[3]}, x.options());
      status = call();
    }
    check(status, "deform_sample_depthwise backward");
    return {dx, doff, dr, dw};
  }
  std::string name() const override { return "DeformableSampleDepthwiseFunctionBackward"; }
  void release_variables() override {
    input.reset_data(), offset.reset_data(), rotation.reset_data(), weight.reset_data();
  }
};

Tensor deform_sample_depthwise(const Tensor& input, const Tensor& offset, const Tensor& rotation, const Tensor& weight,
                               const ConvArgs& a) {
  require_cuda({&input, &offset, &rotation, &weight});
  same_dtype(input, {&offset, &rotation, &weight});
  same_device(input, {&offset, &rotation, &weight});
  no_forward_ad({&input, &offset, &rotation, &weight});
  const int code = dtype_code(input);
  std::array<int64_t, 4> out_size;
  const dk_geom g = make_geom(input, offset, rotation, weight, a, out_size.data());
  const bool grad = wants_grad({&input, &offset, &rotation, &weight});
  Tensor out, x, o, r, w;
  {
    at::NoGradGuard no_grad;
    const c10::DeviceGuard guard(input.device());
    x = input.contiguous(), o = offset.contiguous(), w = weight.contiguous();
    if (rotation.defined()) r = rotation.contiguous();
    out = empty_as(x, out_size);
    const size_t bytes = lib.dk_deform_sample_depthwise_forward_workspace_bytes(&g, code);
    Tensor ws = workspace(bytes, x);
    auto call = [&] {
      return lib.dk_deform_sample_depthwise_forward_ws(cptr(x), cptr(o), cptr(r), cptr(w), mptr(out), &g, code, mptr(ws), bytes,
                                                       stream_of(x));
    };
    int status = call();
    if (status == DK_ERR_UNSUPPORTED && !r.defined()) {
      // zero kernel-space offsets: the library builds the (pixel-independent) kernel once where it can
      r = at::zeros({x.size(0), (int64_t)g.rotation_groups * g.kernel_h * g.kernel_w * 2, out_size[2], out_size[3]}, x.options());
      status = call();
    }
    check(status, "deform_sample_depthwise forward");
  }
  if (grad) {
    auto node = std::make_shared<DeformableSampleDepthwiseBackward>();
    node->set_next_edges(collect_next_edges(input, offset, rotation, weight));
    node->input = SavedVariable(x, false), node->offset = SavedVariable(o, false), node->weight = SavedVariable(w, false);
    node->has_rotation = r.defined();
    if (r.defined()) node->rotation = SavedVariable(r, false);
    node->g = g;
    node->out_size = out_size;
    torch::autograd::set_history(out, node);
  }
  return out;
}

// ------------------------------------------------------------------ N-d linear sample

struct NdShape {
  std::array<int, 8> s{};
  int dims = 0;
};
// dims beyond what the library takes keep their count, so that the call is refused there
NdShape nd_shape(const Tensor& data, int64_t first) {
  NdShape sh;
  sh.dims = (int)(data.dim() - first);
  for (int d = 0; d < sh.dims && d < 8; ++d) sh.s[d] = as_int(data.size(first + d));
  return sh;
}

struct NdLinearSampleBackward : public Node {
  SavedVariable input, coord;

  variable_list apply(variable_list&& grads) override {
    at::NoGradGuard no_grad;
    const Tensor data = input.unpack(), pos = coord.unpack();
    const c10::DeviceGuard guard(data.device());
    const int b = (int)pos.size(0), c = (int)data.size(0);
    const std::array<int64_t, 2> out_size = {b, c};
    const Tensor dy = arrived(grads, out_size, data);
    const NdShape sh = nd_shape(data, 1);
    const int code = dtype_code(data);
    void* stream = stream_of(data);
    Tensor ddata, dpos;
    if (task_should_compute_output(0)) {
      ddata = empty_as(data, data.sizes());
      check(lib.dk_nd_linear_sample_backward_data(cptr(dy), cptr(pos), mptr(ddata), b, c, sh.dims, sh.s.data(), code, stream),
            "nd_linear_sample backward (data)");
    }
    if (task_should_compute_output(1)) {
      dpos = empty_as(pos, pos.sizes());
      check(lib.dk_nd_linear_sample_backward_coord_sum(cptr(dy), cptr(data), cptr(pos), mptr(dpos), b, c, sh.dims, sh.s.data(),
                                                       code, stream),
            "nd_linear_sample backward (coord)");
    }
    return {ddata, dpos};
  }
  std::string name() const override { return "NdLinearSampleFunctionBackward"; }
  void release_variables() override { input.reset_data(), coord.reset_data(); }
};

Tensor nd_linear_sample(const Tensor& input, const Tensor& coord) {
  require_cuda({&input, &coord});
  same_dtype(input, {&coord});
  same_device(input, {&coord});
  no_forward_ad({&input, &coord});
  TORCH_CHECK_VALUE(input.dim() >= 2 && coord.dim() == 2 && coord.size(1) == input.dim() - 1,
                    "expected input [C, s1..sD] and coord [B, D]");
  const int code = dtype_code(input);
  const bool grad = wants_grad({&input, &coord});
  Tensor out, data, pos;
  {
    at::NoGradGuard no_grad;
    const c10::DeviceGuard guard(input.device());
    data = input.contiguous(), pos = coord.contiguous();
    const NdShape sh = nd_shape(data, 1);
    out = empty_as(data, {pos.size(0), data.size(0)});
    check(lib.dk_nd_linear_sample_forward(cptr(data), cptr(pos), mptr(out), as_int(pos.size(0)), as_int(data.size(0)), sh.dims,
                                          sh.s.data(), code, stream_of(data)),
          "nd_linear_sample forward");
  }
  if (grad) {
    auto node = std::make_shared<NdLinearSampleBackward>();
    node->set_next_edges(collect_next_edges(input, coord));
    node->input = SavedVariable(data, false), node->coord = SavedVariable(pos, false);
    torch::autograd::set_history(out, node);
  }
  return out;
}

// ------------------------------------------------------------------ per-plane scale

struct PlaneScaleBackward : public Node {
  SavedVariable input, scale;

  variable_list apply(variable_list&& grads) override {
    at::NoGradGuard no_grad;
    const Tensor x = input.unpack(), k = scale.unpack();
    const c10::DeviceGuard guard(x.device());
    const Tensor dy = arrived(grads, x.sizes(), x);
    Tensor dx, dk;
    if (task_should_compute_output(0)) dx = empty_as(x, x.sizes());
    if (task_should_compute_output(1)) dk = empty_as(k, k.sizes());
    check(lib.dk_plane_scale_backward(cptr(dy), cptr(x), cptr(k), mptr(dx), mptr(dk), x.size(0) * x.size(1),
                                      (int)(x.size(2) * x.size(3)), dtype_code(x), stream_of(x)),
          "plane_scale backward");
    return {dx, dk};
  }
  std::string name() const override { return "PlaneScaleFunctionBackward"; }
  void release_variables() override { input.reset_data(), scale.reset_data(); }
};

Tensor plane_scale(const Tensor& input, const Tensor& scale) {
  require_cuda({&input, &scale});
  same_dtype(input, {&scale});
  same_device(input, {&scale});
  no_forward_ad({&input, &scale});
  TORCH_CHECK_VALUE(input.dim() == 4 && scale.dim() == 2 && scale.size(0) == input.size(0) && scale.size(1) == input.size(1),
                    "expected input [N,C,H,W] and scale [N,C]");
  const int code = dtype_code(input);
  const bool grad = wants_grad({&input, &scale});
  Tensor out, x, k;
  {
    at::NoGradGuard no_grad;
    const c10::DeviceGuard guard(input.device());
    x = input.contiguous(), k = scale.contiguous();
    out = empty_as(x, x.sizes());
    check(lib.dk_plane_scale_forward(cptr(x), cptr(k), mptr(out), x.size(0) * x.size(1), as_int(x.size(2) * x.size(3)), code,
                                     stream_of(x)),
          "plane_scale forward");
  }
  if (grad) {
    auto node = std::make_shared<PlaneScaleBackward>();
    node->set_next_edges(collect_next_edges(input, scale));
    node->input = SavedVariable(x, false), node->scale = SavedVariable(k, false);
    torch::autograd::set_history(out, node);
  }
  return out;
}

// ------------------------------------------------------------------ fused global DK (1x1 depthwise)

struct GlobalDKScaleBackward : public Node {
  SavedVariable input, bank, fc_weight;
  Tensor kept;  // pooled [N,C], scale [N,C], raw and coord [N,D], one after the other; not visible outside: no version to check
  int64_t first_dim = 1;             // where the bank's sampled dimensions start

  variable_list apply(variable_list&& grads) override {
    at::NoGradGuard no_grad;
    const Tensor x = input.unpack(), b = bank.unpack(), fw = fc_weight.unpack();
    TORCH_CHECK(kept.defined(), "Trying to backward through the graph a second time");
    const c10::DeviceGuard guard(x.device());
    const Tensor dy = arrived(grads, x.sizes(), x);
    const NdShape sh = nd_shape(b, first_dim);
    const int n = (int)x.size(0), c = (int)x.size(1), hw = (int)(x.size(2) * x.size(3));
    Tensor dx, db, dfw, dfb;
    if (task_should_compute_output(0)) dx = empty_as(x, x.sizes());
    if (task_should_compute_output(1)) db = empty_as(b, b.sizes());
    if (task_should_compute_output(2)) dfw = empty_as(fw, fw.sizes());
    if (task_should_compute_output(3)) dfb = empty_of(x, {sh.dims}, at::kFloat);
    const size_t bytes = lib.dk_global_dk_backward_workspace_bytes(n, c, sh.dims);
    Tensor ws = workspace(bytes, x);
    const float* pooled = kept.const_data_ptr<float>();
    const float *scale = pooled + (int64_t)n * c, *raw = scale + (int64_t)n * c, *coord = raw + (int64_t)n * sh.dims;
    check(lib.dk_global_dk_backward(cptr(dy), cptr(x), cptr(b), cptr(fw), pooled, raw, coord, scale,
                                    mptr(dx), mptr(db), mptr(dfw), mptr(dfb), n, c, hw, sh.dims, sh.s.data(), dtype_code(x),
                                    mptr(ws), bytes, stream_of(x)),
          "global_dk_scale backward");
    return {dx, db, dfw, dfb, Tensor()};
  }
  std::string name() const override { return "GlobalDKScaleFunctionBackward"; }
  void release_variables() override {
    input.reset_data(), bank.reset_data(), fc_weight.reset_data();
    kept.reset();
  }
};

// `bank` is [C, shape...] or, as the layer stores it, [C, 1, shape...] (told apart by the number of coordinates)
Tensor global_dk_scale(const Tensor& input, const Tensor& bank, const Tensor& fc_weight, const Tensor& fc_bias,
                       const Tensor& tap_bias) {
  require_cuda({&input, &bank, &fc_weight, &fc_bias, &tap_bias});
  no_forward_ad({&input, &bank, &fc_weight, &fc_bias, &tap_bias});
  for (const Tensor* t : {&bank, &fc_weight, &fc_bias, &tap_bias})
    TORCH_CHECK_TYPE(t->scalar_type() == at::kFloat, "the coordinate head's tensors must be float32");
  same_device(input, {&bank, &fc_weight, &fc_bias, &tap_bias});
  TORCH_CHECK_VALUE(input.dim() == 4 && bank.dim() >= 2 && bank.size(0) == input.size(1),
                    "expected input [N,C,H,W] and bank [C, shape...]");
  const int64_t first = bank.dim() == tap_bias.numel() + 2 && bank.size(1) == 1 ? 2 : 1;
  const int64_t dims = bank.dim() - first;
  TORCH_CHECK_VALUE(fc_weight.dim() == 2 && fc_weight.size(0) == dims && fc_weight.size(1) == input.size(1) &&
                        fc_bias.numel() == dims && tap_bias.numel() == dims,
                    "expected fc_weight [dims, C], fc_bias [dims], tap_bias [dims]");
  const int code = dtype_code(input);
  const bool grad = wants_grad({&input, &bank, &fc_weight, &fc_bias});
  Tensor out, x, b, fw, kept;
  {
    at::NoGradGuard no_grad;
    const c10::DeviceGuard guard(input.device());
    x = input.contiguous(), b = bank.contiguous(), fw = fc_weight.contiguous();
    const Tensor fb = fc_bias.contiguous(), tb = tap_bias.contiguous();
    const int64_t n = x.size(0), c = x.size(1);
    out = empty_as(x, x.sizes());
    kept = empty_of(x, {2 * n * (c + dims)}, at::kFloat);
    float* pooled = kept.mutable_data_ptr<float>();
    float *scale = pooled + n * c, *raw = scale + n * c, *coord = raw + n * dims;
    const NdShape sh = nd_shape(b, first);
    check(lib.dk_global_dk_forward(cptr(x), cptr(b), cptr(fw), cptr(fb), cptr(tb), mptr(out), pooled, raw, coord, scale,
                                   as_int(n), as_int(c), as_int(x.size(2) * x.size(3)), sh.dims, sh.s.data(), code,
                                   stream_of(x)),
          "global_dk_scale forward");
  }
  if (grad) {
    auto node = std::make_shared<GlobalDKScaleBackward>();
    node->set_next_edges(collect_next_edges(input, bank, fc_weight, fc_bias, tap_bias));
    node->input = SavedVariable(x, false), node->bank = SavedVariable(b, false), node->fc_weight = SavedVariable(fw, false);
    node->kept = kept;
    node->first_dim = first;
    torch::autograd::set_history(out, node);
  }
  return out;
}

// ------------------------------------------------------------------ offset clipping

struct ClipOffsetsBackward : public Node {
  SavedVariable offsets, bias;
  bool has_bias = false;
  double lo = 0, hi = 0, dilate = 1, post_scale = 1;

  variable_list apply(variable_list&& grads) override {
    at::NoGradGuard no_grad;
    const Tensor o = offsets.unpack(), b = has_bias ? bias.unpack() : Tensor();
    const c10::DeviceGuard guard(o.device());
    const Tensor dy = arrived(grads, o.sizes(), o);
    Tensor grad = empty_as(o, o.sizes());
    check(lib.dk_offset_clip_backward(cptr(dy), cptr(o), cptr(b), mptr(grad), (int)o.size(0), (int)o.size(1),
                                      (int)(o.size(2) * o.size(3)), lo, hi, dilate, post_scale, dtype_code(o), stream_of(o)),
          "clip_offsets backward");
    return {grad, Tensor()};
  }
  std::string name() const override { return "ClipOffsetsFunctionBackward"; }
  void release_variables() override { offsets.reset_data(), bias.reset_data(); }
};

Tensor clip_offsets(const Tensor& offsets, const Tensor& bias, double lo, double hi, double dilate, double post_scale) {
  require_cuda({&offsets, &bias});
  no_forward_ad({&offsets});
  TORCH_CHECK_VALUE(offsets.dim() == 4, "expected offsets [N, C, H, W]");
  TORCH_CHECK_VALUE(!bias.defined() || (bias.scalar_type() == at::kFloat && bias.numel() == offsets.size(1)),
                    "bias must be float32 with one entry per offset channel");
  const int code = dtype_code(offsets);
  const bool grad = wants_grad({&offsets});
  Tensor out, o, b;
  {
    at::NoGradGuard no_grad;
    const c10::DeviceGuard guard(offsets.device());
    o = offsets.contiguous();
    if (bias.defined()) b = bias.contiguous();
    out = empty_as(o, o.sizes());
    check(lib.dk_offset_clip_forward(cptr(o), cptr(b), mptr(out), as_int(o.size(0)), as_int(o.size(1)),
                                     as_int(o.size(2) * o.size(3)), lo, hi, dilate, post_scale, code, stream_of(o)),
          "clip_offsets forward");
  }
  if (grad) {
    auto node = std::make_shared<ClipOffsetsBackward>();
    node->set_next_edges(collect_next_edges(offsets, bias));
    node->offsets = SavedVariable(o, false);
    node->has_bias = b.defined();
    if (b.defined()) node->bias = SavedVariable(b, false);
    node->lo = lo, node->hi = hi, node->dilate = dilate, node->post_scale = post_scale;
    torch::autograd::set_history(out, node);
  }
  return out;
}

// ------------------------------------------------------------------ Python surface

Tensor tensor_arg(PyObject* o, const char* name, bool optional = false) {
  if (optional && o == Py_None) return Tensor();
  TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a Tensor, got ", Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
int int_arg(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return as_int(v);
}
// a number, or one number per spatial dimension
void pair_arg(PyObject* o, int (&out)[2]) {
  if (PyLong_Check(o)) {
    out[0] = out[1] = int_arg(o);
    return;
  }
  if (PyObject* seq = PySequence_Fast(o, "")) {
    THPObjectPtr own(seq);
    TORCH_CHECK_VALUE(PySequence_Fast_GET_SIZE(seq) >= 2, "expected one number per spatial dimension");
    out[0] = int_arg(PySequence_Fast_GET_ITEM(seq, 0));
    out[1] = int_arg(PySequence_Fast_GET_ITEM(seq, 1));
    return;
  }
  PyErr_Clear();
  out[0] = out[1] = int_arg(o);
}
double double_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
ConvArgs conv_args(PyObject* const* a) {
  ConvArgs c;
  pair_arg(a[0], c.kernel), pair_arg(a[1], c.stride), pair_arg(a[2], c.padding), pair_arg(a[3], c.dilation);
  c.groups = int_arg(a[4]);
  return c;
}
void want_args(Py_ssize_t got, Py_ssize_t want) { TORCH_CHECK_TYPE(got == want, "expected ", want, " arguments, got ", got); }

// Offsets produced under autocast and fp32 parameters may differ in dtype from the activations; the kernels want one dtype
// per call, so follow the input's.
inline void follow(Tensor& t, const Tensor& input) {
  if (t.defined() && t.scalar_type() != input.scalar_type()) t = t.to(input.scalar_type());
}

#define DK_METHOD(NAME, NARGS, ...)                                           \
  PyObject* NAME(PyObject*, PyObject* const* a, Py_ssize_t n) {               \
    HANDLE_TH_ERRORS                                                          \
    want_args(n, NARGS);                                                      \
    Tensor out;                                                               \
    __VA_ARGS__;                                                              \
    return THPVariable_Wrap(std::move(out));                                  \
    END_HANDLE_TH_ERRORS                                                      \
  }
// the library calls and the allocator run without the GIL, as any torch operator
#define DK_NOGIL(EXPR)                          \
  do {                                          \
    pybind11::gil_scoped_release no_gil;        \
    out = (EXPR);                               \
  } while (0)

DK_METHOD(py_sample_depthwise, 9, {
  const Tensor x = tensor_arg(a[0], "input");
  Tensor r = tensor_arg(a[1], "rotation"), w = tensor_arg(a[2], "weight");
  const ConvArgs c = conv_args(a + 3);
  if (a[8] == Py_True) follow(r, x), follow(w, x);
  DK_NOGIL(sample_depthwise(x, r, w, c));
})
DK_METHOD(py_deform_sample_depthwise, 10, {
  const Tensor x = tensor_arg(a[0], "input");
  Tensor o = tensor_arg(a[1], "offset"), r = tensor_arg(a[2], "rotation", true), w = tensor_arg(a[3], "weight");
  const ConvArgs c = conv_args(a + 4);
  if (a[9] == Py_True) follow(o, x), follow(r, x), follow(w, x);
  DK_NOGIL(deform_sample_depthwise(x, o, r, w, c));
})
DK_METHOD(py_nd_linear_sample, 2, {
  const Tensor x = tensor_arg(a[0], "input"), c = tensor_arg(a[1], "coord");
  DK_NOGIL(nd_linear_sample(x, c));
})
DK_METHOD(py_plane_scale, 2, {
  const Tensor x = tensor_arg(a[0], "input"), k = tensor_arg(a[1], "scale");
  DK_NOGIL(plane_scale(x, k));
})
DK_METHOD(py_global_dk_scale, 5, {
  const Tensor x = tensor_arg(a[0], "input"), b = tensor_arg(a[1], "bank"), fw = tensor_arg(a[2], "fc_weight");
  const Tensor fb = tensor_arg(a[3], "fc_bias"), tb = tensor_arg(a[4], "tap_bias");
  DK_NOGIL(global_dk_scale(x, b, fw, fb, tb));
})
DK_METHOD(py_clip_offsets, 6, {
  const Tensor o = tensor_arg(a[0], "offsets"), b = tensor_arg(a[1], "bias", true);
  const double lo = double_arg(a[2]), hi = double_arg(a[3]), dilate = double_arg(a[4]), post = double_arg(a[5]);
  DK_NOGIL(clip_offsets(o, b, lo, hi, dilate, post));
})

// bind({name: address}, error class): the loaded library's entry points
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want_args(n, 2);
  auto address = [&](const char* name) -> void* {
    PyObject* v = PyDict_GetItemString(a[0], name);
    TORCH_CHECK(v, "the library has no ", name);
    void* p = PyLong_AsVoidPtr(v);
    if (!p && PyErr_Occurred()) throw python_error();
    return p;
  };
#define DK_TAKE(name) lib.name = reinterpret_cast<decltype(lib.name)>(address(#name));
  DK_BOUND(DK_TAKE)
#undef DK_TAKE
  Py_INCREF(a[1]);
  Py_XSETREF(g_dk_error, a[1]);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
// the names that bind() wants
PyObject* py_entry_points(PyObject*, PyObject*) {
#define DK_NAME(name) #name,
  static const char* const names[] = {DK_BOUND(DK_NAME)};
#undef DK_NAME
  PyObject* t = PyTuple_New(sizeof(names) / sizeof(names[0]));
  if (!t) return nullptr;
  for (size_t i = 0; i < sizeof(names) / sizeof(names[0]); ++i) PyTuple_SET_ITEM(t, i, PyUnicode_FromString(names[i]));
  return t;
}

#define DK_FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f))
PyMethodDef methods[] = {
    {"sample_depthwise", DK_FAST(py_sample_depthwise), METH_FASTCALL, nullptr},
    {"deform_sample_depthwise", DK_FAST(py_deform_sample_depthwise), METH_FASTCALL, nullptr},
    {"nd_linear_sample", DK_FAST(py_nd_linear_sample), METH_FASTCALL, nullptr},
    {"plane_scale", DK_FAST(py_plane_scale), METH_FASTCALL, nullptr},
    {"global_dk_scale", DK_FAST(py_global_dk_scale), METH_FASTCALL, nullptr},
    {"clip_offsets", DK_FAST(py_clip_offsets), METH_FASTCALL, nullptr},
    {"bind", DK_FAST(py_bind), METH_FASTCALL, nullptr},
    {"entry_points", py_entry_points, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "dk_torch", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_dk_torch() { return PyModule_Create(&module); }
