// The host side of one attention or mask call: arguments, allocations, launches, one call per step from Python.
//
// A small call is bound by its host path: the passes of 2 x 128 float32 tokens of 8 heads take 43 us of the device, and took 200 us
// of the host with the argument structures filled in, and the tensors allocated, from Python (136 - 147 us now; create_block_mask of
// 16 x 16 blocks 48 -> 22).  Everything is built for one call and dropped with it; the library's entry points are those of include/bma.h, handed over as addresses by jaxmodules_b200/_native.py,
// so that both sides use the one library that is loaded.
#include <cuda_runtime_api.h>
#include <nvtx3/nvToolsExt.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>
#include <ATen/ATen.h>

#include <algorithm>
#include <cmath>
#include <optional>
#include <string>

#include "../../include/bma.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

// ---- the library ------------------------------------------------------------------------------------------------
#define BMA_FUNCTIONS(X)                                                                                                      \
  X(bma_mask_compile_workspace_bytes) X(bma_mask_compile) X(bma_attn_plan) X(bma_attn_bwd_plan) X(bma_attn_fwd_implies_lists) X(bma_attn_fwd_workspace_bytes) \
  X(bma_attn_fwd_uses_workspace) X(bma_attn_fwd_ws) X(bma_attn_f32_workspace_bytes) X(bma_attn_fwd_f32) X(bma_attn_bwd_f32) X(bma_attn_bwd_f32_o) X(bma_attn_bwd_preprocess)       \
  X(bma_attn_bwd_workspace_bytes) X(bma_attn_bwd_scratch_bytes) X(bma_attn_bwd_scratch_min_bytes) X(bma_attn_bwd) X(bma_attn_bwd_o)
struct Library {
#define X(name) decltype(&::name) name = nullptr;
  BMA_FUNCTIONS(X)
#undef X
} lib;
PyObject* error_class = nullptr;   // _native.BmaError, which lives as long as the process

void bind(const py::dict& addresses, py::object error) {
#define X(name) lib.name = reinterpret_cast<decltype(&::name)>(addresses[#name].cast<uintptr_t>());
  BMA_FUNCTIONS(X)
#undef X
  Py_XDECREF(error_class);
  error_class = error.release().ptr();
}

void check(int status, const char* where) {
  if (status == BMA_OK) return;
  py::object e = py::reinterpret_borrow<py::object>(error_class)(status, where);
  PyErr_SetObject(error_class, e.ptr());
  throw py::error_already_set();
}

// One launch group: a range named after it, visible in a timeline profiler and free otherwise; other Python threads run meanwhile.
struct Group {
  explicit Group(const char* name) { nvtxRangePushA(name); }
  ~Group() { nvtxRangePop(); }
  py::gil_scoped_release no_gil;
};

// ---- arguments --------------------------------------------------------------------------------------------------
template <typename T>
T* at_address(uintptr_t p) { return reinterpret_cast<T*>(p); }

bma_tensor describe(const Tensor& t) {
  TORCH_CHECK_VALUE(t.dim() == 4 && t.stride(3) == 1, "innermost dimension must be contiguous");
  bma_tensor r{};
  r.ptr = t.data_ptr();
  r.stride_b = t.stride(0); r.stride_l = t.stride(1); r.stride_h = t.stride(2);
  TORCH_CHECK_TYPE(t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16, "float32 or bfloat16 expected");
  r.dtype = t.scalar_type() == at::kFloat ? BMA_DTYPE_F32 : BMA_DTYPE_BF16;
  return r;
}

bma_attn_args arguments(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& key_bias, std::optional<double> scale, int backend) {
  bma_attn_args a{};
  a.q = describe(q); a.k = describe(k); a.v = describe(v);
  a.B = (int32_t)q.size(0); a.N = (int32_t)q.size(1); a.Hq = (int32_t)q.size(2); a.d = (int32_t)q.size(3);
  a.L = (int32_t)k.size(1); a.Hkv = (int32_t)k.size(2);
  a.scale = (float)(scale ? *scale : 1.0 / std::sqrt((double)k.size(3)));
  a.backend = backend;
  if (key_bias) a.key_bias = static_cast<const float*>(key_bias->data_ptr());   // [Hq] float32 on the device
  return a;
}

Tensor bytes_on(const Tensor& like, size_t n) { return at::empty({(int64_t)n}, like.options().dtype(at::kByte).requires_grad(false)); }

struct Route {
  int32_t backend = 0, q_tile = 0, kv_tile = 0;
  size_t f32_bytes = 0;
};
// The kernels of one pass: those of the float32 tensor-core entry points where these cover the request, else what the plan says.
Route route_of(const bma_attn_args& a, bool backward) {
  Route r;
  if (a.q.dtype == BMA_DTYPE_F32 && (r.f32_bytes = lib.bma_attn_f32_workspace_bytes(&a, backward))) {
    r.backend = BMA_BACKEND_SIMT;
    r.q_tile = r.kv_tile = BMA_F32_TILE;
    return r;
  }
  check((backward ? lib.bma_attn_bwd_plan : lib.bma_attn_plan)(&a, &r.backend, &r.q_tile, &r.kv_tile), "bma_attn_plan");
  return r;
}

// (backend, q_tile, kv_tile, workspace bytes of the float32 kernels) of the forward pass and, `backward`, of the backward pass
py::tuple routes(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& key_bias, std::optional<double> scale, int backend,
                 bool forward, bool backward) {
  const bma_attn_args a = arguments(q, k, v, key_bias, scale, backend);
  auto one = [&](bool wanted, bool bwd) -> py::object {
    if (!wanted) return py::none();
    const Route r = route_of(a, bwd);
    return py::make_tuple(r.backend, r.q_tile, r.kv_tile, r.f32_bytes);
  };
  return py::make_tuple(one(forward, false), one(backward, true));
}

bool implies_lists(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& key_bias, std::optional<double> scale, int backend, uintptr_t spec_at) {
  const bma_attn_args a = arguments(q, k, v, key_bias, scale, backend);
  return lib.bma_attn_fwd_implies_lists(&a, at_address<bma_mask_spec>(spec_at));
}

// ---- block lists ------------------------------------------------------------------------------------------------
// Compiles the lists that `lists` describes by its sizes; returns the tensors that hold them, in the order kv_num, kv_idx,
// full_kv_num, full_kv_idx [, q_num, q_idx, full_q_num, full_q_idx], workspace.  Without `views` the arrays lie in one buffer with the
// workspace.  `flags` are added to those of the mask; the valid lengths are cut at `q_valid`, `k_valid`.
std::vector<Tensor> compile_lists(uintptr_t spec_at, uintptr_t lists_at, int B, int H, bool q_side, bool views, int flags, int q_valid, int k_valid,
                                  int device, uintptr_t stream) {
  bma_mask_spec spec = *at_address<bma_mask_spec>(spec_at);
  bma_block_lists& l = *at_address<bma_block_lists>(lists_at);
  spec.flags |= flags;
  spec.q_valid = std::min(spec.q_valid, q_valid);
  spec.k_valid = std::min(spec.k_valid, k_valid);
  const size_t ws_bytes = lib.bma_mask_compile_workspace_bytes(&spec, B, H, l.NQ, l.NKV);
  const at::TensorOptions on = at::TensorOptions().device(at::kCUDA, (c10::DeviceIndex)device);
  std::vector<Tensor> out;
  uint8_t* ws;
  if (views) {
    const at::TensorOptions i32 = on.dtype(at::kInt);
    auto side = [&](int rows, int cols, int32_t*& num, int32_t*& idx, int32_t*& full_num, int32_t*& full_idx) {
      auto array = [&](at::IntArrayRef shape) {
        out.push_back(at::empty(shape, i32));
        return out.back().data_ptr<int32_t>();
      };
      num = array({l.B, l.H, rows});
      idx = array({l.B, l.H, rows, cols});
      full_num = array({l.B, l.H, rows});
      full_idx = array({l.B, l.H, rows, cols});
    };
    side(l.NQ, l.NKV, l.kv_num, l.kv_idx, l.full_kv_num, l.full_kv_idx);
    if (q_side) side(l.NKV, l.NQ, l.q_num, l.q_idx, l.full_q_num, l.full_q_idx);
    out.push_back(at::empty({(int64_t)std::max<size_t>(ws_bytes, 1)}, on.dtype(at::kByte)));
    ws = out.back().data_ptr<uint8_t>();
  } else {
    auto pad = [](int64_t n) { return (4 * n + 255) / 256 * 256; };   // bytes of n int32, every array on a 256-byte boundary
    const int64_t heads = (int64_t)l.B * l.H, rows = pad(heads * l.NQ), cols = pad(heads * l.NKV), cells = pad(heads * l.NQ * l.NKV);
    const int64_t total = 2 * (rows + cells) + (q_side ? 2 * (cols + cells) : 0);
    out.push_back(at::empty({total + (int64_t)ws_bytes + 1}, on.dtype(at::kByte)));
    uint8_t* at = out.back().data_ptr<uint8_t>();
    auto array = [&](int64_t bytes) {
      int32_t* r = reinterpret_cast<int32_t*>(at);
      at += bytes;
      return r;
    };
    l.kv_num = array(rows); l.kv_idx = array(cells); l.full_kv_num = array(rows); l.full_kv_idx = array(cells);
    if (q_side) { l.q_num = array(cols); l.q_idx = array(cells); l.full_q_num = array(cols); l.full_q_idx = array(cells); }
    ws = at;
  }
  int rc;
  {
    Group group("bma.mask_compile");
    rc = lib.bma_mask_compile(&spec, B, H, &l, ws, ws_bytes, reinterpret_cast<bma_stream_t>(stream));
  }
  check(rc, "bma_mask_compile");
  return out;
}

// ---- attention --------------------------------------------------------------------------------------------------
// `f32_bytes`: workspace of the float32 kernels, 0 for the others; `planes` is that workspace, None where there is no room for it.
std::tuple<Tensor, Tensor> forward(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& key_bias, std::optional<double> scale, int backend,
                                   uintptr_t spec_at, uintptr_t lists_at, size_t f32_bytes, const OptTensor& planes, bool bf16_out, uintptr_t stream) {
  bma_attn_args a = arguments(q, k, v, key_bias, scale, backend);
  const bma_mask_spec* spec = at_address<bma_mask_spec>(spec_at);
  const bma_block_lists* lists = at_address<bma_block_lists>(lists_at);
  const at::TensorOptions f32 = q.options().dtype(at::kFloat).requires_grad(false);
  Tensor o = at::empty({a.B, a.N, a.Hq, a.d}, bf16_out ? f32.dtype(at::kBFloat16) : f32), lse = at::empty({a.B, a.Hq, a.N}, f32), ws;
  a.o = describe(o);
  a.lse = lse.data_ptr<float>();
  size_t ws_bytes = 0;
  if (!f32_bytes && lib.bma_attn_fwd_uses_workspace(&a, lists)) ws = bytes_on(q, ws_bytes = lib.bma_attn_fwd_workspace_bytes(&a, lists));
  int rc;
  {
    Group group("bma.fwd");
    const bma_stream_t st = reinterpret_cast<bma_stream_t>(stream);
    if (f32_bytes) rc = lib.bma_attn_fwd_f32(&a, spec, lists, planes ? planes->data_ptr() : nullptr, planes ? f32_bytes : 0, st);
    else rc = lib.bma_attn_fwd_ws(&a, spec, lists, ws_bytes ? ws.data_ptr() : nullptr, ws_bytes, st);
  }
  check(rc, f32_bytes ? "bma_attn_fwd_f32" : "bma_attn_fwd");
  return {o, lse};
}

// (delta, bf16 copy of the cotangent or None)
std::tuple<Tensor, OptTensor> preprocess(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& d_o, const OptTensor& key_bias,
                                        std::optional<double> scale, int backend, bool bf16_copy, uintptr_t stream) {
  bma_attn_args a = arguments(q, k, v, key_bias, scale, backend);
  const at::TensorOptions f32 = q.options().dtype(at::kFloat).requires_grad(false);
  Tensor delta = at::empty({a.B, a.Hq, a.N}, f32);
  OptTensor copy;
  if (bf16_copy) copy = at::empty({a.B, a.N, a.Hq, a.d}, f32.dtype(at::kBFloat16));
  a.o = describe(o);
  a.d_o = describe(d_o);
  a.delta = delta.data_ptr<float>();
  int rc;
  {
    Group group("bma.bwd_preprocess");
    rc = lib.bma_attn_bwd_preprocess(&a, copy ? copy->data_ptr() : nullptr, reinterpret_cast<bma_stream_t>(stream));
  }
  check(rc, "bma_attn_bwd_preprocess");
  return {delta, copy};
}

// Bytes of the tensor-core backward: (workspace without hand-over, hand-over of everything, of the largest unit); `visited`: host array of
// visited blocks per list head, 0 where the dS tiles cannot be handed over.
std::tuple<size_t, size_t, size_t> backward_bytes(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& key_bias, std::optional<double> scale,
                                                  int backend, uintptr_t lists_at, uintptr_t visited) {
  const bma_attn_args a = arguments(q, k, v, key_bias, scale, backend);
  const bma_block_lists* lists = at_address<bma_block_lists>(lists_at);
  const int64_t* counts = at_address<const int64_t>(visited);
  return {lib.bma_attn_bwd_workspace_bytes(&a), counts ? lib.bma_attn_bwd_scratch_bytes(&a, lists, counts) : 0,
          counts ? lib.bma_attn_bwd_scratch_min_bytes(&a, lists, counts) : 0};
}

// Where `delta` is left out the pass takes it itself, from `d_o` as it came.
std::tuple<Tensor, Tensor, Tensor> backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& d_o,
                                            OptTensor delta, const OptTensor& key_bias, std::optional<double> scale, int backend, uintptr_t spec_at,
                                            uintptr_t lists_at, size_t f32_bytes, const OptTensor& workspace, size_t ws_bytes, uintptr_t visited,
                                            uintptr_t mid_event, uintptr_t stream) {
  bma_attn_args a = arguments(q, k, v, key_bias, scale, backend);
  const bma_mask_spec* spec = at_address<bma_mask_spec>(spec_at);
  const bma_block_lists* lists = at_address<bma_block_lists>(lists_at);
  Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
  a.o = describe(o); a.d_o = describe(d_o);
  const bool own_delta = !delta;
  Tensor copy;
  if (own_delta && !f32_bytes && d_o.scalar_type() != at::kBFloat16) copy = at::empty({a.B, a.N, a.Hq, a.d}, q.options().dtype(at::kBFloat16).requires_grad(false));
  if (own_delta) delta = at::empty({a.B, a.Hq, a.N}, q.options().dtype(at::kFloat).requires_grad(false));
  a.lse = lse.data_ptr<float>(); a.delta = delta->data_ptr<float>();
  a.dq = describe(dq); a.dk = describe(dk); a.dv = describe(dv);
  Tensor small;
  void* ws = workspace ? workspace->data_ptr() : nullptr;
  if (!f32_bytes && !ws) {
    small = bytes_on(q, std::max<size_t>(ws_bytes, 1));
    ws = small.data_ptr();
  }
  int rc;
  {
    Group group("bma.bwd");
    const bma_stream_t st = reinterpret_cast<bma_stream_t>(stream);
    if (f32_bytes) rc = (own_delta ? lib.bma_attn_bwd_f32_o : lib.bma_attn_bwd_f32)(&a, spec, lists, ws, ws ? f32_bytes : 0, st);
    else if (own_delta)
      rc = lib.bma_attn_bwd_o(&a, copy.defined() ? copy.data_ptr() : nullptr, spec, lists, ws, ws_bytes, at_address<const int64_t>(visited), at_address<void>(mid_event), st);
    else rc = lib.bma_attn_bwd(&a, spec, lists, ws, ws_bytes, at_address<const int64_t>(visited), at_address<void>(mid_event), st);
  }
  check(rc, f32_bytes ? "bma_attn_bwd_f32" : "bma_attn_bwd");
  return {dq, dk, dv};
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  m.attr("torch_version") = BMA_TORCH_VERSION;   // the one whose headers this was built with
  m.def("bind", &bind);
  m.def("routes", torch::wrap_pybind_function(routes));
  m.def("implies_lists", torch::wrap_pybind_function(implies_lists));
  m.def("compile_lists", torch::wrap_pybind_function(compile_lists));
  m.def("forward", torch::wrap_pybind_function(forward));
  m.def("preprocess", torch::wrap_pybind_function(preprocess));
  m.def("backward_bytes", torch::wrap_pybind_function(backward_bytes));
  m.def("backward", torch::wrap_pybind_function(backward));
}
