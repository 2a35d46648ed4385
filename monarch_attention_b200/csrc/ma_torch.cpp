// Native half of the Python entry point: one call from Python does the input checks, allocates the result and the
// workspace from PyTorch's caching allocator, and enqueues the kernels through the C ABI.
//
// What bounds the small calls is the host: one image through a vision transformer layer keeps the GPU busy for a few
// microseconds, while the same steps in Python (checks, a ctypes structure, a device context, a workspace lookup) took
// 25 us per call.  The workspace is allocated per call and released as soon as the kernels are queued: the allocator
// is stream-ordered, so the memory is reused by the next call on the stream, nothing is held between calls, and calls
// from several threads or streams cannot meet in one workspace.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>
#include <torch/extension.h>

#include "../../include/monarch_attention_b200.h"

namespace {

using at::Tensor;
using std::optional;

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return MA_B200_F32;
    case at::kBFloat16: return MA_B200_BF16;
    case at::kHalf: return MA_B200_F16;
    default: return -1;
  }
}

void raise_for_status(int code) {
  if (code == MA_B200_OK) return;
  const std::string msg = std::string("monarch_attention_b200: ") + ma_b200_status_string(code) + ": " + ma_b200_last_error();
  TORCH_CHECK_VALUE(code != MA_B200_INVALID_ARGUMENT && code != MA_B200_UNSUPPORTED && code != MA_B200_WORKSPACE_TOO_SMALL, msg);
  TORCH_CHECK(false, msg);
}

ma_b200_tensor view4(const Tensor& t) {
  const auto s = t.strides();
  return {t.data_ptr(), s[0], s[1], s[2]};
}

Tensor unit_inner(const Tensor& t) { return t.stride(-1) == 1 || t.size(-1) == 1 ? t : t.contiguous(); }

void check_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const optional<Tensor>& mask) {
  TORCH_CHECK_VALUE(q.dim() == 4 && k.dim() == 4 && v.dim() == 4, "query, key and value must have shape (batch, heads, tokens, width)");
  TORCH_CHECK(q.is_cuda(), "monarch_attention_b200 runs on CUDA tensors only (there is no CPU path)");
  TORCH_CHECK_VALUE(k.device() == q.device() && v.device() == q.device(), "query, key and value must be on the same device");
  TORCH_CHECK_VALUE(k.sizes() == q.sizes(), "key shape ", k.sizes(), " differs from query shape ", q.sizes());
  TORCH_CHECK_VALUE(v.sizes().slice(0, 3) == q.sizes().slice(0, 3), "value shape ", v.sizes(), " does not match query shape ", q.sizes());
  TORCH_CHECK_VALUE(dtype_code(q.scalar_type()) >= 0 && dtype_code(v.scalar_type()) >= 0, "unsupported dtype ", q.scalar_type(), " / ",
                    v.scalar_type());
  TORCH_CHECK_VALUE(k.scalar_type() == q.scalar_type(), "query and key must have the same dtype");
  if (mask.has_value())
    TORCH_CHECK_VALUE(mask->dim() == 2 && mask->size(0) == q.size(0) && mask->size(1) == q.size(2),
                      "attention_mask must have shape (batch, tokens) = (", q.size(0), ", ", q.size(2), ")");
}

int mask_type(at::ScalarType t) {
  switch (t) {
    case at::kBool: case at::kByte: case at::kChar: return MA_B200_MASK_U8;
    case at::kShort: return MA_B200_MASK_I16;
    case at::kInt: return MA_B200_MASK_I32;
    case at::kLong: return MA_B200_MASK_I64;
    case at::kHalf: case at::kBFloat16: return MA_B200_MASK_F16;
    case at::kFloat: return MA_B200_MASK_F32;
    case at::kDouble: return MA_B200_MASK_F64;
    default: return -1;
  }
}

// A mask the kernels can read (non-zero counts as valid): on the queries' device, unit inner stride.
Tensor readable_mask(const Tensor& mask, const Tensor& q) {
  Tensor m = mask.device() == q.device() ? mask : mask.to(q.device());
  if (mask_type(m.scalar_type()) < 0) m = m.ne(0);
  return m.stride(-1) == 1 || m.size(-1) == 1 ? m : m.contiguous();
}

struct Call {
  int64_t T, B;
  bool pre_pad;
  int kernel;
};

ma_b200_problem make_problem(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& mask, const Call& c) {
  ma_b200_problem p{};
  p.abi_version = MA_B200_ABI_VERSION;
  p.E = q.size(0); p.H = q.size(1); p.N = q.size(2); p.D = q.size(3); p.Dv = v.size(3);
  p.block_size = c.B; p.num_steps = c.T; p.pre_pad = c.pre_pad;
  p.qk_dtype = dtype_code(q.scalar_type());
  p.v_dtype = dtype_code(v.scalar_type());
  p.kernel = c.kernel;
  p.q = view4(q); p.k = view4(k); p.v = view4(v); p.out = view4(out);
  if (mask.defined()) {
    p.mask = static_cast<const uint8_t*>(mask.data_ptr());
    p.mask_stride_e = mask.stride(0);
  }
  return p;
}

Tensor new_output(const Tensor& q, const Tensor& v, bool token_major) {
  const int64_t E = q.size(0), H = q.size(1), N = q.size(2), W = v.size(3);
  const at::TensorOptions o = at::TensorOptions().dtype(v.scalar_type()).device(v.device());
  if (token_major) return at::detail::empty_strided_cuda({E, H, N, W}, {N * H * W, W, H * W, 1}, o);
  return at::detail::empty_cuda({E, H, N, W}, o);
}

Tensor run_kernels(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& mask, const Call& c, const Tensor& out_in,
                   bool token_major) {
  // A bounded wait of an earlier asynchronous call on this device that gave up is reported here, at the next call,
  // without a synchronisation (the kernel leaves its code in mapped host memory).
  raise_for_status(ma_b200_poll_device_status(q_in.device().index()));
  const c10::cuda::CUDAGuard guard(q_in.device());
  const Tensor q = unit_inner(q_in), k = unit_inner(k_in), v = unit_inner(v_in);
  const Tensor out = out_in.defined() ? out_in : new_output(q, v, token_major);
  const ma_b200_problem p = make_problem(q, k, v, out, mask, c);
  ma_b200_workspace_layout layout;
  raise_for_status(ma_b200_workspace_layout_of(&p, &layout));
  const auto stream = c10::cuda::getCurrentCUDAStream();
  const c10::DataPtr ws = c10::cuda::CUDACachingAllocator::get()->allocate(layout.total);
  raise_for_status(ma_b200_forward_typed_mask(&p, mask.defined() ? mask_type(mask.scalar_type()) : MA_B200_MASK_U8, ws.get(), layout.total, stream.stream()));
  return out;
}

bool backward_kernels_take(const Tensor& q, const Tensor& k, const Tensor& v, const Call& c) {
  if (q.stride(-1) != 1 || k.stride(-1) != 1 || v.stride(-1) != 1) return false;
  ma_b200_problem p = make_problem(q, k, v, v, Tensor(), c);
  return ma_b200_backward_workspace_bytes(&p) != 0;
}

// Forward by the kernels, gradients by the backward kernels (which recompute the stage inputs from q, k, v).
struct AttentionFunction : torch::autograd::Function<AttentionFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const optional<Tensor>& mask,
                        int64_t T, int64_t B, bool pre_pad, int64_t kernel, bool token_major) {
    at::AutoDispatchBelowADInplaceOrView below;
    ctx->save_for_backward({q, k, v});
    ctx->saved_data["mask"] = mask.has_value() ? c10::IValue(*mask) : c10::IValue();
    ctx->saved_data["T"] = T;
    ctx->saved_data["B"] = B;
    ctx->saved_data["pre_pad"] = pre_pad;
    return run_kernels(q, k, v, mask.value_or(Tensor()), Call{T, B, pre_pad, (int)kernel}, Tensor(), token_major);
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2];
    const auto& mask_v = ctx->saved_data["mask"];
    const Tensor mask = mask_v.isNone() ? Tensor() : mask_v.toTensor();
    const Call c{ctx->saved_data["T"].toInt(), ctx->saved_data["B"].toInt(), ctx->saved_data["pre_pad"].toBool(), MA_B200_KERNEL_AUTO};
    const c10::cuda::CUDAGuard guard(q.device());
    const at::NoGradGuard no_grad;
    Tensor dz = grads[0];
    const int64_t per = 16 / dz.element_size();
    bool in_place = dz.stride(-1) == 1 && reinterpret_cast<uintptr_t>(dz.data_ptr()) % 16 == 0;
    for (int i = 0; i < 3; ++i) in_place = in_place && dz.stride(i) % per == 0;
    if (!in_place) dz = dz.contiguous();
    const ma_b200_problem p = make_problem(q, k, v, dz, mask, c);
    const size_t need = ma_b200_backward_workspace_bytes(&p);
    if (need == 0) raise_for_status(MA_B200_UNSUPPORTED);
    ma_b200_gradients g{};
    g.grad_out = view4(dz);
    Tensor dq, dk, dv;
    if (ctx->needs_input_grad(0)) { dq = at::empty_like(q); g.dq = view4(dq); }
    if (ctx->needs_input_grad(1)) { dk = at::empty_like(k); g.dk = view4(dk); }
    if (ctx->needs_input_grad(2)) { dv = at::empty_like(v); g.dv = view4(dv); }
    const auto stream = c10::cuda::getCurrentCUDAStream();
    const c10::DataPtr ws = c10::cuda::CUDACachingAllocator::get()->allocate(need);
    raise_for_status(ma_b200_backward_typed_mask(&p, mask.defined() ? mask_type(mask.scalar_type()) : MA_B200_MASK_U8, &g, ws.get(), need, stream.stream()));
    return {dq, dk, dv, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// int(x): block sizes and iteration counts of a configuration may be floats.
int64_t as_integer(PyObject* x) {
  if (PyLong_Check(x)) return PyLong_AsLongLong(x);
  PyObject* i = PyNumber_Long(x);
  if (i == nullptr) return -1;
  const int64_t value = PyLong_AsLongLong(i);
  Py_DECREF(i);
  return value;
}

// forward(q, k, v, mask | None, T, B, pre_pad, kernel, out | None, token_major) -> Tensor, or None when an input
// requires a gradient that the backward kernels do not give.
PyObject* py_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n == 10, "forward() takes 10 arguments");
  for (int i = 0; i < 3; ++i) TORCH_CHECK_TYPE(THPVariable_Check(args[i]), "query, key and value must be tensors");
  const Tensor &q = THPVariable_Unpack(args[0]), &k = THPVariable_Unpack(args[1]), &v = THPVariable_Unpack(args[2]);
  optional<Tensor> mask_in;
  if (args[3] != Py_None) {
    TORCH_CHECK_TYPE(THPVariable_Check(args[3]), "attention_mask must be a tensor or None");
    mask_in = THPVariable_Unpack(args[3]);
  }
  Call c;
  c.T = as_integer(args[4]);
  c.B = as_integer(args[5]);
  if (PyErr_Occurred()) return nullptr;
  c.pre_pad = PyObject_IsTrue(args[6]) == 1;
  c.kernel = (int)PyLong_AsLong(args[7]);
  Tensor out;
  if (args[8] != Py_None) {
    TORCH_CHECK_TYPE(THPVariable_Check(args[8]), "out must be a tensor or None");
    out = THPVariable_Unpack(args[8]);
  }
  const bool token_major = PyObject_IsTrue(args[9]) == 1;
  if (PyErr_Occurred()) return nullptr;
  Tensor result;
  {
    pybind11::gil_scoped_release no_gil;
    check_inputs(q, k, v, mask_in);
    const bool grad = at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
    TORCH_CHECK_VALUE(!grad || !out.defined(), "out= cannot be combined with inputs that require a gradient");
    if (!grad) {
      result = run_kernels(q, k, v, mask_in.has_value() ? readable_mask(*mask_in, q) : Tensor(), c, out, token_major);
    } else if (backward_kernels_take(q, k, v, c)) {
      result = AttentionFunction::apply(q, k, v, mask_in.has_value() ? optional<Tensor>(readable_mask(*mask_in, q)) : std::nullopt, c.T, c.B, c.pre_pad,
                                        (int64_t)c.kernel, token_major);
    }
  }
  if (!result.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(result));
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {{"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_forward)), METH_FASTCALL,
                          "forward(q, k, v, mask, T, B, pre_pad, kernel, out, token_major) -> Tensor | None"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
