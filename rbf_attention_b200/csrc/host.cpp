// The host side of an operator call: checks, operands the TMA engine can address, outputs and workspaces from PyTorch's
// allocator, one call into the C ABI (include/rbf_b200.h). A CPython extension, because this is what short calls wait for:
// the same steps in Python, with the C ABI reached through ctypes, took 31 us for a forward whose kernels run 15 us (B2 H4
// N256 D64; now 15 to 17 us) and 175 us for a forward + backward whose kernels run 71 us (B4 H8 N1024; now 118 us, of which
// autograd's engine is 43), 262 us in fp32 (now 145), 2050 us for the language model on 4 x 777 tokens (now 1155).
// The entry points take and return tensors; ops.py calls them from the operators' implementations. What an entry point
// cannot allocate or copy raises as it would in Python (out of memory included); bad arguments raise ValueError or
// RuntimeError. The attention calls, which post a status word, are checked and prepared first: they return a callable that
// takes the address of the word's slot, enqueues the kernels and returns the C ABI's error code, and the tensors that the
// kernels will fill, so that a slot is only taken for a call that has all it needs.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <cmath>
#include <functional>
#include <optional>
#include <utility>
#include <vector>

#include "../../include/rbf_b200.h"

namespace {

using at::Tensor;
using Optional = std::optional<Tensor>;

// ------------------------------------------------------------------ arguments and results
struct Args {
  PyObject* const* v;
  Py_ssize_t n;
  const char* fn;

  void expect(Py_ssize_t want) const {
    TORCH_CHECK_TYPE(n == want, fn, ": expected ", want, " arguments, got ", n);
  }
  Tensor tensor(Py_ssize_t i, const char* name) const {
    TORCH_CHECK_TYPE(THPVariable_Check(v[i]), name, " must be a tensor");
    return THPVariable_Unpack(v[i]);
  }
  Optional optional(Py_ssize_t i, const char* name) const {
    if (v[i] == Py_None) return std::nullopt;
    return tensor(i, name);
  }
  bool flag(Py_ssize_t i) const {
    const int t = PyObject_IsTrue(v[i]);
    if (t < 0) throw python_error();
    return t != 0;
  }
  int64_t integer(Py_ssize_t i) const {
    const long long x = PyLong_AsLongLong(v[i]);
    if (x == -1 && PyErr_Occurred()) throw python_error();
    return x;
  }
  double number(Py_ssize_t i) const {
    const double x = PyFloat_AsDouble(v[i]);
    if (x == -1.0 && PyErr_Occurred()) throw python_error();
    return x;
  }
};

PyObject* wrap(const Optional& t) {
  if (!t) Py_RETURN_NONE;
  return THPVariable_Wrap(*t);
}

// (items...) as a new tuple; takes the references
template <typename... Items>
PyObject* tuple(Items... items) {
  PyObject* list[] = {items...};
  constexpr Py_ssize_t count = sizeof...(items);
  PyObject* out = PyTuple_New(count);
  bool ok = out != nullptr;
  for (PyObject* x : list) ok = ok && x != nullptr;
  if (!ok) {
    for (PyObject* x : list) Py_XDECREF(x);
    Py_XDECREF(out);
    throw python_error();
  }
  for (Py_ssize_t i = 0; i < count; ++i) PyTuple_SET_ITEM(out, i, list[i]);
  return out;
}

// A prepared call: enqueue(slot address, 0 for none) -> error code. It owns what it was prepared with.
using Enqueue = std::function<int(unsigned int*)>;
constexpr const char* kEnqueue = "rbf_attention_b200.enqueue";

PyObject* enqueue_entry(PyObject* self, PyObject* address) {
  HANDLE_TH_ERRORS
  const auto* call = static_cast<const Enqueue*>(PyCapsule_GetPointer(self, kEnqueue));
  if (call == nullptr) throw python_error();
  void* slot = PyLong_AsVoidPtr(address);
  if (slot == nullptr && PyErr_Occurred()) throw python_error();
  return PyLong_FromLong((*call)(static_cast<unsigned int*>(slot)));
  END_HANDLE_TH_ERRORS
}
PyMethodDef enqueue_method = {"enqueue", enqueue_entry, METH_O, nullptr};

PyObject* callable(Enqueue fn) {
  auto* held = new Enqueue(std::move(fn));
  PyObject* capsule = PyCapsule_New(held, kEnqueue, [](PyObject* c) {
    delete static_cast<Enqueue*>(PyCapsule_GetPointer(c, kEnqueue));
  });
  if (capsule == nullptr) {
    delete held;
    throw python_error();
  }
  PyObject* out = PyCFunction_New(&enqueue_method, capsule);
  Py_DECREF(capsule);
  if (out == nullptr) throw python_error();
  return out;
}

// What _lib.check raises for an error code: ValueError for arguments and layouts, RuntimeError otherwise.
void check(int rc, const char* what) {
  if (rc == RBF_B200_OK) return;
  const bool value = rc == RBF_B200_ERR_BAD_ARGUMENT || rc == RBF_B200_ERR_BAD_LAYOUT;
  static const char* const names[] = {"ok", "bad argument", "bad layout", "workspace", "tensor map", "launch", "device"};
  const char* name = rc > 0 && rc < 7 ? names[rc] : "error";
  if (value) TORCH_CHECK_VALUE(false, what, ": ", name, ": ", rbf_b200_last_error());
  TORCH_CHECK(false, what, ": ", name, ": ", rbf_b200_last_error());
}

// The interpreter's lock is not held while a call copies, allocates or enqueues: a full launch queue blocks, an allocation may
// wait for the device, and what they wait for may need it. An entry point takes its arguments with the lock, does the rest
// without it and takes it back for the results.
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  void lock() {
    if (state != nullptr) PyEval_RestoreThread(std::exchange(state, nullptr));
  }
  ~Unlocked() { lock(); }
};

// ------------------------------------------------------------------ tensors
int dtype_code(at::ScalarType t) {
  return t == at::kBFloat16 ? 0 : t == at::kHalf ? 1 : t == at::kFloat ? 2 : -1;
}
bool is_16bit(const Tensor& t) { return t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf; }

Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Device& device) {
  if (at::globalContext().deterministicAlgorithms())     // which may fill uninitialised memory
    return at::empty(size, at::TensorOptions().dtype(type).device(device));
  return Tensor(at::detail::empty_cuda(size, type, device, std::nullopt));
}

Tensor workspace(size_t bytes, const at::Device& device) {
  // the caching allocator's blocks are 512-byte aligned, which satisfies the 256-byte rule
  return empty({static_cast<int64_t>(bytes)}, at::kByte, device);
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// `t` if the TMA engine can address it in place (unit stride on D, 16-byte aligned base, strides of dims b, h, n multiples
// of 16 bytes), else a contiguous copy
Tensor tma_ready(const Tensor& t) {
  const auto size = t.sizes();
  const auto stride = t.strides();
  const int64_t per16 = 16 / static_cast<int64_t>(t.element_size());
  bool ok = stride[3] == 1 && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
  if (ok && size[3] % per16 == 0 && t.is_contiguous()) return t;
  for (int i = 0; i < 3; ++i)
    if (size[i] > 1 && (stride[i] <= 0 || stride[i] % per16 != 0)) ok = false;
  if (size[2] > 1 && stride[2] < size[3]) ok = false;
  return ok ? t : t.contiguous();
}

Tensor pad_columns(const Tensor& t, int64_t columns) {
  const int64_t d = t.size(3);
  return d == columns ? t : at::constant_pad_nd(t, {0, columns - d});
}
void validate(const char* name, const Tensor& t, const Tensor* like) {
  TORCH_CHECK_VALUE(t.dim() == 4, name, " must have shape (B, H, N, D), got ", t.sizes());
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor: rbf_attention_b200 has no CPU path");
  if (like == nullptr) return;
  TORCH_CHECK_VALUE(t.sizes() == like->sizes(), name, " shape ", t.sizes(), " differs from q shape ", like->sizes());
  TORCH_CHECK_VALUE(t.scalar_type() == like->scalar_type(), name, " dtype ", t.scalar_type(), " differs from q dtype ",
                    like->scalar_type());
  TORCH_CHECK_VALUE(t.device() == like->device(), name, " is on ", t.device(), ", q is on ", like->device());
}

// Head dim the kernels run at. Others up to 128 run zero-padded to the next of the two, which is exact: zero columns add
// nothing to q.k, to |k|^2 or to |q|^2, and zero value columns give zero output columns (the reference pads to the next power
// of two inside its kernels, rbf_attention.py:661). The softmax scale keeps using the caller's head dim.
int64_t padded_head_dim(int64_t d) {
  TORCH_CHECK_VALUE(d <= 128, "head dim ", d, " is not supported (at most 128)");
  return d <= 64 ? 64 : 128;
}
// columns the tensors of a call get: their own where the kernels' loads can pad them, else those the kernels run at
int64_t columns_of(int64_t d, at::ScalarType t) { return t != at::kFloat && d % 8 == 0 ? d : padded_head_dim(d); }

const int64_t* strides3(const Tensor& t) { return t.strides().data(); }

// The same two rules for calls that are prepared in Python: (name, tensor, tensor that it has to go with or None), (tensor)
PyObject* validate_entry(const Args& a) {
  a.expect(3);
  const char* name = PyUnicode_AsUTF8(a.v[0]);
  if (name == nullptr) throw python_error();
  const Optional like = a.optional(2, "like");
  validate(name, a.tensor(1, name), like ? &*like : nullptr);
  Py_RETURN_NONE;
}

PyObject* tma_ready_entry(const Args& a) {
  a.expect(1);
  const Tensor t = a.tensor(0, "t");
  TORCH_CHECK_VALUE(t.dim() == 4, "t must have shape (B, H, N, D), got ", t.sizes());
  Unlocked unlocked;
  const Tensor ready = tma_ready(t);
  unlocked.lock();
  return wrap(ready);
}

// ------------------------------------------------------------------ attention operators
// (q, k, v, causal, softmax) -> (enqueue, out, lse or None). 16-bit tensors, or fp32 at head dims up to 64; `out` has the
// columns that the kernels fill (columns_of).
PyObject* attention_fwd(const Args& a) {
  a.expect(5);
  const Tensor q = a.tensor(0, "q"), k = a.tensor(1, "k"), v = a.tensor(2, "v");
  const bool causal = a.flag(3), softmax = a.flag(4);
  validate("q", q, nullptr);
  validate("k", k, &q);
  validate("v", v, &q);
  const at::ScalarType type = q.scalar_type();
  const int64_t B = q.size(0), H = q.size(1), N = q.size(2), D0 = q.size(3);
  const int64_t D = padded_head_dim(D0);
  TORCH_CHECK_VALUE(is_16bit(q) || (type == at::kFloat && D == 64), "unsupported dtype ", type,
                    " (bfloat16, float16 or float32)");
  const int64_t Dc = columns_of(D0, type);
  Unlocked unlocked;
  const c10::cuda::CUDAGuard guard(q.device());
  const Tensor qc = tma_ready(pad_columns(q, Dc)), kc = tma_ready(pad_columns(k, Dc)), vc = tma_ready(pad_columns(v, Dc));
  const Tensor out = empty({B, H, N, Dc}, type, q.device());
  Optional lse;
  if (softmax) lse = empty({B, H, N}, at::kFloat, q.device());
  const Tensor ws = workspace(rbf_b200_workspace_bytes(B, H, N, D, softmax, 0), q.device());
  const float scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(D0)));
  void* stream = stream_of(q);
  Enqueue call = [=](unsigned int* slot) {
    const c10::cuda::CUDAGuard on(out.device());
    const Unlocked unlocked;
    return rbf_b200_fwd_posting(qc.const_data_ptr(), kc.const_data_ptr(), vc.const_data_ptr(), out.data_ptr(),
                                lse ? lse->data_ptr<float>() : nullptr, ws.data_ptr(), ws.nbytes(), B, H, N, Dc, strides3(qc),
                                strides3(kc), strides3(vc), strides3(out), dtype_code(type), causal, softmax, scale, stream,
                                RBF_B200_PHASE_ALL, slot);
  };
  unlocked.lock();
  return tuple(callable(std::move(call)), wrap(out), wrap(lse));
}

// (q, k, v, out or None, lse or None, dout, causal, scale, softmax) -> (enqueue, dq, dk, dv). 16-bit tensors; the gradients
// have the columns that the kernels fill.
PyObject* attention_bwd(const Args& a) {
  a.expect(9);
  const Tensor q = a.tensor(0, "q"), k = a.tensor(1, "k"), v = a.tensor(2, "v"), dout = a.tensor(5, "dout");
  const Optional out = a.optional(3, "out"), lse = a.optional(4, "lse");
  const bool causal = a.flag(6), softmax = a.flag(8);
  const float scale = static_cast<float>(a.number(7));
  validate("q", q, nullptr);
  validate("k", k, &q);
  validate("v", v, &q);
  validate("dout", dout, &q);
  const at::ScalarType type = q.scalar_type();
  TORCH_CHECK_VALUE(is_16bit(q), "unsupported dtype ", type, " (bfloat16, float16 or float32)");
  const int64_t B = q.size(0), H = q.size(1), N = q.size(2), D0 = q.size(3);
  const int64_t D = padded_head_dim(D0), Dc = columns_of(D0, type);
  TORCH_CHECK_VALUE(!out || (out->sizes() == q.sizes() && out->device() == q.device()),
                    "out must have the shape and device of q, ", q.sizes());
  TORCH_CHECK_VALUE(!softmax || !lse || (lse->numel() == B * H * N && lse->scalar_type() == at::kFloat &&
                                         lse->device() == q.device()),
                    "L must be (B, H, N) float32 on the device of q");
  Unlocked unlocked;
  const c10::cuda::CUDAGuard guard(q.device());
  const Tensor qc = tma_ready(pad_columns(q, Dc)), kc = tma_ready(pad_columns(k, Dc)), vc = tma_ready(pad_columns(v, Dc)),
               doc = tma_ready(pad_columns(dout, Dc));
  Optional oc;
  if (out) oc = tma_ready(pad_columns(out->scalar_type() == type ? *out : out->to(type), Dc));
  const Tensor dq = empty({B, H, N, Dc}, type, q.device()), dk = empty({B, H, N, Dc}, type, q.device()),
               dv = empty({B, H, N, Dc}, type, q.device());
  const Tensor ws = workspace(rbf_b200_workspace_bytes(B, H, N, D, softmax, 1), q.device());
  Optional l;
  if (softmax && lse) l = lse->contiguous();
  void* stream = stream_of(q);
  Enqueue call = [=](unsigned int* slot) {
    const c10::cuda::CUDAGuard on(dq.device());
    const int64_t none[3] = {0, 0, 0};
    // torch.use_deterministic_algorithms(True) selects the backward whose summation order is fixed
    rbf_b200_set_deterministic(at::globalContext().deterministicAlgorithms());
    const Unlocked unlocked;
    return rbf_b200_bwd_posting(qc.const_data_ptr(), kc.const_data_ptr(), vc.const_data_ptr(), oc ? oc->const_data_ptr() : nullptr,
                                l ? l->const_data_ptr<float>() : nullptr, doc.const_data_ptr(), dq.data_ptr(), dk.data_ptr(),
                                dv.data_ptr(), ws.data_ptr(), ws.nbytes(), B, H, N, Dc, strides3(qc), strides3(kc), strides3(vc),
                                oc ? strides3(*oc) : none, strides3(doc), strides3(dq), strides3(dk), strides3(dv),
                                dtype_code(type), causal, softmax, scale, stream, RBF_B200_PHASE_ALL, slot);
  };
  unlocked.lock();
  return tuple(callable(std::move(call)), wrap(dq), wrap(dk), wrap(dv));
}

// ------------------------------------------------------------------ fp32 tensors on the fp16-operand kernels
std::vector<Tensor> tensors(PyObject* sequence) {
  THPObjectPtr list(PySequence_Fast(sequence, "expected a sequence of tensors"));
  if (!list) throw python_error();
  std::vector<Tensor> out;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(list.get()); ++i) {
    PyObject* t = PySequence_Fast_GET_ITEM(list.get(), i);
    TORCH_CHECK_TYPE(THPVariable_Check(t), "expected a sequence of tensors");
    out.push_back(THPVariable_Unpack(t));
  }
  return out;
}

PyObject* wrap_all(const std::vector<Tensor>& list) {
  THPObjectPtr out(PyList_New(static_cast<Py_ssize_t>(list.size())));
  if (!out) throw python_error();
  for (size_t i = 0; i < list.size(); ++i) {
    PyObject* t = THPVariable_Wrap(list[i]);
    if (t == nullptr) throw python_error();
    PyList_SET_ITEM(out.get(), static_cast<Py_ssize_t>(i), t);
  }
  return out.release();
}

// ((B, H, N, D) tensors, how many of them are checked) -> (enqueue, their fp16 copies), or None where the kernel's 16-byte
// loads cannot take them. The word that is posted is 1 if one of the checked left fp16's range.
PyObject* narrow_f32(const Args& a) {
  a.expect(2);
  const std::vector<Tensor> src = tensors(a.v[0]);
  const int64_t checked = a.integer(1);
  TORCH_CHECK_VALUE(!src.empty() && checked >= 0 && checked <= static_cast<int64_t>(src.size()), "narrow_f32: bad count");
  const Tensor& first = src[0];
  if (first.dim() != 4) Py_RETURN_NONE;
  const int64_t B = first.size(0), H = first.size(1), N = first.size(2), D = first.size(3);
  padded_head_dim(D);                              // refused before anything is enqueued
  bool ok = D > 0 && D % 8 == 0;
  std::vector<int64_t> strides;
  for (const Tensor& t : src) {
    ok = ok && t.is_cuda() && t.scalar_type() == at::kFloat && t.sizes() == first.sizes() && t.device() == first.device() &&
         t.stride(3) == 1 && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
    for (int i = 0; ok && i < 3; ++i) {
      ok = t.size(i) <= 1 || t.stride(i) % 4 == 0;
      strides.push_back(t.stride(i));
    }
  }
  if (!ok) Py_RETURN_NONE;
  const at::Device dev = first.device();
  Unlocked unlocked;
  const c10::cuda::CUDAGuard guard(dev);
  std::vector<Tensor> halves;
  for (size_t i = 0; i < src.size(); ++i) halves.push_back(empty({B, H, N, D}, at::kHalf, dev));
  const Tensor flag = empty({2}, at::kInt, dev);
  void* stream = stream_of(first);
  Enqueue call = [=](unsigned int* slot) {
    const c10::cuda::CUDAGuard on(dev);
    std::vector<const void*> from;
    std::vector<void*> to;
    for (const Tensor& t : src) from.push_back(t.const_data_ptr());
    for (const Tensor& t : halves) to.push_back(t.data_ptr());
    const Unlocked unlocked;
    return rbf_b200_narrow_f32_posting(static_cast<int>(src.size()), from.data(), to.data(), strides.data(), B, H, N, D, checked,
                                       static_cast<unsigned int*>(flag.data_ptr()), stream, slot);
  };
  unlocked.lock();
  return tuple(callable(std::move(call)), wrap_all(halves));
}

// Dense fp16 tensors of one shape as fp32, in one launch
PyObject* widen_f16(const Args& a) {
  a.expect(1);
  const std::vector<Tensor> src = tensors(a.v[0]);
  TORCH_CHECK_VALUE(!src.empty(), "widen_f16: no tensors");
  const int64_t count = src[0].numel();
  const at::Device dev = src[0].device();
  Unlocked unlocked;
  std::vector<const void*> from;
  std::vector<void*> to;
  std::vector<Tensor> out;
  bool ok = count % 8 == 0;
  for (const Tensor& t : src)
    ok = ok && t.is_cuda() && t.scalar_type() == at::kHalf && t.is_contiguous() && t.numel() == count && t.device() == dev &&
         reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
  for (const Tensor& t : src) {
    out.push_back(ok ? empty(t.sizes(), at::kFloat, dev) : t.to(at::kFloat));
    from.push_back(t.const_data_ptr());
    to.push_back(out.back().data_ptr());
  }
  int rc = RBF_B200_OK;
  if (ok) {
    const c10::cuda::CUDAGuard guard(dev);
    rc = rbf_b200_widen_f16(static_cast<int>(src.size()), from.data(), to.data(), count, stream_of(src[0]));
  }
  check(rc, "rbf_b200_widen_f16");
  unlocked.lock();
  return wrap_all(out);
}

// ------------------------------------------------------------------ the attention block's RBF branch
// strides of dims b, h, n of memory laid out (B, S, n_rows * H, D), seen as (B, H, S, D)
struct BshdStrides {
  int64_t s[3];
  BshdStrides(int64_t S, int64_t row, int64_t D) : s{S * row, D, row} {}
};

// (qkv, pos_weight, reg_pos_emb or None, table, heads, softmax) -> (enqueue, out, lse, qk)
PyObject* block_fwd(const Args& a) {
  a.expect(6);
  Tensor qkv = a.tensor(0, "qkv");
  const Tensor pos_weight = a.tensor(1, "pos_weight");
  const Optional reg = a.optional(2, "reg_pos_emb");
  Tensor table = a.tensor(3, "table");
  const int64_t H = a.integer(4);
  const bool softmax = a.flag(5);
  TORCH_CHECK(qkv.is_cuda(), "qkv must be a CUDA tensor: rbf_attention_b200 has no CPU path");
  TORCH_CHECK_VALUE(is_16bit(qkv), "unsupported dtype ", qkv.scalar_type(), " (bfloat16 or float16)");
  TORCH_CHECK_VALUE(qkv.dim() == 3, "qkv must have shape (B, S, 3 H D), got ", qkv.sizes());
  TORCH_CHECK_VALUE(H > 0, "the number of heads must be positive");
  const int64_t B = qkv.size(0), S = qkv.size(1), E = qkv.size(2) / 3, D = E / H;
  const int64_t R = reg ? reg->size(-2) : 0;
  TORCH_CHECK_VALUE(D == 64 || D == 128, "head dim ", D, " is not supported (64 or 128)");
  // the kernels walk qkv, and k behind q, by H * D columns
  TORCH_CHECK(qkv.size(2) == 3 * H * D, "qkv ", qkv.sizes(), " is not (B, S, 3 x ", H, " heads x ", D, ")");
  TORCH_CHECK_VALUE(pos_weight.scalar_type() == at::kFloat || pos_weight.scalar_type() == qkv.scalar_type(),
                    "pos_weight must be float32 or have the dtype of qkv");
  const at::Device dev = qkv.device();
  TORCH_CHECK_VALUE(pos_weight.numel() == H * (D / 2) && pos_weight.device() == dev, "pos_weight must be (", H, ", ", D / 2,
                    ") on the device of qkv, got ", pos_weight.sizes());
  TORCH_CHECK_VALUE(R == 0 || (reg->numel() == H * R * D && reg->device() == dev), "reg_pos_emb must be (", H, ", R, ", D,
                    ") on the device of qkv");
  Unlocked unlocked;
  const c10::cuda::CUDAGuard guard(dev);
  qkv = qkv.contiguous();
  const Tensor pw = pos_weight.contiguous();
  Tensor rp;
  if (R > 0) rp = (reg->scalar_type() == pw.scalar_type() ? *reg : reg->to(pw.scalar_type())).contiguous();
  if (table.device() != dev || table.scalar_type() != at::kFloat) table = table.to(dev, at::kFloat);
  table = table.contiguous();
  TORCH_CHECK_VALUE(table.size(0) >= S - R && table.numel() >= (S - R) * D, "the position table holds ", table.size(0),
                    " rows, ", S - R, " text positions of ", D, " columns are needed");
  const at::ScalarType type = qkv.scalar_type();
  const Tensor qk = empty({2, B, S, H, D}, type, dev), out = empty({B, S, E}, type, dev);
  const Tensor lse = softmax ? empty({B, H, S}, at::kFloat, dev) : empty({0}, at::kFloat, dev);
  const Tensor ws = workspace(rbf_b200_workspace_bytes(B, H, S, D, softmax, 0), dev);
  void* stream = stream_of(qkv);
  Enqueue call = [=](unsigned int* slot) {
    const c10::cuda::CUDAGuard on(dev);
    const BshdStrides packed(S, E, D), fused(S, 3 * E, D);
    const int code = dtype_code(type);
    const int64_t item = qkv.element_size();
    char* q = static_cast<char*>(qk.data_ptr());
    char* k = q + B * S * E * item;
    const char* v = static_cast<const char*>(qkv.const_data_ptr()) + 2 * E * item;
    const float scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(D)));
    const Unlocked unlocked;
    const int rc = rbf_b200_qkv_prep(qkv.const_data_ptr(), pw.const_data_ptr(), R > 0 ? rp.const_data_ptr() : nullptr,
                                     pw.scalar_type() == at::kFloat, table.const_data_ptr<float>(), q, k, packed.s, packed.s,
                                     ws.data_ptr(), ws.nbytes(), B, S, H, D, R, code, softmax, scale, stream);
    if (rc != RBF_B200_OK) return rc;
    return rbf_b200_fwd_posting(q, k, v, out.data_ptr(), softmax ? lse.data_ptr<float>() : nullptr, ws.data_ptr(), ws.nbytes(),
                                B, H, S, D, packed.s, packed.s, fused.s, packed.s, code, 1, softmax, scale, stream,
                                RBF_B200_PHASE_MAIN, slot);
  };
  unlocked.lock();
  return tuple(callable(std::move(call)), wrap(out), wrap(lse), wrap(qk));
}

// (qkv, qk, out, lse, dout, table, registers, softmax) -> (enqueue, dqkv, d_pos_weight, d_reg_pos_emb)
PyObject* block_bwd(const Args& a) {
  a.expect(8);
  Tensor qkv = a.tensor(0, "qkv"), dout = a.tensor(4, "dout"), table = a.tensor(5, "table");
  const Tensor qk = a.tensor(1, "qk"), out = a.tensor(2, "out"), lse = a.tensor(3, "lse");
  const int64_t R = a.integer(6);
  const bool softmax = a.flag(7);
  TORCH_CHECK(qkv.is_cuda(), "qkv must be a CUDA tensor: rbf_attention_b200 has no CPU path");
  TORCH_CHECK_VALUE(is_16bit(qkv), "unsupported dtype ", qkv.scalar_type(), " (bfloat16 or float16)");
  TORCH_CHECK_VALUE(qk.dim() == 5 && qk.size(0) == 2, "qk must have shape (2, B, S, H, D), got ", qk.sizes());
  const int64_t B = qk.size(1), S = qk.size(2), H = qk.size(3), D = qk.size(4), E = H * D;
  const at::Device dev = qkv.device();
  const at::ScalarType type = qkv.scalar_type();
  TORCH_CHECK_VALUE(D == 64 || D == 128, "head dim ", D, " is not supported (64 or 128)");
  TORCH_CHECK_VALUE(R >= 0 && R <= S, R, " registers in a sequence of ", S);
  // the kernels walk every tensor by qk's sizes
  TORCH_CHECK(qkv.numel() == 3 * B * S * E && out.numel() == B * S * E && dout.numel() == B * S * E &&
                  (!softmax || lse.numel() == B * H * S) && table.numel() >= (S - R) * D,
              "qkv ", qkv.sizes(), ", out ", out.sizes(), ", lse ", lse.sizes(), ", dout ", dout.sizes(), " or table ",
              table.sizes(), " does not go with qk ", qk.sizes());
  TORCH_CHECK_VALUE(qk.scalar_type() == type && out.scalar_type() == type && (!softmax || lse.scalar_type() == at::kFloat),
                    "qk and out must have the dtype of qkv and lse float32, got ", qk.scalar_type(), ", ", out.scalar_type(),
                    ", ", lse.scalar_type(), " with ", type);
  TORCH_CHECK_VALUE(qk.device() == dev && out.device() == dev && dout.device() == dev && (!softmax || lse.device() == dev),
                    "qkv, qk, out, lse and dout must be on one device");
  Unlocked unlocked;
  const c10::cuda::CUDAGuard guard(dev);
  qkv = qkv.contiguous();
  dout = (dout.scalar_type() == type ? dout : dout.to(type)).contiguous();
  if (table.device() != dev || table.scalar_type() != at::kFloat) table = table.to(dev, at::kFloat);
  table = table.contiguous();
  const Tensor qk_c = qk.contiguous(), out_c = out.contiguous(), lse_c = softmax ? lse.contiguous() : lse;
  const Tensor dqkv = empty({B, S, 3 * E}, type, dev), d_pw = empty({H, D / 2}, at::kFloat, dev),
               d_rp = empty({H, R, D}, at::kFloat, dev);
  const Tensor ws = workspace(rbf_b200_workspace_bytes(B, H, S, D, softmax, 1), dev);
  const Tensor ws2 = workspace(rbf_b200_qkv_prep_bwd_workspace_bytes(B, S, H, D, R), dev);
  void* stream = stream_of(qkv);
  Enqueue call = [=](unsigned int* slot) {
    const c10::cuda::CUDAGuard on(dev);
    const BshdStrides packed(S, E, D), fused(S, 3 * E, D);
    const int code = dtype_code(type);
    const int64_t item = qkv.element_size();
    const char* q = static_cast<const char*>(qk_c.const_data_ptr());
    const char* k = q + B * S * E * item;
    const char* v = static_cast<const char*>(qkv.const_data_ptr()) + 2 * E * item;
    char* dq = static_cast<char*>(dqkv.data_ptr());
    char* dk = dq + E * item;
    const float scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(D)));
    rbf_b200_set_deterministic(at::globalContext().deterministicAlgorithms());
    int rc2 = RBF_B200_OK;
    {
      const Unlocked unlocked;
      const int rc =
          rbf_b200_bwd_posting(q, k, v, out_c.const_data_ptr(), softmax ? lse_c.const_data_ptr<float>() : nullptr,
                               dout.const_data_ptr(), dq, dk, dk + E * item, ws.data_ptr(), ws.nbytes(), B, H, S, D, packed.s,
                               packed.s, fused.s, packed.s, packed.s, fused.s, fused.s, fused.s, code, 1, softmax, scale, stream,
                               RBF_B200_PHASE_ALL, slot);
      if (rc != RBF_B200_OK) return rc;
      rc2 = rbf_b200_qkv_prep_bwd(dq, dk, fused.s, fused.s, table.const_data_ptr<float>(), d_pw.data_ptr<float>(),
                                  R > 0 ? d_rp.data_ptr<float>() : nullptr, ws2.data_ptr(), ws2.nbytes(), B, S, H, D, R, code,
                                  stream);
    }
    check(rc2, "rbf_b200_qkv_prep_bwd");     // raised, not returned: the backward is enqueued and posts its word
    return static_cast<int>(RBF_B200_OK);
  };
  unlocked.lock();
  return tuple(callable(std::move(call)), wrap(dqkv), wrap(d_pw), wrap(d_rp));
}

// ------------------------------------------------------------------ the language model's other layers
// Columns sums over the leading dims: fp32 sums of a 16-bit matrix (rows, cols), cols a multiple of 8.
PyObject* column_sums(const Args& a) {
  a.expect(1);
  Tensor x = a.tensor(0, "x");
  TORCH_CHECK_VALUE(x.dim() == 2 && x.is_cuda() && is_16bit(x) && x.size(1) % 8 == 0,
                    "column_sums: a 16-bit CUDA matrix whose width is a multiple of 8");
  Unlocked unlocked;
  const c10::cuda::CUDAGuard guard(x.device());
  const bool ok = x.stride(1) == 1 && x.stride(0) >= x.size(1) && x.stride(0) % 8 == 0 &&
                  reinterpret_cast<uintptr_t>(x.const_data_ptr()) % 16 == 0;
  if (!ok) x = x.contiguous();
  const int64_t rows = x.size(0), cols = x.size(1);
  const Tensor out = empty({cols}, at::kFloat, x.device());
  const Tensor ws = workspace(std::max<size_t>(rbf_b200_column_sums_workspace_bytes(rows, cols), 16), x.device());
  const int rc = rbf_b200_column_sums(x.const_data_ptr(), out.data_ptr<float>(), ws.data_ptr(), ws.nbytes(), rows, cols,
                                      rows > 1 ? x.stride(0) : cols, dtype_code(x.scalar_type()), stream_of(x));
  check(rc, "rbf_b200_column_sums");
  unlocked.lock();
  return wrap(out);
}

PyObject* gelu_fwd(const Args& a) {
  a.expect(1);
  Tensor h = a.tensor(0, "h");
  TORCH_CHECK_VALUE(h.is_cuda() && is_16bit(h) && h.numel() % 8 == 0,
                    "gelu_fwd: a 16-bit CUDA tensor with a multiple of 8 elements");
  Unlocked unlocked;
  const c10::cuda::CUDAGuard guard(h.device());
  h = h.contiguous();
  const Tensor out = empty(h.sizes(), h.scalar_type(), h.device());
  const int rc = rbf_b200_gelu_fwd(h.const_data_ptr(), out.data_ptr(), h.numel(), dtype_code(h.scalar_type()), stream_of(h));
  check(rc, "rbf_b200_gelu_fwd");
  unlocked.lock();
  return wrap(out);
}

// (h, dy, with_bias) -> (dh, fp32 column sums of dh or an empty tensor)
PyObject* gelu_bwd(const Args& a) {
  a.expect(3);
  Tensor h = a.tensor(0, "h"), dy = a.tensor(1, "dy");
  const bool with_bias = a.flag(2);
  TORCH_CHECK_VALUE(h.is_cuda() && is_16bit(h), "gelu_bwd: a 16-bit CUDA tensor");
  TORCH_CHECK_VALUE(h.dim() > 0 && h.size(-1) > 0, "gelu_bwd: no columns in ", h.sizes());
  TORCH_CHECK_VALUE(dy.numel() == h.numel() && dy.device() == h.device(), "gelu_bwd: dy must have the size and device of h");
  Unlocked unlocked;
  const c10::cuda::CUDAGuard guard(h.device());
  const at::ScalarType type = h.scalar_type();
  h = h.contiguous();
  dy = (dy.scalar_type() == type ? dy : dy.to(type)).contiguous();
  const int64_t cols = h.size(-1), rows = h.numel() / cols;
  const Tensor dh = empty(h.sizes(), type, h.device());
  const Tensor dbias = empty({with_bias ? cols : 0}, at::kFloat, h.device());
  const size_t bytes = with_bias ? rbf_b200_column_sums_workspace_bytes(rows, cols) : 0;
  const Tensor ws = workspace(std::max<size_t>(bytes, 16), h.device());
  const int rc = rbf_b200_gelu_bwd(h.const_data_ptr(), dy.const_data_ptr(), dh.data_ptr(),
                                   with_bias ? dbias.data_ptr<float>() : nullptr, ws.data_ptr(), ws.nbytes(), rows, cols,
                                   dtype_code(type), stream_of(h));
  check(rc, "rbf_b200_gelu_bwd");
  unlocked.lock();
  return tuple(wrap(dh), wrap(dbias));
}

bool layer_norm_takes(const Tensor& x, const Tensor& weight, const Tensor& bias) {
  const at::ScalarType type = x.scalar_type();
  return x.is_cuda() && is_16bit(x) && weight.scalar_type() == type && bias.scalar_type() == type && x.dim() > 0 &&
         x.size(-1) > 0 && x.size(-1) % 256 == 0 && x.size(-1) <= 1024;
}

// (x, residual or None, weight, bias, eps) -> (x + residual or None, y, mean, rstd)
PyObject* layer_norm_fwd(const Args& a) {
  a.expect(5);
  Tensor x = a.tensor(0, "x");
  Optional residual = a.optional(1, "residual");
  const Tensor weight = a.tensor(2, "weight"), bias = a.tensor(3, "bias");
  const float eps = static_cast<float>(a.number(4));
  const char* name = residual ? "add_layer_norm_fwd" : "layer_norm_fwd";
  TORCH_CHECK_VALUE(layer_norm_takes(x, weight, bias), name, ": 16-bit CUDA tensors with 256, 512, 768 or 1024 columns");
  if (residual)
    TORCH_CHECK_VALUE(residual->sizes() == x.sizes() && residual->scalar_type() == x.scalar_type() &&
                          residual->device() == x.device(),
                      "residual must have the shape, dtype and device of x: ", residual->sizes(), " ",
                      residual->scalar_type(), " against ", x.sizes(), " ", x.scalar_type());
  TORCH_CHECK_VALUE(weight.numel() == x.size(-1) && bias.numel() == x.size(-1) && weight.device() == x.device() &&
                        bias.device() == x.device(),
                    name, ": weight and bias must have the columns and the device of x, got ", weight.sizes(), " and ",
                    bias.sizes(), " with ", x.sizes());
  Unlocked unlocked;
  const c10::cuda::CUDAGuard guard(x.device());
  const at::ScalarType type = x.scalar_type();
  const at::Device dev = x.device();
  x = x.contiguous();
  const int64_t cols = x.size(-1), rows = x.numel() / cols;
  Optional sum;
  if (residual) {
    residual = residual->contiguous();
    sum = empty(x.sizes(), type, dev);
  }
  const Tensor y = empty(x.sizes(), type, dev), mean = empty({rows}, at::kFloat, dev), rstd = empty({rows}, at::kFloat, dev);
  const Tensor wc = weight.contiguous(), bc = bias.contiguous();
  const int rc = rbf_b200_add_layer_norm_fwd(x.const_data_ptr(), residual ? residual->const_data_ptr() : nullptr,
                                             sum ? sum->data_ptr() : nullptr, wc.const_data_ptr(), bc.const_data_ptr(),
                                             y.data_ptr(), mean.data_ptr<float>(), rstd.data_ptr<float>(), rows, cols, eps,
                                             dtype_code(type), stream_of(x));
  check(rc, residual ? "rbf_b200_add_layer_norm_fwd" : "rbf_b200_layer_norm_fwd");
  unlocked.lock();
  return tuple(wrap(sum), wrap(y), wrap(mean), wrap(rstd));
}

// (x, dy, gradient of the skip path or None, weight, mean, rstd) -> (dx, dgamma, dbeta)
PyObject* layer_norm_bwd(const Args& a) {
  a.expect(6);
  Tensor x = a.tensor(0, "x"), dy = a.tensor(1, "dy");
  Optional dres = a.optional(2, "dres");
  const Tensor weight = a.tensor(3, "weight"), mean = a.tensor(4, "mean"), rstd = a.tensor(5, "rstd");
  TORCH_CHECK(x.is_cuda(), "x must be a CUDA tensor: rbf_attention_b200 has no CPU path");
  TORCH_CHECK_VALUE(x.dim() > 0 && x.size(-1) > 0, "layer_norm_bwd: no columns in ", x.sizes());
  Unlocked unlocked;
  const c10::cuda::CUDAGuard guard(x.device());
  const at::ScalarType type = x.scalar_type();
  const at::Device dev = x.device();
  const int64_t cols = x.size(-1), rows = x.numel() / cols;
  TORCH_CHECK_VALUE(is_16bit(x) && weight.scalar_type() == type && mean.scalar_type() == at::kFloat &&
                        rstd.scalar_type() == at::kFloat,
                    "layer_norm_bwd: 16-bit x and weight of one type, mean and rstd float32");
  TORCH_CHECK_VALUE(dy.numel() == x.numel() && weight.numel() == cols && mean.numel() == rows && rstd.numel() == rows,
                    "layer_norm_bwd: dy ", dy.sizes(), ", weight ", weight.sizes(), ", mean ", mean.sizes(), " or rstd ",
                    rstd.sizes(), " does not go with x ", x.sizes());
  TORCH_CHECK_VALUE(dy.device() == dev && weight.device() == dev && mean.device() == dev && rstd.device() == dev &&
                        (!dres || dres->device() == dev),
                    "layer_norm_bwd: tensors on several devices");
  x = x.contiguous();
  dy = (dy.scalar_type() == type ? dy : dy.to(type)).contiguous();
  const Tensor wc = weight.contiguous(), mean_c = mean.contiguous(), rstd_c = rstd.contiguous();
  if (dres) {
    dres = (dres->scalar_type() == type ? *dres : dres->to(type)).contiguous();
    TORCH_CHECK_VALUE(dres->sizes() == x.sizes(), "dres must have the shape of x: ", dres->sizes(), " against ", x.sizes());
  }
  const Tensor dx = empty(x.sizes(), type, dev), dgamma = empty({cols}, at::kFloat, dev), dbeta = empty({cols}, at::kFloat, dev);
  const Tensor ws = workspace(std::max<size_t>(rbf_b200_layer_norm_bwd_workspace_bytes(rows, cols), 16), dev);
  const int rc =
      rbf_b200_layer_norm_bwd_add(x.const_data_ptr(), dy.const_data_ptr(), dres ? dres->const_data_ptr() : nullptr,
                                  wc.const_data_ptr(), mean_c.const_data_ptr<float>(), rstd_c.const_data_ptr<float>(),
                                  dx.data_ptr(), dgamma.data_ptr<float>(), dbeta.data_ptr<float>(), ws.data_ptr(), ws.nbytes(),
                                  rows, cols, dtype_code(type), stream_of(x));
  check(rc, dres ? "rbf_b200_layer_norm_bwd_add" : "rbf_b200_layer_norm_bwd");
  const Tensor dgamma_out = dgamma.to(type), dbeta_out = dbeta.to(type);      // the type of weight
  unlocked.lock();
  return tuple(wrap(dx), wrap(dgamma_out), wrap(dbeta_out));
}

// (device index) -> whether the current stream of that device, which is the one that a call on its tensors uses, is being
// captured into a graph. (The question without a device is answered for the thread's current one.)
PyObject* capturing(const Args& a) {
  a.expect(1);
  const int64_t index = a.integer(0);
  if (c10::cuda::device_count() == 0) Py_RETURN_FALSE;
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(index));
  return PyBool_FromLong(c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None);
}

// ------------------------------------------------------------------ module
template <PyObject* (*kFn)(const Args&)>
PyObject* entry(PyObject* self, PyObject* const* argv, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return kFn(Args{argv, n, PyModule_GetName(self)});
  END_HANDLE_TH_ERRORS
}

template <PyObject* (*kFn)(const Args&)>
PyMethodDef method(const char* name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<kFn>)), METH_FASTCALL, nullptr};
}

PyMethodDef methods[] = {
    method<attention_fwd>("attention_fwd"),   method<attention_bwd>("attention_bwd"),
    method<block_fwd>("block_fwd"),           method<block_bwd>("block_bwd"),
    method<narrow_f32>("narrow_f32"),         method<widen_f16>("widen_f16"),
    method<column_sums>("column_sums"),       method<gelu_fwd>("gelu_fwd"),
    method<gelu_bwd>("gelu_bwd"),             method<layer_norm_fwd>("layer_norm_fwd"),
    method<layer_norm_bwd>("layer_norm_bwd"), method<capturing>("capturing"),
    method<validate_entry>("validate"),       method<tma_ready_entry>("tma_ready"),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  PyObject* m = PyModule_Create(&module);
  // the torch that this file was compiled against: no other one has the interface it calls
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", RBF_TORCH_VERSION) != 0) Py_CLEAR(m);
  return m;
}
