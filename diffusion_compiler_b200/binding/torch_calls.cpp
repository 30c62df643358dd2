// The short way into libdifb200.so for calls on ordinary tensors: arguments read, outputs allocated and the C entry point
// called in native code. A small call is a few microseconds on the GPU (a linear of two rows 5), and interpreted glue
// around the same entry point took 7 to 10 of its 13: two allocations through the Python API 4, the conversion of 14
// arguments 2, attribute reads and checks the rest. us of the host per call, before -> here: a linear of 2 rows 13.4 -> 8.1,
// quantising 16 rows 13.0 -> 6.0, attention of 64 tokens 14.1 -> 10.7 (then the GPU).
//
// A function here takes what it can serve without a copy: dense tensors of torch.Tensor itself on the current CUDA device,
// of the right type, with the shapes that the entry point wants. For everything else it returns None, and ops.py goes its
// general way, which copies, converts or raises. A status other than 0 comes back as an int.
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>

#include "difb200/difb200.h"

namespace {

using Args = PyObject *const *;

PyObject *none() { Py_RETURN_NONE; }

// The current CUDA device where `o` is a CUDA tensor and no mode stands between a call and its tensors, else -1.
c10::DeviceIndex device_of_call(PyObject *o) {
  if (!THPVariable_CheckExact(o) || !THPVariable_Unpack(o).is_cuda() || c10::impl::TorchDispatchModeTLS::any_modes_set())
    return -1;
  return c10::cuda::current_device();
}

// The tensor behind `o` if it is one of these; the reference is borrowed from the object.
const at::Tensor *dense(PyObject *o, at::ScalarType type, c10::DeviceIndex device) {
  if (!THPVariable_CheckExact(o))
    return nullptr;
  const at::Tensor &t = THPVariable_Unpack(o);
  return t.layout() == at::kStrided && t.is_cuda() && t.get_device() == device && t.scalar_type() == type && t.has_storage() && t.is_contiguous() &&
                 !t.requires_grad() && !t.is_conj() && !t.is_neg()
             ? &t
             : nullptr;
}

at::Tensor make(at::IntArrayRef shape, at::ScalarType type, const at::Tensor &like) {
  return at::empty(shape, like.options().dtype(type).requires_grad(false));
}

template <typename T = void>
const T *in(const at::Tensor *t) {
  return t ? static_cast<const T *>(t->const_data_ptr()) : nullptr;
}
template <typename T = void>
T *out_of(const at::Tensor &t) {
  return static_cast<T *>(t.mutable_data_ptr());
}

// `call` holds plain pointers and numbers: nothing in it may throw, the interpreter's lock is given up around it.
template <typename F>
PyObject *finish(F call, const at::Tensor &a, const at::Tensor *b = nullptr) {
  int status;
  Py_BEGIN_ALLOW_THREADS status = call();
  Py_END_ALLOW_THREADS if (status != 0) return PyLong_FromLong(status);
  if (!b)
    return THPVariable_Wrap(a);
  PyObject *first = THPVariable_Wrap(a), *second = THPVariable_Wrap(*b);
  PyObject *both = first && second ? PyTuple_Pack(2, first, second) : nullptr;
  Py_XDECREF(first);
  Py_XDECREF(second);
  return both;
}

// Where an allocation fails the general way does it again, and raises as torch does. Nothing was launched by then.
template <typename F>
PyObject *guarded(F body) {
  try {
    return body();
  } catch (const std::exception &) {
    return none();
  }
}

// (x, w8, col_scales, bias or None, gelu, implementation, clip)
PyObject *w8a8_linear(PyObject *, Args args, Py_ssize_t n) {
  return guarded([&]() -> PyObject * {
    const auto device = n == 7 ? device_of_call(args[0]) : -1;
    if (device < 0)
      return none();
    const at::Tensor *x = dense(args[0], at::kBFloat16, device), *w = dense(args[1], at::kChar, device),
                     *ws = dense(args[2], at::kFloat, device), *bias = nullptr;
    if (!x || !w || !ws || x->dim() < 1 || w->dim() != 2 || x->numel() == 0)
      return none();
    if (args[3] != Py_None && !(bias = dense(args[3], at::kBFloat16, device)))
      return none();
    const int64_t K = x->size(-1), M = x->numel() / K, N = w->size(0);
    if (w->size(1) != K || ws->numel() != N || (bias && bias->numel() != N))
      return none();
    const int gelu = PyObject_IsTrue(args[4]);
    const long implementation = PyLong_AsLong(args[5]);
    const double clip = PyFloat_AsDouble(args[6]);
    if (PyErr_Occurred()) {
      PyErr_Clear();
      return none();
    }
    const uint32_t flags = (bias ? 1u : 0u) | (gelu ? 2u : 0u);
    const int64_t at = (M * K + 15) / 16 * 16; // the codes, then the row scales on the next 16 bytes
    const at::Tensor scratch = make({at + 4 * M}, at::kByte, *x);
    auto shape = x->sizes().vec();
    shape.back() = N;
    const at::Tensor out = make(shape, at::kBFloat16, *x);
    int8_t *codes = out_of<int8_t>(scratch);
    const void *px = in(x), *pb = in(bias);
    const int8_t *pw = in<int8_t>(w);
    const float *ps = in<float>(ws);
    void *po = out_of(out), *stream = c10::cuda::getCurrentCUDAStream(device).stream();
    return finish(
        [=] {
          return difb200_w8a8_linear(px, pw, ps, pb, flags, (int32_t)implementation, (float)clip, (uint64_t)M, (uint64_t)N, (uint64_t)K,
                                     codes, reinterpret_cast<float *>(codes + at), po, stream);
        },
        out);
  });
}

// (list of inputs, implementation, clip)
PyObject *quantize_int8_rows(PyObject *, Args args, Py_ssize_t n) {
  return guarded([&]() -> PyObject * {
    const Py_ssize_t count = n == 3 && PyList_CheckExact(args[0]) ? PyList_GET_SIZE(args[0]) : 0;
    const auto device = count >= 1 && count <= 8 ? device_of_call(PyList_GET_ITEM(args[0], 0)) : -1;
    if (device < 0)
      return none();
    const void *parts[8];
    uint64_t widths[8], total = 0;
    at::Tensor held[8]; // the list may change while arguments are converted and while the lock is given up
    const at::Tensor *first = nullptr;
    for (Py_ssize_t i = 0; i < count; ++i) {
      const at::Tensor *t = dense(PyList_GET_ITEM(args[0], i), at::kBFloat16, device);
      if (!t || t->dim() < 1 || t->numel() == 0)
        return none();
      held[i] = *t;
      if (i == 0)
        first = &held[0];
      else if (t->dim() != first->dim() || t->sizes().slice(0, t->dim() - 1) != first->sizes().slice(0, t->dim() - 1))
        return none();
      parts[i] = in(t);
      total += widths[i] = (uint64_t)t->size(-1);
    }
    const long implementation = PyLong_AsLong(args[1]);
    const double clip = PyFloat_AsDouble(args[2]);
    if (PyErr_Occurred()) {
      PyErr_Clear();
      return none();
    }
    const int64_t rows = first->numel() / first->size(-1);
    auto shape = first->sizes().vec();
    shape.back() = (int64_t)total;
    const at::Tensor codes = make(shape, at::kChar, *first), scales = make({rows}, at::kFloat, *first);
    int8_t *pc = out_of<int8_t>(codes);
    float *ps = out_of<float>(scales);
    void *stream = c10::cuda::getCurrentCUDAStream(device).stream();
    return finish(
        [&] {
          return difb200_quantize_int8_rows(parts, widths, (uint32_t)count, (uint64_t)rows, (int32_t)implementation, (float)clip, nullptr,
                                            pc, ps, nullptr, nullptr, stream);
        },
        codes, &scales);
  });
}

// (x, weight, bias or None, scale, shift, epsilon, implementation, clip): the layer norm where there is a bias
PyObject *norm_modulate_quant(PyObject *, Args args, Py_ssize_t n) {
  return guarded([&]() -> PyObject * {
    const auto device = n == 8 ? device_of_call(args[0]) : -1;
    if (device < 0)
      return none();
    const bool layer = args[2] != Py_None;
    const at::Tensor *x = dense(args[0], at::kBFloat16, device), *weight = nullptr, *bias = nullptr,
                     *scale = dense(args[3], at::kBFloat16, device), *shift = dense(args[4], at::kBFloat16, device);
    if (!x || !scale || !shift || x->dim() != 2 || x->numel() == 0 || scale->dim() != 2 || scale->sizes() != shift->sizes() ||
        scale->size(1) != x->size(1) || scale->size(0) == 0)
      return none();
    if ((layer || args[1] != Py_None) && !(weight = dense(args[1], at::kBFloat16, device)))
      return none();
    if (layer && !(bias = dense(args[2], at::kBFloat16, device)))
      return none();
    if ((weight && weight->numel() != x->size(1)) || (bias && bias->numel() != x->size(1)))
      return none();
    const double epsilon = PyFloat_AsDouble(args[5]), clip = PyFloat_AsDouble(args[7]);
    const long implementation = PyLong_AsLong(args[6]);
    if (PyErr_Occurred()) {
      PyErr_Clear();
      return none();
    }
    const int64_t M = x->size(0), K = x->size(1), mods = scale->size(0);
    if (layer ? M % mods != 0 : mods != M)
      return none();
    const at::Tensor codes = make({M, K}, at::kChar, *x), scales = make({M}, at::kFloat, *x);
    int8_t *pc = out_of<int8_t>(codes);
    float *ps = out_of<float>(scales);
    const void *px = in(x), *pw = in(weight), *pb = in(bias), *pscale = in(scale), *pshift = in(shift);
    void *stream = c10::cuda::getCurrentCUDAStream(device).stream();
    return finish(
        [=] {
          return layer ? difb200_layer_norm_modulate_quant(px, pw, pb, pscale, pshift, (uint64_t)M, (uint64_t)K, (uint64_t)(M / mods),
                                                           (float)epsilon, (int32_t)implementation, (float)clip, pc, ps, stream)
                       : difb200_rms_norm_modulate_quant(px, pw, pscale, pshift, (uint64_t)M, (uint64_t)K, (float)epsilon,
                                                         (int32_t)implementation, (float)clip, pc, ps, stream);
        },
        codes, &scales);
  });
}

// (q, k, v, key_valid or None, scale or None)
PyObject *attention(PyObject *, Args args, Py_ssize_t n) {
  return guarded([&]() -> PyObject * {
    const auto device = n == 5 ? device_of_call(args[0]) : -1;
    if (device < 0)
      return none();
    const at::Tensor *q = dense(args[0], at::kBFloat16, device), *k = dense(args[1], at::kBFloat16, device),
                     *v = dense(args[2], at::kBFloat16, device), *valid = nullptr;
    if (!q || !k || !v || q->dim() != 4 || k->dim() != 4 || q->numel() == 0 || k->numel() == 0 || v->sizes() != k->sizes() ||
        k->size(0) != q->size(0) || k->size(1) != q->size(1) || k->size(3) != q->size(3))
      return none();
    const int64_t B = q->size(0), S = q->size(1), H = q->size(2), D = q->size(3), KV = k->size(2);
    if (args[3] != Py_None && (!(valid = dense(args[3], at::kByte, device)) || valid->numel() != B * S))
      return none();
    const double scale = args[4] == Py_None ? 1.0 / std::sqrt((double)D) : PyFloat_AsDouble(args[4]);
    if (PyErr_Occurred()) {
      PyErr_Clear();
      return none();
    }
    const uint64_t bytes = difb200_attention_scratch_bytes((uint64_t)B, (uint64_t)S, (uint64_t)H, (uint64_t)KV);
    const at::Tensor out = make({B, S, H, D}, at::kBFloat16, *q), scratch = make({(int64_t)bytes}, at::kByte, *q);
    const void *pq = in(q), *pk = in(k), *pv = in(v);
    const uint8_t *pm = in<uint8_t>(valid);
    void *ps = out_of(scratch), *po = out_of(out), *stream = c10::cuda::getCurrentCUDAStream(device).stream();
    return finish(
        [=] {
          return difb200_attention(pq, pk, pv, pm, (uint64_t)B, (uint64_t)S, (uint64_t)H, (uint64_t)KV, (uint64_t)D, (float)scale, ps,
                                   bytes, po, stream);
        },
        out);
  });
}

#define DIFB200_METHOD(NAME) {#NAME, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(NAME)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {DIFB200_METHOD(w8a8_linear), DIFB200_METHOD(quantize_int8_rows), DIFB200_METHOD(norm_modulate_quant),
                         DIFB200_METHOD(attention), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__torch_calls() { return PyModule_Create(&module); }
