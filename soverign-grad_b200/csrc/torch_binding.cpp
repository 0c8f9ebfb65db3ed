// Native side of the Python package's hot calls: takes torch tensors and the package's own objects, allocates the
// outputs, and calls the C ABI of include/sgq.h.
//
// Why it exists: a decode-sized forward takes 5-10 us on the GPU, and the Python form of the call (attribute walks,
// contiguous / float checks, a ctypes call with sixteen converted arguments, the stream lookup) took 15-20 us on the
// host, so an eager token loop was bound by the host at every small size.  Arguments are parsed by hand
// (METH_FASTCALL), the GIL is released around the library call as ctypes does.
//
// No computation happens here, and nothing falls back: unusual inputs are converted by the same torch operations the
// Python code used (contiguous, float).
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>
#include <utility>
#include <vector>

#include "../../include/sgq.h"

namespace {

PyObject* g_error_class = nullptr;      // SgqError(status, what, detail)
PyObject* g_tensor_class = nullptr;     // QuantizedTensor(qdata, scales, scheme, original_shape, group_size, bits)
PyObject* g_workspace_class = nullptr;  // Workspace: .buf, .get(nbytes)

PyObject *s_qdata, *s_scales, *s_scheme, *s_shape, *s_group, *s_bits, *s_buf, *s_get;

// A reference that is given back at the end of the scope.
struct Ref {
    PyObject* p;
    explicit Ref(PyObject* o = nullptr) : p(o) {}
    ~Ref() { Py_XDECREF(p); }
    Ref(const Ref&) = delete;
    Ref& operator=(const Ref&) = delete;
    PyObject* release() { PyObject* o = p; p = nullptr; return o; }
    explicit operator bool() const { return p != nullptr; }
};

struct PythonError {};      // a Python exception is set

[[noreturn]] void raise(PyObject* type, const char* msg) {
    PyErr_SetString(type, msg);
    throw PythonError();
}

void check(int status, const char* what) {
    if (status == SGQ_OK) return;
    Ref args(Py_BuildValue("(iss)", status, (std::string(what) + " failed: " + sgq_status_string(status)).c_str(), sgq_last_error()));
    Ref exc(args ? PyObject_CallObject(g_error_class, args.p) : nullptr);
    if (exc) PyErr_SetObject(g_error_class, exc.p);
    throw PythonError();
}

int64_t as_int(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PythonError();
    return v;
}

const at::Tensor& as_tensor(PyObject* o) {
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, "a torch tensor is needed here");
    return THPVariable_Unpack(o);
}

// fp32, contiguous, on the GPU; the tensor itself where it already is
at::Tensor f32_cuda(PyObject* o) {
    const at::Tensor& t = as_tensor(o);
    if (!t.is_cuda()) raise(PyExc_ValueError, "this library computes on CUDA tensors only");
    if (t.scalar_type() == at::kFloat && t.is_contiguous()) return t;
    return t.contiguous().to(at::kFloat);
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Tensor& like) {
    return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt);
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// What a QuantizedTensor holds.  Its scheme is read for INT8 only and its group for INT4 only: what a checkpoint loader left
// in the other one does not matter.
struct Quantized {
    at::Tensor qdata, scales;
    int64_t scheme = SGQ_PER_TENSOR, group = 0, bits, rows = 0, cols = 0, numel = 1;
    size_t dims;
    Ref shape;
    explicit Quantized(PyObject* q) {
        Ref d(PyObject_GetAttr(q, s_qdata)), s(PyObject_GetAttr(q, s_scales)), b(PyObject_GetAttr(q, s_bits));
        shape.p = PyObject_GetAttr(q, s_shape);
        if (!d || !s || !b || !shape) throw PythonError();
        qdata = as_tensor(d.p);
        scales = as_tensor(s.p);
        bits = as_int(b.p);
        Ref v(PyObject_GetAttr(q, bits == 4 ? s_group : s_scheme));
        if (!v) throw PythonError();
        (bits == 4 ? group : scheme) = as_int(v.p);
        Ref seq(PySequence_Fast(shape.p, "original_shape is a sequence"));
        if (!seq) throw PythonError();
        dims = static_cast<size_t>(PySequence_Fast_GET_SIZE(seq.p));
        for (size_t i = 0; i < dims; ++i) {
            const int64_t v = as_int(PySequence_Fast_GET_ITEM(seq.p, i));
            if (i == 0) rows = v;
            if (i == 1) cols = v;
            numel *= v;
        }
    }
    // a single scale counts as per tensor whatever the scheme says (src/quantization.cpp:91)
    int scheme_now() const { return scheme == SGQ_PER_TENSOR || scales.numel() == 1 ? SGQ_PER_TENSOR : SGQ_PER_ROW; }
};

// The scratch of a call: what the caller's workspace gives for `need` bytes (None: nothing), or a buffer of this call.  The
// package's own Workspace is read directly while its buffer is large enough; any other object, a class derived from it
// included, is asked through its get().
struct Scratch {
    at::Tensor buf;
    void* ptr = nullptr;
    size_t bytes = 0;
    Scratch(PyObject* workspace, size_t need, const at::Tensor& like) {
        if (need == 0) return;
        if (workspace == Py_None) {
            buf = empty({static_cast<int64_t>(need)}, at::kByte, like);
        } else {
            Ref b;
            if (reinterpret_cast<PyObject*>(Py_TYPE(workspace)) == g_workspace_class) {
                b.p = PyObject_GetAttr(workspace, s_buf);
                if (!b) throw PythonError();
            }
            if (b && b.p != Py_None && static_cast<size_t>(as_tensor(b.p).numel()) >= need) {
                buf = as_tensor(b.p);
            } else {
                Ref n(PyLong_FromSize_t(need));
                Ref given(n ? PyObject_CallMethodOneArg(workspace, s_get, n.p) : nullptr);
                if (!given) throw PythonError();
                if (given.p == Py_None) return;
                buf = as_tensor(given.p);
            }
        }
        ptr = buf.data_ptr();
        bytes = static_cast<size_t>(buf.numel());
    }
};

// Calls into the library without the GIL, as ctypes does.
template <typename F>
int without_gil(F&& f) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f();
    Py_END_ALLOW_THREADS
    return rc;
}

template <PyObject* (*F)(PyObject* const*, Py_ssize_t)>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    try {
        return F(args, n);
    } catch (const PythonError&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

float* fptr(const at::Tensor& t) { return static_cast<float*>(t.data_ptr()); }

// bias as N fp32 values, or an empty tensor
at::Tensor bias_of(PyObject* o, int64_t N) {
    if (o == Py_None) return at::Tensor();
    at::Tensor b = f32_cuda(o);
    if (b.numel() != N) raise(PyExc_RuntimeError, "Incompatible shapes for broadcasting!");      // src/ops.cpp:60
    return b;
}

// quantized_matmul(x, q, bias, layout, path, out, workspace, ldy, workspace_limit)
PyObject* quantized_matmul(PyObject* const* a, Py_ssize_t n) {
    if (n != 9) raise(PyExc_TypeError, "quantized_matmul takes nine arguments");
    const at::Tensor x = f32_cuda(a[0]);
    if (x.dim() != 2) raise(PyExc_RuntimeError, "matmul currently requires 2D tensors!");
    const Quantized q(a[1]);
    const int layout = static_cast<int>(as_int(a[3])), path = static_cast<int>(as_int(a[4]));
    if (q.dims != 2) raise(PyExc_RuntimeError, "matmul currently requires 2D tensors!");                     // src/ops.cpp:380-382
    const int64_t K = layout == SGQ_LAYOUT_KN ? q.rows : q.cols, N = layout == SGQ_LAYOUT_KN ? q.cols : q.rows, M = x.size(0);
    if (x.size(1) != K) raise(PyExc_RuntimeError, "Matrix inner dimensions must match for matmul!");         // src/ops.cpp:387-389
    const at::Tensor bias = bias_of(a[2], N);
    at::Tensor out;
    int64_t ldy = N;
    if (a[5] == Py_None) {
        out = empty({M, N}, at::kFloat, x);
    } else {
        out = as_tensor(a[5]);
        ldy = a[7] == Py_None ? out.stride(0) : as_int(a[7]);
    }
    size_t need = sgq_linear_workspace_bytes(static_cast<int>(q.bits), M, K, N, layout, path);
    const bool limited = a[8] != Py_None;
    const size_t limit = limited ? static_cast<size_t>(as_int(a[8])) : 0;
    if (limited && need > limit) need = limit;
    Scratch ws(a[6], need, x);
    if (limited && ws.bytes > limit) ws.bytes = limit;
    void* s = stream();
    const float* b = bias.defined() ? fptr(bias) : nullptr;
    check(without_gil([&] {
              return q.bits == 4 ? sgq_linear_int4(fptr(x), M, K, N, static_cast<const uint8_t*>(q.qdata.data_ptr()), fptr(q.scales), layout,
                                                   q.group, b, fptr(out), ldy, path, ws.ptr, ws.bytes, s)
                                 : sgq_linear_int8(fptr(x), M, K, N, static_cast<const int8_t*>(q.qdata.data_ptr()), fptr(q.scales), layout,
                                                   q.scheme_now(), b, fptr(out), ldy, path, ws.ptr, ws.bytes, s);
          }),
          "sgq_linear");
    if (a[5] != Py_None) {
        Py_INCREF(a[5]);
        return a[5];
    }
    return THPVariable_Wrap(std::move(out));
}

// quantized_matmul_backward_x(dy, q, layout, path, workspace)
PyObject* backward_x(PyObject* const* a, Py_ssize_t n) {
    if (n != 5) raise(PyExc_TypeError, "quantized_matmul_backward_x takes five arguments");
    const at::Tensor dy = f32_cuda(a[0]);
    const Quantized q(a[1]);
    const int layout = static_cast<int>(as_int(a[2])), path = static_cast<int>(as_int(a[3]));
    if (q.dims != 2) raise(PyExc_RuntimeError, "matmul currently requires 2D tensors!");
    const int64_t K = layout == SGQ_LAYOUT_KN ? q.rows : q.cols, N = layout == SGQ_LAYOUT_KN ? q.cols : q.rows;
    if (dy.dim() != 2 || dy.size(1) != N) raise(PyExc_RuntimeError, "Matrix inner dimensions must match for matmul!");
    const int64_t M = dy.size(0);
    at::Tensor dx = empty({M, K}, at::kFloat, dy);
    Scratch ws(a[4], sgq_linear_backward_x_workspace_bytes(static_cast<int>(q.bits), M, K, N, layout, path), dy);
    void* s = stream();
    check(without_gil([&] {
              return q.bits == 4 ? sgq_linear_int4_backward_x(fptr(dy), M, K, N, static_cast<const uint8_t*>(q.qdata.data_ptr()),
                                                              fptr(q.scales), layout, q.group, fptr(dx), K, path, ws.ptr, ws.bytes, s)
                                 : sgq_linear_int8_backward_x(fptr(dy), M, K, N, static_cast<const int8_t*>(q.qdata.data_ptr()),
                                                              fptr(q.scales), layout, q.scheme_now(), fptr(dx), K, path, ws.ptr, ws.bytes, s);
          }),
          "sgq_linear_backward_x");
    return THPVariable_Wrap(std::move(dx));
}

// linear_w8a8(x, q, bias, want_parts).  Every shape is checked here, before the device: the library below sees pointers and
// M, K, N only, and a narrower x, packed INT4 codes or a short bias would be read past their end.
PyObject* linear_w8a8(PyObject* const* a, Py_ssize_t n) {
    if (n != 4) raise(PyExc_TypeError, "linear_w8a8 takes four arguments");
    const at::Tensor& given = as_tensor(a[0]);
    const Quantized q(a[1]);
    if (given.dim() != 2 || q.dims != 2) raise(PyExc_RuntimeError, "matmul currently requires 2D tensors!");
    if (q.bits != 8) raise(PyExc_RuntimeError, "linear_w8a8 needs an INT8 weight stored [N,K]");
    const int64_t N = q.rows, K = q.cols, M = given.size(0);
    if (given.size(1) != K) raise(PyExc_RuntimeError, "Matrix inner dimensions must match for matmul!");
    if (a[2] != Py_None && as_tensor(a[2]).numel() != N) raise(PyExc_RuntimeError, "Incompatible shapes for broadcasting!");
    const int parts_asked = PyObject_IsTrue(a[3]);
    if (parts_asked < 0) throw PythonError();
    const at::Tensor x = f32_cuda(a[0]), bias = bias_of(a[2], N);
    at::Tensor y = empty({M, N}, at::kFloat, x), xq, sx, acc;
    const bool parts = parts_asked == 1;
    if (parts) {
        xq = empty({M, K}, at::kChar, x);
        sx = empty({M}, at::kFloat, x);
        acc = empty({M, N}, at::kInt, x);
    }
    const size_t need = sgq_linear_w8a8_workspace_bytes(M, K, N);
    at::Tensor ws = empty({static_cast<int64_t>(need > 256 ? need : 256)}, at::kByte, x);
    void* s = stream();
    check(without_gil([&] {
              return sgq_linear_w8a8(fptr(x), M, K, N, static_cast<const int8_t*>(q.qdata.data_ptr()), fptr(q.scales), q.scheme_now(),
                                     bias.defined() ? fptr(bias) : nullptr, fptr(y), N,
                                     parts ? static_cast<int8_t*>(xq.data_ptr()) : nullptr, parts ? fptr(sx) : nullptr,
                                     parts ? static_cast<int32_t*>(acc.data_ptr()) : nullptr, ws.data_ptr(),
                                     static_cast<size_t>(ws.numel()), s);
          }),
          "sgq_linear_w8a8");
    if (!parts) return THPVariable_Wrap(std::move(y));
    return Py_BuildValue("(NNNN)", THPVariable_Wrap(y), THPVariable_Wrap(xq), THPVariable_Wrap(sx), THPVariable_Wrap(acc));
}

// A QuantizedTensor object; `shape` as the package keeps it (a plain tuple)
PyObject* wrap_quantized(const at::Tensor& x, at::Tensor& qdata, at::Tensor& scales, int64_t scheme, int64_t group, int64_t bits) {
    Ref shape(PyTuple_New(x.dim()));
    if (!shape) throw PythonError();
    for (int64_t i = 0; i < x.dim(); ++i) PyTuple_SET_ITEM(shape.p, i, PyLong_FromLongLong(x.size(i)));
    Ref q(THPVariable_Wrap(qdata)), s(THPVariable_Wrap(scales)), sch(PyLong_FromLongLong(scheme)), g(PyLong_FromLongLong(group)),
        b(PyLong_FromLongLong(bits));
    PyObject* args[6] = {q.p, s.p, sch.p, shape.p, g.p, b.p};
    PyObject* r = PyObject_Vectorcall(g_tensor_class, args, 6, nullptr);
    if (!r) throw PythonError();
    return r;
}

// quantize_int8(x, scheme)
PyObject* quantize_int8(PyObject* const* a, Py_ssize_t n) {
    if (n != 2) raise(PyExc_TypeError, "quantize_int8 takes two arguments");
    const at::Tensor x = f32_cuda(a[0]);
    const int64_t scheme = as_int(a[1]), numel = x.numel();
    const bool tensor = scheme == SGQ_PER_TENSOR || x.dim() < 2;        // src/quantization.cpp:22
    const int64_t rows = tensor ? 1 : x.size(0), cols = tensor ? numel : (rows ? numel / rows : 0);
    at::Tensor codes = empty(x.sizes(), at::kChar, x), scales = empty({rows}, at::kFloat, x);
    void* s = stream();
    check(without_gil([&] {
              return sgq_quantize_int8(fptr(x), rows, cols, tensor ? SGQ_PER_TENSOR : SGQ_PER_ROW, static_cast<int8_t*>(codes.data_ptr()),
                                       fptr(scales), s);
          }),
          "sgq_quantize_int8");
    return wrap_quantized(x, codes, scales, scheme, numel, 8);
}

// quantize_int4(x, group_size)
PyObject* quantize_int4(PyObject* const* a, Py_ssize_t n) {
    if (n != 2) raise(PyExc_TypeError, "quantize_int4 takes two arguments");
    const at::Tensor x = f32_cuda(a[0]);
    const int64_t asked = as_int(a[1]), group = asked <= 0 ? 32 : asked, numel = x.numel();
    at::Tensor packed = empty({(numel + 1) / 2}, at::kByte, x), scales = empty({(numel + group - 1) / group}, at::kFloat, x);
    void* s = stream();
    check(without_gil([&] {
              return sgq_quantize_int4(fptr(x), numel, group, static_cast<uint8_t*>(packed.data_ptr()), fptr(scales), s);
          }),
          "sgq_quantize_int4");
    return wrap_quantized(x, packed, scales, SGQ_PER_TENSOR, group, 4);
}

// dequantize(q): either bit width
PyObject* dequantize(PyObject* const* a, Py_ssize_t n) {
    if (n != 1) raise(PyExc_TypeError, "dequantize takes one argument");
    const Quantized q(a[0]);
    std::vector<int64_t> sizes;
    Ref seq(PySequence_Fast(q.shape.p, "original_shape is a sequence"));
    if (!seq) throw PythonError();
    for (size_t i = 0; i < q.dims; ++i) sizes.push_back(as_int(PySequence_Fast_GET_ITEM(seq.p, i)));
    at::Tensor out = empty(sizes, at::kFloat, q.qdata);
    void* s = stream();
    if (q.bits == 4) {
        check(without_gil([&] {
                  return sgq_dequantize_int4(static_cast<const uint8_t*>(q.qdata.data_ptr()), fptr(q.scales), q.numel, q.group, fptr(out), s);
              }),
              "sgq_dequantize_int4");
    } else {
        const int scheme = q.scheme_now();
        const int64_t rows = scheme == SGQ_PER_TENSOR ? 1 : q.rows, cols = rows ? q.numel / rows : 0;
        check(without_gil([&] {
                  return sgq_dequantize_int8(static_cast<const int8_t*>(q.qdata.data_ptr()), fptr(q.scales), rows, cols, scheme, fptr(out), s);
              }),
              "sgq_dequantize_int8");
    }
    return THPVariable_Wrap(std::move(out));
}

// set_classes(SgqError, QuantizedTensor, Workspace)
PyObject* set_classes(PyObject* const* a, Py_ssize_t n) {
    if (n != 3) raise(PyExc_TypeError, "set_classes takes three arguments");
    PyObject** const classes[] = {&g_error_class, &g_tensor_class, &g_workspace_class};
    for (int i = 0; i < 3; ++i) {
        Py_INCREF(a[i]);
        Py_XDECREF(*classes[i]);
        *classes[i] = a[i];
    }
    Py_RETURN_NONE;
}

#define SGQ_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<name>)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {
    SGQ_METHOD(quantized_matmul), SGQ_METHOD(backward_x), SGQ_METHOD(linear_w8a8), SGQ_METHOD(quantize_int8),
    SGQ_METHOD(quantize_int4),    SGQ_METHOD(dequantize), SGQ_METHOD(set_classes), {nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_sgq_torch", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__sgq_torch(void) {
    s_qdata = PyUnicode_InternFromString("qdata");
    s_scales = PyUnicode_InternFromString("scales");
    s_scheme = PyUnicode_InternFromString("scheme");
    s_shape = PyUnicode_InternFromString("original_shape");
    s_group = PyUnicode_InternFromString("group_size");
    s_bits = PyUnicode_InternFromString("bits");
    s_buf = PyUnicode_InternFromString("buf");
    s_get = PyUnicode_InternFromString("get");
    return PyModule_Create(&g_module);
}
