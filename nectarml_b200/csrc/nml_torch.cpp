// Tensor-level host path in native code: unpacks torch tensors, checks them, allocates the result and calls
// the C ABI of include/nectarml_b200.h.  Built into nectarml_b200/_native.so; nectarml_b200/ops.py and
// train.py are the only callers.
//
// Why it exists: a layer call from Python spent 12 us around a C-ABI call of 4 us (ctypes conversions, stream
// lookup through torch.cuda, descriptor fields set one by one, shape tuples), more than most small layers run
// on the GPU.  Here the same work is about 2 us: linear 32 x 512 -> 2048 forward 16.2 -> 7 us per call.
//
// Nothing is kept between calls except the parsed geometry of a layer (a capsule owned by the Python
// ConvGeometry object).  The GIL stays held: every function returns within a few microseconds.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <exception>

#include "../../include/nectarml_b200.h"

namespace {

PyObject* g_error = nullptr;  // nectarml_b200._lib.NectarB200Error

struct Fail {};  // a Python exception is set

[[noreturn]] void fail(const char* msg) {
    PyErr_SetString(g_error, msg);
    throw Fail();
}
[[noreturn]] void fail_assert(const char* what) {
    PyErr_SetString(PyExc_AssertionError, what);
    throw Fail();
}
inline void require(bool ok, const char* what) {
    if (!ok) fail_assert(what);
}
inline void check(int status) {
    if (status == NML_OK) return;
    PyErr_Format(g_error, "nectarml_b200 status %d: %s", status, nml_status_string(status));
    throw Fail();
}

const at::Tensor& tensor(PyObject* o, const char* what) {
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s: a tensor is expected", what);
        throw Fail();
    }
    return THPVariable_Unpack(o);
}
inline const at::Tensor* tensor_or_none(PyObject* o, const char* what) { return o == Py_None ? nullptr : &tensor(o, what); }

int dtype_of(const at::Tensor& t) {
    const auto s = t.scalar_type();
    if (s == at::kFloat) return NML_F32;
    if (s == at::kHalf) return NML_F16;
    fail("only float32 and float16 tensors are supported");
}
void* ptr(const at::Tensor& t) {
    if (!t.is_cuda()) fail("tensors must live on a CUDA device (there is no CPU path)");
    if (!t.is_contiguous()) fail("tensors must be contiguous");
    return t.data_ptr();
}
inline void* ptr_or_null(const at::Tensor* t) { return t ? ptr(*t) : nullptr; }
inline void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

long as_int(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw Fail();
    return v;
}
double as_double(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Fail();
    return v;
}

// An output: the caller's tensor, or a new one (dtype code -1: like `like`).
at::Tensor output(PyObject* given, at::IntArrayRef shape, long dtype_code, const at::Tensor& like) {
    if (given != Py_None) return tensor(given, "out");
    const auto st = dtype_code < 0 ? like.scalar_type() : dtype_code == NML_F16 ? at::kHalf : at::kFloat;
    return at::empty(shape, at::TensorOptions().dtype(st).device(like.device()));
}

// Scratch from the caller's Workspace object (a grow-only buffer, see ops.Workspace): its tensor as it is while it is
// large enough and on the right device, else through its own get().
struct Scratch {
    void* p = nullptr;
    size_t bytes = 0;
};
Scratch scratch(PyObject* ws, size_t need, const at::Tensor& like) {
    static PyObject* const kBuf = PyUnicode_InternFromString("buf");
    static PyObject* const kGet = PyUnicode_InternFromString("get");
    Scratch s;
    if (need == 0) return s;
    for (int attempt = 0; attempt < 2; ++attempt) {
        PyObject* buf = PyObject_GetAttr(ws, kBuf);
        if (!buf) throw Fail();
        if (THPVariable_Check(buf)) {
            const at::Tensor& t = THPVariable_Unpack(buf);
            if (static_cast<size_t>(t.numel()) >= need && t.device() == like.device()) {
                s.p = t.data_ptr();
                s.bytes = t.numel();
                Py_DECREF(buf);
                return s;
            }
        }
        Py_DECREF(buf);
        if (attempt == 1) break;
        PyObject* size = PyLong_FromSize_t(need);
        PyObject* dev = THPVariable_Wrap(like);
        PyObject* device = dev ? PyObject_GetAttrString(dev, "device") : nullptr;
        PyObject* r = (size && device) ? PyObject_CallMethodObjArgs(ws, kGet, size, device, nullptr) : nullptr;
        Py_XDECREF(device);
        Py_XDECREF(dev);
        Py_XDECREF(size);
        if (!r) throw Fail();
        Py_DECREF(r);
    }
    fail("the workspace object did not grow");
}

// Runs a function body with C++ exceptions turned into Python ones.
template <class F>
PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (const Fail&) {
    } catch (const std::exception& e) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}
PyObject* pair(const at::Tensor& a, const at::Tensor* b) {
    PyObject* pa = THPVariable_Wrap(a);
    PyObject* pb = b ? THPVariable_Wrap(*b) : Py_NewRef(Py_None);
    if (!pa || !pb) {
        Py_XDECREF(pa);
        Py_XDECREF(pb);
        return nullptr;
    }
    PyObject* t = PyTuple_New(2);
    PyTuple_SET_ITEM(t, 0, pa);
    PyTuple_SET_ITEM(t, 1, pb);
    return t;
}
bool arity(Py_ssize_t n, Py_ssize_t want) {
    if (n == want) return true;
    PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, n);
    return false;
}

// ------------------------------------------------------------------ convolution --
struct Geometry {
    nml_conv_desc d;
    int ho = 0, wo = 0, status = 0;
};
const char* const kGeometryName = "nectarml_b200.geometry";

// geometry(batch, c_in, h, w, c_out, kh, kw, sh, sw, ph, pw, dh, dw, oph, opw, transposed)
PyObject* py_geometry(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 16)) return nullptr;
    return guarded([&]() -> PyObject* {
        auto* g = new Geometry();
        std::memset(&g->d, 0, sizeof(g->d));
        int* const f[16] = {&g->d.batch, &g->d.c_in, &g->d.h, &g->d.w, &g->d.c_out, &g->d.kh, &g->d.kw, &g->d.stride_h,
                            &g->d.stride_w, &g->d.pad_h, &g->d.pad_w, &g->d.dil_h, &g->d.dil_w, &g->d.outpad_h,
                            &g->d.outpad_w, &g->d.transposed};
        try {
            for (int i = 0; i < 16; ++i) *f[i] = static_cast<int>(as_int(a[i]));
        } catch (...) {
            delete g;
            throw;
        }
        g->status = nml_conv_output_size(&g->d, &g->ho, &g->wo);
        return PyCapsule_New(g, kGeometryName, [](PyObject* c) {
            delete static_cast<Geometry*>(PyCapsule_GetPointer(c, kGeometryName));
        });
    });
}
const Geometry& geometry(PyObject* o) {
    auto* g = static_cast<Geometry*>(PyCapsule_GetPointer(o, kGeometryName));
    if (!g) throw Fail();
    check(g->status);
    return *g;
}
bool is_act(const at::Tensor& t, const Geometry& g, bool input, int layout) {
    const int64_t c = input ? g.d.c_in : g.d.c_out, h = input ? g.d.h : g.ho, w = input ? g.d.w : g.wo;
    if (t.dim() != 4 || t.size(0) != g.d.batch) return false;
    return layout == NML_NCHW ? (t.size(1) == c && t.size(2) == h && t.size(3) == w)
                              : (t.size(1) == h && t.size(2) == w && t.size(3) == c);
}
void act_shape(const Geometry& g, bool input, int layout, int64_t (&s)[4]) {
    const int64_t c = input ? g.d.c_in : g.d.c_out, h = input ? g.d.h : g.ho, w = input ? g.d.w : g.wo;
    s[0] = g.d.batch;
    s[1] = layout == NML_NCHW ? c : h;
    s[2] = layout == NML_NCHW ? h : w;
    s[3] = layout == NML_NCHW ? w : c;
}
void weight_shape(const Geometry& g, int64_t (&s)[4]) {
    s[0] = g.d.transposed ? g.d.c_in : g.d.c_out;
    s[1] = g.d.transposed ? g.d.c_out : g.d.c_in;
    s[2] = g.d.kh;
    s[3] = g.d.kw;
}
bool is_weight(const at::Tensor& t, const Geometry& g) {
    int64_t s[4];
    weight_shape(g, s);
    return t.dim() == 4 && t.size(0) == s[0] && t.size(1) == s[1] && t.size(2) == s[2] && t.size(3) == s[3];
}

// conv_forward(geometry, x, w, bias, out, layout, out_layout, math, out_dtype, round_f16, workspace)
PyObject* py_conv_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 11)) return nullptr;
    return guarded([&]() -> PyObject* {
        const Geometry& g = geometry(a[0]);
        const at::Tensor &x = tensor(a[1], "x"), &w = tensor(a[2], "w");
        const at::Tensor* bias = tensor_or_none(a[3], "bias");
        nml_conv_desc d = g.d;
        d.in_layout = static_cast<int>(as_int(a[5]));
        d.out_layout = static_cast<int>(as_int(a[6]));
        require(is_act(x, g, true, d.in_layout), "x does not have the layer's input shape");
        require(is_weight(w, g), "w does not have the layer's weight shape");
        if (bias) require(bias->scalar_type() == w.scalar_type() && bias->numel() == g.d.c_out, "bias: dtype of w, one value per output channel");
        int64_t s[4];
        act_shape(g, false, d.out_layout, s);
        const at::Tensor out = output(a[4], s, as_int(a[8]), x);
        d.in_dtype = dtype_of(x);
        d.out_dtype = dtype_of(out);
        d.w_dtype = dtype_of(w);
        d.math = static_cast<int>(as_int(a[7]));
        d.round_out_f16 = static_cast<int>(as_int(a[9]));
        size_t need = 0;
        check(nml_conv_workspace_size(&d, NML_PASS_FORWARD, &need));
        const Scratch ws = scratch(a[10], need, x);
        check(nml_conv_forward(&d, ptr(x), ptr(w), ptr_or_null(bias), ptr(out), ws.p, ws.bytes, stream()));
        return THPVariable_Wrap(out);
    });
}

// conv_backward_data(geometry, dy, w, out, layout, out_layout, math, out_dtype, workspace)
PyObject* py_conv_backward_data(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 9)) return nullptr;
    return guarded([&]() -> PyObject* {
        const Geometry& g = geometry(a[0]);
        const at::Tensor &dy = tensor(a[1], "dy"), &w = tensor(a[2], "w");
        nml_conv_desc d = g.d;
        d.in_layout = static_cast<int>(as_int(a[4]));
        d.out_layout = static_cast<int>(as_int(a[5]));
        require(is_act(dy, g, false, d.in_layout), "dy does not have the layer's output shape");
        require(is_weight(w, g), "w does not have the layer's weight shape");
        int64_t s[4];
        act_shape(g, true, d.out_layout, s);
        const at::Tensor out = output(a[3], s, as_int(a[7]), dy);
        d.in_dtype = dtype_of(dy);
        d.out_dtype = dtype_of(out);
        d.w_dtype = dtype_of(w);
        d.math = static_cast<int>(as_int(a[6]));
        size_t need = 0;
        check(nml_conv_workspace_size(&d, NML_PASS_BACKWARD_DATA, &need));
        const Scratch ws = scratch(a[8], need, dy);
        check(nml_conv_backward_data(&d, ptr(dy), ptr(w), ptr(out), ws.p, ws.bytes, stream()));
        return THPVariable_Wrap(out);
    });
}

// conv_backward_weight(geometry, x, dy, dw, db, layout, math, want_bias_grad, workspace) -> (dw, db)
PyObject* py_conv_backward_weight(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 9)) return nullptr;
    return guarded([&]() -> PyObject* {
        const Geometry& g = geometry(a[0]);
        const at::Tensor &x = tensor(a[1], "x"), &dy = tensor(a[2], "dy");
        nml_conv_desc d = g.d;
        d.in_layout = d.out_layout = static_cast<int>(as_int(a[5]));
        require(is_act(x, g, true, d.in_layout), "x does not have the layer's input shape");
        require(is_act(dy, g, false, d.in_layout), "dy does not have the layer's output shape");
        require(x.scalar_type() == dy.scalar_type(), "x and dy have one dtype");
        int64_t s[4];
        weight_shape(g, s);
        const at::Tensor dw = output(a[3], s, NML_F32, x);
        at::Tensor db;
        const bool has_db = a[4] != Py_None || as_int(a[7]) != 0;
        if (has_db) db = output(a[4], {g.d.c_out}, NML_F32, x);
        require(dw.scalar_type() == at::kFloat && dw.numel() == s[0] * s[1] * s[2] * s[3], "dw is float32 and has the weight's elements");
        d.in_dtype = dtype_of(x);
        d.out_dtype = d.w_dtype = NML_F32;
        d.math = static_cast<int>(as_int(a[6]));
        size_t need = 0;
        check(nml_conv_workspace_size(&d, NML_PASS_BACKWARD_WEIGHT, &need));
        const Scratch ws = scratch(a[8], need, x);
        check(nml_conv_backward_weight(&d, ptr(x), ptr(dy), static_cast<float*>(ptr(dw)),
                                       has_db ? static_cast<float*>(ptr(db)) : nullptr, ws.p, ws.bytes, stream()));
        return pair(dw, has_db ? &db : nullptr);
    });
}

// ------------------------------------------------------------------ linear --
nml_linear_desc linear_desc(int64_t rows, int64_t fin, int64_t fout, long math) {
    nml_linear_desc d;
    std::memset(&d, 0, sizeof(d));
    d.rows = static_cast<int>(rows);
    d.in_features = static_cast<int>(fin);
    d.out_features = static_cast<int>(fout);
    d.math = static_cast<int>(math);
    return d;
}

// linear_forward(x, w, bias, out, math, out_dtype, round_f16, workspace)
PyObject* py_linear_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 8)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &x = tensor(a[0], "x"), &w = tensor(a[1], "w");
        const at::Tensor* bias = tensor_or_none(a[2], "bias");
        require(x.dim() == 2 && w.dim() == 2 && w.size(1) == x.size(1), "x [rows, in], w [out, in]");
        nml_linear_desc d = linear_desc(x.size(0), x.size(1), w.size(0), as_int(a[4]));
        const at::Tensor out = output(a[3], {x.size(0), w.size(0)}, as_int(a[5]), x);
        d.in_dtype = dtype_of(x);
        d.out_dtype = dtype_of(out);
        d.w_dtype = dtype_of(w);
        d.round_out_f16 = static_cast<int>(as_int(a[6]));
        size_t need = 0;
        check(nml_linear_workspace_size(&d, NML_PASS_FORWARD, &need));
        const Scratch ws = scratch(a[7], need, x);
        check(nml_linear_forward(&d, ptr(x), ptr(w), ptr_or_null(bias), ptr(out), ws.p, ws.bytes, stream()));
        return THPVariable_Wrap(out);
    });
}

// linear_backward_data(dy, w, out, math, out_dtype, workspace)
PyObject* py_linear_backward_data(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 6)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &dy = tensor(a[0], "dy"), &w = tensor(a[1], "w");
        require(dy.dim() == 2 && w.dim() == 2 && w.size(0) == dy.size(1), "dy [rows, out], w [out, in]");
        nml_linear_desc d = linear_desc(dy.size(0), w.size(1), dy.size(1), as_int(a[3]));
        const at::Tensor out = output(a[2], {dy.size(0), w.size(1)}, as_int(a[4]), dy);
        d.in_dtype = dtype_of(dy);
        d.out_dtype = dtype_of(out);
        d.w_dtype = dtype_of(w);
        size_t need = 0;
        check(nml_linear_workspace_size(&d, NML_PASS_BACKWARD_DATA, &need));
        const Scratch ws = scratch(a[5], need, dy);
        check(nml_linear_backward_data(&d, ptr(dy), ptr(w), ptr(out), ws.p, ws.bytes, stream()));
        return THPVariable_Wrap(out);
    });
}

// linear_backward_weight(x, dy, dw, db, math, want_bias_grad, workspace) -> (dw, db)
PyObject* py_linear_backward_weight(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 7)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &x = tensor(a[0], "x"), &dy = tensor(a[1], "dy");
        require(x.dim() == 2 && dy.dim() == 2 && x.size(0) == dy.size(0) && x.scalar_type() == dy.scalar_type(),
                "x [rows, in], dy [rows, out] of one dtype");
        nml_linear_desc d = linear_desc(x.size(0), x.size(1), dy.size(1), as_int(a[4]));
        const at::Tensor dw = output(a[2], {dy.size(1), x.size(1)}, NML_F32, x);
        at::Tensor db;
        const bool has_db = a[3] != Py_None || as_int(a[5]) != 0;
        if (has_db) db = output(a[3], {dy.size(1)}, NML_F32, x);
        d.in_dtype = dtype_of(x);
        d.out_dtype = d.w_dtype = NML_F32;
        size_t need = 0;
        check(nml_linear_workspace_size(&d, NML_PASS_BACKWARD_WEIGHT, &need));
        const Scratch ws = scratch(a[6], need, x);
        check(nml_linear_backward_weight(&d, ptr(x), ptr(dy), static_cast<float*>(ptr(dw)),
                                         has_db ? static_cast<float*>(ptr(db)) : nullptr, ws.p, ws.bytes, stream()));
        return pair(dw, has_db ? &db : nullptr);
    });
}

// ------------------------------------------------------------------ batch norm, activation --
// Concatenations along the channels are not made by a pass of their own: the first of the two layers whose outputs meet
// allocates the wide tensor and writes a second copy of its output into its last channels (`skip`), the other one writes its
// output into the first channels (`join`).  In the backward each reads its part of the wide tensor's gradient in place.
PyObject* wrap_or_none(const at::Tensor& t) { return t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None); }
template <class... T>
PyObject* tuple_of(const T&... t) {
    PyObject* const items[] = {wrap_or_none(t)...};
    PyObject* r = PyTuple_New(sizeof...(t));
    for (size_t i = 0; i < sizeof...(t); ++i) PyTuple_SET_ITEM(r, i, items[i]);
    return r;
}
at::Tensor wide_like(const at::Tensor& x) {
    auto shape = x.sizes().vec();
    shape.back() *= 2;
    return at::empty(shape, x.options());
}
void* channels_from(const at::Tensor& wide, int64_t c) { return static_cast<char*>(ptr(wide)) + c * wide.element_size(); }
void require_half_rows(const at::Tensor& t, const at::Tensor& x, int64_t c, const char* what) {
    require(t.scalar_type() == at::kHalf && t.numel() / t.size(-1) == x.numel() / x.size(-1) && t.size(-1) == c, what);
}

// The gradient of an output: dy and, for an output that also is the last channels of a wide tensor, that tensor's
// gradient; for an output that is the first channels of a wide tensor (join), that tensor's gradient alone.
struct OutputGrad {
    const void *a, *b = nullptr;
    int pitch = 0, pitch2 = 0;
};
OutputGrad output_grad(const at::Tensor& dy, const at::Tensor* dskip, bool join, const at::Tensor& x) {
    const int64_t c = x.size(-1);
    require_half_rows(dy, x, join ? 2 * c : c, "dy does not have the output's shape");
    OutputGrad g{ptr(dy)};
    if (join) g.pitch = static_cast<int>(2 * c);
    if (dskip) {
        require_half_rows(*dskip, x, 2 * c, "the wide gradient has twice the channels");
        g.b = channels_from(*dskip, c);
        g.pitch2 = static_cast<int>(2 * c);
    }
    return g;
}

// bn_forward(x, residual, gamma, beta, act, slope, eps, join, skip, workspace) -> (y, wide, mean, rstd, mask): y is join's
// storage where one is given; the mask of y > 0 where the backward cannot tell it from x, else None
PyObject* py_bn_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 10)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &x = tensor(a[0], "x"), &gamma = tensor(a[2], "gamma"), &beta = tensor(a[3], "beta");
        const at::Tensor *res = tensor_or_none(a[1], "residual"), *join = tensor_or_none(a[7], "join");
        const int64_t c = x.size(-1), rows = x.numel() / c;
        const int act = static_cast<int>(as_int(a[4]));
        if (join) require_half_rows(*join, x, 2 * c, "join has twice the channels of x");
        const at::Tensor y = join ? join->variable_data() : at::empty(x.sizes(), x.options());
        const auto fopt = at::TensorOptions().dtype(at::kFloat).device(x.device());
        const at::Tensor mean = at::empty({c}, fopt), rstd = at::empty({c}, fopt);
        at::Tensor mask, wide;
        if (res != nullptr && act != 0) mask = at::empty({x.numel() / 8}, fopt.dtype(at::kByte));
        if (as_int(a[8]) != 0) wide = wide_like(x);
        const int pitch = static_cast<int>(2 * c);
        size_t need = 0;
        check(nml_bn_workspace_size(rows, static_cast<int>(c), &need));
        const Scratch ws = scratch(a[9], need, x);
        check(nml_bn_forward_masked(ptr(x), rows, static_cast<int>(c), static_cast<const float*>(ptr(gamma)),
                                    static_cast<const float*>(ptr(beta)), ptr_or_null(res), act, static_cast<float>(as_double(a[5])),
                                    static_cast<float>(as_double(a[6])), ptr(y), join ? pitch : 0,
                                    wide.defined() ? channels_from(wide, c) : nullptr, pitch, mask.defined() ? ptr(mask) : nullptr,
                                    static_cast<float*>(ptr(mean)), static_cast<float*>(ptr(rstd)), ws.p, ws.bytes, stream()));
        return tuple_of(y, wide, mean, rstd, mask);
    });
}

// bn_backward(dy, dwide, join, mask, x, gamma, beta, mean, rstd, act, slope, want_residual_grad, dgamma, dbeta, workspace)
// -> (dx, dres)
PyObject* py_bn_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 15)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &dy = tensor(a[0], "dy"), &x = tensor(a[4], "x"), &gamma = tensor(a[5], "gamma"), &beta = tensor(a[6], "beta"),
                         &mean = tensor(a[7], "mean"), &rstd = tensor(a[8], "rstd"), &dgamma = tensor(a[12], "dgamma"), &dbeta = tensor(a[13], "dbeta");
        const at::Tensor* mask = tensor_or_none(a[3], "mask");
        const int64_t c = x.size(-1), rows = x.numel() / c;
        const OutputGrad g = output_grad(dy, tensor_or_none(a[1], "dwide"), as_int(a[2]) != 0, x);
        const at::Tensor dx = at::empty(x.sizes(), x.options());
        at::Tensor dres;
        if (as_int(a[11]) != 0) dres = at::empty(x.sizes(), x.options());
        size_t need = 0;
        check(nml_bn_workspace_size(rows, static_cast<int>(c), &need));
        const Scratch ws = scratch(a[14], need, x);
        check(nml_bn_backward_masked(g.a, g.pitch, g.b, g.pitch2, ptr_or_null(mask), ptr(x), rows, static_cast<int>(c),
                                     static_cast<const float*>(ptr(gamma)), static_cast<const float*>(ptr(beta)),
                                     static_cast<const float*>(ptr(mean)), static_cast<const float*>(ptr(rstd)),
                                     static_cast<int>(as_int(a[9])), static_cast<float>(as_double(a[10])), ptr(dx),
                                     dres.defined() ? ptr(dres) : nullptr, static_cast<float*>(ptr(dgamma)),
                                     static_cast<float*>(ptr(dbeta)), ws.p, ws.bytes, stream()));
        return tuple_of(dx, dres);
    });
}

// act_forward(x, act, slope, skip) -> (y, wide)
PyObject* py_act_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 4)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor& x = tensor(a[0], "x");
        const int64_t c = x.size(-1);
        require_half_rows(x, x, c, "x is float16");
        const at::Tensor y = at::empty(x.sizes(), x.options());
        at::Tensor wide;
        if (as_int(a[3]) != 0) wide = wide_like(x);
        check(nml_act_forward(ptr(x), x.numel() / c, static_cast<int>(c), static_cast<int>(as_int(a[1])), static_cast<float>(as_double(a[2])),
                              ptr(y), wide.defined() ? channels_from(wide, c) : nullptr, static_cast<int>(2 * c), stream()));
        return tuple_of(y, wide);
    });
}

// act_backward(dy, dwide, x, act, slope) -> dx
PyObject* py_act_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 5)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &dy = tensor(a[0], "dy"), &x = tensor(a[2], "x");
        const int64_t c = x.size(-1);
        const OutputGrad g = output_grad(dy, tensor_or_none(a[1], "dwide"), false, x);
        const at::Tensor dx = at::empty(x.sizes(), x.options());
        check(nml_act_backward(g.a, g.pitch, g.b, g.pitch2, ptr(x), x.numel() / c, static_cast<int>(c), static_cast<int>(as_int(a[3])),
                               static_cast<float>(as_double(a[4])), ptr(dx), stream()));
        return THPVariable_Wrap(dx);
    });
}

// ------------------------------------------------------------------ loss --
// l1_forward(a, b, denom, workspace) -> loss
PyObject* py_l1_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (!arity(n, 4)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &a = tensor(args[0], "a"), &b = tensor(args[1], "b");
        require(a.scalar_type() == at::kHalf && b.scalar_type() == at::kHalf && a.numel() == b.numel(), "two float16 tensors of one size");
        const at::Tensor loss = at::empty({}, a.options().dtype(at::kFloat));
        size_t need = 0;
        check(nml_l1_workspace_size(&need));
        const Scratch ws = scratch(args[3], need, a);
        check(nml_l1_forward(ptr(a), ptr(b), a.numel(), static_cast<float>(as_double(args[2])), static_cast<float*>(ptr(loss)), ws.p, ws.bytes,
                             stream()));
        return THPVariable_Wrap(loss);
    });
}

// l1_backward(a, b, dloss, denom) -> da
PyObject* py_l1_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (!arity(n, 4)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &a = tensor(args[0], "a"), &b = tensor(args[1], "b"), &dloss = tensor(args[2], "dloss");
        require(dloss.scalar_type() == at::kFloat && dloss.numel() == 1, "the gradient of the loss is one float32");
        const at::Tensor da = at::empty(a.sizes(), a.options());
        check(nml_l1_backward(ptr(a), ptr(b), a.numel(), static_cast<const float*>(ptr(dloss)), static_cast<float>(as_double(args[3])), ptr(da),
                              stream()));
        return THPVariable_Wrap(da);
    });
}

#define NML_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {NML_FAST(geometry), NML_FAST(conv_forward), NML_FAST(conv_backward_data), NML_FAST(conv_backward_weight),
                          NML_FAST(linear_forward), NML_FAST(linear_backward_data), NML_FAST(linear_backward_weight),
                          NML_FAST(bn_forward), NML_FAST(bn_backward), NML_FAST(act_forward), NML_FAST(act_backward),
                          NML_FAST(l1_forward), NML_FAST(l1_backward), {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    PyObject* lib = PyImport_ImportModule("nectarml_b200._lib");
    if (!lib) return nullptr;
    g_error = PyObject_GetAttrString(lib, "NectarB200Error");
    Py_DECREF(lib);
    if (!g_error) return nullptr;
    return PyModule_Create(&kModule);
}
