// Tensor-level host path in native code: unpacks torch tensors, checks them, allocates the result and calls
// the C ABI of include/nectarml_b200.h.  Built into nectarml_b200/_native.so; nectarml_b200/ops.py and
// train.py are the only callers.
//
// Why it exists: a layer call from Python spent 12 us around a C-ABI call of 4 us (ctypes conversions, stream
// lookup through torch.cuda, descriptor fields set one by one, shape tuples), more than most small layers run
// on the GPU.  Here the same work is about 2 us: linear 32 x 512 -> 2048 forward 16.2 -> 7 us per call.
//
// Nothing is kept between calls except the parsed geometry of a layer (a capsule owned by the Python
// ConvGeometry object).  The GIL is released while memory is allocated and while kernels are launched: an allocation may
// synchronise the device, and a launch waits where the stream's queue is full, for as long as the GPU is behind.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/engine.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <cstring>
#include <initializer_list>
#include <memory>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

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
// (Callers take every pointer before they ask for the stream: a tensor in the wrong place is reported as such even where there
// is no GPU to have a stream on.)
void* ptr(const at::Tensor& t) {
    if (!t.is_cuda()) fail("tensors must live on a CUDA device (there is no CPU path)");
    if (!t.is_contiguous()) fail("tensors must be contiguous");
    return t.data_ptr();
}
inline float* floats(const at::Tensor& t) { return static_cast<float*>(ptr(t)); }
inline void* ptr_or_null(const at::Tensor* t) { return t ? ptr(*t) : nullptr; }

struct NoGil {
    PyThreadState* const state = PyEval_SaveThread();
    NoGil() = default;
    NoGil(const NoGil&) = delete;
    ~NoGil() { PyEval_RestoreThread(state); }
};
template <class F>
auto without_gil(F&& f) {
    NoGil off;
    return f();
}
at::Tensor new_empty(at::IntArrayRef shape, const at::TensorOptions& options) {
    return without_gil([&] { return at::empty(shape, options); });
}

// Launches a pass, f(stream) -> status, on the current stream.  A pass is several kernels that share the workspace, so the
// passes that threads issue on one stream follow one another whole: a lock per stream (streams that share one by their hash only
// take turns), taken without the GIL and given back before it.
template <class F>
void issue(F&& f) {
    static std::mutex order[64];
    const auto s = c10::cuda::getCurrentCUDAStream();
    const int status = without_gil([&] {
        const size_t key = reinterpret_cast<size_t>(s.stream()) / 64 + 7u * static_cast<size_t>(s.device_index());
        std::lock_guard<std::mutex> turn(order[(key ^ key >> 6 ^ key >> 12) % 64]);
        return f(static_cast<void*>(s.stream()));
    });
    check(status);
}

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
    return new_empty(shape, at::TensorOptions().dtype(st).device(like.device()));
}

// Scratch from the caller's Workspace object (a grow-only buffer, see ops.Workspace): its tensor as it is while it is
// large enough and on the right device, else through its own get().
struct Scratch {
    void* p = nullptr;
    size_t bytes = 0;
    at::Tensor hold;  // until the pass is launched: another thread may make the workspace grow meanwhile
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
                s.hold = t;
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

// Runs a function body with C++ exceptions turned into the Python ones torch's own functions raise (out of memory and index
// errors have types of their own).
template <class F>
PyObject* guarded(F&& f) {
    HANDLE_TH_ERRORS
    try {
        return f();
    } catch (const Fail&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
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

at::Tensor run_conv_forward(const Geometry& g, const at::Tensor& x, const at::Tensor& w, const at::Tensor* bias, PyObject* given,
                            int layout, int out_layout, int math, long out_dtype, int round_f16, PyObject* workspace) {
    nml_conv_desc d = g.d;
    d.in_layout = layout;
    d.out_layout = out_layout;
    require(is_act(x, g, true, layout), "x does not have the layer's input shape");
    require(is_weight(w, g), "w does not have the layer's weight shape");
    if (bias) require(bias->scalar_type() == w.scalar_type() && bias->numel() == g.d.c_out, "bias: dtype of w, one value per output channel");
    int64_t s[4];
    act_shape(g, false, out_layout, s);
    const at::Tensor out = output(given, s, out_dtype, x);
    d.in_dtype = dtype_of(x);
    d.out_dtype = dtype_of(out);
    d.w_dtype = dtype_of(w);
    d.math = math;
    d.round_out_f16 = round_f16;
    size_t need = 0;
    check(nml_conv_workspace_size(&d, NML_PASS_FORWARD, &need));
    const Scratch ws = scratch(workspace, need, x);
    void *const px = ptr(x), *const pw = ptr(w), *const pb = ptr_or_null(bias), *const po = ptr(out);
    issue([&](void* st) {
        return nml_conv_forward(&d, px, pw, pb, po, ws.p, ws.bytes, st);
    });
    return out;
}

at::Tensor run_conv_backward_data(const Geometry& g, const at::Tensor& dy, const at::Tensor& w, PyObject* given, int layout, int out_layout,
                                  int math, long out_dtype, PyObject* workspace) {
    nml_conv_desc d = g.d;
    d.in_layout = layout;
    d.out_layout = out_layout;
    require(is_act(dy, g, false, layout), "dy does not have the layer's output shape");
    require(is_weight(w, g), "w does not have the layer's weight shape");
    int64_t s[4];
    act_shape(g, true, out_layout, s);
    const at::Tensor out = output(given, s, out_dtype, dy);
    d.in_dtype = dtype_of(dy);
    d.out_dtype = dtype_of(out);
    d.w_dtype = dtype_of(w);
    d.math = math;
    size_t need = 0;
    check(nml_conv_workspace_size(&d, NML_PASS_BACKWARD_DATA, &need));
    const Scratch ws = scratch(workspace, need, dy);
    void *const pd = ptr(dy), *const pw = ptr(w), *const po = ptr(out);
    issue([&](void* st) {
        return nml_conv_backward_data(&d, pd, pw, po, ws.p, ws.bytes, st);
    });
    return out;
}

// The same on fp16 NHWC tensors with another gradient of the layer's input added: `add`, scaled by `below` where `mask` has no bit.
at::Tensor run_conv_backward_data_add(const Geometry& g, const at::Tensor& dy, const at::Tensor& w, const at::Tensor& add, const at::Tensor& mask,
                                      float below, PyObject* workspace) {
    nml_conv_desc d = g.d;
    d.in_layout = d.out_layout = NML_NHWC;
    int64_t s[4];
    act_shape(g, true, NML_NHWC, s);
    const at::Tensor out = new_empty(s, dy.options());
    d.in_dtype = d.out_dtype = d.w_dtype = NML_F16;
    d.math = NML_MATH_F16;
    size_t need = 0;
    check(nml_conv_workspace_size(&d, NML_PASS_BACKWARD_DATA, &need));
    const Scratch ws = scratch(workspace, need, dy);
    void *const pd = ptr(dy), *const pw = ptr(w), *const pa = ptr(add), *const pm = mask.defined() ? ptr(mask) : nullptr, *const po = ptr(out);
    issue([&](void* st) {
        return nml_conv_backward_data_add(&d, pd, pw, pa, pm, below, po, ws.p, ws.bytes, st);
    });
    return out;
}

// dw and, where defined, db are written
void run_conv_backward_weight(const Geometry& g, const at::Tensor& x, const at::Tensor& dy, const at::Tensor& dw, const at::Tensor& db,
                              int layout, int math, PyObject* workspace) {
    nml_conv_desc d = g.d;
    d.in_layout = d.out_layout = layout;
    require(is_act(x, g, true, layout), "x does not have the layer's input shape");
    require(is_act(dy, g, false, layout), "dy does not have the layer's output shape");
    require(x.scalar_type() == dy.scalar_type(), "x and dy have one dtype");
    int64_t s[4];
    weight_shape(g, s);
    require(dw.scalar_type() == at::kFloat && dw.numel() == s[0] * s[1] * s[2] * s[3], "dw is float32 and has the weight's elements");
    d.in_dtype = dtype_of(x);
    d.out_dtype = d.w_dtype = NML_F32;
    d.math = math;
    size_t need = 0;
    check(nml_conv_workspace_size(&d, NML_PASS_BACKWARD_WEIGHT, &need));
    const Scratch ws = scratch(workspace, need, x);
    void *const px = ptr(x), *const pd = ptr(dy);
    float *const pdw = floats(dw), *const pdb = db.defined() ? floats(db) : nullptr;
    issue([&](void* st) {
        return nml_conv_backward_weight(&d, px, pd, pdw, pdb, ws.p, ws.bytes, st);
    });
}

// conv_forward(geometry, x, w, bias, out, layout, out_layout, math, out_dtype, round_f16, workspace)
PyObject* py_conv_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 11)) return nullptr;
    return guarded([&]() -> PyObject* {
        return THPVariable_Wrap(run_conv_forward(geometry(a[0]), tensor(a[1], "x"), tensor(a[2], "w"), tensor_or_none(a[3], "bias"), a[4],
                                                 static_cast<int>(as_int(a[5])), static_cast<int>(as_int(a[6])),
                                                 static_cast<int>(as_int(a[7])), as_int(a[8]), static_cast<int>(as_int(a[9])), a[10]));
    });
}

// conv_backward_data(geometry, dy, w, out, layout, out_layout, math, out_dtype, workspace)
PyObject* py_conv_backward_data(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 9)) return nullptr;
    return guarded([&]() -> PyObject* {
        return THPVariable_Wrap(run_conv_backward_data(geometry(a[0]), tensor(a[1], "dy"), tensor(a[2], "w"), a[3],
                                                       static_cast<int>(as_int(a[4])), static_cast<int>(as_int(a[5])),
                                                       static_cast<int>(as_int(a[6])), as_int(a[7]), a[8]));
    });
}

// conv_backward_weight(geometry, x, dy, dw, db, layout, math, want_bias_grad, workspace) -> (dw, db)
PyObject* py_conv_backward_weight(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 9)) return nullptr;
    return guarded([&]() -> PyObject* {
        const Geometry& g = geometry(a[0]);
        const at::Tensor& x = tensor(a[1], "x");
        int64_t s[4];
        weight_shape(g, s);
        const at::Tensor dw = output(a[3], s, NML_F32, x);
        at::Tensor db;
        const bool has_db = a[4] != Py_None || as_int(a[7]) != 0;
        if (has_db) db = output(a[4], {g.d.c_out}, NML_F32, x);
        run_conv_backward_weight(g, x, tensor(a[2], "dy"), dw, db, static_cast<int>(as_int(a[5])), static_cast<int>(as_int(a[6])), a[8]);
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
        void *const px = ptr(x), *const pw = ptr(w), *const pb = ptr_or_null(bias), *const po = ptr(out);
        issue([&](void* st) {
            return nml_linear_forward(&d, px, pw, pb, po, ws.p, ws.bytes, st);
        });
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
        void *const pd = ptr(dy), *const pw = ptr(w), *const po = ptr(out);
        issue([&](void* st) {
            return nml_linear_backward_data(&d, pd, pw, po, ws.p, ws.bytes, st);
        });
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
        void *const px = ptr(x), *const pd = ptr(dy);
        float *const pdw = floats(dw), *const pdb = has_db ? floats(db) : nullptr;
        issue([&](void* st) {
            return nml_linear_backward_weight(&d, px, pd, pdw, pdb, ws.p, ws.bytes, st);
        });
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
int64_t channels(const at::Tensor& x) {
    const int64_t c = x.size(-1);
    require(c > 0, "a tensor without channels");
    return c;
}
at::Tensor wide_like(const at::Tensor& x) {
    auto shape = x.sizes().vec();
    shape.back() *= 2;
    return new_empty(shape, x.options());
}
void* channels_from(const at::Tensor& wide, int64_t c) { return static_cast<char*>(ptr(wide)) + c * wide.element_size(); }
void require_half_rows(const at::Tensor& t, const at::Tensor& x, int64_t c, const char* what) {
    require(t.scalar_type() == at::kHalf && t.size(-1) == c && t.numel() / c == x.numel() / channels(x), what);
}

// The gradient of an output: dy and, for an output that also is the last channels of a wide tensor, that tensor's
// gradient; for an output that is the first channels of a wide tensor (join), that tensor's gradient alone.
struct OutputGrad {
    const void *a, *b = nullptr;
    int pitch = 0, pitch2 = 0;
};
OutputGrad output_grad(const at::Tensor& dy, const at::Tensor* dskip, bool join, const at::Tensor& x) {
    const int64_t c = channels(x);
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

struct BnSaved {
    at::Tensor y, wide, mean, rstd, mask;
};
BnSaved run_bn_forward(const at::Tensor& x, const at::Tensor* res, const at::Tensor& gamma, const at::Tensor& beta, int act, float slope,
                       float eps, const at::Tensor* join, bool skip, PyObject* workspace) {
    const int64_t c = channels(x), rows = x.numel() / c;
    if (join) require_half_rows(*join, x, 2 * c, "join has twice the channels of x");
    BnSaved r;
    r.y = join ? join->variable_data() : new_empty(x.sizes(), x.options());
    const auto fopt = at::TensorOptions().dtype(at::kFloat).device(x.device());
    r.mean = new_empty({c}, fopt);
    r.rstd = new_empty({c}, fopt);
    if (res != nullptr && act != 0) r.mask = new_empty({x.numel() / 8}, fopt.dtype(at::kByte));
    if (skip) r.wide = wide_like(x);
    const int pitch = static_cast<int>(2 * c);
    size_t need = 0;
    check(nml_bn_workspace_size(rows, static_cast<int>(c), &need));
    const Scratch ws = scratch(workspace, need, x);
    void *const px = ptr(x), *const pres = ptr_or_null(res), *const py = ptr(r.y);
    void *const py2 = skip ? channels_from(r.wide, c) : nullptr, *const pmask = r.mask.defined() ? ptr(r.mask) : nullptr;
    float *const pg = floats(gamma), *const pb = floats(beta), *const pm = floats(r.mean), *const pr = floats(r.rstd);
    issue([&](void* st) {
        return nml_bn_forward_masked(px, rows, static_cast<int>(c), pg, pb, pres, act, slope, eps, py, join ? pitch : 0, py2, pitch, pmask,
                                     pm, pr, ws.p, ws.bytes, st);
    });
    return r;
}

// -> dx, and dz in dres where that is defined
at::Tensor run_bn_backward(const OutputGrad& g, const at::Tensor* mask, const at::Tensor& x, const at::Tensor& gamma, const at::Tensor& beta,
                           const at::Tensor& mean, const at::Tensor& rstd, int act, float slope, const at::Tensor& dres,
                           const at::Tensor& dgamma, const at::Tensor& dbeta, PyObject* workspace) {
    const int64_t c = channels(x), rows = x.numel() / c;
    const at::Tensor dx = new_empty(x.sizes(), x.options());
    size_t need = 0;
    check(nml_bn_workspace_size(rows, static_cast<int>(c), &need));
    const Scratch ws = scratch(workspace, need, x);
    void *const px = ptr(x), *const pmask = ptr_or_null(mask), *const pdx = ptr(dx), *const pdres = dres.defined() ? ptr(dres) : nullptr;
    float *const pg = floats(gamma), *const pb = floats(beta), *const pm = floats(mean), *const pr = floats(rstd);
    float *const pdg = floats(dgamma), *const pdb = floats(dbeta);
    issue([&](void* st) {
        return nml_bn_backward_masked(g.a, g.pitch, g.b, g.pitch2, pmask, px, rows, static_cast<int>(c), pg, pb, pm, pr, act, slope, pdx,
                                      pdres, pdg, pdb, ws.p, ws.bytes, st);
    });
    return dx;
}

// bn_forward(x, residual, gamma, beta, act, slope, eps, join, skip, workspace) -> (y, wide, mean, rstd, mask): y is join's
// storage where one is given; the mask of y > 0 where the backward cannot tell it from x, else None
PyObject* py_bn_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 10)) return nullptr;
    return guarded([&]() -> PyObject* {
        const BnSaved r = run_bn_forward(tensor(a[0], "x"), tensor_or_none(a[1], "residual"), tensor(a[2], "gamma"), tensor(a[3], "beta"),
                                         static_cast<int>(as_int(a[4])), static_cast<float>(as_double(a[5])),
                                         static_cast<float>(as_double(a[6])), tensor_or_none(a[7], "join"), as_int(a[8]) != 0, a[9]);
        return tuple_of(r.y, r.wide, r.mean, r.rstd, r.mask);
    });
}

// bn_backward(dy, dwide, join, mask, x, gamma, beta, mean, rstd, act, slope, want_residual_grad, dgamma, dbeta, workspace)
// -> (dx, dres)
PyObject* py_bn_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 15)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor& x = tensor(a[4], "x");
        const OutputGrad g = output_grad(tensor(a[0], "dy"), tensor_or_none(a[1], "dwide"), as_int(a[2]) != 0, x);
        at::Tensor dres;
        if (as_int(a[11]) != 0) dres = new_empty(x.sizes(), x.options());
        const at::Tensor dx = run_bn_backward(g, tensor_or_none(a[3], "mask"), x, tensor(a[5], "gamma"), tensor(a[6], "beta"),
                                              tensor(a[7], "mean"), tensor(a[8], "rstd"), static_cast<int>(as_int(a[9])),
                                              static_cast<float>(as_double(a[10])), dres, tensor(a[12], "dgamma"), tensor(a[13], "dbeta"),
                                              a[14]);
        return tuple_of(dx, dres);
    });
}

// act_forward(x, act, slope, skip) -> (y, wide)
PyObject* py_act_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 4)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor& x = tensor(a[0], "x");
        const int64_t c = channels(x);
        require_half_rows(x, x, c, "x is float16");
        const at::Tensor y = new_empty(x.sizes(), x.options());
        at::Tensor wide;
        if (as_int(a[3]) != 0) wide = wide_like(x);
        const int act = static_cast<int>(as_int(a[1]));
        const float slope = static_cast<float>(as_double(a[2]));
        void *const px = ptr(x), *const py = ptr(y), *const py2 = wide.defined() ? channels_from(wide, c) : nullptr;
        issue([&](void* st) {
            return nml_act_forward(px, x.numel() / c, static_cast<int>(c), act, slope, py, py2, static_cast<int>(2 * c), st);
        });
        return tuple_of(y, wide);
    });
}

// act_backward(dy, dwide, x, act, slope) -> dx
PyObject* py_act_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 5)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &dy = tensor(a[0], "dy"), &x = tensor(a[2], "x");
        const int64_t c = channels(x);
        const OutputGrad g = output_grad(dy, tensor_or_none(a[1], "dwide"), false, x);
        const at::Tensor dx = new_empty(x.sizes(), x.options());
        const int act = static_cast<int>(as_int(a[3]));
        const float slope = static_cast<float>(as_double(a[4]));
        void *const px = ptr(x), *const pdx = ptr(dx);
        issue([&](void* st) {
            return nml_act_backward(g.a, g.pitch, g.b, g.pitch2, px, x.numel() / c, static_cast<int>(c), act, slope, pdx, st);
        });
        return THPVariable_Wrap(dx);
    });
}

// ------------------------------------------------------------------ autograd nodes of train.py's layers --
// A convolution and a batch norm of a training step as nodes of torch's autograd tape.  As Python autograd functions their
// bookkeeping (contexts, saved tensors, wrappers, a Python frame in each direction) was half of the host time of a step: a
// U-Net step of 29 such layers was issued in 2.2 ms and ran 2.0 ms.
//
// Weight gradients go straight into the flat gradient buffer, before the input gradient (so that the buffer's bucket can
// leave early).  `flags` is the parameter store's bytearray, read when the backward runs: [0] gradients add to the buffer,
// [1] buckets are exchanged, so the layer reports back.
namespace autograd = torch::autograd;

struct Gil {
    PyGILState_STATE state = PyGILState_Ensure();
    ~Gil() { PyGILState_Release(state); }
};

// What a node holds of the Python side; released under the GIL, wherever the tape is dropped.
struct Owner {
    PyObject *layer, *flags, *workspace;
    Owner(PyObject* l, PyObject* f, PyObject* w) : layer(Py_NewRef(l)), flags(Py_NewRef(f)), workspace(Py_NewRef(w)) {}
    Owner(const Owner&) = delete;
    Owner& operator=(const Owner&) = delete;
    ~Owner() {
        if (!Py_IsInitialized()) return;
        Gil gil;
        Py_DECREF(layer);
        Py_DECREF(flags);
        Py_DECREF(workspace);
    }
    bool flag(int i) const { return PyByteArray_AS_STRING(flags)[i] != 0; }

    // run(a, b) writes a layer's gradients: into the buffer, or beside it and then added
    template <class F>
    void weight_gradient(const at::Tensor& a, const at::Tensor& b, F&& run) const {
        if (!flag(0)) {
            run(a, b);
        } else {
            const at::Tensor ta = new_empty(a.sizes(), a.options());
            at::Tensor tb;
            if (b.defined()) tb = new_empty(b.sizes(), b.options());
            run(ta, tb);
            without_gil([&] {
                a.add_(ta);
                if (b.defined()) b.add_(tb);
            });
        }
        if (flag(1)) {
            PyObject* r = PyObject_CallMethod(layer, "gradient_written", nullptr);
            if (!r) throw Fail();
            Py_DECREF(r);
        }
    }
};
void require_flags(PyObject* flags) {
    require(PyByteArray_Check(flags) && PyByteArray_GET_SIZE(flags) >= 2, "flags: a bytearray of two");
}

struct LayerNode : autograd::Node {
    std::unique_ptr<Owner> owner;
    autograd::SavedVariable x;
    at::Tensor grad_a, grad_b;  // the layer's parts of the flat gradient buffer

    void release_variables() override { x.reset_data(); }

    // A backward body: under the GIL (the workspaces are Python objects), Python errors handed on as they are.
    template <class F>
    autograd::variable_list guarded_backward(F&& f) {
        Gil gil;
        try {
            return f();
        } catch (const Fail&) {
            python_error e;
            e.persist();
            throw e;
        }
    }
};
template <class N>
std::shared_ptr<N> make_node(PyObject* layer, PyObject* flags, PyObject* workspace) {
    std::shared_ptr<N> node(new N(), autograd::deleteNode);
    node->owner = std::make_unique<Owner>(layer, flags, workspace);
    return node;
}
autograd::Edge edge_of(const at::Tensor* t) {
    return t && t->defined() && t->requires_grad() ? autograd::impl::gradient_edge(*t) : autograd::Edge();
}
// The layers have no forward-mode derivative: a tangent would be dropped in silence.
void require_no_tangent(std::initializer_list<const at::Tensor*> inputs) {
    for (const at::Tensor* t : inputs)
        if (t && t->defined() && t->_fw_grad(0).defined()) {
            PyErr_SetString(PyExc_NotImplementedError, "this layer has no forward-mode derivative");
            throw Fail();
        }
}
// An output nobody differentiated through has no gradient: zeros.
at::Tensor grad_or_zeros(const at::Tensor& g, at::IntArrayRef shape, const at::Tensor& like) {
    return without_gil([&] { return g.defined() ? g.contiguous() : at::zeros(shape, like.options()); });
}

// A residual block's input has two gradients: its first convolution's input gradient, and the gradient of the normalisation that
// the input is added to at the block's end.  Made by two nodes and added by the engine, the second one is stored, and
// three tensors are read and written for the sum (1.2 of the 10.8 GB a 256-channel 56 x 56 block at batch 256 moves).  Instead the
// normalisation's node leaves a description of it (its output's gradient and the mask of the activation) with the
// convolution's node and returns no gradient for its residual, and the convolution adds it as it stores its result.
//
// That is sound where both nodes are run whenever one is, the normalisation first: the convolution's input and the residual
// are one output of the graph (equal edges, so the engine needs both gradients or neither), and the way from the
// normalisation back to the convolution leads through input edges of nodes of this file alone (ancestors, so run later).
// All of this is read off the graph when it is built; that no hook waits for either node's own gradients, when the
// normalisation runs.  What is left is kept per backward pass (its task's id), so passes over one graph, one after another or in
// several threads, do not meet.  (A pass that raises between the two leaves its part until the graph goes or runs to its end.)
struct Handoff {
    struct Part {
        int task;
        at::Tensor dy, mask;  // no mask: no activation
        float below;
    };
    std::weak_ptr<autograd::Node> taker;  // the convolution's node
    // (its hooks are given the input gradient it returns, which has to be its own)
    bool wanted() const {
        const auto node = taker.lock();
        return node && node->post_hooks().empty();
    }
    std::mutex lock;
    std::vector<Part> parts;
    void leave(Part p) {
        std::lock_guard<std::mutex> l(lock);
        parts.push_back(std::move(p));
    }
    bool take(int task, Part& p) {
        std::lock_guard<std::mutex> l(lock);
        for (size_t i = 0; i < parts.size(); ++i)
            if (parts[i].task == task) {
                p = std::move(parts[i]);
                parts.erase(parts.begin() + i);
                return true;
            }
        return false;
    }
    void clear() {
        std::lock_guard<std::mutex> l(lock);
        parts.clear();
    }
};

struct ConvNode : LayerNode {
    Geometry g;
    at::Tensor w;
    bool needs_dx = true;
    std::shared_ptr<Handoff> incoming;  // set by the normalisation at the end of the block
    c10::cuda::CUDAStream made_on = c10::cuda::getCurrentCUDAStream();

    void release_variables() override {
        LayerNode::release_variables();
        if (incoming) incoming->clear();
    }
    std::string name() const override { return "ConvBackward"; }
    autograd::variable_list apply(autograd::variable_list&& grads) override {
        return guarded_backward([&]() -> autograd::variable_list {
            const at::Tensor in = x.unpack();
            int64_t s[4];
            act_shape(g, false, NML_NHWC, s);
            const at::Tensor dy = grad_or_zeros(grads[0], s, in);
            owner->weight_gradient(grad_a, grad_b, [&](const at::Tensor& dw, const at::Tensor& db) {
                run_conv_backward_weight(g, in, dy, dw, db, NML_NHWC, NML_MATH_F16, owner->workspace);
            });
            autograd::variable_list out(2);
            Handoff::Part other;
            const bool sum = incoming && incoming->take(autograd::get_current_graph_task_id(), other);
            if (needs_dx && task_should_compute_output(0) && sum)
                out[0] = run_conv_backward_data_add(g, dy, w, other.dy, other.mask, other.below, owner->workspace);
            else if (needs_dx && task_should_compute_output(0))
                out[0] = run_conv_backward_data(g, dy, w, Py_None, NML_NHWC, NML_NHWC, NML_MATH_F16, -1, owner->workspace);
            return out;
        });
    }
};

// conv_layer(geometry, x, token, w, bias, dw, db, needs_dx, layer, flags, workspace) -> y
PyObject* py_conv_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 11)) return nullptr;
    return guarded([&]() -> PyObject* {
        const Geometry& g = geometry(a[0]);
        const at::Tensor &x = tensor(a[1], "x"), &token = tensor(a[2], "token"), &w = tensor(a[3], "w"), &dw = tensor(a[5], "dw");
        const at::Tensor* db = tensor_or_none(a[6], "db");
        const bool needs_dx = as_int(a[7]) != 0;
        require_flags(a[9]);
        require_no_tangent({&x, &token});
        at::Tensor y = run_conv_forward(g, x, w, tensor_or_none(a[4], "bias"), Py_None, NML_NHWC, NML_NHWC, NML_MATH_F16, -1, 0, a[10]);
        if (at::GradMode::is_enabled() && (x.requires_grad() || token.requires_grad())) {
            auto node = make_node<ConvNode>(a[8], a[9], a[10]);
            node->g = g;
            node->w = w;
            node->needs_dx = needs_dx;
            node->grad_a = dw;
            if (db) node->grad_b = *db;
            node->x = autograd::SavedVariable(x, false);
            node->set_next_edges({edge_of(&x), edge_of(&token)});
            autograd::create_gradient_edge(y, node);
        }
        return THPVariable_Wrap(y);
    });
}

struct BnNode : LayerNode {
    at::Tensor gamma, beta;
    autograd::SavedVariable mean, rstd, mask;  // (saved like x, so that hooks on saved tensors see all a layer keeps)
    bool masked = false;
    int act = 0;
    float slope = 0.f;
    bool residual = false, join = false;
    std::shared_ptr<Handoff> outgoing;  // where the residual's gradient may be left

    // The first convolution of the block that this normalisation ends, if it can take the residual's gradient over.
    void find_block(const autograd::Edge& x_edge, const autograd::Edge& res_edge, const at::Tensor& x) {
        const auto here = c10::cuda::getCurrentCUDAStream();
        if (!res_edge.is_valid() || x.scalar_type() != at::kHalf) return;
        autograd::Node* n = x_edge.function.get();
        for (int depth = 0; n && depth < 16; ++depth) {
            if (auto* c = dynamic_cast<ConvNode*>(n)) {
                const auto& e = c->next_edge(0);
                if (e.function == res_edge.function && e.input_nr == res_edge.input_nr) {
                    const auto& d = c->g.d;
                    if (!c->incoming && c->needs_dx && c->made_on == here && d.c_in % 8 == 0 && d.stride_h * d.stride_w * d.c_in > 16) {
                        outgoing = c->incoming = std::make_shared<Handoff>();
                        outgoing->taker = c->getptr();
                    }
                    return;
                }
                n = e.function.get();
            } else if (auto* b = dynamic_cast<BnNode*>(n)) {
                n = b->next_edge(0).function.get();
            } else {
                return;
            }
        }
    }

    void release_variables() override {
        LayerNode::release_variables();
        mean.reset_data();
        rstd.reset_data();
        mask.reset_data();
    }
    std::string name() const override { return "BatchNormBackward"; }
    autograd::variable_list apply(autograd::variable_list&& grads) override {
        return guarded_backward([&]() -> autograd::variable_list {
            const at::Tensor in = x.unpack(), mu = mean.unpack(), rs = rstd.unpack();
            at::Tensor positive;
            if (masked) positive = mask.unpack();
            auto shape = in.sizes().vec();
            if (join) shape.back() *= 2;
            const at::Tensor dy = grad_or_zeros(grads[0], shape, in);
            at::Tensor dwide;
            if (grads.size() > 1 && grads[1].defined()) dwide = without_gil([&] { return grads[1].contiguous(); });
            const OutputGrad g = output_grad(dy, dwide.defined() ? &dwide : nullptr, join, in);
            autograd::variable_list out(4);
            // (a hook on this node would miss the gradient it returns)
            const bool leave = outgoing && !join && !dwide.defined() && task_should_compute_output(1) && post_hooks().empty() && outgoing->wanted() &&
                               (reinterpret_cast<uintptr_t>(dy.data_ptr()) & 15) == 0;
            if (residual && !leave) out[1] = new_empty(in.sizes(), in.options());
            owner->weight_gradient(grad_a, grad_b, [&](const at::Tensor& dgamma, const at::Tensor& dbeta) {
                out[0] = run_bn_backward(g, masked ? &positive : nullptr, in, gamma, beta, mu, rs, act, slope, out[1], dgamma, dbeta,
                                         owner->workspace);
            });
            if (join) out[3] = dy;
            if (leave) outgoing->leave({autograd::get_current_graph_task_id(), dy, positive, act == 1 ? 0.f : slope});
            return out;
        });
    }
};

// bn_layer(x, residual, token, join, gamma, beta, dgamma, dbeta, act, slope, eps, skip, layer, flags, workspace)
// -> y, or (y, wide) with skip
PyObject* py_bn_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arity(n, 15)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &x = tensor(a[0], "x"), &token = tensor(a[2], "token"), &gamma = tensor(a[4], "gamma"), &beta = tensor(a[5], "beta");
        const at::Tensor *res = tensor_or_none(a[1], "residual"), *join = tensor_or_none(a[3], "join");
        const int act = static_cast<int>(as_int(a[8]));
        const float slope = static_cast<float>(as_double(a[9]));
        const bool skip = as_int(a[11]) != 0;
        require_flags(a[13]);
        require_no_tangent({&x, res, &token, join});
        BnSaved r = run_bn_forward(x, res, gamma, beta, act, slope, static_cast<float>(as_double(a[10])), join, skip, a[14]);
        const bool differentiable = x.requires_grad() || token.requires_grad() || (res && res->requires_grad()) || (join && join->requires_grad());
        if (at::GradMode::is_enabled() && differentiable) {
            auto node = make_node<BnNode>(a[12], a[13], a[14]);
            node->gamma = gamma;
            node->beta = beta;
            node->mean = autograd::SavedVariable(r.mean, false);
            node->rstd = autograd::SavedVariable(r.rstd, false);
            node->masked = r.mask.defined();
            if (node->masked) node->mask = autograd::SavedVariable(r.mask, false);
            node->act = act;
            node->slope = slope;
            node->residual = res != nullptr;
            node->join = join != nullptr;
            node->grad_a = tensor(a[6], "dgamma");
            node->grad_b = tensor(a[7], "dbeta");
            node->x = autograd::SavedVariable(x, false);
            node->set_next_edges({edge_of(&x), edge_of(res), edge_of(&token), edge_of(join)});
            if (res && !join && !skip && res->is_cuda()) node->find_block(node->next_edge(0), node->next_edge(1), x);
            autograd::create_gradient_edge(r.y, node);
            if (skip) autograd::create_gradient_edge(r.wide, node);
        }
        return skip ? tuple_of(r.y, r.wide) : THPVariable_Wrap(r.y);
    });
}

// ------------------------------------------------------------------ loss --
// l1_forward(a, b, denom, workspace) -> loss
PyObject* py_l1_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (!arity(n, 4)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &a = tensor(args[0], "a"), &b = tensor(args[1], "b");
        require(a.scalar_type() == at::kHalf && b.scalar_type() == at::kHalf && a.numel() == b.numel(), "two float16 tensors of one size");
        const at::Tensor loss = new_empty({}, a.options().dtype(at::kFloat));
        size_t need = 0;
        check(nml_l1_workspace_size(&need));
        const Scratch ws = scratch(args[3], need, a);
        const float denom = static_cast<float>(as_double(args[2]));
        void *const pa = ptr(a), *const pb = ptr(b);
        float* const pl = floats(loss);
        issue([&](void* st) {
            return nml_l1_forward(pa, pb, a.numel(), denom, pl, ws.p, ws.bytes, st);
        });
        return THPVariable_Wrap(loss);
    });
}

// l1_backward(a, b, dloss, denom) -> da
PyObject* py_l1_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (!arity(n, 4)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &a = tensor(args[0], "a"), &b = tensor(args[1], "b"), &dloss = tensor(args[2], "dloss");
        require(dloss.scalar_type() == at::kFloat && dloss.numel() == 1, "the gradient of the loss is one float32");
        const at::Tensor da = new_empty(a.sizes(), a.options());
        const float denom = static_cast<float>(as_double(args[3]));
        void *const pa = ptr(a), *const pb = ptr(b), *const pda = ptr(da);
        float* const pl = floats(dloss);
        issue([&](void* st) {
            return nml_l1_backward(pa, pb, a.numel(), pl, denom, pda, st);
        });
        return THPVariable_Wrap(da);
    });
}

#define NML_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {NML_FAST(geometry), NML_FAST(conv_forward), NML_FAST(conv_backward_data), NML_FAST(conv_backward_weight),
                          NML_FAST(linear_forward), NML_FAST(linear_backward_data), NML_FAST(linear_backward_weight),
                          NML_FAST(bn_forward), NML_FAST(bn_backward), NML_FAST(act_forward), NML_FAST(act_backward),
                          NML_FAST(l1_forward), NML_FAST(l1_backward), NML_FAST(conv_layer), NML_FAST(bn_layer), {nullptr, nullptr, 0, nullptr}};
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
