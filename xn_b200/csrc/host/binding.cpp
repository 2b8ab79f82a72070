// Native host path of the Python operators (xn_b200/ops.py, decoder.py, prefill.py): argument checks, output
// allocation and the call into libxn_mm.so, as CPython functions over torch tensors.
//
// Why native: a decode-sized call runs 5-15 us on the GPU, and the same checks in Python (tensor attributes, ctypes
// argument conversion, torch.empty through the dispatcher, the stream lookup) took 12-35 us on the host, so the
// host, not the kernel, set the rate of a loop of such calls.  Here a call costs what its launches cost.
//
// All arithmetic stays in libxn_mm.so; this file launches nothing itself.  Errors are raised as xn_b200.XnError with
// the code and the text the Python checks used.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>

#include "../../../include/xn_mm.h"

namespace {

PyObject *g_error_class = nullptr;  // xn_b200._lib.XnError

struct Raised {};  // a Python exception is set

[[noreturn]] void raise_xn(int code, const char *fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    PyObject *e = PyObject_CallFunction(g_error_class ? g_error_class : PyExc_RuntimeError, "is", code, buf);
    if (e) {
        PyErr_SetObject((PyObject *)Py_TYPE(e), e);
        Py_DECREF(e);
    }
    throw Raised();
}

void check(int rc) {
    if (rc) raise_xn(rc, "%s", xn_mm_last_error());
}

// The library call runs without the interpreter lock, as it does through ctypes.
#define XN_CALL(expr)                                                                         \
    do {                                                                                      \
        int _rc;                                                                              \
        Py_BEGIN_ALLOW_THREADS _rc = (expr);                                                  \
        Py_END_ALLOW_THREADS check(_rc);                                                      \
    } while (0)

const at::Tensor &tensor(PyObject *o) {
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "expected a torch.Tensor, got %s", Py_TYPE(o)->tp_name);
        throw Raised();
    }
    return THPVariable_Unpack(o);
}

const at::Tensor *maybe_tensor(PyObject *o) { return o == Py_None ? nullptr : &tensor(o); }

size_t size_arg(PyObject *o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw Raised();
    if (v < 0) raise_xn(XN_ERR_INVALID, "negative size %lld", v);
    return (size_t)v;
}

double float_arg(PyObject *o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Raised();
    return v;
}

void require_cuda(const at::Tensor &t) {
    if (!t.is_cuda()) raise_xn(XN_ERR_INVALID, "xn_b200 runs on CUDA tensors only; there is no CPU path");
}

// as torch prints them
const char *dtype_name(at::ScalarType s) {
    switch (s) {
        case at::kFloat: return "torch.float32";
        case at::kHalf: return "torch.float16";
        case at::kBFloat16: return "torch.bfloat16";
        case at::kDouble: return "torch.float64";
        case at::kLong: return "torch.int64";
        case at::kInt: return "torch.int32";
        case at::kShort: return "torch.int16";
        case at::kChar: return "torch.int8";
        case at::kByte: return "torch.uint8";
        case at::kBool: return "torch.bool";
        default: return c10::toString(s);
    }
}

xn_dtype dtype_code(at::ScalarType s) {
    if (s == at::kFloat) return XN_F32;
    if (s == at::kHalf) return XN_F16;
    if (s == at::kBFloat16) return XN_BF16;
    // the reference refuses other element types at the same point (xn-core/src/cuda_backend.rs:862)
    raise_xn(XN_ERR_UNSUPPORTED, "GEMM not supported for dtype %s", dtype_name(s));
}

void *stream() { return (void *)c10::cuda::getCurrentCUDAStream().stream(); }

at::Tensor empty(at::IntArrayRef shape, at::ScalarType dt, const at::Device &dev) {
    return at::Tensor(at::detail::empty_cuda(shape, dt, dev, std::nullopt));
}

PyObject *wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

std::string shape_text(const at::Tensor &t) {
    std::string s = "[";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + "]";
}

struct Shape {  // an output shape: leading dimensions of another tensor, then given ones
    c10::SmallVector<int64_t, 8> d;
    void lead(const at::Tensor &t, int64_t upto) {
        for (int64_t i = 0; i < upto; ++i) d.push_back(t.size(i));
    }
};

// 0-based argument access with a count check
void want_args(Py_ssize_t n, Py_ssize_t want, const char *name) {
    if (n != want) {
        PyErr_Format(PyExc_TypeError, "%s takes %zd arguments (%zd given)", name, want, n);
        throw Raised();
    }
}

// Runs a binding's body; C++ exceptions (torch's among them) become Python exceptions.
template <typename F> PyObject *guarded(F &&body) {
    try {
        return body();
    } catch (const Raised &) {
        return nullptr;
    } catch (const c10::Error &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
        return nullptr;
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

#define XN_BINDING(name, nargs)                                                                                  \
    PyObject *name##_body(PyObject *const *a);                                                                   \
    PyObject *py_##name(PyObject *, PyObject *const *a, Py_ssize_t n) {                                          \
        return guarded([&]() -> PyObject * {                                                                     \
            want_args(n, nargs, #name);                                                                          \
            return name##_body(a);                                                                               \
        });                                                                                                      \
    }                                                                                                            \
    PyObject *name##_body(PyObject *const *a)

// ---------------------------------------------------------------------------------------------
// matmul / Linear (xn-core/src/ops.rs:631-714, inplace_ops.rs:318-436, nn/linear.rs:4-71)
// ---------------------------------------------------------------------------------------------
// Where a view begins in its storage, also when it has no elements (data_ptr() is null then): a product over no elements
// is zeros, and a live tensor's empty slice is a valid operand of it.
const void *view_ptr(const at::Tensor &t) {
    const char *base = static_cast<const char *>(t.storage().data());
    return base ? base + (size_t)t.storage_offset() * t.itemsize() : nullptr;
}

void matmul_into(const at::Tensor &dst, const at::Tensor &lhs, const at::Tensor &rhs, bool rhs_t) {
    require_cuda(dst);
    require_cuda(lhs);
    require_cuda(rhs);
    if (dst.scalar_type() != lhs.scalar_type() || lhs.scalar_type() != rhs.scalar_type())
        raise_xn(XN_ERR_INVALID, "matmul dtype mismatch: %s, %s, %s", dtype_name(dst.scalar_type()), dtype_name(lhs.scalar_type()),
                 dtype_name(rhs.scalar_type()));
    const xn_dtype dt = dtype_code(dst.scalar_type());
    static_assert(sizeof(size_t) == sizeof(int64_t), "sizes are passed as they are");
    const size_t *ls = (const size_t *)lhs.sizes().data(), *lt = (const size_t *)lhs.strides().data();
    const size_t *rs = (const size_t *)rhs.sizes().data(), *rt = (const size_t *)rhs.strides().data();
    size_t p[12];
    check(xn_mm_matmul_plan((size_t)lhs.dim(), ls, lt, (size_t)rhs.dim(), rs, rt, rhs_t ? 1 : 0, (size_t)dst.numel(), p));
    void *d = dst.data_ptr();
    const void *l = view_ptr(lhs), *r = view_ptr(rhs);
    void *st = stream();
    XN_CALL(xn_mm_gemm(dt, d, l, 0, r, 0, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], p[8], p[9], p[10], p[11], st));
}

XN_BINDING(matmul_, 4) {
    matmul_into(tensor(a[0]), tensor(a[1]), tensor(a[2]), PyObject_IsTrue(a[3]) != 0);
    Py_RETURN_NONE;
}

XN_BINDING(matmul_with_t, 3) {
    const at::Tensor &lhs = tensor(a[0]), &rhs = tensor(a[1]);
    const bool rhs_t = PyObject_IsTrue(a[2]) != 0;
    if (lhs.dim() < 2 || rhs.dim() < 2) raise_xn(XN_ERR_INVALID, "matmul requires at least 2D tensors");
    require_cuda(lhs);
    require_cuda(rhs);
    Shape s;
    s.lead(lhs, lhs.dim() - 1);
    s.d.push_back(rhs.size(rhs_t ? -2 : -1));
    at::Tensor out = empty(s.d, lhs.scalar_type(), lhs.device());
    matmul_into(out, lhs, rhs, rhs_t);
    return wrap(std::move(out));
}

// Contiguous-row activations and weight (what every model layer passes): the Linear entry point, which may prefetch
// the weight -- a parameter, never the previous kernel's output -- ahead of the stream order.  None where the views
// need the general route.
XN_BINDING(linear, 3) {
    const at::Tensor &x = tensor(a[0]), &w = tensor(a[1]);
    const at::Tensor *b = maybe_tensor(a[2]);
    if (b) {
        require_cuda(*b);
        if (b->scalar_type() != x.scalar_type() || b->dim() != 1 || b->size(0) != w.size(0))
            raise_xn(XN_ERR_INVALID, "bias shape mismatch: expected [%lld] of %s, got %s of %s", (long long)w.size(0),
                     dtype_name(x.scalar_type()), shape_text(*b).c_str(), dtype_name(b->scalar_type()));
    }
    if (!(x.is_cuda() && w.is_cuda() && x.scalar_type() == w.scalar_type() && x.dim() >= 2 && w.dim() == 2 &&
          x.size(-1) == w.size(1) && w.size(1) != 0 && w.stride(1) == 1 && x.is_contiguous()))
        Py_RETURN_NONE;
    const xn_dtype dt = dtype_code(x.scalar_type());
    const size_t n = (size_t)w.size(0), k = (size_t)w.size(1), m = (size_t)x.numel() / k, ldw = (size_t)w.stride(0);
    Shape s;
    s.lead(x, x.dim() - 1);
    s.d.push_back((int64_t)n);
    at::Tensor y = empty(s.d, x.scalar_type(), x.device());
    at::Tensor bc;
    if (b) bc = b->contiguous();
    void *yp = y.data_ptr(), *st = stream();
    const void *xp = x.data_ptr(), *wp = w.data_ptr(), *bp = b ? bc.data_ptr() : nullptr;
    XN_CALL(xn_mm_linear(dt, yp, xp, wp, bp, m, n, k, k, ldw, n, st));
    return wrap(std::move(y));
}

// ---------------------------------------------------------------------------------------------
// Quantized linears
// ---------------------------------------------------------------------------------------------
// The rows of x [..., k], counted over its leading dimensions, which are also the output's: a last dimension that is not the
// layer's k is refused here, before anything is allocated or launched (as many rows of k elements as x holds would not be as
// many as the output has).
size_t rows_in(const char *name, const at::Tensor &x, int64_t k) {
    size_t m = 1;
    for (int64_t i = 0; i + 1 < x.dim(); ++i) m *= (size_t)x.size(i);
    if (x.dim() < 1 || (m != 0 && x.size(-1) != k))
        raise_xn(XN_ERR_INVALID, "%s expects rows of %lld elements, got %s", name, (long long)k, shape_text(x).c_str());
    return m;
}

XN_BINDING(quantize_rows_i8, 3) {  // x [m, k], xq or None, x_scale or None
    const at::Tensor &x = tensor(a[0]);
    require_cuda(x);
    if (x.dim() != 2) raise_xn(XN_ERR_INVALID, "quantize_rows_i8 expects a matrix, got %s", shape_text(x).c_str());
    const at::Tensor xc = x.contiguous();
    const int64_t m = x.size(0), k = x.size(1);
    at::Tensor xq, xs;
    if (a[1] != Py_None) {
        xq = tensor(a[1]);
        xs = tensor(a[2]);
        if (xq.sizes() != at::IntArrayRef({m, k}) || xq.scalar_type() != at::kChar || xs.sizes() != at::IntArrayRef({m}) ||
            xs.scalar_type() != at::kFloat) {
            PyErr_SetString(PyExc_ValueError, "quantize_rows_i8: out must be (int8 [m,k], float32 [m])");
            throw Raised();
        }
        require_cuda(xq);
        require_cuda(xs);
    } else {
        xq = empty({m, k}, at::kChar, x.device());
        xs = empty({m}, at::kFloat, x.device());
    }
    const xn_dtype dt = dtype_code(x.scalar_type());
    int8_t *q = (int8_t *)xq.data_ptr();
    float *s = (float *)xs.data_ptr();
    const void *xp = xc.data_ptr();
    void *st = stream();
    XN_CALL(xn_mm_quantize_rows_i8(q, s, xp, dt, (size_t)m, (size_t)k, st));
    PyObject *r = PyTuple_New(2);
    if (!r) throw Raised();
    PyTuple_SET_ITEM(r, 0, wrap(std::move(xq)));
    PyTuple_SET_ITEM(r, 1, wrap(std::move(xs)));
    return r;
}

XN_BINDING(linear_block, 7) {  // bits, xq, x_scale, packed weights, n, partials or None, out or None
    const size_t bits = size_arg(a[0]), n = size_arg(a[4]);
    const at::Tensor &xq = tensor(a[1]), &xs = tensor(a[2]), &wq = tensor(a[3]);
    const at::Tensor *part = maybe_tensor(a[5]), *out = maybe_tensor(a[6]);
    require_cuda(xq);
    require_cuda(wq);
    if (xq.dim() != 2) raise_xn(XN_ERR_INVALID, "linear_q%zu expects a matrix of activations, got %s", bits, shape_text(xq).c_str());
    const size_t m = (size_t)xq.size(0), k = (size_t)xq.size(1);
    at::Tensor y = out ? *out : empty({(int64_t)m, (int64_t)n}, at::kFloat, xq.device());
    float *yp = (float *)y.data_ptr();
    const int8_t *q = (const int8_t *)xq.data_ptr();
    const float *s = (const float *)xs.data_ptr();
    const void *w = wq.data_ptr();
    int32_t *pp = part ? (int32_t *)part->data_ptr() : nullptr;
    void *st = stream();
    XN_CALL(bits == 4 ? xn_mm_linear_q4(yp, q, s, w, m, n, k, pp, st) : xn_mm_linear_q8(yp, q, s, w, m, n, k, pp, st));
    return wrap(std::move(y));
}

XN_BINDING(linear_q4_forward, 4) {  // x [..., k], packed weights, n, k: quantize the rows, then the linear
    const at::Tensor &x = tensor(a[0]), &wq = tensor(a[1]);
    const int64_t n = (int64_t)size_arg(a[2]), k = (int64_t)size_arg(a[3]);
    const size_t m = rows_in("linear_q4", x, k);
    require_cuda(x);
    require_cuda(wq);
    const at::Tensor xr = x.contiguous();
    const xn_dtype dt = dtype_code(x.scalar_type());
    // codes and row scales in one block, the scales behind the codes at a 256-byte boundary
    const size_t codes = (m * (size_t)k + 255) / 256 * 256;
    at::Tensor ws = empty({(int64_t)(codes + m * sizeof(float))}, at::kByte, x.device());
    Shape s;
    s.lead(x, x.dim() - 1);
    s.d.push_back(n);
    at::Tensor y = empty(s.d, at::kFloat, x.device());
    int8_t *q = (int8_t *)ws.data_ptr();
    float *sc = (float *)(q + codes), *yp = (float *)y.data_ptr();
    const void *xp = xr.data_ptr(), *w = wq.data_ptr();
    void *st = stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = xn_mm_quantize_rows_i8(q, sc, xp, dt, m, (size_t)k, st);
    if (!rc) rc = xn_mm_linear_q4(yp, q, sc, w, m, (size_t)n, (size_t)k, nullptr, st);
    Py_END_ALLOW_THREADS check(rc);
    return wrap(std::move(y));
}

XN_BINDING(split_rows_e4m3, 2) {  // x [m, k], want_lo
    const at::Tensor &x = tensor(a[0]);
    const bool want_lo = PyObject_IsTrue(a[1]) != 0;
    require_cuda(x);
    if (x.dim() != 2) raise_xn(XN_ERR_INVALID, "split_rows_e4m3 expects a matrix, got %s", shape_text(x).c_str());
    const at::Tensor xc = x.contiguous();
    const int64_t m = x.size(0), k = x.size(1);
    at::Tensor hi = empty({m, k}, at::kByte, x.device()), lo, xs = empty({m}, at::kFloat, x.device());
    if (want_lo) lo = empty({m, k}, at::kByte, x.device());
    const xn_dtype dt = dtype_code(x.scalar_type());
    uint8_t *h = (uint8_t *)hi.data_ptr(), *l = want_lo ? (uint8_t *)lo.data_ptr() : nullptr;
    float *s = (float *)xs.data_ptr();
    const void *xp = xc.data_ptr();
    void *st = stream();
    XN_CALL(xn_mm_split_rows_e4m3(h, l, s, xp, dt, (size_t)m, (size_t)k, st));
    PyObject *r = PyTuple_New(3);
    if (!r) throw Raised();
    PyTuple_SET_ITEM(r, 0, wrap(std::move(hi)));
    PyTuple_SET_ITEM(r, 1, want_lo ? wrap(std::move(lo)) : Py_NewRef(Py_None));
    PyTuple_SET_ITEM(r, 2, wrap(std::move(xs)));
    return r;
}

XN_BINDING(linear_fp8, 6) {  // x [..., k] bf16, weights, scales, variant, workspace or None, out or None
    const at::Tensor &x = tensor(a[0]), &wq = tensor(a[1]), &wsc = tensor(a[2]);
    const int variant = (int)size_arg(a[3]);
    const at::Tensor *work = maybe_tensor(a[4]), *out = maybe_tensor(a[5]);
    const int64_t n = wq.size(0), k = n ? wq.numel() / n : x.size(-1);  // a weight holds whole rows of k bytes
    const size_t m = rows_in("linear_fp8", x, k);
    require_cuda(x);
    require_cuda(wq);
    if (x.scalar_type() != at::kBFloat16) raise_xn(XN_ERR_INVALID, "linear_fp8 takes bf16 activations");
    const at::Tensor xr = x.contiguous();
    const size_t need = xn_mm_linear_fp8_workspace_bytes(m, (size_t)k);
    at::Tensor ws = work ? *work : empty({(int64_t)need}, at::kByte, x.device());
    at::Tensor y;
    if (out) {
        y = *out;
    } else {
        Shape s;
        s.lead(x, x.dim() - 1);
        s.d.push_back(n);
        y = empty(s.d, at::kBFloat16, x.device());
    }
    void *yp = y.data_ptr(), *wp = ws.data_ptr(), *st = stream();
    const void *xp = xr.data_ptr();
    const uint8_t *q = (const uint8_t *)wq.data_ptr();
    const float *s = (const float *)wsc.data_ptr();
    const size_t wbytes = (size_t)ws.numel();
    XN_CALL(xn_mm_linear_fp8(yp, xp, q, s, m, (size_t)n, (size_t)k, variant, wp, wbytes, st));
    return wrap(std::move(y));
}

// ---------------------------------------------------------------------------------------------
// Row operations
// ---------------------------------------------------------------------------------------------
XN_BINDING(rms_norm, 3) {  // x, alpha, eps
    const at::Tensor &x = tensor(a[0]), &al = tensor(a[1]);
    require_cuda(x);
    require_cuda(al);
    const at::Tensor xc = x.contiguous();
    at::Tensor out = empty(x.sizes(), x.scalar_type(), x.device());
    const size_t cols = (size_t)x.size(-1), rows = cols ? (size_t)x.numel() / cols : 0;
    const xn_dtype dt = dtype_code(x.scalar_type());
    const float eps = (float)float_arg(a[2]);
    void *o = out.data_ptr(), *st = stream();
    const void *xp = xc.data_ptr(), *ap = al.data_ptr();
    XN_CALL(xn_mm_rms_norm(dt, o, xp, ap, rows, cols, eps, st));
    return wrap(std::move(out));
}

XN_BINDING(softmax, 1) {
    const at::Tensor &x = tensor(a[0]);
    require_cuda(x);
    const at::Tensor xc = x.contiguous();
    at::Tensor out = empty(x.sizes(), x.scalar_type(), x.device());
    const size_t cols = (size_t)x.size(-1), rows = cols ? (size_t)x.numel() / cols : 0;
    const xn_dtype dt = dtype_code(x.scalar_type());
    void *o = out.data_ptr(), *st = stream();
    const void *xp = xc.data_ptr();
    XN_CALL(xn_mm_softmax(dt, o, xp, rows, cols, st));
    return wrap(std::move(out));
}

XN_BINDING(silu_mul, 1) {
    const at::Tensor &x = tensor(a[0]);
    require_cuda(x);
    const at::Tensor xc = x.contiguous();
    const int64_t width = x.size(-1), hidden = width / 2;
    Shape s;
    s.lead(x, x.dim() - 1);
    s.d.push_back(hidden);
    at::Tensor out = empty(s.d, x.scalar_type(), x.device());
    const size_t rows = width ? (size_t)(x.numel() / width) : 0;
    const xn_dtype dt = dtype_code(x.scalar_type());
    void *o = out.data_ptr(), *st = stream();
    const void *xp = xc.data_ptr();
    XN_CALL(xn_mm_silu_mul(dt, o, xp, rows, (size_t)hidden, st));
    return wrap(std::move(out));
}

XN_BINDING(add, 2) {
    const at::Tensor &x = tensor(a[0]), &y = tensor(a[1]);
    require_cuda(x);
    require_cuda(y);
    if (x.numel() != y.numel() || x.scalar_type() != y.scalar_type())
        raise_xn(XN_ERR_INVALID, "add expects two tensors of one shape and type, got %s and %s", shape_text(x).c_str(), shape_text(y).c_str());
    at::Tensor out = empty(x.sizes(), x.scalar_type(), x.device());  // contiguous, like the copies it is written from
    const at::Tensor xc = x.contiguous(), yc = y.contiguous();
    const xn_dtype dt = dtype_code(x.scalar_type());
    void *o = out.data_ptr(), *st = stream();
    const void *xp = xc.data_ptr(), *yp = yc.data_ptr();
    const size_t count = (size_t)x.numel();
    XN_CALL(xn_mm_add(dt, o, xp, yp, count, st));
    return wrap(std::move(out));
}

// ---------------------------------------------------------------------------------------------
// Convolutions: Tensor::conv1d / Tensor::conv_transpose1d (xn-core/src/ops.rs:253-300, 305-350), same arguments, same
// shape rules and error texts
// ---------------------------------------------------------------------------------------------
void check_conv_bias(const at::Tensor *bias, int64_t out_channels) {
    if (bias && (bias->dim() != 1 || bias->size(0) != out_channels))
        raise_xn(XN_ERR_INVALID, "bias shape mismatch: expected [%lld], got %s", (long long)out_channels, shape_text(*bias).c_str());
}

void check_conv_channels(const char *name, const at::Tensor &x, const at::Tensor &kernel, size_t groups) {
    if (x.dim() != 3 || kernel.dim() != 3)
        raise_xn(XN_ERR_INVALID, "%s expects rank-3 input and kernel, got %s and %s", name, shape_text(x).c_str(),
                 shape_text(kernel).c_str());
    if (groups < 1 || x.size(1) % (int64_t)groups)
        raise_xn(XN_ERR_INVALID, "in_channels (%lld) must be divisible by groups (%zu)", (long long)x.size(1), groups);
}

XN_BINDING(conv1d, 7) {  // x, kernel, bias or None, stride, padding, dilation, groups
    const at::Tensor &x = tensor(a[0]), &kernel = tensor(a[1]);
    const at::Tensor *bias = maybe_tensor(a[2]);
    const size_t stride = size_arg(a[3]), padding = size_arg(a[4]), dilation = size_arg(a[5]), groups = size_arg(a[6]);
    require_cuda(x);
    require_cuda(kernel);
    check_conv_channels("conv1d", x, kernel, groups);
    const size_t batch = (size_t)x.size(0), c_in = (size_t)x.size(1), length = (size_t)x.size(2);
    const size_t c_out = (size_t)kernel.size(0), ks = (size_t)kernel.size(2);
    if (c_out % groups) raise_xn(XN_ERR_INVALID, "out_channels (%zu) must be divisible by groups (%zu)", c_out, groups);
    if ((size_t)kernel.size(1) != c_in / groups)
        raise_xn(XN_ERR_INVALID, "kernel in_channels/groups mismatch: expected %zu, got %lld", c_in / groups, (long long)kernel.size(1));
    check_conv_bias(bias, (int64_t)c_out);
    const size_t span = dilation * (ks - 1) + 1;
    if (length + 2 * padding < span)
        raise_xn(XN_ERR_INVALID, "kernel span %zu exceeds the padded length %zu", span, length + 2 * padding);
    if (stride == 0) raise_xn(XN_ERR_INVALID, "conv1d: stride must be positive");
    const size_t out_length = (length + 2 * padding - span) / stride + 1;
    const at::Tensor xc = x.contiguous(), kc = kernel.contiguous();
    at::Tensor bc;
    if (bias) bc = bias->contiguous();
    at::Tensor out = empty({(int64_t)batch, (int64_t)c_out, (int64_t)out_length}, x.scalar_type(), x.device());
    const xn_dtype dt = dtype_code(x.scalar_type());
    const size_t need = xn_mm_conv1d_workspace_bytes(dt, batch, c_in, c_out, length, ks, stride, padding, dilation, groups);
    at::Tensor ws;
    if (need) ws = empty({(int64_t)need}, at::kByte, x.device());
    void *o = out.data_ptr(), *wp = need ? ws.data_ptr() : nullptr, *st = stream();
    const void *xp = xc.data_ptr(), *kp = kc.data_ptr(), *bp = bias ? bc.data_ptr() : nullptr;
    XN_CALL(xn_mm_conv1d(dt, o, xp, kp, bp, batch, c_in, c_out, length, out_length, ks, stride, padding, dilation, groups, wp, need, st));
    return wrap(std::move(out));
}

XN_BINDING(conv_transpose1d, 7) {  // x, kernel, bias or None, stride, padding, output_padding, groups
    const at::Tensor &x = tensor(a[0]), &kernel = tensor(a[1]);
    const at::Tensor *bias = maybe_tensor(a[2]);
    const size_t stride = size_arg(a[3]), padding = size_arg(a[4]), opad = size_arg(a[5]), groups = size_arg(a[6]);
    require_cuda(x);
    require_cuda(kernel);
    check_conv_channels("conv_transpose1d", x, kernel, groups);
    const size_t batch = (size_t)x.size(0), c_in = (size_t)x.size(1), length = (size_t)x.size(2);
    const size_t c_out = (size_t)kernel.size(1) * groups, ks = (size_t)kernel.size(2);
    if ((size_t)kernel.size(0) != c_in)
        raise_xn(XN_ERR_INVALID, "kernel in_channels mismatch: expected %zu, got %lld", c_in, (long long)kernel.size(0));
    check_conv_bias(bias, (int64_t)c_out);
    const long long out_length = ((long long)length - 1) * (long long)stride + (long long)ks + (long long)opad - 2 * (long long)padding;
    if (out_length < 0) raise_xn(XN_ERR_INVALID, "padding %zu leaves no output", padding);
    const at::Tensor xc = x.contiguous(), kc = kernel.contiguous();
    at::Tensor bc;
    if (bias) bc = bias->contiguous();
    at::Tensor out = empty({(int64_t)batch, (int64_t)c_out, (int64_t)out_length}, x.scalar_type(), x.device());
    const xn_dtype dt = dtype_code(x.scalar_type());
    const size_t need = xn_mm_conv_transpose1d_workspace_bytes(dt, batch, c_in, c_out, length, ks, stride, padding, opad, groups);
    at::Tensor ws;
    if (need) ws = empty({(int64_t)need}, at::kByte, x.device());
    void *o = out.data_ptr(), *wp = need ? ws.data_ptr() : nullptr, *st = stream();
    const void *xp = xc.data_ptr(), *kp = kc.data_ptr(), *bp = bias ? bc.data_ptr() : nullptr;
    XN_CALL(xn_mm_conv_transpose1d(dt, o, xp, kp, bp, batch, c_in, c_out, length, (size_t)out_length, ks, stride, padding, opad,
                                   groups, wp, need, st));
    return wrap(std::move(out));
}

// ---------------------------------------------------------------------------------------------
// Layer loops of xn_b200/decoder.py and xn_b200/prefill.py.  The Python object stays the owner of every buffer and
// weight (attributes and layer dicts are read on each call, so replacing one takes effect on the next); only the walk
// over the layers, with its ten or so library calls each, is native.
// ---------------------------------------------------------------------------------------------
struct Ref {  // an owned reference
    PyObject *p;
    explicit Ref(PyObject *o) : p(o) {
        if (!o) throw Raised();
    }
    Ref(const Ref &) = delete;
    ~Ref() { Py_DECREF(p); }
};

const char *const ATTR_NAMES[] = {"B", "T", "d", "H", "hid", "ctx", "eps", "variant", "attention", "layers", "hi", "lo", "xs",
                                  "qkv", "attn", "attn_ws", "attn_ws_bytes", "proj", "h", "x_mid", "x_out", "pos", "mask",
                                  "attn_full", "proj_full", "h_l", "t", "norm1", "norm2", "in_proj", "out_proj", "linear_in",
                                  "linear_out", "k", "v"};
enum Attr { A_B, A_T, A_d, A_H, A_hid, A_ctx, A_eps, A_variant, A_attention, A_layers, A_hi, A_lo, A_xs,
            A_qkv, A_attn, A_attn_ws, A_attn_ws_bytes, A_proj, A_h, A_x_mid, A_x_out, A_pos, A_mask,
            A_attn_full, A_proj_full, A_h_l, A_t, A_norm1, A_norm2, A_in_proj, A_out_proj, A_linear_in,
            A_linear_out, A_k, A_v, A_COUNT };
PyObject *g_attr[A_COUNT];

// Attributes are read from the object under the interpreter lock; the object keeps what they refer to alive (a caller
// that replaces a buffer while a step is being enqueued on another thread was never supported).
void *attr_ptr(PyObject *o, Attr at, bool none_ok = false) {
    Ref r(PyObject_GetAttr(o, g_attr[at]));
    if (none_ok && r.p == Py_None) return nullptr;
    return tensor(r.p).data_ptr();
}
size_t attr_size(PyObject *o, Attr at) {
    Ref r(PyObject_GetAttr(o, g_attr[at]));
    return size_arg(r.p);
}
double attr_float(PyObject *o, Attr at) {
    Ref r(PyObject_GetAttr(o, g_attr[at]));
    return float_arg(r.p);
}
void *item_ptr(PyObject *dict, Attr key) {
    PyObject *o = PyDict_GetItemWithError(dict, g_attr[key]);  // borrowed
    if (!o) {
        if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, g_attr[key]);
        throw Raised();
    }
    return tensor(o).data_ptr();
}

struct Weight {
    const uint8_t *q;
    const float *s;
};
Weight item_weight(PyObject *dict, Attr key) {
    PyObject *o = PyDict_GetItemWithError(dict, g_attr[key]);
    if (!o || !PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 2) {
        if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, g_attr[key]);
        throw Raised();
    }
    return {(const uint8_t *)tensor(PyTuple_GET_ITEM(o, 0)).data_ptr(), (const float *)tensor(PyTuple_GET_ITEM(o, 1)).data_ptr()};
}

struct Layer {
    const void *norm1, *norm2;
    Weight in_proj, out_proj, linear_in, linear_out;
    void *k, *v;
};
void read_layers(PyObject *o, bool caches, c10::SmallVectorImpl<Layer> &out) {
    Ref list(PyObject_GetAttr(o, g_attr[A_layers]));
    if (!PyList_Check(list.p)) {
        PyErr_SetString(PyExc_TypeError, "layers must be a list of dicts");
        throw Raised();
    }
    const size_t n = (size_t)PyList_GET_SIZE(list.p);
    out.resize(n);
    for (size_t i = 0; i < n; ++i) {
        PyObject *d = PyList_GET_ITEM(list.p, (Py_ssize_t)i);
        if (!PyDict_Check(d)) {
            PyErr_SetString(PyExc_TypeError, "layers must be a list of dicts");
            throw Raised();
        }
        out[i] = Layer{item_ptr(d, A_norm1), item_ptr(d, A_norm2), item_weight(d, A_in_proj), item_weight(d, A_out_proj),
                       item_weight(d, A_linear_in), item_weight(d, A_linear_out), caches ? item_ptr(d, A_k) : nullptr,
                       caches ? item_ptr(d, A_v) : nullptr};
    }
}

XN_BINDING(decoder_step, 2) {  // DecoderStack, x -> x_out
    PyObject *o = a[0];
    const at::Tensor &x = tensor(a[1]);
    const size_t B = attr_size(o, A_B), d = attr_size(o, A_d), H = attr_size(o, A_H), hid = attr_size(o, A_hid), ctx = attr_size(o, A_ctx);
    const float eps = (float)attr_float(o, A_eps);
    const bool two_pieces = attr_size(o, A_variant) == 0;
    int mode = 0;  // 0 separate launches, 1 fused, 2 fused in one launch
    {
        Ref at(PyObject_GetAttr(o, g_attr[A_attention]));
        const char *t = PyUnicode_AsUTF8(at.p);
        if (!t) throw Raised();
        mode = !strcmp(t, "separate") ? 0 : !strcmp(t, "fused_one_launch") ? 2 : 1;
    }
    uint8_t *hi = (uint8_t *)attr_ptr(o, A_hi), *lo = two_pieces ? (uint8_t *)attr_ptr(o, A_lo) : nullptr;
    float *xs = (float *)attr_ptr(o, A_xs);
    char *qkv = (char *)attr_ptr(o, A_qkv);
    void *attn = attr_ptr(o, A_attn), *ws = attr_ptr(o, A_attn_ws), *proj = attr_ptr(o, A_proj), *h = attr_ptr(o, A_h);
    void *x_mid = attr_ptr(o, A_x_mid), *x_out = attr_ptr(o, A_x_out);
    const size_t ws_bytes = attr_size(o, A_attn_ws_bytes);
    const int64_t *pos = (const int64_t *)attr_ptr(o, A_pos);
    const float *mask = (const float *)attr_ptr(o, A_mask, true);
    c10::SmallVector<Layer, 64> layers;
    read_layers(o, true, layers);
    const void *cur = x.data_ptr();
    void *st = stream();
    const float scale = (float)(1.0 / std::sqrt(128.0));
    auto steps = [&]() -> int {
        for (size_t i = 0; i < layers.size(); ++i) {
            const Layer &y = layers[i];
            int rc = 0;
            if (i == 0)  // later layers get their pieces from the fused add + norm that ends the previous layer
                rc = xn_mm_rms_norm_split_e4m3(hi, lo, xs, nullptr, cur, y.norm1, XN_BF16, B, d, eps, st);
            if (!rc) rc = xn_mm_linear_fp8_pieces(qkv, hi, lo, xs, y.in_proj.q, y.in_proj.s, B, 3 * d, d, st);
            if (rc) return rc;
            const char *q = qkv, *kn = qkv + 2 * d, *vn = qkv + 4 * d;
            if (mode == 0) {
                rc = xn_mm_kv_append2(XN_BF16, y.k, y.v, kn, vn, 3 * d, pos, B, H, ctx, 128, st);
                // the merge of the context slices also writes the e4m3 pieces of the output row
                if (!rc)
                    rc = xn_mm_decode_attention_split_e4m3(hi, lo, xs, attn, q, 3 * d, y.k, y.v, mask, B, H, ctx, 128, scale, ws,
                                                           ws_bytes, st);
            } else {
                // append the new key / value rows, attend over the cache, merge the slices, write the pieces
                rc = xn_mm_decode_attention_append_e4m3(hi, lo, xs, attn, q, kn, vn, 3 * d, y.k, y.v, pos, mask, B, H, ctx, 128, scale,
                                                        mode == 2 ? 1 : 0, ws, ws_bytes, st);
            }
            if (!rc) rc = xn_mm_linear_fp8_pieces(proj, hi, lo, xs, y.out_proj.q, y.out_proj.s, B, d, d, st);
            if (!rc) rc = xn_mm_add_rms_norm_split_e4m3(hi, lo, xs, x_mid, cur, proj, y.norm2, XN_BF16, B, d, eps, st);
            if (!rc) rc = xn_mm_linear_fp8_pieces(h, hi, lo, xs, y.linear_in.q, y.linear_in.s, B, 2 * hid, d, st);
            if (!rc) rc = xn_mm_silu_mul_split_e4m3(hi, lo, xs, h, XN_BF16, B, hid, st);
            if (!rc) rc = xn_mm_linear_fp8_pieces(proj, hi, lo, xs, y.linear_out.q, y.linear_out.s, B, d, hid, st);
            if (!rc)  // x_out = x_mid + proj, and the pieces of the next layer's norm1(x_out)
                rc = i + 1 < layers.size()
                         ? xn_mm_add_rms_norm_split_e4m3(hi, lo, xs, x_out, x_mid, proj, layers[i + 1].norm1, XN_BF16, B, d, eps, st)
                         : xn_mm_add(XN_BF16, x_out, x_mid, proj, B * d, st);
            if (rc) return rc;
            cur = x_out;
        }
        return 0;
    };
    XN_CALL(steps());
    PyObject *out = PyObject_GetAttr(o, g_attr[A_x_out]);
    if (!out) throw Raised();
    return out;
}

// One rank with every head and channel: nothing is exchanged, the attention writes the rows the out projection reads.
XN_BINDING(prefill_forward, 2) {  // PrefillStack (world 1, fused attention), x -> x_out
    PyObject *o = a[0];
    const at::Tensor &x = tensor(a[1]);
    const size_t T = attr_size(o, A_T), d = attr_size(o, A_d), H = attr_size(o, A_H), hid = attr_size(o, A_hid);
    const float eps = (float)attr_float(o, A_eps);
    const bool two_pieces = attr_size(o, A_variant) == 0;
    uint8_t *hi = (uint8_t *)attr_ptr(o, A_hi), *lo = two_pieces ? (uint8_t *)attr_ptr(o, A_lo) : nullptr;
    float *xs = (float *)attr_ptr(o, A_xs);
    char *qkv = (char *)attr_ptr(o, A_qkv);
    void *h = attr_ptr(o, A_h_l), *x_mid = attr_ptr(o, A_x_mid), *x_out = attr_ptr(o, A_x_out);
    Ref attn_full(PyObject_GetAttr(o, g_attr[A_attn_full])), proj_full(PyObject_GetAttr(o, g_attr[A_proj_full]));
    void *attn = attr_ptr(attn_full.p, A_t), *proj = attr_ptr(proj_full.p, A_t);
    c10::SmallVector<Layer, 64> layers;
    read_layers(o, false, layers);
    const void *cur = x.data_ptr();
    void *st = stream();
    const float scale = (float)(1.0 / std::sqrt(128.0));
    void *dst[1] = {proj};
    auto steps = [&]() -> int {
        for (size_t i = 0; i < layers.size(); ++i) {
            const Layer &y = layers[i];
            int rc = 0;
            if (i == 0) rc = xn_mm_rms_norm_split_e4m3(hi, lo, xs, nullptr, cur, y.norm1, XN_BF16, T, d, eps, st);
            if (!rc) rc = xn_mm_linear_fp8_pieces(qkv, hi, lo, xs, y.in_proj.q, y.in_proj.s, T, 3 * d, d, st);
            if (!rc)
                rc = xn_mm_attention_prefill(XN_BF16, attn, d, qkv, qkv + 2 * d, qkv + 4 * d, 3 * d, 128, H, 128, T, T, scale, st);
            if (!rc) rc = xn_mm_split_rows_e4m3(hi, lo, xs, attn, XN_BF16, T, d, st);
            if (!rc) rc = xn_mm_linear_fp8_pieces_scatter(dst, 1, d, 0, hi, lo, xs, y.out_proj.q, y.out_proj.s, T, d, d, st);
            if (!rc) rc = xn_mm_add_rms_norm_split_e4m3(hi, lo, xs, x_mid, cur, proj, y.norm2, XN_BF16, T, d, eps, st);
            if (!rc) rc = xn_mm_linear_fp8_pieces(h, hi, lo, xs, y.linear_in.q, y.linear_in.s, T, 2 * hid, d, st);
            if (!rc) rc = xn_mm_silu_mul_split_e4m3(hi, lo, xs, h, XN_BF16, T, hid, st);
            if (!rc) rc = xn_mm_linear_fp8_pieces_scatter(dst, 1, d, 0, hi, lo, xs, y.linear_out.q, y.linear_out.s, T, d, hid, st);
            if (!rc)
                rc = i + 1 < layers.size()
                         ? xn_mm_add_rms_norm_split_e4m3(hi, lo, xs, x_out, x_mid, proj, layers[i + 1].norm1, XN_BF16, T, d, eps, st)
                         : xn_mm_add(XN_BF16, x_out, x_mid, proj, T * d, st);
            if (rc) return rc;
            cur = x_out;
        }
        return 0;
    };
    XN_CALL(steps());
    PyObject *out = PyObject_GetAttr(o, g_attr[A_x_out]);
    if (!out) throw Raised();
    return out;
}

XN_BINDING(set_error_class, 1) {
    Py_INCREF(a[0]);
    Py_XDECREF(g_error_class);
    g_error_class = a[0];
    Py_RETURN_NONE;
}

#define XN_METHOD(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr}
PyMethodDef METHODS[] = {
    XN_METHOD(matmul_), XN_METHOD(matmul_with_t), XN_METHOD(linear), XN_METHOD(quantize_rows_i8), XN_METHOD(linear_block),
    XN_METHOD(linear_q4_forward), XN_METHOD(split_rows_e4m3), XN_METHOD(linear_fp8), XN_METHOD(rms_norm), XN_METHOD(softmax),
    XN_METHOD(silu_mul), XN_METHOD(add), XN_METHOD(conv1d), XN_METHOD(conv_transpose1d), XN_METHOD(decoder_step),
    XN_METHOD(prefill_forward), XN_METHOD(set_error_class), {nullptr, nullptr, 0, nullptr}};
PyModuleDef MODULE = {PyModuleDef_HEAD_INIT, "_host", "Native host path of the operators.", -1, METHODS, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    static_assert(sizeof ATTR_NAMES / sizeof *ATTR_NAMES == A_COUNT, "one name per attribute");
    for (int i = 0; i < A_COUNT; ++i)
        if (!(g_attr[i] = PyUnicode_InternFromString(ATTR_NAMES[i]))) return nullptr;
    return PyModule_Create(&MODULE);
}
