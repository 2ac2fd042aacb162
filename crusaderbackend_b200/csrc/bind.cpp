// CPython face of the C ABI: takes torch tensors, reads their extents, strides and device pointers natively and calls
// libcrusader_b200.so. A call through ctypes costs 4 to 10 us of interpreter work (shape tuples, pointer objects, up to 18
// converted arguments), more than most of the small kernels run; here it is well under one.
//
// Every function: first argument the cb_ctx* as an integer, then tensors (None where the ABI allows NULL) and plain values;
// ValueError for operands the ABI cannot take, the exception class handed to attach() for a CB_E* return code. The GIL is
// released while the library runs.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/crusader_b200.h"

namespace {

#define CB_FUNCTIONS(X)                                                                                              \
    X(cb_last_error) X(cb_gemm) X(cb_gemm_batch_reduce) X(cb_conv_fwd) X(cb_conv_dgrad) X(cb_conv_wgrad) X(cb_conv_bias) \
    X(cb_conv_bias_grad) X(cb_linear_fwd) X(cb_linear_xgrad) X(cb_linear_paramgrad) X(cb_bn_fwd) X(cb_bn_bwd)          \
    X(cb_bn_paramgrad) X(cb_bn_bwd_fused) X(cb_bn_fwd_relu) X(cb_add_relu) X(cb_relu_grad2) X(cb_relu) X(cb_relu_grad) \
    X(cb_tensor_op) X(cb_grad_handover) X(cb_avgpool) X(cb_avgpool_back) X(cb_global_avgpool) X(cb_global_avgpool_back) \
    X(cb_softmax) X(cb_cross_entropy) X(cb_momentum)
struct Library {
#define X(name) decltype(&::name) name = nullptr;
    CB_FUNCTIONS(X)
#undef X
} lib;
PyObject* error_class = nullptr;

struct BadCall {
    const char* what;  // nullptr: a Python error is already set
};

struct Args {
    PyObject* const* a;
    Py_ssize_t n;
    cb_ctx* ctx;
    Args(PyObject* const* args, Py_ssize_t count, Py_ssize_t want) : a(args), n(count) {
        if (count != want) throw BadCall{"wrong number of arguments"};
        if (!lib.cb_gemm) throw BadCall{"the CUDA library is not attached"};
        ctx = static_cast<cb_ctx*>(PyLong_AsVoidPtr(a[0]));
        if (!ctx && PyErr_Occurred()) throw BadCall{nullptr};
    }
    const at::Tensor& tensor(int i) const {
        if (!THPVariable_Check(a[i])) throw BadCall{"operands must be fp32 CUDA tensors"};
        return THPVariable_Unpack(a[i]);
    }
    static float* ptr(const at::Tensor& t) {
        if (!t.is_cuda() || t.scalar_type() != at::kFloat) throw BadCall{"operands must be fp32 CUDA tensors"};
        return static_cast<float*>(t.data_ptr());
    }
    float* ptr(int i) const { return a[i] == Py_None ? nullptr : ptr(tensor(i)); }
    int flag(int i) const {
        const int v = PyObject_IsTrue(a[i]);
        if (v < 0) throw BadCall{nullptr};
        return v;
    }
    long long integer(int i) const {
        const long long v = PyLong_AsLongLong(a[i]);
        if (v == -1 && PyErr_Occurred()) throw BadCall{nullptr};
        return v;
    }
    float real(int i) const {
        const double v = PyFloat_AsDouble(a[i]);
        if (v == -1.0 && PyErr_Occurred()) throw BadCall{nullptr};
        return static_cast<float>(v);
    }
    PyObject* returning(int i) const {
        Py_INCREF(a[i]);
        return a[i];
    }
};

// Runs `call` without the GIL and turns its status into a Python exception.
template <class F>
void run(const Args& a, F call) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = call();
    Py_END_ALLOW_THREADS
    if (rc == CB_OK) return;
    PyObject* e = PyObject_CallFunction(error_class, "is", rc, lib.cb_last_error(a.ctx));
    if (e) {
        PyErr_SetObject(error_class, e);
        Py_DECREF(e);
    }
    throw BadCall{nullptr};
}

typedef PyObject* (*Body)(const Args&);
template <int kArgs, Body body>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    try {
        return body(Args(args, n, kArgs));
    } catch (const BadCall& e) {
        if (e.what) PyErr_SetString(PyExc_ValueError, e.what);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_ValueError, e.what());
    }
    return nullptr;
}

int to_int(int64_t v) {
    if (v > INT_MAX || v < INT_MIN) throw BadCall{"an extent does not fit 32 bits"};
    return static_cast<int>(v);
}

struct Matrix {
    int64_t batch, rows, cols, ld, stride;
    float* p;
    explicit Matrix(const at::Tensor& t) {
        const int64_t d = t.dim();
        if (d != 2 && d != 3) throw BadCall{"operands are 2-D or 3-D"};
        if (t.stride(d - 1) != 1) throw BadCall{"operands must be row-major (unit inner stride)"};
        batch = d == 3 ? t.size(0) : 1;
        stride = d == 3 ? t.stride(0) : 0;
        rows = t.size(d - 2);
        cols = t.size(d - 1);
        ld = t.stride(d - 2);
        p = Args::ptr(t);
    }
};

// (ctx, A, B, C, transA, transB, accumulate) -> C
PyObject* gemm(const Args& a) {
    const Matrix A(a.tensor(1)), B(a.tensor(2)), C(a.tensor(3));
    const int tA = a.flag(4), tB = a.flag(5), acc = a.flag(6);
    const int64_t K = tA ? A.rows : A.cols;
    if ((tA ? A.cols : A.rows) != C.rows || (tB ? B.cols : B.rows) != K || (tB ? B.rows : B.cols) != C.cols)
        throw BadCall{"gemm: shapes do not agree"};
    const int64_t nb = C.batch;
    if ((A.batch != 1 && A.batch != nb) || (B.batch != 1 && B.batch != nb)) throw BadCall{"gemm: batch sizes do not agree"};
    const int M = to_int(C.rows), N = to_int(C.cols), k = to_int(K), lda = to_int(A.ld), ldb = to_int(B.ld), ldc = to_int(C.ld),
              n = to_int(nb);
    run(a, [&] {
        return lib.cb_gemm(a.ctx, tA, tB, M, N, k, A.p, lda, B.p, ldb, C.p, ldc, n, A.batch == nb ? A.stride : 0,
                           B.batch == nb ? B.stride : 0, C.stride, acc);
    });
    return a.returning(3);
}

// (ctx, A, B, C) -> C: C += sum over n of A[n] B[n]^T
PyObject* gemm_nta(const Args& a) {
    const at::Tensor &tA = a.tensor(1), &tB = a.tensor(2), &tC = a.tensor(3);
    if (tA.dim() != 3 || tB.dim() != 3 || tC.dim() != 2) throw BadCall{"sgemmNTA: A and B are 3-D (batch first), C is 2-D"};
    const Matrix A(tA), B(tB), C(tC);
    if (B.batch != A.batch || B.cols != A.cols || C.rows != A.rows || C.cols != B.rows) throw BadCall{"sgemmNTA: shapes do not agree"};
    const int M = to_int(A.rows), N = to_int(B.rows), K = to_int(A.cols), lda = to_int(A.ld), ldb = to_int(B.ld), ldc = to_int(C.ld),
              n = to_int(A.batch);
    run(a, [&] { return lib.cb_gemm_batch_reduce(a.ctx, 0, 1, M, N, K, A.p, lda, B.p, ldb, C.p, ldc, n, A.stride, B.stride, 1); });
    return a.returning(3);
}

struct Geometry {
    int N, IC, IH, IW, OC, FH, FW, s[2], p[2];
    Geometry(const Args& a, const at::Tensor& W, const at::Tensor& X, int first) {
        if (W.dim() != 4 || X.dim() != 4) throw BadCall{"conv: filters and maps are 4-D"};
        if (W.size(1) != X.size(1)) throw BadCall{"conv: channel counts do not agree"};
        N = to_int(X.size(0)); IC = to_int(X.size(1)); IH = to_int(X.size(2)); IW = to_int(X.size(3));
        OC = to_int(W.size(0)); FH = to_int(W.size(2)); FW = to_int(W.size(3));
        for (int i = 0; i < 2; ++i) {
            s[i] = to_int(a.integer(first + i));
            p[i] = to_int(a.integer(first + 2 + i));
        }
    }
};

// (ctx, W, X, Y, strideH, strideW, padH, padW, bias, relu) -> Y
PyObject* conv(const Args& a) {
    const Geometry g(a, a.tensor(1), a.tensor(2), 4);
    float *W = a.ptr(1), *X = a.ptr(2), *Y = a.ptr(3), *b = a.ptr(8);
    const int relu = a.flag(9);
    run(a, [&] {
        return lib.cb_conv_fwd(a.ctx, W, X, Y, b, g.N, g.IC, g.IH, g.IW, g.OC, g.FH, g.FW, g.s[0], g.s[1], g.p[0], g.p[1], relu);
    });
    return a.returning(3);
}
// (ctx, W, dY, dX, strideH, strideW, padH, padW) -> dX
PyObject* conv_dgrad(const Args& a) {
    const Geometry g(a, a.tensor(1), a.tensor(3), 4);
    float *W = a.ptr(1), *dY = a.ptr(2), *dX = a.ptr(3);
    run(a, [&] {
        return lib.cb_conv_dgrad(a.ctx, W, dY, dX, g.N, g.IC, g.IH, g.IW, g.OC, g.FH, g.FW, g.s[0], g.s[1], g.p[0], g.p[1]);
    });
    return a.returning(3);
}
// (ctx, dY, X, dW, strideH, strideW, padH, padW, accumulate) -> dY
PyObject* conv_wgrad(const Args& a) {
    const Geometry g(a, a.tensor(3), a.tensor(2), 4);
    float *dY = a.ptr(1), *X = a.ptr(2), *dW = a.ptr(3);
    const int acc = a.flag(8);
    run(a, [&] {
        return lib.cb_conv_wgrad(a.ctx, dY, X, dW, g.N, g.IC, g.IH, g.IW, g.OC, g.FH, g.FW, g.s[0], g.s[1], g.p[0], g.p[1], acc);
    });
    return a.returning(1);
}

void map_extents(const at::Tensor& t, int (&d)[4]) {
    if (t.dim() != 4) throw BadCall{"feature maps are 4-D"};
    for (int i = 0; i < 4; ++i) d[i] = to_int(t.size(i));
}
int64_t leading(const at::Tensor& t) {
    if (t.dim() < 1 || t.size(0) < 1) throw BadCall{"an operand without samples"};
    return t.size(0);
}

// (ctx, Y, bias) -> Y
PyObject* conv_bias(const Args& a) {
    int d[4];
    map_extents(a.tensor(1), d);
    float *Y = a.ptr(1), *b = a.ptr(2);
    run(a, [&] { return lib.cb_conv_bias(a.ctx, Y, b, d[0], d[1], d[2] * d[3]); });
    return a.returning(1);
}
// (ctx, dY, db, accumulate) -> db
PyObject* conv_bias_grad(const Args& a) {
    int d[4];
    map_extents(a.tensor(1), d);
    float *dY = a.ptr(1), *db = a.ptr(2);
    const int acc = a.flag(3);
    run(a, [&] { return lib.cb_conv_bias_grad(a.ctx, dY, db, d[0], d[1], d[2] * d[3], acc); });
    return a.returning(2);
}

struct Dense {
    int batch, ins, outs;
    Dense(int64_t b, int64_t i, const at::Tensor& W) : batch(to_int(b)), ins(to_int(i)) {
        if (W.dim() < 2) throw BadCall{"dense weights are at least 2-D"};
        outs = to_int(W.size(W.dim() - 2));
    }
};
// (ctx, X, W, b, Y) -> Y
PyObject* linear(const Args& a) {
    const at::Tensor& X = a.tensor(1);
    const int64_t n = leading(X);
    const Dense d(n, X.numel() / n, a.tensor(2));
    float *x = a.ptr(1), *W = a.ptr(2), *b = a.ptr(3), *Y = a.ptr(4);
    run(a, [&] { return lib.cb_linear_fwd(a.ctx, x, W, b, Y, d.batch, d.ins, d.outs); });
    return a.returning(4);
}
// (ctx, dY, W, dX) -> dX
PyObject* linear_xgrad(const Args& a) {
    const at::Tensor &W = a.tensor(2), &dX = a.tensor(3);
    if (W.dim() < 2) throw BadCall{"dense weights are at least 2-D"};
    const Dense d(leading(dX), W.size(W.dim() - 1), W);
    float *dY = a.ptr(1), *w = a.ptr(2), *dx = a.ptr(3);
    run(a, [&] { return lib.cb_linear_xgrad(a.ctx, dY, w, dx, d.batch, d.ins, d.outs); });
    return a.returning(3);
}
// (ctx, dY, X, dW, db) -> dW
PyObject* linear_paramgrad(const Args& a) {
    const at::Tensor& dW = a.tensor(3);
    if (dW.dim() < 2) throw BadCall{"dense weights are at least 2-D"};
    const Dense d(leading(a.tensor(2)), dW.size(dW.dim() - 1), dW);
    float *dY = a.ptr(1), *X = a.ptr(2), *dw = a.ptr(3), *db = a.ptr(4);
    run(a, [&] { return lib.cb_linear_paramgrad(a.ctx, dY, X, dw, db, d.batch, d.ins, d.outs); });
    return a.returning(3);
}

struct Samples {
    int N;
    long long P;
    explicit Samples(const at::Tensor& t) : N(to_int(leading(t))), P(t.numel() / t.size(0)) {}
};
// (ctx, X, beta, gamma, mean, var, Y, xhat) -> Y
PyObject* bn_fwd(const Args& a) {
    const Samples s(a.tensor(1));
    float* v[8];
    for (int i = 1; i < 8; ++i) v[i] = a.ptr(i);
    run(a, [&] { return lib.cb_bn_fwd(a.ctx, v[1], v[2], v[3], v[4], v[5], v[6], v[7], s.N, s.P); });
    return a.returning(6);
}
// (ctx, dY, gamma, X, dX) -> dX
PyObject* bn_bwd(const Args& a) {
    const Samples s(a.tensor(3));
    float *dY = a.ptr(1), *gamma = a.ptr(2), *X = a.ptr(3), *dX = a.ptr(4);
    run(a, [&] { return lib.cb_bn_bwd(a.ctx, dY, gamma, X, dX, s.N, s.P); });
    return a.returning(4);
}
// (ctx, dY, xhat, dgamma, dbeta) -> None
PyObject* bn_paramgrad(const Args& a) {
    const Samples s(a.tensor(1));
    float *dY = a.ptr(1), *xhat = a.ptr(2), *dgamma = a.ptr(3), *dbeta = a.ptr(4);
    run(a, [&] { return lib.cb_bn_paramgrad(a.ctx, dY, xhat, dgamma, dbeta, s.N, s.P); });
    Py_RETURN_NONE;
}
// (ctx, dY, gamma, X, dX, dgamma, dbeta, relu_out) -> dX
PyObject* bn_bwd_fused(const Args& a) {
    const Samples s(a.tensor(3));
    float* v[8];
    for (int i = 1; i < 8; ++i) v[i] = a.ptr(i);
    run(a, [&] { return lib.cb_bn_bwd_fused(a.ctx, v[1], v[2], v[3], v[4], v[5], v[6], v[7], s.N, s.P); });
    return a.returning(4);
}
// (ctx, X, beta, gamma, Y) -> Y
PyObject* bn_fwd_relu(const Args& a) {
    const Samples s(a.tensor(1));
    float *X = a.ptr(1), *beta = a.ptr(2), *gamma = a.ptr(3), *Y = a.ptr(4);
    run(a, [&] { return lib.cb_bn_fwd_relu(a.ctx, X, beta, gamma, Y, s.N, s.P); });
    return a.returning(4);
}

// (ctx, A, B, Out) -> Out
PyObject* add_relu(const Args& a) {
    const long long n = a.tensor(1).numel();
    float *A = a.ptr(1), *B = a.ptr(2), *out = a.ptr(3);
    run(a, [&] { return lib.cb_add_relu(a.ctx, A, B, out, n); });
    return a.returning(3);
}
// (ctx, Y, dY, dA, dB) -> dA
PyObject* relu_grad2(const Args& a) {
    const long long n = a.tensor(1).numel();
    float *Y = a.ptr(1), *dY = a.ptr(2), *dA = a.ptr(3), *dB = a.ptr(4);
    run(a, [&] { return lib.cb_relu_grad2(a.ctx, Y, dY, dA, dB, n); });
    return a.returning(3);
}
// (ctx, X, Y) -> Y
PyObject* relu(const Args& a) {
    const long long n = a.tensor(1).numel();
    float *X = a.ptr(1), *Y = a.ptr(2);
    run(a, [&] { return lib.cb_relu(a.ctx, X, Y, n); });
    return a.returning(2);
}
// (ctx, X, dY, dX) -> dX
PyObject* relu_grad(const Args& a) {
    const long long n = a.tensor(1).numel();
    float *X = a.ptr(1), *dY = a.ptr(2), *dX = a.ptr(3);
    run(a, [&] { return lib.cb_relu_grad(a.ctx, X, dY, dX, n); });
    return a.returning(3);
}
// (ctx, op, A, B, scalar) -> A
PyObject* tensor_op(const Args& a) {
    const int op = to_int(a.integer(1));
    const long long n = a.tensor(2).numel();
    float *A = a.ptr(2), *B = a.ptr(3), scalar = a.real(4);
    run(a, [&] { return lib.cb_tensor_op(a.ctx, op, A, B, scalar, n); });
    return a.returning(2);
}
// (ctx, dA, dA_reserve) -> dA
PyObject* grad_handover(const Args& a) {
    const long long n = a.tensor(1).numel();
    float *dA = a.ptr(1), *reserve = a.ptr(2);
    run(a, [&] { return lib.cb_grad_handover(a.ctx, dA, reserve, n); });
    return a.returning(1);
}

// (ctx, X, Y, rangeH, rangeW) -> Y
PyObject* avgpool(const Args& a) {
    int d[4];
    map_extents(a.tensor(1), d);
    float *X = a.ptr(1), *Y = a.ptr(2);
    const int rh = to_int(a.integer(3)), rw = to_int(a.integer(4));
    run(a, [&] { return lib.cb_avgpool(a.ctx, X, Y, (long long)d[0] * d[1], d[2], d[3], rh, rw); });
    return a.returning(2);
}
// (ctx, dX, dY, rangeH, rangeW) -> dX
PyObject* avgpool_back(const Args& a) {
    int d[4];
    map_extents(a.tensor(1), d);
    float *dX = a.ptr(1), *dY = a.ptr(2);
    const int rh = to_int(a.integer(3)), rw = to_int(a.integer(4));
    run(a, [&] { return lib.cb_avgpool_back(a.ctx, dX, dY, (long long)d[0] * d[1], d[2], d[3], rh, rw); });
    return a.returning(1);
}
// (ctx, X, Y) -> Y
PyObject* global_avgpool(const Args& a) {
    int d[4];
    map_extents(a.tensor(1), d);
    float *X = a.ptr(1), *Y = a.ptr(2);
    run(a, [&] { return lib.cb_global_avgpool(a.ctx, X, Y, (long long)d[0] * d[1], d[2] * d[3]); });
    return a.returning(2);
}
// (ctx, dX, dY) -> dX
PyObject* global_avgpool_back(const Args& a) {
    int d[4];
    map_extents(a.tensor(1), d);
    float *dX = a.ptr(1), *dY = a.ptr(2);
    run(a, [&] { return lib.cb_global_avgpool_back(a.ctx, dX, dY, (long long)d[0] * d[1], d[2] * d[3]); });
    return a.returning(1);
}

// (ctx, A, out, step) -> out; step 0: one row per sample
PyObject* softmax(const Args& a) {
    const at::Tensor& A = a.tensor(1);
    long long step = a.integer(3);
    if (step == 0) step = A.numel() / leading(A);
    if (step < 1) throw BadCall{"softmax: empty rows"};
    float *x = a.ptr(1), *y = a.ptr(2);
    const int rows = to_int(A.numel() / step), width = to_int(step);
    run(a, [&] { return lib.cb_softmax(a.ctx, x, y, rows, width); });
    return a.returning(2);
}
// (ctx, Y, labels, dY, loss) -> loss
PyObject* cross_entropy(const Args& a) {
    const long long n = a.tensor(1).numel();
    float *Y = a.ptr(1), *labels = a.ptr(2), *dY = a.ptr(3), *loss = a.ptr(4);
    run(a, [&] { return lib.cb_cross_entropy(a.ctx, Y, labels, dY, loss, n); });
    return a.returning(4);
}
// (ctx, w, g, m, lr, beta, l2, is_weight) -> None
PyObject* momentum(const Args& a) {
    const long long n = a.tensor(1).numel();
    float *w = a.ptr(1), *g = a.ptr(2), *m = a.ptr(3), lr = a.real(4), beta = a.real(5), l2 = a.real(6);
    const int is_weight = a.flag(7);
    run(a, [&] { return lib.cb_momentum(a.ctx, w, g, m, n, lr, beta, l2, is_weight); });
    Py_RETURN_NONE;
}

// (dlopen handle of libcrusader_b200.so, exception class): resolves the library's entry points
PyObject* attach(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2) {
        PyErr_SetString(PyExc_ValueError, "attach takes the library handle and the exception class");
        return nullptr;
    }
    void* handle = PyLong_AsVoidPtr(args[0]);
    if (!handle) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null library handle");
        return nullptr;
    }
    Library found;
#define X(name)                                                                     \
    found.name = reinterpret_cast<decltype(found.name)>(dlsym(handle, #name));      \
    if (!found.name) {                                                              \
        PyErr_SetString(PyExc_RuntimeError, "libcrusader_b200.so lacks " #name);    \
        return nullptr;                                                             \
    }
    CB_FUNCTIONS(X)
#undef X
    Py_INCREF(args[1]);
    Py_XDECREF(error_class);
    error_class = args[1];
    lib = found;
    Py_RETURN_NONE;
}

#define ENTRY(name, nargs) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<nargs, name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"attach", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&attach)), METH_FASTCALL, nullptr},
    ENTRY(gemm, 7), ENTRY(gemm_nta, 4), ENTRY(conv, 10), ENTRY(conv_dgrad, 8), ENTRY(conv_wgrad, 9), ENTRY(conv_bias, 3),
    ENTRY(conv_bias_grad, 4), ENTRY(linear, 5), ENTRY(linear_xgrad, 4), ENTRY(linear_paramgrad, 5), ENTRY(bn_fwd, 8),
    ENTRY(bn_bwd, 5), ENTRY(bn_paramgrad, 5), ENTRY(bn_bwd_fused, 8), ENTRY(bn_fwd_relu, 5), ENTRY(add_relu, 4),
    ENTRY(relu_grad2, 5), ENTRY(relu, 3), ENTRY(relu_grad, 4), ENTRY(tensor_op, 5), ENTRY(grad_handover, 3), ENTRY(avgpool, 5),
    ENTRY(avgpool_back, 5), ENTRY(global_avgpool, 3), ENTRY(global_avgpool_back, 3), ENTRY(softmax, 4), ENTRY(cross_entropy, 5),
    ENTRY(momentum, 8), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
