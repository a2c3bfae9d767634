// Python module _torch_calls: the calls of capi.py that take torch tensors, with everything between the
// Python call and the C ABI in native code: the checks of the tensors, their addresses and sizes, the
// current stream and the device switch.  capi.py keeps the public functions (names, defaults,
// allocation of outputs that are not given) and hands the rest to this module.
//
// What bounds a small call is this host path: a 4096 x 4096 linear takes 4 us on the device, and with
// the same steps as Python statements around a ctypes call one call took 9.9 us (now 4.1).
//
// The library is not linked but bound: capi.py passes the addresses of the functions it has loaded,
// so the range-checked debug build is reached the same way as the normal one.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>

#include "../../../include/jq_b200.h"

namespace {

// ---- functions of the library, bound by capi.py -----------------------------------------------------
decltype(&jq_quantize_q8_1_device) f_quantize = nullptr;
decltype(&jq_mul_mat_q4_0_q8_1_device_ex) f_mul_mat = nullptr;
decltype(&jq_linear_q4_0_device) f_linear = nullptr;
decltype(&jq_linear_q4_0_multi_device) f_multi = nullptr;
decltype(&jq_rms_norm_q8_1_device) f_rms_norm = nullptr;
decltype(&jq_swiglu_q8_1_device) f_swiglu = nullptr;

struct Binding {
    const char *name;
    void **slot;
};
const Binding bindings[] = {
    {"jq_quantize_q8_1_device", reinterpret_cast<void **>(&f_quantize)},
    {"jq_mul_mat_q4_0_q8_1_device_ex", reinterpret_cast<void **>(&f_mul_mat)},
    {"jq_linear_q4_0_device", reinterpret_cast<void **>(&f_linear)},
    {"jq_linear_q4_0_multi_device", reinterpret_cast<void **>(&f_multi)},
    {"jq_rms_norm_q8_1_device", reinterpret_cast<void **>(&f_rms_norm)},
    {"jq_swiglu_q8_1_device", reinterpret_cast<void **>(&f_swiglu)},
};

PyObject *bind(PyObject *, PyObject *addresses) {
    for (const Binding &b : bindings) {
        PyObject *v = PyDict_GetItemString(addresses, b.name);
        if (v == nullptr) {
            PyErr_Format(PyExc_KeyError, "no address given for %s", b.name);
            return nullptr;
        }
        *b.slot = PyLong_AsVoidPtr(v);
        if (PyErr_Occurred()) return nullptr;
    }
    Py_RETURN_NONE;
}

// a reference that is given back on every way out, an exception's included
struct Owned {
    PyObject *p = nullptr;
    ~Owned() { Py_XDECREF(p); }
};

// ---- arguments -------------------------------------------------------------------------------------
const char *dtype_text(at::ScalarType t) { return t == at::kFloat ? "torch.float32" : "torch.uint8"; }

// The tensor behind `o` when it is a contiguous CUDA tensor of this type, else nullptr with ValueError set.
const at::Tensor *tensor_arg(PyObject *o, at::ScalarType type, const char *name) {
    if (THPVariable_Check(o)) {
        const at::Tensor &t = THPVariable_Unpack(o);
        if (t.is_cuda() && t.scalar_type() == type && t.is_contiguous()) return &t;
    }
    PyErr_Format(PyExc_ValueError, "%s must be a contiguous CUDA tensor of dtype %s", name, dtype_text(type));
    return nullptr;
}
bool pointer_arg(PyObject *o, at::ScalarType type, const char *name, void **out) {
    const at::Tensor *t = tensor_arg(o, type, name);
    if (t == nullptr) return false;
    *out = t->data_ptr();
    return true;
}
bool optional_pointer_arg(PyObject *o, at::ScalarType type, const char *name, void **out) {
    *out = nullptr;
    return o == Py_None || pointer_arg(o, type, name, out);
}
// any tensor (its bytes are what counts) or None
bool optional_bytes_arg(PyObject *o, const char *name, void **out) {
    *out = nullptr;
    if (o == Py_None) return true;
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_ValueError, "%s must be a tensor", name);
        return false;
    }
    *out = THPVariable_Unpack(o).data_ptr();
    return true;
}
bool size_arg(PyObject *o, int64_t *out) {
    *out = PyLong_AsLongLong(o);
    return !(*out == -1 && PyErr_Occurred());
}
bool two_sizes(const at::Tensor &t, const char *name, int64_t *rows, int64_t *cols) {
    if (t.dim() != 2) {
        PyErr_Format(PyExc_ValueError, "%s must have two dimensions (has %d)", name, (int)t.dim());
        return false;
    }
    *rows = t.size(0);
    *cols = t.size(1);
    return true;
}
bool argument_count(Py_ssize_t n, Py_ssize_t want) {
    if (n == want) return true;
    PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, n);
    return false;
}

// The device of the call made current for its duration, and the stream that torch would use on it.
class OnDevice {
  public:
    explicit OnDevice(const at::Tensor &t) : want_(t.get_device()) {
        had_ = c10::cuda::current_device();
        if (had_ != want_) c10::cuda::set_device(want_);
    }
    ~OnDevice() {
        if (had_ != want_) (void)c10::cuda::SetDevice(had_);  // no exception from here: restore() has reported the error
    }
    void restore() {
        const c10::DeviceIndex back = had_;
        had_ = want_;
        if (back != want_) c10::cuda::set_device(back);
    }
    void *stream() const { return c10::cuda::getCurrentCUDAStream(want_).stream(); }

  private:
    c10::DeviceIndex want_, had_;
};

// Other Python threads run while this is in scope: no Python object and no tensor is touched meanwhile.
class WithoutGil {
  public:
    WithoutGil() : state_(PyEval_SaveThread()) {}
    ~WithoutGil() { PyEval_RestoreThread(state_); }

  private:
    PyThreadState *state_;
};

// Runs `call` (which returns a jq_status) and hands the status to Python.  A launch can wait: for room in the queue, for a
// kernel's module to be loaded on its first use.  So `call` has only plain values left to pass on, and runs without the GIL.
template <typename F>
PyObject *status_of(const at::Tensor &on, F &&call) {
    OnDevice device(on);
    void *const stream = device.stream();
    int status;
    {
        const WithoutGil released;
        status = call(stream);
    }
    device.restore();
    return PyLong_FromLong(status);
}

// What Python calls.  Almost everything of torch can throw, is_contiguous() and data_ptr() of a tensor without storage
// (under vmap, for instance) included, and no exception may leave a C function: each becomes the Python exception that
// torch's own functions raise for it.
template <PyObject *(*Call)(PyObject *const *, Py_ssize_t)>
PyObject *entry(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    return Call(a, n);
    END_HANDLE_TH_ERRORS
}

// ---- the calls: every one returns the library's status -------------------------------------------------
// (x, out, order, s_mode)
PyObject *quantize(PyObject *const *a, Py_ssize_t n) {
    int64_t M, K, order, s_mode;
    void *xp, *op;
    if (!argument_count(n, 4)) return nullptr;
    const at::Tensor *x = tensor_arg(a[0], at::kFloat, "x");
    if (x == nullptr || !two_sizes(*x, "x", &M, &K) || !pointer_arg(a[1], at::kByte, "out", &op) || !size_arg(a[2], &order) ||
        !size_arg(a[3], &s_mode))
        return nullptr;
    xp = x->data_ptr();
    return status_of(*x, [&](void *st) { return f_quantize(st, static_cast<const float *>(xp), op, K, M, (int)order, (int)s_mode); });
}

// (w, xq, out, K, N, M, order, kernel)
PyObject *mul_mat(PyObject *const *a, Py_ssize_t n) {
    int64_t K, N, M, order, kernel;
    void *xp, *yp;
    if (!argument_count(n, 8)) return nullptr;
    const at::Tensor *w = tensor_arg(a[0], at::kByte, "w");
    if (w == nullptr || !pointer_arg(a[1], at::kByte, "xq", &xp) || !pointer_arg(a[2], at::kFloat, "out", &yp) || !size_arg(a[3], &K) ||
        !size_arg(a[4], &N) || !size_arg(a[5], &M) || !size_arg(a[6], &order) || !size_arg(a[7], &kernel))
        return nullptr;
    const void *wp = w->data_ptr();
    return status_of(*w, [&](void *st) {
        return f_mul_mat(st, wp, xp, static_cast<float *>(yp), K, N, M, (int)order, (int)kernel);
    });
}

// (w, x, ws, out, N, s_mode)
PyObject *linear(PyObject *const *a, Py_ssize_t n) {
    int64_t K, N, M, s_mode;
    void *wp, *wsp, *yp;
    if (!argument_count(n, 6)) return nullptr;
    if (!pointer_arg(a[0], at::kByte, "w", &wp)) return nullptr;
    const at::Tensor *x = tensor_arg(a[1], at::kFloat, "x");
    if (x == nullptr || !two_sizes(*x, "x", &M, &K) || !pointer_arg(a[2], at::kByte, "ws", &wsp) ||
        !pointer_arg(a[3], at::kFloat, "out", &yp) || !size_arg(a[4], &N) || !size_arg(a[5], &s_mode))
        return nullptr;
    const void *xp = x->data_ptr();
    return status_of(*x, [&](void *st) {
        return f_linear(st, wp, static_cast<const float *>(xp), wsp, static_cast<float *>(yp), K, N, M, (int)s_mode);
    });
}

// (ws_list, N_list, outs, x or None, xq or None, ws or None, K, M, s_mode); the first three are sequences of one length
PyObject *multi(PyObject *const *a, Py_ssize_t n) {
    constexpr Py_ssize_t MOST = 16;  // the library says how many it takes; this only bounds the arrays here
    const void *w[MOST];
    float *y[MOST];
    int64_t rows[MOST];
    int64_t K, M, s_mode;
    void *xp, *xqp, *wsp;
    if (!argument_count(n, 9)) return nullptr;
    Owned seq[3];  // tuples of the call's own: converting a row count may run Python code that changes the caller's lists
    for (int i = 0; i < 3; ++i) {
        seq[i].p = PySequence_Tuple(a[i]);
        if (seq[i].p == nullptr) return nullptr;
    }
    const Py_ssize_t n_mats = PyTuple_GET_SIZE(seq[0].p);
    if (n_mats < 1 || n_mats > MOST || PyTuple_GET_SIZE(seq[1].p) != n_mats || PyTuple_GET_SIZE(seq[2].p) != n_mats) {
        PyErr_SetString(PyExc_ValueError, "weights, row counts and outputs must be sequences of one length (1 to 16)");
        return nullptr;
    }
    const at::Tensor *first = nullptr;
    for (Py_ssize_t i = 0; i < n_mats; ++i) {
        void *yp = nullptr;
        const at::Tensor *t = tensor_arg(PyTuple_GET_ITEM(seq[0].p, i), at::kByte, "w");
        if (t == nullptr || !pointer_arg(PyTuple_GET_ITEM(seq[2].p, i), at::kFloat, "out", &yp)) return nullptr;
        Owned r{PyNumber_Long(PyTuple_GET_ITEM(seq[1].p, i))};
        if (r.p == nullptr || !size_arg(r.p, &rows[i])) return nullptr;
        if (i == 0) first = t;
        w[i] = t->data_ptr();
        y[i] = static_cast<float *>(yp);
    }
    if (!optional_pointer_arg(a[3], at::kFloat, "x", &xp) || !optional_pointer_arg(a[4], at::kByte, "xq", &xqp) ||
        !optional_pointer_arg(a[5], at::kByte, "ws", &wsp) || !size_arg(a[6], &K) || !size_arg(a[7], &M) || !size_arg(a[8], &s_mode))
        return nullptr;
    return status_of(*first, [&](void *st) {
        return f_multi(st, (int)n_mats, w, rows, y, static_cast<const float *>(xp), xqp, wsp, K, M, (int)s_mode);
    });
}

// (x, weight, epsilon, residual or None, normed or None, xq or None, order, s_mode)
PyObject *rms_norm(PyObject *const *a, Py_ssize_t n) {
    int64_t T, H, order, s_mode;
    void *wp, *rp, *np, *qp;
    if (!argument_count(n, 8)) return nullptr;
    const at::Tensor *x = tensor_arg(a[0], at::kFloat, "x");
    if (x == nullptr || !two_sizes(*x, "x", &T, &H) || !pointer_arg(a[1], at::kFloat, "weight", &wp)) return nullptr;
    const double epsilon = PyFloat_AsDouble(a[2]);
    if (epsilon == -1.0 && PyErr_Occurred()) return nullptr;
    if (!optional_pointer_arg(a[3], at::kFloat, "residual", &rp) || !optional_pointer_arg(a[4], at::kFloat, "normed", &np) ||
        !optional_bytes_arg(a[5], "xq", &qp) || !size_arg(a[6], &order) || !size_arg(a[7], &s_mode))
        return nullptr;
    void *xp = x->data_ptr();
    return status_of(*x, [&](void *st) {
        return f_rms_norm(st, static_cast<float *>(xp), static_cast<float *>(rp), static_cast<const float *>(wp),
                          static_cast<float *>(np), qp, H, T, (float)epsilon, (int)order, (int)s_mode);
    });
}

// (gate, up, mid or None, xq or None, order, s_mode)
PyObject *swiglu(PyObject *const *a, Py_ssize_t n) {
    int64_t T, I, order, s_mode;
    void *up, *mp, *qp;
    if (!argument_count(n, 6)) return nullptr;
    const at::Tensor *g = tensor_arg(a[0], at::kFloat, "gate");
    if (g == nullptr || !two_sizes(*g, "gate", &T, &I) || !pointer_arg(a[1], at::kFloat, "up", &up) ||
        !optional_pointer_arg(a[2], at::kFloat, "mid", &mp) || !optional_bytes_arg(a[3], "xq", &qp) || !size_arg(a[4], &order) ||
        !size_arg(a[5], &s_mode))
        return nullptr;
    const void *gp = g->data_ptr();
    return status_of(*g, [&](void *st) {
        return f_swiglu(st, static_cast<const float *>(gp), static_cast<const float *>(up), static_cast<float *>(mp), qp, I, T,
                        (int)order, (int)s_mode);
    });
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&entry<f>)), METH_FASTCALL
PyMethodDef methods[] = {
    {"bind", bind, METH_O, "Addresses of the library's functions, by name."},
    {"quantize", FAST(quantize), "(x, out, order, s_mode) -> status"},
    {"mul_mat", FAST(mul_mat), "(w, xq, out, K, N, M, order, kernel) -> status"},
    {"linear", FAST(linear), "(w, x, ws, out, N, s_mode) -> status"},
    {"multi", FAST(multi), "(ws_list, N_list, outs, x, xq, ws, K, M, s_mode) -> status"},
    {"rms_norm", FAST(rms_norm), "(x, weight, epsilon, residual, normed, xq, order, s_mode) -> status"},
    {"swiglu", FAST(swiglu), "(gate, up, mid, xq, order, s_mode) -> status"},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_calls", "Native part of capi.py's tensor calls.", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__torch_calls(void) { return PyModule_Create(&module); }
