/* Native half of the Python front end: the calls a program makes per step, without ctypes.
 *
 * DeviceBase and ModelBase hold the library handles and implement the hot methods of Device and
 * Model as functions of this extension: they read pointers, shapes and strides off the tensors, allocate the
 * output, and call the C ABI through function pointers taken from the loaded library (bind()).
 * A ctypes call of ag_gemm with its twenty converted arguments, torch.cuda.current_stream and the
 * surrounding Python cost 13 us; the same call here about 4 us, most of it the kernel launch.
 * Tensors are read and made through torch's C++ interface: through its Python objects (attributes, tuples of
 * ints, torch.empty) a convolution, pool or bias gradient took the host 6.4 to 7.0 us a call, now 4.4 to 4.8.
 *
 * Anything but the plain case -- other argument types, views that need a copy, shapes that do not
 * match, another current stream, a torch mode that wants to see operations (a default device does not: outputs have
 * theirs), output guards switched on -- goes to the Python implementation of the method (set_fallback()), which also
 * raises the errors. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <structmember.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/PyInterpreter.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/autograph_b200.h"

/* ------------------------------------------------------------------ library and torch objects */
#define FUNCTIONS(X)                                                                               \
    X(ag_gemm) X(ag_dense_forward) X(ag_conv2_forward) X(ag_conv2_backward_input)                  \
    X(ag_conv2_backward_weight) X(ag_conv2_output_shape) X(ag_max_pool2)                           \
    X(ag_max_pool2_backward_from_input) X(ag_relu) X(ag_relu_backward) X(ag_bias_add)              \
    X(ag_bias_grad) X(ag_model_infer) X(ag_model_infer_u8) X(ag_model_forward_device)              \
    X(ag_model_train_step) X(ag_model_train_forward_backward) X(ag_model_apply_update)

#define DECLARE(name) static __typeof__(&name) p_##name;
FUNCTIONS(DECLARE)
#undef DECLARE

static PyObject *py_check, *device_context;

enum Method {
    M_DOT, M_GEMM, M_DENSE, M_CONV_FWD, M_CONV_DX, M_CONV_DW, M_POOL, M_POOL_BWD, M_RELU, M_RELU_BWD,
    M_BIAS_ADD, M_BIAS_GRAD, M_INFER, M_INFER_U8, M_FORWARD, M_TRAIN, M_TRAIN_FB, M_UPDATE, M_COUNT
};
static const char *method_names[M_COUNT] = {
    "dot", "gemm", "dense_forward", "conv2_forward", "conv2_backward_input", "conv2_backward_weight",
    "max_pool2", "max_pool2_backward_from_input", "relu", "relu_backward", "bias_add", "bias_grad",
    "infer", "infer_u8", "forward_device", "train_step", "train_forward_backward", "apply_update"};
static PyObject *fallbacks[M_COUNT];

typedef struct {
    PyObject_HEAD
    ag_device *h;
    uintptr_t stream;
    int index;
    int guarded;
} DeviceObject;

typedef struct {
    PyObject_HEAD
    ag_model *h;
    int dtype, index;
    int64_t out_features;
} ModelObject;

static PyObject *fall_back(enum Method m, PyObject *self, PyObject *const *args, Py_ssize_t nargs,
                           PyObject *kwnames) {
    if (PyErr_Occurred()) PyErr_Clear();
    if (fallbacks[m] == NULL) {
        PyErr_SetString(PyExc_RuntimeError, "the front end is not bound");
        return NULL;
    }
    const Py_ssize_t nkw = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
    PyObject *stack[64];
    if (nargs + nkw + 1 > 64) {
        PyErr_SetString(PyExc_TypeError, "too many arguments");
        return NULL;
    }
    stack[0] = self;
    for (Py_ssize_t i = 0; i < nargs + nkw; ++i) stack[i + 1] = args[i];
    return PyObject_Vectorcall(fallbacks[m], stack, (size_t)(nargs + 1), kwnames);
}

/* Arguments by position or name; 0 when the call does not have the plain form. */
static int parse(PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames, const char *const *names,
                 int n, int required, PyObject **out) {
    if (nargs > n) return 0;
    for (int i = 0; i < n; ++i) out[i] = i < nargs ? args[i] : NULL;
    const Py_ssize_t nkw = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
    for (Py_ssize_t j = 0; j < nkw; ++j) {
        int found = -1;
        for (int i = (int)nargs; i < n && found < 0; ++i)
            if (PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(kwnames, j), names[i]) == 0) found = i;
        if (found < 0 || out[found] != NULL) return 0;
        out[found] = args[nargs + j];
    }
    for (int i = 0; i < required; ++i)
        if (out[i] == NULL) return 0;
    return 1;
}

typedef struct {
    void *p;
    int64_t shape[4], stride[2];
    int ndim, dtype;
} View;

static int tuple_ints(PyObject *t, int64_t *out, int most) {
    if (!PyTuple_Check(t)) return -1;
    const Py_ssize_t n = PyTuple_GET_SIZE(t);
    if (n > most) return -1;
    for (Py_ssize_t i = 0; i < n; ++i) {
        out[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(t, i));
        if (out[i] == -1 && PyErr_Occurred()) return -1;
    }
    return (int)n;
}

/* Whether a torch mode wants to see operations.  torch.set_default_device and `with torch.device(...)` are modes too, of
 * a class that only adds a device where none is given. */
static int watched(void) {
    if (c10::impl::dispatch_mode_enabled()) return 1;
    if (!at::impl::torch_function_mode_enabled()) return 0;
    const int64_t n = at::impl::PythonTorchFunctionTLS::stack_len();
    for (int64_t i = 0; i < n; ++i) {
        PyObject *mode = at::impl::PythonTorchFunctionTLS::get_stack_at(i)->ptr(getPyInterpreter());
        if ((PyObject *)Py_TYPE(mode) != device_context) return 1;
    }
    return 0;
}

/* Reads a tensor of `ndim` dimensions (0: any up to 4) on the GPU `index`, or in host memory for index -1: its
 * address goes to a kernel or a copy as it is.  Strides only when asked for, otherwise the tensor must be
 * contiguous. */
static int view_of(PyObject *o, int ndim, int with_strides, int index, View *v) {
    if (o == NULL || !THPVariable_CheckExact(o)) return 0;
    if (watched()) return 0;
    const at::Tensor &t = THPVariable_Unpack(o);
    const c10::TensorImpl *impl = t.unsafeGetTensorImpl();
    if (impl->layout() != c10::kStrided || impl->has_symbolic_sizes_strides() || !impl->has_storage()) return 0;
    try {
        switch (t.scalar_type()) {
            case at::kFloat: v->dtype = AG_F32; break;
            case at::kBFloat16: v->dtype = AG_BF16; break;
            case at::kByte: v->dtype = AG_U8; break;
            default: return 0;
        }
        v->ndim = (int)t.dim();
        if (v->ndim > 4 || (ndim && v->ndim != ndim)) return 0;
        for (int i = 0; i < v->ndim; ++i) v->shape[i] = t.size(i);
        if (with_strides) {
            if (v->ndim > 2) return 0;
            for (int i = 0; i < v->ndim; ++i) v->stride[i] = t.stride(i);
        } else if (!t.is_contiguous()) {
            return 0;
        }
        const c10::Device device = t.device();
        if (index != (device.is_cpu() ? -1 : device.is_cuda() ? device.index() : -2)) return 0;
        v->p = t.data_ptr();   /* throws where there is no pointer to give (wrappers of function transforms) */
    } catch (const std::exception &) {
        return 0;
    }
    return 1;
}

static int64_t count_of(const View *v) {
    int64_t n = 1;
    for (int i = 0; i < v->ndim; ++i) n *= v->shape[i];
    return n;
}

/* The plain case of a device call: no guards, and the device's own stream is torch's current one. */
static int plain(DeviceObject *d) {
    if (d->guarded || d->h == NULL) return 0;
    try {
        return (uintptr_t)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)d->index).stream() == d->stream;
    } catch (const std::exception &) {
        return 0;
    }
}

static PyObject *new_tensor(DeviceObject *d, int dtype, int ndim, const int64_t *shape, void **p) {
    HANDLE_TH_ERRORS
    at::Tensor t;
    {
        pybind11::gil_scoped_release no_gil;
        t = at::empty(at::IntArrayRef(shape, (size_t)ndim),
                      at::TensorOptions(dtype == AG_F32 ? at::kFloat : at::kBFloat16)
                          .device(c10::Device(c10::kCUDA, (c10::DeviceIndex)d->index)));
        *p = t.data_ptr();
    }
    return THPVariable_Wrap(std::move(t));
    END_HANDLE_TH_ERRORS
}

/* `result` (a new reference) when status is AG_OK, else the library's error raised by Python. */
static PyObject *finish(int status, PyObject *result) {
    if (status == AG_OK) return result;
    Py_XDECREF(result);
    PyObject *r = PyObject_CallFunction(py_check, "i", status);
    Py_XDECREF(r);
    return NULL;
}

#define CALL(status, expr)        \
    do {                          \
        Py_BEGIN_ALLOW_THREADS    \
        status = (expr);          \
        Py_END_ALLOW_THREADS      \
    } while (0)

static int pair_of(PyObject *o, int32_t *out, int def) {
    if (o == NULL) {
        out[0] = out[1] = def;
        return 1;
    }
    int64_t v[2];
    if (tuple_ints(o, v, 2) != 2) return 0;
    out[0] = (int32_t)v[0];
    out[1] = (int32_t)v[1];
    return 1;
}

static int flag_of(PyObject *o, int *out) {
    if (o == NULL) {
        *out = 0;
        return 1;
    }
    *out = o == Py_True;
    return o == Py_True || o == Py_False;
}

static int float_of(PyObject *o, double def, float *out) {
    if (o == NULL) {
        *out = (float)def;
        return 1;
    }
    if (!PyFloat_Check(o) && !PyLong_Check(o)) return 0;
    *out = (float)PyFloat_AsDouble(o);
    return !PyErr_Occurred();
}

static int options_of(PyObject *padding, PyObject *stride, PyObject *dilation, int64_t fh, int64_t fw,
                      ag_conv2_options *o) {
    o->filter[0] = (int32_t)fh;
    o->filter[1] = (int32_t)fw;
    return pair_of(padding, o->padding, 0) && pair_of(stride, o->stride, 1) && pair_of(dilation, o->dilation, 1);
}

/* bias: None or a contiguous vector */
static int bias_of(PyObject *o, int index, const void **p) {
    *p = NULL;
    if (o == NULL || o == Py_None) return 1;
    View v;
    if (!view_of(o, 1, 0, index, &v)) return 0;
    *p = v.p;
    return 1;
}

/* --------------------------------------------------------------------------------- Device */
#define ENTRY(name) static PyObject *name(PyObject *self, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames)
#define FALL_BACK(m) return fall_back(m, self, args, nargs, kwnames)

static int run_gemm(DeviceObject *d, float alpha, const View *a, const View *b, float beta, void *c,
                    int64_t rs, int64_t cs) {
    int st;
    CALL(st, p_ag_gemm(d->h, (ag_dtype)a->dtype, a->shape[0], a->shape[1], b->shape[1], alpha, a->p, 0,
                       a->stride[0], a->stride[1], b->p, 0, b->stride[0], b->stride[1], beta, c, 0, rs, cs));
    return st;
}

ENTRY(dot) {
    static const char *const names[] = {"a", "b"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[2];
    View a, b;
    if (!parse(args, nargs, kwnames, names, 2, 2, o) || !plain(d) || !view_of(o[0], 2, 1, d->index, &a) ||
        !view_of(o[1], 2, 1, d->index, &b) || a.dtype != b.dtype || a.dtype == AG_U8 || a.shape[1] != b.shape[0])
        FALL_BACK(M_DOT);
    void *c;
    const int64_t shape[2] = {a.shape[0], b.shape[1]};
    PyObject *out = new_tensor(d, a.dtype, 2, shape, &c);
    if (out == NULL) return NULL;
    return finish(run_gemm(d, 1.f, &a, &b, 0.f, c, shape[1] > 1 ? shape[1] : 1, 1), out);
}

ENTRY(gemm) {
    static const char *const names[] = {"alpha", "a", "b", "beta", "c"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[5];
    View a, b, c;
    float alpha, beta;
    if (!parse(args, nargs, kwnames, names, 5, 5, o) || !plain(d) || !float_of(o[0], 0, &alpha) ||
        !float_of(o[3], 0, &beta) || !view_of(o[1], 2, 1, d->index, &a) || !view_of(o[2], 2, 1, d->index, &b) ||
        !view_of(o[4], 2, 1, d->index, &c) || a.dtype != b.dtype || a.dtype != c.dtype || a.dtype == AG_U8 ||
        a.shape[1] != b.shape[0] || a.shape[0] != c.shape[0] || b.shape[1] != c.shape[1])
        FALL_BACK(M_GEMM);
    return finish(run_gemm(d, alpha, &a, &b, beta, c.p, c.stride[0], c.stride[1]), Py_NewRef(o[4]));
}

ENTRY(dense_forward) {
    static const char *const names[] = {"x", "w", "bias", "relu"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[4];
    View x, w;
    const void *bias;
    int relu, st;
    if (!parse(args, nargs, kwnames, names, 4, 2, o) || !plain(d) || !view_of(o[0], 2, 0, d->index, &x) ||
        !view_of(o[1], 2, 0, d->index, &w) || x.dtype != w.dtype || x.dtype == AG_U8 || x.shape[1] != w.shape[0] ||
        !bias_of(o[2], d->index, &bias) || !flag_of(o[3], &relu))
        FALL_BACK(M_DENSE);
    void *y;
    const int64_t shape[2] = {x.shape[0], w.shape[1]};
    PyObject *out = new_tensor(d, x.dtype, 2, shape, &y);
    if (out == NULL) return NULL;
    CALL(st, p_ag_dense_forward(d->h, (ag_dtype)x.dtype, x.p, x.shape[0], x.shape[1], w.p, w.shape[1], bias,
                                relu, y));
    return finish(st, out);
}

ENTRY(conv2_forward) {
    static const char *const names[] = {"x", "w", "bias", "padding", "stride", "dilation", "relu"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[7];
    View x, w;
    const void *bias;
    ag_conv2_options opt;
    int relu, st;
    int64_t oh, ow;
    if (!parse(args, nargs, kwnames, names, 7, 2, o) || !plain(d) || !view_of(o[0], 4, 0, d->index, &x) ||
        !view_of(o[1], 4, 0, d->index, &w) || x.dtype == AG_U8 || x.dtype != w.dtype || x.shape[1] != w.shape[1] ||
        !bias_of(o[2], d->index, &bias) || !options_of(o[3], o[4], o[5], w.shape[2], w.shape[3], &opt) ||
        !flag_of(o[6], &relu) || p_ag_conv2_output_shape(x.shape[2], x.shape[3], &opt, &oh, &ow) != AG_OK)
        FALL_BACK(M_CONV_FWD);
    void *y;
    const int64_t shape[4] = {x.shape[0], w.shape[0], oh, ow};
    PyObject *out = new_tensor(d, x.dtype, 4, shape, &y);
    if (out == NULL) return NULL;
    CALL(st, p_ag_conv2_forward(d->h, (ag_dtype)x.dtype, x.p, x.shape[0], x.shape[1], x.shape[2], x.shape[3],
                                w.p, w.shape[0], bias, &opt, relu, y));
    return finish(st, out);
}

ENTRY(conv2_backward_input) {
    static const char *const names[] = {"w", "dy", "input_hw", "padding", "stride", "dilation"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[6];
    View w, dy;
    ag_conv2_options opt;
    int st;
    int32_t hw[2];
    if (!parse(args, nargs, kwnames, names, 6, 3, o) || !plain(d) || !view_of(o[0], 4, 0, d->index, &w) ||
        !view_of(o[1], 4, 0, d->index, &dy) || dy.dtype == AG_U8 || dy.dtype != w.dtype || !pair_of(o[2], hw, 0) ||
        !options_of(o[3], o[4], o[5], w.shape[2], w.shape[3], &opt))
        FALL_BACK(M_CONV_DX);
    void *dx;
    const int64_t shape[4] = {dy.shape[0], w.shape[1], hw[0], hw[1]};
    PyObject *out = new_tensor(d, dy.dtype, 4, shape, &dx);
    if (out == NULL) return NULL;
    CALL(st, p_ag_conv2_backward_input(d->h, (ag_dtype)dy.dtype, w.p, w.shape[0], w.shape[1], dy.p,
                                       dy.shape[0], hw[0], hw[1], &opt, dx));
    return finish(st, out);
}

ENTRY(conv2_backward_weight) {
    static const char *const names[] = {"x", "dy", "filter", "padding", "stride", "dilation", "beta", "dw"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[8];
    View x, dy, w;
    ag_conv2_options opt;
    int st;
    int32_t f[2];
    float beta;
    if (!parse(args, nargs, kwnames, names, 8, 3, o) || !plain(d) || !view_of(o[0], 4, 0, d->index, &x) ||
        !view_of(o[1], 4, 0, d->index, &dy) || x.dtype == AG_U8 || x.dtype != dy.dtype || !pair_of(o[2], f, 0) ||
        !options_of(o[3], o[4], o[5], f[0], f[1], &opt) || !float_of(o[6], 0, &beta))
        FALL_BACK(M_CONV_DW);
    PyObject *out;
    if (o[7] == NULL || o[7] == Py_None) {
        const int64_t shape[4] = {dy.shape[1], x.shape[1], f[0], f[1]};
        out = new_tensor(d, x.dtype, 4, shape, &w.p);
        if (out == NULL) return NULL;
    } else {
        if (!view_of(o[7], 4, 0, d->index, &w) || w.dtype != x.dtype) FALL_BACK(M_CONV_DW);
        out = Py_NewRef(o[7]);
    }
    CALL(st, p_ag_conv2_backward_weight(d->h, (ag_dtype)x.dtype, x.p, x.shape[0], x.shape[1], x.shape[2],
                                        x.shape[3], dy.p, dy.shape[1], &opt, beta, w.p));
    return finish(st, out);
}

/* window and strides of a pool (strides default to the window); 0 when it does not fit */
static int pool_of(PyObject *size, PyObject *strides, const View *x, int32_t *h, int32_t *s) {
    if (!pair_of(size, h, 2)) return 0;
    if (strides == NULL || strides == Py_None) {
        s[0] = h[0];
        s[1] = h[1];
    } else if (!pair_of(strides, s, 0)) {
        return 0;
    }
    return h[0] > 0 && h[1] > 0 && s[0] > 0 && s[1] > 0 && x->shape[2] >= h[0] && x->shape[3] >= h[1];
}

ENTRY(max_pool2) {
    static const char *const names[] = {"x", "size", "strides"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[3];
    View x;
    int32_t h[2], s[2];
    int st;
    if (!parse(args, nargs, kwnames, names, 3, 1, o) || !plain(d) || !view_of(o[0], 4, 0, d->index, &x) ||
        x.dtype == AG_U8 || !pool_of(o[1], o[2], &x, h, s))
        FALL_BACK(M_POOL);
    void *y;
    const int64_t shape[4] = {x.shape[0], x.shape[1], (x.shape[2] - h[0]) / s[0] + 1,
                              (x.shape[3] - h[1]) / s[1] + 1};
    PyObject *out = new_tensor(d, x.dtype, 4, shape, &y);
    if (out == NULL) return NULL;
    CALL(st, p_ag_max_pool2(d->h, (ag_dtype)x.dtype, x.p, x.shape[0], x.shape[1], x.shape[2], x.shape[3], h[0],
                            h[1], s[0], s[1], y));
    return finish(st, out);
}

ENTRY(max_pool2_backward_from_input) {
    static const char *const names[] = {"x", "dy", "size", "strides"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[4];
    View x, dy;
    int32_t h[2], s[2];
    int st;
    if (!parse(args, nargs, kwnames, names, 4, 2, o) || !plain(d) || !view_of(o[0], 4, 0, d->index, &x) ||
        !view_of(o[1], 4, 0, d->index, &dy) || x.dtype == AG_U8 || x.dtype != dy.dtype || !pool_of(o[2], o[3], &x, h, s))
        FALL_BACK(M_POOL_BWD);
    void *dx;
    PyObject *out = new_tensor(d, x.dtype, 4, x.shape, &dx);
    if (out == NULL) return NULL;
    CALL(st, p_ag_max_pool2_backward_from_input(d->h, (ag_dtype)x.dtype, x.p, x.shape[0], x.shape[1],
                                                x.shape[2], x.shape[3], h[0], h[1], s[0], s[1], dy.p, dx));
    return finish(st, out);
}

ENTRY(relu) {
    static const char *const names[] = {"x", "inplace"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[2];
    View x;
    int inplace, st;
    if (!parse(args, nargs, kwnames, names, 2, 1, o) || !plain(d) || !view_of(o[0], 0, 0, d->index, &x) ||
        x.dtype == AG_U8 || !flag_of(o[1], &inplace))
        FALL_BACK(M_RELU);
    void *y = x.p;
    PyObject *out = inplace ? Py_NewRef(o[0]) : new_tensor(d, x.dtype, x.ndim, x.shape, &y);
    if (out == NULL) return NULL;
    CALL(st, p_ag_relu(d->h, (ag_dtype)x.dtype, x.p, y, count_of(&x)));
    return finish(st, out);
}

ENTRY(relu_backward) {
    static const char *const names[] = {"x", "dy", "inplace"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[3];
    View x, dy;
    int inplace, st;
    if (!parse(args, nargs, kwnames, names, 3, 2, o) || !plain(d) || !view_of(o[0], 0, 0, d->index, &x) ||
        !view_of(o[1], 0, 0, d->index, &dy) || x.dtype == AG_U8 || x.dtype != dy.dtype || count_of(&x) != count_of(&dy) ||
        !flag_of(o[2], &inplace))
        FALL_BACK(M_RELU_BWD);
    void *dx = dy.p;
    PyObject *out = inplace ? Py_NewRef(o[1]) : new_tensor(d, dy.dtype, dy.ndim, dy.shape, &dx);
    if (out == NULL) return NULL;
    CALL(st, p_ag_relu_backward(d->h, (ag_dtype)x.dtype, x.p, dy.p, dx, count_of(&x)));
    return finish(st, out);
}

static int rows_cols_inner(const View *v, int64_t *inner) {
    if (v->ndim < 2) return 0;
    *inner = 1;
    for (int i = 2; i < v->ndim; ++i) *inner *= v->shape[i];
    return *inner > 0 && v->shape[0] > 0 && v->shape[1] > 0;
}

ENTRY(bias_add) {
    static const char *const names[] = {"y", "bias"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[2];
    View y, b;
    int64_t inner;
    int st;
    if (!parse(args, nargs, kwnames, names, 2, 2, o) || !plain(d) || !view_of(o[0], 0, 0, d->index, &y) ||
        !view_of(o[1], 1, 0, d->index, &b) || y.dtype == AG_U8 || y.dtype != b.dtype || !rows_cols_inner(&y, &inner))
        FALL_BACK(M_BIAS_ADD);
    CALL(st, p_ag_bias_add(d->h, (ag_dtype)y.dtype, y.p, b.p, y.shape[0], y.shape[1], inner));
    return finish(st, Py_NewRef(o[0]));
}

ENTRY(bias_grad) {
    static const char *const names[] = {"dy", "beta", "out"};
    DeviceObject *d = (DeviceObject *)self;
    PyObject *o[3];
    View dy, b;
    int64_t inner;
    float beta;
    int st;
    if (!parse(args, nargs, kwnames, names, 3, 1, o) || !plain(d) || !view_of(o[0], 0, 0, d->index, &dy) ||
        dy.dtype == AG_U8 || !float_of(o[1], 0, &beta) || !rows_cols_inner(&dy, &inner))
        FALL_BACK(M_BIAS_GRAD);
    PyObject *out;
    if (o[2] == NULL || o[2] == Py_None) {
        out = new_tensor(d, dy.dtype, 1, &dy.shape[1], &b.p);
        if (out == NULL) return NULL;
    } else {
        if (!view_of(o[2], 1, 0, d->index, &b) || b.dtype != dy.dtype) FALL_BACK(M_BIAS_GRAD);
        out = Py_NewRef(o[2]);
    }
    CALL(st, p_ag_bias_grad(d->h, (ag_dtype)dy.dtype, dy.p, dy.shape[0], dy.shape[1], inner, beta, b.p));
    return finish(st, out);
}

/* _bind(handle, stream, index): handle 0 when the device is closed */
static PyObject *device_bind(PyObject *self, PyObject *args) {
    DeviceObject *d = (DeviceObject *)self;
    unsigned long long h, stream;
    int index;
    if (!PyArg_ParseTuple(args, "KKi", &h, &stream, &index)) return NULL;
    d->h = (ag_device *)(uintptr_t)h;
    d->stream = (uintptr_t)stream;
    d->index = index;
    Py_RETURN_NONE;
}

static PyObject *device_guarded(PyObject *self, PyObject *on) {
    ((DeviceObject *)self)->guarded = PyObject_IsTrue(on);
    Py_RETURN_NONE;
}

#define FAST(fn) {#fn, (PyCFunction)(void (*)(void))fn, METH_FASTCALL | METH_KEYWORDS, NULL}
static PyMethodDef device_methods[] = {
    FAST(dot), FAST(gemm), FAST(dense_forward), FAST(conv2_forward), FAST(conv2_backward_input),
    FAST(conv2_backward_weight), FAST(max_pool2), FAST(max_pool2_backward_from_input), FAST(relu),
    FAST(relu_backward), FAST(bias_add), FAST(bias_grad),
    {"_bind", device_bind, METH_VARARGS, NULL},
    {"_set_guarded", device_guarded, METH_O, NULL},
    {NULL, NULL, 0, NULL}};

static PyTypeObject DeviceType = {PyVarObject_HEAD_INIT(NULL, 0)};

/* ---------------------------------------------------------------------------------- Model */
/* A batch [bs, c, h, w] (or a vector / matrix) of the given type on the GPU `index`, or in host
 * memory for index -1. */
static int batch_of(PyObject *t, int ndim, int dtype, int index, View *v) {
    return view_of(t, ndim, 0, index, v) && v->dtype == dtype;
}

/* logits: given, or a new tensor; NULL without an exception when the given one does not fit */
static PyObject *logits_of(ModelObject *m, PyObject *given, int64_t bs, int index, View *out) {
    if (given == NULL || given == Py_None) return NULL;
    if (!batch_of(given, 2, m->dtype, index, out) || out->shape[0] != bs || out->shape[1] != m->out_features)
        return NULL;
    return Py_NewRef(given);
}

ENTRY(infer) {
    static const char *const names[] = {"x_host", "out_host"};
    ModelObject *m = (ModelObject *)self;
    PyObject *o[2], *out;
    View x, y;
    int st;
    if (m->h == NULL || !parse(args, nargs, kwnames, names, 2, 2, o) || !batch_of(o[0], 4, m->dtype, -1, &x) ||
        (out = logits_of(m, o[1], x.shape[0], -1, &y)) == NULL)
        FALL_BACK(M_INFER);
    CALL(st, p_ag_model_infer(m->h, x.p, x.shape[0], x.shape[1], x.shape[2], x.shape[3], y.p));
    return finish(st, out);
}

ENTRY(infer_u8) {
    static const char *const names[] = {"x_host_u8", "alpha", "out_host"};
    ModelObject *m = (ModelObject *)self;
    PyObject *o[3], *out;
    View x, y;
    float alpha;
    int st;
    if (m->h == NULL || !parse(args, nargs, kwnames, names, 3, 1, o) || !float_of(o[1], 1.0 / 255.0, &alpha) ||
        !batch_of(o[0], 4, AG_U8, -1, &x) || (out = logits_of(m, o[2], x.shape[0], -1, &y)) == NULL)
        FALL_BACK(M_INFER_U8);
    CALL(st, p_ag_model_infer_u8(m->h, (const uint8_t *)x.p, x.shape[0], x.shape[1], x.shape[2], x.shape[3], alpha, y.p));
    return finish(st, out);
}

ENTRY(forward_device) {
    static const char *const names[] = {"x_dev", "out_dev"};
    ModelObject *m = (ModelObject *)self;
    PyObject *o[2], *out;
    View x, y;
    int st;
    if (m->h == NULL || !parse(args, nargs, kwnames, names, 2, 2, o) ||
        !batch_of(o[0], 4, m->dtype, m->index, &x) ||
        (out = logits_of(m, o[1], x.shape[0], m->index, &y)) == NULL)
        FALL_BACK(M_FORWARD);
    CALL(st, p_ag_model_forward_device(m->h, x.p, x.shape[0], x.shape[1], x.shape[2], x.shape[3], y.p));
    return finish(st, out);
}

ENTRY(train_step) {
    static const char *const names[] = {"x_host", "t_host", "lr"};
    ModelObject *m = (ModelObject *)self;
    PyObject *o[3];
    View x, t;
    float lr, loss = 0.f;
    int st;
    if (m->h == NULL || !parse(args, nargs, kwnames, names, 3, 3, o) || !float_of(o[2], 0, &lr) ||
        !batch_of(o[0], 4, m->dtype, -1, &x) || !batch_of(o[1], 1, AG_U8, -1, &t) || t.shape[0] != x.shape[0])
        FALL_BACK(M_TRAIN);
    CALL(st, p_ag_model_train_step(m->h, x.p, (const uint8_t *)t.p, x.shape[0], x.shape[1], x.shape[2],
                                   x.shape[3], lr, &loss));
    return finish(st, PyFloat_FromDouble(loss));
}

ENTRY(train_forward_backward) {
    static const char *const names[] = {"x_dev", "t_dev", "sync"};
    ModelObject *m = (ModelObject *)self;
    PyObject *o[3];
    View x, t;
    float loss = 0.f;
    void *bucket = NULL;
    int64_t length = 0;
    int st;
    if (m->h == NULL || !parse(args, nargs, kwnames, names, 3, 2, o) ||
        (o[2] != NULL && o[2] != Py_True && o[2] != Py_False) || !batch_of(o[0], 4, m->dtype, m->index, &x) ||
        !batch_of(o[1], 1, AG_U8, m->index, &t) || t.shape[0] != x.shape[0])
        FALL_BACK(M_TRAIN_FB);
    const int sync = o[2] != Py_False;
    CALL(st, p_ag_model_train_forward_backward(m->h, x.p, (const uint8_t *)t.p, x.shape[0], x.shape[1],
                                               x.shape[2], x.shape[3], sync ? &loss : NULL, &bucket, &length));
    if (st != AG_OK) return finish(st, NULL);
    return Py_BuildValue("(NKL)", sync ? PyFloat_FromDouble(loss) : Py_NewRef(Py_None),
                         (unsigned long long)(uintptr_t)bucket, (long long)length);
}

ENTRY(apply_update) {
    static const char *const names[] = {"lr"};
    ModelObject *m = (ModelObject *)self;
    PyObject *o[1];
    float lr;
    int st;
    if (m->h == NULL || !parse(args, nargs, kwnames, names, 1, 1, o) || !float_of(o[0], 0, &lr))
        FALL_BACK(M_UPDATE);
    CALL(st, p_ag_model_apply_update(m->h, lr));
    return finish(st, Py_NewRef(Py_None));
}

/* _bind(handle, dtype code, device index, out_features): handle 0 when the model is closed */
static PyObject *model_bind(PyObject *self, PyObject *args) {
    ModelObject *m = (ModelObject *)self;
    unsigned long long h;
    long long out;
    if (!PyArg_ParseTuple(args, "KiiL", &h, &m->dtype, &m->index, &out)) return NULL;
    m->h = (ag_model *)(uintptr_t)h;
    m->out_features = out;
    Py_RETURN_NONE;
}

static PyMethodDef model_methods[] = {
    FAST(infer), FAST(infer_u8), FAST(forward_device), FAST(train_step), FAST(train_forward_backward),
    FAST(apply_update),
    {"_bind", model_bind, METH_VARARGS, NULL},
    {NULL, NULL, 0, NULL}};

static PyTypeObject ModelType = {PyVarObject_HEAD_INIT(NULL, 0)};

/* --------------------------------------------------------------------------------- module */
/* bind({name: address}, check): once, before the first device */
static PyObject *bind(PyObject *mod, PyObject *args) {
    (void)mod;
    PyObject *fns, *check;
    if (!PyArg_ParseTuple(args, "OO", &fns, &check)) return NULL;
#define TAKE(name)                                                              \
    {                                                                           \
        PyObject *v = PyDict_GetItemString(fns, #name);                         \
        void *p = v ? PyLong_AsVoidPtr(v) : NULL;                               \
        if (p == NULL) {                                                        \
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_KeyError, #name);      \
            return NULL;                                                        \
        }                                                                       \
        p_##name = (__typeof__(p_##name))p;                                     \
    }
    FUNCTIONS(TAKE)
#undef TAKE
    py_check = Py_NewRef(check);
    PyObject *modes = PyImport_ImportModule("torch.utils._device");
    device_context = modes ? PyObject_GetAttrString(modes, "DeviceContext") : NULL;
    Py_XDECREF(modes);
    PyErr_Clear();   /* without it every mode is one that watches */
    Py_RETURN_NONE;
}

/* set_fallback(name, function): the Python implementation of a method */
static PyObject *set_fallback(PyObject *mod, PyObject *args) {
    (void)mod;
    const char *name;
    PyObject *fn;
    if (!PyArg_ParseTuple(args, "sO", &name, &fn)) return NULL;
    for (int i = 0; i < M_COUNT; ++i)
        if (strcmp(name, method_names[i]) == 0) {
            Py_XSETREF(fallbacks[i], Py_NewRef(fn));
            Py_RETURN_NONE;
        }
    PyErr_SetString(PyExc_KeyError, name);
    return NULL;
}

static PyMethodDef module_methods[] = {{"bind", bind, METH_VARARGS, NULL},
                                       {"set_fallback", set_fallback, METH_VARARGS, NULL},
                                       {NULL, NULL, 0, NULL}};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_front", NULL, -1, module_methods,
                                    NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__front(void) {
    const auto type = [](PyTypeObject &t, const char *name, size_t size, PyMethodDef *methods) {
        t.tp_name = name;
        t.tp_basicsize = (Py_ssize_t)size;
        t.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE;
        t.tp_methods = methods;
        t.tp_new = PyType_GenericNew;
    };
    type(DeviceType, "autograph_b200._front.DeviceBase", sizeof(DeviceObject), device_methods);
    type(ModelType, "autograph_b200._front.ModelBase", sizeof(ModelObject), model_methods);
    if (PyType_Ready(&DeviceType) < 0 || PyType_Ready(&ModelType) < 0) return NULL;
    PyObject *m = PyModule_Create(&module);
    if (m == NULL) return NULL;
    PyObject *names = PyList_New(0);
    for (int i = 0; i < M_COUNT; ++i) {
        PyObject *s = PyUnicode_FromString(method_names[i]);
        PyList_Append(names, s);
        Py_DECREF(s);
    }
    PyObject *fns = PyList_New(0);
#define NAME(name)                                 \
    {                                              \
        PyObject *s = PyUnicode_FromString(#name); \
        PyList_Append(fns, s);                     \
        Py_DECREF(s);                              \
    }
    FUNCTIONS(NAME)
#undef NAME
    PyModule_AddObject(m, "METHODS", names);
    PyModule_AddObject(m, "FUNCTIONS", fns);
    PyModule_AddObjectRef(m, "DeviceBase", (PyObject *)&DeviceType);
    PyModule_AddObjectRef(m, "ModelBase", (PyObject *)&ModelType);
    return m;
}
