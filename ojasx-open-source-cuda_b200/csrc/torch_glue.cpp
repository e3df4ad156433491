// The hot entry points as a CPython extension module on torch tensors: checks, output and scratch allocation, stream
// look-up and the C ABI call of one operation in one native call.
//
// A decode-shape linear takes a few microseconds on the GPU; the same steps through Python and ctypes took ~30 us per
// call, so they bounded every small call (one row of 4096 -> 1024: 36 us a pass, 6.6 us of it on the GPU).
//
// A function returns None when the call is not of the plain form it handles (another device or dtype, non-contiguous
// operands, tensor subclasses that dispatch in Python, ...): ops.py then runs its general path, which converts or raises.
// A negative int is a status of the C ABI, 1 a pending failure of an earlier launch.
#define PY_SSIZE_T_CLEAN
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include "../../include/ojx_e8t.h"

namespace {

int dtype_code(at::ScalarType t) {
    return t == at::kBFloat16 ? OJX_BF16 : (t == at::kHalf ? OJX_F16 : (t == at::kFloat ? OJX_F32 : -1));
}
at::ScalarType scalar_type(long code) {
    return code == OJX_BF16 ? at::kBFloat16 : (code == OJX_F16 ? at::kHalf : at::kFloat);
}

const at::Tensor* as_tensor(PyObject* o) { return o != Py_None && THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// A dense CUDA tensor that holds data (no fake or wrapper tensors).
bool plain(const at::Tensor* t) {
    return t != nullptr && t->defined() && t->is_cuda() && t->layout() == at::kStrided && t->is_contiguous() &&
           !t->unsafeGetTensorImpl()->key_set().has(c10::DispatchKey::Python) && !t->is_conj() && !t->is_neg();
}

bool packed_pair(const at::Tensor* packed, const at::Tensor* scales, c10::Device dev) {
    return plain(packed) && plain(scales) && packed->scalar_type() == at::kByte && scales->scalar_type() == at::kHalf &&
           packed->device() == dev && scales->device() == dev;
}

// The buffers hold the codes and scales of an [n, k] weight: every kernel reads all of them.  (What is too short takes the general
// path, which raises; a group that no format has is refused by the library.)
bool holds(int fmt, const at::Tensor& packed, const at::Tensor& scales, int64_t n, int64_t k, int64_t group) {
    if (n > (int64_t{1} << 31) || k > (int64_t{1} << 31)) return false;
    if (fmt == 0 && (group <= 0 || group % 16 != 0)) group = 16;
    if (group <= 0) return true;
    const int64_t total = n * k, codes = fmt == 0 ? (total + 15) / 16 * 3 : (fmt == 2 ? (total + 3) / 4 : (total + 7) / 8);
    return packed.numel() >= codes && scales.numel() >= (total + group - 1) / group;
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType t, c10::Device dev) {
    return at::detail::empty_cuda(sizes, t, dev, std::nullopt);
}
void* stream_of(c10::Device dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }
void* data(const at::Tensor& t) { return t.data_ptr(); }

// Other Python threads run while this one allocates and launches: a launch waits as long as the launch queue is full.
struct NoGil {
    PyThreadState* const state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

struct Args {
    PyObject* const* v;
    Py_ssize_t n;
    bool ok = true;
    long long i(int k) {
        const long long r = PyLong_AsLongLong(v[k]);
        if (r == -1 && PyErr_Occurred()) { PyErr_Clear(); ok = false; }
        return r;
    }
    const at::Tensor* t(int k) { return as_tensor(v[k]); }
};

#define OJX_ARGS(count)                                                                    \
    if (nargs != (count)) { PyErr_SetString(PyExc_TypeError, "wrong number of arguments"); return nullptr; } \
    Args a{args, nargs}

PyObject* status_or(int32_t st, at::Tensor&& y) {
    if (st != OJX_OK) return PyLong_FromLong(st);
    return THPVariable_Wrap(std::move(y));
}

// direct(x, parameters) -> bool: nothing records, transforms or differentiates operations on these tensors (gradients of either
// mode, the tracer, a dispatch mode, a function transform), so a call may pass by the dispatcher.
PyObject* py_direct(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 2 || !PyDict_Check(args[1])) { PyErr_SetString(PyExc_TypeError, "direct() takes x and a dict of parameters"); return nullptr; }
    bool ok = !torch::jit::tracer::isTracing() && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
              !c10::impl::tls_local_dispatch_key_set().included_.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
    const bool grad = c10::GradMode::is_enabled();
    auto look = [&](PyObject* o) {
        const at::Tensor* t = as_tensor(o);
        if (t != nullptr && t->defined() && ((grad && t->requires_grad()) || t->_fw_grad(0).defined())) ok = false;
    };
    look(args[0]);
    PyObject *name, *value;
    for (Py_ssize_t at = 0; ok && PyDict_Next(args[1], &at, &name, &value);) look(value);
    return PyBool_FromLong(ok);
    END_HANDLE_TH_ERRORS
}

// linear(fmt, x, packed, scales, bias, n, k, group, y_dtype, flags, hadamard) -> y [..., n]
PyObject* py_linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    OJX_ARGS(11);
    const int fmt = (int)a.i(0);
    const at::Tensor *x = a.t(1), *pk = a.t(2), *sc = a.t(3), *bias = args[4] == Py_None ? nullptr : a.t(4);
    const int64_t n = a.i(5), k = a.i(6);
    const int group = (int)a.i(7), yd = (int)a.i(8), flags = (int)a.i(9);
    const bool hadamard = args[10] == Py_True;
    if (!a.ok || !plain(x) || x->dim() < 1 || n <= 0 || k <= 0 || x->size(-1) != k || x->numel() == 0) Py_RETURN_NONE;
    const c10::Device dev = x->device();
    const int xd = dtype_code(x->scalar_type());
    if (xd < 0 || !packed_pair(pk, sc, dev) || !holds(fmt, *pk, *sc, n, k, group)) Py_RETURN_NONE;
    if (args[4] != Py_None &&
        (!plain(bias) || bias->device() != dev || bias->scalar_type() != x->scalar_type() || bias->numel() != n))
        Py_RETURN_NONE;
    const bool rotate = hadamard && k % 32 == 0;         // rotated weights: the transform of x first
    if (rotate && (reinterpret_cast<uintptr_t>(data(*x)) & 15) != 0) Py_RETURN_NONE;
    if (ojx_e8t_poll_status() != OJX_OK) return PyLong_FromLong(1);
    const int64_t m = x->numel() / k;
    c10::SmallVector<int64_t, 6> sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = n;
    const int y_code = yd < 0 ? xd : yd;
    at::Tensor y, rot, ws;
    int32_t st = OJX_OK;
    {
        const NoGil others;
        const c10::cuda::CUDAGuard guard(dev);
        void* s = stream_of(dev);
        y = empty(sizes, scalar_type(y_code), dev);
        const void* xp = data(*x);
        if (rotate) {
            rot = empty({x->numel()}, x->scalar_type(), dev);
            st = ojx_e8t_fwht32(xp, xd, x->numel(), data(rot), s);
            xp = data(rot);
        }
        const size_t need = ojx_e8t_linear_workspace_bytes(fmt, xd, m, n, k, group, flags);
        if (need > 0) ws = empty({(int64_t)need}, at::kByte, dev);
        if (st == OJX_OK)
            st = ojx_e8t_linear(fmt, xp, xd, m, static_cast<const uint8_t*>(data(*pk)), static_cast<const uint16_t*>(data(*sc)),
                                bias ? data(*bias) : nullptr, n, k, group, data(y), y_code, need ? data(ws) : nullptr, need, flags, s);
    }
    return status_or(st, std::move(y));
    END_HANDLE_TH_ERRORS
}

// linear_adapter(fmt, x, packed, scales, bias, n, k, group, y_dtype, hadamard, lora_a, lora_b, scaling) -> y [..., n]; decode shapes
PyObject* py_linear_adapter(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    OJX_ARGS(13);
    const int fmt = (int)a.i(0);
    const at::Tensor *x = a.t(1), *pk = a.t(2), *sc = a.t(3), *bias = args[4] == Py_None ? nullptr : a.t(4), *la = a.t(10), *lb = a.t(11);
    const int64_t n = a.i(5), k = a.i(6);
    const int group = (int)a.i(7), yd = (int)a.i(8), hadamard = args[9] == Py_True && k % 32 == 0;
    const double scaling = PyFloat_AsDouble(args[12]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if (!a.ok || !plain(x) || x->dim() < 1 || n <= 0 || k <= 0 || x->size(-1) != k || x->numel() == 0 || x->numel() / k > 16) Py_RETURN_NONE;
    const c10::Device dev = x->device();
    const at::ScalarType xt = x->scalar_type();
    const int xd = dtype_code(xt);
    if ((xd != OJX_BF16 && xd != OJX_F16) || !packed_pair(pk, sc, dev) || !holds(fmt, *pk, *sc, n, k, group)) Py_RETURN_NONE;
    if (args[4] != Py_None && (!plain(bias) || bias->device() != dev || bias->scalar_type() != xt || bias->numel() != n)) Py_RETURN_NONE;
    if (!plain(la) || !plain(lb) || la->device() != dev || lb->device() != dev || la->scalar_type() != xt || lb->scalar_type() != xt ||
        la->dim() != 2 || lb->dim() != 2 || la->size(0) != k || lb->size(1) != n || la->size(1) != lb->size(0))
        Py_RETURN_NONE;
    if (ojx_e8t_poll_status() != OJX_OK) return PyLong_FromLong(1);
    const int64_t m = x->numel() / k;
    const int rank = (int)la->size(1);
    const size_t need = ojx_e8t_linear_adapter_workspace_bytes(m, k, rank, hadamard);
    if (need == 0) Py_RETURN_NONE;
    c10::SmallVector<int64_t, 6> sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = n;
    const int y_code = yd < 0 ? xd : yd;
    at::Tensor y, ws;
    int32_t st;
    {
        const NoGil others;
        const c10::cuda::CUDAGuard guard(dev);
        y = empty(sizes, scalar_type(y_code), dev);
        ws = empty({(int64_t)need}, at::kByte, dev);
        st = ojx_e8t_linear_adapter(fmt, data(*x), xd, m, static_cast<const uint8_t*>(data(*pk)), static_cast<const uint16_t*>(data(*sc)),
                                    bias ? data(*bias) : nullptr, n, k, group, data(*la), data(*lb), rank, (float)scaling, hadamard,
                                    data(y), y_code, data(ws), need, stream_of(dev));
    }
    if (st == OJX_ERR_UNSUPPORTED) Py_RETURN_NONE;
    return status_or(st, std::move(y));
    END_HANDLE_TH_ERRORS
}

// linear_dx(fmt, grad_y [m, n], packed, scales, n, k, group, out_dtype) -> dx [m, k]; 16-bit gradients
PyObject* py_linear_dx(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    OJX_ARGS(8);
    const int fmt = (int)a.i(0);
    const at::Tensor *gy = a.t(1), *pk = a.t(2), *sc = a.t(3);
    const int64_t n = a.i(4), k = a.i(5);
    const int group = (int)a.i(6), od = (int)a.i(7);
    if (!a.ok || !plain(gy) || gy->dim() != 2 || n <= 0 || k <= 0 || gy->size(1) != n || gy->size(0) == 0) Py_RETURN_NONE;
    const c10::Device dev = gy->device();
    const int gd = dtype_code(gy->scalar_type());
    if ((gd != OJX_BF16 && gd != OJX_F16) || !packed_pair(pk, sc, dev) || !holds(fmt, *pk, *sc, n, k, group)) Py_RETURN_NONE;
    if (ojx_e8t_poll_status() != OJX_OK) return PyLong_FromLong(1);
    const int64_t m = gy->size(0);
    const int code = od < 0 ? gd : od;
    at::Tensor dx, ws;
    int32_t st;
    {
        const NoGil others;
        const c10::cuda::CUDAGuard guard(dev);
        dx = empty({m, k}, scalar_type(code), dev);
        const size_t need = ojx_e8t_gemm_dx_workspace_bytes(m, n, k);
        ws = empty({(int64_t)need}, at::kByte, dev);
        const uint8_t* p = static_cast<const uint8_t*>(data(*pk));
        const uint16_t* q = static_cast<const uint16_t*>(data(*sc));
        void* s = stream_of(dev);
        st = fmt == 0 ? ojx_e8t_gemm_dx(data(*gy), gd, m, p, q, n, k, group, data(dx), code, data(ws), need, s)
                      : ojx_e8t_gemm_dx_lowbit(fmt, data(*gy), gd, m, p, q, n, k, group, data(dx), code, data(ws), need, s);
    }
    return status_or(st, std::move(dx));
    END_HANDLE_TH_ERRORS
}

// encode(fmt, w [rows, cols], group, code_bytes, scale_count, flags) -> (packed, scales)
PyObject* py_encode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    OJX_ARGS(6);
    const int fmt = (int)a.i(0);
    const at::Tensor* w = a.t(1);
    const int group = (int)a.i(2);
    const int64_t bytes = a.i(3), count = a.i(4);
    const uint32_t flags = (uint32_t)a.i(5);
    if (!a.ok || !plain(w) || w->dim() != 2 || w->numel() == 0) Py_RETURN_NONE;
    const int wd = dtype_code(w->scalar_type());
    if (wd < 0) Py_RETURN_NONE;
    const c10::Device dev = w->device();
    at::Tensor pk, sc;
    int32_t st;
    {
        const NoGil others;
        const c10::cuda::CUDAGuard guard(dev);
        pk = empty({bytes}, at::kByte, dev);
        sc = empty({count}, at::kHalf, dev);
        uint8_t* p = static_cast<uint8_t*>(data(pk));
        uint16_t* q = static_cast<uint16_t*>(data(sc));
        void* s = stream_of(dev);
        const int64_t rows = w->size(0), cols = w->size(1);
        st = fmt == 0 ? ojx_e8t_encode_ex(data(*w), wd, rows, cols, group, flags, p, q, s)
           : fmt == 2 ? ojx_e8t_encode_2bit(data(*w), wd, rows, cols, group, p, q, s)
                      : ojx_e8t_encode_1bit(data(*w), wd, rows, cols, group, p, q, s);
    }
    if (st != OJX_OK) return PyLong_FromLong(st);
    PyObject* tp = THPVariable_Wrap(std::move(pk));
    PyObject* ts = THPVariable_Wrap(std::move(sc));
    PyObject* pair = (tp && ts) ? PyTuple_Pack(2, tp, ts) : nullptr;
    Py_XDECREF(tp);
    Py_XDECREF(ts);
    return pair;
    END_HANDLE_TH_ERRORS
}

// decode(fmt, packed, scales, rows, cols, group, dtype) -> w [rows, cols]; the caller has checked the sizes
PyObject* py_decode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    OJX_ARGS(7);
    const int fmt = (int)a.i(0);
    const at::Tensor *pk = a.t(1), *sc = a.t(2);
    const int64_t rows = a.i(3), cols = a.i(4);
    const int group = (int)a.i(5), od = (int)a.i(6);
    if (!a.ok || !plain(pk) || !packed_pair(pk, sc, pk->device()) || rows <= 0 || cols <= 0) Py_RETURN_NONE;
    const c10::Device dev = pk->device();
    at::Tensor w;
    int32_t st;
    {
        const NoGil others;
        const c10::cuda::CUDAGuard guard(dev);
        w = empty({rows, cols}, scalar_type(od), dev);
        const uint8_t* p = static_cast<const uint8_t*>(data(*pk));
        const uint16_t* q = static_cast<const uint16_t*>(data(*sc));
        void* s = stream_of(dev);
        st = fmt == 0 ? ojx_e8t_decode(p, q, rows, cols, group, od, data(w), s)
           : fmt == 2 ? ojx_e8t_decode_2bit(p, q, rows, cols, group, od, data(w), s)
                      : ojx_e8t_decode_1bit(p, q, rows, cols, group, od, data(w), s);
    }
    return status_or(st, std::move(w));
    END_HANDLE_TH_ERRORS
}

// fwht32(x) -> rotated x
PyObject* py_fwht32(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    OJX_ARGS(1);
    const at::Tensor* x = a.t(0);
    if (!plain(x) || x->numel() == 0 || x->dim() < 1 || x->size(-1) % 32 != 0 || (reinterpret_cast<uintptr_t>(data(*x)) & 15) != 0)
        Py_RETURN_NONE;
    const int xd = dtype_code(x->scalar_type());
    if (xd < 0) Py_RETURN_NONE;
    const c10::Device dev = x->device();
    at::Tensor y;
    int32_t st;
    {
        const NoGil others;
        const c10::cuda::CUDAGuard guard(dev);
        y = empty(x->sizes(), x->scalar_type(), dev);
        st = ojx_e8t_fwht32(data(*x), xd, x->numel(), data(y), stream_of(dev));
    }
    return status_or(st, std::move(y));
    END_HANDLE_TH_ERRORS
}

// grouped(device, table, count, tiles, m, x_dtype, y_dtype, needs_reduce, peer_deltas, world, peer_sync, flags) -> status
PyObject* py_grouped(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    OJX_ARGS(12);
    const c10::DeviceIndex index = (c10::DeviceIndex)a.i(0);
    if (ojx_e8t_poll_status() != OJX_OK) return PyLong_FromLong(1);
    const long long table = a.i(1), peers = a.i(8), sync = a.i(10);
    const int count = (int)a.i(2), tiles = (int)a.i(3), m = (int)a.i(4), xd = (int)a.i(5), yd = (int)a.i(6), reduce = (int)a.i(7);
    const int world = (int)a.i(9), flags = (int)a.i(11);
    if (!a.ok) { PyErr_SetString(PyExc_TypeError, "grouped() takes integers"); return nullptr; }
    int32_t st;
    {
        const NoGil others;
        const c10::cuda::CUDAGuard guard(index);
        st = ojx_e8t_gemv_grouped_ex(reinterpret_cast<const ojx_e8t_gemv_problem*>(table), count, tiles, m, xd, yd, reduce,
                                     reinterpret_cast<const int64_t*>(peers), world, reinterpret_cast<ojx_e8t_peer_sync*>(sync), flags,
                                     c10::cuda::getCurrentCUDAStream(index).stream());
    }
    return PyLong_FromLong(st);
    END_HANDLE_TH_ERRORS
}

#define OJX_METHOD(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {OJX_METHOD(direct), OJX_METHOD(linear), OJX_METHOD(linear_adapter), OJX_METHOD(linear_dx), OJX_METHOD(encode), OJX_METHOD(decode), OJX_METHOD(fwht32),
                         OJX_METHOD(grouped), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ojx_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ojx_torch() { return PyModule_Create(&module); }
