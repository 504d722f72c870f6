// Native host path of the Python operators: what quantforge_b200/ops.py does around one C-ABI call (reading the
// tensors, checking them, allocating the result, finding stream and workspace, filling the descriptor), without the
// interpreter. Only the ordinary case is handled here: CUDA tensors of one device, contiguous, right shapes and types,
// a workspace that this stream already has. Whatever differs - an argument in error included - returns None, and
// ops.py takes the call from the start: it makes the copies and allocations that are needed, and raises what it has to.
// None means that nothing was enqueued: a status that says otherwise is raised here.
//
// The interpreter lock is held while Python objects are read and released around allocation and launch, both of which can
// block (a full launch queue, a free of cached memory): other Python threads go on meanwhile, as around a foreign call. The
// caller's references keep the arguments alive.
//
// Why: the interpreter needed 15 to 17 us per linear (attribute reads, two foreign calls, a device context manager,
// ctypes conversions), more than the kernels of small layers take on the GPU.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <unordered_map>
#include <vector>

#include "quantforge_rt.h"

namespace {

using at::ScalarType;
using at::Tensor;

constexpr int kMaxDevices = 64;
qf_ctx *g_ctx[kMaxDevices] = {nullptr};  // ops.py registers a device's context when it creates it

// The workspaces that ops.py has made, by device and stream, ascending in size. The tensors live in ops.py.
struct Buffer {
    size_t bytes;
    void *ptr;
};
struct StreamKey {
    int device;
    cudaStream_t stream;
    bool operator==(const StreamKey &o) const { return device == o.device && stream == o.stream; }
};
struct StreamKeyHash {
    size_t operator()(const StreamKey &k) const { return std::hash<void *>()((void *)k.stream) * 31u + (size_t)k.device; }
};
std::unordered_map<StreamKey, std::vector<Buffer>, StreamKeyHash> g_workspaces;

bool find_workspace(int device, cudaStream_t stream, size_t need, void **ptr, size_t *bytes) {
    *ptr = nullptr;
    *bytes = 0;
    if (need == 0) return true;
    const auto it = g_workspaces.find(StreamKey{device, stream});
    if (it == g_workspaces.end()) return false;
    for (const Buffer &b : it->second)
        if (b.bytes >= need) {
            *ptr = b.ptr;
            *bytes = b.bytes;
            return true;
        }
    return false;
}

// Other Python threads run while this exists.
class Unlocked {
  public:
    Unlocked() : state_(PyEval_SaveThread()) {}
    ~Unlocked() { PyEval_RestoreThread(state_); }
    Unlocked(const Unlocked &) = delete;
    Unlocked &operator=(const Unlocked &) = delete;

  private:
    PyThreadState *state_;
};

PyObject *g_error = nullptr;  // QuantForgeError(status, name, message)

// What a call of the C ABI that did not succeed becomes. Its checks come before any launch, and ops.py may start over after
// them; anything else is an error of CUDA.
PyObject *failed(int status, int device) {
    if (status == QF_ERR_BAD_ARG || status == QF_ERR_UNSUPPORTED || status == QF_ERR_WORKSPACE) Py_RETURN_NONE;
    PyObject *e = PyObject_CallFunction(g_error ? g_error : PyExc_RuntimeError, "iss", status, qf_status_string(status),
                                        qf_last_error(g_ctx[device]));
    if (e) {
        PyErr_SetObject((PyObject *)Py_TYPE(e), e);
        Py_DECREF(e);
    }
    return nullptr;
}

int type_code(ScalarType t) {
    return t == at::kHalf ? QF_F16 : t == at::kBFloat16 ? QF_BF16 : t == at::kFloat ? QF_F32 : -1;
}
bool is_byte(ScalarType t) { return t == at::kChar || t == at::kByte; }

// A plain contiguous CUDA tensor on `device` (-1: any; then `device` becomes its device).
const Tensor *cuda_tensor(PyObject *o, int *device) {
    if (!THPVariable_Check(o)) return nullptr;
    const Tensor &t = THPVariable_Unpack(o);
    if (!t.is_cuda() || t.layout() != at::kStrided || !t.is_contiguous() || !t.has_storage() ||
        t.key_set().has(c10::DispatchKey::Python) || t.is_conj() || t.is_neg())
        return nullptr;
    const int d = t.get_device();
    if (*device >= 0 && d != *device) return nullptr;
    *device = d;
    return &t;
}

bool shape_is(const Tensor &t, int64_t a, int64_t b) { return t.dim() == 2 && t.size(0) == a && t.size(1) == b; }

// The layout helpers (pack, pack_zeros, quantize) are tensor programs in ops.py, which autograd, tracing and function transforms
// see operator by operator. Whether any of them watches this call on `t`.
bool watched(PyObject *o, const Tensor &t) {
    const c10::DispatchKeySet in = c10::impl::tls_local_dispatch_key_set().included_;
    return !THPVariable_CheckExact(o) || in.has(c10::DispatchKey::Python) || in.has(c10::DispatchKey::Tracer) ||
           in.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) || in.has(c10::DispatchKey::Functionalize) ||
           at::impl::torch_function_mode_enabled() || (t.requires_grad() && c10::GradMode::is_enabled()) ||
           t._fw_grad(0).defined();
}

// The device must be the current one and must have a context.
bool ready(int device) {
    return device >= 0 && device < kMaxDevices && g_ctx[device] != nullptr && c10::cuda::current_device() == device;
}

cudaStream_t stream_of(int device) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }

Tensor empty(at::IntArrayRef size, ScalarType type, int device) {
    return at::detail::empty_cuda(size, type, c10::Device(c10::kCUDA, (c10::DeviceIndex)device), std::nullopt);
}

// A small integer argument; false leaves no error set.
bool as_int(PyObject *o, long long *v) {
    if (!PyLong_Check(o)) return false;
    *v = PyLong_AsLongLong(o);
    if (*v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}
bool attr_int(PyObject *o, PyObject *name, long long *v) {
    PyObject *a = PyObject_GetAttr(o, name);
    if (!a) {
        PyErr_Clear();
        return false;
    }
    const bool ok = as_int(a, v);
    Py_DECREF(a);
    return ok;
}

// Zero points [G, N]: none (constant), int8, or packed four-bit codes.
bool read_zeros(PyObject *o, int64_t G, int64_t N, int *device, qf_linear_desc *d, const void **ptr) {
    *ptr = nullptr;
    if (o == Py_None) {
        d->zero_mode = QF_ZERO_CONST;
        return true;
    }
    const Tensor *z = cuda_tensor(o, device);
    if (!z) return false;
    if (z->scalar_type() == at::kChar && shape_is(*z, G, N)) d->zero_mode = QF_ZERO_I8;
    else if (z->scalar_type() == at::kInt && N % 8 == 0 && shape_is(*z, G, N / 8)) d->zero_mode = QF_ZERO_U4;
    else return false;
    *ptr = z->const_data_ptr();
    return true;
}

// Packed weights [N, K/2] bytes or [N, K/8] words, scales [K/group, N], zeros. `K` < 0: taken from the weights.
bool read_weights(PyObject *qw_o, PyObject *sc_o, PyObject *z_o, int *device, qf_linear_desc *d, int64_t K,
                  const void **qw_ptr, const void **sc_ptr, const void **z_ptr, ScalarType *act) {
    const Tensor *qw = cuda_tensor(qw_o, device), *sc = cuda_tensor(sc_o, device);
    if (!qw || !sc || qw->dim() != 2) return false;
    const int64_t per = is_byte(qw->scalar_type()) ? 2 : qw->scalar_type() == at::kInt ? 8 : 0;
    if (per == 0) return false;
    d->N = qw->size(0);
    d->K = qw->size(1) * per;
    if (K >= 0 && d->K != K) return false;
    if (d->group_size <= 0 || d->K % d->group_size != 0) return false;
    *act = sc->scalar_type();
    if (*act != at::kHalf && *act != at::kBFloat16) return false;
    const int64_t G = d->K / d->group_size;
    if (!shape_is(*sc, G, d->N)) return false;
    d->act_dtype = type_code(*act);
    *qw_ptr = qw->const_data_ptr();
    *sc_ptr = sc->const_data_ptr();
    return read_zeros(z_o, G, d->N, device, d, z_ptr);
}

// Allocates or checks the result, finds the workspace and makes the call. None where any of it does not apply.
PyObject *finish(qf_linear_desc *d, int device, const Tensor &x, const void *qw, const void *sc, const void *z,
                 PyObject *out_dtype_o, PyObject *out_o, PyObject *residual_o) {
    ScalarType out_type = x.scalar_type();
    if (out_dtype_o != Py_None) {
        if (!THPDtype_Check(out_dtype_o)) Py_RETURN_NONE;
        out_type = ((THPDtype *)out_dtype_o)->scalar_type;
    }
    d->out_dtype = type_code(out_type);
    if (d->out_dtype < 0 || d->M <= 0) Py_RETURN_NONE;
    const int64_t cols = d->epilogue == QF_EPI_SILU_MUL ? d->N / 2 : d->N;
    const void *res = nullptr;
    if (residual_o != Py_None) {
        const Tensor *r = cuda_tensor(residual_o, &device);
        if (!r) Py_RETURN_NONE;
        if (d->epilogue == QF_EPI_RESIDUAL_ADD && (!shape_is(*r, d->M, cols) || r->scalar_type() != out_type)) Py_RETURN_NONE;
        res = r->const_data_ptr();
    } else if (d->epilogue == QF_EPI_RESIDUAL_ADD) {
        Py_RETURN_NONE;
    }
    if (!ready(device)) Py_RETURN_NONE;
    const cudaStream_t stream = stream_of(device);
    void *ws;
    size_t ws_bytes;
    if (!find_workspace(device, stream, qf_w4a16_workspace_bytes(d), &ws, &ws_bytes)) Py_RETURN_NONE;
    Tensor y;
    if (out_o != Py_None) {
        const Tensor *o = cuda_tensor(out_o, &device);
        if (!o || !shape_is(*o, d->M, cols) || o->scalar_type() != out_type) Py_RETURN_NONE;
        y = *o;
    }
    int st;
    {
        Unlocked u;
        if (!y.defined()) y = empty({d->M, cols}, out_type, device);
        st = qf_w4a16_linear_fused(g_ctx[device], d, x.const_data_ptr(), qw, sc, z, y.data_ptr(), res, ws, ws_bytes, stream);
    }
    if (st != QF_OK) return failed(st, device);
    if (out_o != Py_None) return Py_NewRef(out_o);
    return THPVariable_Wrap(std::move(y));
}

// ------------------------------------------------------------------------------------------------
// entry points (positional arguments only; None = not handled here)
// ------------------------------------------------------------------------------------------------
PyObject *s_blob, *s_N, *s_K, *s_group, *s_act, *s_zmode, *s_zconst;  // interned attribute names of SlabWeight

// linear(x, qweight, scales, zeros, group_size, zero_const, out_dtype, path, split_k, out, weight_layout, epilogue, residual)
PyObject *linear_impl(PyObject *const *a) {
    int device = -1;
    const Tensor *x = cuda_tensor(a[0], &device);
    if (!x || x->dim() != 2) Py_RETURN_NONE;
    qf_linear_desc d = {};
    long long group, zero_const, path, split_k, layout, epilogue;
    if (!as_int(a[8], &split_k) || !as_int(a[11], &epilogue)) Py_RETURN_NONE;
    d.M = x->size(0);
    d.split_k = (int32_t)split_k;
    d.epilogue = (int32_t)epilogue;
    const void *qw, *sc = nullptr, *z = nullptr;
    Tensor blob;
    if (THPVariable_Check(a[1])) {
        ScalarType act;
        if (!as_int(a[4], &group) || !as_int(a[5], &zero_const) || !as_int(a[7], &path) || !as_int(a[10], &layout)) Py_RETURN_NONE;
        if (group > INT32_MAX || zero_const < -128 || zero_const > 127) Py_RETURN_NONE;
        d.group_size = (int32_t)group;
        d.path = (int32_t)path;
        d.weight_layout = (int32_t)layout;
        if (!read_weights(a[1], a[2], a[3], &device, &d, x->size(1), &qw, &sc, &z, &act) || act != x->scalar_type()) Py_RETURN_NONE;
        if (d.zero_mode == QF_ZERO_CONST) d.zero_const = (int32_t)zero_const;
    } else {
        // a SlabWeight: blob, shape and converter facts come from the object
        PyObject *blob_o = PyObject_GetAttr(a[1], s_blob);
        if (!blob_o) {
            PyErr_Clear();
            Py_RETURN_NONE;
        }
        const Tensor *t = cuda_tensor(blob_o, &device);
        if (t) blob = *t;  // another thread may give the object another blob
        Py_DECREF(blob_o);
        qw = blob.defined() ? blob.const_data_ptr() : nullptr;
        const size_t have = blob.defined() ? (size_t)blob.nbytes() : 0;
        PyObject *act_o = PyObject_GetAttr(a[1], s_act);
        if (!act_o) PyErr_Clear();
        const bool act_ok = act_o && THPDtype_Check(act_o) && ((THPDtype *)act_o)->scalar_type == x->scalar_type();
        Py_XDECREF(act_o);
        long long N, K, zmode;
        if (!qw || !act_ok || !attr_int(a[1], s_N, &N) || !attr_int(a[1], s_K, &K) || !attr_int(a[1], s_group, &group) ||
            !attr_int(a[1], s_zmode, &zmode) || !attr_int(a[1], s_zconst, &zero_const))
            Py_RETURN_NONE;
        if (x->size(1) != K || have < qf_prepack_bytes(QF_LAYOUT_GEMV_SLAB, N, K)) Py_RETURN_NONE;
        d.N = N;
        d.K = K;
        d.group_size = (int32_t)group;
        d.act_dtype = type_code(x->scalar_type());
        d.zero_mode = (int32_t)zmode;
        d.zero_const = (int32_t)zero_const;
        d.path = QF_PATH_AUTO;
        d.weight_layout = QF_LAYOUT_GEMV_SLAB;
    }
    return finish(&d, device, *x, qw, sc, z, a[6], a[9], a[12]);
}

// gemv(x, w_packed, scale, zero_point): per-channel quantisation
PyObject *gemv_impl(PyObject *const *a) {
    int device = -1;
    const Tensor *x = cuda_tensor(a[0], &device), *w = cuda_tensor(a[1], &device), *sc = cuda_tensor(a[2], &device),
                 *z = cuda_tensor(a[3], &device);
    if (!x || !w || !sc || !z || x->dim() != 2 || w->dim() != 2 || !is_byte(w->scalar_type())) Py_RETURN_NONE;
    qf_linear_desc d = {};
    d.M = x->size(0);
    d.K = x->size(1);
    d.N = w->size(0);
    const ScalarType act = x->scalar_type();
    if ((act != at::kHalf && act != at::kBFloat16) || sc->scalar_type() != act || z->scalar_type() != at::kChar) Py_RETURN_NONE;
    if (w->size(1) * 2 != d.K || sc->numel() != d.N || z->numel() != d.N || d.K > INT32_MAX) Py_RETURN_NONE;
    d.group_size = (int32_t)d.K;
    d.act_dtype = type_code(act);
    d.zero_mode = QF_ZERO_I8;
    return finish(&d, device, *x, w->const_data_ptr(), sc->const_data_ptr(), z->const_data_ptr(), Py_None, Py_None, Py_None);
}

// unpack(packed)
PyObject *unpack_impl(PyObject *const *a) {
    int device = -1;
    const Tensor *p = cuda_tensor(a[0], &device);
    if (!p || p->dim() < 1 || !is_byte(p->scalar_type()) || p->numel() == 0 || !ready(device)) Py_RETURN_NONE;
    c10::SmallVector<int64_t, 5> shape(p->sizes().begin(), p->sizes().end());
    const int64_t cols = shape.back();
    shape.back() = cols * 2;
    Tensor out;
    int st;
    {
        Unlocked u;
        out = empty(shape, at::kChar, device);
        st = qf_unpack_int4(g_ctx[device], p->const_data_ptr(), out.data_ptr(), p->numel() / cols, cols, stream_of(device));
    }
    if (st != QF_OK) return failed(st, device);
    return THPVariable_Wrap(std::move(out));
}

// dequant(qweight, scales, zeros, group_size, zero_const)
PyObject *dequant_impl(PyObject *const *a) {
    int device = -1;
    qf_linear_desc d = {};
    long long group, zero_const;
    if (!as_int(a[3], &group) || !as_int(a[4], &zero_const) || group > INT32_MAX || zero_const < -128 || zero_const > 127)
        Py_RETURN_NONE;
    d.M = 1;
    d.group_size = (int32_t)group;
    const void *qw, *sc, *z;
    ScalarType act;
    if (!read_weights(a[0], a[1], a[2], &device, &d, -1, &qw, &sc, &z, &act) || !ready(device)) Py_RETURN_NONE;
    if (d.zero_mode == QF_ZERO_CONST) d.zero_const = (int32_t)zero_const;
    d.out_dtype = d.act_dtype;
    Tensor out;
    int st;
    {
        Unlocked u;
        out = empty({d.N, d.K}, act, device);
        st = qf_dequant_w4(g_ctx[device], &d, qw, sc, z, out.data_ptr(), stream_of(device));
    }
    if (st != QF_OK) return failed(st, device);
    return THPVariable_Wrap(std::move(out));
}

// pack(codes): int8 [..., 2n] -> int8 [..., n]
PyObject *pack_impl(PyObject *const *a) {
    int device = -1;
    const Tensor *c = cuda_tensor(a[0], &device);
    if (!c || watched(a[0], *c) || c->dim() < 1 || c->scalar_type() != at::kChar || c->numel() == 0 || c->sizes().back() % 2 != 0 || !ready(device))
        Py_RETURN_NONE;
    c10::SmallVector<int64_t, 5> shape(c->sizes().begin(), c->sizes().end());
    shape.back() /= 2;
    Tensor out;
    int st;
    {
        Unlocked u;
        out = empty(shape, at::kChar, device);
        st = qf_pack_int4(g_ctx[device], c->const_data_ptr(), out.data_ptr(), out.numel(), stream_of(device));
    }
    if (st != QF_OK) return failed(st, device);
    return THPVariable_Wrap(std::move(out));
}

// pack_zeros(zeros): int8 [G, N] -> int32 [G, N/8]
PyObject *pack_zeros_impl(PyObject *const *a) {
    int device = -1;
    const Tensor *z = cuda_tensor(a[0], &device);
    if (!z || watched(a[0], *z) || z->dim() != 2 || z->scalar_type() != at::kChar || z->numel() == 0 || z->size(1) % 8 != 0 || !ready(device))
        Py_RETURN_NONE;
    Tensor out;
    int st;
    {
        Unlocked u;
        out = empty({z->size(0), z->size(1) / 8}, at::kInt, device);
        st = qf_pack_int4(g_ctx[device], z->const_data_ptr(), out.data_ptr(), z->numel() / 2, stream_of(device));
    }
    if (st != QF_OK) return failed(st, device);
    return THPVariable_Wrap(std::move(out));
}

// quantize(weight, group_size, symmetric, scale_dtype) -> (codes, scales, zeros or None)
PyObject *quantize_impl(PyObject *const *a) {
    int device = -1;
    const Tensor *w = cuda_tensor(a[0], &device);
    long long group;
    if (!w || watched(a[0], *w) || w->dim() != 2 || w->numel() == 0 || type_code(w->scalar_type()) < 0 || !as_int(a[1], &group) || !PyBool_Check(a[2]) ||
        !THPDtype_Check(a[3]) || !ready(device))
        Py_RETURN_NONE;
    const ScalarType st = ((THPDtype *)a[3])->scalar_type;
    const int64_t N = w->size(0), K = w->size(1);
    if ((st != at::kHalf && st != at::kBFloat16) || group <= 0 || group > INT32_MAX || K % group != 0) Py_RETURN_NONE;
    const bool sym = a[2] == Py_True;
    Tensor codes, scales, zeros;
    int status;
    {
        Unlocked u;
        codes = empty({N, K}, at::kChar, device);
        scales = empty({K / group, N}, st, device);
        if (!sym) zeros = empty({K / group, N}, at::kChar, device);
        status = qf_quantize_w4(g_ctx[device], w->const_data_ptr(), type_code(w->scalar_type()), N, K, (int)group, sym,
                                codes.data_ptr(), scales.data_ptr(), type_code(st), sym ? nullptr : zeros.data_ptr(),
                                stream_of(device));
    }
    if (status != QF_OK) return failed(status, device);
    PyObject *c = THPVariable_Wrap(std::move(codes)), *s = THPVariable_Wrap(std::move(scales));
    PyObject *z = sym ? Py_NewRef(Py_None) : THPVariable_Wrap(std::move(zeros));
    return Py_BuildValue("(NNN)", c, s, z);
}

// prepack_slab(qweight, scales, zeros, group_size, zero_const) -> (blob, N, K, zero_mode)
PyObject *prepack_slab_impl(PyObject *const *a) {
    int device = -1;
    qf_linear_desc d = {};
    long long group, zero_const;
    if (!as_int(a[3], &group) || !as_int(a[4], &zero_const) || group > INT32_MAX || zero_const < -128 || zero_const > 127)
        Py_RETURN_NONE;
    d.M = 1;
    d.group_size = (int32_t)group;
    const void *qw, *sc, *z;
    ScalarType act;
    if (!read_weights(a[0], a[1], a[2], &device, &d, -1, &qw, &sc, &z, &act) || !ready(device)) Py_RETURN_NONE;
    d.zero_const = (int32_t)zero_const;
    d.out_dtype = d.act_dtype;
    d.weight_layout = QF_LAYOUT_GEMV_SLAB;
    const size_t bytes = qf_prepack_bytes(QF_LAYOUT_GEMV_SLAB, d.N, d.K);
    if (bytes == 0) Py_RETURN_NONE;
    Tensor blob;
    int st;
    {
        Unlocked u;
        blob = empty({(int64_t)bytes}, at::kByte, device);
        st = qf_prepack_gemv_slab(g_ctx[device], &d, qw, sc, z, blob.data_ptr(), stream_of(device));
    }
    if (st != QF_OK) return failed(st, device);
    return Py_BuildValue("(NLLi)", THPVariable_Wrap(std::move(blob)), (long long)d.N, (long long)d.K, (int)d.zero_mode);
}

// prepack(qweight, to_canonical, layout)
PyObject *prepack_impl(PyObject *const *a) {
    int device = -1;
    const Tensor *q = cuda_tensor(a[0], &device);
    long long layout;
    if (!q || q->dim() != 2 || q->numel() == 0 || !PyBool_Check(a[1]) || !as_int(a[2], &layout) || !ready(device)) Py_RETURN_NONE;
    const int64_t per = is_byte(q->scalar_type()) ? 2 : q->scalar_type() == at::kInt ? 8 : 0;
    if (per == 0 || (int64_t)q->nbytes() % 4 != 0) Py_RETURN_NONE;
    const int back = a[1] == Py_True ? 1 : 0;
    Tensor out;
    int st;
    {
        Unlocked u;
        out = empty(q->sizes(), q->scalar_type(), device);
        if (layout == QF_LAYOUT_TILED)
            st = qf_prepack_w4_tiled(g_ctx[device], q->const_data_ptr(), out.data_ptr(), q->size(0), q->size(1) * per, back,
                                     stream_of(device));
        else
            st = qf_prepack_w4(g_ctx[device], q->const_data_ptr(), out.data_ptr(), (int64_t)q->nbytes() / 4, back, stream_of(device));
    }
    if (st != QF_OK) return failed(st, device);
    return THPVariable_Wrap(std::move(out));
}

template <PyObject *(*F)(PyObject *const *), Py_ssize_t N>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
    if (n != N) {
        PyErr_SetString(PyExc_TypeError, "wrong number of arguments");
        return nullptr;
    }
    try {
        return F(args);
    } catch (const std::exception &) {  // no memory, for one: ops.py meets the same and says so
        Py_RETURN_NONE;
    }
}

// set_ctx(device, handle)
PyObject *set_ctx_impl(PyObject *const *a) {
    long long device, handle;
    if (!as_int(a[0], &device) || !as_int(a[1], &handle)) Py_RETURN_NONE;
    if (device >= 0 && device < kMaxDevices) g_ctx[device] = (qf_ctx *)(intptr_t)handle;
    Py_RETURN_NONE;
}

// set_error(class): what `failed` raises
PyObject *set_error_impl(PyObject *const *a) {
    Py_INCREF(a[0]);
    Py_XSETREF(g_error, a[0]);
    Py_RETURN_NONE;
}

// add_workspace(device, stream, pointer, bytes)
PyObject *add_workspace_impl(PyObject *const *a) {
    long long device, stream, ptr, bytes;
    if (!as_int(a[0], &device) || !as_int(a[1], &stream) || !as_int(a[2], &ptr) || !as_int(a[3], &bytes)) Py_RETURN_NONE;
    g_workspaces[StreamKey{(int)device, (cudaStream_t)(intptr_t)stream}].push_back(Buffer{(size_t)bytes, (void *)(intptr_t)ptr});
    Py_RETURN_NONE;
}

#define QF_FAST(name, fn, n) {name, (PyCFunction)(void (*)(void))(entry<fn, n>), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    QF_FAST("linear", linear_impl, 13), QF_FAST("gemv", gemv_impl, 4),       QF_FAST("unpack", unpack_impl, 1),
    QF_FAST("pack", pack_impl, 1),       QF_FAST("pack_zeros", pack_zeros_impl, 1), QF_FAST("quantize", quantize_impl, 4),
    QF_FAST("prepack_slab", prepack_slab_impl, 5), QF_FAST("prepack", prepack_impl, 3),
    QF_FAST("dequant", dequant_impl, 5), QF_FAST("set_ctx", set_ctx_impl, 2), QF_FAST("add_workspace", add_workspace_impl, 4),
    QF_FAST("set_error", set_error_impl, 1),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_qf_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__qf_host(void) {
    s_blob = PyUnicode_InternFromString("blob");
    s_N = PyUnicode_InternFromString("N");
    s_K = PyUnicode_InternFromString("K");
    s_group = PyUnicode_InternFromString("group_size");
    s_act = PyUnicode_InternFromString("act_dtype");
    s_zmode = PyUnicode_InternFromString("zero_mode");
    s_zconst = PyUnicode_InternFromString("zero_const");
    return PyModule_Create(&module);
}
