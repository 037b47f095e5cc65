// Native host path of the Python launchers.
//
// One call of RegularAttention.forward used to spend 16 to 18 us on the host: a dozen attribute reads and
// comparisons on tensors, ctypes conversions of 20 arguments and a periodic copy of the status word --
// more than the small problems take on the device.  The functions here do the same checks on the tensors'
// C++ objects and call the C ABI directly.  They only ever take the ordinary case: plain CUDA tensors on
// the current device, consistent shapes, no debug mode, no reported failure.  For anything else they
// return None without side effects and the Python code, which also words the errors, carries on.
//
// The C ABI entry points are handed over as addresses (bind()), so this module follows whichever build of
// the library splat_native loaded, and the library itself stays free of torch.
#include <Python.h>

#include <ATen/core/CachingHostAllocator.h>
#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <chrono>
#include <cstdint>
#include <cstdlib>
#include <exception>
#include <mutex>

namespace {

constexpr int kPathAuto = 0, kPathGeneric = 1, kPathBand = 2;
constexpr int kMaxDevices = 64;

using FusedFn = int32_t (*)(const void*, const void*, int64_t, int64_t, int64_t, const void*, void*, float*,
                            const float*, const float*, const float*, int64_t, int64_t, int64_t, int64_t, float,
                            int32_t, int32_t, const int32_t*, const int32_t*, int32_t*, int32_t*, void*);
using SddmmBandFn = int32_t (*)(const void*, const void*, int64_t, int64_t, int64_t, void*, const float*, const float*,
                                const float*, int64_t, int64_t, int64_t, int64_t, int64_t, int32_t, const int32_t*,
                                const int32_t*, int32_t*, void*);
using SpmmBandFn = int32_t (*)(const void*, const void*, void*, const float*, const float*, const float*, int64_t, int64_t,
                               int64_t, int64_t, int64_t, int32_t, const int32_t*, const int32_t*, int32_t*, void*);
using SddmmTileFn = int32_t (*)(const void*, const void*, int64_t, int64_t, int64_t, void*, const float*, const float*,
                                const float*, int64_t, int64_t, int64_t, int64_t, int64_t, int32_t, const int32_t*, int32_t*, void*);
using SpmmTileFn = int32_t (*)(const void*, const void*, void*, const float*, const float*, const float*, int64_t, int64_t,
                               int64_t, int64_t, int64_t, int32_t, const int32_t*, int32_t*, void*);
using SddmmFn = int32_t (*)(const void*, const void*, int64_t, int64_t, int64_t, void*, const float*, const float*,
                            const float*, int64_t, int64_t, int64_t, int64_t, int64_t, int32_t, void*);
using SpmmFn = int32_t (*)(const void*, const void*, void*, const float*, const float*, const float*, int64_t, int64_t,
                           int64_t, int64_t, int64_t, int32_t, void*);
using MaskFn = int32_t (*)(const void*, int64_t, int64_t, int64_t, int32_t, float*, float*, float*, float*, float*, float*, float*,
                           int32_t*, int32_t*, void*);
using TransposeFn = int32_t (*)(const void*, void*, int64_t, int64_t, int64_t, void*);
using SoftmaxFn = int32_t (*)(const void*, void*, const float*, int64_t, int64_t, int64_t, float, int32_t, void*);

struct Api {
    FusedFn fused;
    SddmmBandFn sddmm_band;
    SpmmBandFn spmm_band;
    SddmmTileFn sddmm_tile;
    SpmmTileFn spmm_tile;
    SoftmaxFn softmax;
    MaskFn mask;
    TransposeFn transpose;
    SddmmFn sddmm;
    SpmmFn spmm;
} g_api{};

// Per device: the status word (device memory) and its host copy, which the kernels write.
struct Status {
    int32_t* word = nullptr;
    volatile int32_t* mirror = nullptr;
} g_status[kMaxDevices];

PyObject* g_warn = nullptr;   // splat_native's one-time warning, until it has been given

struct PythonError {};        // thrown while a Python exception is set

void warn_once(const char* what) {     // 16-bit operands on the CUDA cores; a warning may be an error to the caller
    if (g_warn == nullptr) return;
    PyObject* cb = g_warn;
    g_warn = nullptr;
    PyObject* r = PyObject_CallFunction(cb, "s", what);
    Py_DECREF(cb);
    if (r == nullptr) throw PythonError{};
    Py_DECREF(r);
}
// return codes of the tile and band kernels that mean "use the row kernels": misaligned, unsupported shape, no tensor map
bool not_applicable(int32_t rc) { return rc == -3 || rc == -6 || rc == -7; }
PyObject *k_lin, *k_tr, *k_nnzs, *k_out, *k_scale, *k_path, *k_plan, *k_lse, *k_cached_plan;

inline const at::Tensor* tensor(PyObject* o) {
    return o != nullptr && THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr;
}
inline int dtype_code(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return 0;
        case at::kHalf: return 1;
        case at::kBFloat16: return 2;
        default: return -1;
    }
}
inline const float* meta(const at::Tensor* t, int64_t n, int device) {
    return t != nullptr && t->scalar_type() == at::kFloat && t->is_cuda() && t->get_device() == device &&
                   t->is_contiguous() && t->numel() >= n
               ? static_cast<const float*>(t->const_data_ptr())
               : nullptr;
}
// the 8 plan integers of a tuple
inline bool read_plan(PyObject* o, int32_t (&plan)[8]) {
    if (o == nullptr || !PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 8) return false;
    for (int i = 0; i < 8; ++i) {
        PyObject* v = PyTuple_GET_ITEM(o, i);
        if (!PyLong_Check(v)) return false;
        plan[i] = static_cast<int32_t>(PyLong_AsLong(v));
    }
    return !PyErr_Occurred();
}
inline bool as_long(PyObject* o, long* v) {
    if (o == nullptr || !PyLong_Check(o)) return false;
    *v = PyLong_AsLong(o);
    return !PyErr_Occurred();
}
// The device of an ordinary operand if it is the current one and nothing unusual is going on, else -1.
inline int ordinary_device(const at::Tensor& t) {
    if (!t.is_cuda()) return -1;
    const int dev = t.get_device();
    if (dev < 0 || dev >= kMaxDevices || g_status[dev].word == nullptr || dev != c10::cuda::current_device()) return -1;
    if (*g_status[dev].mirror != 0) return -1;             // an earlier launch gave up: Python raises
    if (const char* e = std::getenv("SPLAT_B200_DEBUG"); e != nullptr && e[0] != 0) return -1;
    return dev;
}
// (B, H, X, Y) with collapsible (B, H)
inline bool flat_bh(const at::Tensor& t, int64_t* stride_bh) {
    const auto st = t.strides();
    const auto sz = t.sizes();
    if (sz[0] > 1 && sz[1] > 1 && st[0] != sz[1] * st[1]) return false;
    *stride_bh = sz[1] > 1 ? st[1] : (sz[0] > 1 ? st[0] : sz[2] * sz[3]);
    return true;
}
inline bool same4(const at::Tensor& t, int64_t a, int64_t b, int64_t c, int64_t d) {
    const auto s = t.sizes();
    return s.size() == 4 && s[0] == a && s[1] == b && s[2] == c && s[3] == d;
}

// plan remembered by splat_native.classify() on the nnzs tensor: ((id, id, version x 3, numel), plan, lin, tr,
// band table, stream it was made on); false if the metadata is not what it was made from.  With `table`, also its address -- null for a pattern without one -- and false if Python has yet to
// make it.  A captured launch gets no table: a replay has to follow the metadata as they are then, and the table's
// memory goes with the Python objects.  The caller knows nothing of the table, so its use on another stream than its own
// is recorded here.
bool cached_plan(PyObject* nnzs_obj, const at::Tensor& nnzs, PyObject* lin_obj, const at::Tensor& lin, PyObject* tr_obj,
                 const at::Tensor& tr, int32_t (&plan)[8], const int32_t** table = nullptr) {
    PyObject* hit = PyObject_GetAttr(nnzs_obj, k_cached_plan);
    if (hit == nullptr) {
        PyErr_Clear();
        return false;
    }
    bool ok = PyTuple_Check(hit) && PyTuple_GET_SIZE(hit) == 6 && PyTuple_GET_ITEM(hit, 2) == lin_obj &&
              PyTuple_GET_ITEM(hit, 3) == tr_obj;
    if (ok) {
        PyObject* key = PyTuple_GET_ITEM(hit, 0);
        const int64_t now[4] = {static_cast<int64_t>(lin._version()), static_cast<int64_t>(tr._version()),
                                static_cast<int64_t>(nnzs._version()), nnzs.numel()};
        ok = PyTuple_Check(key) && PyTuple_GET_SIZE(key) == 6;
        for (int i = 0; ok && i < 4; ++i) {
            long v;
            ok = as_long(PyTuple_GET_ITEM(key, 2 + i), &v) && v == now[i];
        }
        ok = ok && read_plan(PyTuple_GET_ITEM(hit, 1), plan);
    }
    if (ok && table != nullptr) {
        *table = nullptr;
        PyObject* made = PyTuple_GET_ITEM(hit, 4);          // a tensor, False (no such table) or None (not made)
        const at::Tensor* t = tensor(made);
        const auto stream = c10::cuda::getCurrentCUDAStream(t != nullptr ? t->get_device() : -1);
        // (the legacy stream is never captured: asking costs 0.3 us of a small call)
        if (t != nullptr && (stream.stream() == nullptr ||
                             c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None)) {
            if (PyLong_AsVoidPtr(PyTuple_GET_ITEM(hit, 5)) != stream.stream())
                c10::cuda::CUDACachingAllocator::recordStream(t->storage().data_ptr(), stream);
            *table = static_cast<const int32_t*>(t->const_data_ptr());
        }
        ok = ok && made != Py_None;
    }
    Py_DECREF(hit);
    return ok;
}

// 16-bit K^T as a contiguous (B, H, d, n) array of a band pattern that the tensor-core kernels cannot fetch in
// this layout (a tensor map has to start and step on 16 bytes, and strided rows are not contiguous in it): a
// row-major copy, ordered on the current stream, else an undefined tensor.  One pass over K against kernels on
// the CUDA cores that take 10 to 30 times as long.
at::Tensor rows_of_k(const at::Tensor& kt, int64_t ksb, const int32_t (&plan)[8], int64_t L, int64_t d, void* stream) {
    const int64_t n = kt.size(3), bh = kt.size(0) * kt.size(1);
    const int64_t stride = plan[7] > 0 ? plan[1] : 1;
    const bool contiguous = kt.stride(3) == 1 && kt.stride(2) == n && ksb == n * d;
    const bool band = (plan[7] == 0 || plan[1] == plan[2]) && plan[3] == 0 && plan[5] <= n && n == L && d % 8 == 0 && d <= 128;
    const bool direct = kt.stride(2) == 1 || (stride == 1 && n % 8 == 0);
    if (!contiguous || !band || direct || bh > 65535 || g_api.transpose == nullptr) return {};
    at::Tensor rows;
    try {
        rows = at::empty({bh, n, d}, kt.options());
    } catch (const std::exception&) {      // no memory for it: the kernels that need none
        return {};
    }
    if (g_api.transpose(kt.const_data_ptr(), rows.data_ptr(), bh, d, n, stream) != 0) return {};
    return rows;
}

// True if the call was made; false: nothing happened and the Python code decides.
bool fused(const at::Tensor* q, const at::Tensor* kt, const at::Tensor* v, const at::Tensor* out, const at::Tensor* lin,
           const at::Tensor* tr, const at::Tensor* nnzs, float scale, long path, PyObject* plan_obj, const int32_t* table, const at::Tensor* lse) {
    if (!q || !kt || !v || !out || g_api.fused == nullptr || q->dim() != 4 || kt->dim() != 4) return false;
    const int dtype = dtype_code(*q);
    const int dev = ordinary_device(*q);
    if (dtype < 0 || dev < 0 || q->numel() == 0) return false;
    if (kt->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type() || out->scalar_type() != q->scalar_type())
        return false;
    if (!kt->is_cuda() || !v->is_cuda() || !out->is_cuda() || kt->get_device() != dev || v->get_device() != dev ||
        out->get_device() != dev)
        return false;
    const auto qs = q->sizes();
    const int64_t B = qs[0], H = qs[1], L = qs[2], d = qs[3], n_cols = kt->size(3);
    int64_t ksb;
    if (!same4(*kt, B, H, d, n_cols) || !same4(*v, B, H, n_cols, d) || !same4(*out, B, H, L, d) || !flat_bh(*kt, &ksb))
        return false;
    if (!q->is_contiguous() || !v->is_contiguous() || !out->is_contiguous()) return false;
    const float *pl = meta(lin, L, dev), *pt = meta(tr, L, dev), *pn = meta(nnzs, L, dev);
    if (!pl || !pt || !pn) return false;
    float* plse = nullptr;
    if (lse != nullptr) {
        const auto s = lse->sizes();
        if (lse->scalar_type() != at::kFloat || s.size() != 3 || s[0] != B || s[1] != H || s[2] != L ||
            !lse->is_contiguous() || !lse->is_cuda() || lse->get_device() != dev)
            return false;
        plse = static_cast<float*>(lse->data_ptr());
    }
    int32_t plan[8];
    const bool with_plan = path != kPathGeneric;
    if (with_plan && !read_plan(plan_obj, plan)) return false;
    if (nnzs->numel() != L) table = nullptr;       // (made for as many rows as the metadata have)
    int32_t ran = 0;
    void* stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    at::Tensor rows;
    if (dtype != 0 && path == kPathAuto) rows = rows_of_k(*kt, ksb, plan, L, d, stream);
    const bool copied = rows.defined();
    const int32_t rc = g_api.fused(q->const_data_ptr(), copied ? rows.const_data_ptr() : kt->const_data_ptr(), copied ? n_cols * d : ksb,
                                   copied ? d : kt->stride(3), copied ? 1 : kt->stride(2),
                                   v->const_data_ptr(), out->data_ptr(), plse, pl, pt, pn, B * H, L, n_cols, d, scale, dtype,
                                   static_cast<int32_t>(path), with_plan ? plan : nullptr, table, g_status[dev].word, &ran, stream);
    if (rc != 0) return false;
    if (ran != kPathBand && dtype != 0 && path == kPathAuto) warn_once("attention");
    return true;
}

PyObject* yes_or_none(bool yes) {
    if (PyErr_Occurred()) PyErr_Clear();
    if (yes) Py_RETURN_TRUE;
    Py_RETURN_NONE;
}

// Torch throws for tensors it has no data, strides or version of (fake, functional, sparse ones); nothing of that may
// leave through CPython's frames.  Everything of torch that throws comes before a call's launch, so Python can start over.
template <PyObject* (*F)(PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject*, PyObject* const* args, Py_ssize_t n) {
    try {
        return F(args, n);
    } catch (const PythonError&) {
        return nullptr;
    } catch (...) {
        return yes_or_none(false);
    }
}

// module_forward(module.__dict__, [q, kt, v]) -> the module's output, or None
PyObject* module_forward(PyObject* const* args, Py_ssize_t n) {
    if (n != 2 || !PyDict_Check(args[0])) Py_RETURN_NONE;
    PyObject *dict = args[0], *x = args[1];
    PyObject* item[3];
    if (PyList_Check(x) && PyList_GET_SIZE(x) == 3) {
        for (int i = 0; i < 3; ++i) item[i] = PyList_GET_ITEM(x, i);
    } else if (PyTuple_Check(x) && PyTuple_GET_SIZE(x) == 3) {
        for (int i = 0; i < 3; ++i) item[i] = PyTuple_GET_ITEM(x, i);
    } else {
        Py_RETURN_NONE;
    }
    PyObject* out = PyDict_GetItemWithError(dict, k_out);
    PyObject* scale = PyDict_GetItemWithError(dict, k_scale);
    PyObject* lse = PyDict_GetItemWithError(dict, k_lse);
    long path;
    if (out == nullptr || scale == nullptr || !PyFloat_Check(scale) || !as_long(PyDict_GetItemWithError(dict, k_path), &path))
        return yes_or_none(false);
    const at::Tensor* lse_t = nullptr;
    if (lse != nullptr && lse != Py_None && (lse_t = tensor(lse)) == nullptr) return yes_or_none(false);
    PyObject *lin = PyDict_GetItemWithError(dict, k_lin), *tr = PyDict_GetItemWithError(dict, k_tr),
             *nnzs = PyDict_GetItemWithError(dict, k_nnzs);
    const at::Tensor *lin_t = tensor(lin), *tr_t = tensor(tr), *nnzs_t = tensor(nnzs);
    const int32_t* table = nullptr;
    int32_t unused[8];
    if (lin_t && tr_t && nnzs_t && !cached_plan(nnzs, *nnzs_t, lin, *lin_t, tr, *tr_t, unused, &table)) table = nullptr;
    if (!fused(tensor(item[0]), tensor(item[1]), tensor(item[2]), tensor(out), lin_t, tr_t, nnzs_t,
               static_cast<float>(PyFloat_AS_DOUBLE(scale)), path, PyDict_GetItemWithError(dict, k_plan), table, lse_t))
        return yes_or_none(false);
    Py_INCREF(out);
    return out;
}

// sddmm(x, y, output, sTod_lin, sTod_tr, nnzs, trailing_dim, path) -> True, or None
PyObject* sddmm(PyObject* const* a, Py_ssize_t n) {
    long trailing, path;
    if (n != 8 || !as_long(a[6], &trailing) || !as_long(a[7], &path) || path != kPathAuto) return yes_or_none(false);
    const at::Tensor *x = tensor(a[0]), *y = tensor(a[1]), *out = tensor(a[2]), *lin = tensor(a[3]), *tr = tensor(a[4]),
                     *nnzs = tensor(a[5]);
    if (!x || !y || !out || !lin || !tr || !nnzs || g_api.sddmm_band == nullptr || x->dim() != 4 || y->dim() != 4)
        return yes_or_none(false);
    const int dtype = dtype_code(*x), dev = ordinary_device(*x);
    if (dtype < 0 || dev < 0 || x->numel() == 0 || trailing < 1) return yes_or_none(false);
    const auto xs = x->sizes();
    const int64_t B = xs[0], H = xs[1], L = xs[2], d = xs[3], n_cols = y->size(3);
    int64_t ksb;
    if (y->scalar_type() != x->scalar_type() || out->scalar_type() != x->scalar_type() || !y->is_cuda() || !out->is_cuda() ||
        y->get_device() != dev || out->get_device() != dev || !same4(*y, B, H, d, n_cols) || !same4(*out, B, H, L, trailing) ||
        !flat_bh(*y, &ksb) || !x->is_contiguous() || !out->is_contiguous())
        return yes_or_none(false);
    const float *pl = meta(lin, L, dev), *pt = meta(tr, L, dev), *pn = meta(nnzs, L, dev);
    int32_t plan[8];
    const int32_t* table = nullptr;
    if (!pl || !pt || !pn || !cached_plan(a[5], *nnzs, a[3], *lin, a[4], *tr, plan, dtype != 0 && nnzs->numel() == L ? &table : nullptr))
        return yes_or_none(false);
    void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
    at::Tensor rows;
    if (dtype != 0) rows = rows_of_k(*y, ksb, plan, L, d, st);
    const bool copied = rows.defined();
    const void* yp = copied ? rows.const_data_ptr() : y->const_data_ptr();
    const int64_t ksc = copied ? d : y->stride(3), ksk = copied ? 1 : y->stride(2);
    if (copied) ksb = n_cols * d;
    int32_t rc =
        dtype == 0 ? g_api.sddmm_tile(x->const_data_ptr(), yp, ksb, ksc, ksk, out->data_ptr(), pl, pt, pn, B * H,
                                      L, n_cols, d, trailing, dtype, plan, g_status[dev].word, st)
                   : g_api.sddmm_band(x->const_data_ptr(), yp, ksb, ksc, ksk, out->data_ptr(), pl, pt, pn, B * H,
                                      L, n_cols, d, trailing, dtype, plan, table, g_status[dev].word, st);
    if (not_applicable(rc)) {
        if (dtype != 0) warn_once("sddmm");
        rc = g_api.sddmm(x->const_data_ptr(), yp, ksb, ksc, ksk, out->data_ptr(), pl, pt, pn, B * H, L, n_cols, d, trailing, dtype, st);
    }
    return yes_or_none(rc == 0);
}

// spmm(p, v, output, sTod_lin, sTod_tr, nnzs, trailing_dim, path) -> True, or None
PyObject* spmm(PyObject* const* a, Py_ssize_t n) {
    long trailing, path;
    if (n != 8 || !as_long(a[6], &trailing) || !as_long(a[7], &path) || path != kPathAuto) return yes_or_none(false);
    const at::Tensor *x = tensor(a[0]), *y = tensor(a[1]), *out = tensor(a[2]), *lin = tensor(a[3]), *tr = tensor(a[4]),
                     *nnzs = tensor(a[5]);
    if (!x || !y || !out || !lin || !tr || !nnzs || g_api.spmm_band == nullptr || x->dim() != 4 || y->dim() != 4)
        return yes_or_none(false);
    const int dtype = dtype_code(*x), dev = ordinary_device(*x);
    if (dtype < 0 || dev < 0 || x->numel() == 0) return yes_or_none(false);
    const auto xs = x->sizes();
    const int64_t B = xs[0], H = xs[1], L = xs[2], T = xs[3], n_cols = y->size(2), d = y->size(3);
    if (T != trailing || y->scalar_type() != x->scalar_type() || out->scalar_type() != x->scalar_type() || !y->is_cuda() ||
        !out->is_cuda() || y->get_device() != dev || out->get_device() != dev || !same4(*y, B, H, n_cols, d) ||
        !same4(*out, B, H, L, d) || !x->is_contiguous() || !y->is_contiguous() || !out->is_contiguous())
        return yes_or_none(false);
    const float *pl = meta(lin, L, dev), *pt = meta(tr, L, dev), *pn = meta(nnzs, L, dev);
    int32_t plan[8];
    const int32_t* table = nullptr;
    if (!pl || !pt || !pn || !cached_plan(a[5], *nnzs, a[3], *lin, a[4], *tr, plan, dtype != 0 && nnzs->numel() == L ? &table : nullptr))
        return yes_or_none(false);
    void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
    int32_t rc = dtype == 0 ? g_api.spmm_tile(x->const_data_ptr(), y->const_data_ptr(), out->data_ptr(), pl, pt, pn, B * H, L,
                                                    n_cols, d, T, dtype, plan, g_status[dev].word, st)
                                  : g_api.spmm_band(x->const_data_ptr(), y->const_data_ptr(), out->data_ptr(), pl, pt, pn, B * H, L,
                                                    n_cols, d, T, dtype, plan, table, g_status[dev].word, st);
    if (not_applicable(rc)) {
        if (dtype != 0) warn_once("spmm");
        rc = g_api.spmm(x->const_data_ptr(), y->const_data_ptr(), out->data_ptr(), pl, pt, pn, B * H, L, n_cols, d, T, dtype, st);
    }
    return yes_or_none(rc == 0);
}

// softmax(x, output, nnzs, trailing_dim, scale) -> True, or None
PyObject* softmax(PyObject* const* a, Py_ssize_t n) {
    long trailing;
    if (n != 5 || !as_long(a[3], &trailing) || !PyFloat_Check(a[4])) return yes_or_none(false);
    const at::Tensor *x = tensor(a[0]), *out = tensor(a[1]), *nnzs = tensor(a[2]);
    if (!x || !out || !nnzs || g_api.softmax == nullptr || x->dim() != 4) return yes_or_none(false);
    const int dtype = dtype_code(*x), dev = ordinary_device(*x);
    if (dtype < 0 || dev < 0) return yes_or_none(false);
    const auto xs = x->sizes();
    if (xs[3] != trailing || !same4(*out, xs[0], xs[1], xs[2], xs[3]) || out->scalar_type() != x->scalar_type() ||
        !out->is_cuda() || out->get_device() != dev || !x->is_contiguous() || !out->is_contiguous())
        return yes_or_none(false);
    const float* pn = meta(nnzs, xs[2], dev);
    if (!pn) return yes_or_none(false);
    const int32_t rc = g_api.softmax(x->const_data_ptr(), out->data_ptr(), pn, xs[0] * xs[1], xs[2], trailing,
                                     static_cast<float>(PyFloat_AS_DOUBLE(a[4])), dtype, c10::cuda::getCurrentCUDAStream(dev).stream());
    return yes_or_none(rc == 0);
}

// rows_of_k(K^T (B, H, d, n), plan, query rows) -> the row-major copy (B H, n, d) that the calls above work with where they
// need one, or None: for the launchers' Python path.  K^T's device is the current one.
PyObject* rows_of_k(PyObject* const* a, Py_ssize_t n) {
    long L;
    int32_t plan[8];
    int64_t ksb;
    const at::Tensor* kt = n == 3 ? tensor(a[0]) : nullptr;
    if (!kt || kt->dim() != 4 || !kt->is_cuda() || kt->element_size() != 2 || !read_plan(a[1], plan) || !as_long(a[2], &L) ||
        !flat_bh(*kt, &ksb))
        return yes_or_none(false);
    at::Tensor rows = rows_of_k(*kt, ksb, plan, L, kt->size(2), c10::cuda::getCurrentCUDAStream(kt->get_device()).stream());
    return rows.defined() ? THPVariable_Wrap(rows) : yes_or_none(false);
}

// bind(fused, sddmm_band, spmm_band, sddmm_tile_status, spmm_tile_status, softmax, mask, transpose, sddmm, spmm, warn): addresses of the C ABI entry points
// and the function that warns of 16-bit operands on the CUDA-core kernels
PyObject* bind(PyObject*, PyObject* args) {
    unsigned long long f[10];
    PyObject* warn;
    if (!PyArg_ParseTuple(args, "KKKKKKKKKKO", f, f + 1, f + 2, f + 3, f + 4, f + 5, f + 6, f + 7, f + 8, f + 9, &warn)) return nullptr;
    Py_INCREF(warn);
    g_warn = warn;
    g_api.fused = reinterpret_cast<FusedFn>(f[0]);
    g_api.sddmm_band = reinterpret_cast<SddmmBandFn>(f[1]);
    g_api.spmm_band = reinterpret_cast<SpmmBandFn>(f[2]);
    g_api.sddmm_tile = reinterpret_cast<SddmmTileFn>(f[3]);
    g_api.spmm_tile = reinterpret_cast<SpmmTileFn>(f[4]);
    g_api.softmax = reinterpret_cast<SoftmaxFn>(f[5]);
    g_api.mask = reinterpret_cast<MaskFn>(f[6]);
    g_api.transpose = reinterpret_cast<TransposeFn>(f[7]);
    g_api.sddmm = reinterpret_cast<SddmmFn>(f[8]);
    g_api.spmm = reinterpret_cast<SpmmFn>(f[9]);
    Py_RETURN_NONE;
}

// set_status(device index, address of the status word, address of its host copy)
PyObject* set_status(PyObject*, PyObject* args) {
    int dev;
    unsigned long long word, mirror;
    if (!PyArg_ParseTuple(args, "iKK", &dev, &word, &mirror)) return nullptr;
    if (dev >= 0 && dev < kMaxDevices) {
        g_status[dev].mirror = reinterpret_cast<volatile int32_t*>(mirror);
        g_status[dev].word = reinterpret_cast<int32_t*>(word);
    }
    Py_RETURN_NONE;
}

// Scratch of acsr_from_mask calls in progress, per device: `slots` pairs of device words (zero between calls) and
// `slots` page-locked host words.  Kept by splat_native; a slot is taken for the length of a call.
struct MaskWork {
    int32_t* work = nullptr;
    volatile int32_t* host = nullptr;
    uint32_t free = 0;
} g_mask[kMaxDevices];
std::mutex g_mask_mutex;

// set_mask_work(device index, slots, address of the device words, address of the host words)
PyObject* set_mask_work(PyObject*, PyObject* args) {
    int dev, slots;
    unsigned long long work, host;
    if (!PyArg_ParseTuple(args, "iiKK", &dev, &slots, &work, &host)) return nullptr;
    if (dev >= 0 && dev < kMaxDevices && slots > 0 && slots < 32) {
        std::lock_guard<std::mutex> lock(g_mask_mutex);
        g_mask[dev].work = reinterpret_cast<int32_t*>(work);
        g_mask[dev].host = reinterpret_cast<volatile int32_t*>(host);
        g_mask[dev].free = (1u << slots) - 1;
    }
    Py_RETURN_NONE;
}

// acsr_from_mask(uint8 or bool CUDA tensor (rows, cols), block height) -> the tuple create_acsr returns, or None
PyObject* acsr_from_mask(PyObject*, PyObject* const* a, Py_ssize_t n) {
    long height;
    const at::Tensor* m = n == 2 ? tensor(a[0]) : nullptr;
    if (m == nullptr || !as_long(a[1], &height) || g_api.mask == nullptr || m->dim() != 2 || !m->is_cuda() ||
        m->element_size() != 1 || height < 4 || height > 64)
        return yes_or_none(false);
    const int dev = m->get_device();
    const int64_t rows = m->size(0), cols = m->size(1);
    if (dev >= kMaxDevices || dev != c10::cuda::current_device() || rows < 1 || cols < 1 || m->stride(1) != 1 || m->stride(0) < cols)
        return yes_or_none(false);
    int slot = -1;
    {
        std::lock_guard<std::mutex> lock(g_mask_mutex);
        if (g_mask[dev].free != 0) {
            slot = __builtin_ctz(g_mask[dev].free);
            g_mask[dev].free &= g_mask[dev].free - 1;
        }
    }
    if (slot < 0) return yes_or_none(false);
    volatile int32_t* word = g_mask[dev].host + slot;
    const auto stream = c10::cuda::getCurrentCUDAStream(dev);
    at::Tensor t[7];
    int32_t rc = -1, trailing = -1;
    try {
        // (behind the dispatcher: seven trips through it are a quarter of a small call)
        for (int i = 0; i < 7; ++i)
            t[i] = at::Tensor(at::detail::empty_cuda({i < 5 ? rows : (rows + height - 1) / height}, at::kFloat, m->device(), std::nullopt));
        *word = -1;
        float* p[7];
        for (int i = 0; i < 7; ++i) p[i] = static_cast<float*>(t[i].data_ptr());
        rc = g_api.mask(m->const_data_ptr(), rows, cols, m->stride(0), static_cast<int32_t>(height), p[0], p[1], p[2], p[3], p[4],
                        p[5], p[6], g_mask[dev].work + 2 * slot, const_cast<int32_t*>(word), stream.stream());
        if (rc == 0) {
            // The count reaches the host some microseconds before a stream synchronisation would return; work
            // queued before this call, or an error, is left to the synchronisation.  Other threads run meanwhile.
            std::exception_ptr failed;
            Py_BEGIN_ALLOW_THREADS
            const auto until = std::chrono::steady_clock::now() + std::chrono::milliseconds(2);
            while ((trailing = *word) < 0)
                if (std::chrono::steady_clock::now() > until) break;
            if (trailing < 0) {
                try {
                    c10::cuda::stream_synchronize(stream.stream());
                    trailing = *word;
                } catch (...) {
                    failed = std::current_exception();
                }
            }
            Py_END_ALLOW_THREADS
            if (failed) std::rethrow_exception(failed);
        }
    } catch (const std::exception& e) {
        if (rc == 0) {                  // launched, and the device reports an error: the slot stays taken
            PyErr_SetString(PyExc_RuntimeError, e.what());
            return nullptr;
        }
    }
    {
        std::lock_guard<std::mutex> lock(g_mask_mutex);
        g_mask[dev].free |= 1u << slot;
    }
    if (rc != 0 || trailing < 0) return yes_or_none(false);
    PyObject* out = PyTuple_New(8);
    if (out == nullptr) return nullptr;
    for (int i = 0; i < 8; ++i)
        PyTuple_SET_ITEM(out, i, i == 5 ? PyLong_FromLong(trailing) : THPVariable_Wrap(t[i < 5 ? i : i - 1]));
    return out;
}

// record_pinned(host tensor, stream id, device index, device type): a copy from or to the tensor has been queued on the
// stream by other means than torch's copy_().  The page-locked allocator then keeps the block, once it is
// freed, until what the stream holds at that time is done; memory that is not the allocator's is left alone.
PyObject* record_pinned(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const at::Tensor* t = n == 4 ? tensor(a[0]) : nullptr;
    long id, device, type;
    if (t == nullptr || !as_long(a[1], &id) || !as_long(a[2], &device) || !as_long(a[3], &type)) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "record_pinned(tensor, stream id, device index, device type)");
        return nullptr;
    }
    try {
        const auto stream = c10::Stream::unpack3(id, static_cast<c10::DeviceIndex>(device), static_cast<c10::DeviceType>(type));
        if (t->device().is_cpu())
            at::getHostAllocator(at::kCUDA)->record_event(const_cast<void*>(t->const_data_ptr()),
                                                          t->storage().data_ptr().get_context(), stream);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    {"set_status", set_status, METH_VARARGS, nullptr},
    {"module_forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(guarded<module_forward>)), METH_FASTCALL, nullptr},
    {"sddmm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(guarded<sddmm>)), METH_FASTCALL, nullptr},
    {"spmm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(guarded<spmm>)), METH_FASTCALL, nullptr},
    {"set_mask_work", set_mask_work, METH_VARARGS, nullptr},
    {"acsr_from_mask", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(acsr_from_mask)), METH_FASTCALL, nullptr},
    {"rows_of_k", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(guarded<rows_of_k>)), METH_FASTCALL, nullptr},
    {"record_pinned", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(record_pinned)), METH_FASTCALL, nullptr},
    {"softmax", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(guarded<softmax>)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "splat_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_splat_host() {
    k_lin = PyUnicode_InternFromString("sTod_linear_transformations");
    k_tr = PyUnicode_InternFromString("sTod_translations");
    k_nnzs = PyUnicode_InternFromString("nnzs");
    k_out = PyUnicode_InternFromString("rspmm_output");
    k_scale = PyUnicode_InternFromString("scale");
    k_path = PyUnicode_InternFromString("path");
    k_plan = PyUnicode_InternFromString("plan");
    k_lse = PyUnicode_InternFromString("lse");
    k_cached_plan = PyUnicode_InternFromString("_splat_plan");
    return PyModule_Create(&module_def);
}
