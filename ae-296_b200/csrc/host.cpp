// Native host path of the Python ops: from tensors and pool objects to one C-ABI call.
//
// A decode step makes 64 to 160 applies, each of a few microseconds on the GPU, so what Python spends per
// call decides the step's time.  Reading the tensors through ctypes (a data_ptr() call, two stride() calls
// and a structure field per operand, and a NumPy pass over the ranks) took 35-40 us per fused apply and
// 21 us per operator call; here the operands are read from the tensor objects directly and the whole call
// costs about 1 us besides the CUDA launches.
//
// The functions take the short path only: operands that are exactly what the ops document.  Anything else
// (a wrong shape or type, a table that has to grow) returns kSlow and the Python code beside the call
// raises the error or prepares what is missing.  The GIL is given up around the CUDA calls.
//
// Reading a tensor can throw (one without storage, as under vmap or in a tracer; a driver that is not usable):
// every entry point turns that into the Python exception the same access raises in Python, and no tensor is
// touched while the GIL is given up.
#include <Python.h>

#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>

#include <string.h>

#include <memory>
#include <mutex>
#include <vector>

#include "b200_lora.h"

namespace {

constexpr long kSlow = 1;          // "not for the short path" (status codes are <= 0)

// attribute names, interned once
PyObject *s_wa, *s_wb, *s_h_in, *s_h_out, *s_ranks, *s_scalings, *s_cum_ranks, *s_n_adapters, *s_n_layers, *s_r_pool,
    *s_packed, *s_ranks_host, *s_cum_host, *s_buf, *s_nbytes, *s_max_tokens, *s_n_tokens;

struct Ref {                       // owned reference
    PyObject* o;
    explicit Ref(PyObject* p) : o(p) {}
    ~Ref() { Py_XDECREF(o); }
    Ref(const Ref&) = delete;
    Ref& operator=(const Ref&) = delete;
    explicit operator bool() const { return o != nullptr; }
};

bool get_int(PyObject* obj, PyObject* name, int64_t& out) {
    Ref v(PyObject_GetAttr(obj, name));
    if (!v) return false;
    out = PyLong_AsLongLong(v.o);
    return !(out == -1 && PyErr_Occurred());
}

// A CUDA tensor attribute; None gives a null pointer when `optional`.
bool get_ptr(PyObject* obj, PyObject* name, bool optional, const void*& out, at::ScalarType* dtype = nullptr) {
    Ref v(PyObject_GetAttr(obj, name));
    if (!v) return false;
    out = nullptr;
    if (v.o == Py_None) return optional;
    if (!THPVariable_Check(v.o)) return false;
    const at::Tensor& t = THPVariable_Unpack(v.o);
    if (!t.is_cuda()) return false;
    out = t.data_ptr();
    if (dtype) *dtype = t.scalar_type();
    return true;
}

bool dtype_code(at::ScalarType t, int& code) {
    if (t == at::kHalf) code = B200_LORA_F16;
    else if (t == at::kBFloat16) code = B200_LORA_BF16;
    else if (t == at::kFloat) code = B200_LORA_F32;
    else return false;
    return true;
}

void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// The adapter table of a pool object, or of a ctypes structure of the same layout.  The ranks are read from
// the pool's host copy on every call: a pool manager may change a slot's rank between calls.  Host tables of other
// types than int32 ranks and int64 prefixes are the Python code's to read.
bool read_adapters(PyObject* obj, b200_lora_adapters& ad) {
    if (PyObject_CheckBuffer(obj)) {
        Py_buffer b;
        if (PyObject_GetBuffer(obj, &b, PyBUF_SIMPLE) != 0) return false;
        const bool ok = b.len == (Py_ssize_t)sizeof(ad);
        if (ok) memcpy(&ad, b.buf, sizeof(ad));
        PyBuffer_Release(&b);
        return ok;
    }
    memset(&ad, 0, sizeof(ad));
    int64_t n, l, r, packed;
    const void *ranks, *scalings, *cum;
    if (!get_int(obj, s_n_adapters, n) || !get_int(obj, s_n_layers, l) || !get_int(obj, s_r_pool, r) ||
        !get_int(obj, s_packed, packed) || !get_ptr(obj, s_ranks, true, ranks) ||
        !get_ptr(obj, s_scalings, true, scalings) || !get_ptr(obj, s_cum_ranks, true, cum))
        return false;
    ad.ranks = static_cast<const int32_t*>(ranks);
    ad.scalings = static_cast<const float*>(scalings);
    ad.cum_ranks = static_cast<const int64_t*>(cum);
    ad.n_adapters = (int32_t)n; ad.n_layers = (int32_t)l; ad.r_pool = (int32_t)r; ad.packed = packed ? 1 : 0;
    ad.scale = 1.0f;
    Ref rh(PyObject_GetAttr(obj, s_ranks_host)), ch(PyObject_GetAttr(obj, s_cum_host));
    if (!rh || !ch || !PyObject_CheckBuffer(rh.o) || !PyObject_CheckBuffer(ch.o)) return false;
    Py_buffer b;
    if (PyObject_GetBuffer(rh.o, &b, PyBUF_ND | PyBUF_FORMAT) != 0) return false;
    bool ok = b.format && b.itemsize == 4 && !strcmp(b.format, "i") && b.len == 4 * n;
    if (ok) {
        const int32_t* h = static_cast<const int32_t*>(b.buf);
        bool pow2 = true;
        for (int64_t i = 0; i < n; ++i)
            pow2 &= packed ? (h[i] == 8) | (h[i] == 16) | (h[i] == 32) | (h[i] == 64) : h[i] == (int32_t)r;
        ad.ranks_pow2 = pow2 && (packed || r == 8 || r == 16 || r == 32 || r == 64);
    }
    PyBuffer_Release(&b);
    if (!ok || PyObject_GetBuffer(ch.o, &b, PyBUF_ND | PyBUF_FORMAT) != 0) return false;
    ok = b.format && b.itemsize == 8 && (!strcmp(b.format, "l") || !strcmp(b.format, "q")) && b.len >= 8;
    if (ok) ad.total_rank = static_cast<const int64_t*>(b.buf)[b.len / 8 - 1];
    PyBuffer_Release(&b);
    return ok;
}

struct PlanRef { void* buf; size_t nbytes; int max_tokens; int64_t n_tokens; };
bool read_plan(PyObject* plan, PlanRef& p) {
    const void* buf;
    int64_t nb, cap;
    if (!get_ptr(plan, s_buf, false, buf) || !get_int(plan, s_nbytes, nb) || !get_int(plan, s_max_tokens, cap) ||
        !get_int(plan, s_n_tokens, p.n_tokens))
        return false;
    p.buf = const_cast<void*>(buf); p.nbytes = (size_t)nb; p.max_tokens = (int)cap;
    return true;
}

PyObject* slow() {                 // an attribute or conversion error on the short path is the slow path's to report
    PyErr_Clear();
    return PyLong_FromLong(kSlow);
}

// An entry point whose C++ exceptions become Python exceptions.
using FastCall = PyObject* (*)(PyObject*, PyObject* const*, Py_ssize_t);
template <FastCall F>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
    try {
        return F(self, args, nargs);
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

// apply(projs, plan, layer, workspace, flags, adapters | None) -> status
PyObject* py_apply(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 6) return slow();
    PyObject* const* items;
    Py_ssize_t n;
    if (PyList_CheckExact(args[0])) { items = &PyList_GET_ITEM(args[0], 0); n = PyList_GET_SIZE(args[0]); if (n == 0) return slow(); }
    else if (PyTuple_CheckExact(args[0])) { n = PyTuple_GET_SIZE(args[0]); if (n == 0) return slow(); items = &PyTuple_GET_ITEM(args[0], 0); }
    else return slow();
    if (n > B200_LORA_MAX_PROJ) return slow();
    PlanRef plan;
    if (!read_plan(args[1], plan)) return slow();
    const long layer = PyLong_AsLong(args[2]), flags = PyLong_AsLong(args[4]);
    if (PyErr_Occurred()) return slow();
    const void* ws;
    int64_t ws_bytes;
    if (!get_ptr(args[3], s_buf, false, ws) || !get_int(args[3], s_nbytes, ws_bytes)) return slow();
    b200_lora_proj pj[B200_LORA_MAX_PROJ];
    int io = 0, yd = 0;
    void* stream = nullptr;
    PyObject* pool0 = nullptr;
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject* t = items[i];
        if (!PyTuple_CheckExact(t) || PyTuple_GET_SIZE(t) != 3) return slow();
        PyObject *ox = PyTuple_GET_ITEM(t, 0), *oy = PyTuple_GET_ITEM(t, 1), *pool = PyTuple_GET_ITEM(t, 2);
        if (!THPVariable_Check(ox) || !THPVariable_Check(oy)) return slow();
        const at::Tensor &x = THPVariable_Unpack(ox), &y = THPVariable_Unpack(oy);
        if (!x.is_cuda() || !y.is_cuda() || x.dim() != 2 || y.dim() != 2) return slow();
        int64_t h_in, h_out;
        const void *wa, *wb;
        at::ScalarType wt;
        if (!get_int(pool, s_h_in, h_in) || !get_int(pool, s_h_out, h_out) || !get_ptr(pool, s_wa, false, wa, &wt) ||
            !get_ptr(pool, s_wb, false, wb))
            return slow();
        int xi, yi;
        if (x.size(0) != plan.n_tokens || y.size(0) != plan.n_tokens || x.size(1) != h_in || y.size(1) != h_out ||
            x.stride(1) != 1 || y.stride(1) != 1 || x.scalar_type() != wt || !dtype_code(x.scalar_type(), xi) ||
            !dtype_code(y.scalar_type(), yi) || xi == B200_LORA_F32 || (yi != xi && yi != B200_LORA_F32))
            return slow();
        if (i == 0) { io = xi; yd = yi; stream = stream_of(x); pool0 = pool; }
        else if (xi != io || yi != yd) return slow();
        pj[i] = b200_lora_proj{x.data_ptr(), y.data_ptr(), wa, wb, x.stride(0), y.stride(0), (int32_t)h_in, (int32_t)h_out};
    }
    b200_lora_adapters ad;
    if (!read_adapters(args[5] == Py_None ? pool0 : args[5], ad)) return slow();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = b200_lora_apply(pj, (int32_t)n, &ad, plan.buf, plan.max_tokens, (int32_t)plan.n_tokens, (int32_t)layer, io, yd, (int32_t)flags,
                         const_cast<void*>(ws), (size_t)ws_bytes, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

// plan_build(plan, ids, pool | adapters) -> status; also sets plan.n_tokens
PyObject* py_plan_build(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    PlanRef plan;
    b200_lora_adapters ad;
    if (nargs != 3 || !THPVariable_Check(args[1]) || !read_plan(args[0], plan) || !read_adapters(args[2], ad)) return slow();
    const at::Tensor& ids = THPVariable_Unpack(args[1]);
    if (!ids.is_cuda() || !ids.is_contiguous() || (ids.scalar_type() != at::kInt && ids.scalar_type() != at::kLong)) return slow();
    const int64_t n = ids.numel();
    Ref num(PyLong_FromLongLong(n));
    void* stream = stream_of(ids);
    const void* ids_ptr = ids.data_ptr();
    const int is_i64 = ids.scalar_type() == at::kLong;
    if (!num || PyObject_SetAttr(args[0], s_n_tokens, num.o) != 0) return slow();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = b200_lora_plan_build(plan.buf, plan.nbytes, plan.max_tokens, ids_ptr, is_i64, (int32_t)n, &ad, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

// plan_segments(plan, seg_starts, seg_adapter, n_tokens, pool | adapters) -> status; also sets plan.n_tokens.
// seg_starts has more entries than seg_adapter, or as many (then the last segment ends at n_tokens).
PyObject* py_plan_segments(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    PlanRef plan;
    b200_lora_adapters ad;
    if (nargs != 5 || !THPVariable_Check(args[1]) || !THPVariable_Check(args[2]) || !read_plan(args[0], plan) || !read_adapters(args[4], ad))
        return slow();
    const at::Tensor &starts = THPVariable_Unpack(args[1]), &owner = THPVariable_Unpack(args[2]);
    if (!starts.is_cuda() || !owner.is_cuda() || starts.scalar_type() != at::kInt || owner.scalar_type() != at::kInt ||
        !starts.is_contiguous() || !owner.is_contiguous())
        return slow();
    const int64_t n = owner.numel(), t = PyLong_AsLongLong(args[3]);
    if (PyErr_Occurred() || starts.numel() < n) return slow();
    void* stream = stream_of(starts);
    const bool ends = starts.numel() > n;
    const int32_t *sp = static_cast<const int32_t*>(starts.data_ptr()), *op = static_cast<const int32_t*>(owner.data_ptr());
    if (PyObject_SetAttr(args[0], s_n_tokens, args[3]) != 0) return slow();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = (ends ? b200_lora_plan_from_segments : b200_lora_plan_from_requests)(plan.buf, plan.nbytes, plan.max_tokens, sp, op, (int32_t)n,
                                                                               (int32_t)t, &ad, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

// ---- the reference's operator call ---------------------------------------------------------------
// Plan and workspace behind add_lora_bgmv for one (device, stream, graph capture): the memory belongs to the
// Python side, which registers it here; what the plan was built from is kept here.  A capture has an entry of
// its own, since every replay writes the plan again: an eager call must not find its plan replaced by a replay.
// The index tensor is held weakly: its object stays comparable by address, its storage does not stay alive.
// `mu` holds a call's enqueues together: another thread's plan must not come between a call's plan, its key and
// its apply.  It is only taken without the GIL (a launch may wait for the GPU, and the GPU for a host callback).
struct OpEntry {
    std::mutex mu;
    void* stream = nullptr;
    int device = -1;
    unsigned long long capture = 0;
    void *plan = nullptr, *ws = nullptr;
    size_t plan_bytes = 0, ws_bytes = 0;
    int cap_t = 0, cap_n = 0, cap_h = 0;
    bool built = false;
    c10::weak_intrusive_ptr<c10::TensorImpl> ids{c10::intrusive_ptr<c10::TensorImpl, c10::UndefinedTensorImpl>()};
    const void* ids_ptr = nullptr;
    uint32_t version = 0;
    int ids_type = 0, t = 0, n = 0, r = 0;
    float scale = 0.f;
};
using OpRef = std::shared_ptr<OpEntry>;
std::vector<OpRef>* g_ops;         // guarded by the GIL; a process has a handful of streams

OpRef find_op(void* stream, int device, unsigned long long capture) {
    for (const OpRef& e : *g_ops)
        if (e->stream == stream && e->device == device && e->capture == capture) return e;
    return nullptr;
}

struct NoGil {
    PyThreadState* state;
    NoGil() : state(PyEval_SaveThread()) {}
    ~NoGil() { PyEval_RestoreThread(state); }
};

// bgmv_register(stream, device, capture, plan_ptr, plan_bytes, ws_ptr, ws_bytes, cap_t, cap_n, cap_h)
// A stream is in one capture at a time: entries of its earlier captures go.
bool register_op(PyObject* args) {
    unsigned long long stream, capture, plan, ws, plan_bytes, ws_bytes;
    int device, t, n, h;
    if (!PyArg_ParseTuple(args, "KiKKKKKiii", &stream, &device, &capture, &plan, &plan_bytes, &ws, &ws_bytes, &t, &n, &h)) return false;
    void* s = reinterpret_cast<void*>(stream);
    for (size_t i = g_ops->size(); i-- > 0;) {
        const OpEntry& o = *(*g_ops)[i];
        if (o.stream == s && o.device == device && o.capture != 0 && o.capture != capture) g_ops->erase(g_ops->begin() + i);
    }
    OpRef e = find_op(s, device, capture);
    if (!e) {
        e = std::make_shared<OpEntry>();
        e->stream = s; e->device = device; e->capture = capture;
        g_ops->push_back(e);
    }
    NoGil nogil;
    std::lock_guard<std::mutex> lock(e->mu);
    e->plan = reinterpret_cast<void*>(plan); e->plan_bytes = plan_bytes;
    e->ws = reinterpret_cast<void*>(ws); e->ws_bytes = ws_bytes;
    e->cap_t = t; e->cap_n = n; e->cap_h = h; e->built = false;
    return true;
}
PyObject* py_bgmv_register(PyObject*, PyObject* args) {
    try {
        if (!register_op(args)) return nullptr;
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
    Py_RETURN_NONE;
}

// bgmv_forget(): the plans must be rebuilt on their next use
PyObject* py_bgmv_forget(PyObject*, PyObject* const*, Py_ssize_t) {
    const std::vector<OpRef> all(*g_ops);
    {
        NoGil nogil;
        for (const OpRef& e : all) {
            std::lock_guard<std::mutex> lock(e->mu);
            e->built = false;
        }
    }
    Py_RETURN_NONE;
}

struct OpArgs {
    const at::Tensor *y, *x, *wa, *wb, *ids;
    int64_t t, n, l, r, h_in, h_out;
    long layer;
    double scale;
    int io;
};
// (y, x, wa_T_all, wb_T_all, indicies, layer_idx, scale), checked as the op documents them
bool read_op(PyObject* const* args, OpArgs& a) {
    for (int i = 0; i < 5; ++i)
        if (!THPVariable_Check(args[i])) return false;
    a.y = &THPVariable_Unpack(args[0]); a.x = &THPVariable_Unpack(args[1]); a.wa = &THPVariable_Unpack(args[2]);
    a.wb = &THPVariable_Unpack(args[3]); a.ids = &THPVariable_Unpack(args[4]);
    const at::Tensor &y = *a.y, &x = *a.x, &wa = *a.wa, &wb = *a.wb, &ids = *a.ids;
    if (!y.is_cuda() || !x.is_cuda() || !wa.is_cuda() || !wb.is_cuda() || !ids.is_cuda()) return false;
    if (wa.dim() != 4 || wb.dim() != 4 || x.dim() != 2 || y.dim() != 2) return false;
    a.n = wa.size(0); a.l = wa.size(1); a.r = wa.size(2); a.h_in = wa.size(3); a.h_out = wb.size(2); a.t = x.size(0);
    if (wb.size(0) != a.n || wb.size(1) != a.l || wb.size(3) != a.r || x.size(1) != a.h_in || y.size(0) != a.t ||
        y.size(1) != a.h_out || ids.numel() != a.t)
        return false;
    if (!y.is_contiguous() || !x.is_contiguous() || !wa.is_contiguous() || !wb.is_contiguous() || !ids.is_contiguous()) return false;
    const at::ScalarType dt = x.scalar_type();
    if (y.scalar_type() != dt || wa.scalar_type() != dt || wb.scalar_type() != dt || !dtype_code(dt, a.io) || a.io == B200_LORA_F32) return false;
    if (ids.scalar_type() != at::kInt && ids.scalar_type() != at::kLong) return false;
    a.layer = PyLong_AsLong(args[5]);
    if (PyErr_Occurred()) return false;
    a.scale = PyFloat_AsDouble(args[6]);
    return !PyErr_Occurred();
}

// bgmv(y, x, wa_T_all, wb_T_all, indicies, layer_idx, scale) -> status; kSlow also while the plan and workspace of
// this stream (or of the capture it is in) are missing or too small
PyObject* py_bgmv(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    OpArgs a;
    if (nargs != 7 || !read_op(args, a)) return slow();
    void* stream = stream_of(*a.x);
    unsigned long long cap = 0;
    int rc = b200_lora_stream_capture_id(stream, &cap);
    if (rc) return PyLong_FromLong(rc);
    const OpRef e = find_op(stream, a.ids->get_device(), cap);
    if (!e) return slow();
    const bool versioned = !a.ids->is_inference();                  // inference tensors have no version counter
    const uint32_t version = versioned ? a.ids->_version() : 0;
    const int ids_type = (int)a.ids->scalar_type();
    const float scale = (float)a.scale;
    const void* ids_ptr = a.ids->data_ptr();
    c10::weak_intrusive_ptr<c10::TensorImpl> ids(a.ids->getIntrusivePtr());
    b200_lora_adapters ad;
    memset(&ad, 0, sizeof(ad));
    ad.n_adapters = (int32_t)a.n; ad.n_layers = (int32_t)a.l; ad.r_pool = (int32_t)a.r; ad.scale = scale;
    const b200_lora_proj pj{a.x->data_ptr(), a.y->data_ptr(), a.wa->data_ptr(), a.wb->data_ptr(), a.h_in, a.h_out, (int32_t)a.h_in, (int32_t)a.h_out};
    {
        NoGil nogil;
        std::lock_guard<std::mutex> lock(e->mu);
        if (a.t > e->cap_t || a.n > e->cap_n || a.h_in > e->cap_h) rc = kSlow;
        const bool same = e->built && versioned && e->ids._unsafe_get_target() == ids._unsafe_get_target() && e->ids_ptr == ids_ptr &&
                          e->version == version && e->ids_type == ids_type && e->t == a.t && e->n == a.n && e->r == a.r && e->scale == scale;
        if (rc == 0 && !same) {
            e->built = false;
            rc = b200_lora_plan_build(e->plan, e->plan_bytes, e->cap_t, ids_ptr, ids_type == (int)at::kLong, (int32_t)a.t, &ad, stream);
            if (rc == 0) {
                e->built = true;
                std::swap(e->ids, ids);                             // the former one is released with the GIL held
                e->ids_ptr = ids_ptr; e->version = version; e->ids_type = ids_type;
                e->t = (int)a.t; e->n = (int)a.n; e->r = (int)a.r; e->scale = scale;
            }
        }
        if (rc == 0)
            rc = b200_lora_apply(&pj, 1, &ad, e->plan, e->cap_t, (int32_t)a.t, (int32_t)a.layer, a.io, a.io, B200_LORA_NO_TENSOR, e->ws, e->ws_bytes, stream);
    }
    return rc == kSlow ? slow() : PyLong_FromLong(rc);
}

// bgmv_static(y, x, wa_T_all, wb_T_all, indicies, layer_idx, scale) -> status
PyObject* py_bgmv_static(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    OpArgs a;
    if (nargs != 7 || !read_op(args, a)) return slow();
    void* stream = stream_of(*a.x);
    void* y = a.y->data_ptr();
    const void *x = a.x->data_ptr(), *wa = a.wa->data_ptr(), *wb = a.wb->data_ptr(), *ids = a.ids->data_ptr();
    const int is_i64 = a.ids->scalar_type() == at::kLong;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = b200_add_lora_bgmv_static(y, x, wa, wb, ids, is_i64, (int32_t)a.t, (int32_t)a.h_in, (int32_t)a.h_out, (int32_t)a.n,
                                   (int32_t)a.l, (int32_t)a.r, (int32_t)a.layer, (float)a.scale, a.io, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

// (current stream of the tensor's device, identifier of the capture it is in or 0)
PyObject* stream_and_capture(PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 1 || !THPVariable_Check(args[0]) || !THPVariable_Unpack(args[0]).is_cuda()) {
        PyErr_SetString(PyExc_ValueError, "a CUDA tensor expected");
        return nullptr;
    }
    void* stream = stream_of(THPVariable_Unpack(args[0]));
    unsigned long long cap = 0;
    const int rc = b200_lora_stream_capture_id(stream, &cap);
    if (rc) {
        PyErr_Format(PyExc_RuntimeError, "stream capture status: %s", b200_lora_last_cuda_error());
        return nullptr;
    }
    return Py_BuildValue("(KK)", reinterpret_cast<unsigned long long>(stream), cap);
}
// stream_key(tensor) -> (stream, capture)
PyObject* py_stream_key(PyObject*, PyObject* const* args, Py_ssize_t nargs) { return stream_and_capture(args, nargs); }

// use_key(tensor) -> ((stream, capture), address, version, *sizes, *strides): equal for two uses of the same values in one place
PyObject* py_use_key(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    Ref where(stream_and_capture(args, nargs));
    if (!where) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(args[0]);
    const unsigned long long ptr = reinterpret_cast<uintptr_t>(t.data_ptr());
    const unsigned long version = t._version();                     // (throws for an inference tensor)
    const int64_t dim = t.dim();
    Ref key(PyTuple_New(3 + 2 * dim));
    if (!key) return nullptr;
    Py_INCREF(where.o);
    PyTuple_SET_ITEM(key.o, 0, where.o);
    for (int64_t i = 0; i < 2 + 2 * dim; ++i) {
        PyObject* v = i == 0 ? PyLong_FromUnsignedLongLong(ptr) : i == 1 ? PyLong_FromUnsignedLong(version)
                      : PyLong_FromLongLong(i < 2 + dim ? t.size(i - 2) : t.stride(i - 2 - dim));
        if (!v) return nullptr;
        PyTuple_SET_ITEM(key.o, 1 + i, v);
    }
    Py_INCREF(key.o);
    return key.o;
}

PyMethodDef kMethods[] = {
    {"apply", (PyCFunction)(void*)guarded<py_apply>, METH_FASTCALL, nullptr},
    {"plan_build", (PyCFunction)(void*)guarded<py_plan_build>, METH_FASTCALL, nullptr},
    {"plan_segments", (PyCFunction)(void*)guarded<py_plan_segments>, METH_FASTCALL, nullptr},
    {"bgmv", (PyCFunction)(void*)guarded<py_bgmv>, METH_FASTCALL, nullptr},
    {"bgmv_static", (PyCFunction)(void*)guarded<py_bgmv_static>, METH_FASTCALL, nullptr},
    {"stream_key", (PyCFunction)(void*)guarded<py_stream_key>, METH_FASTCALL, nullptr},
    {"use_key", (PyCFunction)(void*)guarded<py_use_key>, METH_FASTCALL, nullptr},
    {"bgmv_register", py_bgmv_register, METH_VARARGS, nullptr},
    {"bgmv_forget", (PyCFunction)(void*)guarded<py_bgmv_forget>, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_b200host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200host(void) {
    struct { PyObject** slot; const char* name; } names[] = {
        {&s_wa, "wa"}, {&s_wb, "wb"}, {&s_h_in, "h_in"}, {&s_h_out, "h_out"}, {&s_ranks, "ranks"}, {&s_scalings, "scalings"},
        {&s_cum_ranks, "cum_ranks"}, {&s_n_adapters, "n_adapters"}, {&s_n_layers, "n_layers"}, {&s_r_pool, "r_pool"},
        {&s_packed, "packed"}, {&s_ranks_host, "ranks_host"}, {&s_cum_host, "cum_host"}, {&s_buf, "buf"}, {&s_nbytes, "nbytes"},
        {&s_max_tokens, "max_tokens"}, {&s_n_tokens, "n_tokens"}};
    for (auto& e : names)
        if (!(*e.slot = PyUnicode_InternFromString(e.name))) return nullptr;
    g_ops = new std::vector<OpRef>();
    return PyModule_Create(&kModule);
}
