// Native host layer of the Python mirror (deers_b200/ops.py): one CPython call per operator.
//
// What bounds the small calls of the operator interface is the host, not the GPU: around a decode step's 5 - 7 us of kernels
// the same call spent 28 us of Python on argument checks, on filling a ctypes descriptor stride by
// stride and on allocating through the dispatcher (9 us now).  Here the checks, the output and workspace
// allocations (torch's caching allocator, without the dispatcher) and the C-ABI call happen in one native function.
// The functions answer None for anything they do not take as it is (wrong type, shape, device or a layout
// that needs compaction); the Python mirror then raises the matching error or compacts and calls again, saying so: what is
// still not to the library's liking (a head_dim, a contiguous tensor off a 16-byte boundary) is refused with its status.
// Allocations and library calls run without the interpreter lock (a launch waits while the device's queue is full); a lock
// per context keeps the threads that share a stream, and so a context, apart.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string.h>

#include <memory>
#include <mutex>
#include <vector>

#include "../../include/deers_b200.h"

namespace {

PyObject* g_make_context = nullptr;      // ops.Context: device index -> handle as an int
PyObject* g_raise_status = nullptr;      // (status, handle) -> raises CudaError

struct Ctx { int device; cudaStream_t stream; deers_ctx* handle; std::mutex mu; };
std::vector<std::unique_ptr<Ctx>> g_contexts;        // guarded by the GIL; the Python side keeps every context alive

// The library context of the tensor's device and torch's current stream there; nullptr with an exception set.
Ctx* context_for(int device) {
    const cudaStream_t s = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
    for (const auto& e : g_contexts)
        if (e->stream == s && e->device == device) return e.get();
    PyObject* r = PyObject_CallFunction(g_make_context, "i", device);
    if (!r) return nullptr;
    void* p = PyLong_AsVoidPtr(r);
    Py_DECREF(r);
    if (!p) return nullptr;
    for (const auto& e : g_contexts)                 // another thread may have got here while Python ran
        if (e->stream == s && e->device == device) return e.get();
    std::unique_ptr<Ctx> e(new Ctx());
    e->device = device; e->stream = s; e->handle = (deers_ctx*)p;
    g_contexts.push_back(std::move(e));
    return g_contexts.back().get();
}

// The part of an operator that touches no Python object.
struct NoGil {
    PyThreadState* state;
    NoGil() : state(PyEval_SaveThread()) {}
    ~NoGil() { PyEval_RestoreThread(state); }
    NoGil(const NoGil&) = delete;
    NoGil& operator=(const NoGil&) = delete;
};

PyObject* fail(int status, const Ctx* ctx) {
    PyObject* r = PyObject_CallFunction(g_raise_status, "iK", status, (unsigned long long)(uintptr_t)ctx->handle);
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "deers_b200 call failed");
    return nullptr;
}

inline const at::Tensor* tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

inline int dtype_code(const at::Tensor& t) {
    return t.scalar_type() == at::kHalf ? DEERS_F16 : t.scalar_type() == at::kFloat ? DEERS_F32 : -1;
}

// 4-D, on a CUDA device, f16 or f32: the library can be asked.
inline bool offerable(const at::Tensor& t) { return t.dim() == 4 && t.is_cuda() && dtype_code(t) >= 0; }
// The same, and the kernels can read it in place (ops._usable).
inline bool usable(const at::Tensor& t) {
    if (!offerable(t) || t.stride(3) != 1) return false;
    const int64_t align = t.scalar_type() == at::kHalf ? 16 : 4, es = t.element_size();
    if ((uintptr_t)t.data_ptr() % align) return false;
    // a repeated (expanded) axis is compacted where the tile is wider than the row: TMA maps want real strides
    const bool narrow = es == 2 && t.size(3) != 64 && t.size(3) != 128;
    for (int i = 0; i < 3; ++i)
        if (t.size(i) != 1 && ((t.stride(i) * es) % align || (narrow && t.stride(i) == 0))) return false;
    return true;
}
inline bool same(const at::Tensor& a, const at::Tensor& b) {
    return a.sizes() == b.sizes() && a.scalar_type() == b.scalar_type() && a.get_device() == b.get_device();
}
inline void put_strides(int64_t (&dst)[4], const at::Tensor& t) {
    for (int i = 0; i < 4; ++i) dst[i] = t.stride(i);
}
inline at::Tensor empty_like_of(at::IntArrayRef sizes, at::ScalarType st, const at::Tensor& like) {
    return at::Tensor(at::detail::empty_cuda(sizes, st, like.device(), c10::nullopt));
}
inline at::Tensor scratch(size_t bytes, const at::Tensor& like) {
    const int64_t n[1] = {(int64_t)bytes};
    return empty_like_of(at::IntArrayRef(n, 1), at::kByte, like);
}
inline PyObject* wrap2(at::Tensor a, at::Tensor b) {
    PyObject* r = PyTuple_New(2);
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(std::move(a)));
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(std::move(b)));
    return r;
}

void fill_desc(deers_attn_desc* d, const at::Tensor& q, double scale, int causal) {
    memset(d, 0, sizeof(*d));
    d->B = (int)q.size(0); d->H = (int)q.size(1); d->T = (int)q.size(2); d->D = (int)q.size(3);
    d->dtype = dtype_code(q); d->causal = causal; d->scale = (float)scale;
    for (int64_t* s : {d->do_strides, d->dq_strides, d->dk_strides, d->dv_strides}) {
        s[0] = (int64_t)d->H * d->T * d->D; s[1] = (int64_t)d->T * d->D; s[2] = d->D; s[3] = 1;
    }
}

PyObject* oom_class();

// C++ exceptions (the allocator's out-of-memory, a bad cast) become Python errors, as THP functions do.
#define HOST_BEGIN try {
#define HOST_END                                                      \
    } catch (const c10::OutOfMemoryError& e) {                        \
        PyErr_SetString(oom_class(), e.what_without_backtrace()); \
        return nullptr;                                               \
    } catch (const std::exception& e) {                               \
        PyErr_SetString(PyExc_RuntimeError, e.what());                \
        return nullptr;                                               \
    }

PyObject* oom_class() {
    static PyObject* cls = nullptr;
    if (!cls) {
        PyObject* m = PyImport_ImportModule("torch");
        cls = m ? PyObject_GetAttrString(m, "OutOfMemoryError") : nullptr;
        Py_XDECREF(m);
        if (!cls) { PyErr_Clear(); cls = PyExc_MemoryError; }
    }
    return cls;
}

// compatible(a, b, ...) -> True when all are 4-D tensors the attention op takes with equal shape, type and device
PyObject* compatible(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const at::Tensor* q = n > 0 ? tensor(args[0]) : nullptr;
    if (!q || q->dim() != 4 || !q->is_cuda() || dtype_code(*q) < 0) Py_RETURN_FALSE;
    for (Py_ssize_t i = 1; i < n; ++i) {
        const at::Tensor* t = tensor(args[i]);
        if (!t || !t->is_cuda() || !same(*q, *t)) Py_RETURN_FALSE;
    }
    Py_RETURN_TRUE;
}

// attn_fwd(q, k, v, scale, causal, token_major, out | None, compacted) -> (o, lse) | None.  compacted: what compaction could do
// has been done, the library judges the layout.
PyObject* attn_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HOST_BEGIN
    if (n != 8) Py_RETURN_NONE;
    const at::Tensor *q = tensor(args[0]), *k = tensor(args[1]), *v = tensor(args[2]);
    const bool compacted = PyObject_IsTrue(args[7]);
    if (!q || !k || !v) Py_RETURN_NONE;
    for (const at::Tensor* t : {q, k, v})
        if (!(compacted ? offerable(*t) : usable(*t)) || !same(*q, *t)) Py_RETURN_NONE;
    const double scale = PyFloat_AsDouble(args[3]);
    if (scale == -1.0 && PyErr_Occurred()) return nullptr;
    Ctx* ctx = context_for(q->get_device());
    if (!ctx) return nullptr;
    at::Tensor o, lse;
    if (args[6] != Py_None) {
        const at::Tensor* given = tensor(args[6]);
        if (!given || !usable(*given) || !same(*q, *given)) Py_RETURN_NONE;
        o = *given;
    }
    const bool token_major = PyObject_IsTrue(args[5]);
    deers_attn_desc d;
    fill_desc(&d, *q, scale, PyObject_IsTrue(args[4]));
    int rc;
    {
        NoGil unlocked;
        if (!o.defined() && token_major)
            o = empty_like_of({q->size(0), q->size(2), q->size(1), q->size(3)}, q->scalar_type(), *q).permute({0, 2, 1, 3});
        else if (!o.defined())
            o = empty_like_of(q->sizes(), q->scalar_type(), *q);
        lse = empty_like_of(q->sizes().slice(0, 3), at::kFloat, *q);
        put_strides(d.q_strides, *q); put_strides(d.k_strides, *k); put_strides(d.v_strides, *v); put_strides(d.o_strides, o);
        std::lock_guard<std::mutex> one(ctx->mu);
        rc = deers_b200_attn_fwd(ctx->handle, &d, q->data_ptr(), k->data_ptr(), v->data_ptr(), o.data_ptr(), (float*)lse.data_ptr(),
                                 nullptr, 0);
    }
    if (rc) return fail(rc, ctx);
    return wrap2(std::move(o), std::move(lse));
    HOST_END
}

// Whether the backward may take the larger workspace (the dS tiles kept between its kernels): when it is at most a quarter
// of what is free, on the device or in torch's allocator.  Asked anew every time, except for sizes up to 1/512 of the device
// (350 MB of 180 GB): the question costs 74 us of host time, which the forward in front of a larger backward hides (110 us and
// more), a smaller one does not; and so little, when it does not fit, is noticed by the allocation itself.
bool large_workspace_ok(deers_ctx* ctx, const at::Tensor& like, size_t bytes) {
    const c10::DeviceIndex device = like.device().index();
    if (bytes <= at::cuda::getDeviceProperties(device)->totalGlobalMem / 512) return true;
    size_t free_bytes = 0, total = 0;
    if (deers_b200_mem_info(ctx, &free_bytes, &total) != DEERS_OK) return false;
    const auto stats = c10::cuda::CUDACachingAllocator::getDeviceStats(device);
    const int64_t kept = stats.reserved_bytes[0].current - stats.allocated_bytes[0].current;
    return bytes <= (free_bytes + (size_t)(kept > 0 ? kept : 0)) / 4;
}

// Bytes the backward uses of its workspace: what deers_b200_attn_workspace_bytes answers for the tile width, without the room
// it keeps for the padded copies of other f16 head dims.
size_t used_workspace_bytes(const deers_attn_desc& d, int pass) {
    deers_attn_desc tile = d;
    if (d.dtype == DEERS_F16 && d.D % 8 == 0 && d.D < 128) tile.D = d.D <= 64 ? 64 : 128;
    return deers_b200_attn_workspace_bytes(&tile, pass);
}

// attn_bwd(q, k, v, o, lse, d_o, scale, causal, workspace | None, dv_out | None, compacted) -> (dq, dk, dv) | None
PyObject* attn_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HOST_BEGIN
    if (n != 11) Py_RETURN_NONE;
    const at::Tensor *q = tensor(args[0]), *k = tensor(args[1]), *v = tensor(args[2]), *o = tensor(args[3]), *lse = tensor(args[4]),
                     *g = tensor(args[5]);
    const bool compacted = PyObject_IsTrue(args[10]);
    if (!q || !k || !v || !o || !lse || !g) Py_RETURN_NONE;
    for (const at::Tensor* t : {q, k, v, o, g})
        if (!(compacted ? offerable(*t) : usable(*t)) || !same(*q, *t)) Py_RETURN_NONE;
    const double scale = PyFloat_AsDouble(args[6]);
    if (scale == -1.0 && PyErr_Occurred()) return nullptr;
    Ctx* ctx = context_for(q->get_device());
    if (!ctx) return nullptr;
    at::Tensor dq, dk, dv, ws;
    if (args[9] != Py_None) {
        const at::Tensor* given = tensor(args[9]);
        if (!given || !usable(*given) || !same(*q, *given)) Py_RETURN_NONE;
        dv = *given;
    }
    deers_attn_desc d;
    fill_desc(&d, *q, scale, PyObject_IsTrue(args[7]));
    const size_t need = used_workspace_bytes(d, 1);
    if (args[8] != Py_None) {
        const at::Tensor* given = tensor(args[8]);
        if (given && (size_t)(given->numel() * given->element_size()) >= need) ws = *given;
    }
    int rc;
    {
        NoGil unlocked;
        dq = empty_like_of(q->sizes(), q->scalar_type(), *q);
        dk = empty_like_of(q->sizes(), q->scalar_type(), *q);
        if (!dv.defined()) dv = empty_like_of(q->sizes(), q->scalar_type(), *q);
        put_strides(d.q_strides, *q); put_strides(d.k_strides, *k); put_strides(d.v_strides, *v); put_strides(d.o_strides, *o);
        put_strides(d.do_strides, *g); put_strides(d.dq_strides, dq); put_strides(d.dk_strides, dk); put_strides(d.dv_strides, dv);
        if (!ws.defined()) {
            const size_t fast = used_workspace_bytes(d, 2);
            if (fast > need && large_workspace_ok(ctx->handle, *q, fast)) {
                try {
                    ws = scratch(fast, *q);
                } catch (const c10::OutOfMemoryError&) {}        // recompute instead
            }
            if (!ws.defined()) ws = scratch(need < 256 ? 256 : need, *q);
        }
        std::lock_guard<std::mutex> one(ctx->mu);
        rc = deers_b200_attn_bwd(ctx->handle, &d, q->data_ptr(), k->data_ptr(), v->data_ptr(), o->data_ptr(), (const float*)lse->data_ptr(),
                                 g->data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), ws.data_ptr(),
                                 (size_t)(ws.numel() * ws.element_size()));
    }
    if (rc) return fail(rc, ctx);
    PyObject* r = PyTuple_New(3);
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(std::move(dq)));
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(std::move(dk)));
    PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(std::move(dv)));
    return r;
    HOST_END
}

// attn_decode(q, k_cache, v_cache, scale, causal, want_lse) -> o | (o, lse) | None
PyObject* attn_decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HOST_BEGIN
    if (n != 6) Py_RETURN_NONE;
    const at::Tensor *q = tensor(args[0]), *k = tensor(args[1]), *v = tensor(args[2]);
    if (!q || !k || !v) Py_RETURN_NONE;
    for (const at::Tensor* t : {q, k, v})
        if (t->dim() != 4 || !t->is_cuda() || t->stride(3) != 1 || t->scalar_type() != q->scalar_type() || t->get_device() != q->get_device())
            Py_RETURN_NONE;
    if (dtype_code(*q) < 0 || k->sizes() != v->sizes() || k->size(0) != q->size(0) || k->size(1) != q->size(1) ||
        k->size(3) != q->size(3) || k->size(2) < q->size(2))
        Py_RETURN_NONE;
    const double scale = PyFloat_AsDouble(args[3]);
    if (scale == -1.0 && PyErr_Occurred()) return nullptr;
    Ctx* ctx = context_for(q->get_device());
    if (!ctx) return nullptr;
    deers_decode_desc d;
    memset(&d, 0, sizeof(d));
    d.B = (int)q->size(0); d.H = (int)q->size(1); d.Tq = (int)q->size(2); d.Tk = (int)k->size(2); d.D = (int)q->size(3);
    d.dtype = dtype_code(*q); d.causal = PyObject_IsTrue(args[4]); d.scale = (float)scale;
    const bool want_lse = PyObject_IsTrue(args[5]);
    at::Tensor o, lse;
    int rc;
    {
        NoGil unlocked;
        o = empty_like_of(q->sizes(), q->scalar_type(), *q);
        if (want_lse) lse = empty_like_of(q->sizes().slice(0, 3), at::kFloat, *q);
        put_strides(d.q_strides, *q); put_strides(d.k_strides, *k); put_strides(d.v_strides, *v); put_strides(d.o_strides, o);
        // most calls need no workspace (the chunks of a slice meet in shared memory): ask for one only when told so
        float* lse_p = want_lse ? (float*)lse.data_ptr() : nullptr;
        std::lock_guard<std::mutex> one(ctx->mu);
        rc = deers_b200_attn_decode(ctx->handle, &d, q->data_ptr(), k->data_ptr(), v->data_ptr(), o.data_ptr(), lse_p, nullptr, 0);
        if (rc == DEERS_ERR_WORKSPACE) {
            const size_t need = deers_b200_attn_decode_workspace_bytes(&d);
            at::Tensor ws = scratch(need < 256 ? 256 : need, *q);
            rc = deers_b200_attn_decode(ctx->handle, &d, q->data_ptr(), k->data_ptr(), v->data_ptr(), o.data_ptr(), lse_p, ws.data_ptr(), need);
        }
    }
    if (rc) return fail(rc, ctx);
    if (!want_lse) return THPVariable_Wrap(std::move(o));
    return wrap2(std::move(o), std::move(lse));
    HOST_END
}

// gemm_f16(M, N, K, a, a_mn, b, b_mn) -> c: operands already checked by the Linear node
PyObject* gemm_f16(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HOST_BEGIN
    if (n != 7) Py_RETURN_NONE;
    const long M = PyLong_AsLong(args[0]), N = PyLong_AsLong(args[1]), K = PyLong_AsLong(args[2]);
    if (PyErr_Occurred()) return nullptr;
    const at::Tensor *a = tensor(args[3]), *b = tensor(args[5]);
    if (!a || !b || a->dim() != 2 || b->dim() != 2 || !a->is_cuda()) Py_RETURN_NONE;
    Ctx* ctx = context_for(a->get_device());
    if (!ctx) return nullptr;
    const int a_mn = PyObject_IsTrue(args[4]), b_mn = PyObject_IsTrue(args[6]);
    at::Tensor c;
    int rc;
    {
        NoGil unlocked;
        c = empty_like_of({M, N}, a->scalar_type(), *a);
        std::lock_guard<std::mutex> one(ctx->mu);
        rc = deers_b200_gemm_f16(ctx->handle, (int)M, (int)N, (int)K, a->data_ptr(), a->stride(0), a_mn, b->data_ptr(), b->stride(0), b_mn,
                                 c.data_ptr(), c.stride(0));
    }
    if (rc) return fail(rc, ctx);
    return THPVariable_Wrap(std::move(c));
    HOST_END
}

// rope_pack(src, cos, sin, dst, src_is_head_major, inverse) -> True | None.  One of src / dst is [B,T,H,D], the other the
// head-major [B,H,T,D] tensor.
PyObject* rope_pack(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HOST_BEGIN
    if (n != 6) Py_RETURN_NONE;
    const at::Tensor *src = tensor(args[0]), *cs = tensor(args[1]), *sn = tensor(args[2]), *dst = tensor(args[3]);
    if (!src || !cs || !sn || !dst || src->dim() != 4 || dst->dim() != 4 || !src->is_cuda() || dtype_code(*src) < 0) Py_RETURN_NONE;
    const bool head_src = PyObject_IsTrue(args[4]);
    const at::Tensor& tok = head_src ? *dst : *src;
    Ctx* ctx = context_for(src->get_device());
    if (!ctx) return nullptr;
    deers_rope_desc d;
    memset(&d, 0, sizeof(d));
    d.B = (int)tok.size(0); d.T = (int)tok.size(1); d.H = (int)tok.size(2); d.D = (int)tok.size(3);
    d.dtype = dtype_code(*src); d.inverse = PyObject_IsTrue(args[5]);
    static const int tok_order[4] = {0, 1, 2, 3}, head_order[4] = {0, 2, 1, 3};        // (b, t, h, d)
    for (int i = 0; i < 4; ++i) {
        d.src_strides[i] = src->stride(head_src ? head_order[i] : tok_order[i]);
        d.dst_strides[i] = dst->stride(head_src ? tok_order[i] : head_order[i]);
    }
    int rc;
    {
        NoGil unlocked;
        std::lock_guard<std::mutex> one(ctx->mu);
        rc = deers_b200_rope_pack(ctx->handle, &d, src->data_ptr(), cs->data_ptr(), sn->data_ptr(), dst->data_ptr());
    }
    if (rc) return fail(rc, ctx);
    Py_RETURN_TRUE;
    HOST_END
}

// setup(make_context, raise_status)
PyObject* setup(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "setup(make_context, raise_status)"); return nullptr; }
    Py_INCREF(args[0]); Py_INCREF(args[1]);
    Py_XDECREF(g_make_context); Py_XDECREF(g_raise_status);
    g_make_context = args[0]; g_raise_status = args[1];
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"setup", (PyCFunction)(void (*)())setup, METH_FASTCALL, nullptr},
    {"compatible", (PyCFunction)(void (*)())compatible, METH_FASTCALL, nullptr},
    {"attn_fwd", (PyCFunction)(void (*)())attn_fwd, METH_FASTCALL, nullptr},
    {"attn_bwd", (PyCFunction)(void (*)())attn_bwd, METH_FASTCALL, nullptr},
    {"attn_decode", (PyCFunction)(void (*)())attn_decode, METH_FASTCALL, nullptr},
    {"gemm_f16", (PyCFunction)(void (*)())gemm_f16, METH_FASTCALL, nullptr},
    {"rope_pack", (PyCFunction)(void (*)())rope_pack, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_deers_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__deers_host(void) { return PyModule_Create(&kModule); }
