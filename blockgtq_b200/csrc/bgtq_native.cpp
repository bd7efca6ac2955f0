// The frequent calls of the Python host, natively: tensors in, library call, tensors out.
//
// Taking a call's tensors apart in Python (pointers, shapes, some twenty strides, result allocations) and converting
// forty arguments for ctypes cost 5 us of a layer step, 23 of an attention, 16 of a decode operator and 15 to 47 of the
// encoders and the prefill, more than the launches themselves (2.6 us each).  These functions do the same from the tensor
// objects.  A call whose tensors are not of the common form (another type, device, rank or layout) gets None and has
// done nothing: the Python wrapper then converts, stages or reports the error.
//
// The library is not linked: `bind` receives the addresses of its entry points from the ctypes handle.
#include <Python.h>

#include <cstring>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/bgtq.h"

namespace {

constexpr int64_t kHD = BGTQ_HEAD_DIM;

struct Fns {
    decltype(&bgtq_layer_step) layer_step;
    decltype(&bgtq_layer_encode) layer_encode;
    decltype(&bgtq_attend) attend;
    decltype(&bgtq_decode_default_splits) default_splits;
    decltype(&bgtq_encode) encode;
    decltype(&bgtq_rotate_q_rows) rotate_rows;
    decltype(&bgtq_prefill) prefill;
    decltype(&bgtq_prefill_workspace_bytes) prefill_workspace;
} F;

PyObject* none() { Py_RETURN_NONE; }
PyObject* code(int rc) { return PyLong_FromLong(rc); }

// A Python exception is set: the call ends with it (see `guarded`).
struct PythonError {};

struct Args {
    PyObject* const* a;
    // a tensor, or null where the argument is None or no tensor (`bad` then)
    const at::Tensor* tensor(int i, bool& bad) const {
        if (THPVariable_Check(a[i])) return &THPVariable_Unpack(a[i]);
        if (a[i] != Py_None) bad = true;
        return nullptr;
    }
    // Numbers are taken before the tensors are looked at and while the GIL is held; one that is no number, or does not fit,
    // ends the call.
    int64_t num(int i) const {
        const long long x = PyLong_AsLongLong(a[i]);
        if (x == -1 && PyErr_Occurred()) throw PythonError();
        return x;
    }
    int i32(int i) const {
        const int64_t x = num(i);
        if (x < INT32_MIN || x > INT32_MAX) {
            PyErr_SetString(PyExc_OverflowError, "argument does not fit 32 bits");
            throw PythonError();
        }
        return (int)x;
    }
    float real(int i) const {
        const double x = PyFloat_AsDouble(a[i]);
        if (x == -1.0 && PyErr_Occurred()) throw PythonError();
        return (float)x;
    }
    template <typename T> T* ptr(int i) const {
        if (a[i] == Py_None) return nullptr;
        const unsigned long long x = PyLong_AsUnsignedLongLong(a[i]);
        if (x == ~0ull && PyErr_Occurred()) throw PythonError();
        return reinterpret_cast<T*>(x);
    }
    bool truth(int i) const {
        const int r = PyObject_IsTrue(a[i]);
        if (r < 0) throw PythonError();
        return r != 0;
    }
};

void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// A CUDA tensor of `rank` dims on the current device, of this type, unit last stride.
bool is(const at::Tensor* t, int rank, at::ScalarType type) {
    return t && t->is_cuda() && t->dim() == rank && t->scalar_type() == type && t->stride(rank - 1) == 1;
}
bool here(const at::Tensor& t) { return t.get_device() == c10::cuda::current_device(); }
at::Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Tensor& like) {
    return at::detail::empty_cuda(size, type, like.device(), std::nullopt);
}
PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

// The cache's four tensors, checked: packed rows u8 (B, H, T, bytes), K norms fp16 or fp32 (B, H, T, n), V norms fp16 (B, H, T).
bool cache_ok(const at::Tensor* kp, const at::Tensor* kn, const at::Tensor* vp, const at::Tensor* vn) {
    return is(kp, 4, at::kByte) && is(kn, 4, at::kHalf) && is(vp, 4, at::kByte) && vn && vn->is_cuda() && vn->dim() == 3 &&
           vn->scalar_type() == at::kHalf;
}

// layer_step(step address, device, q, k, v, cos | None, sin | None) -> code | None
PyObject* layer_step(PyObject*, PyObject* const* argv, Py_ssize_t n) {
    if (n != 7) return none();
    const Args A{argv};
    const auto* s = A.ptr<const BgtqLayerStep>(0);
    const int dev = A.i32(1);
    bool bad = false;
    const at::Tensor *q = A.tensor(2, bad), *k = A.tensor(3, bad), *v = A.tensor(4, bad), *cs = A.tensor(5, bad), *sn = A.tensor(6, bad);
    if (bad || !is(q, 4, at::kHalf) || !is(k, 4, at::kHalf) || !is(v, 4, at::kHalf)) return none();
    auto shape = [&](const at::Tensor& t, int64_t heads) {
        return t.get_device() == dev && t.size(0) == s->n_batch && t.size(1) == heads && t.size(2) == 1 && t.size(3) == kHD;
    };
    if (!shape(*q, s->n_q) || !shape(*k, s->n_kv) || !shape(*v, s->n_kv)) return none();
    if ((s->flags & BGTQ_STEP_Q_ROTATED) && !q->is_contiguous()) return none();
    int64_t r_sb = 0;
    if (cs || sn) {
        for (const at::Tensor* t : {cs, sn})
            if (!t || !t->is_cuda() || t->get_device() != dev || t->scalar_type() != at::kHalf || t->dim() < 2 || t->numel() != s->n_batch * kHD ||
                t->size(0) != s->n_batch || t->stride(-1) != 1 || t->size(-1) != kHD)
                return none();
        r_sb = cs->stride(0);
        if (sn->stride(0) != r_sb) return none();
    }
    void* const st = stream_of(*q);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = F.layer_step(s, q->data_ptr(), q->stride(0), q->stride(1), k->data_ptr(), k->stride(0), k->stride(1), v->data_ptr(), v->stride(0),
                      v->stride(1), cs ? cs->data_ptr() : nullptr, sn ? sn->data_ptr() : nullptr, r_sb, st);
    Py_END_ALLOW_THREADS
    return code(rc);
}

// layer_encode(step address, device, k, v, t0, flags) -> code | None
PyObject* layer_encode(PyObject*, PyObject* const* argv, Py_ssize_t n) {
    if (n != 6) return none();
    const Args A{argv};
    const auto* s = A.ptr<const BgtqLayerStep>(0);
    const int dev = A.i32(1), t0 = A.i32(4), flags = A.i32(5);
    bool bad = false;
    const at::Tensor *k = A.tensor(2, bad), *v = A.tensor(3, bad);
    if (bad || !is(k, 4, at::kHalf) || !is(v, 4, at::kHalf) || k->get_device() != dev || v->get_device() != dev || k->sizes() != v->sizes() ||
        k->size(0) != s->n_batch || k->size(1) != s->n_kv || k->size(3) != kHD || t0 < 0 || t0 + k->size(2) > s->t_capacity)
        return none();
    void* const st = stream_of(*k);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = F.layer_encode(s, k->data_ptr(), k->stride(0), k->stride(1), k->stride(2), v->data_ptr(), v->stride(0), v->stride(1), v->stride(2),
                        (int)k->size(2), t0, flags, st);
    Py_END_ALLOW_THREADS
    return code(rc);
}

// encode(desc, rot_k, rot_v, n_kv, vpb, k, v, t0, k_packed, k_norms, v_packed, v_norms, flags) -> code | None   (both sides, fp16 norms)
PyObject* encode(PyObject*, PyObject* const* argv, Py_ssize_t n) {
    if (n != 13) return none();
    const Args A{argv};
    const auto* desc = A.ptr<const BgtqHeadDesc>(0);
    const auto* rot_k = A.ptr<const float>(1);
    const auto* rot_v = A.ptr<const float>(2);
    const int n_kv = A.i32(3), vpb = A.i32(4), t0 = A.i32(7), flags = A.i32(12);
    bool bad = false;
    const at::Tensor *k = A.tensor(5, bad), *v = A.tensor(6, bad), *kp = A.tensor(8, bad), *kn = A.tensor(9, bad), *vp = A.tensor(10, bad),
                     *vn = A.tensor(11, bad);
    if (bad || !is(k, 4, at::kHalf) || !is(v, 4, at::kHalf) || !cache_ok(kp, kn, vp, vn) || k->sizes() != v->sizes() || k->size(1) != n_kv ||
        k->size(3) != kHD || t0 < 0 || t0 + k->size(2) > kp->size(2) || vp->size(3) < ((flags & BGTQ_ENC_V_NIBBLE) ? kHD / 2 : vpb))
        return none();
    void* const st = stream_of(*k);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = F.encode(desc, rot_k, rot_v, k->data_ptr(), k->stride(0), k->stride(1),
                  k->stride(2), v->data_ptr(), v->stride(0), v->stride(1), v->stride(2), (int)k->size(0), n_kv, (int)k->size(2), t0,
                  kp->data_ptr<uint8_t>(), kp->stride(0), kp->stride(1), kp->stride(2), (int)kp->size(3), kn->data_ptr(), kn->stride(0),
                  kn->stride(1), kn->stride(2), (int)kn->size(3), vp->data_ptr<uint8_t>(), vp->stride(0), vp->stride(1), vp->stride(2),
                  vn->data_ptr(), vn->stride(0), vn->stride(1), vn->stride(2), nullptr, nullptr, flags | BGTQ_ENC_K_NORMS_F16, nullptr,
                  (int)kp->size(2), nullptr, st);
    Py_END_ALLOW_THREADS
    return code(rc);
}

// compress(desc, rot, n_kv, x, row_bytes, n_norms, flags) -> (packed, norms) | code | None.  x (n_kv, N, 128) contiguous;
// n_norms > 0: keys, fp32 norms (n_kv, N, n_norms); 0: values, fp16 norms (n_kv, N).
PyObject* compress(PyObject*, PyObject* const* argv, Py_ssize_t n) {
    if (n != 7) return none();
    const Args A{argv};
    const auto* desc = A.ptr<const BgtqHeadDesc>(0);
    const auto* rot = A.ptr<const float>(1);
    const int64_t n_kv = A.i32(2), rb = A.i32(4), ng = A.i32(5);
    const int flags = A.i32(6);
    bool bad = false;
    const at::Tensor* x = A.tensor(3, bad);
    if (bad || !is(x, 3, at::kHalf) || !x->is_contiguous() || x->size(0) != n_kv || x->size(2) != kHD) return none();
    const int64_t N = x->size(1);
    at::Tensor packed = empty({n_kv, N, rb}, at::kByte, *x);
    at::Tensor norms = ng ? empty({n_kv, N, ng}, at::kFloat, *x) : empty({n_kv, N}, at::kHalf, *x);
    void* const st = stream_of(*x);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = ng ? F.encode(desc, rot, nullptr, x->data_ptr(), 0, N * kHD, kHD, nullptr, 0, 0, 0, 1, (int)n_kv, (int)N, 0, packed.data_ptr<uint8_t>(), 0,
                       N * rb, rb, (int)rb, norms.data_ptr(), 0, N * ng, ng, (int)ng, nullptr, 0, 0, 0, nullptr, 0, 0, 0, nullptr, nullptr,
                       flags | BGTQ_ENC_SKIP_V, nullptr, (int)N, nullptr, st)
            : F.encode(desc, nullptr, rot, nullptr, 0, 0, 0, x->data_ptr(), 0, N * kHD, kHD, 1, (int)n_kv, (int)N, 0, nullptr, 0, 0, 0, 1, nullptr,
                       0, 0, 0, 1, packed.data_ptr<uint8_t>(), 0, N * rb, rb, norms.data_ptr(), 0, N, 1, nullptr, nullptr,
                       flags | BGTQ_ENC_SKIP_K, nullptr, (int)N, nullptr, st);
    Py_END_ALLOW_THREADS
    if (rc != BGTQ_OK) return code(rc);
    return Py_BuildValue("(NN)", wrap(std::move(packed)), wrap(std::move(norms)));
}

// attend(plan, desc, rot_k | None, q, k_packed, k_norms, v_packed, v_norms, t_begin, t_end, n_splits (0: the library's), scale, v_rot | None,
//        buf_o | None, buf_lse | None, want_f32, want_lse, status | None, n_kv) -> (out, f32 | None, lse | None) | code | None
// q (B, n_q, [1,] 128); out has q's rank.
PyObject* attend(PyObject*, PyObject* const* argv, Py_ssize_t n) {
    if (n != 19) return none();
    const Args A{argv};
    const auto* plan = A.ptr<const BgtqDecodePlan>(0);
    const auto* desc = A.ptr<const BgtqHeadDesc>(1);
    const auto* rot_k = A.ptr<const float>(2);
    const int t0 = A.i32(8), t1 = A.i32(9), n_kv = A.i32(18);
    int ns = A.i32(10);
    const float scale = A.real(11);
    const auto* v_rot = A.ptr<const float>(12);
    const bool want32 = A.truth(15), want_lse = A.truth(16);
    auto* status = A.ptr<int32_t>(17);
    if (ns < 0) return code(BGTQ_E_BADARG);
    bool bad = false;
    const at::Tensor *q = A.tensor(3, bad), *kp = A.tensor(4, bad), *kn = A.tensor(5, bad), *vp = A.tensor(6, bad), *vn = A.tensor(7, bad),
                     *bo = A.tensor(13, bad), *bl = A.tensor(14, bad);
    const bool four = q && q->dim() == 4;
    if (bad || !is(q, four ? 4 : 3, at::kHalf) || (four && q->size(2) != 1) || q->size(-1) != kHD || !here(*q) || !cache_ok(kp, kn, vp, vn))
        return none();
    if (!rot_k && !q->is_contiguous()) return none();
    const int64_t B = q->size(0), n_q = q->size(1);
    if (kp->size(0) < B || kp->size(1) != n_kv || t1 > kp->size(2)) return none();
    if (ns == 0) ns = F.default_splits((int)B, n_kv, t1 - t0);
    at::Tensor scratch, out = four ? empty({B, n_q, 1, kHD}, at::kHalf, *q) : empty({B, n_q, kHD}, at::kHalf, *q);
    at::Tensor o32, lse;
    if (want32) o32 = empty({B, n_q, kHD}, at::kFloat, *q);
    if (want_lse) lse = empty({B, n_q}, at::kFloat, *q);
    void* const st = stream_of(*q);
    int rc;
    bool bare = !rot_k;      // a decode that merges its shares and rotates nothing needs no scratch ...
again:
    if (!bare) scratch = empty({B * n_q * (ns * (kHD + 1) + kHD / 2)}, at::kFloat, *q);
    Py_BEGIN_ALLOW_THREADS
    rc = F.attend(plan, desc, rot_k, q->data_ptr(), q->stride(0), q->stride(1), kp->data_ptr<uint8_t>(), kp->stride(0), kp->stride(1), kp->stride(2),
                  kn->data_ptr(), kn->stride(0), kn->stride(1), kn->stride(2), vp->data_ptr<uint8_t>(), vp->stride(0), vp->stride(1), vp->stride(2),
                  vn->data_ptr(), vn->stride(0), vn->stride(1), vn->stride(2), (int)B, (int)n_q, n_kv, t0, t1, ns, scale, v_rot,
                  bo ? bo->data_ptr<float>() : nullptr, bl ? bl->data_ptr<float>() : nullptr, bare ? nullptr : scratch.data_ptr(), out.data_ptr(),
                  want32 ? o32.data_ptr<float>() : nullptr, want_lse ? lse.data_ptr<float>() : nullptr, status, st);
    Py_END_ALLOW_THREADS
    if (bare && rc == BGTQ_E_UNSUPPORTED) {      // ... any other does, and says so before it launches anything
        bare = false;
        goto again;
    }
    if (rc != BGTQ_OK) return code(rc);
    return Py_BuildValue("(NNN)", wrap(std::move(out)), want32 ? wrap(std::move(o32)) : none(), want_lse ? wrap(std::move(lse)) : none());
}

// rotate_rows(desc, rot_k, n_kv, q) -> tensor | code | None.  q (B, n_q, S, 128) fp16, rows on 16-byte boundaries.
PyObject* rotate_rows(PyObject*, PyObject* const* argv, Py_ssize_t n) {
    if (n != 4) return none();
    const Args A{argv};
    const auto* desc = A.ptr<const BgtqHeadDesc>(0);
    const auto* rot_k = A.ptr<const float>(1);
    const int n_kv = A.i32(2);
    bool bad = false;
    const at::Tensor* q = A.tensor(3, bad);
    if (bad || !is(q, 4, at::kHalf) || q->size(3) != kHD || q->numel() == 0 || !here(*q)) return none();
    if ((reinterpret_cast<uintptr_t>(q->data_ptr()) | (uint64_t)(2 * (q->stride(0) | q->stride(1) | q->stride(2)))) & 15u) return none();
    at::Tensor out = empty(q->sizes(), at::kHalf, *q);
    void* const st = stream_of(*q);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = F.rotate_rows(desc, rot_k, q->data_ptr(), q->stride(0), q->stride(1), q->stride(2), out.data_ptr(),
                       (int)q->size(0), (int)q->size(1), n_kv, (int)q->size(2), st);
    Py_END_ALLOW_THREADS
    return rc == BGTQ_OK ? wrap(std::move(out)) : code(rc);
}

// prefill(desc, n_kv, q, k_packed, k_norms, v_packed, v_norms, n_tokens, q_pos_offset, causal, scale, flags, v_rot | None, bound)
//   -> tensor | code | None; None too when the workspace would be larger than `bound` bytes
PyObject* prefill(PyObject*, PyObject* const* argv, Py_ssize_t n) {
    if (n != 14) return none();
    const Args A{argv};
    const auto* desc = A.ptr<const BgtqHeadDesc>(0);
    const int n_kv = A.i32(1), T = A.i32(7), off = A.i32(8), causal = A.truth(9) ? 1 : 0, flags = A.i32(11);
    const float scale = A.real(10);
    const auto* v_rot = A.ptr<const float>(12);
    const int64_t bound = A.num(13);
    bool bad = false;
    const at::Tensor *q = A.tensor(2, bad), *kp = A.tensor(3, bad), *kn = A.tensor(4, bad), *vp = A.tensor(5, bad), *vn = A.tensor(6, bad);
    if (bad || !is(q, 4, at::kHalf) || q->size(3) != kHD || q->numel() == 0 || !here(*q) || !cache_ok(kp, kn, vp, vn)) return none();
    const int64_t B = q->size(0), n_q = q->size(1), S = q->size(2);
    const int64_t ws_bytes = F.prefill_workspace((int)B, (int)n_q, n_kv, (int)S, T, off, causal, v_rot ? 1 : 0);
    if (ws_bytes > bound) return none();
    at::Tensor ws = empty({ws_bytes > 16 ? ws_bytes : 16}, at::kByte, *q), out = empty({B, n_q, S, kHD}, at::kHalf, *q);
    void* const st = stream_of(*q);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = F.prefill(desc, q->data_ptr(), q->stride(0), q->stride(1), q->stride(2), kp->data_ptr<uint8_t>(), kp->stride(0), kp->stride(1), kp->stride(2),
                   kn->data_ptr(), kn->stride(0), kn->stride(1), kn->stride(2), vp->data_ptr<uint8_t>(), vp->stride(0), vp->stride(1), vp->stride(2),
                   vn->data_ptr(), vn->stride(0), vn->stride(1), vn->stride(2), (int)B, (int)n_q, n_kv, (int)S, T, off, causal,
                   scale, flags, v_rot, ws.data_ptr(), ws.numel(), out.data_ptr(), st);
    Py_END_ALLOW_THREADS
    return rc == BGTQ_OK ? wrap(std::move(out)) : code(rc);
}

// bind(addresses in the order of Fns)
PyObject* bind(PyObject*, PyObject* const* argv, Py_ssize_t n) {
    if (n != (Py_ssize_t)(sizeof(F) / sizeof(void*))) {
        PyErr_SetString(PyExc_ValueError, "bind: wrong number of addresses");
        return nullptr;
    }
    const Args A{argv};
    void* fns[sizeof(F) / sizeof(void*)];
    for (Py_ssize_t i = 0; i < n; ++i) fns[i] = A.ptr<void>((int)i);
    memcpy(&F, fns, sizeof(F));
    return none();
}

// Library errors raised by torch (an allocation that fails) become Python exceptions.
template <PyObject* (*FN)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* argv, Py_ssize_t n) {
    try {
        return FN(self, argv, n);
    } catch (const PythonError&) {
    } catch (const c10::OutOfMemoryError& e) {
        PyObject* torch = PyImport_ImportModule("torch");
        PyObject* type = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
        if (type) PyErr_SetString(type, e.what_without_backtrace());
        Py_XDECREF(type);
        Py_XDECREF(torch);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

#define BGTQ_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {BGTQ_METHOD(bind),   BGTQ_METHOD(layer_step),  BGTQ_METHOD(layer_encode), BGTQ_METHOD(encode), BGTQ_METHOD(compress),
                          BGTQ_METHOD(attend), BGTQ_METHOD(rotate_rows), BGTQ_METHOD(prefill),      {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__native(void) {
    PyObject* m = PyModule_Create(&kModule);
    if (m && PyModule_AddStringConstant(m, "abi", BGTQ_NATIVE_ABI) != 0) Py_CLEAR(m);
    return m;
}
