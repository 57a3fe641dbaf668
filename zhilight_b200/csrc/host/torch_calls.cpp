// The calls that a program makes once per layer and token, from Python tensors to launches in one step: ops.py's general path costs 10 to 30 us of
// interpreter and ctypes per call, more than many of the kernels behind it.  Host time of a call, us, there / here: one row through a 4096 x 4096
// 4-bit Linear 12.9 / 6.6 (the GPU works 4.7), an int8 Linear 30 / 13, an fp8 one 35 / 18, a bf16 one 16 / 8, an attention step over 32 caches
// 88 / 19, a masked prompt portion 37 / 16.  Each function does what the Python function of its name does, on the same stream and with
// the same entry points of the library, and returns the result, the library's error code as an int, or None for anything out of the ordinary (CPU
// tensors, tensor subclasses, wrapped or strided tensors where plain ones are asked for, active torch modes, memory of other owners):
// ops.py then takes its general path, which serves or refuses it.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "../../../include/zhilight_b200.h"

namespace {

// Entry points of the loaded library, by address (the library is found and opened by _lib.py)
struct {
    decltype(&zl_w4a16_gemm_fused) w4;
    decltype(&zl_dense_gemm_skinny) dense;
    decltype(&zl_int8_quant_per_token) int8_quant;
    decltype(&zl_fp8_quant_per_tensor) fp8_quant;
    decltype(&zl_w8a8_gemm) w8;
    decltype(&zl_decode_attention_workspace_bytes) attn_bytes;
    decltype(&zl_decode_attention_host) attn;
} zl;

struct NotPlain {};   // the general path's

const at::Tensor& plain(PyObject* o, bool contiguous) {
    if (!THPVariable_CheckExact(o)) throw NotPlain{};
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || !t.has_storage() || t.layout() != at::kStrided || t.is_neg() || t.unsafeGetTensorImpl()->is_python_dispatch() ||
        (contiguous && !t.is_contiguous()))
        throw NotPlain{};
    return t;
}
void* optional(PyObject* o, bool contiguous) { return o == Py_None ? nullptr : plain(o, contiguous).data_ptr(); }
int dtype_of(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kHalf: return ZL_F16;
        case at::kBFloat16: return ZL_BF16;
        case at::kFloat: return ZL_F32;
        default: throw NotPlain{};
    }
}
int to_int(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        throw NotPlain{};
    }
    if (v != (int)v) throw NotPlain{};
    return (int)v;
}
int truth(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) {
        PyErr_Clear();
        throw NotPlain{};
    }
    return v;
}
void args(Py_ssize_t n, Py_ssize_t want) {
    if (n != want || c10::impl::dispatch_mode_enabled() || at::impl::torch_function_mode_enabled()) throw NotPlain{};
}
zl_stream_t stream() { return (zl_stream_t)c10::cuda::getCurrentCUDAStream().stream(); }
at::Tensor empty(const at::Tensor& like, at::IntArrayRef sizes, at::ScalarType type) { return at::empty(sizes, like.options().dtype(type).requires_grad(false)); }

// as ctypes does, the library's calls run without the interpreter's lock
struct Unlocked {
    PyThreadState* state = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(state); }
};
template <typename F>
int unlocked(F&& f) {
    Unlocked u;
    return f();
}
// pdl of a call: early reads, or a dependent that waits for everything earlier first
int launched(PyObject* pdl) { return truth(pdl) ? 1 : 2; }
PyObject* result(int rc, const at::Tensor& out) { return rc ? PyLong_FromLong(rc) : THPVariable_Wrap(out); }

template <typename F>
PyObject* guarded(F&& f) {
    HANDLE_TH_ERRORS   // what torch throws here becomes what its own calls raise, torch.OutOfMemoryError for one
    try {
        return f();
    } catch (const NotPlain&) {
    }
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// x, packed, n, k, group_size, bias, residual, epilogue, pdl, out, variant
PyObject* w4a16_gemm_fused(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        args(na, 11);
        if (!zl.w4) throw NotPlain{};
        const at::Tensor& x = plain(a[0], false);
        if (x.scalar_type() != at::kHalf || x.dim() != 2) throw NotPlain{};
        zl_w4_fused_args_t p = {};
        p.x = x.data_ptr();
        p.M = (int)x.size(0);
        p.ldx = (int)x.stride(0);
        p.packed = plain(a[1], false).data_ptr();
        p.N = to_int(a[2]);
        p.K = to_int(a[3]);
        p.group_size = to_int(a[4]);
        p.bias = optional(a[5], false);
        p.residual = optional(a[6], false);
        p.epilogue = to_int(a[7]);
        p.pdl = launched(a[8]);
        p.variant = to_int(a[10]);
        if (p.epilogue == ZL_EPI_QKV_ROPE || p.N < 0) throw NotPlain{};
        const at::Tensor y = a[9] == Py_None ? empty(x, {x.size(0), p.epilogue == ZL_EPI_SWIGLU ? p.N / 2 : p.N}, at::kHalf) : plain(a[9], false);
        p.y = y.data_ptr();
        const zl_stream_t s = stream();
        return result(unlocked([&] { return zl.w4(&p, s); }), y);
    });
}

// x, w, bias, out_dtype (ZL_F16 ..., or None: x's), pdl
PyObject* dense_gemm_skinny(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        args(na, 5);
        if (!zl.dense) throw NotPlain{};
        const at::Tensor &x = plain(a[0], true), &w = plain(a[1], true);
        if (x.dim() != 2 || w.dim() < 1) throw NotPlain{};
        void* const bias = optional(a[2], true);
        const int dt = dtype_of(x), od = a[3] == Py_None ? dt : to_int(a[3]), pdl = launched(a[4]);
        if (od != ZL_F16 && od != ZL_BF16 && od != ZL_F32) throw NotPlain{};
        const at::Tensor y = empty(x, {x.size(0), w.size(0)}, od == ZL_F16 ? at::kHalf : od == ZL_BF16 ? at::kBFloat16 : at::kFloat);
        const zl_stream_t s = stream();
        return result(unlocked([&] {
                          return zl.dense(x.data_ptr(), (int)x.stride(0), w.data_ptr(), bias, y.data_ptr(), (int)x.size(0), (int)w.size(0), (int)x.size(1), dt,
                                          od, pdl, s);
                      }),
                      y);
    });
}

// x, w, w_scale, bias, kind (ZL_W8_INT8, ZL_W8_FP8), pdl: quantisation of the rows and the product
PyObject* w8_linear(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        args(na, 6);
        if (!zl.w8 || !zl.int8_quant || !zl.fp8_quant) throw NotPlain{};
        const at::Tensor &x = plain(a[0], true), &w = plain(a[1], true), &ws = plain(a[2], true);
        if (x.dim() != 2 || w.dim() < 1) throw NotPlain{};
        void* const bias = optional(a[3], true);
        const int kind = to_int(a[4]), pdl = launched(a[5]), dt = dtype_of(x), ws_dt = dtype_of(ws);
        const int64_t m = x.size(0), k = x.size(1), scale_at = (m * k + 15) / 16 * 16;
        const at::Tensor y = empty(x, {m, w.size(0)}, x.scalar_type());
        const at::Tensor room = empty(x, {scale_at + 4 * m}, at::kByte);   // the 8-bit rows, then their scales
        uint8_t* const q = static_cast<uint8_t*>(room.data_ptr());
        float* const scale = reinterpret_cast<float*>(q + scale_at);
        const zl_stream_t s = stream();
        return result(unlocked([&] {
                          const int rc = kind == ZL_W8_INT8 ? zl.int8_quant(x.data_ptr(), (int)x.stride(0), q, scale, (int)m, (int)k, dt, pdl, s)
                                                            : zl.fp8_quant(x.data_ptr(), q, scale, (size_t)(m * k), dt, pdl, s);
                          // the GEMM may start on its weights during the quantisation, which itself is behind everything earlier
                          return rc ? rc
                                    : zl.w8(q, scale, w.data_ptr(), ws.data_ptr(), ws_dt, bias, y.data_ptr(), (int)m, (int)w.size(0), (int)k, kind, dt, 1, s);
                      }),
                      y);
    });
}

// q, buf_lens, k_bufs, v_bufs, mask, scale, max_len_buf, num_kv_heads, bshd, pdl (which changes nothing: the call is behind everything earlier)
PyObject* decode_attention(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        args(na, 10);
        if (!zl.attn || !zl.attn_bytes) throw NotPlain{};
        const at::Tensor &q = plain(a[0], true), &lens = plain(a[1], true);
        if (q.dim() != 4) throw NotPlain{};
        void* const mask = optional(a[4], true);
        const double scale = PyFloat_AsDouble(a[5]);
        if (scale == -1.0 && PyErr_Occurred()) {
            PyErr_Clear();
            throw NotPlain{};
        }
        const int max_len = to_int(a[6]), kv_heads = to_int(a[7]), bshd = truth(a[8]), dt = dtype_of(q);
        truth(a[9]);
        const int b = (int)q.size(0), len_q = (int)q.size(1), heads = (int)q.size(2), dim = (int)q.size(3);
        // every tensor whose memory the launches below use; what torch cannot resize belongs to another owner and has to be waited for
        std::vector<const at::Tensor*> used{&q, &lens};
        if (mask) used.push_back(&THPVariable_Unpack(a[4]));
        std::vector<uint64_t> at_;
        for (int i = 2; i < 4; ++i) {
            if (!PyList_CheckExact(a[i]) && !PyTuple_CheckExact(a[i])) throw NotPlain{};
            const Py_ssize_t n = PySequence_Fast_GET_SIZE(a[i]);
            if (n != b) throw NotPlain{};
            for (Py_ssize_t j = 0; j < n; ++j) {
                const at::Tensor& t = plain(PySequence_Fast_GET_ITEM(a[i], j), false);
                used.push_back(&t);
                at_.push_back(reinterpret_cast<uint64_t>(t.data_ptr()));
            }
        }
        for (const at::Tensor* t : used)
            if (!t->storage().resizable()) throw NotPlain{};
        if (b == 0) throw NotPlain{};
        // the caller's lists may change hands once the lock is gone: keep the storages, not the tensors
        std::vector<c10::Storage> storages;
        storages.reserve(used.size());
        for (const at::Tensor* t : used) storages.push_back(t->storage());
        const at::Tensor out = at::empty_like(q);
        const size_t ws_bytes = zl.attn_bytes(b, len_q, heads, dim, max_len), table_at = (ws_bytes + 15) / 16 * 16;
        const at::Tensor room = empty(q, {(int64_t)(table_at + 16 * b)}, at::kByte);   // the kernels' workspace, then the table of addresses
        uint8_t* const ws = static_cast<uint8_t*>(room.data_ptr());
        void* const table = ws + table_at;
        const c10::cuda::CUDAStream cs = c10::cuda::getCurrentCUDAStream();
        const int rc = unlocked([&] {
            return zl.attn(q.data_ptr(), static_cast<const int32_t*>(lens.data_ptr()), at_.data(), table, static_cast<const int8_t*>(mask), (float)scale, max_len,
                           out.data_ptr(), b, len_q, heads, kv_heads, dim, bshd, ws, ws_bytes, dt, (zl_stream_t)cs.stream());
        });
        if (rc == 0)
            for (const c10::Storage& s : storages) c10::cuda::CUDACachingAllocator::recordStream(s.data_ptr(), cs);
        return result(rc, out);
    });
}

// {name of an entry point: its address}
PyObject* bind(PyObject*, PyObject* d) {
    if (!PyDict_Check(d)) {
        PyErr_SetString(PyExc_TypeError, "a dict of addresses");
        return nullptr;
    }
    auto set = [&](auto& f, const char* name) {
        PyObject* v = PyDict_GetItemString(d, name);   // borrowed
        f = reinterpret_cast<std::decay_t<decltype(f)>>(v ? PyLong_AsVoidPtr(v) : nullptr);
    };
    set(zl.w4, "zl_w4a16_gemm_fused");
    set(zl.dense, "zl_dense_gemm_skinny");
    set(zl.int8_quant, "zl_int8_quant_per_token");
    set(zl.fp8_quant, "zl_fp8_quant_per_tensor");
    set(zl.w8, "zl_w8a8_gemm");
    set(zl.attn_bytes, "zl_decode_attention_workspace_bytes");
    set(zl.attn, "zl_decode_attention_host");
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}

#define ZL_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {ZL_FAST(w4a16_gemm_fused), ZL_FAST(dense_gemm_skinny), ZL_FAST(w8_linear), ZL_FAST(decode_attention),
                         {"bind", bind, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
