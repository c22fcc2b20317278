// Native front of the Python operators: argument checks, the current stream and the call into the C ABI, without the
// interpreter in between.  A call of the decode shapes takes the GPU 3 - 10 us; the checks written in Python, ctypes'
// conversion of thirteen arguments and building a stream handle took 6 us on top of the launch itself (gemm 10.9 us of
// host time per call, fp8_linear 12.2).
//
// Every function returns the C ABI's return code, or kNotTaken (-1) when the arguments are not the ordinary case (another
// tensor type, a layout that needs a copy, a failed check): the caller then runs its Python path, which does the copy or
// raises the error.  Nothing is kept between calls and no exception leaves this file.

#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdlib>
#include <cstring>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

// What this file was compiled from and for, read out of the built file before it is loaded (front_key in _lib.py).
extern "C" __attribute__((used)) const char yan_b200_front_key[] = YAN_FRONT_KEY;

namespace {

constexpr int kNotTaken = -1;

using GemmFn = void (*)(const void*, const void*, const void*, const void*, void*, int, int, int, int, void*, int, int, int*);
using LinearFn = void (*)(const void*, const void*, const void*, void*, void*, size_t, int, int, int, int, void*, int, int,
                          int*);
using WorkspaceFn = size_t (*)(int, int);
using CastFn = void (*)(const void*, void*, void*, int, int, int, int, void*, int*);

struct Entries {
    GemmFn gemm_bf16, gemm_f32;
    LinearFn linear;
    WorkspaceFn workspace_bytes;
    CastFn per_token_cast;
};
Entries g_entries = {};

// The tensor behind a plain torch.Tensor with storage on a CUDA device; null for anything else.
const at::Tensor* cuda_tensor(PyObject* o) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.defined() && t.has_storage() && t.is_cuda() && t.layout() == at::kStrided ? &t : nullptr;
}

bool fits_int(int64_t v) { return v > 0 && v <= INT32_MAX; }
bool aligned(const void* p, size_t a) { return reinterpret_cast<uintptr_t>(p) % a == 0; }
int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

bool jit_requested() {
    const char* e = std::getenv("YAN_FP8_GEMM_JIT");
    return e != nullptr && e[0] != '\0' && std::strcmp(e, "0") != 0;
}

void* current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// [rows, cols] fp32 scales that are already row-contiguous per k-block.
bool column_major_scales(const at::Tensor& s, int64_t rows, int64_t cols) {
    if (s.scalar_type() != at::kFloat || s.dim() != 2 || s.size(0) != rows || s.size(1) != cols) return false;
    return rows == 1 ? (cols == 1 || s.stride(1) == 1) : (s.stride(0) == 1 && s.stride(1) == rows);
}

bool weights_ok(const at::Tensor& q, const at::Tensor& s, int64_t n, int64_t k) {
    return q.scalar_type() == at::kFloat8_e4m3fn && q.dim() == 2 && q.size(0) == n && q.size(1) == k && q.is_contiguous() &&
           s.scalar_type() == at::kFloat && s.dim() == 2 && s.size(0) == ceil_div(n, 128) && s.size(1) == k / 128 &&
           s.is_contiguous();
}

bool as_long(PyObject* o, long* v) {
    if (!PyLong_CheckExact(o)) return false;
    *v = PyLong_AsLong(o);
    if (*v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return *v >= 0 && *v <= INT32_MAX;
}

PyObject* code(int rc) { return PyLong_FromLong(rc); }

// gemm_*(lhs_q, lhs_scales, rhs_q, rhs_scales, out, block_n, num_sms, tail_cut)
template <bool bf16>
PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    try {
        long block_n, num_sms;
        if (nargs != 8 || !as_long(args[5], &block_n) || !as_long(args[6], &num_sms)) return code(kNotTaken);
        const at::Tensor *a = cuda_tensor(args[0]), *sa = cuda_tensor(args[1]), *b = cuda_tensor(args[2]),
                         *sb = cuda_tensor(args[3]), *out = cuda_tensor(args[4]);
        if (!a || !sa || !b || !sb || !out || a->dim() != 2 || b->dim() != 2 || out->dim() != 2) return code(kNotTaken);
        const int64_t m = a->size(0), k = a->size(1), n = b->size(0);
        if (!fits_int(m) || !fits_int(n) || !fits_int(k) || k % 128 != 0 || n % 16 != 0) return code(kNotTaken);
        if (out->scalar_type() != (bf16 ? at::kBFloat16 : at::kFloat)) return code(kNotTaken);
        if (a->scalar_type() != at::kFloat8_e4m3fn || !a->is_contiguous() || !weights_ok(*b, *sb, n, k)) return code(kNotTaken);
        if (!column_major_scales(*sa, m, k / 128)) return code(kNotTaken);
        const int64_t ldd = out->stride(0);
        if (out->size(0) != m || out->size(1) != n || out->stride(1) != 1 || ldd < n || ldd > INT32_MAX || ldd % (bf16 ? 8 : 4) != 0)
            return code(kNotTaken);
        // the compiled-per-shape route, the cut last wave (which needs scratch) and whole tiles on request stay with the
        // Python path
        if (bf16 && jit_requested()) return code(kNotTaken);
        if (block_n == 0) {
            const bool cut = PyObject_IsTrue(args[7]) == 1;
            if (bf16 ? (cut ? k >= 96 * 128 && ceil_div(m, 128) * ceil_div(n, 256) > num_sms : m > 64) : !cut) return code(kNotTaken);
        }
        const void *pa = a->data_ptr(), *pb = b->data_ptr();
        void* pout = out->data_ptr();
        if (!aligned(pa, 16) || !aligned(pb, 16) || !aligned(pout, 16)) return code(kNotTaken);
        const void *psa = sa->data_ptr(), *psb = sb->data_ptr();
        void* stream = current_stream();
        int rc = 0;
        Py_BEGIN_ALLOW_THREADS  // a launch waits when the queue is full
        (bf16 ? g_entries.gemm_bf16 : g_entries.gemm_f32)(pa, psa, pb, psb, pout, static_cast<int>(m), static_cast<int>(n),
                                                          static_cast<int>(k), static_cast<int>(ldd), stream,
                                                          static_cast<int>(num_sms), static_cast<int>(block_n), &rc);
        Py_END_ALLOW_THREADS
        return code(rc);
    } catch (...) {
        return code(kNotTaken);
    }
}

// linear(a, rhs_q, rhs_scales, out, workspace or None, workspaces, block_n, num_sms, tail_cut); `workspaces` maps (device,
// stream, bytes) to the caller's buffers
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    try {
        long block_n, num_sms;
        if (nargs != 9 || !as_long(args[6], &block_n) || !as_long(args[7], &num_sms)) return code(kNotTaken);
        const at::Tensor *a = cuda_tensor(args[0]), *b = cuda_tensor(args[1]), *sb = cuda_tensor(args[2]),
                         *out = cuda_tensor(args[3]);
        if (!a || !b || !sb || !out || a->dim() != 2 || b->dim() != 2 || out->dim() != 2) return code(kNotTaken);
        const int64_t m = a->size(0), k = a->size(1), n = b->size(0), ldd = out->stride(0);
        if (!fits_int(m) || !fits_int(n) || !fits_int(k) || k % 128 != 0) return code(kNotTaken);
        if (block_n == 0 && m > 64 && PyObject_IsTrue(args[8]) != 1) return code(kNotTaken);  // whole tiles: see the Python path
        if (a->scalar_type() != at::kBFloat16 || !a->is_contiguous() || !weights_ok(*b, *sb, n, k)) return code(kNotTaken);
        if (out->scalar_type() != at::kBFloat16 || out->size(0) != m || out->size(1) != n || out->stride(1) != 1 || !fits_int(ldd))
            return code(kNotTaken);
        void* stream = current_stream();
        const size_t need = g_entries.workspace_bytes(static_cast<int>(m), static_cast<int>(k));
        PyObject* ws_obj = args[4];
        if (ws_obj == Py_None) {
            if (!PyDict_CheckExact(args[5])) return code(kNotTaken);
            PyObject* key = Py_BuildValue("(iKn)", static_cast<int>(a->get_device()),
                                          static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)),
                                          static_cast<Py_ssize_t>(need));
            if (key == nullptr) {
                PyErr_Clear();
                return code(kNotTaken);
            }
            ws_obj = PyDict_GetItem(args[5], key);  // borrowed; the dictionary outlives the call
            Py_DECREF(key);
            if (ws_obj == nullptr) return code(kNotTaken);
        }
        const at::Tensor* ws_ptr = cuda_tensor(ws_obj);
        if (!ws_ptr || ws_ptr->scalar_type() != at::kByte || static_cast<size_t>(ws_ptr->numel()) < need) return code(kNotTaken);
        const at::Tensor ws = *ws_ptr;  // held: the dictionary may change while the interpreter runs other threads
        const void *pa = a->data_ptr(), *pb = b->data_ptr(), *psb = sb->data_ptr();
        void *pout = out->data_ptr(), *pws = ws.data_ptr();
        const size_t ws_bytes = static_cast<size_t>(ws.numel());
        int rc = 0;
        Py_BEGIN_ALLOW_THREADS
        g_entries.linear(pa, pb, psb, pout, pws, ws_bytes, static_cast<int>(m), static_cast<int>(n), static_cast<int>(k),
                         static_cast<int>(ldd), stream, static_cast<int>(num_sms), static_cast<int>(block_n), &rc);
        Py_END_ALLOW_THREADS
        return code(rc);
    } catch (...) {
        return code(kNotTaken);
    }
}

// per_token_cast(x, q, scales)
PyObject* per_token_cast(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    try {
        if (nargs != 3) return code(kNotTaken);
        const at::Tensor *x = cuda_tensor(args[0]), *q = cuda_tensor(args[1]), *s = cuda_tensor(args[2]);
        if (!x || !q || !s || x->dim() != 2 || q->dim() != 2 || s->dim() != 2) return code(kNotTaken);
        const int64_t m = x->size(0), k = x->size(1);
        if (x->scalar_type() != at::kBFloat16 || !fits_int(m) || !fits_int(k) || k % 128 != 0) return code(kNotTaken);
        if (x->stride(1) != 1 || x->stride(0) % 8 != 0 || !fits_int(x->stride(0)) || !aligned(x->data_ptr(), 16)) return code(kNotTaken);
        if (q->scalar_type() != at::kFloat8_e4m3fn || q->size(0) != m || q->size(1) != k || !q->is_contiguous()) return code(kNotTaken);
        if (s->scalar_type() != at::kFloat || s->size(0) != m || s->size(1) != k / 128 || s->stride(0) != 1 ||
            s->stride(1) < m || !fits_int(s->stride(1)))
            return code(kNotTaken);
        const int64_t scales_ld = k > 128 ? s->stride(1) : m;
        const void* px = x->data_ptr();
        void *pq = q->data_ptr(), *ps = s->data_ptr(), *stream = current_stream();
        const int x_ld = static_cast<int>(x->stride(0));
        int rc = 0;
        Py_BEGIN_ALLOW_THREADS
        g_entries.per_token_cast(px, pq, ps, static_cast<int>(m), static_cast<int>(k), x_ld, static_cast<int>(scales_ld), stream,
                                 &rc);
        Py_END_ALLOW_THREADS
        return code(rc);
    } catch (...) {
        return code(kNotTaken);
    }
}

// bind(gemm_bf16, gemm_f32, linear, workspace_bytes, per_token_cast): addresses of the C ABI's entry points
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 5) {
        PyErr_SetString(PyExc_TypeError, "bind takes five addresses");
        return nullptr;
    }
    void* p[5];
    for (int i = 0; i < 5; ++i) {
        p[i] = PyLong_AsVoidPtr(args[i]);
        if (p[i] == nullptr) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null entry point");
            return nullptr;
        }
    }
    g_entries = {reinterpret_cast<GemmFn>(p[0]), reinterpret_cast<GemmFn>(p[1]), reinterpret_cast<LinearFn>(p[2]),
                 reinterpret_cast<WorkspaceFn>(p[3]), reinterpret_cast<CastFn>(p[4])};
    Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {
    {"gemm_bf16", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(gemm<true>)), METH_FASTCALL, nullptr},
    {"gemm_f32", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(gemm<false>)), METH_FASTCALL, nullptr},
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear)), METH_FASTCALL, nullptr},
    {"per_token_cast", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(per_token_cast)), METH_FASTCALL, nullptr},
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall() { return PyModule_Create(&g_module); }
