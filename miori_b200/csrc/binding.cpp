// Native call path of the Python operators: one C function per operator that checks its tensors,
// allocates the output when the caller gave none, and calls the C ABI on the current stream.
//
// A decode step is a few hundred calls of 2-8 us of device work each, so what a call costs on the
// host is what an eager step takes.  Through ctypes a call cost 9.7 us (14.1 with an allocated
// output) on the B200 box's host: 3.2 us for the Stream object behind torch.cuda.current_stream(),
// 2.5 for torch.empty, about 2 for ctypes' eleven conversions, the rest attribute reads.  Here the
// stream, the pointers and the shapes are read from the C++ objects and the driver's launch (2 us)
// is what is left.  The library's functions come from the handle that _lib.py opened, so that there
// is one library whatever path it was loaded from.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <dlfcn.h>

#include <cstdint>
#include <cstring>
#include <exception>

#include "../../include/miori_b200.h"

namespace {

constexpr int MAX_ARGS = 13;
PyObject* g_error = nullptr;  // _lib.MioriError

#define MIORI_ENTRIES(X)                                                                         \
    X(last_error) X(gemv4) X(gemv8) X(dequant4_rowmajor) X(dequant8_rowmajor) X(dequant4_cache)  \
    X(cache_bytes) X(gemm_bf16_cache_ws) X(gemm_bf16_strided) X(gemv_bf16_cache) X(linear4)      \
    X(rmsnorm) X(post_norm_add) X(silu_mul) X(embed8) X(argmax) X(gemv4_rmsnorm)                 \
    X(gemv8_rmsnorm) X(gemv4_silu) X(gemv4_post_norm_add) X(gemv4_rmsnorm_silu)

struct Abi {
#define X(name) decltype(&miori_##name) name;
    MIORI_ENTRIES(X)
#undef X
} abi;

struct Failed {};  // a Python exception is set

[[noreturn]] void raise(PyObject* type, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    PyErr_FormatV(type, fmt, ap);
    va_end(ap);
    throw Failed();
}

// Arguments of a METH_FASTCALL | METH_KEYWORDS call by position: v[i] is null where none was given.
struct Args {
    PyObject* v[MAX_ARGS] = {};
    Args(const char* fn, const char* const* names, int count, int required, PyObject* const* args, Py_ssize_t n,
         PyObject* kw) {
        if (n > count) raise(PyExc_TypeError, "%s() takes at most %d arguments (%zd given)", fn, count, n);
        for (Py_ssize_t i = 0; i < n; ++i) v[i] = args[i];
        const Py_ssize_t nk = kw ? PyTuple_GET_SIZE(kw) : 0;
        for (Py_ssize_t k = 0; k < nk; ++k) {
            Py_ssize_t len = 0;
            const char* key = PyUnicode_AsUTF8AndSize(PyTuple_GET_ITEM(kw, k), &len);
            if (!key) throw Failed();
            int at = -1;
            for (int i = 0; i < count; ++i)
                if (names[i][0] == key[0] && std::strcmp(names[i], key) == 0) { at = i; break; }
            if (at < 0) raise(PyExc_TypeError, "%s() got an unexpected keyword argument '%s'", fn, key);
            if (v[at]) raise(PyExc_TypeError, "%s() got multiple values for argument '%s'", fn, key);
            v[at] = args[n + k];
        }
        for (int i = 0; i < required; ++i)
            if (!v[i]) raise(PyExc_TypeError, "%s() missing required argument '%s'", fn, names[i]);
    }
    bool given(int i) const { return v[i] && v[i] != Py_None; }
    const at::Tensor& tensor(int i) const {
        if (!v[i] || !THPVariable_Check(v[i])) raise(PyExc_TypeError, "argument %d: a tensor is expected", i + 1);
        return THPVariable_Unpack(v[i]);
    }
    uint32_t u32(int i, uint32_t dflt) const {
        if (!v[i]) return dflt;
        const unsigned long r = PyLong_AsUnsignedLongMask(v[i]);
        if (r == (unsigned long)-1 && PyErr_Occurred()) throw Failed();
        return (uint32_t)r;
    }
    float f32(int i) const {
        if (PyFloat_CheckExact(v[i])) return (float)PyFloat_AS_DOUBLE(v[i]);
        PyObject* f = PyNumber_Float(v[i]);  // whatever float() takes
        if (!f) throw Failed();
        const double d = PyFloat_AS_DOUBLE(f);
        Py_DECREF(f);
        return (float)d;
    }
};

void need_cuda(std::initializer_list<const at::Tensor*> ts) {
    for (const at::Tensor* t : ts) {
        if (!t->is_cuda()) raise(PyExc_ValueError, "miori_b200 ops need CUDA tensors (there is no CPU path)");
        if (!t->is_contiguous()) raise(PyExc_ValueError, "miori_b200 ops need contiguous tensors");
    }
}
void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
at::Tensor empty(at::IntArrayRef shape, at::ScalarType dt, const at::Tensor& like) {
    return at::Tensor(at::detail::empty_cuda(shape, dt, like.device(), std::nullopt));
}
at::ScalarType out_type(uint32_t flags) { return flags & MIORI_OUT_BF16 ? at::kBFloat16 : at::kFloat; }

// The output: the caller's object (returned as it is) or a new tensor.
struct Out {
    PyObject* given = nullptr;
    at::Tensor made;
    void* ptr() const { return given ? THPVariable_Unpack(given).data_ptr() : made.data_ptr(); }
    PyObject* result() {
        if (given) return Py_NewRef(given);
        return THPVariable_Wrap(std::move(made));
    }
};
// Memory of the caller's that a kernel writes: on a GPU or pinned, contiguous, large enough.
void need_room(const at::Tensor& t, const char* what, size_t bytes) {
    if (!t.is_cuda() && !t.is_pinned()) raise(PyExc_ValueError, "%s: a CUDA tensor is expected", what);
    if (!t.is_contiguous()) raise(PyExc_ValueError, "%s: a contiguous tensor is expected", what);
    if ((size_t)t.numel() * t.element_size() < bytes)
        raise(PyExc_ValueError, "%s: %zu bytes needed, the tensor has %zu", what, bytes, (size_t)t.numel() * t.element_size());
}
// `need`: what the kernel writes, where that is not the type of a new tensor.
Out output(const Args& a, int i, at::IntArrayRef shape, at::ScalarType dt, const at::Tensor& like,
           at::ScalarType need = at::ScalarType::Undefined) {
    Out o;
    if (a.given(i)) {
        size_t bytes = c10::elementSize(need == at::ScalarType::Undefined ? dt : need);
        for (const int64_t n : shape) bytes *= (size_t)n;
        need_room(a.tensor(i), "out", bytes);
        o.given = a.v[i];
    } else {
        o.made = empty(shape, dt, like);
    }
    return o;
}

// Call into the library without the interpreter lock (a launch may block on a full queue).  The arguments
// are evaluated before, under the lock: reading a tensor's pointer may throw.
template <class... P, class... A>
void call(int (*fn)(P...), A... args) {
    PyThreadState* ts = PyEval_SaveThread();
    const int rc = fn(static_cast<P>(args)...);
    PyEval_RestoreThread(ts);
    if (rc != MIORI_OK) {
        PyObject* exc = PyObject_CallFunction(g_error, "is", rc, abi.last_error());
        if (exc) {
            PyErr_SetObject(g_error, exc);
            Py_DECREF(exc);
        }
        throw Failed();
    }
}

template <class F>
PyObject* guarded(F body) {
    try {
        return body();
    } catch (const Failed&) {
    } catch (...) {  // torch's own, as its operators raise them: out of memory, no storage, a missing dimension
        torch::translate_exception_to_python(std::current_exception());
    }
    return nullptr;
}

#define OP(name, required, ...)                                                                    \
    const char* const name##_names[] = {__VA_ARGS__};                                              \
    PyObject* name##_body(const Args& a);                                                          \
    PyObject* py_##name(PyObject*, PyObject* const* args, Py_ssize_t n, PyObject* kw) {            \
        constexpr int count = sizeof(name##_names) / sizeof(char*);                                \
        static_assert(count <= MAX_ARGS, "");                                                      \
        return guarded([&] { return name##_body(Args(#name, name##_names, count, required, args, n, kw)); }); \
    }                                                                                              \
    PyObject* name##_body(const Args& a)

// Rows and columns of the activations: [K] counts as [1][K].
void rows_of(const at::Tensor& x, int64_t& M, int64_t& K) {
    if (x.dim() == 1) {
        M = 1, K = x.size(0);
    } else if (x.dim() == 2) {
        M = x.size(0), K = x.size(1);
    } else {
        raise(PyExc_ValueError, "activations of one or two dimensions expected");
    }
}
void check_words(const at::Tensor& q, int64_t per_word, int64_t K) {
    if (q.size(1) * per_word != K)
        raise(PyExc_ValueError, "q has %lld words per row, expected %lld", (long long)q.size(1), (long long)(K / per_word));
}

PyObject* gemv(const Args& a, decltype(abi.gemv4) fn, int64_t per_word) {
    const at::Tensor &q = a.tensor(0), &s = a.tensor(1), &b = a.tensor(2), &x = a.tensor(3);
    need_cuda({&q, &s, &b, &x});
    int64_t M, K;
    rows_of(x, M, K);
    check_words(q, per_word, K);
    const int64_t N = q.size(0);
    const uint32_t group = a.u32(4, 32), flags = a.u32(5, 0);
    Out y = output(a, 6, {M, N}, out_type(flags), x);
    call(fn, q.data_ptr(), s.data_ptr(), b.data_ptr(), x.data_ptr(), y.ptr(), N, K, M, group, flags, stream());
    return y.result();
}
OP(gemv4, 4, "q", "s", "b", "x", "group", "flags", "out") { return gemv(a, abi.gemv4, 8); }
OP(gemv8, 4, "q", "s", "b", "x", "group", "flags", "out") { return gemv(a, abi.gemv8, 4); }

PyObject* dequant(const Args& a, decltype(abi.dequant4_rowmajor) fn, int64_t per_word, bool flat) {
    const at::Tensor &q = a.tensor(0), &s = a.tensor(1), &b = a.tensor(2);
    need_cuda({&q, &s, &b});
    const int64_t N = q.size(0), K = q.size(1) * per_word;
    const uint32_t group = a.u32(3, 32);
    const int64_t flat_shape[1] = {(int64_t)(abi.cache_bytes(N, K) / 2)}, shape[2] = {N, K};
    Out o = output(a, 4, flat ? at::IntArrayRef(flat_shape) : at::IntArrayRef(shape), at::kBFloat16, q);
    call(fn, q.data_ptr(), s.data_ptr(), b.data_ptr(), o.ptr(), N, K, group, stream());
    return o.result();
}
OP(dequant4_rowmajor, 3, "q", "s", "b", "group", "out") { return dequant(a, abi.dequant4_rowmajor, 8, false); }
OP(dequant8_rowmajor, 3, "q", "s", "b", "group", "out") { return dequant(a, abi.dequant8_rowmajor, 4, false); }
OP(dequant4_cache, 3, "q", "s", "b", "group", "out") { return dequant(a, abi.dequant4_cache, 8, true); }

// Pointer and bytes of an optional workspace tensor.
void workspace(const Args& a, int i, void*& p, size_t& bytes) {
    p = nullptr, bytes = 0;
    if (!a.given(i)) return;
    const at::Tensor& w = a.tensor(i);
    need_room(w, "workspace", 0);
    p = w.data_ptr();
    bytes = (size_t)w.numel() * w.element_size();
}

OP(gemm_bf16_cache, 3, "A", "cache", "N", "flags", "out", "workspace") {
    const at::Tensor &A = a.tensor(0), &cache = a.tensor(1);
    need_cuda({&A, &cache});
    if (A.dim() != 2) raise(PyExc_ValueError, "gemm_bf16_cache: A [M][K] expected");
    const int64_t M = A.size(0), K = A.size(1), N = a.u32(2, 0);
    const uint32_t flags = a.u32(3, 0);
    Out c = output(a, 4, {M, N}, out_type(flags), A);
    void* wp;
    size_t wb;
    workspace(a, 5, wp, wb);
    call(abi.gemm_bf16_cache_ws, A.data_ptr(), cache.data_ptr(), c.ptr(), M, N, K, flags, wp, wb, stream());
    return c.result();
}

OP(gemm_bf16_strided, 2, "A", "B", "flags", "out") {
    const at::Tensor &A = a.tensor(0), &B = a.tensor(1);
    if (!A.is_cuda() || !B.is_cuda()) raise(PyExc_ValueError, "miori_b200 ops need CUDA tensors (there is no CPU path)");
    if (A.scalar_type() != at::kBFloat16 || B.scalar_type() != at::kBFloat16)
        raise(PyExc_TypeError, "gemm_bf16_strided: bf16 operands expected");
    if (A.dim() != 2 || B.dim() != 2 || B.size(1) != A.size(1) || A.stride(1) != 1 || B.stride(1) != 1)
        raise(PyExc_ValueError, "gemm_bf16_strided: A [M][K] and B [N][K] with contiguous rows expected");
    const int64_t M = A.size(0), K = A.size(1), N = B.size(0);
    const uint32_t flags = a.u32(2, 0);
    const at::ScalarType dt = out_type(flags);
    Out o;  // rows of a caller's output may lie apart
    if (a.given(3)) a.tensor(3), o.given = a.v[3];
    else o.made = empty({M, N}, dt, A);
    const at::Tensor& c = o.given ? THPVariable_Unpack(o.given) : o.made;
    if (!c.is_cuda() && !c.is_pinned()) raise(PyExc_ValueError, "out: a CUDA tensor is expected");
    if (c.scalar_type() != dt || c.dim() != 2 || c.size(0) != M || c.size(1) != N || c.stride(1) != 1)
        raise(PyExc_ValueError, "gemm_bf16_strided: bad output tensor");
    call(abi.gemm_bf16_strided, A.data_ptr(), A.stride(0), B.data_ptr(), B.stride(0), c.data_ptr(), c.stride(0), M, N,
         K, flags, stream());
    return o.result();
}

OP(gemv_bf16_cache, 3, "x", "cache", "N", "flags", "out") {
    const at::Tensor &x = a.tensor(0), &cache = a.tensor(1);
    need_cuda({&x, &cache});
    if (x.dim() != 2) raise(PyExc_ValueError, "gemv_bf16_cache: x [M][K] expected");
    const int64_t M = x.size(0), K = x.size(1), N = a.u32(2, 0);
    const uint32_t flags = a.u32(3, 0);
    Out y = output(a, 4, {M, N}, out_type(flags), x);
    call(abi.gemv_bf16_cache, x.data_ptr(), cache.data_ptr(), y.ptr(), M, N, K, flags, stream());
    return y.result();
}

OP(linear4, 5, "q", "s", "b", "cache", "x", "group", "flags", "out", "workspace") {
    const at::Tensor &q = a.tensor(0), &s = a.tensor(1), &b = a.tensor(2), &x = a.tensor(4);
    need_cuda({&q, &s, &b, &x});
    if (x.dim() != 2) raise(PyExc_ValueError, "linear4: x [M][K] expected");
    const int64_t M = x.size(0), K = x.size(1), N = q.size(0);
    const void* cache = a.given(3) ? a.tensor(3).data_ptr() : nullptr;
    const uint32_t group = a.u32(5, 32), flags = a.u32(6, 0);
    Out y = output(a, 7, {M, N}, at::kFloat, x, out_type(flags));
    void* wp;
    size_t wb;
    workspace(a, 8, wp, wb);
    call(abi.linear4, q.data_ptr(), s.data_ptr(), b.data_ptr(), cache, x.data_ptr(), y.ptr(), N, K, M, group, flags,
         wp, wb, stream());
    return y.result();
}

OP(rmsnorm, 3, "x", "gamma", "eps", "flags", "out") {
    const at::Tensor &x = a.tensor(0), &gamma = a.tensor(1);
    need_cuda({&x, &gamma});
    if (x.dim() != 2) raise(PyExc_ValueError, "rmsnorm: x [rows][n] expected");
    const int64_t rows = x.size(0), n = x.size(1);
    const float eps = a.f32(2);
    const uint32_t flags = a.u32(3, 0);
    Out y = output(a, 4, {rows, n}, at::kBFloat16, x);
    call(abi.rmsnorm, x.data_ptr(), gamma.data_ptr(), y.ptr(), rows, n, eps, flags, stream());
    return y.result();
}

OP(post_norm_add, 4, "x", "src", "gamma", "eps", "flags", "out") {
    const at::Tensor &x = a.tensor(0), &src = a.tensor(1), &gamma = a.tensor(2);
    need_cuda({&x, &src, &gamma});
    if (x.dim() != 2) raise(PyExc_ValueError, "post_norm_add: x [rows][n] expected");
    const int64_t rows = x.size(0), n = x.size(1);
    const float eps = a.f32(3);
    const uint32_t flags = a.u32(4, 0);
    Out o = output(a, 5, {rows, n}, x.scalar_type(), x, at::kFloat);
    call(abi.post_norm_add, x.data_ptr(), src.data_ptr(), gamma.data_ptr(), o.ptr(), rows, n, eps, flags, stream());
    return o.result();
}

OP(silu_mul, 2, "gate", "up", "flags", "out") {
    const at::Tensor &gate = a.tensor(0), &up = a.tensor(1);
    need_cuda({&gate, &up});
    const uint32_t flags = a.u32(2, 0);
    Out o = output(a, 3, gate.sizes(), at::kBFloat16, gate);
    call(abi.silu_mul, gate.data_ptr(), up.data_ptr(), o.ptr(), gate.numel(), flags, stream());
    return o.result();
}

OP(embed8, 4, "q", "s", "b", "tokens", "group", "flags", "out") {
    const at::Tensor &q = a.tensor(0), &s = a.tensor(1), &b = a.tensor(2), &tokens = a.tensor(3);
    need_cuda({&q, &s, &b, &tokens});
    const int64_t rows = q.size(0), K = q.size(1) * 4, T = tokens.numel();
    const uint32_t group = a.u32(4, 32), flags = a.u32(5, 0);
    Out o = output(a, 6, {T, K}, at::kBFloat16, q);
    call(abi.embed8, q.data_ptr(), s.data_ptr(), b.data_ptr(), tokens.data_ptr(), o.ptr(), T, rows, K, group, flags,
         stream());
    return o.result();
}

OP(argmax, 1, "v", "flags") {
    const at::Tensor& v = a.tensor(0);
    need_cuda({&v});
    const uint32_t flags = a.u32(1, 0) | (v.scalar_type() == at::kBFloat16 ? MIORI_OUT_BF16 : 0u);
    at::Tensor idx = empty({1}, at::kInt, v), val = empty({1}, at::kFloat, v);
    call(abi.argmax, v.data_ptr(), v.numel(), flags, idx.data_ptr(), val.data_ptr(), stream());
    PyObject* pair = PyTuple_New(2);
    if (!pair) throw Failed();
    PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::move(idx)));
    PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(std::move(val)));
    return pair;
}

void need_f32(const at::Tensor& x) {
    if (x.scalar_type() != at::kFloat) raise(PyExc_TypeError, "the fused norm takes fp32 activations");
}
PyObject* gemv_rmsnorm(const Args& a, decltype(abi.gemv4_rmsnorm) fn) {
    const at::Tensor &q = a.tensor(0), &s = a.tensor(1), &b = a.tensor(2), &x = a.tensor(3), &gamma = a.tensor(4);
    need_cuda({&q, &s, &b, &x, &gamma});
    need_f32(x);
    int64_t M, K;
    rows_of(x, M, K);
    const int64_t N = q.size(0);
    const float eps = a.f32(5);
    const uint32_t group = a.u32(6, 32), flags = a.u32(7, 0);
    Out y = output(a, 8, {M, N}, out_type(flags), x);
    call(fn, q.data_ptr(), s.data_ptr(), b.data_ptr(), x.data_ptr(), gamma.data_ptr(), eps, y.ptr(), N, K, M, group,
         flags, stream());
    return y.result();
}
OP(gemv4_rmsnorm, 6, "q", "s", "b", "x", "gamma", "eps", "group", "flags", "out") { return gemv_rmsnorm(a, abi.gemv4_rmsnorm); }
OP(gemv8_rmsnorm, 6, "q", "s", "b", "x", "gamma", "eps", "group", "flags", "out") { return gemv_rmsnorm(a, abi.gemv8_rmsnorm); }

OP(gemv4_silu, 4, "q", "s", "b", "x", "group", "flags", "out") {
    const at::Tensor &q = a.tensor(0), &s = a.tensor(1), &b = a.tensor(2), &x = a.tensor(3);
    need_cuda({&q, &s, &b, &x});
    int64_t M, K;
    rows_of(x, M, K);
    check_words(q, 8, K);
    const int64_t N = q.size(0);
    const uint32_t group = a.u32(4, 32), flags = a.u32(5, 0);
    Out y = output(a, 6, {M, N / 2}, at::kBFloat16, x);
    call(abi.gemv4_silu, q.data_ptr(), s.data_ptr(), b.data_ptr(), x.data_ptr(), y.ptr(), N, K, M, group, flags,
         stream());
    return y.result();
}

OP(gemv4_post_norm_add, 8, "q", "s", "b", "x", "residual", "gamma", "eps", "counter", "group", "flags", "out") {
    const at::Tensor &q = a.tensor(0), &s = a.tensor(1), &b = a.tensor(2), &x = a.tensor(3), &residual = a.tensor(4),
                     &gamma = a.tensor(5), &counter = a.tensor(7);
    need_cuda({&q, &s, &b, &x, &residual, &gamma, &counter});
    int64_t M, K;
    rows_of(x, M, K);
    check_words(q, 8, K);
    const int64_t N = q.size(0);
    if (residual.scalar_type() != at::kFloat || residual.numel() != M * N)
        raise(PyExc_ValueError, "residual: fp32 [M][N] expected");
    const float eps = a.f32(6);
    const uint32_t group = a.u32(8, 32), flags = a.u32(9, 0);
    Out o = output(a, 10, {M, N}, at::kFloat, x);
    call(abi.gemv4_post_norm_add, q.data_ptr(), s.data_ptr(), b.data_ptr(), x.data_ptr(), residual.data_ptr(),
         gamma.data_ptr(), eps, counter.data_ptr(), o.ptr(), N, K, M, group, flags, stream());
    return o.result();
}

OP(gemv4_rmsnorm_silu, 6, "q", "s", "b", "x", "gamma", "eps", "group", "flags", "out") {
    const at::Tensor &q = a.tensor(0), &s = a.tensor(1), &b = a.tensor(2), &x = a.tensor(3), &gamma = a.tensor(4);
    need_cuda({&q, &s, &b, &x, &gamma});
    need_f32(x);
    int64_t M, K;
    rows_of(x, M, K);
    const int64_t N = q.size(0);
    const float eps = a.f32(5);
    const uint32_t group = a.u32(6, 32), flags = a.u32(7, 0);
    Out y = output(a, 8, {M, N / 2}, at::kBFloat16, x);
    call(abi.gemv4_rmsnorm_silu, q.data_ptr(), s.data_ptr(), b.data_ptr(), x.data_ptr(), gamma.data_ptr(), eps,
         y.ptr(), N, K, M, group, flags, stream());
    return y.result();
}

// bind(handle, error): take the library's functions from the handle that ctypes opened.
PyObject* py_bind(PyObject*, PyObject* args) {
    unsigned long long h = 0;
    PyObject* err = nullptr;
    if (!PyArg_ParseTuple(args, "KO", &h, &err)) return nullptr;
#define X(name)                                                                                    \
    abi.name = reinterpret_cast<decltype(abi.name)>(dlsym(reinterpret_cast<void*>(h), "miori_" #name)); \
    if (!abi.name) return PyErr_Format(PyExc_ImportError, "miori_" #name " is missing from the library");
    MIORI_ENTRIES(X)
#undef X
    Py_XSETREF(g_error, Py_NewRef(err));
    Py_RETURN_NONE;
}

#define FAST(name, signature, text)                                                                \
    {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_##name)),            \
     METH_FASTCALL | METH_KEYWORDS, #name "(" signature ")\n--\n\n" text}

PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, "bind(handle, error)\n--\n\nTake the C ABI from an open library handle."},
    FAST(gemv4, "q, s, b, x, group=32, flags=0, out=None",
         "y[M][N] for packed 4-bit weights q[N][K/8] (int32 words), s/b[N][K/group] bf16."),
    FAST(gemv8, "q, s, b, x, group=32, flags=0, out=None", "y[M][N] for packed 8-bit weights q[N][K/4] (int32 words)."),
    FAST(dequant4_rowmajor, "q, s, b, group=32, out=None", "bf16 [N][K] of packed 4-bit weights."),
    FAST(dequant8_rowmajor, "q, s, b, group=32, out=None", "bf16 [N][K] of packed 8-bit weights."),
    FAST(dequant4_cache, "q, s, b, group=32, out=None",
         "Layout-opaque bf16 cache for gemm_bf16_cache (returned as a flat bf16 tensor)."),
    FAST(gemm_bf16_cache, "A, cache, N, flags=0, out=None, workspace=None",
         "C[M][N] = A[M][K] x cache(N,K)^T on the tcgen05 tensor cores (split-K if a workspace tensor is\n"
         "given and the shape has few output tiles)."),
    FAST(gemm_bf16_strided, "A, B, flags=0, out=None",
         "C[M][N] = A[M][K] x B[N][K]^T for bf16 operands whose rows may be strided (views of larger\n"
         "tensors, last dimension contiguous); `out` may be a strided view too."),
    FAST(gemv_bf16_cache, "x, cache, N, flags=0, out=None",
         "y[M][N] = x[M][K] (bf16) against the bf16 cache, M <= 32: the narrow-batch kernel."),
    FAST(linear4, "q, s, b, cache, x, group=32, flags=0, out=None, workspace=None",
         "Projection dispatch: packed-weight GEMV up to four rows, the bf16 cache above (narrow-batch\n"
         "kernel or tensor-core GEMM by shape; lib.miori_linear4_route tells which)."),
    FAST(rmsnorm, "x, gamma, eps, flags=0, out=None",
         "bf16(x * rsqrt(mean(x^2) + eps) * gamma): x fp32 [rows][n], gamma bf16 [n]."),
    FAST(post_norm_add, "x, src, gamma, eps, flags=0, out=None",
         "x + src * rsqrt(mean(src^2) + eps) * gamma, fp32 [rows][n]; gamma bf16 [n]."),
    FAST(silu_mul, "gate, up, flags=0, out=None", "bf16(gate / (1 + exp(-gate)) * up), fp32 inputs of the same shape."),
    FAST(embed8, "q, s, b, tokens, group=32, flags=0, out=None",
         "Rows tokens[t] of the 8-bit table q [rows][K/4] dequantized to bf16 [T][K]."),
    FAST(argmax, "v, flags=0",
         "(index, value) tensors of the largest element of a 1-D fp32 or bf16 vector; ties: lowest index."),
    FAST(gemv4_rmsnorm, "q, s, b, x, gamma, eps, group=32, flags=0, out=None",
         "gemv4 over bf16(rmsnorm(x) * gamma) with the norm fused into the kernel's activation staging."),
    FAST(gemv8_rmsnorm, "q, s, b, x, gamma, eps, group=32, flags=0, out=None",
         "gemv8 over bf16(rmsnorm(x) * gamma) with the norm fused into the kernel's activation staging."),
    FAST(gemv4_silu, "q, s, b, x, group=32, flags=0, out=None",
         "bf16(silu(gate) * up) [M][N/2] for the fused gate + up weights q [N][K/8] (gate rows first):\n"
         "gemv4 with silu_mul as its epilogue."),
    FAST(gemv4_post_norm_add, "q, s, b, x, residual, gamma, eps, counter, group=32, flags=0, out=None",
         "residual + v * rsqrt(mean(v^2) + eps) * gamma for v = gemv4(x), fp32 [M][N], M <= 4: gemv4 with\n"
         "post_norm_add as its epilogue.  `counter`: a zeroed int32 tensor of one element, left zero."),
    FAST(gemv4_rmsnorm_silu, "q, s, b, x, gamma, eps, group=32, flags=0, out=None",
         "bf16(silu(gate) * up) [M][N/2] of the fused gate + up weights applied to bf16(rmsnorm(x) * gamma),\n"
         "x fp32 [M][K], M <= 4: one launch for the norm, both projections and the activation."),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Native call path of the operators, " MIORI_TORCH_TAG, -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
