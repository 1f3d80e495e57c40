// The host side of a decode call in native code: what `forward` of the quantized linears does between its arguments and the C entry point
// (checks, dtype codes, choice of kernel, result and scratch from torch's allocator, stream), for plain CUDA tensors. Anything else, errors included, returns
// None and is left to the Python code, which does the same in about 5 us more (QLinear 8.4 us a call, 6.0 so bound by Python and ctypes).
// Nothing is kept between calls but the addresses of the C entry points and, per device, the flag words and the workspace that gemm.py
// keeps as well.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/oxq.h"

namespace {

constexpr int MAX_DEVICES = 64;
at::Tensor *g_flags[MAX_DEVICES], *g_workspaces[MAX_DEVICES];

#define ENTRIES(X)                                                                                                                        \
    X(oxq_gguf_scratch_bytes) X(oxq_gguf_matmul) X(oxq_gguf_gemv) X(oxq_awq_gemv) X(oxq_w8a16_gemv) X(oxq_gptq_gemv)                      \
    X(oxq_packed4_full_scratch_bytes) X(oxq_packed4_streams) X(oxq_packed4_matmul) X(oxq_awq_gemm) X(oxq_gptq_gemm) X(oxq_awq_ffn_gate_up) X(oxq_gemm_workspace_bytes) X(oxq_fp8_gemv)            \
    X(oxq_fp8_scratch_bytes) X(oxq_fp8_matmul)
struct Entries {
#define X(name) decltype(&::name) name;
    ENTRIES(X)
#undef X
} g;
bool g_bound = false;

int dtype_code(at::ScalarType t)
{
    switch (t) {
    case at::kFloat: return OXQ_F32;
    case at::kHalf: return OXQ_F16;
    case at::kBFloat16: return OXQ_BF16;
    default: return -1;
    }
}

// A dense CUDA tensor that is nothing but that: no subclass, no wrapper of a transform, no lazy negation. Null otherwise.
const at::Tensor *plain(PyObject *o)
{
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor &t = THPVariable_Unpack(o);
    using K = c10::DispatchKey;
    static const c10::DispatchKeySet odd({K::Python, K::PythonTLSSnapshot, K::Functionalize, K::FuncTorchBatched, K::FuncTorchGradWrapper, K::FuncTorchVmapMode,
                                          K::FuncTorchBatchedDecomposition, K::BatchedNestedTensor, K::Batched, K::VmapMode, K::Conjugate, K::Negative,
                                          K::ZeroTensor, K::NestedTensor, K::Fake, K::DeferredInit});
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.key_set().has_any(odd)) return nullptr;
    return &t;
}
// Parameters are torch.nn.Parameter objects: weights may be, x may not (its result would have no gradient; Python says what happens then).
const at::Tensor *weight(PyObject *o)
{
    const at::Tensor *t = plain(o);
    return t && t->is_contiguous() ? t : nullptr;
}

struct Call {
    const at::Tensor *x = nullptr;
    int64_t m = 0;
    void *stream = nullptr;
    c10::DeviceIndex device = -1;
};
// x [..., k] as bf16 rows in order; false: not for this code.
bool begin(Call &c, PyObject *px, int64_t k)
{
    c.x = plain(px);
    if (!c.x || c.x->scalar_type() != at::kBFloat16 || c.x->dim() < 2 || c.x->size(-1) != k || !c.x->is_contiguous() || k <= 0) return false;
    c.m = c.x->numel() / k;
    if (c.m < 1 || c.m > 1 << 20) return false;
    c.device = c.x->device().index();
    if (c.device < 0 || c.device >= MAX_DEVICES || c.device != c10::cuda::current_device()) return false;
    c.stream = c10::cuda::getCurrentCUDAStream(c.device).stream();
    return true;
}
at::Tensor empty(const Call &c, c10::IntArrayRef sizes, at::ScalarType t)
{
    return at::Tensor(at::detail::empty_cuda(sizes, t, c.x->device(), std::nullopt));
}
at::Tensor result(const Call &c, int64_t n, at::ScalarType t)
{
    c10::DimVector sizes(c.x->sizes().begin(), c.x->sizes().end());
    sizes.back() = n;
    return empty(c, sizes, t);
}
bool opt_bias(PyObject *o, const void *&p, int &code)
{
    p = nullptr;
    code = 0;
    if (o == Py_None) return true;
    const at::Tensor *t = weight(o);
    if (!t || (code = dtype_code(t->scalar_type())) < 0) return false;
    p = t->data_ptr();
    return true;
}
uintptr_t bits(const void *p) { return reinterpret_cast<uintptr_t>(p); }
int num(PyObject *o) { return (int)PyLong_AsLong(o); } // True and False are numbers too

// Runs `body` (which returns an OXQ status) without the interpreter lock, as ctypes does; the result, or None where it failed.
template <typename Body> PyObject *finish(at::Tensor &y, Body body)
{
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = body();
    Py_END_ALLOW_THREADS
    if (rc != OXQ_OK) Py_RETURN_NONE; // Python makes the call again and raises what it says
    return THPVariable_Wrap(std::move(y));
}

template <PyObject *(*IMPL)(PyObject *const *), int ARGS> PyObject *guard(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (!g_bound || n != ARGS || at::tracer::impl::is_dispatch_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
        at::impl::torch_function_mode_enabled())
        Py_RETURN_NONE; // tracing, or a mode that wants to see what torch does
    try {
        PyObject *r = IMPL(a);
        if (PyErr_Occurred()) { // an argument of another type than the Python code has
            Py_XDECREF(r);
            PyErr_Clear();
            Py_RETURN_NONE;
        }
        return r;
    } catch (...) { // out of memory among others: Python raises it
        PyErr_Clear();
        Py_RETURN_NONE;
    }
}

// gguf(x, blocks, bias, type, in, out, result dtype code, most tokens of the GEMV)
PyObject *gguf(PyObject *const *a)
{
    const int type = num(a[3]), k = num(a[4]), n = num(a[5]), out = num(a[6]), gemv_max = num(a[7]);
    Call c;
    const at::Tensor *w = weight(a[1]);
    const void *b;
    int b_dt;
    if (out < 0 || !w || !begin(c, a[0], k) || !opt_bias(a[2], b, b_dt)) Py_RETURN_NONE;
    const int m = (int)c.m;
    const void *x = c.x->data_ptr(), *blocks = w->data_ptr();
    const at::ScalarType t = out == OXQ_F32 ? at::kFloat : out == OXQ_F16 ? at::kHalf : at::kBFloat16;
    const size_t need = (bits(x) | bits(blocks)) & 15 ? 0 : g.oxq_gguf_scratch_bytes(type, m, k, n);
    if (need) {
        if (!g_flags[c.device]) Py_RETURN_NONE;
        at::Tensor y = result(c, n, t), scratch = empty(c, {(int64_t)need}, at::kByte);
        void *yp = y.data_ptr(), *flag = g_flags[c.device]->data_ptr(), *sp = scratch.data_ptr();
        return finish(y, [&] { return g.oxq_gguf_matmul(type, x, OXQ_BF16, blocks, b, b_dt, yp, out, m, k, n, flag, sp, need, c.stream); });
    }
    if (m > gemv_max) Py_RETURN_NONE;
    at::Tensor y = result(c, n, t);
    void *yp = y.data_ptr();
    return finish(y, [&] { return g.oxq_gguf_gemv(type, x, OXQ_BF16, blocks, b, b_dt, yp, out, m, k, n, c.stream); });
}

struct Packed {
    const uint32_t *qw, *qz;
    const void *sc;
    int sc_dt;
};
bool packed(Packed &p, PyObject *qw, PyObject *qz, PyObject *sc)
{
    const at::Tensor *w = weight(qw), *s = weight(sc), *z = qz == Py_None ? nullptr : weight(qz);
    if (!w || !s || (qz != Py_None && !z) || (p.sc_dt = dtype_code(s->scalar_type())) < 0) return false;
    p.qw = (const uint32_t *)w->data_ptr();
    p.qz = z ? (const uint32_t *)z->data_ptr() : nullptr;
    p.sc = s->data_ptr();
    return true;
}

// packed4(x, qweight, qzeros, scales, bias, in, out, group, bits, pack along in, symmetric, (grouped, gemv, unaligned gemv) most tokens)
PyObject *packed4(PyObject *const *a)
{
    const int k = num(a[5]), n = num(a[6]), group = num(a[7]), nbits = num(a[8]), in = num(a[9]), sym = num(a[10]);
    if (!PyTuple_CheckExact(a[11]) || PyTuple_GET_SIZE(a[11]) != 3) Py_RETURN_NONE;
    const int grouped = num(PyTuple_GET_ITEM(a[11], 0)), gemv = num(PyTuple_GET_ITEM(a[11], 1)), unaligned = num(PyTuple_GET_ITEM(a[11], 2));
    Call c;
    Packed p;
    const void *b;
    int b_dt;
    if (!begin(c, a[0], k) || !packed(p, a[1], a[2], a[3]) || !opt_bias(a[4], b, b_dt)) Py_RETURN_NONE;
    const int m = (int)c.m;
    const void *x = c.x->data_ptr();
    const bool aligned = ((bits(x) | bits(p.qw) | bits(p.qz) | bits(p.sc)) & 15) == 0;
    // PackedQuantLinear._streams
    const bool streams = aligned && nbits == 4 && p.sc_dt == OXQ_F16 && !(in && grouped && m <= gemv) && g.oxq_packed4_streams(m, k, n, group, in);
    if (!streams && m <= (aligned ? gemv : unaligned)) {
        at::Tensor y = result(c, n, at::kBFloat16);
        void *yp = y.data_ptr();
        return finish(y, [&] {
            if (in) return g.oxq_gptq_gemv(x, OXQ_BF16, p.qw, p.qz, p.sc, p.sc_dt, b, b_dt, yp, OXQ_BF16, m, k, n, group, nbits, sym, c.stream);
            return (nbits == 4 ? g.oxq_awq_gemv : g.oxq_w8a16_gemv)(x, OXQ_BF16, p.qw, p.qz, p.sc, p.sc_dt, b, b_dt, yp, OXQ_BF16, m, k, n, group, c.stream);
        });
    }
    if (!aligned || !g_flags[c.device]) Py_RETURN_NONE;
    if (!streams && m > grouped) { // the dense copy and its GEMM: 15.8 us a call of 327 x 3072 x 1024 by way of Python were the call itself
        if (nbits != 4 || (!in && !p.qz) || !g_workspaces[c.device]) Py_RETURN_NONE;
        const at::Tensor ws = *g_workspaces[c.device]; // ours until the launch is done, should another thread let it grow
        const size_t bytes = (size_t)ws.numel();
        if (bytes < g.oxq_gemm_workspace_bytes(n, k)) Py_RETURN_NONE; // Python lets it grow
        at::Tensor y = result(c, n, at::kBFloat16);
        void *yp = y.data_ptr(), *wp = ws.data_ptr();
        return finish(y, [&] {
            if (in) return g.oxq_gptq_gemm(x, OXQ_BF16, p.qw, p.qz, p.sc, p.sc_dt, b, b_dt, yp, OXQ_BF16, m, k, n, group, nbits, sym || !p.qz, wp, bytes, c.stream);
            return g.oxq_awq_gemm(x, OXQ_BF16, p.qw, p.qz, p.sc, p.sc_dt, b, b_dt, yp, OXQ_BF16, m, k, n, group, wp, bytes, c.stream);
        });
    }
    const size_t need = g.oxq_packed4_full_scratch_bytes(m, k, n, group, in);
    at::Tensor y = result(c, n, at::kBFloat16), scratch = empty(c, {(int64_t)need}, at::kByte);
    void *yp = y.data_ptr(), *flag = g_flags[c.device]->data_ptr(), *sp = scratch.data_ptr();
    return finish(y, [&] {
        return g.oxq_packed4_matmul(x, OXQ_BF16, p.qw, p.qz, p.sc, p.sc_dt, b, b_dt, yp, OXQ_BF16, m, k, n, group, in, sym, flag, sp, need, c.stream);
    });
}

// ffn(x, qweight, qzeros, scales, in, intermediate, group, activation)
PyObject *ffn(PyObject *const *a)
{
    const int k = num(a[4]), inter = num(a[5]), group = num(a[6]), act = num(a[7]);
    Call c;
    Packed p;
    if (!begin(c, a[0], k) || !packed(p, a[1], a[2], a[3]) || !p.qz || !g_workspaces[c.device]) Py_RETURN_NONE;
    const at::Tensor ws = *g_workspaces[c.device]; // ours until the launch is done, should another thread let it grow
    if ((size_t)ws.numel() < g.oxq_gemm_workspace_bytes(2 * inter, k)) Py_RETURN_NONE; // Python lets it grow
    at::Tensor y = result(c, inter, at::kBFloat16);
    const void *x = c.x->data_ptr();
    void *yp = y.data_ptr(), *wp = ws.data_ptr();
    const int m = (int)c.m;
    const size_t bytes = (size_t)ws.numel();
    return finish(y, [&] { return g.oxq_awq_ffn_gate_up(x, OXQ_BF16, p.qw, p.qz, p.sc, p.sc_dt, act, yp, m, k, inter, group, wp, bytes, c.stream); });
}

// fp8(x, weight, scale_inv [s_out, s_in] f32, bias, in, out, most tokens of the GEMV off 16 bytes)
PyObject *fp8(PyObject *const *a)
{
    const int k = num(a[4]), n = num(a[5]), unaligned = num(a[6]);
    Call c;
    const at::Tensor *w = weight(a[1]), *s = weight(a[2]);
    const void *b;
    int b_dt;
    if (!w || !s || s->scalar_type() != at::kFloat || s->dim() != 2 || !begin(c, a[0], k) || !opt_bias(a[3], b, b_dt)) Py_RETURN_NONE;
    const int64_t so = s->size(0), si = s->size(1);
    if (so <= 0 || si <= 0 || n % so || k % si) Py_RETURN_NONE;
    const int s_out = (int)so, s_in = (int)si, bo = n / s_out, bi = k / s_in, m = (int)c.m;
    int few = n % 128 == 0 && k % 128 == 0 && bo % 128 == 0 && bi % 64 == 0 ? 8 : 32; // Fp8Linear.gemv_max_m
    const void *x = c.x->data_ptr();
    const uint8_t *wp = (const uint8_t *)w->data_ptr();
    const float *sp = (const float *)s->data_ptr();
    const bool off = (bits(x) | bits(wp)) & 15;
    if (m > few && m <= unaligned && off) few = unaligned;
    if (m <= few) {
        at::Tensor y = result(c, n, at::kBFloat16);
        void *yp = y.data_ptr();
        return finish(y, [&] { return g.oxq_fp8_gemv(x, OXQ_BF16, wp, sp, s_out, s_in, b, b_dt, yp, OXQ_BF16, m, k, n, c.stream); });
    }
    const size_t need = off ? 0 : g.oxq_fp8_scratch_bytes(m, k, n, s_out, s_in);
    if (!need || !g_flags[c.device]) Py_RETURN_NONE;
    at::Tensor y = result(c, n, at::kBFloat16), scratch = empty(c, {(int64_t)need}, at::kByte);
    void *yp = y.data_ptr(), *flag = g_flags[c.device]->data_ptr(), *scp = scratch.data_ptr();
    return finish(y, [&] { return g.oxq_fp8_matmul(x, OXQ_BF16, wp, sp, s_out, s_in, b, b_dt, yp, OXQ_BF16, m, k, n, flag, scp, need, c.stream); });
}

// keep(0: flag words, 1: workspace; tensor): what gemm.py uses on the tensor's device from now on.
PyObject *keep(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 2 || !THPVariable_Check(a[1])) {
        PyErr_SetString(PyExc_TypeError, "keep(kind, tensor)");
        return nullptr;
    }
    const at::Tensor &t = THPVariable_Unpack(a[1]);
    const int d = t.is_cuda() ? t.device().index() : -1, kind = num(a[0]);
    if (d < 0 || d >= MAX_DEVICES || kind < 0 || kind > 1) {
        PyErr_SetString(PyExc_ValueError, "keep: not a CUDA tensor, or unknown kind");
        return nullptr;
    }
    at::Tensor *&slot = (kind ? g_workspaces : g_flags)[d];
    if (slot) *slot = t;
    else slot = new at::Tensor(t); // lives as long as the process, as the dictionaries of gemm.py do
    Py_RETURN_NONE;
}

// bind({name: address of the C entry point})
PyObject *bind(PyObject *, PyObject *names)
{
    if (!PyDict_Check(names)) {
        PyErr_SetString(PyExc_TypeError, "bind: dict expected");
        return nullptr;
    }
#define X(name)                                                                                     \
    {                                                                                               \
        PyObject *v = PyDict_GetItemString(names, #name);                                           \
        void *p = v ? PyLong_AsVoidPtr(v) : nullptr;                                                \
        if (!p) {                                                                                   \
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_KeyError, #name);                          \
            return nullptr;                                                                         \
        }                                                                                           \
        g.name = reinterpret_cast<decltype(g.name)>(p);                                             \
    }
    ENTRIES(X)
#undef X
    g_bound = true;
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"gguf", (PyCFunction)(void (*)(void))guard<gguf, 8>, METH_FASTCALL, nullptr},
    {"packed4", (PyCFunction)(void (*)(void))guard<packed4, 12>, METH_FASTCALL, nullptr},
    {"ffn", (PyCFunction)(void (*)(void))guard<ffn, 8>, METH_FASTCALL, nullptr},
    {"fp8", (PyCFunction)(void (*)(void))guard<fp8, 7>, METH_FASTCALL, nullptr},
    {"keep", (PyCFunction)(void (*)(void))keep, METH_FASTCALL, nullptr},
    {"bind", bind, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
