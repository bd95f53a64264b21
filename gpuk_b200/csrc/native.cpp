// CPython functions over the C ABI of include/gpuk_b200.h for the calls a decode step makes many of: module
// `gpuk_b200._native`, part of libgpuk_b200.so.  They take tensors as they are, allocate the results, and launch on the
// current stream of the tensors' device, with the interpreter lock released as a dispatcher operator or ctypes would.  Why
// neither of those: a call through them costs several microseconds of host time, which is what bounds a step of a few sequences
// (fused epilogue, 8 rows: 11.0 -> 6.6 us a call; FP8 linear layer, 8 tokens, 1280 x 8192: 14.8 -> 5.7 us).  All but fp8_linear return None for a
// call that belongs to the operators: see NotDirect and add_rms.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <climits>

#include "gpuk_b200.h"

using at::Tensor;

namespace {

void check(int status, const char *what) {
    TORCH_CHECK(status == GPUK_OK, "gpuk::", what, ": ", gpuk_status_string(status), ": ", gpuk_last_error());
}

const Tensor &tensor_arg(PyObject *o, const char *what) {
    TORCH_CHECK(THPVariable_Check(o), "gpuk: ", what, " must be a tensor");
    return THPVariable_Unpack(o);
}
int64_t int_arg(PyObject *o) {
    const int64_t v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}
// A size as the C ABI takes it.
int int_size(int64_t v) {
    TORCH_CHECK(v >= 0 && v <= INT_MAX, "gpuk: a size of ", v, " is out of range");
    return static_cast<int>(v);
}
struct NoGil {
    PyThreadState *state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};
void expect_args(Py_ssize_t n, Py_ssize_t want, const char *what) { TORCH_CHECK(n == want, "gpuk::", what, " takes ", want, " arguments, got ", n); }
void *stream_of(const Tensor &t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
Tensor empty_like_on(const Tensor &t, at::IntArrayRef sizes, at::ScalarType type) { return at::detail::empty_cuda(sizes, type, t.device(), std::nullopt); }

// A tensor whose operators would go straight to the CUDA kernels: of the class Tensor itself, dense and contiguous, no transform or lazy bit on it.
bool plain_class(PyObject *o) {
    if (!THPVariable_CheckExact(o)) return false;
    const Tensor &t = THPVariable_Unpack(o);
    static const c10::DispatchKeySet other({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::Functionalize, c10::DispatchKey::FuncTorchBatched,
                                            c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Batched, c10::DispatchKey::Negative, c10::DispatchKey::Conjugate,
                                            c10::DispatchKey::ZeroTensor, c10::DispatchKey::NestedTensor});
    return !t.key_set().has_any(other);
}
bool plain(PyObject *o, int device) {
    if (!plain_class(o)) return false;
    const Tensor &t = THPVariable_Unpack(o);
    return t.is_cuda() && (device < 0 || t.get_device() == device) && t.layout() == at::kStrided && t.is_contiguous();
}
// No mode that wants to see operators: tracing, functional transforms, dispatch or function modes.
bool no_modes() {
    const c10::impl::LocalDispatchKeySet tls = c10::impl::tls_local_dispatch_key_set();
    static const c10::DispatchKeySet front({c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::FuncTorchVmapMode, c10::DispatchKey::Functionalize,
                                            c10::DispatchKey::Tracer, c10::DispatchKey::Python, c10::DispatchKey::PreDispatch});
    return !tls.included_.has_any(front) && !c10::impl::TorchDispatchModeTLS::any_modes_set() && at::impl::PythonTorchFunctionTLS::stack_len() == 0;
}
// Thrown for a tensor that a decode call below does not read as it is: it returns None, and the caller takes the operators, which accept any strides and types that go
// together.
struct NotDirect {};
// A plain contiguous CUDA tensor of the given type and alignment on the given device (-1: any).
bool direct(PyObject *o, at::ScalarType type, int device, uintptr_t align) {
    if (!plain(o, device)) return false;
    const Tensor &t = THPVariable_Unpack(o);
    return t.scalar_type() == type && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % align == 0;
}
// What is no CUDA tensor, or on another device, is an error.
const Tensor &cuda_arg(PyObject *o, const char *what, at::ScalarType type, int device = -1, uintptr_t align = 16) {
    if (direct(o, type, device, align)) return THPVariable_Unpack(o);
    const Tensor &t = tensor_arg(o, what);
    TORCH_CHECK(t.is_cuda(), "gpuk: ", what, " must be a contiguous CUDA tensor of ", type);
    TORCH_CHECK(device < 0 || t.get_device() == device, "gpuk: ", what, " is on another device");
    throw NotDirect();
}
// The same of a KV cache.  The library's attention reads it in vectors of 16 bytes and faults on one whose rows are not aligned for them: such a cache is refused.
const Tensor &cache_arg(PyObject *o, const char *what, int device) {
    if (direct(o, at::kBFloat16, device, 16)) return THPVariable_Unpack(o);
    if (plain_class(o)) {
        const Tensor &t = THPVariable_Unpack(o);
        if (t.is_cuda() && t.layout() == at::kStrided && t.dim() == 4 && t.stride(3) == 1) {
            bool aligned = reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
            for (int i = 0; i < 3; ++i) aligned = aligned && t.stride(i) * t.element_size() % 16 == 0;
            TORCH_CHECK(aligned, "gpuk: rows of a KV cache must be 16-byte aligned");
        }
    }
    return cuda_arg(o, what, at::kBFloat16, device);
}
// Around such a call: None while a mode wants to see operators, and for tensors that are not direct.
#define DIRECT_CALL(name, count)     \
    HANDLE_TH_ERRORS                 \
    expect_args(n, count, name);     \
    if (!no_modes()) Py_RETURN_NONE; \
    try {
#define END_DIRECT_CALL                                  \
    }                                                    \
    catch (const NotDirect &) { Py_RETURN_NONE; }        \
    END_HANDLE_TH_ERRORS

// rope_append(qkv [rows, (heads + 2 kv_heads) * head_dim], cos, sin, pos [t], k_cache, v_cache, heads) -> q [rows, heads * head_dim]
PyObject *rope_append(PyObject *, PyObject *const *args, Py_ssize_t n) {
    DIRECT_CALL("rope_append", 7)
    const Tensor &qkv = cuda_arg(args[0], "qkv", at::kBFloat16);
    const int dev = qkv.get_device();
    const Tensor &cos = cuda_arg(args[1], "cos", at::kFloat, dev), &sin = cuda_arg(args[2], "sin", at::kFloat, dev);
    const Tensor &pos = cuda_arg(args[3], "positions", at::kLong, dev, 8);
    const Tensor &kc = cache_arg(args[4], "k_cache", dev), &vc = cache_arg(args[5], "v_cache", dev);
    const int64_t heads = int_arg(args[6]);
    TORCH_CHECK(kc.dim() == 4 && vc.sizes() == kc.sizes() && qkv.dim() == 2 && cos.dim() == 2 && sin.sizes() == cos.sizes(), "gpuk: rope_append shapes do not match");
    const int64_t kv = kc.size(1), max_seq = kc.size(2), hd = kc.size(3), t = pos.numel(), rows = qkv.size(0);
    TORCH_CHECK(qkv.size(1) == (heads + 2 * kv) * hd && cos.size(1) * 2 == hd && t > 0 && rows % t == 0 && rows / t <= kc.size(0),
                "gpuk: rope_append shapes do not match");
    Tensor q;
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(qkv.device());
        q = empty_like_on(qkv, {rows, heads * hd}, at::kBFloat16);
        check(gpuk_rope_append(qkv.data_ptr(), cos.data_ptr<float>(), sin.data_ptr<float>(), pos.data_ptr<int64_t>(), q.data_ptr(), kc.data_ptr(), vc.data_ptr(),
                               int_size(rows / t), int_size(t), int_size(heads), int_size(kv), int_size(hd),
                               int_size(cos.size(0)), int_size(max_seq), stream_of(qkv)), "rope_append");
    }
    return THPVariable_Wrap(std::move(q));
    END_DIRECT_CALL
}

// silu_mul(x [rows, 2 f]) -> [rows, f]
PyObject *silu_mul(PyObject *, PyObject *const *args, Py_ssize_t n) {
    DIRECT_CALL("silu_mul", 1)
    const Tensor &x = cuda_arg(args[0], "x", at::kBFloat16);
    TORCH_CHECK(x.dim() == 2 && x.size(1) % 2 == 0, "gpuk: silu_mul takes [rows, 2 f]");
    Tensor out;
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(x.device());
        out = empty_like_on(x, {x.size(0), x.size(1) / 2}, at::kBFloat16);
        check(gpuk_silu_mul(x.data_ptr(), out.data_ptr(), x.size(0), int_size(x.size(1) / 2), stream_of(x)), "silu_mul");
    }
    return THPVariable_Wrap(std::move(out));
    END_DIRECT_CALL
}

// linear(x [m, k], w [n, k]) -> [m, n], bf16, m <= 32
PyObject *linear(PyObject *, PyObject *const *args, Py_ssize_t n) {
    DIRECT_CALL("linear", 2)
    const Tensor &x = cuda_arg(args[0], "x", at::kBFloat16);
    const Tensor &w = cuda_arg(args[1], "w", at::kBFloat16, x.get_device());
    TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1), "gpuk: linear operand shapes do not match");
    Tensor out;
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(x.device());
        out = empty_like_on(x, {x.size(0), w.size(0)}, at::kBFloat16);
        check(gpuk_linear_skinny(x.data_ptr(), w.data_ptr(), out.data_ptr(), int_size(x.size(0)), int_size(w.size(0)), int_size(x.size(1)), 0,
                                 stream_of(x)), "linear");
    }
    return THPVariable_Wrap(std::move(out));
    END_DIRECT_CALL
}

// x [m, k] and w [n, k] in FP8 with their scales, or in bf16 with None for both: checked, and as the C ABI takes them.
struct Operands {
    const Tensor &x, &w;
    const float *x_scale = nullptr, *w_scale = nullptr;
    int m, n, k;
    Operands(PyObject *const *args) : x(cuda_arg(args[0], "x", args[1] == Py_None ? at::kBFloat16 : at::kFloat8_e4m3fn)), w(cuda_arg(args[2], "w", x.scalar_type(), x.get_device())) {
        TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1) && (args[1] == Py_None) == (args[3] == Py_None), "gpuk: linear operand shapes do not match");
        m = int_size(x.size(0)), n = int_size(w.size(0)), k = int_size(w.size(1));
        if (args[1] == Py_None) return;
        const Tensor &xs = cuda_arg(args[1], "x_scale", at::kFloat, x.get_device(), 4), &ws = cuda_arg(args[3], "w_scale", at::kFloat, x.get_device());
        TORCH_CHECK(xs.numel() == m && ws.numel() == n, "gpuk: linear takes a scale per token and per channel");
        x_scale = xs.data_ptr<float>(), w_scale = ws.data_ptr<float>();
    }
};

// swiglu(x, x_scale, w [2 f, k], w_scale) -> [m, f]: silu of the first f channels times the others
PyObject *swiglu(PyObject *, PyObject *const *args, Py_ssize_t n) {
    DIRECT_CALL("swiglu", 4)
    const Operands o(args);
    Tensor out;
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(o.x.device());
        out = empty_like_on(o.x, {o.m, o.n / 2}, at::kBFloat16);
        check(gpuk_swiglu_skinny(o.x.data_ptr(), o.x_scale, o.w.data_ptr(), o.w_scale, out.data_ptr(), o.m, o.n, o.k, 0, stream_of(o.x)), "swiglu");
    }
    return THPVariable_Wrap(std::move(out));
    END_DIRECT_CALL
}

// qkv_rope(x, x_scale, w, w_scale, cos, sin, pos [t], k_cache, v_cache, heads) -> q [m, heads * 128]; keys and values go to the caches
PyObject *qkv_rope(PyObject *, PyObject *const *args, Py_ssize_t n) {
    DIRECT_CALL("qkv_rope", 10)
    const Operands o(args);
    const int dev = o.x.get_device();
    const Tensor &cos = cuda_arg(args[4], "cos", at::kFloat, dev), &sin = cuda_arg(args[5], "sin", at::kFloat, dev), &pos = cuda_arg(args[6], "positions", at::kLong, dev, 8);
    const Tensor &kc = cache_arg(args[7], "k_cache", dev), &vc = cache_arg(args[8], "v_cache", dev);
    const int64_t heads = int_arg(args[9]), t = pos.numel();
    TORCH_CHECK(kc.dim() == 4 && vc.sizes() == kc.sizes() && cos.dim() == 2 && sin.sizes() == cos.sizes() && kc.size(3) == 128 && cos.size(1) == 64 && heads > 0 &&
                    o.n == (heads + 2 * kc.size(1)) * 128 && t > 0 && o.m % t == 0 && o.m / t <= kc.size(0), "gpuk: qkv_rope shapes do not match");
    Tensor q;
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(o.x.device());
        q = empty_like_on(o.x, {o.m, heads * 128}, at::kBFloat16);
        check(gpuk_qkv_rope_skinny(o.x.data_ptr(), o.x_scale, o.w.data_ptr(), o.w_scale, cos.data_ptr<float>(), sin.data_ptr<float>(), pos.data_ptr<int64_t>(), q.data_ptr(),
                                   kc.data_ptr(), vc.data_ptr(), int_size(o.m / t), int_size(t), int_size(heads), int_size(kc.size(1)), o.k,
                                   int_size(cos.size(0)), int_size(kc.size(2)), 0, stream_of(o.x)), "qkv_rope");
    }
    return THPVariable_Wrap(std::move(q));
    END_DIRECT_CALL
}

// decode_attention(q [batch, heads, 128], k_cache, v_cache [>= batch, kv_heads, max_seq, 128], len) -> [batch, heads * 128]
PyObject *decode_attention(PyObject *, PyObject *const *args, Py_ssize_t n) {
    DIRECT_CALL("decode_attention", 4)
    const Tensor &q = cuda_arg(args[0], "q", at::kBFloat16);
    const int dev = q.get_device();
    const Tensor &kc = cache_arg(args[1], "k_cache", dev), &vc = cache_arg(args[2], "v_cache", dev);
    const int64_t len = int_arg(args[3]);
    TORCH_CHECK(q.dim() == 3 && kc.dim() == 4 && vc.sizes() == kc.sizes() && q.size(0) <= kc.size(0) && q.size(2) == kc.size(3) && len <= kc.size(2),
                "gpuk: decode_attention shapes do not match");
    Tensor out;
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(q.device());
        out = empty_like_on(q, {q.size(0), q.size(1) * q.size(2)}, at::kBFloat16);
        check(gpuk_decode_attention(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), out.data_ptr(), int_size(q.size(0)), int_size(q.size(1)),
                                    int_size(kc.size(1)), int_size(q.size(2)), int_size(len), int_size(kc.size(2)), 0, stream_of(q)),
              "decode_attention");
    }
    return THPVariable_Wrap(std::move(out));
    END_DIRECT_CALL
}

// prefill_attention(q [batch, t, heads, 128], k_cache, v_cache, pos [t], len) -> [batch * t, heads * 128]
PyObject *prefill_attention(PyObject *, PyObject *const *args, Py_ssize_t n) {
    DIRECT_CALL("prefill_attention", 5)
    const Tensor &q = cuda_arg(args[0], "q", at::kBFloat16);
    const int dev = q.get_device();
    const Tensor &kc = cache_arg(args[1], "k_cache", dev), &vc = cache_arg(args[2], "v_cache", dev);
    const Tensor &pos = cuda_arg(args[3], "positions", at::kLong, dev, 8);
    const int64_t len = int_arg(args[4]);
    TORCH_CHECK(q.dim() == 4 && kc.dim() == 4 && vc.sizes() == kc.sizes() && q.size(0) <= kc.size(0) && q.size(3) == kc.size(3) && pos.numel() == q.size(1) && len <= kc.size(2),
                "gpuk: prefill_attention shapes do not match");
    Tensor out;
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(q.device());
        out = empty_like_on(q, {q.size(0) * q.size(1), q.size(2) * q.size(3)}, at::kBFloat16);
        check(gpuk_prefill_attention(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), pos.data_ptr<int64_t>(), out.data_ptr(), int_size(q.size(0)),
                                     int_size(q.size(1)), int_size(q.size(2)), int_size(kc.size(1)), int_size(q.size(3)),
                                     int_size(len), int_size(kc.size(2)), stream_of(q)), "prefill_attention");
    }
    return THPVariable_Wrap(std::move(out));
    END_DIRECT_CALL
}

// fp8_linear(x [m, k], x_scale, w [n, k], w_scale, out or None, packed, k_split) -> [m, n]
PyObject *fp8_linear(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect_args(n, 7, "fp8_linear");
    const Tensor &x = tensor_arg(args[0], "x_fp8"), &xs = tensor_arg(args[1], "x_scale"), &w = tensor_arg(args[2], "w_fp8"), &ws = tensor_arg(args[3], "w_scale");
    TORCH_CHECK(x.scalar_type() == at::kFloat8_e4m3fn && w.scalar_type() == at::kFloat8_e4m3fn, "gpuk: fp8_linear takes float8_e4m3fn operands");
    // scales, results and (copied for the call) weights may also be pinned host memory, which the GPU reads
    auto reachable = [](const Tensor &t) { return t.is_cuda() || t.is_pinned(); };
    TORCH_CHECK(x.is_cuda() && reachable(w) && x.is_contiguous() && w.is_contiguous() && x.dim() == 2 && w.dim() == 2, "gpuk: fp8_linear takes contiguous 2-d CUDA tensors");
    const int64_t m = x.size(0), k = x.size(1), channels = w.size(0);
    TORCH_CHECK(w.size(1) == k && xs.numel() == m && ws.numel() == channels, "gpuk: fp8_linear operand shapes do not match");
    TORCH_CHECK(xs.scalar_type() == at::kFloat && ws.scalar_type() == at::kFloat && xs.is_contiguous() && ws.is_contiguous(), "gpuk: fp8_linear takes contiguous fp32 scales");
    TORCH_CHECK(reachable(xs) && reachable(ws), "gpuk: fp8_linear takes CUDA scales");
    const int packed = PyObject_IsTrue(args[5]);
    if (packed < 0) throw python_error();
    const int64_t split = int_arg(args[6]);
    Tensor out;
    if (args[4] != Py_None) {
        out = tensor_arg(args[4], "out");
        TORCH_CHECK(reachable(out) && out.scalar_type() == at::kBFloat16 && out.dim() == 2 && out.size(0) == m && out.size(1) == channels && out.is_contiguous(),
                    "gpuk: fp8_linear writes a contiguous bf16 [tokens, n] tensor");
    }
    TORCH_CHECK(m <= INT_MAX && channels <= INT_MAX && k <= INT_MAX && split >= 0 && split <= INT_MAX, "gpuk: fp8_linear sizes out of range");
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(x.device());
        if (!out.defined()) out = empty_like_on(x, {m, channels}, at::kBFloat16);
        const Tensor here = w.is_cuda() ? w : w.to(x.device());
        TORCH_CHECK(gpuk_fp8_linear_skinny(x.data_ptr(), xs.data_ptr<float>(), here.data_ptr(), ws.data_ptr<float>(), out.data_ptr(), static_cast<int>(m),
                                           static_cast<int>(channels), static_cast<int>(k), packed, static_cast<int>(split), stream_of(x)) == GPUK_OK,
                    gpuk_last_error());
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// add_rms(workspace, x, residual, weight, eps, quant_type, scale or None) -> (residual_out, norm_out, scale), what allreduce_rms computes, with the
// results allocated here; None for a call that should take the operator instead: whatever is not plain tensors of matching sizes and types.
PyObject *add_rms(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect_args(n, 7, "add_rms");
    if (!no_modes() || !plain(args[1], -1)) Py_RETURN_NONE;
    const Tensor &x = THPVariable_Unpack(args[1]);
    const int device = x.get_device();
    if (!plain(args[2], device) || !plain(args[3], device) || !PyLong_CheckExact(args[5])) Py_RETURN_NONE;
    const Tensor &residual = THPVariable_Unpack(args[2]), &weight = THPVariable_Unpack(args[3]);
    const at::ScalarType type = x.scalar_type();
    const int dtype = type == at::kBFloat16 ? GPUK_DTYPE_BF16 : type == at::kHalf ? GPUK_DTYPE_F16 : type == at::kFloat ? GPUK_DTYPE_F32 : -1;
    if (dtype < 0 || x.dim() < 1 || x.numel() == 0 || residual.scalar_type() != type || weight.scalar_type() != type) Py_RETURN_NONE;
    const int64_t numel = x.numel(), hidden = x.size(-1);
    if (residual.numel() != numel || weight.numel() != hidden || hidden > INT_MAX) Py_RETURN_NONE;
    const int64_t ws = int_arg(args[0]), quant = int_arg(args[5]);
    const double eps = PyFloat_AsDouble(args[4]);
    if (eps == -1.0 && PyErr_Occurred()) throw python_error();
    const bool given = args[6] != Py_None, dynamic = quant == GPUK_QUANT_FP8_E4M3FN_240 || quant == GPUK_QUANT_FP8_E4M3FNUZ_120 || quant == GPUK_QUANT_FP8_E4M3FN_448;
    if (given ? quant != GPUK_QUANT_FP8_E4M3FN_448_STATIC : !dynamic && quant != GPUK_QUANT_NONE) Py_RETURN_NONE;
    Tensor scale, residual_out, norm_out;
    if (given) {
        if (!plain(args[6], device)) Py_RETURN_NONE;
        scale = THPVariable_Unpack(args[6]);
        if (scale.scalar_type() != at::kFloat || scale.numel() < 1) Py_RETURN_NONE;
    }
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(x.device());
        residual_out = empty_like_on(x, residual.sizes(), type);
        norm_out = empty_like_on(x, x.sizes(), quant == GPUK_QUANT_NONE ? type : quant == GPUK_QUANT_FP8_E4M3FNUZ_120 ? at::kFloat8_e4m3fnuz : at::kFloat8_e4m3fn);
        if (!given) scale = dynamic ? empty_like_on(x, {x.size(0), 1}, at::kFloat) : empty_like_on(x, {1}, at::kFloat);
        // one scale a row of `hidden`
        TORCH_CHECK(!dynamic || scale.numel() >= numel / hidden, "gpuk: scale_out has ", scale.numel(), " elements, needs ", numel / hidden);
        float *const s = scale.data_ptr<float>();
        check(ws == 0 ? gpuk_residual_rms_quant(x.data_ptr(), residual.data_ptr(), weight.data_ptr(), residual_out.data_ptr(), norm_out.data_ptr(), s, numel,
                                                static_cast<int>(hidden), dtype, static_cast<float>(eps), static_cast<int>(quant), stream_of(x))
                      : gpuk_allreduce_rms(reinterpret_cast<gpuk_ws *>(ws), x.data_ptr(), residual.data_ptr(), weight.data_ptr(), residual_out.data_ptr(),
                                           norm_out.data_ptr(), s, numel, static_cast<int>(hidden), dtype, static_cast<float>(eps), static_cast<int>(quant), stream_of(x)),
              "allreduce_rms");
    }
    PyObject *result = PyTuple_New(3);
    if (!result) throw python_error();
    PyTuple_SET_ITEM(result, 0, THPVariable_Wrap(std::move(residual_out)));
    PyTuple_SET_ITEM(result, 1, THPVariable_Wrap(std::move(norm_out)));
    PyTuple_SET_ITEM(result, 2, THPVariable_Wrap(std::move(scale)));
    return result;
    END_HANDLE_TH_ERRORS
}

// no_modes(): whether nothing but the kernels would see the operators of this thread's next call
PyObject *no_modes_py(PyObject *, PyObject *) {
    HANDLE_TH_ERRORS
    return PyBool_FromLong(no_modes());
    END_HANDLE_TH_ERRORS
}

template <PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)>
constexpr PyCFunction fast() { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(F)); }

PyMethodDef methods[] = {
    {"no_modes", no_modes_py, METH_NOARGS, nullptr},
    {"rope_append", fast<rope_append>(), METH_FASTCALL, nullptr},
    {"swiglu", fast<swiglu>(), METH_FASTCALL, nullptr},
    {"qkv_rope", fast<qkv_rope>(), METH_FASTCALL, nullptr},
    {"linear", fast<linear>(), METH_FASTCALL, nullptr},
    {"decode_attention", fast<decode_attention>(), METH_FASTCALL, nullptr},
    {"prefill_attention", fast<prefill_attention>(), METH_FASTCALL, nullptr},
    {"fp8_linear", fast<fp8_linear>(), METH_FASTCALL, nullptr},
    {"add_rms", fast<add_rms>(), METH_FASTCALL, nullptr},
    {"silu_mul", fast<silu_mul>(), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "gpuk_b200._native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
