// CPython functions over the C ABI of include/gpuk_b200.h for the calls a decode step makes many of: module
// `gpuk_b200._native`, part of libgpuk_b200.so.  They take tensors as they are, allocate the results, and launch on the
// current stream of the tensors' device.  Why not operators of the dispatcher or ctypes: a call through either costs several
// microseconds of host time, which is what bounds a step of a few sequences.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

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
// A contiguous CUDA tensor of the given type on the given device (-1: any).
const Tensor &cuda_arg(PyObject *o, const char *what, at::ScalarType type, int device = -1) {
    const Tensor &t = tensor_arg(o, what);
    TORCH_CHECK(t.is_cuda() && t.is_contiguous() && t.scalar_type() == type, "gpuk: ", what, " must be a contiguous CUDA tensor of ", type);
    TORCH_CHECK(device < 0 || t.get_device() == device, "gpuk: ", what, " is on another device");
    return t;
}
int64_t int_arg(PyObject *o) {
    const int64_t v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}
void expect_args(Py_ssize_t n, Py_ssize_t want, const char *what) { TORCH_CHECK(n == want, "gpuk::", what, " takes ", want, " arguments, got ", n); }
void *stream_of(const Tensor &t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
Tensor empty_like_on(const Tensor &t, at::IntArrayRef sizes, at::ScalarType type) { return at::detail::empty_cuda(sizes, type, t.device(), std::nullopt); }

// rope_append(qkv [rows, (heads + 2 kv_heads) * head_dim], cos, sin, pos [t], k_cache, v_cache, heads) -> q [rows, heads * head_dim]
PyObject *rope_append(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect_args(n, 7, "rope_append");
    const Tensor &qkv = cuda_arg(args[0], "qkv", at::kBFloat16);
    const int dev = qkv.get_device();
    const Tensor &cos = cuda_arg(args[1], "cos", at::kFloat, dev), &sin = cuda_arg(args[2], "sin", at::kFloat, dev);
    const Tensor &pos = cuda_arg(args[3], "positions", at::kLong, dev);
    const Tensor &kc = cuda_arg(args[4], "k_cache", at::kBFloat16, dev), &vc = cuda_arg(args[5], "v_cache", at::kBFloat16, dev);
    const int64_t heads = int_arg(args[6]);
    TORCH_CHECK(kc.dim() == 4 && vc.sizes() == kc.sizes() && qkv.dim() == 2 && cos.dim() == 2 && sin.sizes() == cos.sizes(), "gpuk: rope_append shapes do not match");
    const int64_t kv = kc.size(1), max_seq = kc.size(2), hd = kc.size(3), t = pos.numel(), rows = qkv.size(0);
    TORCH_CHECK(qkv.size(1) == (heads + 2 * kv) * hd && cos.size(1) * 2 == hd && t > 0 && rows % t == 0 && rows / t <= kc.size(0),
                "gpuk: rope_append shapes do not match");
    c10::cuda::CUDAGuard guard(qkv.device());
    Tensor q = empty_like_on(qkv, {rows, heads * hd}, at::kBFloat16);
    check(gpuk_rope_append(qkv.data_ptr(), cos.data_ptr<float>(), sin.data_ptr<float>(), pos.data_ptr<int64_t>(), q.data_ptr(), kc.data_ptr(), vc.data_ptr(),
                           static_cast<int>(rows / t), static_cast<int>(t), static_cast<int>(heads), static_cast<int>(kv), static_cast<int>(hd),
                           static_cast<int>(cos.size(0)), static_cast<int>(max_seq), stream_of(qkv)), "rope_append");
    return THPVariable_Wrap(std::move(q));
    END_HANDLE_TH_ERRORS
}

// silu_mul(x [rows, 2 f]) -> [rows, f]
PyObject *silu_mul(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect_args(n, 1, "silu_mul");
    const Tensor &x = cuda_arg(args[0], "x", at::kBFloat16);
    TORCH_CHECK(x.dim() == 2 && x.size(1) % 2 == 0, "gpuk: silu_mul takes [rows, 2 f]");
    c10::cuda::CUDAGuard guard(x.device());
    Tensor out = empty_like_on(x, {x.size(0), x.size(1) / 2}, at::kBFloat16);
    check(gpuk_silu_mul(x.data_ptr(), out.data_ptr(), x.size(0), static_cast<int>(x.size(1) / 2), stream_of(x)), "silu_mul");
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// linear(x [m, k], w [n, k]) -> [m, n], bf16, m <= 32
PyObject *linear(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect_args(n, 2, "linear");
    const Tensor &x = cuda_arg(args[0], "x", at::kBFloat16);
    const Tensor &w = cuda_arg(args[1], "w", at::kBFloat16, x.get_device());
    TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1), "gpuk: linear operand shapes do not match");
    c10::cuda::CUDAGuard guard(x.device());
    Tensor out = empty_like_on(x, {x.size(0), w.size(0)}, at::kBFloat16);
    check(gpuk_linear_skinny(x.data_ptr(), w.data_ptr(), out.data_ptr(), static_cast<int>(x.size(0)), static_cast<int>(w.size(0)), static_cast<int>(x.size(1)), 0,
                             stream_of(x)), "linear");
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// decode_attention(q [batch, heads, 128], k_cache, v_cache [>= batch, kv_heads, max_seq, 128], len) -> [batch, heads * 128]
PyObject *decode_attention(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect_args(n, 4, "decode_attention");
    const Tensor &q = cuda_arg(args[0], "q", at::kBFloat16);
    const int dev = q.get_device();
    const Tensor &kc = cuda_arg(args[1], "k_cache", at::kBFloat16, dev), &vc = cuda_arg(args[2], "v_cache", at::kBFloat16, dev);
    const int64_t len = int_arg(args[3]);
    TORCH_CHECK(q.dim() == 3 && kc.dim() == 4 && vc.sizes() == kc.sizes() && q.size(0) <= kc.size(0) && q.size(2) == kc.size(3) && len <= kc.size(2),
                "gpuk: decode_attention shapes do not match");
    c10::cuda::CUDAGuard guard(q.device());
    Tensor out = empty_like_on(q, {q.size(0), q.size(1) * q.size(2)}, at::kBFloat16);
    check(gpuk_decode_attention(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), out.data_ptr(), static_cast<int>(q.size(0)), static_cast<int>(q.size(1)),
                                static_cast<int>(kc.size(1)), static_cast<int>(q.size(2)), static_cast<int>(len), static_cast<int>(kc.size(2)), 0, stream_of(q)),
          "decode_attention");
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

template <PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)>
constexpr PyCFunction fast() { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(F)); }

PyMethodDef methods[] = {
    {"rope_append", fast<rope_append>(), METH_FASTCALL, nullptr},
    {"linear", fast<linear>(), METH_FASTCALL, nullptr},
    {"decode_attention", fast<decode_attention>(), METH_FASTCALL, nullptr},
    {"silu_mul", fast<silu_mul>(), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "gpuk_b200._native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
