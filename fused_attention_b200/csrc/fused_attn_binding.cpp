// Torch extension module `fused_attn`: the operator surface of the reference binding
// (src/fused_attn_extention.cu:15-129) over the C ABI of include/fa_b200.h.
//
//   fused_attn.attention_forward(head_dim, chunk_size, queries, keys, values, mask=None) -> Tensor
//
// Same argument names, order and default; the same preconditions raise the same exception type
// (c10::Error -> RuntimeError).  Relaxed on purpose: sequence_len need not be a multiple of
// chunk_size.  Fixed on purpose: the output lives on queries.device() and the launch goes to the
// caller's current stream (the reference allocates on the current device and launches on stream 0,
// src/fused_attn_extention.cu:67-70, include/fused_attn.cuh:885).
#include <torch/extension.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include "fa_b200.h"

namespace {

void check_input(const torch::Tensor& t, const char* name) {
    TORCH_CHECK(t.dtype() == torch::kFloat16 && t.device().type() == torch::kCUDA && t.is_contiguous() &&
                    t.dim() == 3,
                name, " must be a contiguous float16 CUDA tensor with 3 dimensions");
}

torch::Tensor attention_forward(int head_dim, int chunk_size, torch::Tensor queries, torch::Tensor keys,
                                torch::Tensor values, torch::optional<torch::Tensor> mask) {
    check_input(queries, "queries");
    check_input(keys, "keys");
    check_input(values, "values");
    if (mask.has_value()) check_input(*mask, "mask");

    TORCH_CHECK(head_dim > 0 && !(head_dim & (head_dim - 1)) && 16 <= head_dim && head_dim <= 128,
                "head_dim must be a power of two in [16, 128]");
    TORCH_CHECK(chunk_size > 0 && !(chunk_size & (chunk_size - 1)) && 16 <= chunk_size && chunk_size <= 128 &&
                    chunk_size <= 2 * head_dim,
                "chunk_size must be a power of two in [16, 128] and at most 2*head_dim");
    TORCH_CHECK(!(chunk_size == 16 && head_dim == 128), "chunk_size 16 with head_dim 128 is not supported");

    const int64_t B = queries.size(0), L = queries.size(1), F = queries.size(2);
    TORCH_CHECK(keys.size(0) == B && keys.size(1) == L && keys.size(2) == F, "keys must have the shape of queries");
    TORCH_CHECK(values.size(0) == B && values.size(1) == L && values.size(2) == F,
                "values must have the shape of queries");
    TORCH_CHECK(F % head_dim == 0, "the feature size must be divisible by head_dim");
    TORCH_CHECK(B > 0 && L > 0 && F > 0, "empty tensors are not supported");
    TORCH_CHECK(keys.device() == queries.device() && values.device() == queries.device(),
                "queries, keys and values must be on one device");
    if (mask.has_value()) {
        TORCH_CHECK(mask->size(0) == B && mask->size(1) == L && mask->size(2) == L, "mask must have shape [B, L, L]");
        TORCH_CHECK(mask->device() == queries.device(), "mask must be on the device of queries");
    }

    const c10::cuda::CUDAGuard guard(queries.device());
    auto output = torch::empty_like(queries);
    const auto stream = c10::cuda::getCurrentCUDAStream(queries.device().index());
    const int rc = fa_b200_attention_forward(
        queries.data_ptr(), keys.data_ptr(), values.data_ptr(), mask.has_value() ? mask->data_ptr() : nullptr,
        output.data_ptr(), static_cast<uint32_t>(B), static_cast<uint32_t>(L), static_cast<uint32_t>(F),
        static_cast<uint32_t>(head_dim), static_cast<uint32_t>(chunk_size), queries.device().index(),
        static_cast<void*>(stream.stream()), FA_B200_FLAG_DEFAULT);
    TORCH_CHECK(rc == FA_B200_OK, "fa_b200: ", fa_b200_strerror(rc), " (status ", rc, ")");
    return output;
}

// The call behind the package's Python function (fused_attention_b200.attention_forward), positional arguments (entry,
// head_dim, chunk_size, queries, keys, values, mask or None, flags): the output, the status of a launch that failed, or None
// for everything that is not a plain call with every precondition met, which Python then looks at with its own checks (and
// their messages).  `entry` is the address of fa_b200_attention_forward in the library that Python has loaded, which need not
// be the one that this module links (the checked and the clock-counting build).  Checks, allocation and call took 8.4 us in
// Python on B=1 R=4 L=256 H=64, more than the kernel.
bool plain_tensor(PyObject* o, at::Tensor& t) {
    if (!THPVariable_CheckExact(o)) return false;   // a subclass may have its own idea of every operation
    t = THPVariable_Unpack(o);
    using c10::DispatchKey;
    static const c10::DispatchKeySet wrapped({DispatchKey::Python, DispatchKey::FuncTorchBatched, DispatchKey::FuncTorchGradWrapper,
                                              DispatchKey::Functionalize, DispatchKey::Conjugate, DispatchKey::Negative});
    return t.defined() && !t.key_set().has_any(wrapped) && t.scalar_type() == at::kHalf && t.is_cuda() && t.dim() == 3 && t.is_contiguous();
}

PyObject* forward_through(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8 || !PyLong_CheckExact(args[0])) Py_RETURN_NONE;
    auto* const entry = reinterpret_cast<decltype(&fa_b200_attention_forward)>(PyLong_AsVoidPtr(args[0]));
    if (entry == nullptr) {
        PyErr_Clear();
        Py_RETURN_NONE;
    }
    ++args;
    if (!PyLong_CheckExact(args[0]) || !PyLong_CheckExact(args[1]) || !PyLong_CheckExact(args[6]) ||
        at::impl::PythonTorchFunctionTLS::stack_len() > 0)
        Py_RETURN_NONE;
    int over = 0;
    const long H = PyLong_AsLongAndOverflow(args[0], &over), C = over ? 0 : PyLong_AsLongAndOverflow(args[1], &over);
    const long flags = over ? 0 : PyLong_AsLongAndOverflow(args[6], &over);
    auto is_pow2 = [](long x) { return x > 0 && (x & (x - 1)) == 0; };
    if (over || flags < 0 || flags > 0xFFFFFFFFL || !is_pow2(H) || !is_pow2(C) || H < 16 || H > 128 || C < 16 || C > 128 || C > 2 * H ||
        (C == 16 && H == 128))
        Py_RETURN_NONE;
    at::Tensor q, k, v, mask;
    const bool masked = args[5] != Py_None;
    if (!plain_tensor(args[2], q) || !plain_tensor(args[3], k) || !plain_tensor(args[4], v) || (masked && !plain_tensor(args[5], mask)))
        Py_RETURN_NONE;
    const int64_t B = q.size(0), L = q.size(1), F = q.size(2);
    if (k.sizes() != q.sizes() || v.sizes() != q.sizes() || B <= 0 || L <= 0 || F <= 0 || F % H != 0 || B > UINT32_MAX || L > UINT32_MAX ||
        F > UINT32_MAX || k.device() != q.device() || v.device() != q.device() ||
        (masked && (mask.size(0) != B || mask.size(1) != L || mask.size(2) != L || mask.device() != q.device())))
        Py_RETURN_NONE;
    const auto device = q.device().index();
    at::Tensor out = at::empty_like(q);
    const void *pq = q.data_ptr(), *pk = k.data_ptr(), *pv = v.data_ptr(), *pm = masked ? mask.data_ptr() : nullptr;
    void *py = out.data_ptr(), *stream = static_cast<void*>(c10::cuda::getCurrentCUDAStream(device).stream());
    int rc = 0;
    Py_BEGIN_ALLOW_THREADS   // (a call that waits for the stream must not hold other threads up)
    rc = entry(pq, pk, pv, pm, py, static_cast<uint32_t>(B), static_cast<uint32_t>(L), static_cast<uint32_t>(F),
               static_cast<uint32_t>(H), static_cast<uint32_t>(C), device, stream, static_cast<uint32_t>(flags));
    Py_END_ALLOW_THREADS
    if (rc != FA_B200_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}
PyMethodDef forward_through_def = {"_forward_through", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(forward_through)),
                                   METH_FASTCALL, nullptr};

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("attention_forward", &attention_forward, py::arg("head_dim"), py::arg("chunk_size"), py::arg("queries"),
          py::arg("keys"), py::arg("values"), py::arg("mask") = torch::optional<torch::Tensor>(),
          "Fused multihead attention");
    m.add_object("_forward_through", PyCFunction_New(&forward_through_def, nullptr));
}
