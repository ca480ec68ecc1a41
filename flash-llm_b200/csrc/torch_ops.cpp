// CUDA implementations of torch.ops.flashllm.{spmm, spmm_epilogue, encode} (schemas, shape inference and the refusals for
// other devices are registered by torch_op.py).  Checks, result allocation and the call into libSpMM_API.so run here
// because a decode step is launch-bound: from Python the same work took 18-22 us per call, four times the kernel.
//
// The library's entry points are handed over as addresses (flashllm_torch_bind), so that the operators call whichever
// build of the library the package has loaded.
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/library.h>

#include <string>
#include <tuple>

namespace {

using SpmmFn        = int (*)(void*, const void*, const int*, const void*, void*, int, int, int, void*, int, const void*, int,
                       const void*);
using TileOffsetsFn = int (*)(void*, const void*, int, int, int*);
using PackFn        = int (*)(void*, const void*, int, int, const int*, uint32_t*, int);

SpmmFn        g_spmm         = nullptr;
TileOffsetsFn g_tile_offsets = nullptr;
PackFn        g_pack         = nullptr;
PyObject*     g_error_class  = nullptr;  // FlashLLMError

[[noreturn]] void raise_library_error(const std::string& what, int code)
{
    pybind11::gil_scoped_acquire gil;
    PyErr_SetString(g_error_class, (what + " failed with cudaError_t " + std::to_string(code)).c_str());
    throw pybind11::error_already_set();
}

bool is_half_matrix(const at::Tensor& t)
{
    return t.scalar_type() == at::kHalf && t.dim() == 2 && t.is_contiguous();
}

at::Tensor spmm_epilogue(const at::Tensor& compressed, const at::Tensor& tile_offsets, const at::Tensor& B, int64_t M,
                         int64_t split_k, const std::optional<at::Tensor>& bias, int64_t activation,
                         const std::optional<at::Tensor>& residual)
{
    TORCH_CHECK(B.is_cuda(), "flashllm::spmm runs on CUDA tensors only");
    TORCH_CHECK(is_half_matrix(B), "B must be a contiguous fp16 matrix [N][K]");
    TORCH_CHECK(compressed.scalar_type() == at::kInt && tile_offsets.scalar_type() == at::kInt,
                "compressed and tile_offsets must be int32 tensors (tiled-CSL words, offsets in vectors)");
    TORCH_CHECK(compressed.device() == B.device() && tile_offsets.device() == B.device(),
                "all operands must live on one device");
    const int64_t N = B.size(0), K = B.size(1);
    TORCH_CHECK(M % 128 == 0 && K % 64 == 0, "M (", M, ") must be a multiple of 128 and K (", K, ") of 64");
    TORCH_CHECK(tile_offsets.numel() == (M / 128) * (K / 64) + 2, "tile_offsets does not belong to an M x K matrix of this shape");
    const bool has_bias = bias.has_value() && bias->defined(), has_residual = residual.has_value() && residual->defined();
    if (has_bias)
        TORCH_CHECK(bias->scalar_type() == at::kHalf && bias->dim() == 1 && bias->size(0) == M && bias->is_contiguous()
                        && bias->device() == B.device(),
                    "bias must be a contiguous fp16 tensor of shape (", M, ",) on B's device");
    if (has_residual)
        TORCH_CHECK(is_half_matrix(*residual) && residual->size(0) == N && residual->size(1) == M
                        && residual->device() == B.device(),
                    "residual must be a contiguous fp16 tensor of shape (", N, ", ", M, ") on B's device");
    const c10::cuda::CUDAGuard guard(B.device());
    const at::Tensor           C = at::empty({N, M}, B.options());
    at::Tensor                 workspace;
    if (split_k > 1)  // the room the reference's callers bring: Split_K fp16 matrices (reference csrc/SpMM_API.cu:150-152)
        workspace = at::empty({split_k, N, M}, B.options());
    const int code = g_spmm(c10::cuda::getCurrentCUDAStream().stream(), compressed.const_data_ptr(),
                            static_cast<const int*>(tile_offsets.const_data_ptr()), B.const_data_ptr(), C.mutable_data_ptr(),
                            static_cast<int>(M), static_cast<int>(N), static_cast<int>(K),
                            split_k > 1 ? workspace.mutable_data_ptr() : nullptr, static_cast<int>(split_k),
                            has_bias ? bias->const_data_ptr() : nullptr, static_cast<int>(activation),
                            has_residual ? residual->const_data_ptr() : nullptr);
    if (code != 0)
        raise_library_error("SpMM_SplitK_Epilogue(M=" + std::to_string(M) + ", N=" + std::to_string(N) + ", K=" + std::to_string(K)
                                + ", Split_K=" + std::to_string(split_k) + ")",
                            code);
    return C;
}

at::Tensor spmm(const at::Tensor& compressed, const at::Tensor& tile_offsets, const at::Tensor& B, int64_t M, int64_t split_k)
{
    return spmm_epilogue(compressed, tile_offsets, B, M, split_k, std::nullopt, 0, std::nullopt);
}

std::tuple<at::Tensor, at::Tensor> encode(const at::Tensor& A)
{
    TORCH_CHECK(is_half_matrix(A), "A must be a contiguous fp16 matrix [M][K]");
    const int64_t M = A.size(0), K = A.size(1);
    TORCH_CHECK(M % 128 == 0 && K % 64 == 0, "M (", M, ") must be a multiple of 128 and K (", K, ") of 64");
    const c10::cuda::CUDAGuard guard(A.device());
    const cudaStream_t         stream  = c10::cuda::getCurrentCUDAStream().stream();
    const auto                 options = A.options().dtype(at::kInt);
    const int64_t              tiles   = (M / 128) * (K / 64);
    const at::Tensor           offs    = at::empty({tiles + 2}, options);
    int* const                 offs_d  = static_cast<int*>(offs.mutable_data_ptr());
    int                        code    = g_tile_offsets(stream, A.const_data_ptr(), static_cast<int>(M), static_cast<int>(K), offs_d);
    if (code != 0)
        raise_library_error("EncodeOnDevice_TileOffsets", code);
    // The size of the result depends on the data: the one wait of an encoding.  Through page-locked memory (PyTorch's pool of
    // it), a copy to any other is staged.
    const at::Tensor size = at::empty({1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    code = cudaMemcpyAsync(size.mutable_data_ptr(), offs_d + tiles + 1, sizeof(int), cudaMemcpyDeviceToHost, stream);
    if (code == 0)
        code = cudaStreamSynchronize(stream);
    if (code != 0)
        raise_library_error("reading the size of the encoding", code);
    const int64_t    words = static_cast<int64_t>(*static_cast<const int*>(size.const_data_ptr())) * 4;
    const at::Tensor comp  = at::empty({words > 4 ? words : 4}, options);
    code = g_pack(stream, A.const_data_ptr(), static_cast<int>(M), static_cast<int>(K), offs_d,
                  static_cast<uint32_t*>(comp.mutable_data_ptr()), 1);
    if (code != 0)
        raise_library_error("EncodeOnDevice_Pack", code);
    return {words < 4 ? comp.narrow(0, 0, words) : comp, offs};
}

}  // namespace

extern "C" void flashllm_torch_bind(void* spmm_fn, void* tile_offsets_fn, void* pack_fn, PyObject* error_class)
{
    g_spmm         = reinterpret_cast<SpmmFn>(spmm_fn);
    g_tile_offsets = reinterpret_cast<TileOffsetsFn>(tile_offsets_fn);
    g_pack         = reinterpret_cast<PackFn>(pack_fn);
    g_error_class  = error_class;  // kept alive by the package that defines it
}

TORCH_LIBRARY_IMPL(flashllm, CUDA, m)
{
    m.impl("spmm", &spmm);
    m.impl("spmm_epilogue", &spmm_epilogue);
    m.impl("encode", &encode);
}
