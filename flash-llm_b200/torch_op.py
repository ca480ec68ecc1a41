"""``torch.ops.flashllm``: the library's SpMM as PyTorch operators, for integration tests and for callers whose tensors
live in torch.  Importing this module registers

* ``flashllm::encode(Tensor A) -> (Tensor compressed, Tensor tile_offsets)``: a dense fp16 weight ``A[M][K]`` on a CUDA
  device to its tiled-CSL form (int32 words, int32 tile offsets) with the device encoder; what the reference does on
  the host with ``InitSparseMatrixA_API`` (reference csrc/SpMM_API.cu:449-494).
* ``flashllm::spmm(Tensor compressed, Tensor tile_offsets, Tensor B, int M, int split_k=1) -> Tensor``:
  ``C[N][M] = B[N][K] @ A[M][K]^T`` (reference ``SpMM_SplitK_API``, csrc/SpMM_API.cu:124-171).
* ``flashllm::spmm_epilogue(..., Tensor? bias, int activation, Tensor? residual) -> Tensor``: the same with
  ``act(. + bias[M]) + residual[N][M]`` applied to the fp32 sums before the one rounding.

The operators run on the current CUDA stream of B's device and call the library through its C ABI; there is no CPU
implementation (a CPU tensor is refused), only shape inference for meta tensors.  Their CUDA side is native
(csrc/torch_ops.cpp, ``build/libflashllm_torch.so``): a decode step is launch-bound, and from Python the checks, the
result's allocation and the call took 18-22 us of host time around a 6 us kernel.
"""
from __future__ import annotations

import ctypes
import os

import torch

from . import api

OPERATORS_PATH = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "build", "libflashllm_torch.so")

_LIB = torch.library.Library("flashllm", "DEF")
_LIB.define("encode(Tensor A) -> (Tensor, Tensor)")
_LIB.define("spmm(Tensor compressed, Tensor tile_offsets, Tensor B, int M, int split_k=1) -> Tensor")
_LIB.define("spmm_epilogue(Tensor compressed, Tensor tile_offsets, Tensor B, int M, int split_k=1, Tensor? bias=None, "
            "int activation=0, Tensor? residual=None) -> Tensor")


def _load_operators() -> None:
    """Registers the CUDA implementations and binds them to the library build that :mod:`api` has loaded."""
    if not os.path.exists(OPERATORS_PATH):
        raise api.FlashLLMError(f"{OPERATORS_PATH} is missing: build it with `make -C flash-llm_b200/csrc all operators` "
                                "(or __graft_entry__.build()); there is no fallback implementation")
    library = api.library()
    torch.ops.load_library(OPERATORS_PATH)
    bind = ctypes.CDLL(OPERATORS_PATH).flashllm_torch_bind
    bind.restype, bind.argtypes = None, [ctypes.c_void_p] * 3 + [ctypes.py_object]
    bind(*(ctypes.cast(f, ctypes.c_void_p) for f in (library.FlashLLM_SpMM_SplitK_Epilogue,
                                                     library.FlashLLM_EncodeOnDevice_TileOffsets,
                                                     library.FlashLLM_EncodeOnDevice_Pack)), api.FlashLLMError)


try:
    _load_operators()
except (api.FlashLLMError, OSError) as _error:
    # Schemas and shape inference work without the library (a build of torch without CUDA, a host that only traces);
    # whoever runs an operator is told.
    _reason = str(_error)

    def _refuse_cuda(*args, **kwargs):
        raise api.FlashLLMError(f"the flashllm operators could not be loaded: {_reason}")

    for _name in ("encode", "spmm", "spmm_epilogue"):
        _LIB.impl(_name, _refuse_cuda, "CUDA")


def _refuse_cpu(*args, **kwargs):
    raise RuntimeError("flashllm operators have no CPU implementation: move the tensors to a CUDA device")


for _name in ("encode", "spmm", "spmm_epilogue"):
    _LIB.impl(_name, _refuse_cpu, "CPU")


@torch.library.register_fake("flashllm::spmm")
def _spmm_fake(compressed, tile_offsets, B, M, split_k=1):
    return B.new_empty((B.shape[0], M))


@torch.library.register_fake("flashllm::spmm_epilogue")
def _spmm_epilogue_fake(compressed, tile_offsets, B, M, split_k=1, bias=None, activation=0, residual=None):
    return B.new_empty((B.shape[0], M))


def spmm(compressed: torch.Tensor, tile_offsets: torch.Tensor, B: torch.Tensor, M: int, split_k: int = 1) -> torch.Tensor:
    """Python spelling of ``torch.ops.flashllm.spmm``."""
    return torch.ops.flashllm.spmm(compressed, tile_offsets, B, M, split_k)
