"""Workloads the library is timed on: sparse decoder matmuls from single projections to whole layers, prefill widths,
and the device encoder, each through its public entry point.

``listed()`` names the fixed ones, ``draw(rng)`` samples further ones from the same ranges.  A case is a plain dict;
its ``kind`` selects the entry point:

* ``spmm``    the C ABI call a drop-in host makes: ``SpMM_SplitK_API``, or ``spmm_splitk_epilogue`` when the host lets
              the library add bias, ReLU or the residual.  Buffers and workspace belong to the caller.
* ``op``      the same product as a PyTorch operator, ``torch.ops.flashllm.spmm_epilogue``, which allocates its result.
* ``layer``   one pass over a sparse decoder layer held by one GPU, ``tp_chain.DeviceChain.step``.
* ``encode``  dense fp16 weights to tiled-CSL on the GPU, ``torch.ops.flashllm.encode``.

Weights are fp16 with unstructured sparsity: uniform values under a Bernoulli mask, or (``layer``) normal values pruned
by magnitude.  Activations are fp16.  All of it is generated on the GPU from the seed.
"""
from __future__ import annotations

import math
import statistics

import torch

import flash_llm_b200 as fl
from flash_llm_b200 import torch_op  # noqa: F401  (registers torch.ops.flashllm)
from flash_llm_b200.tp_chain import ChainShape, DeviceChain

DEVICE = torch.device("cuda:0")
ROWS_PER_BLOCK = 4096  # rows of a weight matrix generated at a time (bounds the fp32 temporaries)

# Decode batches and prefill widths the SpMM accepts.
DECODE_TOKENS = (8, 16, 32, 64)
PREFILL_TOKENS = (128, 256, 384, 512)
# Values callers pass for Split_K: uncut, powers of two, and the tuned tables of the reference's benchmark (2, 3, 6, 9).
SPLIT_K = (1, 2, 3, 4, 6, 8, 9)

SPMM_DEFAULTS = {"kind": "spmm", "split_k": 1, "bias": False, "relu": False, "residual": False, "scan_order": False,
                 "overlap": False}


def _spmm(name, M, K, N, sparsity, **more):
    return {**SPMM_DEFAULTS, "name": name, "M": M, "K": K, "N": N, "sparsity": sparsity, **more}


def listed():
    return [
        # One small projection, the least work a call can carry: launch and latency.
        _spmm("decode 1024x1024 n8", 1024, 1024, 8, 0.80),
        # The single-SpMM configuration of the benchmark, uncut.
        _spmm("decode 4096x4096 n16", 4096, 4096, 16, 0.80),
        # One GPU's slice of an attention output projection (hidden 9216 over 8 GPUs) called from PyTorch, bias and
        # residual fused.
        {**SPMM_DEFAULTS, "kind": "op", "name": "op 9216x1152 n16", "M": 9216, "K": 1152, "N": 16, "sparsity": 0.80,
         "split_k": 6, "bias": True, "residual": True},
        # Few rows and a long K: every tile row has to be cut to fill the GPU (split-K stress configuration).
        _spmm("decode 2048x32768 n16", 2048, 32768, 16, 0.70, split_k=4),
        # QKV projection of a hidden-9216 layer at the highest sparsity and the smallest batch.
        _spmm("decode 27648x9216 n8 s90", 27648, 9216, 8, 0.90, split_k=2),
        # First feed-forward matmul of the same layer, the benchmark's largest matrix, with its bias and ReLU.
        _spmm("decode 36864x9216 n16", 36864, 9216, 16, 0.80, split_k=3, bias=True, relu=True),
        # Second feed-forward matmul at a larger batch and the lowest sparsity, with bias and residual.
        _spmm("decode 9216x36864 n32 s70", 9216, 36864, 32, 0.70, split_k=6, bias=True, residual=True),
        # First feed-forward matmul of a hidden-12288 layer at the largest decode batch.
        _spmm("decode 49152x12288 n64", 49152, 12288, 64, 0.80, split_k=9),
        # Sizes that divide by nothing but the tile, words in scan order as InitSparseMatrixA_API_NoReorder leaves them.
        _spmm("decode 4736x7232 n32 scan", 4736, 7232, 32, 0.75, split_k=3, scan_order=True),
        # Prompt processing: 512 tokens through the first feed-forward matmul.
        _spmm("prefill 36864x9216 n512", 36864, 9216, 512, 0.80),
        # A whole hidden-9216 decoder layer in a decode loop: four dependent matmuls, launch overlap on.
        {"kind": "layer", "name": "layer 9216 n16", "hidden": 9216, "ffn": 36864, "N": 16, "sparsity": 0.80,
         "overlap": True},
        # Encoding the benchmark's largest matrix when a model is loaded.
        {"kind": "encode", "name": "encode 36864x9216", "M": 36864, "K": 9216, "sparsity": 0.80},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _shape(rng, fewest, most, sparsity):
    """(M, K) with `fewest`..`most` weights (fewer where they are denser than the listed 80 %), spread over the logarithm,
    from 8 times wider than long to 16 times longer than wide; M any multiple of 128, K any multiple of 64."""
    most *= min(1.0, 0.2 / (1 - sparsity))
    weights, aspect = _log_uniform(rng, fewest, most), _log_uniform(rng, 1 / 8, 16)
    M = max(1, round(math.sqrt(weights / aspect) / 128)) * 128
    K = max(1, int(weights / M) // 64) * 64
    return M, K


def draw(rng):
    kind = rng.choices(("spmm", "prefill", "op", "layer", "encode"), (9, 3, 3, 2, 3))[0]
    sparsity = round(rng.uniform(0.60, 0.95), 3)
    if kind == "encode":
        M, K = _shape(rng, 1 << 20, 36864 * 9216, sparsity)
        return {"kind": "encode", "M": M, "K": K, "sparsity": sparsity}
    if kind == "layer":
        most = 9216 * min(1.0, math.sqrt(0.2 / (1 - sparsity)))
        hidden = int(_log_uniform(rng, 1024, most + 128) / 128) * 128
        return {"kind": "layer", "hidden": hidden, "ffn": 4 * hidden, "N": rng.choice(DECODE_TOKENS), "sparsity": sparsity,
                "overlap": rng.random() < 0.75}
    case = dict(SPMM_DEFAULTS)
    if kind == "prefill":
        N = rng.choice(PREFILL_TOKENS)
        M, K = _shape(rng, 1 << 21, 36864 * 9216, sparsity)
    elif kind == "op":
        case["kind"] = "op"
        N = rng.choice(DECODE_TOKENS)
        M, K = _shape(rng, 1 << 20, 9216 * 9216, sparsity)
    else:
        N = rng.choice(DECODE_TOKENS)
        M, K = _shape(rng, 1 << 20, 49152 * 12288, sparsity)
        case["scan_order"] = rng.random() < 0.15
        case["overlap"] = rng.random() < 0.25
    epilogue = rng.choice(((False, False, False), (True, False, False), (True, True, False), (True, False, True)))
    case.update(M=M, K=K, N=N, sparsity=sparsity, split_k=rng.choice(SPLIT_K))
    case.update(zip(("bias", "relu", "residual"), epilogue))
    return case


# --------------------------------------------------------------------------------------------------- inputs

def _uniform(gen, rows, cols):
    return (torch.rand((rows, cols), generator=gen, device=DEVICE) * 2 - 1).to(torch.float16)


def _sparse_weights(gen, M, K, sparsity, pattern=None):
    """fp16 [M][K]: values U(-1, 1), none of them zero, under a Bernoulli(1 - sparsity) mask drawn from `pattern` (from
    `gen` by default)."""
    A = torch.empty((M, K), dtype=torch.float16, device=DEVICE)
    for r in range(0, M, ROWS_PER_BLOCK):
        block = A[r:r + ROWS_PER_BLOCK]
        keep = torch.rand(block.shape, generator=gen if pattern is None else pattern, device=DEVICE) >= sparsity
        value = torch.rand(block.shape, generator=gen, device=DEVICE) * 2 - 1
        block.copy_((value + torch.copysign(torch.full_like(value, 1e-4), value)) * keep)
    return A


def _weights_to_encode(gen, case):
    """Weights whose encoding is equally long for every seed: one sparsity pattern per case, moved by whole 128x64 tiles."""
    M, K = case["M"], case["K"]
    pattern = torch.Generator(device=DEVICE)
    pattern.manual_seed(M * K)
    A = _sparse_weights(gen, M, K, case["sparsity"], pattern)
    rows, cols = (int(torch.randint(n, (1,), generator=gen, device=DEVICE)) for n in (M // 128, K // 64))
    return A.roll((128 * rows, 64 * cols), (0, 1))


def _pruned_weights(gen, M, K, sparsity):
    """fp16 [M][K]: N(0, 0.02) values with (up to sampling) the smallest `sparsity` share by magnitude set to zero."""
    threshold = statistics.NormalDist().inv_cdf((1 + sparsity) / 2)
    A = torch.empty((M, K), dtype=torch.float16, device=DEVICE)
    for r in range(0, M, ROWS_PER_BLOCK):
        block = A[r:r + ROWS_PER_BLOCK]
        w = torch.randn(block.shape, generator=gen, device=DEVICE)
        block.copy_(0.02 * w * (w.abs() >= threshold))
    return A


def _encoded(A, scan_order):
    """(words, tile offsets) of a dense matrix, in the reordered or the scan-order form."""
    if not scan_order:
        return torch.ops.flashllm.encode(A)
    M, K = A.shape
    stream = torch.cuda.current_stream().cuda_stream
    offs = torch.empty((M // 128) * (K // 64) + 2, dtype=torch.int32, device=DEVICE)
    code = fl.library().FlashLLM_EncodeOnDevice_TileOffsets(stream, A.data_ptr(), M, K, offs.data_ptr())
    words = torch.empty(4 * int(offs[-1].item()), dtype=torch.int32, device=DEVICE)
    code |= fl.library().FlashLLM_EncodeOnDevice_Pack(stream, A.data_ptr(), M, K, offs.data_ptr(), words.data_ptr(), 0)
    if code != 0:
        raise RuntimeError(f"device encoder failed with cudaError_t {code}")
    return words, offs


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    stream = torch.cuda.current_stream(DEVICE).cuda_stream
    kind = case["kind"]
    if kind == "encode":
        return {"kind": kind, "A": _weights_to_encode(gen, case)}
    # Process-wide, set once by a serving program whose weights are resident before its loop.
    fl.set_launch_overlap(case["overlap"])
    if kind == "layer":
        shape = ChainShape(hidden=case["hidden"], ffn=case["ffn"], tokens=case["N"], world=1)
        shards = {name: _pruned_weights(gen, M, K, case["sparsity"]) for name, (M, K) in shape.shard_shapes().items()}
        x = torch.randn((case["N"], case["hidden"]), generator=gen, device=DEVICE).to(torch.float16)
        return {"kind": kind, "chain": DeviceChain(fl, shape, shards, DEVICE, split_k=8), "x": x}
    M, K, N, split_k = case["M"], case["K"], case["N"], case["split_k"]
    words, offs = _encoded(_sparse_weights(gen, M, K, case["sparsity"]), case["scan_order"])
    state = {"kind": kind, "M": M, "K": K, "N": N, "split_k": split_k, "stream": stream, "words": words, "offs": offs,
             "B": _uniform(gen, N, K), "relu": case["relu"],
             "bias": _uniform(gen, 1, M).view(M) if case["bias"] else None,
             "residual": _uniform(gen, N, M) if case["residual"] else None}
    if kind == "spmm":
        state["C"] = torch.empty((N, M), dtype=torch.float16, device=DEVICE)
        state["workspace"] = torch.empty((split_k, N, M), dtype=torch.float16, device=DEVICE) if split_k > 1 else None
    return state


# --------------------------------------------------------------------------------------------------- one pass

def _pointer(t):
    return None if t is None else t.data_ptr()


def run(state):
    kind = state["kind"]
    if kind == "encode":
        return torch.ops.flashllm.encode(state["A"])
    if kind == "layer":
        return state["chain"].step(state["x"], all_reduce=lambda t: t)
    activation = fl.ACT_RELU if state["relu"] else fl.ACT_NONE
    if kind == "op":
        return torch.ops.flashllm.spmm_epilogue(state["words"], state["offs"], state["B"], state["M"], state["split_k"],
                                                state["bias"], activation, state["residual"])
    M, N, K = state["M"], state["N"], state["K"]
    C, workspace = state["C"], _pointer(state["workspace"])
    if state["bias"] is None and state["residual"] is None and not state["relu"]:
        fl.SpMM_SplitK_API(state["stream"], None, state["words"].data_ptr(), state["offs"].data_ptr(),
                           state["B"].data_ptr(), C.data_ptr(), M, N, K, workspace, state["split_k"])
    else:
        fl.spmm_splitk_epilogue(state["stream"], state["words"].data_ptr(), state["offs"].data_ptr(),
                                state["B"].data_ptr(), C.data_ptr(), M, N, K, workspace, state["split_k"],
                                _pointer(state["bias"]), activation, _pointer(state["residual"]))
    return C


# --------------------------------------------------------------------------------------------------- accounting

def _weight_bytes(M, K, sparsity):
    """Tiled-CSL bytes of a matrix: a 4-byte word per non-zero (tiles are padded by 1.5 words on average) and the tile
    offsets."""
    tiles = (M // 128) * (K // 64)
    return 4 * (M * K * (1 - sparsity) + 1.5 * tiles) + 4 * (tiles + 2)


def _matmul_work(M, K, N, sparsity):
    """Bytes and multiply-add operations of one product: compressed weights, B and C once; every weight that is not
    zero meets every token."""
    return _weight_bytes(M, K, sparsity) + 2 * N * (K + M), 2 * M * K * N * (1 - sparsity)


def work(case):
    if case["kind"] == "encode":
        M, K = case["M"], case["K"]
        return {"bytes": 2 * M * K + _weight_bytes(M, K, case["sparsity"]), "flops": 0}
    if case["kind"] == "layer":
        H, F, N = case["hidden"], case["ffn"], case["N"]
        parts = [_matmul_work(M, K, N, case["sparsity"]) for M, K in ((3 * H, H), (H, H), (F, H), (H, F))]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    total, flops = _matmul_work(case["M"], case["K"], case["N"], case["sparsity"])
    total += 2 * case["M"] * case["bias"] + 2 * case["N"] * case["M"] * case["residual"]
    if case["N"] >= 128:  # prefill runs on the tensor cores as a dense contraction
        flops = 2 * case["M"] * case["K"] * case["N"]
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Encoded words are exact.  Products are fp32 sums in some order rounded to fp16 once: neighbouring fp16 values may
    be chosen (2^-11 of a value), rarely, so 5e-4 over the whole output; a layer rounds four times in a row."""
    if case["kind"] == "encode":
        return "exact"
    return {"rel": 2e-3, "max": 2e-2} if case["kind"] == "layer" else {"rel": 5e-4, "max": 4e-3}
