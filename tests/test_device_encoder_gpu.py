"""The device tiled-CSL encoder must reproduce the host encoder (and so the reference) bit for bit."""
import numpy as np
import pytest
import torch

from flash_llm_b200 import torch_op  # noqa: F401  (registers torch.ops.flashllm)

pytestmark = pytest.mark.gpu


def _encode_on_device(lib, A_np: np.ndarray, reorder: bool):
    M, K = A_np.shape
    T = (M // 128) * (K // 64)
    A_d = torch.from_numpy(np.ascontiguousarray(A_np.view(np.float16))).cuda()
    offs = torch.full((T + 2,), -7, dtype=torch.int32, device="cuda")
    L = lib.library()
    stream = torch.cuda.current_stream().cuda_stream
    assert L.FlashLLM_EncodeOnDevice_TileOffsets(stream, A_d.data_ptr(), M, K, offs.data_ptr()) == 0
    words = int(offs[T + 1].item()) * 4
    comp = torch.full((max(words, 4),), -1, dtype=torch.int32, device="cuda")
    assert L.FlashLLM_EncodeOnDevice_Pack(stream, A_d.data_ptr(), M, K, offs.data_ptr(), comp.data_ptr(),
                                          1 if reorder else 0) == 0
    torch.cuda.synchronize()
    assert lib.consume_status() == 0
    return comp.cpu().numpy().view(np.uint32)[:words], offs.cpu().numpy()


@pytest.mark.parametrize("M,K,sparsity", [(128, 64, 0.8), (128, 64, 0.0), (128, 64, 1.0), (256, 192, 0.7),
                                          (384, 128, 0.999), (1024, 1024, 0.9), (4096, 4096, 0.8), (128, 128, 0.5)])
@pytest.mark.parametrize("reorder", [True, False])
def test_device_encoder_bit_exact(lib, M, K, sparsity, reorder):
    A = lib.synthetic.sparse_uniform_matrix(M, K, sparsity, seed=M + K).numpy()
    comp_h, offs_h, _ = (lib.InitSparseMatrixA_API if reorder else lib.InitSparseMatrixA_API_NoReorder)(A)
    comp_d, offs_d = _encode_on_device(lib, A, reorder)
    assert np.array_equal(offs_d, offs_h)
    assert np.array_equal(comp_d, comp_h)


def test_device_encoder_golden_and_special_values(lib):
    import glob
    import os
    for path in sorted(glob.glob(os.path.join(os.path.dirname(__file__), "golden", "*.npz"))):
        g = np.load(path)
        for reorder, key in ((True, "compressed_reorder"), (False, "compressed_noreorder")):
            comp_d, offs_d = _encode_on_device(lib, g["A"], reorder)
            assert np.array_equal(offs_d, g["tile_offsets"]), path
            assert np.array_equal(comp_d, g[key]), (path, reorder)


def test_device_encoded_buffers_feed_the_kernel(lib, oracle):
    from helpers import assert_close
    M, K, N = 1024, 2048, 16
    A = lib.synthetic.sparse_uniform_matrix(M, K, 0.8, seed=9)
    B = lib.synthetic.dense_uniform_matrix(N, K, 10)
    A_d, B_d = A.cuda(), B.cuda()
    T = (M // 128) * (K // 64)
    stream = torch.cuda.current_stream().cuda_stream
    comp, offs, n, words = lib.encode_on_device(
        stream, A_d.data_ptr(), M, K,
        lambda n: (lambda t: (t, t.data_ptr()))(torch.empty(n, dtype=torch.int32, device="cuda")),
        lambda n: (lambda t: (t, t.data_ptr()))(torch.empty(n, dtype=torch.int32, device="cuda")),
        lambda owner, i: owner[i].item())
    assert n == T + 2
    C = torch.empty((N, M), dtype=torch.float16, device="cuda")
    lib.SpMM_SplitK_API(stream, None, comp.data_ptr(), offs.data_ptr(), B_d.data_ptr(), C.data_ptr(), M, N, K, None, 1)
    torch.cuda.synchronize()
    assert lib.consume_status() == 0
    assert_close(C.cpu().numpy(), oracle.gemm_f32(A.numpy(), B.numpy()), "device-encoded SpMM")


@pytest.mark.parametrize("reorder", [1, 0])
def test_an_overlapped_spmm_right_behind_the_encoder(lib, oracle, reorder):
    """With launch overlap on an SpMM reads its words before it waits for its predecessors; enqueued right behind the encoder,
    into buffers that still hold another matrix of another sparsity, it must find the new words and offsets."""
    from helpers import assert_close
    M, K, N = 4096, 2048, 16
    B = lib.synthetic.dense_uniform_matrix(N, K, 10)
    As = [lib.synthetic.sparse_uniform_matrix(M, K, s, seed) for seed, s in ((11, 0.8), (12, 0.6))]
    wants = [oracle.gemm_f32(A.numpy(), B.numpy()) for A in As]
    As, B_d = [A.cuda() for A in As], B.cuda()
    words = torch.zeros(M * K, dtype=torch.int32, device="cuda")
    offs = torch.zeros((M // 128) * (K // 64) + 2, dtype=torch.int32, device="cuda")
    outs = [torch.empty((N, M), dtype=torch.float16, device="cuda") for _ in range(12)]
    L, stream = lib.library(), torch.cuda.current_stream().cuda_stream
    lib.set_launch_overlap(True)
    try:
        for i, C in enumerate(outs):
            A = As[i % 2]
            assert L.FlashLLM_EncodeOnDevice_TileOffsets(stream, A.data_ptr(), M, K, offs.data_ptr()) == 0
            assert L.FlashLLM_EncodeOnDevice_Pack(stream, A.data_ptr(), M, K, offs.data_ptr(), words.data_ptr(), reorder) == 0
            lib.SpMM_SplitK_API(stream, None, words.data_ptr(), offs.data_ptr(), B_d.data_ptr(), C.data_ptr(), M, N, K, None, 1)
        torch.cuda.synchronize()
    finally:
        lib.set_launch_overlap(False)
    assert lib.consume_status() == 0
    for i, C in enumerate(outs):
        assert_close(C.cpu().numpy(), wants[i % 2], f"call {i}")


@pytest.mark.parametrize("shift", [0, 2])
def test_tiles_of_every_density_and_special_values(lib, shift):
    """Tiles on both sides of the density that has a kernel of its own (1088 vectors), sparse ones with a full bucket (a warp's
    lists hold 164 words), zeros, NaN, infinities and subnormals among them; groups of 32 tiles that end in the middle of a row; A only 4-byte aligned."""
    M, K = 128 * 5, 64 * 27
    rng = np.random.default_rng(5)
    A = rng.uniform(-1, 1, (M, K)).astype(np.float16)
    density = rng.choice([0.0, 0.05, 0.2, 0.4, 0.5, 0.53, 0.54, 0.6, 0.9, 1.0], size=(M // 128, K // 64))
    A[rng.random((M, K)) >= np.kron(density, np.ones((128, 64)))] = 0
    bits = A.view(np.uint16)
    special = rng.random((M, K))
    for i, b in enumerate((0x8000, 0x7C00, 0xFC00, 0x7E00, 0xFFFF, 0x0001, 0x83FF)):
        bits[(special > i * 0.004) & (special <= (i + 1) * 0.004)] = b
    for r in range(128):  # bucket 3 of the first tile full, bucket 31 of the last one but for its last cells
        for tile_row, tile_col, bucket in ((0, 0, 3), (4, 26, 31)):
            c = tile_col * 64 + ((2 * bucket) ^ ((r & 7) << 3))
            if r % 3:
                A[tile_row * 128 + r, tile_col * 64:tile_col * 64 + 64] = 0
            A[tile_row * 128 + r, c:c + 2] = 0.5 if r < 126 or tile_row == 0 else 0
    comp_h, offs_h, _ = lib.InitSparseMatrixA_API(A)
    flat = torch.zeros(M * K + 8, dtype=torch.float16, device="cuda")
    A_d = flat[shift:shift + M * K]
    A_d.copy_(torch.from_numpy(A).view(-1))
    assert (A_d.data_ptr() % 16 == 0) == (shift == 0)
    T = offs_h.size - 2
    offs = torch.full((T + 2,), -7, dtype=torch.int32, device="cuda")
    comp = torch.full((comp_h.size + 4,), -1, dtype=torch.int32, device="cuda")
    L, stream = lib.library(), torch.cuda.current_stream().cuda_stream
    assert L.FlashLLM_EncodeOnDevice_TileOffsets(stream, A_d.data_ptr(), M, K, offs.data_ptr()) == 0
    for start in (0, 1):  # words to a 16-byte aligned place, and to a 4-byte aligned one
        comp.fill_(-1)
        assert L.FlashLLM_EncodeOnDevice_Pack(stream, A_d.data_ptr(), M, K, offs.data_ptr(), comp.data_ptr() + 4 * start, 1) == 0
        torch.cuda.synchronize()
        assert lib.consume_status() == 0
        assert np.array_equal(offs.cpu().numpy(), offs_h)
        got = comp.cpu().numpy().view(np.uint32)
        assert np.array_equal(got[start:start + comp_h.size], comp_h)
        assert (got[:start] == 0xFFFFFFFF).all() and (got[start + comp_h.size:] == 0xFFFFFFFF).all()


@pytest.mark.parametrize("tiles", [31, 33, 32 * 1024, 32 * 1024 + 1])
def test_offsets_over_many_groups(lib, tiles):
    """The offsets' two levels at the edges of a group (32 tiles) and of a round (1024 groups), against a plain cumulative sum."""
    A = torch.zeros((128, 64 * tiles), dtype=torch.float16, device="cuda")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(tiles)
    A[:3] = (torch.rand((3, 64 * tiles), generator=gen, device="cuda") < 0.3).half()
    vectors = ((A[:3] != 0).view(3, tiles, 64).sum((0, 2)) + 3) // 4
    _, offs = torch.ops.flashllm.encode(A)
    want = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), vectors.cumsum(0), vectors.sum().view(1)])
    assert torch.equal(offs.long(), want)
