"""The wide form of the SpMM kernel (a CTA multiplies a tile by 256, 384 or 512 output columns) at its widths' edges: output
columns beyond N, one K tile, fewer K tiles than stages, K cut in clusters and in the workspace, tiles above the register
budget, every output epilogue, malformed offsets."""
import numpy as np
import pytest
import torch

from helpers import DeviceProblem, assert_close, random_problem

pytestmark = pytest.mark.gpu


@pytest.fixture
def pinned(lib):
    yield lambda **plan: lib.set_plan(path=lib.api.PATH_WIDE, **plan)
    lib.set_plan()


@pytest.mark.parametrize("width", [2, 3, 4])
@pytest.mark.parametrize("M,K,N,sparsity", [
    (128, 64, 512, 0.8),         # one tile; at width 384 columns beyond N
    (384, 64 * 5, 512, 0.9),     # fewer K tiles than stages
    (256, 64 * 9, 640, 0.8),     # one K tile more than eight stages; groups of columns partly and wholly beyond N
    (256, 64 * 31, 896, 0.7),
    (128, 64 * 13, 1024, 0.4),   # tiles above the register budget
    (128, 64 * 7, 512, 0.0),     # dense tiles
    (128, 64 * 900, 512, 0.995), # more offsets than shared memory stages
])
def test_widths(lib, oracle, pinned, width, M, K, N, sparsity):
    A, B = random_problem(lib, M, K, N, sparsity, M + K + N)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    pinned(producers=width)
    assert_close(DeviceProblem(lib, comp, offs, B, M, N, K, 1).run(), oracle.gemm_f32(A, B), f"{width * 128} columns, {M}x{K} N={N}")


@pytest.mark.parametrize("width,cluster_k,workspace_k", [(2, 2, 1), (2, 8, 1), (3, 3, 1), (3, 8, 2), (2, 1, 4), (4, 1, 3), (2, 5, 3)])
def test_cut_k(lib, oracle, pinned, width, cluster_k, workspace_k):
    M, K, N = 256, 64 * 29, 512
    A, B = random_problem(lib, M, K, N, 0.8, 41)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    pinned(producers=width, cluster_k=cluster_k, workspace_k=workspace_k)
    prob = DeviceProblem(lib, comp, offs, B, M, N, K, 8)
    first = prob.run().copy()
    assert_close(first, oracle.gemm_f32(A, B), f"{width * 128} columns, {cluster_k} x {workspace_k} parts")
    assert np.array_equal(prob.run(), first)


@pytest.mark.parametrize("bias,relu,residual", [(True, False, False), (True, True, False), (True, False, True), (False, True, True)])
@pytest.mark.parametrize("cluster_k", [1, 2])
def test_output_epilogues(lib, oracle, pinned, bias, relu, residual, cluster_k):
    M, K, N = 384, 64 * 11, 384
    A, B = random_problem(lib, M, K, N, 0.8, 17)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    rng = np.random.default_rng(18)
    b = (rng.standard_normal(M) * 2).astype(np.float16)
    r = (rng.standard_normal((N, M)) * 4).astype(np.float16)
    want = oracle.gemm_f32(A, B) + (b.astype(np.float32)[None, :] if bias else 0)
    want = (np.maximum(want, 0) if relu else want) + (r.astype(np.float32) if residual else 0)
    to_dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    comp_d, offs_d, B_d, b_d, r_d = to_dev(comp.view(np.int32)), to_dev(offs), to_dev(B), to_dev(b), to_dev(r)
    pinned(producers=3, cluster_k=cluster_k)
    for shift in (0, 1):  # C only two-byte aligned takes narrow stores
        C = torch.full((N * M + 8,), float("nan"), dtype=torch.float16, device="cuda")[shift:shift + N * M]
        lib.spmm_splitk_epilogue(torch.cuda.current_stream().cuda_stream, comp_d.data_ptr(), offs_d.data_ptr(), B_d.data_ptr(),
                                 C.data_ptr(), M, N, K, None, 1, b_d.data_ptr() if bias else None,
                                 lib.ACT_RELU if relu else lib.ACT_NONE, r_d.data_ptr() if residual else None)
        torch.cuda.synchronize()
        assert lib.consume_status() == 0
        assert_close(C.view(N, M).cpu().numpy(), want, f"bias={bias} relu={relu} residual={residual} shift={shift}")


def test_chosen_where_it_saves_decompression(lib, oracle):
    M, K, N = 128 * 150, 64 * 16, 512
    assert lib.get_plan(M, N, K, 1)["path"] == lib.api.PATH_WIDE
    assert lib.get_plan(M, 128, K, 1)["path"] != lib.api.PATH_WIDE
    A, B = random_problem(lib, M, K, N, 0.8, 3)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    assert_close(DeviceProblem(lib, comp, offs, B, M, N, K, 1).run(), oracle.gemm_f32(A, B), "automatic")


def test_two_accumulators_at_256_columns(lib):
    """As the streaming form's test of the same kind: sums of positive products, whose mean shortfall against 64-bit products
    must not be larger than that of 128 columns per CTA, which alternate between two accumulators (allowance 1e-6: ten times
    the 2^-11 / sqrt(12 * 2400000) that rounding to fp16 leaves)."""
    from flash_llm_b200 import torch_op  # noqa: F401  (registers torch.ops.flashllm)
    M, K, N = 128 * 74, 9216, 256
    gen = torch.Generator(device="cuda")
    gen.manual_seed(7)
    A = torch.rand((M, K), generator=gen, device="cuda").half()
    A *= torch.rand((M, K), generator=gen, device="cuda") >= 0.8
    B = torch.rand((N, K), generator=gen, device="cuda").half()
    want = torch.cat([B.double() @ A[r:r + 1024].double().T for r in range(0, M, 1024)], dim=1)
    words, offs = torch.ops.flashllm.encode(A)
    share = {}
    try:
        for path, width in ((lib.api.PATH_WIDE, 2), (lib.api.PATH_DIRECT, 0)):
            lib.set_plan(path=path, producers=width, cluster_k=1)
            share[path] = float(((want - torch.ops.flashllm.spmm(words, offs, B, M).double()) / want).mean())
    finally:
        lib.set_plan()
    assert lib.consume_status() == 0
    assert abs(share[lib.api.PATH_WIDE]) <= abs(share[lib.api.PATH_DIRECT]) + 1e-6, share


def test_malformed_offsets_are_reported_not_followed(lib, oracle, pinned):
    M, K, N = 384, 64 * 20, 256
    A, B = random_problem(lib, M, K, N, 0.8, 31)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    broken = offs.copy()
    broken[25] = broken[24] - 3
    pinned(producers=2, cluster_k=1)
    got = DeviceProblem(lib, comp, broken, B, M, N, K, 1).run(check_status=False)
    assert lib.consume_status() & 2
    want = oracle.gemm_f32(A, B)
    assert np.isnan(got[:, 128:256]).all(), "the row with the malformed offsets is not stored"
    assert_close(np.delete(got, np.s_[128:256], axis=1), np.delete(want, np.s_[128:256], axis=1), "the other rows")
    assert_close(DeviceProblem(lib, comp, offs, B, M, N, K, 1).run(), want, "call after a malformed one")
