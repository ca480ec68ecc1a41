"""The streaming form of the SpMM kernel (a persistent grid over the linear tile sequence) where its shares of the
sequence can go wrong: fewer tiles than CTAs, shares inside one tile row, shares that end exactly at a row's end, rows cut
into two and into many parts, tiles above the register budget; with every output epilogue, on several streams, and with
malformed offsets."""
import numpy as np
import pytest
import torch

from helpers import DeviceProblem, assert_close, random_problem

pytestmark = pytest.mark.gpu


@pytest.fixture
def streaming(lib):
    lib.set_plan(path=lib.api.PATH_STREAM)
    yield
    lib.set_plan()


@pytest.mark.parametrize("M,K,N,sparsity", [
    (128, 64, 16, 0.8),          # one tile, one CTA
    (128, 64 * 37, 8, 0.8),      # one row in 37 single-tile parts
    (384, 64 * 5, 32, 0.7),      # fewer tiles than CTAs, three rows
    (128 * 37, 64 * 8, 16, 0.9), # 296 tiles: one per CTA on 148 SMs, eight parts to a row
    (128 * 37, 64 * 16, 64, 0.8),# two tiles per CTA, shares ending at row ends
    (128 * 41, 64 * 13, 16, 0.8),# nothing divides anything
    (128 * 74, 64 * 9, 32, 0.75),# rows cut into two or three parts
    (128 * 300, 64 * 3, 16, 0.8),# more rows than CTAs: whole rows inside a share
    (256, 64 * 700, 16, 0.5),    # long shares, tiles above the register budget
    (256, 64 * 400, 64, 0.99),   # many parts of a wide output, nearly empty tiles
])
def test_shares_of_the_tile_sequence(lib, oracle, streaming, M, K, N, sparsity):
    A, B = random_problem(lib, M, K, N, sparsity, M + K + N)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    prob = DeviceProblem(lib, comp, offs, B, M, N, K, 1)
    first = prob.run().copy()
    assert_close(first, oracle.gemm_f32(A, B), f"M={M} K={K} N={N} s={sparsity}")
    for _ in range(5):  # parts are added in CTA order, whichever CTA finishes the row
        assert np.array_equal(prob.run(), first)


@pytest.mark.parametrize("M,K", [
    (128 * 300, 64 * 40),  # 40.5 tiles a CTA, 40 a row: last segments of one tile and more, first ones of 39 and fewer
    (128 * 150, 64 * 64),  # 32.4 tiles a CTA: every row is cut once or twice
    (128 * 148, 64 * 24),  # 12 tiles a CTA: every row belongs to two, neither of which has begun before it
])
@pytest.mark.parametrize("N", [8, 32, 64])
def test_rows_of_two_shares(lib, streaming, M, K, N):
    """The CTA that holds a row's first part finishes the row from tensor memory when the other part is there already, and
    parks its own when it is not; either way the same bits."""
    from flash_llm_b200 import torch_op  # noqa: F401  (registers torch.ops.flashllm)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + K + N)
    A = (torch.rand((M, K), generator=gen, device="cuda") - 0.5).half()
    A *= torch.rand((M, K), generator=gen, device="cuda") >= 0.8
    B = (torch.rand((N, K), generator=gen, device="cuda") - 0.5).half()
    bias = (torch.rand(M, generator=gen, device="cuda") - 0.5).half()
    residual = (torch.rand((N, M), generator=gen, device="cuda") - 0.5).half()
    words, offs = torch.ops.flashllm.encode(A)
    want = (B.double() @ A.double().T + bias.double() + residual.double()).float().cpu().numpy()
    first = torch.ops.flashllm.spmm_epilogue(words, offs, B, M, 1, bias, 0, residual)
    assert_close(first.cpu().numpy(), want, f"M={M} K={K} N={N}")
    for _ in range(20):
        assert torch.equal(torch.ops.flashllm.spmm_epilogue(words, offs, B, M, 1, bias, 0, residual), first)
    assert lib.consume_status() == 0


@pytest.mark.parametrize("M,K,N", [(27648, 9216, 16), (27648, 9216, 32), (49152, 4608, 64)])
def test_sums_are_as_exact_as_the_row_forms(lib, M, K, N):
    """The tensor core truncates its additions, so sums of positive products come out too small by a share that grows with
    the tiles added up in one accumulator.  The mean of that share over all outputs, against 64-bit products, must not be
    larger than the row form's; rounding to fp16 leaves the mean of 440 thousand and more outputs uncertain by
    2^-11 / sqrt(12 * 440000) = 2e-7, so 1e-6 is allowed."""
    from flash_llm_b200 import torch_op  # noqa: F401  (registers torch.ops.flashllm)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + N)
    A = torch.rand((M, K), generator=gen, device="cuda").half()
    A *= torch.rand((M, K), generator=gen, device="cuda") >= 0.8
    B = torch.rand((N, K), generator=gen, device="cuda").half()
    want = torch.cat([B.double() @ A[r:r + 1024].double().T for r in range(0, M, 1024)], dim=1)
    words, offs = torch.ops.flashllm.encode(A)
    share = {}
    try:
        for path in (lib.api.PATH_STREAM, lib.api.PATH_DIRECT):
            if path == lib.api.PATH_DIRECT:
                lib.set_plan(path=path)
            assert lib.get_plan(M, N, K, 1)["path"] == path
            share[path] = float(((want - torch.ops.flashllm.spmm(words, offs, B, M).double()) / want).mean())
    finally:
        lib.set_plan()
    assert lib.consume_status() == 0
    assert abs(share[lib.api.PATH_STREAM]) <= abs(share[lib.api.PATH_DIRECT]) + 1e-6, share


@pytest.mark.parametrize("bias,relu,residual", [(True, False, False), (True, True, False), (True, False, True), (False, True, True)])
def test_output_epilogues(lib, oracle, streaming, bias, relu, residual):
    """Whole rows leave through one epilogue and summed rows through another; C only two-byte aligned takes narrow stores."""
    M, K, N = 128 * 41, 64 * 13, 16
    A, B = random_problem(lib, M, K, N, 0.8, 17)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    rng = np.random.default_rng(18)
    b = (rng.standard_normal(M) * 2).astype(np.float16)
    r = (rng.standard_normal((N, M)) * 4).astype(np.float16)
    want = oracle.gemm_f32(A, B) + (b.astype(np.float32)[None, :] if bias else 0)
    want = (np.maximum(want, 0) if relu else want) + (r.astype(np.float32) if residual else 0)
    to_dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    comp_d, offs_d, B_d, b_d, r_d = to_dev(comp.view(np.int32)), to_dev(offs), to_dev(B), to_dev(b), to_dev(r)
    for shift in (0, 1):
        C = torch.full((N * M + 8,), float("nan"), dtype=torch.float16, device="cuda")[shift:shift + N * M]
        lib.spmm_splitk_epilogue(torch.cuda.current_stream().cuda_stream, comp_d.data_ptr(), offs_d.data_ptr(), B_d.data_ptr(),
                                 C.data_ptr(), M, N, K, None, 1, b_d.data_ptr() if bias else None,
                                 lib.ACT_RELU if relu else lib.ACT_NONE, r_d.data_ptr() if residual else None)
        torch.cuda.synchronize()
        assert lib.consume_status() == 0
        assert_close(C.view(N, M).cpu().numpy(), want, f"bias={bias} relu={relu} residual={residual} shift={shift}")


class _Forms:
    """One problem that is streamed, with the bits of its result in the streaming and in the row form (they differ, since the
    forms add up in another order)."""

    def __init__(self, lib, oracle, seed):
        self.lib = lib
        M, K, N = 128 * 100, 64 * 40, 16
        A, B = random_problem(lib, M, K, N, 0.8, seed)
        comp, offs, _ = lib.InitSparseMatrixA_API(A)
        self.want = oracle.gemm_f32(A, B)
        assert lib.get_plan(M, N, K, 1)["path"] == lib.api.PATH_STREAM, "this case is meant to be streamed"
        self.prob = DeviceProblem(lib, comp, offs, B, M, N, K, 1)
        lib.release_scratch()
        self.streamed = self.prob.run().copy()
        lib.set_plan(path=lib.api.PATH_DIRECT)
        self.by_rows = self.prob.run().copy()
        lib.set_plan()
        lib.release_scratch()
        assert not np.array_equal(self.streamed, self.by_rows)

    def enqueue(self, stream, C=None):
        p = self.prob
        self.lib.SpMM_SplitK_API(stream.cuda_stream, None, p.comp.data_ptr(), p.offs.data_ptr(), p.B.data_ptr(),
                                 (p.C if C is None else C).data_ptr(), p.M, p.N, p.K, None, 1)


def test_streams_without_a_scratch_of_their_own_run_another_form(lib, oracle):
    """At most eight streams hold scratch; calls on further streams, and after the scratch was given back, are still right."""
    f = _Forms(lib, oracle, 23)
    for i, s in enumerate([torch.cuda.current_stream()] + [torch.cuda.Stream() for _ in range(12)]):
        with torch.cuda.stream(s):
            got = f.prob.run()
        assert_close(got, f.want, "one of many streams")
        assert np.array_equal(got, f.streamed if i < 8 else f.by_rows), i
    lib.release_scratch()
    assert np.array_equal(f.prob.run(), f.streamed), "after the scratch was released"


def test_streams_that_come_and_go_give_their_scratch_back(lib, oracle):
    """More streams than places, each giving its scratch back at its end, right behind work that it has not waited for."""
    f = _Forms(lib, oracle, 24)
    outs = [torch.full_like(f.prob.C, float("nan")) for _ in range(20)]
    torch.cuda.synchronize()
    for C in outs:
        stream = torch.cuda.Stream()
        for _ in range(5):
            f.enqueue(stream, C)
        lib.release_stream_scratch(stream.cuda_stream)
        assert stream.query(), "waits for the stream's work"
    for C in outs:
        assert np.array_equal(C.cpu().numpy(), f.streamed)
    lib.release_stream_scratch(torch.cuda.Stream().cuda_stream)  # one that has none
    assert lib.consume_status() == 0


def test_a_captured_call_needs_no_scratch(lib, oracle):
    M, K, N = 128 * 100, 64 * 40, 16
    A, B = random_problem(lib, M, K, N, 0.8, 29)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    prob = DeviceProblem(lib, comp, offs, B, M, N, K, 1)
    prob.run()
    prob.C.fill_(float("nan"))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        lib.SpMM_SplitK_API(torch.cuda.current_stream().cuda_stream, None, prob.comp.data_ptr(), prob.offs.data_ptr(),
                            prob.B.data_ptr(), prob.C.data_ptr(), M, N, K, None, 1)
    graph.replay()
    torch.cuda.synchronize()
    assert lib.consume_status() == 0
    assert_close(prob.C.cpu().numpy(), oracle.gemm_f32(A, B), "replayed")


def test_malformed_offsets_are_reported_not_followed(lib, oracle, streaming):
    """The CTA that meets them gives up, its rows are not stored, the counters are left clean for the next call."""
    M, K, N = 128 * 37, 64 * 16, 16
    A, B = random_problem(lib, M, K, N, 0.8, 31)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    broken = offs.copy()
    broken[5] = broken[4] - 3
    got = DeviceProblem(lib, comp, broken, B, M, N, K, 1).run(check_status=False)
    assert lib.consume_status() & 2
    want = oracle.gemm_f32(A, B)
    assert np.isnan(got[:, :128]).all(), "the row whose tiles 4 and 5 were given up is not stored"
    assert_close(got[:, 128:], want[:, 128:], "the other rows")
    assert_close(DeviceProblem(lib, comp, offs, B, M, N, K, 1).run(), want, "call after a malformed one")


@pytest.mark.parametrize("M,K,split_k,cluster_k,workspace_k", [(25472, 11264, 2, 4, 1), (27648, 12288, 4, 2, 2),
                                                               (27648, 20480, 1, 5, 1)])
def test_sums_are_as_exact_as_in_the_cut_that_bounds_them(lib, M, K, split_k, cluster_k, workspace_k):
    """149 to 296 tile rows fill the GPU uncut, and a cut by cost alone would add up 88 to 160 tiles in each of a K range's two
    accumulators.  Streamed or not, no sum in the tensor core may be longer than in the cut by tiles (22, 24, 32 of them), so
    that the mean share a sum of positive products loses is no larger; 1e-6 for rounding and sums in fp32, as above."""
    from flash_llm_b200 import torch_op  # noqa: F401  (registers torch.ops.flashllm)
    N = 64
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + K)
    A = torch.rand((M, K), generator=gen, device="cuda").half()
    A *= torch.rand((M, K), generator=gen, device="cuda") >= 0.8
    B = torch.rand((N, K), generator=gen, device="cuda").half()
    want = torch.cat([B.double() @ A[r:r + 1024].double().T for r in range(0, M, 1024)], dim=1)
    words, offs = torch.ops.flashllm.encode(A)
    share = {}
    assert lib.get_plan(M, N, K, split_k)["path"] == lib.api.PATH_STREAM
    try:
        for name, plan in (("streamed", {}), ("rows", dict(path=2)), ("by tiles", dict(path=2, cluster_k=cluster_k, workspace_k=workspace_k))):
            lib.set_plan(**plan)
            share[name] = abs(float(((want - torch.ops.flashllm.spmm(words, offs, B, M, split_k).double()) / want).mean()))
    finally:
        lib.set_plan()
    assert lib.consume_status() == 0
    assert max(share["streamed"], share["rows"]) <= share["by tiles"] + 1e-6, share
