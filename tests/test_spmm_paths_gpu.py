"""Every form of the SpMM kernel against the CPU oracle, whichever of them the automatic plan prefers: the ring form
(bulk copies of the compressed stream into shared memory) and the register-streaming form (global loads of a whole tile
into the scatter warps' registers) in its three shapes: 8 stages with one CTA per SM, 4 stages with two CTAs per SM,
and 4 stages with two warps sharing every tile.  Calls go through the C ABI of libSpMM_API.so."""
import numpy as np
import pytest
import torch

from helpers import DeviceProblem, assert_close, random_problem

pytestmark = pytest.mark.gpu

FORMS = [dict(path=1), dict(path=2, scatter_warps=8), dict(path=2, scatter_warps=4),
         dict(path=2, scatter_warps=4, producers=2)]
FORM_IDS = ["ring", "direct8", "direct4", "direct4x2"]


def _check(lib, oracle, A, B, N, split_k, plan, note):
    M, K = A.shape
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    want = oracle.gemm_f32(A, B)
    lib.set_plan(**plan)
    try:
        got = DeviceProblem(lib, comp, offs, B, M, N, K, split_k).run()
        used = lib.get_plan(M, N, K, split_k)
    finally:
        lib.set_plan()
    assert used["path"] == plan["path"]
    assert_close(got, want, f"{note} plan={plan}")
    return got


@pytest.mark.parametrize("form", FORMS, ids=FORM_IDS)
@pytest.mark.parametrize("N", [8, 16, 32, 64, 128])
def test_every_n_tile(lib, oracle, form, N):
    A, B = random_problem(lib, 384, 1024, N, 0.8, 100 + N)
    _check(lib, oracle, A, B, N, 1, dict(cluster_k=1, **form), f"N={N}")


@pytest.mark.parametrize("form", FORMS, ids=FORM_IDS)
@pytest.mark.parametrize("sparsity", [0.0, 0.3, 0.6, 0.7, 0.75, 0.95, 0.999, 1.0])
def test_densities(lib, oracle, form, sparsity):
    """From fully dense tiles (2048 vectors, far beyond what the register-streaming form keeps in registers) through
    the densities around its register budget (512 and 768 vectors per tile) down to empty tiles."""
    A, B = random_problem(lib, 256, 1536, 16, sparsity, 7)
    _check(lib, oracle, A, B, 16, 1, dict(cluster_k=1, **form), f"s={sparsity}")


@pytest.mark.parametrize("form", FORMS, ids=FORM_IDS)
def test_dense_and_sparse_tiles_alternate_in_a_stage(lib, oracle, form):
    """Successive tiles of one stage switch between tiles above the register budget of the register-streaming form,
    tiles within it and empty tiles, in every order."""
    M, K, N = 256, 64 * 48, 16
    rng = np.random.default_rng(11)
    A = np.zeros((M, K), np.float16)
    density = rng.choice([0.0, 0.02, 0.2, 0.3, 0.45, 1.0], size=(M // 128, K // 64))
    for r in range(M // 128):
        for c in range(K // 64):
            tile = rng.uniform(-1, 1, (128, 64)).astype(np.float16)
            tile[tile == 0] = np.float16(0.5)
            tile[rng.random((128, 64)) >= density[r, c]] = 0
            A[r * 128:(r + 1) * 128, c * 64:(c + 1) * 64] = tile
    B = lib.synthetic.dense_uniform_matrix(N, K, 12).numpy()
    _check(lib, oracle, A, B, N, 1, dict(cluster_k=1, **form), "alternating densities")


@pytest.mark.parametrize("form", FORMS, ids=FORM_IDS)
@pytest.mark.parametrize("reduce", [1, 2], ids=["second-kernel", "last-cta"])
@pytest.mark.parametrize("cluster_k,workspace_k,split_k", [(2, 1, 1), (4, 1, 1), (1, 3, 6), (2, 2, 4), (8, 1, 1), (3, 1, 1),
                                                           (5, 2, 4), (6, 1, 1), (7, 1, 1), (1, 32, 64), (1, 2, 5)])
def test_k_splits(lib, oracle, form, reduce, cluster_k, workspace_k, split_k):
    """Every way of cutting K: parts summed inside clusters of any size up to 8, workspace parts summed by the last
    CTA of an output tile to finish or by the second kernel, and both at once."""
    if workspace_k == 1 and reduce == 1:
        pytest.skip("no workspace parts: the reduce mode does not matter")
    A, B = random_problem(lib, 256, 2048, 16, 0.8, 13)
    _check(lib, oracle, A, B, 16, split_k,
           dict(cluster_k=cluster_k, workspace_k=workspace_k, reduce=reduce, **form), "K split")


@pytest.mark.parametrize("form", FORMS[1:], ids=FORM_IDS[1:])
@pytest.mark.parametrize("cluster_k", [2, 3, 7, 8])
@pytest.mark.parametrize("N", [8, 32, 64, 128, 256])
def test_cluster_sums_of_every_width(lib, oracle, form, cluster_k, N):
    """The CTAs of a cluster send one another their rows of the partial tile: into shared memory set aside for that (up to 64
    columns, where two CTAs per SM leave the room) or over the operands; rows that the cluster size does not divide, columns
    beyond N, an epilogue, and the same bits every time."""
    M, K = 384, 64 * 19
    A, B = random_problem(lib, M, K, N, 0.8, 700 + N + cluster_k)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    bias = torch.rand(M, device="cuda").half()
    want = oracle.gemm_f32(A, B) + bias.float().cpu().numpy()
    lib.set_plan(cluster_k=cluster_k, **form)
    try:
        prob = DeviceProblem(lib, comp, offs, B, M, N, K, 1)
        stream = torch.cuda.current_stream().cuda_stream
        outs = []
        for _ in range(3):
            C = torch.full((N, M), float("nan"), dtype=torch.float16, device="cuda")
            lib.spmm_splitk_epilogue(stream, prob.comp.data_ptr(), prob.offs.data_ptr(), prob.B.data_ptr(), C.data_ptr(), M, N, K,
                                     None, 1, bias.data_ptr())
            outs.append(C)
        assert lib.get_plan(M, N, K, 1)["cluster_k"] == cluster_k
    finally:
        lib.set_plan()
    assert lib.consume_status() == 0
    assert_close(outs[0].cpu().numpy(), want, f"N={N} S={cluster_k} {form}")
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("rows,tiles,cluster_k,N", [
    (33, 8, 2, 32), (33, 9, 2, 32), (3, 10, 2, 32),     # 4 tiles a CTA and more: the receiving area goes, launch overlap off
    (33, 32, 2, 32), (33, 33, 2, 32), (10, 115, 7, 32),  # 16 and more: it goes with launch overlap on
    (100, 38, 2, 32), (100, 38, 2, 64), (40, 33, 7, 64), (12, 16, 4, 64), (13, 16, 4, 64), (8, 24, 6, 64), (72, 9, 2, 64),
    (8, 130, 8, 32), (9, 130, 8, 32),                    # 64 CTAs and more: off, only few of them have it at this length
    (75, 9, 2, 64), (16, 16, 8, 64),                     # 64 columns: CTAs with an SM to themselves, and pairs on every SM
])
def test_cluster_sums_by_length_and_crowding(lib, rows, tiles, cluster_k, N, overlap):
    """What a cluster's sum goes through (an area of its own, the operands' buffers, the parked tiles) depends on the K tiles of
    a CTA, on how many CTAs there are and on launch overlap.  Calls back to back, the same bits every time."""
    from flash_llm_b200 import torch_op  # noqa: F401  (registers torch.ops.flashllm)
    M, K = 128 * rows, 64 * tiles
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows * tiles + N)
    A = (torch.rand((M, K), generator=gen, device="cuda") * 2 - 1).half()
    A *= torch.rand((M, K), generator=gen, device="cuda") >= 0.8
    B = (torch.rand((N, K), generator=gen, device="cuda") * 2 - 1).half()
    bias = (torch.rand(M, generator=gen, device="cuda") - 0.5).half()
    residual = (torch.rand((N, M), generator=gen, device="cuda") - 0.5).half()
    want = (B.double() @ A.double().T + bias.double() + residual.double()).float().cpu().numpy()
    words, offs = torch.ops.flashllm.encode(A)
    torch.cuda.synchronize()
    lib.set_launch_overlap(overlap)
    lib.set_plan(path=lib.api.PATH_DIRECT, cluster_k=cluster_k)
    try:
        outs = [torch.ops.flashllm.spmm_epilogue(words, offs, B, M, 1, bias, 0, residual) for _ in range(6)]
        torch.cuda.synchronize()
    finally:
        lib.set_plan()
        lib.set_launch_overlap(False)
    assert lib.consume_status() == 0
    assert_close(outs[0].cpu().numpy(), want, f"{rows}x{tiles} S={cluster_k} N={N}")
    assert all(torch.equal(C, outs[0]) for C in outs[1:])


@pytest.mark.parametrize("N", [16, 64, 256])
def test_sum_by_last_cta_is_deterministic_and_leaves_its_counters_clean(lib, oracle, N):
    """The order in which the CTAs of an output tile finish changes from launch to launch; the sum must not.  Repeated
    launches on one stream reuse the same counters, which therefore have to be back at zero every time; a second
    stream gets counters of its own."""
    M, K, split_k = 1152, 4096, 16
    A, B = random_problem(lib, M, K, N, 0.8, 77 + N)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    want = oracle.gemm_f32(A, B)
    lib.set_plan(cluster_k=1, workspace_k=8, reduce=2)
    try:
        prob = DeviceProblem(lib, comp, offs, B, M, N, K, split_k)
        first = prob.run().copy()
        assert_close(first, want, f"N={N}")
        for _ in range(20):
            assert np.array_equal(prob.run(), first)
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            assert np.array_equal(prob.run(), first)
        second_kernel = None
        lib.set_plan(cluster_k=1, workspace_k=8, reduce=1)
        second_kernel = prob.run().copy()
    finally:
        lib.set_plan()
    assert np.array_equal(second_kernel, first)  # both add the parts in part order from the same fp32 partial sums


@pytest.mark.parametrize("form", FORMS, ids=FORM_IDS)
def test_fewer_tiles_than_scatter_warps(lib, oracle, form):
    for k_tiles in (1, 2, 3, 5, 9):
        A, B = random_problem(lib, 128, 64 * k_tiles, 16, 0.8, 20 + k_tiles)
        _check(lib, oracle, A, B, 16, 1, dict(cluster_k=1, **form), f"{k_tiles} K tiles")


@pytest.mark.parametrize("form", FORMS, ids=FORM_IDS)
def test_forms_agree(lib, oracle, form):
    """The forms differ in how words reach the stage and in how many accumulators the tiles are dealt to (the
    register-streaming form keeps one per MMA-issuing thread and adds them at the end), so results agree to fp32
    summation order."""
    M, K, N = 1024, 4096, 32
    A, B = random_problem(lib, M, K, N, 0.8, 31)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    prob = DeviceProblem(lib, comp, offs, B, M, N, K, 1)
    results = []
    for plan in (dict(path=1, cluster_k=2), dict(cluster_k=2, **form)):
        lib.set_plan(**plan)
        try:
            results.append(prob.run().copy())
        finally:
            lib.set_plan()
    assert_close(results[1], results[0].astype(np.float32), f"{form} against the ring form")


@pytest.mark.parametrize("form", FORMS, ids=FORM_IDS)
def test_malformed_offsets_are_reported_not_followed(lib, oracle, form):
    """A TileOffsets entry that runs backwards makes the kernel give up with status bit 2 instead of reading there."""
    M, K, N = 256, 1024, 16
    A, B = random_problem(lib, M, K, N, 0.8, 41)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    offs = offs.copy()
    offs[5] = offs[4] - 3
    lib.set_plan(cluster_k=1, **form)
    try:
        DeviceProblem(lib, comp, offs, B, M, N, K, 1).run(check_status=False)
        # A caller of the reference interface never reads the status word: the next call, made without clearing it,
        # must compute as if nothing had happened (a give-up belongs to the launch it happened in).
        comp, offs, _ = lib.InitSparseMatrixA_API(A)
        got = DeviceProblem(lib, comp, offs, B, M, N, K, 1).run(check_status=False)
        status = lib.consume_status()
    finally:
        lib.set_plan()
    assert status & 2
    assert_close(got, oracle.gemm_f32(A, B), "call after a malformed one")
    assert lib.consume_status() == 0


@pytest.mark.parametrize("form,N", [(f, N) for f in FORMS for N in (16, 64, 128)] + [(dict(path=4, producers=2), 256)],
                         ids=[f"{i}-{N}" for i in FORM_IDS for N in (16, 64, 128)] + ["wide-256"])
def test_a_cta_that_gives_up_does_not_leave_its_cluster_with_wrong_sums(lib, oracle, form, N):
    """Of a tile row's three CTAs the first finds its offsets malformed: the row's outputs are not stored or not a number,
    never what happened to lie in tensor memory; the other row is as ever."""
    M, K = 256, 1024
    A, B = random_problem(lib, M, K, N, 0.8, 43)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    want = oracle.gemm_f32(A, B)
    bad = offs.copy()
    bad[3] = bad[2] - 3
    lib.set_plan(cluster_k=3, **form)
    try:
        for _ in range(2):  # the second time tensor memory holds the sums of a good call
            got = DeviceProblem(lib, comp, bad, B, M, N, K, 1).run(check_status=False)
            assert lib.consume_status() & 2
            assert np.isnan(got[:, :128]).all()
            assert_close(got[:, 128:], want[:, 128:], "the other row")
            assert_close(DeviceProblem(lib, comp, offs, B, M, N, K, 1).run(), want, "call after a malformed one")
    finally:
        lib.set_plan()


@pytest.mark.parametrize("form", FORMS, ids=FORM_IDS)
@pytest.mark.parametrize("N", [256, 384])
def test_n_beyond_one_mma_tile(lib, oracle, form, N):
    """N a multiple of 128 (the reference's large-N dispatch, csrc/SpMM_API.cu:97-112): several N tiles per tile row."""
    A, B = random_problem(lib, 256, 1024, N, 0.8, 500 + N)
    _check(lib, oracle, A, B, N, 4, dict(**form), f"N={N}")


def test_more_streams_than_counter_sets_fall_back_to_the_second_kernel(lib, oracle):
    """The in-kernel split-K sum binds a set of arrival counters to each stream it is used on (32 sets per device);
    calls on further streams must still be right (they are summed by the second kernel)."""
    M, K, N, split_k = 512, 2048, 16, 8
    A, B = random_problem(lib, M, K, N, 0.8, 91)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    want = oracle.gemm_f32(A, B)
    prob = DeviceProblem(lib, comp, offs, B, M, N, K, split_k)
    lib.set_plan(cluster_k=1, workspace_k=4, reduce=2)
    try:
        first = prob.run().copy()
        assert_close(first, want, "default stream")
        streams = [torch.cuda.Stream() for _ in range(40)]
        for s_ in streams:
            with torch.cuda.stream(s_):
                assert np.array_equal(prob.run(), first)
    finally:
        lib.set_plan()


@pytest.mark.parametrize("plan", [dict(cluster_k=1), dict(cluster_k=2), dict(cluster_k=1, workspace_k=4),
                                  dict(cluster_k=1, workspace_k=4, reduce=2)], ids=["plain", "cluster", "parts", "parts-last-cta"])
@pytest.mark.parametrize("offset_halves", [1, 2, 3])
def test_output_that_is_only_two_byte_aligned(lib, oracle, plan, offset_halves):
    """The reference interface asks nothing of C's alignment beyond that of a half; the wide stores of the cluster sum
    and of the sums over workspace parts must give way to narrow ones (or to an uncut launch) for such a C."""
    M, K, N, split_k = 256, 2048, 16, 8
    A, B = random_problem(lib, M, K, N, 0.8, 97)
    comp, offs, _ = lib.InitSparseMatrixA_API(A)
    want = oracle.gemm_f32(A, B)
    dev = torch.device("cuda:0")
    comp_d = torch.from_numpy(np.ascontiguousarray(comp.view(np.int32))).to(dev)
    offs_d, B_d = torch.from_numpy(offs).to(dev), torch.from_numpy(B).to(dev)
    backing = torch.full((N * M + 8,), float("nan"), dtype=torch.float16, device=dev)
    C = backing[offset_halves:offset_halves + N * M]
    ws = torch.empty((split_k, N, M), dtype=torch.float16, device=dev)
    lib.set_plan(**plan)
    try:
        lib.SpMM_SplitK_API(torch.cuda.current_stream().cuda_stream, None, comp_d.data_ptr(), offs_d.data_ptr(),
                            B_d.data_ptr(), C.data_ptr(), M, N, K, ws.data_ptr(), split_k)
        torch.cuda.synchronize()
    finally:
        lib.set_plan()
    assert lib.consume_status() == 0
    assert_close(C.view(N, M).cpu().numpy(), want, f"C at +{2 * offset_halves} bytes, plan {plan}")
    assert torch.isnan(backing[:offset_halves]).all() and torch.isnan(backing[offset_halves + N * M:]).all()


@pytest.mark.parametrize("M,K,N,split_k,cluster_k", [(2048, 32768, 16, 4, 8), (9216, 18432, 32, 6, 2)])
def test_workspace_parts_that_do_not_fit(lib, M, K, N, split_k, cluster_k):
    """A call whose C is not aligned for workspace parts is planned without them: right, and its sums no longer in the tensor
    core than in the cluster parts of the plan with them (`cluster_k`, 7e-8 to 1.4e-7 of a sum per tile).  The mean over the
    outputs, rounding to fp16 included, is uncertain by 2^-11 / sqrt(12 * 32768) = 8e-7 at most; 2e-6 is allowed."""
    from flash_llm_b200 import torch_op  # noqa: F401  (registers torch.ops.flashllm)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + K)
    A = torch.rand((M, K), generator=gen, device="cuda").half()
    A *= torch.rand((M, K), generator=gen, device="cuda") >= 0.8
    B = torch.rand((N, K), generator=gen, device="cuda").half()
    want = torch.cat([B.double() @ A[r:r + 1024].double().T for r in range(0, M, 1024)], dim=1)
    words, offs = torch.ops.flashllm.encode(A)
    ws = torch.empty((split_k, N, M), dtype=torch.float16, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    share = {}
    try:
        for name, shift, plan in (("moved", 1, {}), ("cut", 0, dict(cluster_k=cluster_k, workspace_k=1))):
            C = torch.full((N * M + 8,), float("nan"), dtype=torch.float16, device="cuda")[shift:shift + N * M]
            lib.set_plan(path=lib.api.PATH_DIRECT, **plan)
            lib.SpMM_SplitK_API(stream, None, words.data_ptr(), offs.data_ptr(), B.data_ptr(), C.data_ptr(), M, N, K, ws.data_ptr(),
                                split_k)
            torch.cuda.synchronize()
            assert lib.consume_status() == 0
            assert_close(C.view(N, M).cpu().numpy(), want.float().cpu().numpy(), name)
            share[name] = abs(float(((want - C.view(N, M).double()) / want).mean()))
    finally:
        lib.set_plan()
    assert share["moved"] <= share["cut"] + 2e-6, share
