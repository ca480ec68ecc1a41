"""Kernels are launched before their predecessors on the stream have ended.  Calls enqueued back to back, without the host
waiting in between, must see what the work before them produces and must not disturb what it still reads, in the forms of the
kernel that share scratch between launches or own all of tensor memory: with launch overlap off (weights may be produced by
the stream's earlier work) and on (resident weights; B and C are produced and consumed along the chain)."""
import numpy as np
import pytest
import torch

from flash_llm_b200 import torch_op  # noqa: F401  (registers torch.ops.flashllm)
from helpers import assert_close

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["stream-16", "stream-64", "wide-256", "wide-512"])
def form(request, lib):
    """N of a form that every call is pinned to, whatever its sizes."""
    kind, N = request.param.split("-")
    lib.release_scratch()  # a place for every stream below, whatever streams earlier tests have used
    if kind == "stream":
        lib.set_plan(path=lib.api.PATH_STREAM)
    else:
        lib.set_plan(path=lib.api.PATH_WIDE, producers=int(N) // 128)
    yield int(N)
    lib.set_plan()
    lib.set_launch_overlap(False)


class _Weights:
    """A sparse matrix on the device, dense and encoded, with `exact(B)` by 64-bit arithmetic."""

    def __init__(self, M, K, sparsity, seed):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        A = torch.rand((M, K), generator=gen, device="cuda") * 2 - 1
        self.A = (A * (torch.rand((M, K), generator=gen, device="cuda") >= sparsity)).half()
        self.M, self.K = M, K
        self.words, self.offs = torch.ops.flashllm.encode(self.A)
        torch.cuda.synchronize()

    def exact(self, B):
        return (B.double() @ self.A.double().T).float().cpu().numpy()


def _call(lib, stream, words, offs, B, C, w):
    lib.SpMM_SplitK_API(stream.cuda_stream, None, words.data_ptr(), offs.data_ptr(), B.data_ptr(), C.data_ptr(), w.M, B.shape[0],
                        w.K, None, 1)


def _activations(N, K, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return (torch.rand((N, K), generator=gen, device="cuda") * 2 - 1).half()


def test_weights_written_earlier_in_the_stream_are_seen(lib, form):
    """The copies sit behind a long kernel, and the buffers hold another matrix until they run.  37 rows of 45 tiles: rows cut
    into parts at other places for either matrix would show as soon as one call's parts met another's."""
    N, M, K = form, 128 * 37, 64 * 45
    ws = [_Weights(M, K, s, seed) for seed, s in ((1, 0.8), (2, 0.6))]
    B = _activations(N, K, 3)
    words = torch.zeros(max(w.words.numel() for w in ws), dtype=torch.int32, device="cuda")
    offs = torch.zeros_like(ws[0].offs)
    outs = [torch.full((N, M), float("nan"), dtype=torch.float16, device="cuda") for _ in range(8)]
    slow = torch.zeros(1 << 26, dtype=torch.float32, device="cuda")
    stream = torch.cuda.current_stream()
    torch.cuda.synchronize()
    for i, C in enumerate(outs):
        w = ws[i % 2]
        slow.add_(1.0)
        words[:w.words.numel()].copy_(w.words)
        offs.copy_(w.offs)
        _call(lib, stream, words, offs, B, C, w)
    torch.cuda.synchronize()
    assert lib.consume_status() == 0
    for i, C in enumerate(outs):
        assert_close(C.cpu().numpy(), ws[i % 2].exact(B), f"call {i}")


@pytest.mark.parametrize("overlap", [False, True])
def test_calls_back_to_back_share_a_stream(lib, form, overlap):
    """Calls of different shapes, whose rows are cut at different places, follow one another on one stream and its scratch;
    every second one multiplies what the one before it has just computed, and C is overwritten while it may still be read."""
    N = form
    first, second, other = _Weights(128 * 41, 64 * 30, 0.8, 4), _Weights(128 * 10, 128 * 41, 0.9, 5), _Weights(128 * 75, 64 * 13, 0.6, 6)
    second.A.mul_(0.05)
    second.words, second.offs = torch.ops.flashllm.encode(second.A)
    X = [_activations(N, first.K, 10 + i) for i in range(3)]
    Y = _activations(N, other.K, 20)
    H = torch.empty((N, first.M), dtype=torch.float16, device="cuda")
    outs = [(torch.full((N, second.M), float("nan"), dtype=torch.float16, device="cuda"),
             torch.full((N, other.M), float("nan"), dtype=torch.float16, device="cuda")) for _ in range(12)]
    stream = torch.cuda.current_stream()
    torch.cuda.synchronize()
    lib.set_launch_overlap(overlap)
    for i, (C, D) in enumerate(outs):
        _call(lib, stream, first.words, first.offs, X[i % 3], H, first)
        _call(lib, stream, second.words, second.offs, H, C, second)
        _call(lib, stream, other.words, other.offs, Y, D, other)
    torch.cuda.synchronize()
    assert lib.consume_status() == 0
    want_d = other.exact(Y)
    want_c = [second.exact(torch.from_numpy(first.exact(x)).cuda().half()) for x in X]
    for i, (C, D) in enumerate(outs):
        assert_close(C.cpu().numpy(), want_c[i % 3], f"chained call {i}")
        assert_close(D.cpu().numpy(), want_d, f"unrelated call {i}")
        assert np.array_equal(D.cpu().numpy(), outs[0][1].cpu().numpy())


@pytest.mark.parametrize("overlap", [False, True])
def test_two_streams_at_once(lib, form, overlap):
    """Two streams run the form at the same time, each with its own scratch."""
    N = form
    ws = [_Weights(128 * 41, 64 * 30, 0.8, 7), _Weights(128 * 37, 64 * 45, 0.7, 8)]
    Bs = [_activations(N, w.K, 30 + i) for i, w in enumerate(ws)]
    outs = [[torch.full((N, w.M), float("nan"), dtype=torch.float16, device="cuda") for _ in range(20)] for w in ws]
    streams = [torch.cuda.Stream() for _ in ws]
    torch.cuda.synchronize()
    lib.set_launch_overlap(overlap)
    for i in range(20):
        for w, B, C, s in zip(ws, Bs, outs, streams):
            _call(lib, s, w.words, w.offs, B, C[i], w)
    torch.cuda.synchronize()
    assert lib.consume_status() == 0
    for w, B, C in zip(ws, Bs, outs):
        want = w.exact(B)
        for i, c in enumerate(C):
            assert_close(c.cpu().numpy(), want, f"call {i}")
            assert torch.equal(c, C[0])


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("N", [16, 512])
def test_encoding_into_buffers_an_spmm_has_just_read(lib, N, overlap):
    """Encode, multiply, encode another matrix into the same buffers, multiply, ... at a size that the streaming and the wide
    form take by themselves."""
    M, K = 128 * 216, 64 * 36
    gen = torch.Generator(device="cuda")
    gen.manual_seed(9)
    As = [((torch.rand((M, K), generator=gen, device="cuda") * 2 - 1)
           * (torch.rand((M, K), generator=gen, device="cuda") >= s)).half() for s in (0.8, 0.6)]
    B = _activations(N, K, 40)
    assert lib.get_plan(M, N, K, 1)["path"] == (lib.api.PATH_STREAM if N == 16 else lib.api.PATH_WIDE)
    words = torch.zeros(M * K // 2, dtype=torch.int32, device="cuda")
    offs = torch.zeros((M // 128) * (K // 64) + 2, dtype=torch.int32, device="cuda")
    outs = [torch.full((N, M), float("nan"), dtype=torch.float16, device="cuda") for _ in range(8)]
    L, stream = lib.library(), torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    lib.set_launch_overlap(overlap)
    try:
        for i, C in enumerate(outs):
            A = As[i % 2]
            assert L.FlashLLM_EncodeOnDevice_TileOffsets(stream, A.data_ptr(), M, K, offs.data_ptr()) == 0
            assert L.FlashLLM_EncodeOnDevice_Pack(stream, A.data_ptr(), M, K, offs.data_ptr(), words.data_ptr(), 1) == 0
            lib.SpMM_SplitK_API(stream, None, words.data_ptr(), offs.data_ptr(), B.data_ptr(), C.data_ptr(), M, N, K, None, 1)
        torch.cuda.synchronize()
    finally:
        lib.set_launch_overlap(False)
    assert lib.consume_status() == 0
    for i, C in enumerate(outs):
        want = (B.double() @ As[i % 2].double().T).float().cpu().numpy()
        assert_close(C.cpu().numpy(), want, f"call {i}")


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("operand", ["bias", "residual"])
@pytest.mark.parametrize("N", [16, 64])
@pytest.mark.parametrize("plan", [dict(path=3), dict(path=2, cluster_k=1), dict(path=2, cluster_k=3)],
                         ids=["stream", "rows", "clusters"])
def test_bias_and_residual_written_by_the_call_before(lib, plan, N, operand, overlap):
    """The call before runs on few SMs and for long, so that the next one's CTAs are there while it still computes what they
    are to add; the operand holds another call's values until then."""
    first, second = _Weights(128 * 16, 64 * 256, 0.8, 50), _Weights(128 * 16, 64 * 45, 0.8, 51)
    X = [_activations(N, first.K, 60 + i) for i in range(3)]
    Y = _activations(N, second.K, 70)
    H = torch.full((N, first.M), float("nan"), dtype=torch.float16, device="cuda")
    outs = [torch.full((N, second.M), float("nan"), dtype=torch.float16, device="cuda") for _ in range(12)]
    bias, residual = (H.data_ptr(), None) if operand == "bias" else (None, H.data_ptr())
    stream = torch.cuda.current_stream()
    lib.release_scratch()
    torch.cuda.synchronize()
    lib.set_launch_overlap(overlap)
    try:
        for i, C in enumerate(outs):
            lib.set_plan(path=lib.api.PATH_DIRECT, cluster_k=1)
            _call(lib, stream, first.words, first.offs, X[i % 3], H, first)
            lib.set_plan(**plan)
            lib.spmm_splitk_epilogue(stream.cuda_stream, second.words.data_ptr(), second.offs.data_ptr(), Y.data_ptr(), C.data_ptr(),
                                     second.M, N, second.K, None, 1, bias, lib.ACT_NONE, residual)
        torch.cuda.synchronize()
    finally:
        lib.set_plan()
        lib.set_launch_overlap(False)
    assert lib.consume_status() == 0
    product = second.exact(Y)
    added = []  # what the call before computes when it runs alone: a value it rounds the other way may be an ulp of 2^-5
    lib.set_plan(path=lib.api.PATH_DIRECT, cluster_k=1)
    try:
        for x in X:
            _call(lib, stream, first.words, first.offs, x, H, first)
            assert_close(H.cpu().numpy(), first.exact(x), "the call before")
            added.append(H.float().cpu().numpy())
    finally:
        lib.set_plan()
    for i, C in enumerate(outs):
        assert_close(C.cpu().numpy(), product + (added[i % 3][:1] if operand == "bias" else added[i % 3]), f"call {i}")
