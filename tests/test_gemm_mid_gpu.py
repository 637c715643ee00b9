"""Products of a few hundred rows on CTA pairs with the last round of tiles split over k (``csrc/gemm_mid.cuh``): sizes around its tiles, against fp64."""
import pytest
import torch

from fastllm_b200.ops import _lib
from fastllm_b200.ops import basic as B

gpu = pytest.mark.gpu


def _run(x, w, tiles, out, res=None, bias=None, flags=0):
    (M, K), N = x.shape, w.shape[0]
    lib = _lib.kernels()
    need = lib.fb_gemm_mid_workspace(M, N, K, tiles, 0)
    if need < 0:
        return None
    # what the workspace holds before must not matter
    ws = torch.full((max(need, 16),), 0xFF, device=x.device, dtype=torch.uint8)
    rc = lib.fb_gemm_16bit_mid(B._ptr(x), B._ptr(w), B._ptr(out), B._ptr(bias), B._ptr(res), M, N, K, x.stride(0), w.stride(0), out.stride(0),
                               res.stride(0) if res is not None else 0, B.dtype_code(x.dtype), flags, tiles, B._ptr(ws), need, B._stream())
    assert rc == 0
    return out


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tiles", [1, 2, 4])
# k of one block, with a remainder, in one to eight splits; features below, at and past a 256-row tile and past one round of tiles (75 on 74 pairs)
@pytest.mark.parametrize("N,K", [(256, 64), (136, 520), (576, 2048), (4096, 1024), (19200, 512), (1024, 14336)])
@pytest.mark.parametrize("M", [1, 33, 256, 257, 352, 512, 777])
def test_edges(M, N, K, tiles, dtype):
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N + K)
    x = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    res = torch.randn(M, N, device="cuda", generator=g).to(dtype)
    bias = torch.randn(N, device="cuda", generator=g).to(dtype)
    ref = x.double() @ w.double().t()
    y = _run(x, w, tiles, torch.full((M, N), float("nan"), device="cuda"), flags=B.GEMM_OUT_F32)
    if y is None:
        assert (M + tiles - 1) // tiles > 512
        return
    # 16-bit products are exact in fp32: only the sums round, 2^-24 of a partial sum each, sqrt(K) of them for random terms
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -24 * K ** 0.5 + 1e-5
    half = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11          # half a step of the result's type
    y = _run(x, w, tiles, torch.empty(M, N, device="cuda", dtype=dtype), res, bias, B.GEMM_BIAS | B.GEMM_RESIDUAL)
    want = ref + bias.double() + res.double()
    assert ((y.double() - want).norm() / want.norm()).item() < half
    if N % 128 == 0:
        y = _run(x, w, tiles, torch.empty(M, N // 2, device="cuda", dtype=dtype), flags=B.GEMM_SWIGLU)
        t = ref.view(M, N // 128, 2, 64)
        want = (torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(M, N // 2)
        assert ((y.double() - want).norm() / want.norm()).item() < half
    _lib.check_device_errors()


@gpu
def test_graph_replays_leave_no_flags():
    """A captured launch has the same tag in every replay: each must wait for its own partial tiles."""
    N, K, M = 4096, 14336, 200
    assert _lib.kernels().fb_gemm_mid_pick(M, N, K, 148) > 0
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()
    x = torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    B.linear(x, w)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ys = [B.linear(x, w) for _ in range(3)]
    for seed in range(4):
        x.copy_(torch.randn(M, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)))
        graph.replay()
        ref = x.double() @ w.double().t()
        for y in ys:
            assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -8
    _lib.check_device_errors()


@gpu
@pytest.mark.parametrize("M,N,K", [(300, 18944, 1024), (1250, 4096, 2056)])
def test_whole_tiles_give_the_bits_of_the_other_kernels(M, N, K):
    """More than 256 rows: the sums and their order do not depend on the kernel, so portions of a prompt give what the whole gives."""
    assert _lib.kernels().fb_gemm_mid_pick(M, N, K, 148) > 0 and _lib.kernels().fb_gemm_mid_pick(4 * M, N, K, 148) == 0
    g = torch.Generator(device="cuda").manual_seed(N)
    x, w = torch.randn(4 * M, K, device="cuda", generator=g).bfloat16(), torch.randn(N, K, device="cuda", generator=g).bfloat16()
    assert torch.equal(B.linear(x[:M], w, swiglu=True), B.linear(x, w, swiglu=True)[:M])
    assert torch.equal(B.linear(x[:M], w, out_f32=True), B.linear(x, w, out_f32=True)[:M])


def test_refusals():
    lib = _lib.kernels()
    for M, N, K, tiles in ((513, 256, 64, 1), (100, 256, 63, 1), (100, 252, 64, 1), (100, 256, 64, 0)):
        assert lib.fb_gemm_mid_workspace(M, N, K, tiles, 148) == -1
    assert lib.fb_gemm_mid_pick(64, 4096, 14336, 148) == 0 and lib.fb_gemm_mid_pick(2049, 4096, 14336, 148) == 0
