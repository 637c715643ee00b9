"""16-bit products of large batches on CTA pairs: tile edges, epilogues and block-diagonal weights against 64 bits."""
import pytest
import torch

from fastllm_b200.ops import _lib, basic as B

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _tol(ref, err, dtype):
    # one rounding, fp16 below its smallest normal value included
    return err + ref.abs() * (torch.finfo(dtype).eps / 2 + 2.0 ** -20) + 2.0 ** -24


# one row past a tile, a last tile of one token half, ragged k and n, several rounds of pairs
@pytest.mark.parametrize("M,N,K", [(513, 5120, 200), (600, 4096, 64), (640, 2080, 72), (1000, 544, 2048), (1025, 4352, 136), (4001, 3072, 512)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("form", ["plain", "bias+residual", "f32", "gelu", "swiglu"])
def test_products(M, N, K, dtype, form):
    if form == "swiglu" and N % 128:
        pytest.skip("gate and up rows come in tiles of 128")
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x, w = torch.randn(M, K, device=DEV, generator=g).to(dtype), (torch.randn(N, K, device=DEV, generator=g) * 0.1).to(dtype)
    y = x.double() @ w.double().t()
    # products are exact, each of the K steps of the sum may cut off one unit of fp32 of the largest partial sum
    err = K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())
    if form == "bias+residual":
        b, r = torch.randn(N, device=DEV, generator=g).to(dtype), torch.randn(M, N, device=DEV, generator=g).to(dtype)
        got, ref = B.linear(x, w, bias=b, residual=r), y + b.double() + r.double()
        err = err + 2.0 ** -22 * (y.abs() + b.double().abs() + r.double().abs())
    elif form == "f32":
        got, ref = B.linear(x, w, out_f32=True), y
        assert got.dtype == torch.float32
        assert bool(((got.double() - ref).abs() <= err + 2.0 ** -24).all())
        return
    elif form == "gelu":
        got, ref = B.linear_act(x, w, act="gelu"), torch.nn.functional.gelu(y)
        err = 1.13 * err + 2.0 ** -20                                   # |gelu'| < 1.13
    elif form == "swiglu":
        got = B.linear(x, B.interleave_gate_up(w[:N // 2], w[N // 2:]), swiglu=True)
        a, b = y[:, :N // 2], y[:, N // 2:]
        ref = torch.nn.functional.silu(a) * b
        err = 1.1 * err[:, :N // 2] * b.abs() + torch.nn.functional.silu(a).abs() * err[:, N // 2:] + 2.0 ** -20 * (1 + ref.abs())
    else:
        got, ref = B.linear(x, w), y
    _lib.check_device_errors()
    assert got.dtype == dtype and bool(((got.double() - ref).abs() <= _tol(ref, err, dtype)).all())


@pytest.mark.parametrize("M,N,K,blocks", [(600, 256, 128, 16), (4001, 512, 192, 4)])
def test_block_diagonal(M, N, K, blocks):
    g = torch.Generator(device=DEV).manual_seed(M)
    x, w = torch.randn(M, blocks * K, device=DEV, generator=g).bfloat16(), torch.randn(blocks * N, K, device=DEV, generator=g).bfloat16()
    out = torch.empty(M, blocks * N, device=DEV)
    rc = _lib.kernels().fb_gemm_16bit_blocks(x.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, blocks, x.stride(0), out.stride(0), 1,
                                             torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    xd, wd = x.double().view(M, blocks, K), w.double().view(blocks, N, K)
    ref, size = torch.einsum("mbk,bnk->mbn", xd, wd), torch.einsum("mbk,bnk->mbn", xd.abs(), wd.abs())
    assert bool(((out.double().view(M, blocks, N) - ref).abs() <= K * 2.0 ** -23 * size).all())


@pytest.mark.parametrize("M,N,K", [(1025, 4352, 136), (4001, 3072, 512), (1000, 4096, 14336)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("form", ["plain", "bias+residual", "f32", "swiglu"])
def test_pairs_give_the_bits_of_one_cta(M, N, K, dtype, form):
    """Every output is the same sum in the same order whichever kernel makes it: portions of rows that stay with one CTA a tile against the whole."""
    g = torch.Generator(device=DEV).manual_seed(K)
    x, w = torch.randn(M, K, device=DEV, generator=g).to(dtype), (torch.randn(N, K, device=DEV, generator=g) * 0.1).to(dtype)
    b, r = torch.randn(N, device=DEV, generator=g).to(dtype), torch.randn(M, N, device=DEV, generator=g).to(dtype)
    call = {"plain": lambda s: B.linear(x[s], w), "bias+residual": lambda s: B.linear(x[s], w, bias=b, residual=r[s]), "f32": lambda s: B.linear(x[s], w, out_f32=True),
            "swiglu": lambda s: B.linear(x[s], w, swiglu=True)}[form]
    got = call(slice(None))
    for lo in range(0, M - 257, 333):                          # 333 rows: three row tiles of one CTA, never pairs at these widths
        s = slice(lo, min(lo + 333, M))
        if s.stop - s.start > 256:
            assert torch.equal(call(s), got[s])
