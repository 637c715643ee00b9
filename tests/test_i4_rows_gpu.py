"""int4 groups of 128 x int8 activations for up to 32 rows (``csrc/gemm_i4_rows.cu``), against the same quantised operands in fp64."""
import pytest
import torch

from fastllm_b200.ops import _lib
from fastllm_b200.ops import basic as B
from fastllm_b200.ops import quant_gemm as QG
from fastllm_b200.ops.quant import LinearWeight

pytestmark = pytest.mark.gpu


# row counts around the tiles of eight tokens; N below, at and past a 16-row tile, two, three and four CTAs an SM; k blocks fewer, as many and more than warps
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(8, 128), (136, 640), (128, 1152), (4096, 2048), (6144, 1024), (7680, 256), (256, 14336)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rows(M, N, K, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    lw = LinearWeight.from_dense(rnd(N, K) * K ** -0.5, "int4g128", act_dtype=dtype, interleaved=True)
    bias, res = rnd(N).to(dtype), rnd(M, N).to(dtype)
    xq, sa, xs, ld_a = QG.quant_act_i8(rnd(M, K).to(dtype))
    w, pairs, _, _ = QG._a8_tensors(lw)
    act = (xq.double().view(M, K // 128, 128) * sa[:, :M].t().double()[:, :, None]).reshape(M, K)
    q = torch.stack([(lw.w >> 4) & 0xF, lw.w & 0xF], dim=2).reshape(N, K // 128, 128).double()
    w64 = (q * lw.scale.double()[:, :, None] + lw.zero.double()[:, :, None]).reshape(N, K)
    y, size = act @ w64.t(), act.abs() @ w64.abs().t()

    def run(out, flags, b=None, r=None):
        rc = _lib.kernels().fb_gemm_i4_rows(B._ptr(xq), K, B._ptr(sa), B._ptr(xs), ld_a, B._ptr(w), B._ptr(pairs), B._ptr(out), B._ptr(b), B._ptr(r), M, N, K,
                                            out.stride(0), r.stride(0) if r is not None else 0, B.dtype_code(dtype), flags, B._stream())
        if rc == -1:
            assert M > 16 and (N + 15) // 16 > 2 * torch.cuda.get_device_properties(0).multi_processor_count
            pytest.skip("the tcgen05 route is faster")
        assert rc == 0
        return out.double()

    # the sums of a k block are exact; s * sum and min * xs cancel, each at most 15 / 8 of what it sums up; four fp32 roundings a block and one a sum
    err = (K // 128 + 16) * 2.0 ** -22 * size + 2.0 ** -30
    got = run(torch.full((M, N), float("nan"), device="cuda"), B.GEMM_OUT_F32)
    assert bool(((got - y).abs() <= err).all())
    half = torch.finfo(dtype).eps / 2
    want = y + bias.double() + res.double()
    got = run(torch.empty(M, N, device="cuda", dtype=dtype), B.GEMM_BIAS | B.GEMM_RESIDUAL, bias, res)
    assert bool(((got - want).abs() <= err + want.abs() * (half + 2.0 ** -20) + 2.0 ** -20).all())
    if N % 128 == 0:
        t, e = y.view(M, N // 128, 2, 64), err.view(M, N // 128, 2, 64)
        want = (torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(M, N // 2)
        e = (1.1 * e[:, :, 0] * t[:, :, 1].abs() + torch.nn.functional.silu(t[:, :, 0]).abs() * e[:, :, 1]).reshape(M, N // 2)
        got = run(torch.empty(M, N // 2, device="cuda", dtype=dtype), B.GEMM_SWIGLU)
        assert bool(((got - want).abs() <= e + want.abs() * (half + 2.0 ** -18) + 2.0 ** -20).all())
    _lib.check_device_errors()
