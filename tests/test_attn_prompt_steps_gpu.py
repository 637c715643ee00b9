"""Prompt attention around the edges of its pipelines: few and many steps of keys, ragged rows, maxima that grow by less and by more than what lets an
accumulator stand (2^8), by leaps and not at all."""
import pytest
import torch

from fastllm_b200.ops import _lib, attention as A
from fastllm_b200.ops import grouped as G          # noqa: F401  (signatures)

pytestmark = pytest.mark.gpu
DEV, PAGE = "cuda", 128

# (keys, new tokens) of the requests: one to six steps of 64 and 128 keys, even and odd, a last step of one key, one new row behind a history, full blocks
LENS = [[(1, 1), (64, 64), (65, 1), (127, 127)], [(128, 128), (129, 129), (193, 2), (256, 256)], [(257, 130), (385, 385), (500, 255), (640, 257), (700, 1)]]


def _problem(lens, H, Hkv, D, V, growth, dtype):
    """Scores of a row climb by ``growth`` powers of two every 64 keys (with noise of about one); in 64 bits: outputs, and a bound of their error."""
    g = torch.Generator().manual_seed(len(lens) * 1000 + D + V + int(10 * growth) + 500)
    n_pages = sum((k + PAGE - 1) // PAGE for k, _ in lens) + 1
    perm = torch.randperm(n_pages, generator=g).int()
    table = torch.zeros(len(lens), max((k + PAGE - 1) // PAGE for k, _ in lens), dtype=torch.int32)
    kp, vp = torch.full((n_pages, PAGE, Hkv, D), 30.0, dtype=dtype), torch.full((n_pages, PAGE, Hkv, V), -30.0, dtype=dtype)       # stale rows are finite
    cu, at = [0], 0
    scale = D ** -0.5
    for b, (k, n) in enumerate(lens):
        pages = (k + PAGE - 1) // PAGE
        table[b, :pages] = perm[at:at + pages]
        at += pages
        keys = torch.randn(k, Hkv, D, generator=g)
        keys[:, :, 0] = growth / 1.4426950408889634 / scale / 4 * (torch.arange(k)[:, None] / 64)          # times a query component of 4
        rows = [(table[b, i // PAGE].item(), i % PAGE) for i in range(k)]
        idx = torch.tensor(rows)
        kp[idx[:, 0], idx[:, 1]] = keys.to(dtype)
        vp[idx[:, 0], idx[:, 1]] = torch.randn(k, Hkv, V, generator=g).to(dtype)
        cu.append(cu[-1] + n)
    q = torch.randn(cu[-1], H, D, generator=g)
    q[:, :, 0] = 4.0
    q = q.to(dtype)
    want, tol = torch.zeros(cu[-1], H, V, dtype=torch.float64), torch.zeros(cu[-1], H, V, dtype=torch.float64)
    u = torch.finfo(dtype).eps / 2
    for b, (k, n) in enumerate(lens):
        idx = torch.tensor([(table[b, i // PAGE].item(), i % PAGE) for i in range(k)])
        K, W = (t[idx[:, 0], idx[:, 1]].double().repeat_interleave(H // Hkv, dim=1) for t in (kp, vp))
        Q = q[cu[b]:cu[b + 1]].double()
        s = torch.einsum("nhd,khd->hnk", Q, K) * scale
        s.masked_fill_(torch.arange(k)[None, None] > (k - n + torch.arange(n))[None, :, None], float("-inf"))
        p = torch.softmax(s, -1)
        want[cu[b]:cu[b + 1]] = torch.einsum("hnk,khv->nhv", p, W)
        # a score's fp32 sum of D exact products, cut off by at most a unit each, then a product and the exponential (2^-21 of the exponent's size)
        ds = (D * 2.0 ** -23 + 2.0 ** -20) * torch.einsum("nhd,khd->hnk", Q.abs(), K.abs()).amax(-1) * scale + 2.0 ** -20
        size = torch.einsum("hnk,khv->nhv", p, W.abs())
        # weights rounded to 16 bits (fp16: subnormal ones to 2^-25 of a weight that is at least 2^-8 of the sum's), sums in fp32, one rounding
        tol[cu[b]:cu[b + 1]] = size * (u + 2 * ds.transpose(0, 1)[:, :, None] + k * 2.0 ** -22) + want[cu[b]:cu[b + 1]].abs() * u \
            + (k * 2.0 ** -25 * 2.0 ** 8 * W.abs().amax() if dtype == torch.float16 else 0.0) + 1e-6
    return q.reshape(cu[-1], H * D), kp, vp, table, torch.tensor([k for k, _ in lens], dtype=torch.int32), torch.tensor(cu, dtype=torch.int32), scale, want, tol


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("growth", [0.0, 5.0, 12.0, -9.0])
@pytest.mark.parametrize("H,Hkv", [(4, 2), (8, 1)])
def test_paged_heads(H, Hkv, growth, lens, dtype):
    q, kp, vp, table, kvl, cu, scale, want, tol = _problem(lens, H, Hkv, 128, 128, growth, dtype)
    out = A.attn_prefill(q.to(DEV), kp.to(DEV), vp.to(DEV), table.to(DEV), kvl.to(DEV), cu.to(DEV), scale, H, Hkv, 128)
    _lib.check_device_errors()
    err = (out.cpu().double().view_as(want) - want).abs() / tol
    assert bool((err <= 1).all()), err.max().item()


# values of at most 128: two score tiles a block; wider ones: one
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("growth", [0.0, 12.0, -9.0])
@pytest.mark.parametrize("D,V", [(64, 64), (192, 128), (128, 192)])
def test_windowed_kernel(D, V, growth, lens, dtype):
    H, Hkv = 4, 2
    q, kp, vp, table, kvl, cu, scale, want, tol = _problem(lens, H, Hkv, D, V, growth, dtype)
    blocks = [(int(cu[b]) + r, k - n + r, min(256, n - r), 0, 0, b) for b, (k, n) in enumerate(lens) for r in range(0, n, 256)]
    d = [t.to(DEV) for t in (q, kp, vp, table, torch.tensor(blocks, dtype=torch.int32))]
    out = torch.empty(q.shape[0], H * V, device=DEV, dtype=dtype)
    rc = _lib.kernels().fb_attn_window_paged(d[0].data_ptr(), H * D, q.shape[0], d[1].data_ptr(), d[2].data_ptr(), kp.shape[0] * PAGE, d[3].data_ptr(), table.shape[1],
                                             out.data_ptr(), H * V, None, 0, d[4].data_ptr(), len(blocks), H, Hkv, D, V, 0, 0, 0, scale, 0.0, None, None, 0, None, None,
                                             None, 0, 0, 1 if dtype == torch.bfloat16 else 0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    _lib.check_device_errors()
    err = (out.cpu().double().view_as(want) - want).abs() / tol
    assert bool((err <= 1).all()), err.max().item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("growth", [0.0, 5.0, 12.0, -9.0])
def test_wide_heads(growth, lens, dtype):
    q, kp, vp, table, kvl, cu, scale, want, tol = _problem(lens, 4, 2, 256, 256, growth, dtype)
    out = A.attn_prefill(q.to(DEV), kp.to(DEV), vp.to(DEV), table.to(DEV), kvl.to(DEV), cu.to(DEV), scale, 4, 2, 256)
    _lib.check_device_errors()
    err = (out.cpu().double().view_as(want) - want).abs() / tol
    assert bool((err <= 1).all()), err.max().item()
