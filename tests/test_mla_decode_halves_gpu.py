"""Latent decode attention by halves of a page: ends of requests around the halves, items of several pages, maxima that grow by more than what lets an accumulator
stand (2^8), by leaps and not at all; values that take 256 and 512 columns of tensor memory."""
import pytest
import torch

from fastllm_b200.ops import _lib, attention as A

pytestmark = pytest.mark.gpu
DEV, PAGE = "cuda", 128
LENS = [1, 63, 64, 65, 127, 129, 191, 193, 640, 1300, 2700]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("growth", [0.0, 12.0, -9.0])
@pytest.mark.parametrize("H,dq,dv", [(16, 576, 512), (40, 576, 512), (5, 320, 256), (32, 64, 64)])
@pytest.mark.parametrize("copies", [1, 14])                                # 14: several pages an item
def test_halves(copies, H, dq, dv, growth, dtype):
    g = torch.Generator().manual_seed(H + dq + int(growth))
    lens = LENS * copies
    pages = [(n + PAGE - 1) // PAGE for n in LENS]
    pool = torch.full((sum(pages) + 1, PAGE, 1, dq), 30.0, dtype=dtype)       # stale rows are finite
    perm, table, at = torch.randperm(sum(pages) + 1, generator=g).int(), torch.zeros(len(LENS), max(pages), dtype=torch.int32), 0
    scale = dq ** -0.5
    q = torch.randn(len(LENS), H, dq, generator=g)
    q[:, :, 0] = 4.0
    q = q.to(dtype)
    want, tol, u = torch.zeros(len(LENS), H, dv, dtype=torch.float64), torch.zeros(len(LENS), H, dv, dtype=torch.float64), torch.finfo(dtype).eps / 2
    for b, n in enumerate(LENS):
        table[b, :pages[b]] = perm[at:at + pages[b]]
        at += pages[b]
        lat = torch.randn(n, dq, generator=g)
        lat[:, 0] = growth / 1.4426950408889634 / scale / 4 * (torch.arange(n) // 64 % 7)          # scores climb (fall) over seven halves, then start again
        lat = lat.to(dtype)
        for i in range(pages[b]):
            k = min(PAGE, n - i * PAGE)
            pool[table[b, i], :k, 0] = lat[i * PAGE:i * PAGE + k]
        K, Q = lat.double(), q[b].double()
        p = torch.softmax(Q @ K.t() * scale, -1)
        V = K[:, :dv]
        want[b] = p @ V
        # a score's fp32 sum of dq exact products, cut off by at most a unit each, a product and the exponential; weights rounded to 16 bits (fp16: subnormal
        # ones to 2^-25 of a weight that is at least 2^-8 of the sum's), sums in fp32, one rounding
        ds = (dq * 2.0 ** -23 + 2.0 ** -20) * (Q.abs() @ K.abs().t()).amax(-1, keepdim=True) * scale + 2.0 ** -20
        tol[b] = (p @ V.abs()) * (u + 2 * ds + n * 2.0 ** -22) + want[b].abs() * u + (n * 2.0 ** -17 * V.abs().amax() if dtype == torch.float16 else 0.0) + 1e-6
    rep = lambda t: t.repeat(copies, *([1] * (t.dim() - 1))).to(DEV)
    out = A.mla_decode(rep(q), pool.to(DEV), rep(table), torch.tensor(lens, dtype=torch.int32, device=DEV), scale, lora=dv)
    torch.cuda.synchronize()
    _lib.check_device_errors()
    err = (out.cpu().double().view(copies, len(LENS), H, dv) - want).abs() / tol
    assert bool((err <= 1).all()), err.max().item()
