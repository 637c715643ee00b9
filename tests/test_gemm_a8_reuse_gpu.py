"""8-bit-activation GEMMs whose k loop comes round to a stage again: repeated launches give the same bits, and every row is scaled by its
own block factors."""
import pytest
import torch

from fastllm_b200.ops import quant_gemm as QG
from fastllm_b200.ops.quant import LinearWeight

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["fp8", "int8", "int4g128"])
@pytest.mark.parametrize("rows", [9, 32, 64, 128])
def test_stages_are_not_refilled_under_their_readers(kind, rows):
    if kind == "int4g128" and rows > 64:
        rows = 61
    g = torch.Generator(device="cuda").manual_seed(rows)
    n, k = 28672, 4096                       # one CTA per output tile: 32 k blocks through at most 8 stages
    w = LinearWeight.from_dense((torch.randn(n, k, device="cuda", generator=g) * 0.02).bfloat16(), kind)
    # blocks of very different sizes: a factor of another block is off by orders of magnitude
    x = (torch.randn(rows, k, device="cuda", generator=g) * torch.exp2(torch.randint(-6, 7, (rows, k // 128, 1), device="cuda", generator=g).float())
         .expand(-1, -1, 128).reshape(rows, k)).bfloat16()
    first = w(x)
    for _ in range(20):
        assert torch.equal(w(x), first)
    # both grids are symmetric around what the kernel read; 2^-8: the result's rounding, and fp32 sums of 4096 products
    want = QG.round_act(x, 1 if kind == "fp8" else 0).double()
    # the rounded activations are stored in bf16 for this statement: 2^-9 per factor on top
    want = want @ w.dequant(torch.bfloat16).double().t()
    err = (first.double() - want).norm(dim=1) / want.norm(dim=1)
    assert err.max() < 3 * 2.0 ** -8, err


@pytest.mark.parametrize("kind", ["fp8", "int8", "int4g128"])
@pytest.mark.parametrize("rows", [8, 40, 100])
def test_grouped_stages_are_not_refilled_under_their_readers(kind, rows):
    """The same of the grouped products: a few experts, every one with rows, 32 k blocks; the dequantised weights' products per expert."""
    from fastllm_b200.ops import basic as B
    from fastllm_b200.ops import moe as MOE
    from fastllm_b200.ops import moe_grouped

    g = torch.Generator(device="cuda").manual_seed(rows)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    E, topk, H, inter, dt = 3, 2, 4096, 1024, torch.bfloat16
    load = lambda w, **k: LinearWeight.from_dense((0.02 * w).to(dt), kind, act_dtype=dt, **k)
    gu = [load(B.interleave_gate_up(rnd(inter, H), rnd(inter, H)), interleaved=True) for _ in range(E)]
    experts = MOE.ExpertWeights(E, 0, gu, [load(rnd(H, inter)) for _ in range(E)])
    experts.stacked = moe_grouped.stack_experts(experts)
    assert experts.stacked is not None and experts.stacked.kind != "dense"
    scale = torch.exp2(torch.randint(-6, 7, (rows, H // 128, 1), device="cuda", generator=g).float()).expand(-1, -1, 128).reshape(rows, H)
    x = (rnd(rows, H) * scale * 0.05).to(dt)
    idx, wts = MOE.route_topk(rnd(rows, E), None, topk, 0, True)
    first = moe_grouped.forward(x, idx, wts, experts)
    for _ in range(20):
        assert torch.equal(moe_grouped.forward(x, idx, wts, experts), first)
    # rows by themselves: each row's factors are its own whatever stands beside it (the products' sums and roundings are the same)
    for t in (0, rows // 2, rows - 1):
        one = moe_grouped.forward(x[t:t + 1].contiguous(), idx[t:t + 1].contiguous(), wts[t:t + 1].contiguous(), experts)
        assert ((one - first[t:t + 1]).double().norm() <= 2.0 ** -6 * one.double().norm())
