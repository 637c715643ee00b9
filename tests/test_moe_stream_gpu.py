"""Grouped dense expert GEMM in one persistent launch, routing plan on many blocks, combine with a gated shared expert: edges of tiles and of row chunks."""
import pytest
import torch

from fastllm_b200.ops import _lib, basic as B
from fastllm_b200.ops import moe_grouped as MG

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _stream():
    return torch.cuda.current_stream().cuda_stream


# rows per expert around the tile widths 16 .. 256, unequal chunks, experts without rows (first, last and in between)
COUNTS = [[1], [0, 16, 17, 0, 15], [33, 0, 31, 64, 65, 1], [127, 129, 0, 200], [257, 0, 256, 511, 1, 0, 300]]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("form", ["plain", "swiglu", "clamp", "gelu"])
@pytest.mark.parametrize("counts,hint", [(c, h) for c in COUNTS for h in (1, 20, 40, 100, 256) if h <= max(16, 2 * max(c))])
def test_grouped_gemm(counts, hint, form, dtype):
    E, N, K = len(counts), 384, 200                                     # a k tail of 8, three weight tiles
    g = torch.Generator(device=DEV).manual_seed(sum(counts) + hint)
    offsets, at = [], 0
    for c in counts:
        offsets.append(at)
        at += (c + MG.PAD - 1) // MG.PAD * MG.PAD
    cap = at + 128
    x = torch.randn(cap, K, device=DEV, generator=g).to(dtype)
    w = (torch.randn(E, N, K, device=DEV, generator=g) * (0.3 if form == "clamp" else 0.1)).to(dtype)
    half = form in ("swiglu", "clamp")
    stacked = torch.stack([B.interleave_gate_up(w[e, :N // 2], w[e, N // 2:]) for e in range(E)]).contiguous() if half else w
    cols = N // 2 if half else N
    out = torch.full((cap, cols), 7.0, device=DEV, dtype=dtype)
    cd, od = (torch.tensor(t, dtype=torch.int32, device=DEV) for t in (counts, offsets))
    flags = {"plain": 0, "swiglu": B.GEMM_SWIGLU, "clamp": B.GEMM_SWIGLU | B.GEMM_GLU_CLAMP, "gelu": B.GEMM_GELU}[form]
    rc = _lib.kernels().fb_moe_grouped_gemm_act(x.data_ptr(), stacked.data_ptr(), out.data_ptr(), None, cd.data_ptr(), od.data_ptr(), cap, E, N, K, cols,
                                                max(counts) | (hint << 16), 1 if dtype == torch.bfloat16 else 0, flags, sum(counts), 2.0, 1.7, _stream())
    assert rc == 0
    torch.cuda.synchronize()
    _lib.check_device_errors()
    u = torch.finfo(dtype).eps / 2
    for e, (o, n) in enumerate(zip(offsets, counts)):
        xs = x[o:o + n].double()
        y = xs @ w[e].double().t()
        # the products are exact; each of the sum's K steps may cut off one unit of fp32 of the largest partial sum
        err = K * 2.0 ** -23 * (xs.abs() @ w[e].double().abs().t())
        if form == "gelu":
            y, err = torch.nn.functional.gelu(y), 1.13 * err            # |gelu'| < 1.13
        elif half:
            a, b, ea, eb = y[:, :cols], y[:, cols:], err[:, :cols], err[:, cols:]
            if form == "clamp":
                a, b = a.clamp(max=2.0), b.clamp(-2.0, 2.0) + 1.0
                y, slope = a * torch.sigmoid(1.7 * a), 1.1              # |d/da a sigmoid(c a)| < 1.1 for every c
            else:
                y, slope = torch.nn.functional.silu(a), 1.1
            y, err = y * b, slope * ea * b.abs() + y.abs() * eb
        # the activations in fp32 with fast exponentials (2^-20), then one rounding
        tol = err + y.abs() * (u + 2.0 ** -20) + 2.0 ** -22
        if dtype == torch.float16:
            tol = tol + 2.0 ** -25
        assert bool(((out[o:o + n].double() - y).abs() <= tol).all()), (e, n, ((out[o:o + n].double() - y).abs() / tol).max().item())
        assert bool((out[o + n:offsets[e + 1] if e + 1 < E else cap] == 7.0).all())          # rows between the segments stay as they are


@pytest.mark.parametrize("T,topk,E,first,n_local", [(513, 8, 8, 0, 8), (700, 6, 1024, 0, 1024), (4001, 10, 512, 0, 512), (2049, 2, 16, 9, 7), (34, 31, 512, 128, 256)])
def test_plan_on_many_blocks(T, topk, E, first, n_local):
    g = torch.Generator().manual_seed(T)
    idx = torch.rand(T, E, generator=g).topk(topk, dim=1).indices.int()
    idx[:T // 2, 0] = first                                               # a busy expert; a token may name it twice
    flat = idx.flatten().long() - first
    mine = (flat >= 0) & (flat < n_local)
    onehot = torch.zeros(T * topk, n_local, dtype=torch.int32)
    onehot[mine, flat[mine]] = 1
    cnt = onehot.sum(0)
    padded = (cnt + 15) // 16 * 16
    off = padded.cumsum(0) - padded
    rank = onehot.cumsum(0) - 1
    want = torch.full((T * topk,), -1, dtype=torch.long)
    want[mine] = off[flat[mine]] + rank[mine, flat[mine]]
    plan = [torch.full((n,), -7, dtype=torch.int32, device=DEV) for n in (n_local, n_local, T * topk, 1)]
    d = idx.to(DEV)
    rc = _lib.kernels().fb_moe_plan(d.data_ptr(), T, topk, first, n_local, *(t.data_ptr() for t in plan), 16, _stream())
    assert rc == 0
    for got, w in zip(plan, (cnt, off, want, padded.sum().reshape(1))):
        assert torch.equal(got.cpu().long(), w.long())


# a CTA a place below 256 tokens, a CTA a token from there; rows narrower and wider than a CTA, places in and beside multiples of 4
@pytest.mark.parametrize("T,H,topk", [(1, 8, 1), (255, 264, 5), (256, 2056, 3), (300, 2048, 8), (257, 4104, 10)])
def test_rows_reach_their_places(T, H, topk):
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randint(-32768, 32767, (T, H), device=DEV, generator=g, dtype=torch.int16)
    pos = torch.randperm(T * topk + 9, device=DEV, generator=g)[:T * topk].int()
    pos[3::7] = -1                                                        # experts of another rank
    xs = torch.full((T * topk + 9, H), 7, device=DEV, dtype=torch.int16)
    want = xs.clone()
    want[pos[pos >= 0].long()] = x.repeat_interleave(topk, dim=0)[pos >= 0]
    assert _lib.kernels().fb_moe_gather(x.data_ptr(), pos.data_ptr(), xs.data_ptr(), T, topk, H, _stream()) == 0
    assert torch.equal(xs, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,H,topk,ld", [(1, 8, 1, 1), (37, 264, 8, 13), (300, 4096, 3, 544)])
def test_combine_with_gated_rows(T, H, topk, ld, dtype):
    g = torch.Generator(device=DEV).manual_seed(T)
    ys, add = torch.randn(T * topk + 5, H, device=DEV, generator=g).to(dtype), torch.randn(T, H, device=DEV, generator=g).to(dtype)
    pos = torch.randperm(T * topk + 5, device=DEV, generator=g)[:T * topk].int()
    pos[::7] = -1                                                         # experts of another rank
    w = torch.rand(T, topk, device=DEV, generator=g)
    gate = (4 * torch.randn(T, ld, device=DEV, generator=g))[:, ld // 2]
    out = torch.empty(T, H, device=DEV, dtype=dtype)
    picked = (ys.double()[pos.clamp(min=0).long()] * (pos >= 0)[:, None]).view(T, topk, H) * w.double()[:, :, None]
    for a, gt in ((None, None), (add, None), (add, gate)):
        rc = _lib.kernels().fb_moe_combine_gated(ys.data_ptr(), pos.data_ptr(), w.data_ptr(), a.data_ptr() if a is not None else None,
                                                 gt.data_ptr() if gt is not None else None, gt.stride(0) if gt is not None else 0, out.data_ptr(), T, topk, H,
                                                 1 if dtype == torch.bfloat16 else 0, _stream())
        assert rc == 0
        extra = 0.0 if a is None else add.double() * (1.0 if gt is None else torch.sigmoid(gate.double())[:, None])
        ref = picked.sum(1) + extra
        size = picked.abs().sum(1) + (extra.abs() if a is not None else 0.0)
        # topk + 1 sums in fp32 and a fast sigmoid (2^-20), then one rounding
        tol = ref.abs() * torch.finfo(dtype).eps / 2 + size * ((topk + 1) * 2.0 ** -23 + 2.0 ** -20) + 2.0 ** -25
        assert bool(((out.double() - ref).abs() <= tol).all())


@pytest.mark.parametrize("mode,bias,groups", [(0, False, (1, 1)), (1, True, (1, 1)), (1, True, (4, 2)), (2, False, (1, 1))])
@pytest.mark.parametrize("E", [1, 31, 32, 33, 64, 65, 128, 129, 256, 257, 511, 512])
def test_route_at_every_width(E, mode, bias, groups):
    from fastllm_b200.ops import moe as MOE

    n_group, keep = groups if E % 4 == 0 else (1, 1)
    g = torch.Generator(device=DEV).manual_seed(E)
    wide = torch.randn(67, E + 3, device=DEV, generator=g)
    b = 0.1 * torch.randn(E, device=DEV, generator=g) if bias else None
    topk = min(10, E // n_group * keep)
    for logits in (wide[:, :E].contiguous(), wide[:, 3:]):
        idx, w = MOE.route_topk(logits, b, topk, mode, mode != 2, n_group, keep, 2.5)
        ri, rw = MOE.route_topk_ref(logits.double(), b.double() if bias else None, topk, mode, mode != 2, n_group, keep, 2.5)
        # picked in order of their scores; a score is an fp32 exponential (2^-20) over a sum, the weights are renormalised: no near-tie at this seed
        assert torch.equal(idx.long(), ri.long())
        torch.testing.assert_close(w.double(), rw.double(), rtol=2.0 ** -18, atol=1e-7)


@pytest.mark.parametrize("counts,hint", [([33, 0, 31, 64, 65, 1], 20), ([257, 0, 300], 256)])
@pytest.mark.parametrize("form", ["bias", "swiglu+bias", "clamp+bias", "geglu", "relu2", "gelu tanh+bias"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_grouped_gemm_epilogues(counts, hint, form, dtype):
    """A bias per expert and the less common activations: what the entry took before the tiles went through one launch."""
    E, N, K = len(counts), 384, 200
    g = torch.Generator(device=DEV).manual_seed(sum(counts))
    offsets, at = [], 0
    for c in counts:
        offsets.append(at)
        at += (c + MG.PAD - 1) // MG.PAD * MG.PAD
    x, bias = torch.randn(at + 128, K, device=DEV, generator=g).to(dtype), torch.randn(E, N, device=DEV, generator=g).to(dtype)
    w = (torch.randn(E, N, K, device=DEV, generator=g) * 0.1).to(dtype)
    half = form.split("+")[0] in ("swiglu", "clamp", "geglu")
    mix = lambda t: torch.stack([B.interleave_gate_up(t[e, :N // 2], t[e, N // 2:]) for e in range(E)]).contiguous()
    wk, bk = (mix(w), mix(bias[..., None])[..., 0].contiguous()) if half else (w, bias)
    cols = N // 2 if half else N
    out = torch.empty(at + 128, cols, device=DEV, dtype=dtype)
    cd, od = (torch.tensor(t, dtype=torch.int32, device=DEV) for t in (counts, offsets))
    flags = {"bias": 0, "swiglu": B.GEMM_SWIGLU, "clamp": B.GEMM_SWIGLU | B.GEMM_GLU_CLAMP, "geglu": B.GEMM_SWIGLU | B.GEMM_GEGLU, "relu2": B.GEMM_RELU2,
             "gelu tanh": B.GEMM_GELU_TANH}[form.split("+")[0]] | (B.GEMM_BIAS if "bias" in form else 0)
    call = lambda b, f: _lib.kernels().fb_moe_grouped_gemm_act(x.data_ptr(), wk.data_ptr(), out.data_ptr(), b, cd.data_ptr(), od.data_ptr(), at + 128, E, N, K, cols,
                                                               max(counts) | (hint << 16), 1 if dtype == torch.bfloat16 else 0, f, sum(counts), 2.0, 1.7, _stream())
    assert call(bk.data_ptr(), flags) == 0
    _lib.check_device_errors()
    for e, (o, n) in enumerate(zip(offsets, counts)):
        xs = x[o:o + n].double()
        y = xs @ w[e].double().t()
        err = K * 2.0 ** -23 * (xs.abs() @ w[e].double().abs().t())            # as above
        if "bias" in form:
            y, err = y + bias[e].double(), err + 2.0 ** -23 * (y.abs() + bias[e].double().abs())
        if form == "relu2":
            y, err = y.relu().square(), 2.0 * y.abs() * err + err * err
        elif form.startswith("gelu"):
            y, err = torch.nn.functional.gelu(y, approximate="tanh"), 1.13 * err
        elif half:
            a, b, ea, eb = y[:, :cols], y[:, cols:], err[:, :cols], err[:, cols:]
            if form.startswith("clamp"):
                a, b = a.clamp(max=2.0), b.clamp(-2.0, 2.0) + 1.0
                y = a * torch.sigmoid(1.7 * a)
            else:
                y = torch.nn.functional.silu(a) if form.startswith("swiglu") else torch.nn.functional.gelu(a, approximate="tanh")
            y, err = y * b, 1.13 * ea * b.abs() + y.abs() * eb
        tol = err + y.abs() * (torch.finfo(dtype).eps / 2 + 2.0 ** -19) + 2.0 ** -22 + (2.0 ** -25 if dtype == torch.float16 else 0.0)
        assert bool(((out[o:o + n].double() - y).abs() <= tol).all()), (e, ((out[o:o + n].double() - y).abs() / tol).max().item())
    # a bias that the flags do not ask for is not looked at; a bias, residual or 32-bit result that the entry cannot give is refused
    assert call(bk.data_ptr(), flags & ~B.GEMM_BIAS) == 0
    assert call(None, flags | B.GEMM_BIAS) == -1 and call(None, B.GEMM_RESIDUAL) == -1 and call(None, B.GEMM_OUT_F32) == -1


@pytest.mark.parametrize("counts", [[1], [16], [40], [128], [0, 17, 0, 3], [5, 0]])
@pytest.mark.parametrize("N,K,form", [(1536, 2048, "swiglu+bias"), (520, 4104, "plain"), (2048, 4160, "gelu"), (4096, 4096, "swiglu"), (4096, 14336, "plain")])
def test_few_tiles_share_out_their_k(counts, N, K, form):
    """Two and four CTAs a tile (k blocks that do not divide, a last tile of 8 rows, experts without rows) against 64 bits, and the same bits again."""
    E, dtype = len(counts), torch.bfloat16
    g = torch.Generator(device=DEV).manual_seed(N + sum(counts))
    offsets, at = [], 0
    for c in counts:
        offsets.append(at)
        at += (c + MG.PAD - 1) // MG.PAD * MG.PAD
    x = torch.randn(at + 128, K, device=DEV, generator=g).to(dtype)
    w = (torch.randn(E, (N + 127) // 128 * 128, K, device=DEV, generator=g) * K ** -0.5).to(dtype)
    bias = torch.randn(E, N, device=DEV, generator=g).to(dtype)
    half = form.startswith("swiglu")
    cols = N // 2 if half else N
    flags = {"plain": 0, "gelu": B.GEMM_GELU, "swiglu": B.GEMM_SWIGLU, "swiglu+bias": B.GEMM_SWIGLU | B.GEMM_BIAS}[form]
    cd, od = (torch.tensor(t, dtype=torch.int32, device=DEV) for t in (counts, offsets))
    outs = []
    for _ in range(3):
        out = torch.full((at + 128, cols), 7.0, device=DEV, dtype=dtype)
        rc = _lib.kernels().fb_moe_grouped_gemm_act(x.data_ptr(), w.data_ptr(), out.data_ptr(), bias.data_ptr(), cd.data_ptr(), od.data_ptr(), at + 128, E, N, K, cols,
                                                    max(counts), 1, flags, sum(counts), 0.0, 1.0, _stream())
        assert rc == 0
        outs.append(out)
    _lib.check_device_errors()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    for e, (o, n) in enumerate(zip(offsets, counts)):
        xs, wd = x[o:o + n].double(), w[e, :N].double()
        y, err = xs @ wd.t(), K * 2.0 ** -23 * (xs.abs() @ wd.abs().t())
        if form == "gelu":
            y, err = torch.nn.functional.gelu(y), 1.13 * err
        elif half:
            if "bias" in form:
                y, err = y + bias[e].double(), err + 2.0 ** -23 * (y.abs() + bias[e].double().abs())
            t = torch.arange(cols, device=DEV)
            gate = t // 64 * 128 + t % 64                                   # rows of a 128-row tile: 64 of the gate, 64 of the other factor
            a, b, ea, eb = y[:, gate], y[:, gate + 64], err[:, gate], err[:, gate + 64]
            y = torch.nn.functional.silu(a)
            y, err = y * b, 1.1 * ea * b.abs() + y.abs() * eb
        tol = err + y.abs() * (torch.finfo(dtype).eps / 2 + 2.0 ** -20) + 2.0 ** -22
        assert bool(((outs[0][o:o + n].double() - y).abs() <= tol).all()), (e, n)
        assert bool((outs[0][o + n:offsets[e + 1] if e + 1 < E else None] == 7.0).all())
