"""Attention at head widths other than 128: the kernels against 64-bit attention, and no further off than the fp32 evaluation."""
import pytest
import torch

from fastllm_b200.ops import attention as A

pytestmark = pytest.mark.gpu
PAGE = A.PAGE_LEN


def _setup(dtype, D, Hq, Hkv, lens, news, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    counts = [(n + PAGE - 1) // PAGE for n in lens]
    order = torch.randperm(sum(counts), generator=g, device="cuda").to(torch.int32)
    table = torch.zeros(len(lens), max(counts) + 1, dtype=torch.int32, device="cuda")
    for b, c in enumerate(counts):
        table[b, :c] = order[sum(counts[:b]):sum(counts[:b]) + c]
    pools = [rnd(sum(counts), PAGE, Hkv, D).to(dtype) for _ in range(2)]
    q, gate = (1.5 * rnd(sum(news), Hq * D)).to(dtype), rnd(sum(news), Hq * D).to(dtype)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    return q, gate, *pools, table, i32(lens), i32([sum(news[:i]) for i in range(len(news) + 1)])


def _exact(q, gate, k_pool, v_pool, table, lens, cu, scale, Hq, Hkv, D):
    out = torch.empty(q.shape, dtype=torch.float64, device=q.device)
    cu = cu.tolist()
    for b, L in enumerate(lens.tolist()):
        r0, r1 = cu[b], cu[b + 1]
        pg = table[b, :(L + PAGE - 1) // PAGE].long()
        k, v = (p[pg].reshape(-1, Hkv, D)[:L].double().repeat_interleave(Hq // Hkv, dim=1) for p in (k_pool, v_pool))
        s = torch.einsum("qhd,khd->hqk", q[r0:r1].double().view(-1, Hq, D), k) * scale
        hidden = torch.arange(L, device=q.device)[None, :] > torch.arange(L - (r1 - r0), L, device=q.device)[:, None]
        out[r0:r1] = torch.einsum("hqk,khd->qhd", torch.softmax(s.masked_fill(hidden, float("-inf")), -1), v).reshape(r1 - r0, -1)
    return out if gate is None else out * torch.sigmoid(gate.double())


rel = lambda x, y: ((x.double() - y).norm() / y.norm()).item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,Hq,Hkv", [(64, 4, 2), (72, 3, 3), (192, 2, 1), (256, 8, 1), (256, 20, 1)])
def test_wide_attention(dtype, D, Hq, Hkv):
    scale = D ** -0.5
    # prompts: one token, tile edges, a continuation, several steps
    lens, news = [1, 128, 129, 300, 700], [1, 128, 129, 57, 700]
    q, gate, kp, vp, pt, ln, cu = _setup(dtype, D, Hq, Hkv, lens, news, D)
    assert A.wide_ok(q, kp, Hq, Hkv, D)
    for gt in (None, gate):
        got = A.attn_prefill(q, kp, vp, pt, ln, cu, scale, Hq, Hkv, D, gate=gt)
        want = _exact(q, gt, kp, vp, pt, ln, cu, scale, Hq, Hkv, D)
        old = A.paged_attention_ref(q, kp, vp, pt, ln.cpu(), cu.cpu(), scale, Hq, Hkv, D)
        if gt is not None:
            old = (old.float() * torch.sigmoid(gt.float())).to(old.dtype)
        # both end in one rounding to 16 bits; 2 %: which of two neighbours a tie goes to
        assert rel(got, want) <= 1.02 * rel(old, want)
        assert (got.double() - want).abs().max() <= 1.5 * (old.double() - want).abs().max()
    # decoded tokens
    lens = [1, 127, 128, 129, 1000]
    q, gate, kp, vp, pt, ln, cu = _setup(dtype, D, Hq, Hkv, lens, [1] * 5, D + 1)
    for gt in (None, gate):
        got = A.attn_decode(q, kp, vp, pt, ln, scale, Hq, Hkv, D, gate=gt)
        want = _exact(q, gt, kp, vp, pt, ln, cu, scale, Hq, Hkv, D)
        old = A.paged_attention_ref(q, kp, vp, pt, ln.cpu(), cu.cpu(), scale, Hq, Hkv, D)
        if gt is not None:
            old = (old.float() * torch.sigmoid(gt.float())).to(old.dtype)
        assert rel(got, want) <= 1.05 * rel(old, want)


def test_large_scores_and_empty_rows():
    """Scores far apart, a row whose request holds nothing (a padded decode row), a batch larger than a workspace made for another one."""
    D, Hq, Hkv = 256, 4, 2
    q, gate, kp, vp, pt, ln, cu = _setup(torch.bfloat16, D, Hq, Hkv, [400, 64], [200, 64], 3)
    q = q * 30
    want = _exact(q, None, kp, vp, pt, ln, cu, D ** -0.5, Hq, Hkv, D)
    old = A.paged_attention_ref(q, kp, vp, pt, ln.cpu(), cu.cpu(), D ** -0.5, Hq, Hkv, D)
    assert rel(A.attn_prefill(q, kp, vp, pt, ln, cu, D ** -0.5, Hq, Hkv, D), want) <= 1.02 * rel(old, want)
    ln[1] = 0
    out = A.attn_decode(q[:2].contiguous(), kp, vp, pt, ln, D ** -0.5, Hq, Hkv, D)
    assert torch.isfinite(out).all() and (out[1] == 0).all()


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("D,Hq,Hkv", [(64, 4, 2), (72, 3, 3), (256, 20, 1)])
@pytest.mark.parametrize("lens,news", [([1, 63, 64, 130, 700], [1, 63, 40, 130, 300]), ([1, 63, 128, 130, 700], None)])
def test_values_behind_a_request_stay_out(lens, news, D, Hq, Hkv, value):
    """A page's slots behind its request's end hold whatever an earlier owner left there (``news`` None: decoded tokens)."""
    scale = D ** -0.5
    q, gate, kp, vp, pt, ln, cu = _setup(torch.float16, D, Hq, Hkv, lens, news or [1] * len(lens), D + 2)

    def run():
        return (A.attn_prefill(q, kp, vp, pt, ln, cu, scale, Hq, Hkv, D, gate=gate) if news else A.attn_decode(q, kp, vp, pt, ln, scale, Hq, Hkv, D, gate=gate))

    want = run()
    assert torch.isfinite(want).all()
    for b, n in enumerate(lens):
        last = pt[b, (n - 1) // PAGE]
        kp[last, (n - 1) % PAGE + 1:], vp[last, (n - 1) % PAGE + 1:] = value, value
    assert torch.equal(run(), want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 256])
def test_small_weights_keep_their_digits(D, dtype):
    """One key takes nearly all of the weight and has no value: what comes out is the 2^-20 of the weight that another one gets."""
    T, L = 150, 200
    q = torch.zeros(T, D, device="cuda")
    q[:, 0] = torch.linspace(1.0, 1.1, T, device="cuda")
    k, v = torch.zeros(2, PAGE, 1, D, device="cuda"), torch.randn(2, PAGE, 1, D, device="cuda")
    k[..., 0] = -300.0
    k[0, 0, 0, 0], k[0, 1, 0, 0] = 0.0, -13.0
    v[0, 0], v[0, 1] = 0.0, 1000.0
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    p = torch.exp(q[:, 0].double() * k[0, 1, 0, 0].double())
    want = (p / (1 + p) * v[0, 1, 0, 0].double())[:, None].expand(T, D)
    # One rounding to 16 bits.  The weight in two terms: 2^-17 of it in bf16; in fp16 what the scaled second term leaves, 2^-38 of the largest
    # weight and 2^-17.3 of this one (above 2^-20.7).  Its exponent has three roundings to fp32 (the scale, the product, the difference):
    # 21 ln 2 * 3 * 2^-24 < 2^-18.4; exponential, sum and quotient add less than 2^-21.
    bound = torch.finfo(dtype).eps / 2 + 2.0 ** -16
    got = A.attn_prefill(q, k, v, i32([[0, 1]]), i32([L]), i32([0, T]), 1.0, 1, 1, D)
    assert ((got.double() - want).abs() <= bound * want).all()
    got = A.attn_decode(q, k, v, i32([[0, 1]] * T), i32([L] * T), 1.0, 1, 1, D)
    assert ((got.double() - want).abs() <= bound * want).all()


@pytest.mark.parametrize("form", ["int64 lists", "lists on the host", "pools with gaps", "values of another type"])
def test_other_operands_take_the_general_evaluation(form):
    """What the kernels cannot read as it is gives what it gave before there were kernels."""
    D, Hq, Hkv, scale = 64, 4, 2, 0.125
    q, gate, kp, vp, pt, ln, cu = _setup(torch.bfloat16, D, Hq, Hkv, [300, 5, 129], [40, 5, 129], 11)
    assert A.wide_ok(q, kp, Hq, Hkv, D)
    ref = lambda q, cu: A.paged_attention_ref(q, kp, vp, pt, ln.cpu(), cu.cpu(), scale, Hq, Hkv, D)
    want, one = ref(q, cu), ref(q[:3], torch.arange(4))
    k, v, t, n, c = kp, vp, pt, ln, cu
    if form == "int64 lists":
        t, n, c = pt.long(), ln.long(), cu.long()
    elif form == "lists on the host":
        n, c = ln.cpu(), cu.cpu()
    elif form == "pools with gaps":
        k, v = (torch.stack([x, x], dim=1)[:, 0] for x in (kp, vp))
    else:
        v = vp.float()
    assert torch.equal(A.attn_prefill(q, k, v, t, n, c, scale, Hq, Hkv, D), want)
    assert torch.equal(A.attn_decode(q[:3], k, v, t, n, scale, Hq, Hkv, D), one)
    assert torch.equal(A.attn_prefill(q, k, v, t, n, c, scale, Hq, Hkv, D, gate=gate), (want.float() * torch.sigmoid(gate.float())).to(q.dtype))
    assert torch.equal(A.attn_decode(q[:3], k, v, t, n, scale, Hq, Hkv, D, gate=gate[:3]), (one.float() * torch.sigmoid(gate[:3].float())).to(q.dtype))


@pytest.mark.parametrize("n,made_for", [(3, (2, 8)), (3, (8, 1)), (1030, (8, 8))])
def test_decode_beyond_a_workspace(n, made_for):
    """More rows or pages than the workspace was made for, and more rows than a plan takes."""
    D, Hq, Hkv, scale = 64, 4, 2, 0.125
    lens = [300, 5, 129] + [1] * (n - 3)
    q, _, kp, vp, pt, ln, cu = _setup(torch.bfloat16, D, Hq, Hkv, lens, [1] * n, n)
    ws = A.DecodeWorkspace(made_for[0], Hkv, Hq // Hkv, made_for[1], q.device, D)
    got = A.attn_decode(q, kp, vp, pt, ln, scale, Hq, Hkv, D, ws=ws)
    want = _exact(q, None, kp, vp, pt, ln, cu, scale, Hq, Hkv, D)
    assert rel(got, want) <= 1.05 * rel(A.paged_attention_ref(q, kp, vp, pt, ln.cpu(), cu.cpu(), scale, Hq, Hkv, D), want)
