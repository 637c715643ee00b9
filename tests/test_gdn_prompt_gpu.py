"""Chunked gated delta rule: packed prompts through the kernels against the rule token by token in 64 bits."""
import pytest
import torch
import torch.nn.functional as F

from fastllm_b200.ops import _lib
from fastllm_b200.ops import linear_attn as L

pytestmark = pytest.mark.gpu


def _conv64(proj, conv_w, conv, cu, slots, C):
    """silu(convolution) in 64 bits; the requests' windows advance."""
    out = torch.empty(proj.shape[0], C, dtype=torch.float64, device=proj.device)
    for i, s in enumerate(slots):
        lo, hi = cu[i], cu[i + 1]
        seq = torch.cat([conv[s].t().double(), proj[lo:hi, :C].double()])
        conv[s] = seq[-3:].t().to(proj.dtype)
        out[lo:hi] = F.silu(sum(seq[j:j + hi - lo] * conv_w.double()[:, j] for j in range(4)))
    return out


def _rule64(y, proj, A_log, dt_bias, norm_w, eps, rec, cu, slots, Hk, Hv):
    """The rule behind the convolution, token by token; the head row is rounded where the kernels store it."""
    kd, vd = Hk * 128, Hv * 128
    C = 2 * kd + vd
    out = torch.empty(proj.shape[0], vd, dtype=torch.float64, device=proj.device)
    for i, s in enumerate(slots):
        lo, hi = cu[i], cu[i + 1]
        yd = y[lo:hi].double()
        q, k, v = yd[:, :kd].view(-1, Hk, 128), yd[:, kd:2 * kd].view(-1, Hk, 128), yd[:, 2 * kd:].view(-1, Hv, 128)
        q, k = (t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(Hv // Hk, dim=1) for t in (q * 128 ** -0.5, k))
        b, a = proj[lo:hi, C + vd:C + vd + Hv].double(), proj[lo:hi, C + vd + Hv:C + vd + 2 * Hv].double()
        g = torch.exp(-A_log.double().exp() * F.softplus(a + dt_bias.double()))
        S, o = rec[s], []
        for t in range(hi - lo):
            S = S * g[t, :, None, None]
            d = (v[t] - torch.einsum("hkv,hk->hv", S, k[t])) * torch.sigmoid(b[t])[:, None]
            S = S + k[t][:, :, None] * d[:, None, :]
            o.append(torch.einsum("hkv,hk->hv", S, q[t]))
        rec[s] = S
        z = proj[lo:hi, C:C + vd].double().view(-1, Hv, 128)
        o = torch.stack(o).to(proj.dtype).double()
        out[lo:hi] = (o * torch.rsqrt(o.square().mean(-1, keepdim=True) + eps) * norm_w.double() * F.silu(z)).reshape(-1, vd)
    return out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens,decay", [([1], 0.0), ([2, 3, 64], 0.0), ([65, 1, 127, 200], -2.0), ([63, 130], 3.0), ([700], -6.0)])
def test_prompt_matches_the_rule(dtype, lens, decay, monkeypatch):
    Hk, Hv = (2, 4) if len(lens) > 1 else (3, 3)
    dev, kd, vd, T = "cuda", Hk * 128, Hv * 128, sum(lens)
    gen = torch.Generator(device=dev).manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device=dev, generator=gen)
    C, width = 2 * kd + vd, (2 * kd + 2 * vd + 2 * Hv + 7) // 8 * 8
    proj = rnd(T, width).to(dtype)
    conv_w, norm_w = (0.5 * rnd(C, 4)).to(dtype), (1 + 0.1 * rnd(128)).to(dtype)
    A_log, dt_bias = torch.log(0.3 + rnd(Hv).abs()), rnd(Hv) + decay       # from hardly any to nearly full forgetting
    slots = [4, 1, 0, 3][:len(lens)]
    first = (rnd(5, C, 3).to(dtype), 0.2 * rnd(5, Hv, 128, 128))
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    plan = L._PromptPlan(cu, slots, dev)
    rel = lambda x, y: ((x.double() - y).norm() / y.norm()).item()
    # the convolution: its exact value rounded, but for ties that fp32 sums of four products do not settle
    conv64, conv = first[0].clone(), first[0].clone()
    y64, y = _conv64(proj, conv_w, conv64, cu, slots, C), torch.empty(T, C, device=dev, dtype=dtype)
    rc = _lib.kernels().fb_gdn_conv_prompt(proj.data_ptr(), width, conv_w.data_ptr(), conv.data_ptr(), plan.chunks.data_ptr(), plan.n_chunks, plan.reqs.data_ptr(),
                                           plan.n_reqs, y.data_ptr(), C, 1 if dtype == torch.bfloat16 else 0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(conv, conv64)
    assert (y != y64.to(dtype)).double().mean() < 1e-3
    torch.testing.assert_close(y.double(), y64, rtol=torch.finfo(dtype).eps, atol=1e-6)
    # the rule on that output, in 64 bits and with the operators in fp32
    rec64, rec32 = first[1].double(), first[1].clone()
    want = _rule64(y, proj, A_log, dt_bias, norm_w, 1e-6, rec64, cu, slots, Hk, Hv)
    b, a = proj[:, C + vd:C + vd + Hv], proj[:, C + vd + Hv:C + vd + 2 * Hv]
    o = L.gated_delta_rule(y[:, :kd].reshape(T, Hk, 128), y[:, kd:2 * kd].reshape(T, Hk, 128), y[:, 2 * kd:].reshape(T, Hv, 128), a, b, A_log, dt_bias, rec32,
                           cu, slots, Hv // Hk)
    old = L.rmsnorm_gated(o, proj[:, C:C + vd].reshape(T, Hv, 128), norm_w, 1e-6).reshape(T, vd)
    assert L.prompt_kernels_ok(proj, conv_w, conv, first[1], Hk, Hv, 128, 128)
    for scratch in (L.SCRATCH_BYTES, 1):                     # 1: a head at a time
        monkeypatch.setattr(L, "SCRATCH_BYTES", scratch)
        conv, rec = first[0].clone(), first[1].clone()
        got = L.gated_delta_prompt(proj, conv_w, conv, A_log, dt_bias, norm_w, 1e-6, rec, plan, Hk, Hv)
        assert torch.equal(conv, conv64)
        # fp32 sums in another order: 8 units in the last place (2^-21) beside the operators' own error
        assert rel(rec[slots], rec64[slots]) <= 1.2 * rel(rec32[slots], rec64[slots]) + 2.0 ** -21
        assert rel(got, want) <= 1.02 * rel(old, want) + 2.0 ** -21
        untouched = [s for s in range(5) if s not in slots]
        assert torch.equal(rec[untouched], first[1][untouched]) and torch.equal(conv[untouched], first[0][untouched])


def test_convolution_rounds_as_often_wrongly_as_fp32():
    """SiLU in full precision: results that are not the nearest fp16 value are as rare as with the fp32 operators (1700 of 16 million, spread 2.5 %)."""
    T, C, dev, dtype = 4000, 4096, "cuda", torch.float16
    gen = torch.Generator(device=dev).manual_seed(8)
    x, w = torch.randn(T, C, device=dev, generator=gen).to(dtype), (0.5 * torch.randn(C, 4, device=dev, generator=gen)).to(dtype)
    state = torch.zeros(1, C, 3, device=dev, dtype=dtype)
    plan, y = L._PromptPlan([0, T], [0], dev), torch.empty(T, C, device=dev, dtype=dtype)
    rc = _lib.kernels().fb_gdn_conv_prompt(x.data_ptr(), C, w.data_ptr(), state.clone().data_ptr(), plan.chunks.data_ptr(), plan.n_chunks, plan.reqs.data_ptr(),
                                           plan.n_reqs, y.data_ptr(), C, 0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    want = _conv64(x, w, state.clone(), [0, T], [0], C).to(dtype)
    off = lambda t: (t != want).double().mean().item()
    assert off(y) <= 1.1 * off(L.causal_conv1d(x, w, state.clone(), [0, T], [0])), (off(y), off(L.causal_conv1d(x, w, state.clone(), [0, T], [0])))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens,decay,Hk,Hv", [([30, 64], 0.0, 2, 4), ([63, 130], 3.0, 2, 4), ([65, 127, 200], -2.0, 2, 4), ([700], -6.0, 3, 3), ([1500], -8.0, 2, 4),
                                              ([900], 1.0, 8, 16), ([333], -2.0, 8, 16)])
@pytest.mark.parametrize("fresh", [False, True])
def test_states_keep_fp32(dtype, lens, decay, Hk, Hv, fresh):
    """The states' error against 64 bits is that of the operators in fp32."""
    dev, kd, vd, T = "cuda", Hk * 128, Hv * 128, sum(lens)
    gen = torch.Generator(device=dev).manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device=dev, generator=gen)
    C, width = 2 * kd + vd, (2 * kd + 2 * vd + 2 * Hv + 7) // 8 * 8
    proj, conv_w, norm_w = rnd(T, width).to(dtype), (0.5 * rnd(C, 4)).to(dtype), (1 + 0.1 * rnd(128)).to(dtype)
    A_log, dt_bias = torch.log(0.3 + rnd(Hv).abs()), rnd(Hv) + decay
    slots, cu = list(range(len(lens))), [sum(lens[:i]) for i in range(len(lens) + 1)]
    conv, first = rnd(len(lens), C, 3).to(dtype), (0.0 if fresh else 0.2) * rnd(len(lens), Hv, 128, 128)
    plan, rec, rec32, rec64 = L._PromptPlan(cu, slots, dev), first.clone(), first.clone(), first.double()
    y = _conv64(proj, conv_w, conv.clone(), cu, slots, C).to(dtype)
    _rule64(y, proj, A_log, dt_bias, norm_w, 1e-6, rec64, cu, slots, Hk, Hv)
    b, a = proj[:, C + vd:C + vd + Hv], proj[:, C + vd + Hv:C + vd + 2 * Hv]
    L.gated_delta_rule(y[:, :kd].reshape(T, Hk, 128), y[:, kd:2 * kd].reshape(T, Hk, 128), y[:, 2 * kd:].reshape(T, Hv, 128), a, b, A_log, dt_bias, rec32, cu, slots,
                       Hv // Hk)
    scratch = [torch.empty(plan.n_chunks * Hv * k, device=dev) for k in (64 * 64, 9 * 64, 128 * 64, 128 * 128)]
    out, p = torch.empty(T, vd, device=dev, dtype=dtype), lambda t: t.data_ptr()
    rc = _lib.kernels().fb_gdn_prompt(p(y), C, p(a), p(b), width, p(proj[:, C:]), width, p(A_log), p(dt_bias), p(norm_w), p(rec), p(out), p(plan.chunks), plan.n_chunks,
                                      p(plan.reqs), plan.n_reqs, *map(p, scratch), Hk, Hv, 0, Hv, 1e-6, 1 if dtype == torch.bfloat16 else 0,
                                      torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    rel = lambda x: ((x.double() - rec64).norm() / rec64.norm()).item()
    # 2^-25: half a unit in the last place of the states themselves, whichever way their last addition rounds
    assert rel(rec) <= rel(rec32) + 2.0 ** -25, (rel(rec), rel(rec32))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T", [1, 65, 200])
def test_gates_at_odd_addresses(dtype, T):
    """Gates are read in pairs where pairs are aligned: the other reads give the same bits."""
    dev, Hk, Hv = "cuda", 2, 4
    kd, vd = Hk * 128, Hv * 128
    gen = torch.Generator(device=dev).manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device=dev, generator=gen)
    y, ab, norm_w = rnd(T, 2 * kd + vd).to(dtype), rnd(T, 2 * Hv).to(dtype), (1 + 0.1 * rnd(128)).to(dtype)
    A_log, dt_bias, first = torch.log(0.3 + rnd(Hv).abs()), rnd(Hv), 0.2 * rnd(1, Hv, 128, 128)
    plan, z, p = L._PromptPlan([0, T], [0], dev), rnd(T, vd).to(dtype), lambda t: t.data_ptr()
    scratch = [torch.empty(plan.n_chunks * Hv * k, device=dev) for k in (64 * 64, 9 * 64, 128 * 64, 128 * 128)]
    outs = []
    for pad, at in ((0, 0), (1, 0), (2, 1)):                  # aligned; odd row distance; odd start
        wide = torch.zeros(T, vd + pad, device=dev, dtype=dtype)
        wide[:, at:at + vd] = z
        rec, out = first.clone(), torch.empty(T, vd, device=dev, dtype=dtype)
        rc = _lib.kernels().fb_gdn_prompt(p(y), 2 * kd + vd, p(ab[:, Hv:]), p(ab), 2 * Hv, p(wide[:, at:]), vd + pad, p(A_log), p(dt_bias), p(norm_w), p(rec), p(out),
                                          p(plan.chunks), plan.n_chunks, p(plan.reqs), plan.n_reqs, *map(p, scratch), Hk, Hv, 0, Hv, 1e-6,
                                          1 if dtype == torch.bfloat16 else 0, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
