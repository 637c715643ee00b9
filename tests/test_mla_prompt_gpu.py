"""Prompts of multi-head latent attention: expanded keys and values against 64-bit attention, and no further off than the absorbed products."""
import pytest
import torch

from fastllm_b200.models.decoder import ForwardBatch
from fastllm_b200.ops import attention as A
from fastllm_b200.ops import basic as B
from fastllm_b200.ops import latent as LA
from fastllm_b200.ops import moe as MOE

pytestmark = pytest.mark.gpu
PAGE = A.PAGE_LEN


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("mode", [A.ROPE_INTERLEAVED, A.ROPE_NEOX])
@pytest.mark.parametrize("H,lens,news", [(16, [700, 300, 90], [700, 44, 1]), (5, [17, 256, 16], [17, 255, 16])])
def test_mla_prompt(dtype, mode, H, lens, news):
    nope, rope, lora, vd = 128, 64, 512, 128
    g = torch.Generator(device="cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    T, counts = sum(news), [(n + PAGE - 1) // PAGE for n in lens]
    order = torch.randperm(sum(counts), generator=g, device="cuda").to(torch.int32)
    table = torch.zeros(len(lens), max(counts) + 1, dtype=torch.int32, device="cuda")
    for b, c in enumerate(counts):
        table[b, :c] = order[sum(counts[:b]):sum(counts[:b]) + c]
    pool = rnd(sum(counts) + 1, PAGE, 1, lora + rope).to(dtype)
    w_uk, w_uv = ((lora ** -0.5 * rnd(H, n, lora)).to(dtype) for n in (nope, vd))
    q = rnd(T, H * (nope + rope)).to(dtype)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu = [sum(news[:i]) for i in range(len(news) + 1)]
    pos = [lens[b] - n + j for b, n in enumerate(news) for j in range(n)]
    fb = ForwardBatch(ids=i32([0] * T), positions=i32(pos), slots=i32([-1] * T), page_table=table, kv_lens=i32(lens), cu_q=i32(cu), cu_q_host=cu, kv_lens_host=lens)
    cos, sin = A.build_rope_tables(rope, 1024, 1e4, None, "cuda")
    scale = (nope + rope) ** -0.5
    la = LA.from_absorbed(H, nope, rope, lora, vd, w_uk, w_uk.transpose(1, 2).contiguous(), w_uv, scale, mode == A.ROPE_NEOX)
    assert LA.prompt_ok(la, q, pool)
    # the absorbed products
    q3 = q.view(T, H, nope + rope)
    q_full = torch.empty(T, H, lora + rope, device="cuda", dtype=dtype)
    q_full[..., lora:] = A.apply_rope_ref(q3[..., nope:], fb.positions, cos, sin, mode, rope)
    B.linear_batched(q, la.w_uk_t, H, nope + rope, q_full.view(T, -1), lora + rope)
    old = torch.empty(T, H * vd, device="cuda", dtype=dtype)
    B.linear_batched(MOE.mla_paged_attention(q_full, pool, fb, scale, lora).reshape(T, H * lora), w_uv, H, lora, old, vd)
    # 64 bits
    want = torch.empty(T, H, vd, dtype=torch.float64, device="cuda")
    qr = torch.cat([q3[..., :nope].double(), A.apply_rope_ref(q3[..., nope:].float(), fb.positions, cos, sin, mode, rope).double()], dim=-1)
    for b, L in enumerate(lens):
        rows = pool[table[b, :counts[b]].long()].reshape(-1, lora + rope)[:L].double()
        k = torch.cat([torch.einsum("kr,hdr->khd", rows[:, :lora], w_uk.double()), rows[:, None, lora:].expand(-1, H, -1)], dim=-1)
        s = torch.einsum("qhd,khd->hqk", qr[cu[b]:cu[b + 1]], k) * scale
        s = s.masked_fill(torch.arange(L, device="cuda")[None, :] > torch.arange(L - news[b], L, device="cuda")[:, None], float("-inf"))
        want[cu[b]:cu[b + 1]] = torch.einsum("hqk,khv->qhv", torch.softmax(s, -1), torch.einsum("kr,hvr->khv", rows[:, :lora], w_uv.double()))
    want = want.view(T, -1)
    qc = q.clone()
    got = LA.attention(la, qc, pool, fb, qc, None, (cos, sin))
    rel = lambda x: ((x.double() - want).norm() / want.norm()).item()
    # both ways round four times to 16 bits between the projections
    assert rel(got) <= 1.05 * rel(old), (rel(got), rel(old))


@pytest.mark.parametrize("form", ["absorbed", "expanded", "folded", "mixed"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_form(dtype, form, monkeypatch):
    picks = iter(["folded", "expanded", "absorbed"])
    monkeypatch.setattr(LA, "prompt_form", lambda *a: next(picks) if form == "mixed" else form)
    test_mla_prompt(dtype, A.ROPE_INTERLEAVED, 16, [700, 300, 90], [700, 44, 1])


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_neighbours_stay_out(value, monkeypatch):
    """Requests are expanded side by side: the first keys of one must not reach the rows of the one before."""
    H, nope, rope, lora, vd, dtype = 5, 128, 64, 512, 128, torch.float16
    lens, g = [700, 300, 250], torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    T, counts = sum(lens), [(n + PAGE - 1) // PAGE for n in lens]
    table = torch.zeros(len(lens), max(counts), dtype=torch.int32, device="cuda")
    for b, c in enumerate(counts):
        table[b, :c] = torch.arange(sum(counts[:b]), sum(counts[:b]) + c)
    pool = rnd(sum(counts), PAGE, 1, lora + rope).to(dtype)
    w_uk, w_uv = ((lora ** -0.5 * rnd(H, n, lora)).to(dtype) for n in (nope, vd))
    q = rnd(T, H * (nope + rope)).to(dtype)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    pos = [j for n in lens for j in range(n)]
    tables = A.build_rope_tables(rope, 1024, 1e4, None, "cuda")
    la = LA.from_absorbed(H, nope, rope, lora, vd, w_uk, w_uk.transpose(1, 2).contiguous(), w_uv, (nope + rope) ** -0.5, True)

    monkeypatch.setattr(LA, "prompt_form", lambda *a: "expanded")

    def run():
        fb = ForwardBatch(ids=i32([0] * T), positions=i32(pos), slots=i32([-1] * T), page_table=table, kv_lens=i32(lens), cu_q=i32(cu), cu_q_host=cu, kv_lens_host=lens)
        qc = q.clone()
        return LA.attention(la, qc, pool, fb, qc, None, tables)

    want = run()
    pool[counts[0]] = value
    got = run()
    assert torch.equal(got[:cu[1]], want[:cu[1]]) and torch.equal(got[cu[2]:], want[cu[2]:])


@pytest.mark.parametrize("form", ["absorbed", "expanded", "folded"])
@pytest.mark.parametrize("H", [5, 40])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_earlier_owners_stay_out(value, H, form, monkeypatch):
    """What stands in a request's last page behind its end, left by the page's earlier owner, must not reach its rows."""
    nope, rope, lora, vd, dtype, lens, n = 128, 64, 512, 128, torch.float16, [300, 129, 256], 3
    g = torch.Generator(device="cuda").manual_seed(2)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    pages = (max(lens) + PAGE - 1) // PAGE
    table = torch.arange(len(lens) * pages, device="cuda", dtype=torch.int32).view(len(lens), pages)
    pool = rnd(len(lens) * pages, PAGE, 1, lora + rope).to(dtype)
    w_uk, w_uv = ((lora ** -0.5 * rnd(H, d, lora)).to(dtype) for d in (nope, vd))
    q = rnd(n * len(lens), H * (nope + rope)).to(dtype)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu, pos = [n * i for i in range(len(lens) + 1)], [j for L in lens for j in range(L - n, L)]
    tables = A.build_rope_tables(rope, 1024, 1e4, None, "cuda")
    la = LA.from_absorbed(H, nope, rope, lora, vd, w_uk, w_uk.transpose(1, 2).contiguous(), w_uv, (nope + rope) ** -0.5, True)
    monkeypatch.setattr(LA, "prompt_form", lambda *a: form)
    outs = []
    for fill in (0.0, value):
        for b, L in enumerate(lens):
            pool[b * pages:(b + 1) * pages].view(-1, lora + rope)[L:] = fill
        fb = ForwardBatch(ids=i32([0] * len(pos)), positions=i32(pos), slots=i32([-1] * len(pos)), page_table=table, kv_lens=i32(lens), cu_q=i32(cu), cu_q_host=cu,
                          kv_lens_host=lens)
        qc = q.clone()
        outs.append(LA.attention(la, qc, pool, fb, qc, None, tables))
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("form", ["expanded", "folded"])
def test_scratch_is_bounded(form, monkeypatch):
    """One request behind a long history alone may need more than the limit: slices of heads, or of rows."""
    H, nope, rope, lora, vd, dtype, keys, n, limit = 12, 128, 64, 512, 128, torch.bfloat16, 4000, 70, 16 << 20
    g = torch.Generator(device="cuda").manual_seed(4)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)
    pages = (keys + PAGE - 1) // PAGE
    pool, q = rnd(pages, PAGE, 1, lora + rope), rnd(n, H * (nope + rope))
    w_uk, w_uv = (lora ** -0.5 * rnd(H, d, lora) for d in (nope, vd))
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    tables = A.build_rope_tables(rope, 4096, 1e4, None, "cuda")
    la = LA.from_absorbed(H, nope, rope, lora, vd, w_uk, w_uk.transpose(1, 2).contiguous(), w_uv, (nope + rope) ** -0.5, True)
    monkeypatch.setattr(LA, "prompt_form", lambda *a: form)

    def run():
        fb = ForwardBatch(ids=i32([0] * n), positions=i32(list(range(keys - n, keys))), slots=i32([-1] * n), page_table=i32([list(range(pages))]), kv_lens=i32([keys]),
                          cu_q=i32([0, n]), cu_q_host=[0, n], kv_lens_host=[keys])
        qc = q.clone()
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        out = LA.attention(la, qc, pool, fb, qc, None, tables)
        return out, torch.cuda.max_memory_allocated() - before

    monkeypatch.setattr(LA, "EXPAND_BYTES", 1 << 30)
    want, free = run()
    monkeypatch.setattr(LA, "EXPAND_BYTES", limit)
    got, bounded = run()
    # heads by themselves: the same sums; rows in other portions: sums over k in another order before two roundings to bf16
    assert torch.equal(got, want) if form == "expanded" else (got.double() - want.double()).norm() <= 2.0 ** -8 * want.double().norm()
    # folded: the gathered latents (4.6 MB) and their values beside the scores; both: plan, queries and result (below 2 MB)
    assert free > 1.5 * limit and bounded < limit + (12 << 20)
