"""RMS norm with the row in registers and query / key / value rows with 16-byte accesses: vector counts, widths and rotations at their edges."""
import pytest
import torch

from fastllm_b200.ops import attention as A, basic as B

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H", [8, 264, 1024, 1032, 2048, 2056, 8192, 8200, 32768])
@pytest.mark.parametrize("M", [1, 296, 297])
def test_rmsnorm_rows(M, H, dtype):
    g = torch.Generator(device=DEV).manual_seed(M + H)
    x = torch.randn(M, H + 8, device=DEV, generator=g).to(dtype)[:, :H]              # rows further apart than they are long
    res, w = torch.randn(M, H, device=DEV, generator=g).to(dtype), (1 + 0.1 * torch.randn(H, device=DEV, generator=g)).to(dtype)
    for residual in (None, res.clone()):
        y = B.rmsnorm(x, w, 1e-6, residual=residual, unit_offset=1.0)
        h = x if residual is None else (x.float() + res.float()).to(dtype)
        if residual is not None:
            assert torch.equal(residual, h)
        hd = h.double()
        ref = hd * torch.rsqrt(hd.square().mean(-1, keepdim=True) + 1e-6) * (w.double() + 1.0)
        # fp32 sums over threads (far below 2^-20), one rounding; fp16 below its smallest normal value rounds to 2^-25
        tol = ref.abs() * (torch.finfo(dtype).eps / 2 + 2.0 ** -20) + 2.0 ** -24
        assert bool(((y.double() - ref).abs() <= tol).all())


@pytest.mark.parametrize("T", [1, 255, 300])
@pytest.mark.parametrize("D,rot,mode,norm", [(32, 32, A.ROPE_NEOX, False), (64, 32, A.ROPE_INTERLEAVED, True), (128, 128, A.ROPE_NEOX, True), (128, 32, A.ROPE_NEOX, False),
                                             (256, 64, A.ROPE_NEOX, True), (256, 256, A.ROPE_INTERLEAVED, False), (512, 128, A.ROPE_NEOX, True), (128, 0, A.ROPE_NONE, False),
                                             (128, 24, A.ROPE_NEOX, True), (96, 96, A.ROPE_NEOX, False)])
@pytest.mark.parametrize("Hq,Hkv", [(7, 1), (16, 4)])
def test_qkv_rows(T, D, rot, mode, norm, Hq, Hkv):
    """Norm, rotation and page append against their statement in 64 bits; the last two forms take the general kernel."""
    dt, g = torch.bfloat16, torch.Generator().manual_seed(T + D + rot)
    rnd = lambda *s: torch.randn(*s, generator=g)
    qkv = rnd(T, (Hq + 2 * Hkv) * D).to(dt)
    pos, slots = torch.randint(0, 500, (T,), generator=g).int(), torch.randperm(3 * 128, generator=g)[:T].int()
    slots[T // 2] = -1
    cos, sin = A.build_rope_tables(rot or D, 512, 10000.0)
    qn, kn = ((1 + 0.1 * rnd(D)).to(dt), (1 + 0.1 * rnd(D)).to(dt)) if norm else (None, None)
    kp, vp = torch.zeros(3, 128, Hkv, D, dtype=dt, device=DEV), torch.zeros(3, 128, Hkv, D, dtype=dt, device=DEV)
    mv = lambda t: t.to(DEV) if t is not None else None
    q = A.qkv_post(mv(qkv), mv(pos), mv(slots), kp, vp, Hq, Hkv, D, mv(cos), mv(sin), mode, rot, mv(qn), mv(kn), 1e-6)

    def want(x, w):
        """The rotated rows and the sum of the magnitudes that each was made of."""
        if w is not None:
            x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double()
        y, size = x.clone(), x.abs()
        if mode != A.ROPE_NONE:
            c, s = (t[pos.long(), :rot // 2].double()[:, None] for t in (cos, sin))
            ia = torch.arange(rot // 2) if mode == A.ROPE_NEOX else torch.arange(0, rot, 2)
            ib = ia + (rot // 2 if mode == A.ROPE_NEOX else 1)
            xa, xb = x[..., ia], x[..., ib]
            y[..., ia], y[..., ib] = xa * c - xb * s, xb * c + xa * s
            size[..., ia], size[..., ib] = (xa * c).abs() + (xb * s).abs(), (xb * c).abs() + (xa * s).abs()
        return y, size

    rows = qkv.double().view(T, Hq + 2 * Hkv, D)
    live = slots >= 0
    at = slots[live].long()
    (rq, sq), (rk, sk) = want(rows[:, :Hq], qn), want(rows[:, Hq:Hq + Hkv], kn)
    for got, ref, size in ((q.view(T, Hq, D).cpu(), rq, sq), (kp.view(-1, Hkv, D).cpu()[at], rk[live], sk[live])):
        # one rounding to bf16 (2^-8 of the result); behind a norm another one before the rotation, 2^-8 of either element that it joins and 2^-16 of it
        # when it is rounded again; products of values below 8 have fp32 errors below 2^-18
        tol = 2.0 ** -8 * ref.abs() + (2.0 ** -8 + 2.0 ** -16) * size * norm + 2.0 ** -18
        assert bool(((got.double() - ref).abs() <= tol).all())
    assert torch.equal(vp.view(-1, Hkv, D).cpu()[at], qkv.view(T, Hq + 2 * Hkv, D)[live][:, Hq + Hkv:])
    unused = torch.ones(3 * 128, dtype=torch.bool)
    unused[at] = False
    assert not kp.view(3 * 128, -1).cpu()[unused].any() and not vp.view(3 * 128, -1).cpu()[unused].any()


# rows behind two waves of the SMs (four and two vectors a thread), a last round that half a warp or one warp has part in, more than 1024 vectors
@pytest.mark.parametrize("M,H", [(1, 8320), (64, 1152), (64, 8320), (297, 1152), (297, 1920), (297, 2944), (297, 8320), (330, 4096)])
@pytest.mark.parametrize("mode", [1, 2, 3, 4])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rmsnorm_with_8_bit_rows(M, H, mode, dtype):
    """The quantised rows beside the norm, or the norm rounded to their grid: the separate launches' bits."""
    from fastllm_b200.ops import quant_gemm as QG

    if mode < 3 and M > 128:
        pytest.skip("8-bit rows are made for up to 128")
    g = torch.Generator(device=DEV).manual_seed(M + H)
    x, res = torch.randn(M, H, device=DEV, generator=g).to(dtype), torch.randn(M, H, device=DEV, generator=g).to(dtype)
    w = (1 + 0.1 * torch.randn(H, device=DEV, generator=g)).to(dtype)
    for residual in (None, res):
        r0, r1 = (t.clone() if t is not None else None for t in (residual, residual))
        plain, y = B.rmsnorm(x, w, 1e-5, residual=r0), B.rmsnorm(x, w, 1e-5, residual=r1, quant_mode=mode)
        assert y.fb_quant[0] == mode and (residual is None or torch.equal(r0, r1))
        if mode >= 3:
            assert torch.equal(y, QG.round_act(plain, mode - 3))
            continue
        _, xq, scales, sums, _ = y.fb_quant
        want = QG.quant_act_i8(plain) if mode == 1 else QG.quant_act_fp8(plain)
        assert torch.equal(y, plain) and torch.equal(xq, want[0]) and torch.equal(scales[:, :M], want[1][:, :M])
        assert mode == 2 or torch.equal(sums[:, :M], want[2][:, :M])


def test_norm_rule_follows_the_device():
    """Rows on either side of the count from which a thread takes more vectors (two rows an SM)."""
    n = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device=DEV).manual_seed(n)
    x, w = torch.randn(n + 1, 4096, device=DEV, generator=g).bfloat16(), (1 + 0.1 * torch.randn(4096, device=DEV, generator=g)).bfloat16()
    many, few = B.rmsnorm(x, w, 1e-6), B.rmsnorm(x[:n], w, 1e-6)
    ref = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6) * w.double()
    for y in (many[:n], few):
        assert bool(((y.double() - ref[:n]).abs() <= ref[:n].abs() * (torch.finfo(y.dtype).eps / 2 + 2.0 ** -20) + 2.0 ** -24).all())
