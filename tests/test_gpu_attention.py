"""tcgen05 flash attention forward/backward vs an fp32 PyTorch restatement."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(q, k, v, causal):
    # q: [B,S,Hq,D], k/v: [B,S,Hkv,D] fp32
    b, s, hq, d = q.shape
    hkv = k.shape[2]
    k = k.repeat_interleave(hq // hkv, dim=2)
    v = v.repeat_interleave(hq // hkv, dim=2)
    att = torch.einsum("bqhd,bkhd->bhqk", q, k) / math.sqrt(d)
    if causal:
        mask = torch.ones(s, s, device=q.device, dtype=torch.bool).tril()
        att = att.masked_fill(~mask, float("-inf"))
    p = att.softmax(-1)
    return torch.einsum("bhqk,bkhd->bqhd", p, v)


@pytest.mark.parametrize("b,s,hq,hkv", [(1, 128, 1, 1), (2, 384, 4, 4), (1, 512, 8, 2), (2, 200, 2, 1), (1, 2048, 2, 2),
                                         (1, 4096, 32, 8), (1, 4096, 16, 2), (2, 1000, 8, 1), (1, 8192, 8, 1)])
@pytest.mark.parametrize("causal", [True, False])
def test_attention_fwd_bwd(b, s, hq, hkv, causal):
    from yafsdp_b200.ops import kernels

    if not causal and s >= 4096:
        pytest.skip("long sequences are checked in the causal form the models use")
    torch.manual_seed(0)
    d = 128
    t = b * s
    width = (hq + 2 * hkv) * d
    qkv = torch.randn(t, width, device="cuda", dtype=torch.bfloat16)
    q = qkv[:, : hq * d]
    k = qkv[:, hq * d : (hq + hkv) * d]
    v = qkv[:, (hq + hkv) * d :]
    scale = 1.0 / math.sqrt(d)
    out, lse = kernels.attn_fwd(q, k, v, b, s, hq, hkv, scale, causal)
    qf = q.float().view(b, s, hq, d).detach().requires_grad_(True)
    kf = k.float().view(b, s, hkv, d).detach().requires_grad_(True)
    vf = v.float().view(b, s, hkv, d).detach().requires_grad_(True)
    ref = _ref(qf, kf, vf, causal)
    torch.cuda.synchronize()
    kernels.check_status()
    err = (out.float().view(b, s, hq, d) - ref).abs().max().item()
    assert err < 2e-2, f"forward max err {err}"
    dout = torch.randn(t, hq * d, device="cuda", dtype=torch.bfloat16)
    ref.backward(dout.float().view(b, s, hq, d))
    dqkv = torch.zeros_like(qkv)
    kernels.attn_bwd(q, k, v, out, dout, lse, dqkv[:, : hq * d], dqkv[:, hq * d : (hq + hkv) * d], dqkv[:, (hq + hkv) * d :],
                     b, s, hq, hkv, scale, causal)
    torch.cuda.synchronize()
    kernels.check_status()
    for name, got, want in (
        ("dq", dqkv[:, : hq * d], qf.grad.reshape(t, -1)),
        ("dk", dqkv[:, hq * d : (hq + hkv) * d], kf.grad.reshape(t, -1)),
        ("dv", dqkv[:, (hq + hkv) * d :], vf.grad.reshape(t, -1)),
    ):
        e = (got.float() - want).abs().max().item()
        ref_scale = want.abs().max().item()
        assert e <= 2e-2 * ref_scale + 2e-2, f"{name} max err {e} (scale {ref_scale})"


def test_attention_forward_with_growing_scores():
    """Scores that keep growing along the key axis force the forward kernel to move its reference maximum many times
    (the output then is rescaled in TMEM); a large constant offset exercises the exponent range."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(1)
    b, s, hq, hkv, d = 1, 1024, 2, 1, 128
    t = b * s
    qkv = torch.randn(t, (hq + 2 * hkv) * d, device="cuda", dtype=torch.bfloat16)
    ramp = torch.linspace(0.0, 6.0, s, device="cuda").view(s, 1)
    qkv[:, hq * d : (hq + hkv) * d] = (qkv[:, hq * d : (hq + hkv) * d].float() * (1.0 + ramp)).to(torch.bfloat16)  # later keys score higher
    q, k, v = qkv[:, : hq * d], qkv[:, hq * d : (hq + hkv) * d], qkv[:, (hq + hkv) * d :]
    out, lse = kernels.attn_fwd(q, k, v, b, s, hq, hkv, 1.0 / math.sqrt(d), True)
    ref = _ref(q.float().view(b, s, hq, d), k.float().view(b, s, hkv, d), v.float().view(b, s, hkv, d), True)
    torch.cuda.synchronize()
    kernels.check_status()
    assert (out.float().view(b, s, hq, d) - ref).abs().max().item() < 3e-2
    att = torch.einsum("bqhd,bkhd->bhqk", q.float().view(b, s, hq, d), k.float().view(b, s, hkv, d).repeat_interleave(hq // hkv, dim=2)) / math.sqrt(d)
    att = att.masked_fill(~torch.ones(s, s, device="cuda", dtype=torch.bool).tril(), float("-inf"))
    assert torch.allclose(lse, att.logsumexp(-1), atol=2e-2, rtol=1e-3)


@pytest.mark.parametrize("b,s,hq,hkv", [(1, 300, 8, 2), (2, 129, 4, 1), (1, 64, 6, 1), (3, 45, 8, 8)])
@pytest.mark.parametrize("causal", [True, False])
def test_attention_bwd_shared_key_tiles(b, s, hq, hkv, causal):
    """The query heads of a KV head dealt to one or several CTAs: the same gradients but for the order of fp32 sums, which may
    move a bf16 result by one rounding (2^-8 of it)."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(5)
    t, d = b * s, 128
    qkv = torch.randn(t, (hq + 2 * hkv) * d, device="cuda").bfloat16()
    q, k, v = qkv[:, : hq * d], qkv[:, hq * d : (hq + hkv) * d], qkv[:, (hq + hkv) * d :]
    scale = 1.0 / math.sqrt(d)
    out, lse = kernels.attn_fwd(q, k, v, b, s, hq, hkv, scale, causal)
    dout = torch.randn_like(out)
    got = []
    for parts in [p for p in range(1, hq // hkv + 1) if (hq // hkv) % p == 0]:
        g = torch.full_like(qkv, float("nan"))
        kernels.attn_bwd(q, k, v, out, dout, lse, g[:, : hq * d], g[:, hq * d : (hq + hkv) * d], g[:, (hq + hkv) * d :], b, s, hq, hkv,
                         scale, causal, head_parts=parts)
        got.append(g)
    torch.cuda.synchronize()
    kernels.check_status()
    for g in got[1:]:
        assert torch.allclose(g.float(), got[0].float(), rtol=2.0**-7, atol=1e-5)
    qf, kf, vf = (x.double().view(b, s, -1, d).requires_grad_(True) for x in (q, k, v))
    _ref(qf, kf, vf, causal).backward(dout.double().view(b, s, hq, d))
    want = torch.cat([x.grad.reshape(t, -1) for x in (qf, kf, vf)], dim=1)
    assert ((got[0].double() - want).norm() / want.norm()).item() < 2.0**-7  # P, dS and the results are rounded to bf16


@pytest.mark.parametrize("b,s,hq,hkv,parts", [(2, 200, 4, 2, 1), (1, 333, 4, 1, 4), (2, 64, 2, 2, 1)])
def test_attention_bwd_through_rotation(b, s, hq, hkv, parts):
    """dq and dk straight back through RoPE, against the rotation kernel on the rounded gradients (one bf16 rounding less)."""
    from yafsdp_b200.ops import kernels
    from yafsdp_b200.ops.functional import rope_table

    torch.manual_seed(16)
    t, d = b * s, 128
    qkv = torch.randn(t, (hq + 2 * hkv) * d, device="cuda").bfloat16()
    q, k, v = qkv[:, : hq * d], qkv[:, hq * d : (hq + hkv) * d], qkv[:, (hq + hkv) * d :]
    scale, table = 1.0 / math.sqrt(d), rope_table(s + 5, d, 10000.0, "cuda")
    out, lse = kernels.attn_fwd(q, k, v, b, s, hq, hkv, scale, True)
    dout = torch.randn_like(out)
    got, want = torch.empty_like(qkv), torch.empty_like(qkv)
    for g, rope in ((got, table), (want, None)):
        kernels.attn_bwd(q, k, v, out, dout, lse, g[:, : hq * d], g[:, hq * d : (hq + hkv) * d], g[:, (hq + hkv) * d :], b, s, hq, hkv,
                         scale, True, head_parts=parts, rope=rope)
    kernels.rope_(want, table, s, 0, hq + hkv, d, backward=True)
    torch.cuda.synchronize()
    kernels.check_status()
    assert ((got.double() - want.double()).norm() / want.double().norm()).item() < 2.0**-8


@pytest.mark.parametrize("b,s,hq,hkv,parts", [(1, 777, 16, 2, 8), (1, 2048, 16, 2, 4), (2, 300, 14, 2, 7), (1, 640, 8, 8, 1)])
@pytest.mark.parametrize("rotated", [False, True])
def test_attention_bwd_key_gradients_repeat(b, s, hq, hkv, parts, rotated):
    """dk and dv do not vary from run to run, however many CTAs share a key tile: every part's sums have a place of their own."""
    from yafsdp_b200.ops import kernels
    from yafsdp_b200.ops.functional import rope_table

    torch.manual_seed(18)
    t, d = b * s, 128
    qkv = torch.randn(t, (hq + 2 * hkv) * d, device="cuda").bfloat16()
    q, k, v = qkv[:, : hq * d], qkv[:, hq * d : (hq + hkv) * d], qkv[:, (hq + hkv) * d :]
    scale, table = 1.0 / math.sqrt(d), rope_table(s, d, 10000.0, "cuda") if rotated else None
    out, lse = kernels.attn_fwd(q, k, v, b, s, hq, hkv, scale, True)
    dout = torch.randn_like(out)
    runs = []
    for _ in range(6):
        g = torch.empty_like(qkv)
        kernels.attn_bwd(q, k, v, out, dout, lse, g[:, : hq * d], g[:, hq * d : (hq + hkv) * d], g[:, (hq + hkv) * d :], b, s, hq, hkv,
                         scale, True, head_parts=parts, rope=table)
        runs.append(g[:, hq * d :])
    torch.cuda.synchronize()
    kernels.check_status()
    assert all(torch.equal(r, runs[0]) for r in runs[1:])


def test_attention_bwd_refuses_short_scratch():
    from yafsdp_b200 import _native

    b, s, hq, hkv, d = 1, 64, 4, 1, 128
    x = torch.zeros(s, hq * d, device="cuda").bfloat16()
    f = torch.zeros(s * hq * d, device="cuda")
    p, fp = x.data_ptr(), f.data_ptr()
    for parts, floats in ((2, 2 * 2 * 128 * d - 1), (4, 2 * 2 * 128 * d), (2, 0)):
        assert _native.lib().yf_attn_bwd_parts(p, p, p, p, p, fp, fp, fp, fp, floats, parts, None, p, p, p, b, s, hq, hkv, hq * d, d, hq * d, hq * d,
                                               hq * d, d, 0.1, 1, torch.cuda.current_stream().cuda_stream) == -1


def test_attention_fwd_adds_row_sums_in_the_order_of_the_keys():
    """The sums of a row's even and odd groups of 64 keys run through the keys one pair after the other, so that the results of
    ordinary rows repeat bit for bit from version to version.  One weight of 1 and 127 of 2^-25 tell the orders apart: every pair
    of small ones is lost next to the 1 (2^-24, ties to even), while those of the other group add up to 2^-19."""
    from yafsdp_b200.ops import kernels

    s, d, scale = 128, 128, 0.6931471824645996  # scale * log2(e) is 1 in fp32
    qkv = torch.zeros(s, 3 * d, device="cuda").bfloat16()
    qkv[:, 0] = 1.0
    qkv[1:, d] = -25.0
    _, lse = kernels.attn_fwd(qkv[:, :d], qkv[:, d : 2 * d], qkv[:, 2 * d :], 1, s, 1, 1, scale, False)
    torch.cuda.synchronize()
    kernels.check_status()
    assert (lse.double() - math.log1p(2.0**-19)).abs().max().item() < 2.0**-24  # the next sum is 2^-20 away


def test_attention_bwd_heads_in_several_groups():
    """A dQ accumulator beyond 64 MB and heads for more than three groups: the CTAs go group by group, the last group is smaller.
    Some heads against fp64 (P, dS and the results are rounded to bf16)."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(22)
    b, s, h, d = 2, 2304, 32, 128
    assert b * s * h * d * 4 > 64 << 20 and (2 * 148 + s // 128 - 1) // (s // 128) < b * h / 3  # the rule's two conditions on 148 SMs
    qkv = torch.randn(b * s, 3 * h * d, device="cuda").bfloat16()
    q, k, v = qkv[:, : h * d], qkv[:, h * d : 2 * h * d], qkv[:, 2 * h * d :]
    scale = 1.0 / math.sqrt(d)
    out, lse = kernels.attn_fwd(q, k, v, b, s, h, h, scale, True)
    dout = torch.randn_like(out)
    g = torch.full_like(qkv, float("nan"))
    kernels.attn_bwd(q, k, v, out, dout, lse, g[:, : h * d], g[:, h * d : 2 * h * d], g[:, 2 * h * d :], b, s, h, h, scale, True)
    torch.cuda.synchronize()
    kernels.check_status()
    assert not g.isnan().any()
    for bi, hi in ((0, 0), (0, 16), (0, 17), (1, 1), (1, 2), (1, 19), (1, 31)):  # both sides of the groups' borders, first and last
        rows = slice(bi * s, (bi + 1) * s)
        qf, kf, vf = (x[rows, hi * d : (hi + 1) * d].double().view(1, s, 1, d).requires_grad_(True) for x in (q, k, v))
        _ref(qf, kf, vf, True).backward(dout[rows, hi * d : (hi + 1) * d].double().view(1, s, 1, d))
        for x, at in ((qf, hi), (kf, h + hi), (vf, 2 * h + hi)):
            want = x.grad.reshape(s, d)
            assert ((g[rows, at * d : (at + 1) * d].double() - want).norm() / want.norm()).item() < 2.0**-7


def test_attention_fwd_moves_the_reference_of_a_whole_tile():
    """A row whose scores grow by more than 2^8 behind the first key block moves the reference of the exponents for the 128 rows of
    its tile, and for no others: a row's bits do not depend on how rows are dealt to warps.  The second weight is 2^0.5 relative to
    the first block's maximum, which bf16 rounds to 181 / 128, and cancels the first value exactly; relative to its own maximum it is 1
    and leaves 1 - 181 / 128 * 2^-0.5 of a row sum of 1 + 2^-0.5."""
    from yafsdp_b200.ops import kernels

    s, d, scale = 256, 128, 0.6931471824645996  # scale * log2(e) is 1 in fp32: weights are powers of two
    qkv = torch.zeros(s, 3 * d, device="cuda").bfloat16()
    q, k, v = qkv[:, :d], qkv[:, d : 2 * d], qkv[:, 2 * d :]
    q[:, 0] = 1.0
    q[70, 1] = 1.0  # the row that grows: third warp of the first tile
    k[:, 0] = -100.0
    k[0, 0], k[128, 0], k[128, 1] = 0.0, 0.5, 16.0
    v[0], v[128] = -181.0 / 128.0, 1.0
    out, _ = kernels.attn_fwd(q, k, v, 1, s, 1, 1, scale, False)
    torch.cuda.synchronize()
    kernels.check_status()
    moved = (1.0 - 181.0 / 128.0 * 0.5**0.5) / (1.0 + 0.5**0.5)
    rows = [r for r in range(128) if r != 70]
    assert torch.allclose(out[rows].double(), torch.tensor(moved, dtype=torch.float64, device="cuda"), rtol=2.0**-6)  # bf16, and a difference near 1e-4
    assert (out[128:] == 0).all()
    assert (out[70].double() - 1.0).abs().max().item() < 2.0**-8
