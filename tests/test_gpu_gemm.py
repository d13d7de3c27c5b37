"""tcgen05 GEMM family vs an fp32 PyTorch restatement, every operand-major combination."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, a_mn, b_mn):
    af = a.float().t() if a_mn else a.float()
    bf = b.float().t() if b_mn else b.float()
    return af @ bf.t()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (256, 512, 256), (384, 640, 192), (200, 328, 136), (2048, 1024, 2048),
                                   (448, 1000, 136), (2304, 512, 64), (512, 2304, 4096)])
def test_gemm_matches_fp32(m, n, k, a_mn, b_mn):
    from yafsdp_b200.ops import kernels

    torch.manual_seed(0)
    a = torch.randn((k, m) if a_mn else (m, k), device="cuda", dtype=torch.bfloat16)
    b = torch.randn((k, n) if b_mn else (n, k), device="cuda", dtype=torch.bfloat16)
    out = kernels.gemm(a, b, a_mn_major=a_mn, b_mn_major=b_mn)
    ref = _ref(a, b, a_mn, b_mn)
    torch.cuda.synchronize()
    kernels.check_status()
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, f"max err {err} vs scale {scale}"


def test_gemm_fp32_out_accumulate_alpha():
    from yafsdp_b200.ops import kernels

    torch.manual_seed(1)
    m, n, k = 512, 768, 320
    a = torch.randn(k, m, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(k, n, device="cuda", dtype=torch.bfloat16)
    out = torch.randn(m, n, device="cuda", dtype=torch.float32)
    ref = out + 0.5 * (a.float().t() @ b.float())
    kernels.gemm(a, b, a_mn_major=True, b_mn_major=True, out=out, accumulate=True, alpha=0.5)
    torch.cuda.synchronize()
    kernels.check_status()
    assert torch.allclose(out, ref, rtol=1e-3, atol=1e-2)


def test_gemm_strided_views():
    """Operands and output that are column slices of wider buffers (row pitch > row length)."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(2)
    big_a = torch.randn(256, 512, device="cuda", dtype=torch.bfloat16)
    big_b = torch.randn(384, 512, device="cuda", dtype=torch.bfloat16)
    big_c = torch.zeros(256, 1024, device="cuda", dtype=torch.bfloat16)
    a = big_a[:, 128:384]
    b = big_b[:, 256:512]
    c = big_c[:, 256:640]
    kernels.gemm(a, b, out=c)
    torch.cuda.synchronize()
    kernels.check_status()
    ref = a.float() @ b.float().t()
    assert (c.float() - ref).abs().max().item() <= 1e-2 * ref.abs().max().item() + 1e-2
    assert big_c[:, :256].abs().max().item() == 0 and big_c[:, 640:].abs().max().item() == 0


def test_gemm_fused_sum_of_squares():
    """The fp32 epilogue can add the squared norm of what it writes to a device scalar (gradient-norm fusion)."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(3)
    m, n, k = 640, 1000, 256  # n not a multiple of the tile: clipped columns must not contribute
    a = torch.randn(k, m, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(k, n, device="cuda", dtype=torch.bfloat16)
    out = torch.empty(m, n, device="cuda", dtype=torch.float32)
    acc = torch.full((1,), 5.0, device="cuda")
    kernels.gemm(a, b, a_mn_major=True, b_mn_major=True, out=out, sumsq=acc)
    torch.cuda.synchronize()
    kernels.check_status()
    want = 5.0 + out.double().pow(2).sum().item()
    assert abs(acc.item() - want) <= 1e-4 * want


@pytest.mark.parametrize("m,n,k", [(256, 512, 256), (200, 328, 136), (2048, 4096, 1024), (448, 1000, 136), (130, 136, 64)])
def test_gemm_residual_epilogue(m, n, k):
    """out = A @ B^T + R with the bf16 residual added in fp32 inside the epilogue (single-CTA and CTA-pair tiles, ragged
    edges, a residual with a row pitch, and in place on the residual)."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(3)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(n, k, device="cuda", dtype=torch.bfloat16)
    wide = (8 * torch.randn(m, n + 24, device="cuda")).bfloat16()
    res = wide[:, 8 : 8 + n]  # 16-byte aligned view with a pitch of n + 24
    ref = a.float() @ b.float().t() + res.float()
    out = kernels.gemm(a, b, residual=res)
    torch.cuda.synchronize()
    kernels.check_status()
    scale = ref.abs().max().item()
    assert (out.float() - ref).abs().max().item() <= 1e-2 * scale + 1e-2
    # one rounding only: no worse than rounding the exact sum to bf16, up to the accumulation order
    assert (out.float() - ref).abs().max().item() <= (ref.bfloat16().float() - ref).abs().max().item() + 1e-3 * scale
    inplace = res.contiguous()
    kernels.gemm(a, b, residual=inplace, out=inplace)
    torch.cuda.synchronize()
    assert torch.equal(inplace, out)


@pytest.mark.parametrize("tile", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("splits", [1, 2, 3, 4])
@pytest.mark.parametrize("m,n,k,a_mn,b_mn", [(45, 1024, 1048, False, False), (264, 520, 1032, True, True), (1337, 2056, 1024, False, True),
                                             (8, 8, 2048, False, False), (4096, 4104, 256, True, True)])
def test_gemm_tile_shapes_and_split_last_wave(tile, splits, m, n, k, a_mn, b_mn):
    """Every tile shape, whole and with its last wave's tiles split along K: fp32 output (plain, accumulating, with the squared
    norm) and bf16 output with a residual.  fp32 sums of k products: a few sqrt(k) * 2^-24; a bf16 result: 2^-8."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(7)
    a = torch.randn((k, m) if a_mn else (m, k), device="cuda", dtype=torch.bfloat16)
    b = torch.randn((k, n) if b_mn else (n, k), device="cuda", dtype=torch.bfloat16)
    res = torch.randn(m, n, device="cuda", dtype=torch.bfloat16)
    ref = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    kw = dict(a_mn_major=a_mn, b_mn_major=b_mn, tile=tile, splits=splits)
    sq = torch.zeros(1, device="cuda")
    f32 = kernels.gemm(a, b, out_dtype=torch.float32, sumsq=sq, **kw)
    acc = kernels.gemm(a, b, out=torch.full_like(f32, 3.0), accumulate=True, **kw)
    low = kernels.gemm(a, b, residual=res, **kw)
    again = kernels.gemm(a, b, out_dtype=torch.float32, **kw)
    torch.cuda.synchronize()
    kernels.check_status()

    def off(x, y):
        return ((x.double() - y).norm() / y.norm()).item()

    lim = 3.0 * k ** 0.5 * 2.0**-24
    assert off(f32, ref) < lim and off(acc, ref + 3.0) < lim
    assert abs(sq.item() / ref.pow(2).sum().item() - 1.0) < 2 * lim + 2.0**-16
    assert off(low, ref + res.double()) < 2.0**-8
    assert torch.equal(f32, again)  # the order of the sums does not depend on which range comes last


@pytest.mark.parametrize("rows", [[512, 256, 256], [128, 64], [64, 64, 72], [192, 320, 256, 8]])
@pytest.mark.parametrize("tile,splits", [(0, 0), (3, 1), (4, 2)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_gemm_weight_in_pieces(rows, tile, splits, b_mn):
    """A weight in several pieces of memory gives what the concatenated one gives, bit for bit (same tiles, same order)."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(8)
    cols, m = 328, 200
    parts = [torch.randn(r, cols, device="cuda").bfloat16() for r in rows]
    whole = torch.cat(parts)
    tile = 4 if not b_mn else tile  # the tile that every start of a piece is a multiple of
    a = torch.randn(m, sum(rows) if b_mn else cols, device="cuda").bfloat16()
    got = kernels.gemm_parts(a, parts, b_mn_major=b_mn, tile=tile, splits=splits)
    want = kernels.gemm(a, whole, b_mn_major=b_mn, tile=tile, splits=splits)
    torch.cuda.synchronize()
    kernels.check_status()
    assert torch.equal(got, want)


@pytest.mark.parametrize("t,f,k", [(1, 128, 64), (200, 384, 136), (300, 1408, 512), (777, 256, 1032), (2048, 1408, 512)])
@pytest.mark.parametrize("keep", [True, False])
def test_gemm_swiglu_epilogue(t, f, k, keep):
    """Gate, up and their activation from one kernel, against the separate kernels (same rounding points) and fp64 (results
    rounded to bf16: 2^-8)."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(9)
    x = torch.randn(t, k, device="cuda").bfloat16()
    wg, wu = (torch.randn(f, k, device="cuda").bfloat16() * k**-0.5 for _ in range(2))
    gu, a = kernels.gemm_swiglu(x, wg, wu, keep_gu=keep)
    want_gu = torch.cat([x.double() @ wg.double().t(), x.double() @ wu.double().t()], dim=1)
    if keep:
        assert ((gu.double() - want_gu).norm() / want_gu.norm()).item() < 2.0**-8
        assert torch.equal(a, kernels.swiglu_fwd(gu))
    else:
        assert gu is None
        gu = torch.cat([kernels.gemm(x, wg), kernels.gemm(x, wu)], dim=1)
        want = kernels.swiglu_fwd(gu).double()
        assert ((a.double() - want).norm() / want.norm()).item() < 2.0**-8
    torch.cuda.synchronize()
    kernels.check_status()


def test_gemm_alpha_from_device():
    from yafsdp_b200.ops import kernels

    torch.manual_seed(10)
    a, b = torch.randn(300, 1032, device="cuda").bfloat16(), torch.randn(520, 1032, device="cuda").bfloat16()
    alpha = torch.tensor(0.37, device="cuda")
    for splits in (1, 3):
        got = kernels.gemm(a, b, out_dtype=torch.float32, alpha=2.0, alpha_tensor=alpha, tile=3, splits=splits)
        want = kernels.gemm(a, b, out_dtype=torch.float32, tile=3, splits=splits) * (2.0 * alpha)
        assert torch.allclose(got, want, rtol=2.0**-22, atol=0.0)


@pytest.mark.parametrize("m", [1, 16, 45, 208, 250, 257, 333, 777, 1337])
@pytest.mark.parametrize("n,k", [(8, 72), (256, 1032), (1000, 264), (2056, 512)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_gemm_swapped_form(m, n, k, b_mn):
    """Tokens as the narrow operand: every width of a tile, ragged edges on both sides, residual and alpha (bf16 results: 2^-8),
    and the weight in pieces."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(13)
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = torch.randn((k, n) if b_mn else (n, k), device="cuda").bfloat16()
    res = torch.randn(m, n, device="cuda").bfloat16()
    big = torch.full((m + 2, n + 8), 7.0, device="cuda").bfloat16()
    ref = a.double() @ (b.double() if b_mn else b.double().t())
    got = kernels.gemm(a, b, b_mn_major=b_mn, tile=6, out=big[1 : m + 1, :n])
    with_res = kernels.gemm(a, b, b_mn_major=b_mn, tile=6, residual=res, alpha=0.5)
    if b_mn:
        parts = [b[: k // 128 * 64], b[k // 128 * 64 :]] if k >= 128 else None
    else:
        parts = [b[:256], b[256:]] if n > 256 else None
    torch.cuda.synchronize()
    kernels.check_status()
    assert ((got.double() - ref).norm() / ref.norm()).item() < 2.0**-8
    assert (big[0] == 7).all() and (big[m + 1] == 7).all() and (big[1 : m + 1, n:] == 7).all()
    want = 0.5 * ref + res.double()
    assert ((with_res.double() - want).norm() / want.norm()).item() < 2.0**-8
    if parts is not None:
        assert torch.equal(kernels.gemm_parts(a, parts, b_mn_major=b_mn, tile=6), got)


@pytest.mark.parametrize("tile,splits", [(0, 0), (0, 3), (3, 3), (1, 2)])
@pytest.mark.parametrize("given", ["none", "short", "unaligned"])
def test_gemm_without_a_usable_workspace(tile, splits, given):
    """No workspace, one that is too short or one at an odd address: no tile is split, whether or not a split was asked for."""
    from yafsdp_b200 import _native
    from yafsdp_b200.ops import kernels

    torch.manual_seed(17)
    m, n, k = 300, 520, 4096
    a, b = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    out = torch.empty(m, n, device="cuda")
    ws = torch.empty(1 << 24, device="cuda", dtype=torch.uint8)
    at, nbytes = {"none": (None, 0), "short": (ws.data_ptr(), 256), "unaligned": (ws.data_ptr() + 128, (1 << 24) - 128)}[given]
    rc = _native.lib().yf_gemm_bf16_ws(a.data_ptr(), b.data_ptr(), out.data_ptr(), None, m, n, k, k, k, n, 0, 0, 0, 1, 0, 1.0, 0, None, None,
                                       at, nbytes, tile, splits, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    want = kernels.gemm(a, b, out_dtype=torch.float32, tile=tile, splits=1)
    torch.cuda.synchronize()
    kernels.check_status()
    # the same plan as for a caller that asks for whole tiles
    assert torch.equal(out, want)


@pytest.mark.parametrize("m,n,k,f32,split", [(45, 4096, 4096, False, False), (1337, 4096, 11008, False, False), (1337, 4096, 11008, True, True),
                                             (999, 5120, 13824, True, True), (333, 5120, 13824, False, False), (2048, 2816, 512, False, False)])
def test_gemm_plans_chosen_from_the_shape(m, n, k, f32, split):
    """Nothing forced: few tokens (narrow tiles), ragged ones (swapped), a last wave in K ranges, whole pair tiles; against fp64.
    fp32 sums of k products: a few sqrt(k) * 2^-24; a bf16 result: 2^-8."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(19)
    a, b = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    assert (kernels._gemm_workspace(m, n, k, int(f32), 0, 0, 0, 0, 0) > 0) == split
    got = kernels.gemm(a, b, out_dtype=torch.float32 if f32 else torch.bfloat16)
    again = kernels.gemm(a, b, out_dtype=got.dtype)
    ref = a.double() @ b.double().t()
    torch.cuda.synchronize()
    kernels.check_status()
    assert ((got.double() - ref).norm() / ref.norm()).item() < (3.0 * k**0.5 * 2.0**-24 if f32 else 2.0**-8)
    assert torch.equal(got, again)


@pytest.mark.parametrize("rows", [[512, 256, 256], [256, 768, 24]])
@pytest.mark.parametrize("tile,splits", [(1, 1), (5, 1), (2, 1), (1, 2)])
def test_gemm_weight_in_pieces_wide_tiles(rows, tile, splits):
    """Pieces of an [N, K] weight that start where pair tiles do: every CTA of a pair reads its half from the right piece."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(20)
    cols, m = 1032, 600
    parts = [torch.randn(r, cols, device="cuda").bfloat16() for r in rows]
    a = torch.randn(m, cols, device="cuda").bfloat16()
    got = kernels.gemm_parts(a, parts, tile=tile, splits=splits)
    want = kernels.gemm(a, torch.cat(parts), tile=tile, splits=splits)
    torch.cuda.synchronize()
    kernels.check_status()
    assert torch.equal(got, want)


def test_entries_without_scratch():
    """The C entries that Python does not call, against the general forms: plain GEMMs without a workspace, RMSNorm backward with atomic
    weight sums, embedding backward without a norm, attention backward without parts."""
    from yafsdp_b200 import _native
    from yafsdp_b200.ops import kernels

    torch.manual_seed(21)
    lib, st = _native.lib(), torch.cuda.current_stream().cuda_stream
    m, n, k = 333, 520, 1032
    a, b = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    r = torch.randn(m, n, device="cuda").bfloat16()
    low, f32, sq, res = torch.empty_like(r), torch.empty(m, n, device="cuda"), torch.zeros(1, device="cuda"), torch.empty_like(r)
    p = [t.data_ptr() for t in (a, b)]
    assert lib.yf_gemm_bf16(*p, low.data_ptr(), m, n, k, k, k, n, 0, 0, 0, 0, 0.5, 0, st) == 0
    assert lib.yf_gemm_bf16_sumsq(*p, f32.data_ptr(), m, n, k, k, k, n, 0, 0, 1, 0, 1.0, 0, sq.data_ptr(), st) == 0
    assert lib.yf_gemm_bf16_residual(*p, res.data_ptr(), r.data_ptr(), m, n, k, k, k, n, n, 0, 0, 1.0, 0, st) == 0
    # whole tiles of every shape add the products in the same order
    assert torch.equal(low, kernels.gemm(a, b, alpha=0.5, splits=1)) and torch.equal(f32, kernels.gemm(a, b, out_dtype=torch.float32, splits=1))
    assert torch.equal(res, kernels.gemm(a, b, residual=r, splits=1))
    assert abs(sq.item() / f32.double().pow(2).sum().item() - 1.0) < 2.0**-14  # fp32 sums over a thread's rows, then atomics

    t, d = 700, 1032
    x, dy = (torch.randn(t, d, device="cuda").bfloat16() for _ in range(2))
    w = torch.ones(d, device="cuda").bfloat16()
    _, rstd = kernels.rmsnorm_fwd(x, w, 1e-5)
    for zero in (1, 0):
        dw, want = torch.full((d,), 2.0, device="cuda"), torch.full((d,), 2.0, device="cuda")
        dx = torch.empty_like(x)
        assert lib.yf_rmsnorm_bwd(x.data_ptr(), w.data_ptr(), dy.data_ptr(), rstd.data_ptr(), None, dx.data_ptr(), dw.data_ptr(), zero, t, d, st) == 0
        assert torch.equal(dx, kernels.rmsnorm_bwd(x, w, dy, rstd, want, zero_dw=bool(zero)))
        assert torch.allclose(dw, want, rtol=1e-5, atol=t**0.5 * 1e-5)  # fp32 sums of t terms of about one in two orders

    ids = torch.randint(0, 40, (t,), device="cuda")
    table, want = torch.zeros(40, d, device="cuda"), torch.zeros(40, d, device="cuda")
    assert lib.yf_embedding_bwd(dy.data_ptr(), ids.data_ptr(), table.data_ptr(), t, d, 40, st) == 0
    kernels.embedding_bwd_(dy, ids, want)
    assert torch.allclose(table, want, rtol=1e-5, atol=1e-4)  # some twenty fp32 additions in any order

    bsz, s, hq, hkv = 1, 200, 4, 2
    qkv = torch.randn(s, (hq + 2 * hkv) * 128, device="cuda").bfloat16()
    q, kk, v = qkv[:, : hq * 128], qkv[:, hq * 128 : (hq + hkv) * 128], qkv[:, (hq + hkv) * 128 :]
    out, lse = kernels.attn_fwd(q, kk, v, bsz, s, hq, hkv, 0.09, True)
    dout = torch.randn_like(out)
    got, want = torch.empty_like(qkv), torch.empty_like(qkv)
    delta, acc = torch.empty(hq * s, device="cuda"), torch.empty(s * hq * 128, device="cuda")
    ld = qkv.stride(0)

    def views(g):
        return g[:, : hq * 128], g[:, hq * 128 : (hq + hkv) * 128], g[:, (hq + hkv) * 128 :]

    assert lib.yf_attn_bwd(*[x.data_ptr() for x in (q, kk, v, out, dout, lse, delta, acc, *views(got))], bsz, s, hq, hkv, ld, ld, out.stride(0),
                           dout.stride(0), ld, ld, 0.09, 1, st) == 0
    kernels.attn_bwd(q, kk, v, out, dout, lse, *views(want), bsz, s, hq, hkv, 0.09, True, head_parts=1)
    torch.cuda.synchronize()
    kernels.check_status()
    assert torch.equal(got[:, hq * 128 :], want[:, hq * 128 :])
    assert torch.allclose(got.float(), want.float(), rtol=2.0**-7, atol=1e-5)  # dq: fp32 sums in any order, one bf16 rounding
