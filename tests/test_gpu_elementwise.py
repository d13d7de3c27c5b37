"""Memory-bound sm_100a kernels vs fp32 PyTorch restatements."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(a, b, rtol=2e-2, atol=2e-2):
    assert torch.allclose(a.float(), b.float(), rtol=rtol, atol=atol), (a.float() - b.float()).abs().max().item()


@pytest.mark.parametrize("t,d", [(64, 256), (300, 4096), (17, 8192), (33, 1000 * 8), (2049, 2048), (130, 5120), (5, 2056)])
def test_rmsnorm_fwd_bwd(t, d):
    from yafsdp_b200.ops import kernels

    torch.manual_seed(0)
    x = torch.randn(t, d, device="cuda", dtype=torch.bfloat16)
    w = (1 + 0.1 * torch.randn(d, device="cuda")).bfloat16()
    dy = torch.randn(t, d, device="cuda", dtype=torch.bfloat16)
    y, rstd = kernels.rmsnorm_fwd(x, w, 1e-5)
    xf = x.float().requires_grad_(True)
    wf = w.float().requires_grad_(True)
    yr = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
    _close(y, yr)
    yr.backward(dy.float())
    dw = torch.zeros(d, device="cuda", dtype=torch.float32)
    dres = torch.randn(t, d, device="cuda", dtype=torch.bfloat16)
    dx = kernels.rmsnorm_bwd(x, w, dy, rstd, dw, dres)
    _close(dx, xf.grad + dres.float(), rtol=3e-2, atol=3e-2)
    assert torch.allclose(dw, wf.grad, rtol=2e-2, atol=5e-2 * math.sqrt(t))
    # without the residual gradient, and with the weight gradient cleared by the kernel itself
    dw2 = torch.full((d,), 7.0, device="cuda", dtype=torch.float32)
    dx2 = kernels.rmsnorm_bwd(x, w, dy, rstd, dw2, zero_dw=True)
    _close(dx2, xf.grad, rtol=3e-2, atol=3e-2)
    assert torch.allclose(dw2, wf.grad, rtol=2e-2, atol=5e-2 * math.sqrt(t))


def test_rope_roundtrip_and_reference():
    from yafsdp_b200.ops import kernels
    from yafsdp_b200.ops.functional import rope_table

    torch.manual_seed(0)
    seq, b, h, hd = 128, 2, 4, 128
    t = seq * b
    qkv = torch.randn(t, 3 * h * hd, device="cuda", dtype=torch.bfloat16)
    orig = qkv.clone()
    cs = rope_table(seq, hd, 10000.0, qkv.device)
    kernels.rope_(qkv, cs, seq, 0, h, hd)
    q = orig[:, : h * hd].float().view(b, seq, h, hd)
    cos = cs[..., 0].view(1, seq, 1, hd // 2)
    sin = cs[..., 1].view(1, seq, 1, hd // 2)
    q1, q2 = q[..., : hd // 2], q[..., hd // 2 :]
    ref = torch.cat([q1 * cos - q2 * sin, q2 * cos + q1 * sin], -1).view(t, h * hd)
    _close(qkv[:, : h * hd], ref)
    assert torch.equal(qkv[:, h * hd :], orig[:, h * hd :])
    kernels.rope_(qkv, cs, seq, 0, h, hd, backward=True)
    _close(qkv, orig, rtol=3e-2, atol=3e-2)


def test_swiglu():
    from yafsdp_b200.ops import kernels

    torch.manual_seed(0)
    t, f = 130, 688
    gu = torch.randn(t, 2 * f, device="cuda", dtype=torch.bfloat16)
    dh = torch.randn(t, f, device="cuda", dtype=torch.bfloat16)
    h = kernels.swiglu_fwd(gu)
    guf = gu.float().requires_grad_(True)
    ref = torch.nn.functional.silu(guf[:, :f]) * guf[:, f:]
    _close(h, ref)
    ref.backward(dh.float())
    dgu = kernels.swiglu_bwd(gu, dh)
    _close(dgu, guf.grad, rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("v", [1024, 32000, 1003])
def test_cross_entropy(v):
    from yafsdp_b200.ops import kernels

    torch.manual_seed(0)
    t = 96
    vp = (v + 7) // 8 * 8
    buf = torch.randn(t, vp, device="cuda", dtype=torch.bfloat16) * 3
    logits = buf[:, :v]
    labels = torch.randint(0, v, (t,), device="cuda")
    labels[5] = -100
    lf = logits.float().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(lf, labels, ignore_index=-100, reduction="sum")
    ref.backward()
    loss_rows = kernels.cross_entropy_(logits, labels, 1.0)
    assert abs(loss_rows.sum().item() - ref.item()) <= 2e-3 * abs(ref.item()) + 1e-2
    assert torch.allclose(logits.float(), lf.grad, rtol=2e-2, atol=4e-3)
    # the gradient scale as host value x device scalar (what the mean over valid labels uses)
    buf2 = torch.zeros_like(buf)
    logits2 = buf2[:, :v]
    logits2.copy_(lf.detach())
    dev_scale = torch.tensor([0.25], device="cuda")
    kernels.cross_entropy_(logits2, labels, 0.5, scale=dev_scale)
    assert torch.allclose(logits2.float(), lf.grad * 0.125, rtol=2e-2, atol=1e-3)


def test_embedding():
    from yafsdp_b200.ops import kernels

    torch.manual_seed(0)
    v, d, t = 500, 256, 777
    table = torch.randn(v, d, device="cuda", dtype=torch.bfloat16)
    ids = torch.randint(0, v, (t,), device="cuda")
    out = kernels.embedding_fwd(table, ids)
    assert torch.equal(out, table[ids])
    dout = torch.randn(t, d, device="cuda", dtype=torch.bfloat16)
    dt = torch.zeros(v, d, device="cuda", dtype=torch.float32)
    kernels.embedding_bwd_(dout, ids, dt)
    ref = torch.zeros_like(dt).index_add_(0, ids, dout.float())
    assert torch.allclose(dt, ref, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("n", [1024, 1000003])
def test_adamw_matches_torch(n):
    from yafsdp_b200.ops import kernels

    torch.manual_seed(0)
    p = torch.randn(n, device="cuda")
    ref_p = torch.nn.Parameter(p.clone())
    opt = torch.optim.AdamW([ref_p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    m = torch.zeros_like(p)
    v = torch.zeros_like(p)
    pb = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    for step in range(1, 4):
        g = torch.randn(n, device="cuda")
        ref_p.grad = g.clone()
        opt.step()
        kernels.adamw_(p, g, m, v, pb, None, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step)
    assert torch.allclose(p, ref_p.detach(), rtol=1e-5, atol=1e-6)
    assert torch.equal(pb, p.bfloat16())


def test_sumsq_clip_and_casts():
    from yafsdp_b200.ops import kernels

    torch.manual_seed(0)
    g = torch.randn(3 * 1000 * 1000 + 3, device="cuda")
    acc = torch.zeros(1, device="cuda")
    kernels.sumsq_(g, acc)
    assert abs(acc.item() - g.double().pow(2).sum().item()) <= 1e-4 * acc.item()
    coef = torch.empty(1, device="cuda")
    nrm = torch.empty(1, device="cuda")
    kernels.clip_coef_(acc, 1.0, coef, nrm)
    assert abs(nrm.item() - math.sqrt(acc.item())) < 1e-2 and abs(coef.item() - 1.0 / nrm.item()) < 1e-5
    dst = torch.empty(g.numel(), device="cuda", dtype=torch.bfloat16)
    kernels.cast_f32_to_bf16_(g, dst)
    assert torch.equal(dst, g.bfloat16())
    back = torch.ones_like(g)
    kernels.accum_bf16_to_f32_(dst, back, scale=0.5, accumulate=True)
    assert torch.allclose(back, 1 + 0.5 * dst.float())
    s = kernels.add_bf16(dst, dst)
    assert torch.equal(s, (dst.float() * 2).bfloat16())


@pytest.mark.parametrize("n,off", [(1, 0), (2, 3), (7, 1), (4096, 0), (100003, 2), (3_000_001, 1)])
def test_sumsq_and_scale_of_flat_runs(n, off):
    """Runs that start anywhere in a flat buffer: neighbours stay untouched; a coefficient of one changes nothing, NaN spreads."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(3)
    flat = torch.randn(n + off + 5, device="cuda")
    run = flat[off : off + n]
    want = flat.clone()
    other = torch.randn(77, device="cuda")[1:]
    got = kernels.sumsq_runs([run, other])
    ref = run.double().pow(2).sum() + other.double().pow(2).sum()
    assert abs(got.item() / ref.item() - 1.0) < 1e-6  # fp32 partial sums of at most a few hundred terms each
    assert torch.equal(got, kernels.sumsq_runs([run, other]))
    kernels.scale_(run, torch.ones(1, device="cuda"))
    assert torch.equal(flat, want)
    kernels.scale_(run, torch.full((1,), 0.37, device="cuda"))
    want[off : off + n] *= torch.full((1,), 0.37, device="cuda")
    assert torch.equal(flat, want)
    kernels.scale_(run, torch.full((1,), float("nan"), device="cuda"))
    assert run.isnan().all() and not flat[off + n :].isnan().any() and not flat[:off].isnan().any()


@pytest.mark.parametrize("max_norm", [1e-3, 1e9])
def test_clip_grad_norm_of_adjacent_sharded_gradients(max_norm):
    """Parameters of odd sizes behind each other in a group's flat gradient, against the norm and scale of each one."""
    import torch.distributed as dist

    from yafsdp_b200 import fully_shard
    from yafsdp_b200.optim import clip_grad_norm_

    torch.cuda.set_device(0)
    created = not dist.is_initialized()
    if created:
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    try:
        torch.manual_seed(4)
        model = torch.nn.Sequential(torch.nn.Linear(33, 7, device="cuda"), torch.nn.Linear(7, 5, device="cuda"))
        fully_shard(model[0])
        fully_shard(model)
        model(torch.randn(9, 33, device="cuda")).square().sum().backward()
        grads = [p.grad._local_tensor for p in model.parameters()]
        before = [g.clone() for g in grads]
        norm = torch.stack([g.double().norm() for g in before]).norm()
        got = clip_grad_norm_(model, max_norm)
        assert abs(got.item() / norm.item() - 1.0) < 1e-6
        coef = min(1.0, max_norm / (norm.item() + 1e-6))
        for g, b in zip(grads, before):
            assert torch.allclose(g, b * coef, rtol=1e-6, atol=0.0)
    finally:
        if created:
            dist.destroy_process_group()


@pytest.mark.parametrize("max_norm", [1e-3, 1e9])
@pytest.mark.parametrize("form", ["float64", "float64 on the CPU", "float64 vector", "float16 on the CPU", "int64"])
def test_clip_grad_norm_with_a_tensor_as_limit(max_norm, form):
    """``max_norm`` as a tensor of another type than the gradients, below and above their norm: what multiplying each gradient
    by the coefficient gives."""
    import torch.distributed as dist

    from yafsdp_b200 import fully_shard
    from yafsdp_b200.optim import clip_grad_norm_

    dtype = getattr(torch, form.split()[0])
    if dtype in (torch.float16, torch.int64):
        max_norm = min(max(max_norm, 2.0 if dtype == torch.int64 else 0.0), 1000.0)
    limit = torch.tensor([max_norm] if "vector" in form else max_norm, dtype=dtype, device="cpu" if "CPU" in form else "cuda")
    torch.cuda.set_device(0)
    created = not dist.is_initialized()
    if created:
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    try:
        torch.manual_seed(4)
        model = torch.nn.Sequential(torch.nn.Linear(33, 7, device="cuda"), torch.nn.Linear(7, 5, device="cuda"))
        fully_shard(model)
        model(torch.randn(9, 33, device="cuda")).square().sum().backward()
        grads = [p.grad._local_tensor for p in model.parameters()]
        before = [g.clone() for g in grads]
        got = clip_grad_norm_(model, limit)
        coef = torch.clamp(limit / (got + 1e-6), max=1.0)
        for g, b in zip(grads, before):
            assert torch.equal(g, b.clone().mul_(coef))
    finally:
        if created:
            dist.destroy_process_group()


def test_in_place_writes_of_gradients_move_their_version():
    """What the kernels change in place counts as changed for autograd: gradients that a backward pass adds to, and clipped ones."""
    import torch.distributed as dist

    from yafsdp_b200 import MixedPrecisionPolicy, fully_shard
    from yafsdp_b200.optim import clip_grad_norm_

    torch.cuda.set_device(0)
    created = not dist.is_initialized()
    if created:
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    try:
        model = torch.nn.Sequential(torch.nn.Linear(64, 64, device="cuda"), torch.nn.Linear(64, 8, device="cuda"))
        fully_shard(model, mp_policy=MixedPrecisionPolicy(param_dtype=torch.bfloat16, reduce_dtype=torch.float32))
        x = torch.randn(16, 64, device="cuda").bfloat16()
        model(x).square().sum().backward()
        grads = [p.grad._local_tensor for p in model.parameters()]
        before = [g._version for g in grads]
        values = [g.clone() for g in grads]
        model(x).square().sum().backward()  # added to the gradients that are there
        assert all(p.grad._local_tensor is g or p.grad._local_tensor.data_ptr() == g.data_ptr() for p, g in zip(model.parameters(), grads))
        assert all(torch.allclose(g, 2 * v) for g, v in zip(grads, values))
        added = [g._version for g in grads]
        assert all(a > b for a, b in zip(added, before))
        grads = [p.grad._local_tensor for p in model.parameters()]
        added = [g._version for g in grads]
        clip_grad_norm_(model, 1e-3)
        assert all(g._version > a for g, a in zip(grads, added))
    finally:
        if created:
            dist.destroy_process_group()


@pytest.mark.parametrize("t,d", [(1, 8), (7, 1024), (700, 1032), (601, 2048), (1200, 4096), (297, 4104), (599, 8192)])
def test_rmsnorm_bwd_weight_gradient_over_many_rows(t, d):
    """Every width class of the row walk, more rows than a wave holds: the weight gradient in a fixed order, cleared or added to,
    against fp64 sums (fp32 sums of t terms)."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(6)
    x, dy = (torch.randn(t, d, device="cuda").bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(d, device="cuda")).bfloat16()
    _, rstd = kernels.rmsnorm_fwd(x, w, 1e-5)
    want = (dy.double() * x.double() * rstd.double()[:, None]).sum(0)
    got = torch.full((d,), 3.0, device="cuda")
    dx = kernels.rmsnorm_bwd(x, w, dy, rstd, got, zero_dw=True)
    again = torch.empty_like(got)
    dx2 = kernels.rmsnorm_bwd(x, w, dy, rstd, again, zero_dw=True)
    assert torch.equal(got, again) and torch.equal(dx, dx2)
    lim = 4.0 * t**0.5 * 2.0**-24 * (dy.double() * x.double() * rstd.double()[:, None]).abs().sum(0).max().item() + 1e-7
    assert (got.double() - want).abs().max().item() < lim
    kernels.rmsnorm_bwd(x, w, dy, rstd, again)
    assert (again.double() - 2 * want).abs().max().item() < 2 * lim


@pytest.mark.parametrize("v", [8, 1024, 32000, 32768, 32776, 1001, 128256])
@pytest.mark.parametrize("t", [3, 700])
def test_cross_entropy_row_lengths(v, t):
    """Short, long and odd rows; ignored labels; logits at -inf."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(11)
    pitch = (v + 7) // 8 * 8
    logits = (3 * torch.randn(t, pitch, device="cuda")).bfloat16()[:, :v]
    labels = torch.randint(0, v, (t,), device="cuda")
    labels[1] = -100
    if v > 8:
        logits[0, 1:5] = -math.inf
        labels[0] = 0
    ref = logits.double().requires_grad_(True)
    rows = torch.nn.functional.cross_entropy(ref, labels, ignore_index=-100, reduction="none")
    (rows.sum() * 0.25).backward()
    work = torch.empty(t, pitch, device="cuda", dtype=torch.bfloat16)[:, :v]
    work.copy_(logits)
    got = kernels.cross_entropy_(work, labels, 0.25)
    assert torch.allclose(got.double(), rows, rtol=1e-5, atol=1e-5)  # fast exponentials of up to 2^17 terms in fp32
    assert torch.allclose(work.double(), ref.grad, rtol=2.0**-7, atol=1e-6)


def test_loss_scalars_and_embedding_norm():
    from yafsdp_b200.ops import kernels

    torch.manual_seed(12)
    labels = torch.randint(-100, 50, (5003,), device="cuda")
    inv = kernels.inv_valid_labels(labels)
    assert abs(inv.item() * max(1, int((labels >= 0).sum())) - 1.0) < 1e-6
    assert kernels.inv_valid_labels(torch.full((7,), -100, device="cuda")).item() == 1.0
    x = torch.rand(5003, device="cuda")
    assert abs(kernels.scaled_sum(x, inv).item() / (x.double().sum() * inv.double()).item() - 1.0) < 1e-6
    for off in (0, 1):  # a table gradient that starts anywhere in a flat buffer
        flat = torch.zeros(off + 300 * 264, device="cuda")
        table = flat[off:].view(300, 264)
        ids = torch.randint(0, 300, (900,), device="cuda")
        ids[:200] = 17
        dout = torch.randn(900, 264, device="cuda").bfloat16()
        sq = torch.zeros(1, device="cuda")
        kernels.embedding_bwd_(dout, ids, table, sq)
        want = torch.zeros(300, 264, device="cuda", dtype=torch.float64).index_add_(0, ids, dout.double())
        assert torch.allclose(table.double(), want, rtol=1e-4, atol=1e-4)  # up to 200 fp32 additions in any order
        assert abs(sq.item() / table.double().pow(2).sum().item() - 1.0) < 1e-5


@pytest.mark.parametrize("accumulate", [False, True])
def test_accumulate_many_bf16_tensors(accumulate):
    """Tensors of odd sizes at odd places of one flat buffer, more of them than fit a launch, some empty."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(14)
    sizes = [1, 0, 7, 8, 16384, 16385, 40000, 3] * 8
    flat = torch.randn(sum(sizes) + 1, device="cuda")
    want, pairs, at = flat.clone(), [], 1
    for n in sizes:
        src = torch.randn(n, device="cuda").bfloat16()
        pairs.append((flat[at : at + n], src))
        want[at : at + n] = want[at : at + n] + src.float() if accumulate else src.float()
        at += n
    kernels.accum_bf16_to_f32_multi_(pairs, accumulate)
    assert torch.equal(flat, want)


def test_shift_labels_and_rmsnorm_weight_norm():
    from yafsdp_b200.ops import kernels

    labels = torch.arange(30, device="cuda").view(3, 10)
    for x in (labels, labels[:, 2:7], labels[:, :1]):
        want = torch.cat([x[:, 1:], x.new_full((3, 1), -100)], dim=1)
        assert torch.equal(kernels.shift_labels(x), want)
    torch.manual_seed(15)
    x, dy = (torch.randn(50, 1032, device="cuda").bfloat16() for _ in range(2))
    w = torch.ones(1032, device="cuda").bfloat16()
    _, rstd = kernels.rmsnorm_fwd(x, w, 1e-5)
    dw, sq = torch.randn(1032, device="cuda"), torch.full((1,), 2.0, device="cuda")
    kernels.rmsnorm_bwd(x, w, dy, rstd, dw, zero_dw=True, sumsq=sq)
    assert abs((sq.item() - 2.0) / dw.double().pow(2).sum().item() - 1.0) < 1e-5


@pytest.mark.parametrize("v", [1024, 32000, 50257, 128256])
def test_cross_entropy_extreme_logits(v):
    """Masks of the type's lowest value and of -inf over whole batches of loads, sure predictions, the smallest probabilities."""
    from yafsdp_b200.ops import kernels

    torch.manual_seed(13)
    pitch = (v + 7) // 8 * 8
    logits = torch.randn(5, pitch, device="cuda").bfloat16()[:, :v]
    lowest = torch.finfo(torch.bfloat16).min
    logits[0] = lowest
    logits[1, : v - 100] = lowest
    logits[2, : v - 100] = -math.inf
    logits[3] -= 84.0
    logits[3, 7] = 5.0
    logits[4, v - 1] = 25.0
    labels = torch.tensor([3, v - 5, v - 1, 7, v - 1], device="cuda")
    ref = logits.double().requires_grad_(True)
    rows = torch.nn.functional.cross_entropy(ref, labels, reduction="none")
    rows.sum().backward()
    work = torch.empty(5, pitch, device="cuda", dtype=torch.bfloat16)[:, :v]
    work.copy_(logits)
    got = kernels.cross_entropy_(work, labels, 1.0)
    # the sum's fp32 rounding, relative to logsumexp <= 25 and to the loss
    assert torch.allclose(got.double(), rows, rtol=1e-5, atol=1e-5)
    grad, want = work.double(), ref.grad
    rest = torch.ones(5, v, dtype=torch.bool, device="cuda")
    rest[torch.arange(5), labels] = False
    # probabilities: bf16's 2^-9 and the exponentials' error; 2^-133 is the smallest bf16 (half of it for rounding)
    assert torch.allclose(grad[rest], want[rest], rtol=2.0**-8, atol=2.0**-133)
    assert torch.allclose(grad[~rest], want[~rest], rtol=2.0**-8, atol=4e-6)  # p - 1: p to fp32's precision of logsumexp
