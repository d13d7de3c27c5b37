"""Thin tensor-level wrappers over the native sm_100a kernels (``csrc/*.cu``).

Each function checks its arguments on the host, launches on the current CUDA stream and raises on a
non-zero return code.  ``launch_count()`` counts every launch made through this module (the
benchmark reports it).  Nothing here falls back to PyTorch: a missing library on a GPU machine is an
error, and the autograd-level ops in :mod:`yafsdp_b200.ops.functional` choose between this module
(CUDA tensors) and plain PyTorch math (CPU tensors).
"""

from __future__ import annotations

import ctypes
import functools
import math
from typing import Any

import torch

from .. import _native

_launches = 0


def launch_count() -> int:
    return _launches


def reset_launch_count() -> None:
    global _launches
    _launches = 0


def _stream() -> int:
    # torch.cuda.current_stream() without the Stream object around it (some 5 us a call)
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())  # type: ignore[no-any-return]


def _check(rc: int, name: str) -> None:
    global _launches
    if rc != 0:
        raise RuntimeError(f"{name} failed with code {rc}")
    _launches += 1


def _ptr(t: torch.Tensor | None) -> int | None:
    return None if t is None else t.data_ptr()


def status(clear: bool = True) -> tuple[int, int]:
    """(code, site) of the first error any kernel recorded since the last clearing read.  The status word sits in host
    memory: this is a plain read that neither synchronises nor touches the GPU; synchronise first to cover kernels that
    are still running."""
    code = ctypes.c_int(0)
    site = ctypes.c_int(0)
    rc = _native.lib().yf_status_read(ctypes.byref(code), ctypes.byref(site), int(clear))
    if rc != 0:
        raise RuntimeError(f"yf_status_read failed with code {rc}")
    return code.value, site.value


def check_status() -> None:
    code, site = status()
    if code != 0:
        raise RuntimeError(f"a native kernel reported error {code} at site {site} (a bounded wait ran out: a peer rank is late or "
                           "gone); the results of the kernels that ran since are undefined")


def poll_status() -> None:
    """:func:`check_status` when the native library is loaded in this process, nothing otherwise (CPU runs).  Cheap enough
    for once per step: the framework calls it at every root pre-forward and in the fused optimizer step."""
    if _native.loaded():
        check_status()


# --------------------------------------------------------------------------------------- GEMM
def gemm(
    a: torch.Tensor,
    b: torch.Tensor,
    *,
    a_mn_major: bool = False,
    b_mn_major: bool = False,
    out: torch.Tensor | None = None,
    out_dtype: torch.dtype = torch.bfloat16,
    accumulate: bool = False,
    alpha: float = 1.0,
    sm_limit: int = 0,
    sumsq: torch.Tensor | None = None,
    residual: torch.Tensor | None = None,
    tile: int = 0,
    splits: int = 0,
    alpha_tensor: torch.Tensor | None = None,
) -> torch.Tensor:
    """``out[M,N] = alpha * A @ B^T (+ out)`` with bf16 inputs and fp32 accumulation (tcgen05).

    ``a`` is ``[M,K]`` (K-major) or, with ``a_mn_major``, the stored tensor is ``[K,M]``; ``b`` is
    ``[N,K]`` or, with ``b_mn_major``, stored ``[K,N]``.  Rows must be contiguous (stride 1 in the last
    dimension); the row pitch may exceed the row length.  ``sumsq`` (fp32 output without accumulation only): a
    one-element fp32 tensor that receives ``+= sum(out**2)`` from the same kernel.  ``residual`` (bf16 output without
    accumulation only): a bf16 ``[M,N]`` tensor added in fp32 inside the epilogue, before the output is rounded.
    ``tile`` (1-6) and ``splits`` (1-4): tile shape and K ranges of the last wave's tiles; 0 chooses them from the shape.
    ``alpha_tensor``: one fp32 value on the device that ``alpha`` is multiplied by (read by the kernel).
    """
    assert a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and a.is_cuda and b.is_cuda
    assert a.dim() == 2 and b.dim() == 2 and a.stride(1) == 1 and b.stride(1) == 1
    if a_mn_major:
        k, m = a.shape
    else:
        m, k = a.shape
    if b_mn_major:
        kb, n = b.shape
    else:
        n, kb = b.shape
    assert k == kb, f"inner dimensions differ: {k} vs {kb}"
    if out is None:
        assert not accumulate
        out = torch.empty((m, n), device=a.device, dtype=out_dtype)
    assert out.shape == (m, n) and out.stride(1) == 1 and out.dtype in (torch.bfloat16, torch.float32)
    if residual is not None:
        assert out.dtype == torch.bfloat16 and not accumulate and sumsq is None
        assert residual.dtype == torch.bfloat16 and residual.shape == (m, n) and residual.stride(1) == 1
    assert alpha_tensor is None or (alpha_tensor.dtype == torch.float32 and alpha_tensor.numel() == 1 and alpha_tensor.device == a.device)
    kind = 1 if out.dtype == torch.float32 else (2 if a_mn_major or accumulate else 0)
    nbytes = _gemm_workspace(m, n, k, kind, 0, sm_limit, tile, splits, a.device.index)
    ws = torch.empty(nbytes, device=a.device, dtype=torch.uint8) if nbytes else None
    rc = _native.lib().yf_gemm_bf16_ws(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), _ptr(residual), m, n, k, a.stride(0), b.stride(0), out.stride(0),
        0 if residual is None else residual.stride(0), int(a_mn_major), int(b_mn_major), int(out.dtype == torch.float32),
        int(accumulate), float(alpha), int(sm_limit), _ptr(alpha_tensor), _ptr(sumsq), _ptr(ws), nbytes, tile, splits, _stream(),
    )
    _check(rc, "yf_gemm_bf16")
    return out


@functools.lru_cache(maxsize=4096)
def _gemm_workspace(m: int, n: int, k: int, kind: int, n_align: int, sm_limit: int, tile: int, splits: int, device: int | None) -> int:
    """Workspace bytes that a GEMM wants (a function of its shape and the device's number of SMs)."""
    nbytes = ctypes.c_longlong(0)
    rc = _native.lib().yf_gemm_workspace(m, n, k, kind, n_align, int(sm_limit), tile, splits, ctypes.byref(nbytes))
    if rc != 0:
        raise RuntimeError(f"yf_gemm_workspace failed with code {rc}")
    return nbytes.value


def gemm_parts(a: torch.Tensor, parts: "list[torch.Tensor]", *, b_mn_major: bool = False, tile: int = 0, splits: int = 0) -> torch.Tensor:
    """:func:`gemm` (bf16 output) with ``b`` given as two to four tensors that lie one below the other: ``torch.cat(parts)``
    without the copy.  Every part but the last has a multiple of 64 rows (:func:`can_be_parts`)."""
    m, k = a.shape
    rows = [p.shape[0] for p in parts]
    cols = parts[0].shape[1]
    n = cols if b_mn_major else sum(rows)
    assert k == (sum(rows) if b_mn_major else cols) and a.dtype == torch.bfloat16 and a.stride(1) == 1
    assert all(p.dtype == torch.bfloat16 and p.is_cuda and p.dim() == 2 and p.shape[1] == cols and p.stride(1) == 1 for p in parts)
    out = torch.empty((m, n), device=a.device, dtype=torch.bfloat16)
    align = 0 if b_mn_major else math.gcd(*(sum(rows[:i]) for i in range(1, len(rows))))
    nbytes = _gemm_workspace(m, n, k, 0, align, 0, tile, splits, a.device.index)
    ws = torch.empty(nbytes, device=a.device, dtype=torch.uint8) if nbytes else None
    np_ = len(parts)
    _check(_native.lib().yf_gemm_bf16_parts(
        a.data_ptr(), np_, (ctypes.c_void_p * np_)(*[p.data_ptr() for p in parts]), (ctypes.c_int * np_)(*rows),
        (ctypes.c_longlong * np_)(*[p.stride(0) for p in parts]), out.data_ptr(), m, n, k, a.stride(0), out.stride(0), int(b_mn_major),
        _ptr(ws), nbytes, tile, splits, _stream()), "yf_gemm_bf16_parts")
    return out


def can_be_parts(ts: "list[torch.Tensor]") -> bool:
    """Whether :func:`gemm_parts` takes these tensors."""
    first = ts[0]
    return 2 <= len(ts) <= 4 and all(
        t.is_cuda and t.dtype == torch.bfloat16 and t.dim() == 2 and t.is_contiguous() and t.shape[1] == first.shape[1] and t.shape[1] % 8 == 0
        and t.data_ptr() % 16 == 0 for t in ts) and all(t.shape[0] % 64 == 0 and t.shape[0] > 0 for t in ts)


@functools.lru_cache(maxsize=4096)
def swiglu_pays(t: int, f: int, k: int, device: int | None) -> bool:
    """Whether :func:`gemm_swiglu` takes this shape and is expected to beat the two separate kernels."""
    return _native.lib().yf_gemm_swiglu_pays(t, f, k) == 1


def can_fuse_swiglu(wg: torch.Tensor, wu: torch.Tensor) -> bool:
    """Whether :func:`gemm_swiglu` takes these weights where they are (TMA: 16-byte aligned addresses and rows).  What it does not
    take goes through the separate kernels, on a concatenated copy if need be."""
    return wg.shape == wu.shape and can_be_parts([wg, wu])


def gemm_swiglu(x: torch.Tensor, wg: torch.Tensor, wu: torch.Tensor, keep_gu: bool = True) -> tuple[torch.Tensor | None, torch.Tensor]:
    """``(gu, a)``: ``gu = [x wg^T | x wu^T]`` (``None`` unless kept) and ``a = silu(gate) * up`` from one kernel."""
    (t, k), f = x.shape, wg.shape[0]
    assert x.dtype == wg.dtype == wu.dtype == torch.bfloat16 and wg.shape == wu.shape == (f, k) and x.stride(1) == wg.stride(1) == wu.stride(1) == 1
    gu = torch.empty((t, 2 * f), device=x.device, dtype=torch.bfloat16) if keep_gu else None
    act = torch.empty((t, f), device=x.device, dtype=torch.bfloat16)
    _check(_native.lib().yf_gemm_swiglu(x.data_ptr(), wg.data_ptr(), wu.data_ptr(), _ptr(gu), act.data_ptr(), t, f, k, x.stride(0), wg.stride(0),
                                        wu.stride(0), 2 * f, f, _stream()), "yf_gemm_swiglu")
    return gu, act


def gemm_gathered(a: torch.Tensor, n: int, k: int, *, peer_in: Any, layer_buf: torch.Tensor, shard_bytes: int, b_byte_off: int,
                  rank: int, world: int, counters: torch.Tensor, epoch: int, out: torch.Tensor | None = None,
                  out_dtype: torch.dtype = torch.bfloat16, a_mn_major: bool = False) -> torch.Tensor:
    """All-gather -> GEMM in one kernel: ``out = A @ B^T`` where ``B [n, k]`` (bf16, contiguous) starts ``b_byte_off`` bytes
    into ``layer_buf``, which the same kernel fills from every rank's shard (``peer_in``: ctypes array of ``world`` peer
    pointers).  ``counters``: int64 tensor with one word per 256-row block of ``B``, zero before the first call;
    ``epoch`` = 1, 2, ... counts the calls made with these counters."""
    m = a.shape[1] if a_mn_major else a.shape[0]
    if out is None:
        out = torch.empty((m, n), device=a.device, dtype=out_dtype)
    assert counters.dtype == torch.int64 and counters.numel() >= (n + 127) // 128 and epoch >= 1
    rc = _native.lib().yf_gemm_bf16_gathered(
        a.data_ptr(), out.data_ptr(), m, n, k, a.stride(0), out.stride(0), int(a_mn_major), int(out.dtype == torch.float32),
        peer_in, layer_buf.data_ptr(), shard_bytes, b_byte_off, rank, world, counters.data_ptr(), epoch, _stream())
    _check(rc, "yf_gemm_bf16_gathered")
    return out


def gemm_scatter(a: torch.Tensor, b: torch.Tensor, *, a_mn_major: bool, b_mn_major: bool, peer_grad: Any, c_flat_off: int,
                 shard_numel: int, rank: int, world: int, alpha: float = 1.0, sm_limit: int = 0, wire_bf16: bool = False) -> None:
    """GEMM -> reduce-scatter push: the fp32 product goes piece by piece to the owners' staging slots for this rank
    (``peer_grad``: ctypes array of every rank's reduce-buffer base); nothing is stored locally."""
    m = a.shape[1] if a_mn_major else a.shape[0]
    n = b.shape[1] if b_mn_major else b.shape[0]
    k = a.shape[0] if a_mn_major else a.shape[1]
    rc = _native.lib().yf_gemm_bf16_scatter(a.data_ptr(), b.data_ptr(), m, n, k, a.stride(0), b.stride(0), int(a_mn_major),
                                            int(b_mn_major), float(alpha), peer_grad, c_flat_off, shard_numel, rank, world,
                                            int(wire_bf16), int(sm_limit), _stream())
    _check(rc, "yf_gemm_bf16_scatter")


def gemm_scatter_grouped(problems: list[tuple[torch.Tensor, torch.Tensor, int]], *, peer_grad: Any, shard_numel: int, rank: int,
                         world: int, alpha: float = 1.0, sm_limit: int = 0, wire_bf16: bool = False) -> None:
    """The weight-gradient GEMMs of a layer as one launch pushed to their owners.  ``problems``: up to four
    ``(dy [T, out], x [T, in], flat offset of the [out, in] gradient)`` in ascending flat order; every ``dW = dy^T x``
    goes to the owners' slots for this rank.  The owners' tiles are dealt round-robin, so every rank pushes to all owners
    all the time and no owner's NVLink ingress becomes a hot spot."""
    n = len(problems)
    assert 1 <= n <= 4
    k = problems[0][0].shape[0]
    a_ptrs = (ctypes.c_void_p * n)(*[dy.data_ptr() for dy, _, _ in problems])
    b_ptrs = (ctypes.c_void_p * n)(*[x.data_ptr() for _, x, _ in problems])
    ms = (ctypes.c_int * n)(*[dy.shape[1] for dy, _, _ in problems])
    ns = (ctypes.c_int * n)(*[x.shape[1] for _, x, _ in problems])
    ldas = (ctypes.c_longlong * n)(*[dy.stride(0) for dy, _, _ in problems])
    ldbs = (ctypes.c_longlong * n)(*[x.stride(0) for _, x, _ in problems])
    offs = (ctypes.c_longlong * n)(*[off for _, _, off in problems])
    for dy, x, _ in problems:
        assert dy.dtype == x.dtype == torch.bfloat16 and dy.shape[0] == x.shape[0] == k and dy.stride(1) == 1 and x.stride(1) == 1
    rc = _native.lib().yf_gemm_bf16_scatter_grouped(n, a_ptrs, b_ptrs, ms, ns, k, ldas, ldbs, 1, 1, float(alpha), peer_grad, offs,
                                                    shard_numel, rank, world, int(wire_bf16), int(sm_limit), _stream())
    _check(rc, "yf_gemm_bf16_scatter_grouped")


def push_flat(src: torch.Tensor | None, numel: int, flat_off: int, peer_grad: Any, shard_numel: int, rank: int, world: int,
              wire_bf16: bool = False) -> None:
    """Push ``numel`` fp32 values (``src``, or zeros when ``None``) that start at position ``flat_off`` of the flat layer
    gradient into the owners' reduce-scatter slots for this rank."""
    if src is not None:
        assert src.dtype == torch.float32 and src.is_contiguous() and src.numel() == numel
    rc = _native.lib().yf_push_flat(_ptr(src), numel, flat_off, peer_grad, shard_numel, rank, world, int(wire_bf16), _stream())
    _check(rc, "yf_push_flat")


# --------------------------------------------------------------------------------------- norms etc.
def rmsnorm_fwd(x: torch.Tensor, w: torch.Tensor, eps: float) -> tuple[torch.Tensor, torch.Tensor]:
    t, d = x.shape
    y = torch.empty_like(x)
    rstd = torch.empty(t, device=x.device, dtype=torch.float32)
    _check(_native.lib().yf_rmsnorm_fwd(x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr(), t, d, float(eps), _stream()),
           "yf_rmsnorm_fwd")
    return y, rstd


def rmsnorm_bwd(x: torch.Tensor, w: torch.Tensor, dy: torch.Tensor, rstd: torch.Tensor, dw_f32: torch.Tensor,
                dres: torch.Tensor | None = None, zero_dw: bool = False, sumsq: torch.Tensor | None = None) -> torch.Tensor:
    """Returns dx (+ dres when given); accumulates the weight gradient into the fp32 tensor ``dw_f32`` (``zero_dw``: what
    it held before does not count, the caller need not clear it; ``sumsq``: ``+= sum(dw_f32**2)`` of the result)."""
    t, d = x.shape
    dx = torch.empty_like(x)
    assert dw_f32.dtype == torch.float32 and dw_f32.numel() == d
    partials = torch.empty(_rmsnorm_bwd_partials(t, d, x.device.index) * d, device=x.device, dtype=torch.float32)
    _check(_native.lib().yf_rmsnorm_bwd_ws(x.data_ptr(), w.data_ptr(), dy.data_ptr(), rstd.data_ptr(), _ptr(dres), dx.data_ptr(),
                                           dw_f32.data_ptr(), int(zero_dw), partials.data_ptr(), _ptr(sumsq), t, d, _stream()), "yf_rmsnorm_bwd")
    return dx


@functools.lru_cache(maxsize=4096)
def _rmsnorm_bwd_partials(t: int, d: int, device: int | None) -> int:
    rows = _native.lib().yf_rmsnorm_bwd_partials(t, d)
    if rows < 1:
        raise RuntimeError(f"yf_rmsnorm_bwd failed with code {rows}")
    return rows


def rope_(qkv: torch.Tensor, cos_sin: torch.Tensor, seq_len: int, col0: int, n_heads: int, head_dim: int,
          backward: bool = False) -> torch.Tensor:
    """Rotate ``n_heads`` heads of ``qkv[T, :]`` starting at column ``col0`` in place."""
    t = qkv.shape[0]
    assert qkv.dim() == 2 and qkv.stride(1) == 1 and cos_sin.dtype == torch.float32
    _check(_native.lib().yf_rope(qkv.data_ptr(), cos_sin.data_ptr(), t, seq_len, qkv.stride(0), col0, n_heads, head_dim,
                                 int(backward), _stream()), "yf_rope")
    return qkv


def swiglu_fwd(gu: torch.Tensor) -> torch.Tensor:
    t, f2 = gu.shape
    h = torch.empty((t, f2 // 2), device=gu.device, dtype=gu.dtype)
    _check(_native.lib().yf_swiglu_fwd(gu.data_ptr(), h.data_ptr(), t, f2 // 2, _stream()), "yf_swiglu_fwd")
    return h


def swiglu_bwd(gu: torch.Tensor, dh: torch.Tensor) -> torch.Tensor:
    t, f2 = gu.shape
    dgu = torch.empty_like(gu)
    _check(_native.lib().yf_swiglu_bwd(gu.data_ptr(), dh.data_ptr(), dgu.data_ptr(), t, f2 // 2, _stream()), "yf_swiglu_bwd")
    return dgu


def cross_entropy_(logits: torch.Tensor, labels: torch.Tensor, grad_scale: float, write_grad: bool = True,
                   scale: torch.Tensor | None = None) -> torch.Tensor:
    """Per-row losses; ``logits`` is overwritten by ``(softmax - onehot) * grad_scale`` when ``write_grad``.  ``scale``: a
    one-element fp32 device tensor whose value multiplies ``grad_scale`` (read by the kernel: no host synchronisation)."""
    t, v = logits.shape
    assert labels.dtype == torch.int64 and logits.stride(1) == 1
    loss_rows = torch.empty(t, device=logits.device, dtype=torch.float32)
    _check(_native.lib().yf_cross_entropy(logits.data_ptr(), labels.data_ptr(), loss_rows.data_ptr(), t, v, logits.stride(0),
                                          float(grad_scale), _ptr(scale), int(write_grad), _stream()), "yf_cross_entropy")
    return loss_rows


def inv_valid_labels(labels: torch.Tensor) -> torch.Tensor:
    """``1 / max(1, number of labels that are not negative)`` as one fp32 value on the device."""
    assert labels.dtype == torch.int64 and labels.is_contiguous()
    out = torch.empty(1, device=labels.device, dtype=torch.float32)
    _check(_native.lib().yf_inv_valid_labels(labels.data_ptr(), labels.numel(), out.data_ptr(), _stream()), "yf_inv_valid_labels")
    return out


def shift_labels(labels: torch.Tensor) -> torch.Tensor:
    """Next-token labels of ``labels [B, S]``: moved one to the left, -100 at the end of every row."""
    b, s = labels.shape
    assert labels.dtype == torch.int64 and labels.stride(1) == 1
    out = torch.empty((b, s), device=labels.device, dtype=torch.int64)
    _check(_native.lib().yf_shift_labels(labels.data_ptr(), out.data_ptr(), b, s, labels.stride(0), _stream()), "yf_shift_labels")
    return out


def scaled_sum(x: torch.Tensor, scale: torch.Tensor) -> torch.Tensor:
    """``x.sum() * scale`` (fp32, 0-dimensional) in a fixed order."""
    assert x.dtype == scale.dtype == torch.float32 and x.is_contiguous()
    out = torch.empty((), device=x.device, dtype=torch.float32)
    _check(_native.lib().yf_scaled_sum(x.data_ptr(), x.numel(), scale.data_ptr(), out.data_ptr(), _stream()), "yf_scaled_sum")
    return out


def embedding_fwd(table: torch.Tensor, ids: torch.Tensor) -> torch.Tensor:
    v, d = table.shape
    t = ids.numel()
    out = torch.empty((t, d), device=table.device, dtype=table.dtype)
    _check(_native.lib().yf_embedding_fwd(table.data_ptr(), ids.data_ptr(), out.data_ptr(), t, d, v, _stream()), "yf_embedding_fwd")
    return out


def embedding_bwd_(dout: torch.Tensor, ids: torch.Tensor, dtable_f32: torch.Tensor, sumsq: torch.Tensor | None = None) -> None:
    """``dtable[ids[t]] += dout[t]``.  ``sumsq`` (only where ``dtable`` was all zeros before): ``+= sum(dtable**2)``."""
    v, d = dtable_f32.shape
    owner = torch.empty(v, device=dout.device, dtype=torch.int32) if sumsq is not None else None
    _check(_native.lib().yf_embedding_bwd_norm(dout.data_ptr(), ids.data_ptr(), dtable_f32.data_ptr(), _ptr(owner), _ptr(sumsq), ids.numel(),
                                               d, v, _stream()), "yf_embedding_bwd")


def adamw_(p: torch.Tensor, g: torch.Tensor, m: torch.Tensor, v: torch.Tensor, p_bf16: torch.Tensor | None,
           grad_scale: torch.Tensor | None, *, lr: float, beta1: float, beta2: float, eps: float, weight_decay: float,
           step: int, max_ctas: int = 0) -> None:
    n = p.numel()
    assert p.dtype == g.dtype == m.dtype == v.dtype == torch.float32
    _check(_native.lib().yf_adamw(p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), _ptr(p_bf16), _ptr(grad_scale), n,
                                  float(lr), float(beta1), float(beta2), float(eps), float(weight_decay), int(step), int(max_ctas),
                                  _stream()),
           "yf_adamw")


def sumsq_(g: torch.Tensor, out: torch.Tensor) -> None:
    """``out[0] += sum(g*g)`` (fp32)."""
    _check(_native.lib().yf_sumsq(g.data_ptr(), g.numel(), out.data_ptr(), _stream()), "yf_sumsq")


def sumsq_runs(runs: "list[torch.Tensor]") -> torch.Tensor:
    """``sum(g*g)`` over flat fp32 tensors of one device, without atomics (the same inputs give the same bits)."""
    dev = runs[0].device
    assert all(r.is_cuda and r.dtype == torch.float32 and r.is_contiguous() and r.device == dev for r in runs)
    cap = torch.cuda.get_device_properties(dev).multi_processor_count * 8
    ctas = [max(1, min(cap, r.numel() // 4096)) for r in runs]
    partials = torch.empty(sum(ctas), device=dev, dtype=torch.float32)
    at = 0
    for r, n in zip(runs, ctas):
        _check(_native.lib().yf_sumsq_partials(r.data_ptr(), r.numel(), partials.data_ptr() + 4 * at, n, _stream()), "yf_sumsq_partials")
        at += n
    return partials.sum()


def scale_(x: torch.Tensor, coef: torch.Tensor) -> None:
    """``x *= coef`` in place: flat fp32, ``coef`` one fp32 value on the same device."""
    assert x.is_cuda and x.dtype == torch.float32 and x.is_contiguous()
    assert coef.dtype == torch.float32 and coef.numel() == 1 and coef.device == x.device
    _check(_native.lib().yf_scale(x.data_ptr(), x.numel(), coef.data_ptr(), _stream()), "yf_scale")


def clip_coef_(total_sq: torch.Tensor, max_norm: float, coef: torch.Tensor, norm_out: torch.Tensor | None) -> None:
    _check(_native.lib().yf_clip_coef(total_sq.data_ptr(), float(max_norm), coef.data_ptr(), _ptr(norm_out), _stream()), "yf_clip_coef")


def cast_f32_to_bf16_(src: torch.Tensor, dst: torch.Tensor) -> None:
    assert src.numel() == dst.numel()
    _check(_native.lib().yf_cast_f32_to_bf16(src.data_ptr(), dst.data_ptr(), src.numel(), _stream()), "yf_cast_f32_to_bf16")


def accum_bf16_to_f32_(src: torch.Tensor, dst: torch.Tensor, scale: float = 1.0, accumulate: bool = False) -> None:
    assert src.numel() == dst.numel()
    _check(_native.lib().yf_accum_bf16_to_f32(src.data_ptr(), dst.data_ptr(), src.numel(), float(scale), int(accumulate), _stream()),
           "yf_accum_bf16_to_f32")


def accum_bf16_to_f32_multi_(pairs: "list[tuple[torch.Tensor, torch.Tensor]]", accumulate: bool) -> None:
    """``dst (+)= src`` for ``(dst fp32, src bf16)`` pairs of contiguous tensors of one device, in one launch."""
    n = len(pairs)
    assert all(d.is_cuda and d.dtype == torch.float32 and s.dtype == torch.bfloat16 and d.is_contiguous() and s.is_contiguous()
               and d.numel() == s.numel() and d.device == s.device == pairs[0][0].device for d, s in pairs)
    _check(_native.lib().yf_accum_bf16_to_f32_multi(
        n, (ctypes.c_void_p * n)(*[s.data_ptr() for _, s in pairs]), (ctypes.c_void_p * n)(*[d.data_ptr() for d, _ in pairs]),
        (ctypes.c_longlong * n)(*[d.numel() for d, _ in pairs]), int(accumulate), _stream()), "yf_accum_bf16_to_f32_multi")


def add_bf16(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    out = torch.empty_like(a) if out is None else out
    _check(_native.lib().yf_add_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), a.numel(), _stream()), "yf_add_bf16")
    return out


# --------------------------------------------------------------------------------------- attention
def attn_fwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, batch: int, seq: int, n_heads: int, n_kv_heads: int,
             scale: float, causal: bool = True) -> tuple[torch.Tensor, torch.Tensor]:
    """Flash attention forward, head_dim 128.  ``q``: ``[B*S, Hq*128]`` view, ``k``/``v``: ``[B*S, Hkv*128]``
    views (column blocks of the fused QKV projection output are fine).  Returns ``out [B*S, Hq*128]`` and
    ``lse [B, Hq, S]``."""
    t = batch * seq
    assert q.shape == (t, n_heads * 128) and k.shape == (t, n_kv_heads * 128) and v.shape == k.shape
    assert q.stride(1) == 1 and k.stride(1) == 1 and v.stride(1) == 1 and k.stride(0) == v.stride(0)
    out = torch.empty((t, n_heads * 128), device=q.device, dtype=torch.bfloat16)
    lse = torch.empty((batch, n_heads, seq), device=q.device, dtype=torch.float32)
    _check(_native.lib().yf_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), batch, seq,
                                     n_heads, n_kv_heads, q.stride(0), k.stride(0), out.stride(0), float(scale), int(causal),
                                     _stream()), "yf_attn_fwd")
    return out, lse


@functools.lru_cache(maxsize=4096)
def _attn_bwd_head_parts(batch: int, seq: int, n_heads: int, n_kv_heads: int, device: int | None) -> int:
    parts = _native.lib().yf_attn_bwd_head_parts(batch, seq, n_heads, n_kv_heads)
    if parts < 1:
        raise RuntimeError(f"yf_attn_bwd_head_parts failed with code {parts}")
    return parts


def attn_bwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, out: torch.Tensor, dout: torch.Tensor, lse: torch.Tensor,
             dq: torch.Tensor, dk: torch.Tensor, dv: torch.Tensor, batch: int, seq: int, n_heads: int, n_kv_heads: int,
             scale: float, causal: bool = True, head_parts: int = 0, rope: torch.Tensor | None = None) -> None:
    """Flash attention backward into the given ``dq``/``dk``/``dv`` views (bf16, unit column stride).  ``head_parts``: CTAs that
    share a key tile of a KV head (a divisor of the group; 0 = chosen from the shape).  ``rope``: the ``[seq, 64, 2]`` table that
    ``q`` and ``k`` were rotated with; ``dq`` and ``dk`` are then the gradients of what was rotated."""
    assert rope is None or (rope.dtype == torch.float32 and rope.is_contiguous() and rope.numel() >= seq * 128)
    t = batch * seq
    assert dout.stride(1) == 1 and out.stride(1) == 1 and dq.stride(1) == 1 and dk.stride(1) == 1 and dv.stride(1) == 1
    assert dk.stride(0) == dv.stride(0)
    delta = torch.empty((batch, n_heads, seq), device=q.device, dtype=torch.float32)
    dq_acc = torch.empty((t, n_heads * 128), device=q.device, dtype=torch.float32)
    parts = _attn_bwd_head_parts(batch, seq, n_heads, n_kv_heads, q.device.index) if head_parts == 0 else head_parts
    dkv_parts = torch.empty((parts, 2, batch, (seq + 127) // 128 * 128, n_kv_heads * 128), device=q.device, dtype=torch.float32) if parts > 1 else None
    global _launches
    _check(_native.lib().yf_attn_bwd_parts(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), dout.data_ptr(), lse.data_ptr(),
                                           delta.data_ptr(), dq_acc.data_ptr(), _ptr(dkv_parts), 0 if dkv_parts is None else dkv_parts.numel(), parts, _ptr(rope), dq.data_ptr(), dk.data_ptr(),
                                           dv.data_ptr(), batch, seq, n_heads, n_kv_heads, q.stride(0), k.stride(0), out.stride(0),
                                           dout.stride(0), dq.stride(0), dk.stride(0), float(scale), int(causal), _stream()),
           "yf_attn_bwd")
    _launches += 2  # delta pre-pass and dq conversion post-pass
