"""What this framework is measured on: training steps, forward passes and single decoder layers through the public API.

One GPU, one rank.  Widths come from the model configurations of ``yafsdp_b200.models.llama.CONFIGS``; the number of decoder
layers is cut to one or two, so that weights, gradients and optimizer state of a case fit the GPU several times.  Kinds:

* ``train``   ``build_llama`` + ``ShardedAdamW``: a whole step from pinned host tokens to updated weights (bf16 compute,
              fp32 master weights, gradients and moments), with global-norm clipping, micro-batches, prompt-masked labels and
              activation checkpointing as options;
* ``eval``    the logits of an unsharded bf16 model without gradients (scoring, the prompt of a generation);
* ``layer``   forward and backward of one ``LlamaDecoderLayer`` with plain bf16 parameters, as part of somebody's own model;
* ``modules`` somebody's own ``nn.Module`` blocks under ``fully_shard`` with ``torch.optim.AdamW`` and ``clip_grad_norm_``.
"""

from __future__ import annotations

import math
from typing import Any

import torch
import torch.distributed as dist
import torch.nn as nn
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from yafsdp_b200 import MixedPrecisionPolicy, fully_shard
from yafsdp_b200.models.llama import CONFIGS, LlamaConfig, LlamaDecoderLayer, LlamaForCausalLM
from yafsdp_b200.ops.functional import rope_table
from yafsdp_b200.optim import ShardedAdamW, clip_grad_norm_, param_groups_of
from yafsdp_b200.train import TrainStep, build_llama

ARCHS = ("tiny-gpu", "llama2-7b", "llama2-13b", "llama3-8b", "llama2-34b", "llama2-70b")
N_BATCHES = 4  # token batches that a training state walks through


def listed() -> list[dict[str, Any]]:
    return [
        # the smallest training step: a toy model, bound by launches and by the host
        _train("smoke step", "tiny-gpu", layers=2, batch=2, seq=256),
        # the headline pre-training configuration, two of its layers
        _train("pretrain 7b 2048", "llama2-7b", layers=2, batch=1, seq=2048),
        # long-context pre-training: grouped-query attention and the large vocabulary
        _train("pretrain 8b 8192", "llama3-8b", layers=1, batch=1, seq=8192),
        # the largest widths, activations recomputed in backward
        _train("pretrain 70b checkpointed", "llama2-70b", layers=1, batch=1, seq=2048, checkpoint=True),
        # gradient accumulation over micro-batches whose length is no multiple of any tile
        _train("accumulate 7b 2x1337", "llama2-7b", layers=1, batch=1, seq=1337, micro=2),
        # supervised fine-tuning on short ragged conversations, the prompt's labels masked, no clipping
        _train("finetune 13b 3x333", "llama2-13b", layers=1, batch=3, seq=333, masked=True, clip=0.0),
        # a decoder layer inside somebody's own model: ordinary and small ragged
        _layer("layer 7b 2x4096", "llama2-7b", batch=2, seq=4096),
        _layer("layer 34b 1x777", "llama2-34b", batch=1, seq=777),
        # scoring a batch of documents, and the prompt of a chat turn
        _eval("score 8b 4x1024", "llama3-8b", layers=1, batch=4, seq=1024),
        _eval("prompt 7b 1x45", "llama2-7b", layers=2, batch=1, seq=45),
        # own modules with a torch optimizer: the sharding framework around library kernels
        {"name": "modules 4096", "kind": "modules", "hidden": 4096, "ffn": 11008, "layers": 4, "tokens": 2048, "clip": 1.0},
    ]


def _train(name: str, arch: str, *, layers: int, batch: int, seq: int, micro: int = 1, checkpoint: bool = False, masked: bool = False,
           clip: float = 1.0) -> dict[str, Any]:
    return {"name": name, "kind": "train", "arch": arch, "layers": layers, "batch": batch, "seq": seq, "micro": micro,
            "checkpoint": checkpoint, "masked": masked, "clip": clip}


def _layer(name: str, arch: str, *, batch: int, seq: int) -> dict[str, Any]:
    return {"name": name, "kind": "layer", "arch": arch, "layers": 1, "batch": batch, "seq": seq}


def _eval(name: str, arch: str, *, layers: int, batch: int, seq: int) -> dict[str, Any]:
    return {"name": name, "kind": "eval", "arch": arch, "layers": layers, "batch": batch, "seq": seq}


def _log_int(rng: Any, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _cost(case: dict[str, Any]) -> float:
    w = work(case)
    return max(w["bytes"], w["flops"] / 200.0)  # seconds times a few TB/s, either way


def draw(rng: Any) -> dict[str, Any]:
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(("train", "train", "train", "eval", "eval", "layer", "layer", "modules"))
        if kind == "modules":
            hidden = rng.choice((512, 1024, 2048, 4096, 5120))
            case = {"kind": kind, "hidden": hidden, "ffn": 8 * rng.randint(hidden // 8, hidden // 2), "layers": rng.randint(1, 4),
                    "tokens": _log_int(rng, 64, 8192), "clip": rng.choice((0.0, 1.0))}
        else:
            batch = rng.choice((1, 1, 1, 2, 3, 4))
            tokens = _log_int(rng, 16 if kind == "eval" else 128, 8192)
            case = {"kind": kind, "arch": rng.choice(ARCHS), "layers": 1 if kind == "layer" else rng.randint(1, 2), "batch": batch,
                    "seq": max(8, tokens // batch)}
            if kind == "train":
                case.update(micro=rng.choice((1, 1, 2)), checkpoint=rng.random() < 0.25, masked=rng.random() < 0.25,
                            clip=rng.choice((0.0, 1.0, 1.0)))
        if _cost(case) <= most:
            return case


# ----------------------------------------------------------------------------------------- preparation
def _config(case: dict[str, Any]) -> LlamaConfig:
    c = CONFIGS[case["arch"]]
    return LlamaConfig(vocab_size=c.vocab_size, hidden_size=c.hidden_size, intermediate_size=c.intermediate_size,
                       num_hidden_layers=case["layers"], num_attention_heads=c.num_attention_heads,
                       num_key_value_heads=c.num_key_value_heads, rms_norm_eps=c.rms_norm_eps, rope_theta=c.rope_theta,
                       max_position_embeddings=max(c.max_position_embeddings, case["seq"]))


def _device() -> torch.device:
    torch.cuda.set_device(0)
    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    return torch.device("cuda", 0)


def prepare(case: dict[str, Any], seed: int) -> dict[str, Any]:
    return _PREPARE[case["kind"]](case, seed)


def _prepare_train(case: dict[str, Any], seed: int) -> dict[str, Any]:
    dev = _device()
    cfg = _config(case)
    model = build_llama(cfg, dev, seed=seed, checkpoint_layers=cfg.num_hidden_layers if case["checkpoint"] else 0)
    opt = ShardedAdamW(model, lr=1e-5, betas=(0.9, 0.95), weight_decay=0.1, max_grad_norm=case["clip"] or None)
    gen = torch.Generator().manual_seed(seed)
    shape = (case["batch"], case["seq"])
    batches = []
    for _ in range(N_BATCHES * case["micro"]):
        ids = torch.randint(0, cfg.vocab_size, shape, generator=gen).pin_memory()
        labels = ids
        if case["masked"]:  # each row: a prompt of some length without labels, then the answer
            prompt = torch.randint(1, max(2, case["seq"] * 3 // 4), (case["batch"], 1), generator=gen)
            labels = ids.masked_fill(torch.arange(case["seq"])[None, :] < prompt, -100).pin_memory()
        batches.append((ids, labels))
    return {"kind": "train", "model": model, "opt": opt, "step": TrainStep(model, opt, dev), "device": dev, "batches": batches, "at": 0,
            "micro": case["micro"], "masked": case["masked"], "groups": param_groups_of(model)}


def _prepare_eval(case: dict[str, Any], seed: int) -> dict[str, Any]:
    dev = _device()
    cfg = _config(case)
    model = LlamaForCausalLM(cfg, device=dev, dtype=torch.bfloat16)
    model.init_weights(seed)
    gen = torch.Generator().manual_seed(seed)
    ids = torch.randint(0, cfg.vocab_size, (case["batch"], case["seq"]), generator=gen)
    return {"kind": "eval", "model": model, "ids": ids.to(dev)}


def _prepare_layer(case: dict[str, Any], seed: int) -> dict[str, Any]:
    dev = _device()
    cfg = _config(case)
    gen = torch.Generator(device=dev).manual_seed(seed)
    layer = LlamaDecoderLayer(cfg, device=dev, dtype=torch.bfloat16)
    with torch.no_grad():
        for p in layer.parameters():
            if p.dim() > 1:
                p.normal_(0.0, cfg.initializer_range, generator=gen)
    t = case["batch"] * case["seq"]
    x = torch.randn(t, cfg.hidden_size, device=dev, generator=gen).bfloat16().requires_grad_(True)
    dout = torch.randn(t, cfg.hidden_size, device=dev, generator=gen).bfloat16()
    return {"kind": "layer", "layer": layer, "x": x, "dout": dout, "batch": case["batch"], "seq": case["seq"],
            "cos_sin": rope_table(case["seq"], cfg.head_dim, cfg.rope_theta, dev), "params": dict(layer.named_parameters())}


class _Block(nn.Module):
    def __init__(self, hidden: int, ffn: int, device: torch.device):
        super().__init__()
        self.norm = nn.LayerNorm(hidden, device=device)
        self.up = nn.Linear(hidden, ffn, device=device)
        self.down = nn.Linear(ffn, hidden, device=device)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return x + self.down(F.gelu(self.up(self.norm(x))))


def _prepare_modules(case: dict[str, Any], seed: int) -> dict[str, Any]:
    dev = _device()
    torch.manual_seed(seed)
    model = nn.Sequential(*[_Block(case["hidden"], case["ffn"], dev) for _ in range(case["layers"])])
    policy = MixedPrecisionPolicy(param_dtype=torch.bfloat16, reduce_dtype=torch.float32)
    for block in model:
        fully_shard(block, mp_policy=policy)
    fully_shard(model, mp_policy=policy)
    opt = torch.optim.AdamW(model.parameters(), lr=1e-5, betas=(0.9, 0.95), weight_decay=0.1, fused=True)
    x = torch.randn(case["tokens"], case["hidden"], device=dev).bfloat16().requires_grad_(True)
    y = torch.randn(case["tokens"], case["hidden"], device=dev)
    return {"kind": "modules", "model": model, "opt": opt, "x": x, "y": y, "clip": case["clip"], "groups": param_groups_of(model)}


_PREPARE = {"train": _prepare_train, "eval": _prepare_eval, "layer": _prepare_layer, "modules": _prepare_modules}


# ----------------------------------------------------------------------------------------- one pass
def run(state: dict[str, Any]) -> dict[str, Any]:
    return _RUN[state["kind"]](state)


def _run_train(s: dict[str, Any]) -> dict[str, Any]:
    model, opt, dev, micro = s["model"], s["opt"], s["device"], s["micro"]
    at = s["at"]
    s["at"] = (at + micro) % len(s["batches"])
    if micro == 1 and not s["masked"]:
        loss = s["step"](s["batches"][at][0])
    else:
        opt.zero_grad()
        loss = torch.zeros((), device=dev)
        for ids, labels in s["batches"][at : at + micro]:
            ids_dev = ids.to(dev, non_blocking=True)
            part = model(ids_dev, labels=labels.to(dev, non_blocking=True) if labels is not ids else ids_dev) / micro
            part.backward()
            loss += part.detach()
        opt.step()
    return {"loss": loss.detach(), "weights": [g.master_flat for g in s["groups"]], "grads": [g.sharded_grad_flat for g in s["groups"]],
            "exp_avg": list(opt.exp_avg), "exp_avg_sq": list(opt.exp_avg_sq)}


def _run_eval(s: dict[str, Any]) -> dict[str, Any]:
    with torch.no_grad():
        return {"logits": s["model"](s["ids"])}


def _run_layer(s: dict[str, Any]) -> dict[str, Any]:
    layer, x = s["layer"], s["x"]
    x.grad = None
    layer.zero_grad(set_to_none=True)
    out = layer(x, s["cos_sin"], s["batch"], s["seq"])
    out.backward(s["dout"])
    return {"out": out.detach(), "dx": x.grad, "grads": {n: p.grad for n, p in s["params"].items()}}


def _run_modules(s: dict[str, Any]) -> dict[str, Any]:
    model, opt = s["model"], s["opt"]
    s["x"].grad = None
    loss = F.mse_loss(model(s["x"]).float(), s["y"])
    loss.backward()
    if s["clip"]:
        clip_grad_norm_(model, s["clip"])
    opt.step()
    opt.zero_grad()
    return {"loss": loss.detach(), "dx": s["x"].grad, "weights": [g.master_flat for g in s["groups"]],
            "grads": [g.sharded_grad_flat for g in s["groups"]]}


_RUN = {"train": _run_train, "eval": _run_eval, "layer": _run_layer, "modules": _run_modules}


# ----------------------------------------------------------------------------------------- work and tolerance
def work(case: dict[str, Any]) -> dict[str, float]:
    """Training: fp32 weight and two moments read and written, the fp32 gradient and the bf16 weight written (30 bytes per
    parameter); six operations per weight of a projection and token, causal attention with its two products forward and five
    backward at half the square."""
    if case["kind"] == "modules":
        d, f, t = case["hidden"], case["ffn"], case["tokens"]
        n = case["layers"] * (2 * d * f + f + 3 * d)
        return {"bytes": 30.0 * n + 8.0 * t * d, "flops": 6.0 * t * case["layers"] * 2 * d * f}
    c = CONFIGS[case["arch"]]
    d, f, v, layers = c.hidden_size, c.intermediate_size, c.vocab_size, case["layers"]
    kv = c.num_key_value_heads * c.head_dim
    t = float(case["batch"] * case["seq"])
    proj = 2 * d * d + 2 * d * kv + 3 * d * f
    attn = layers * 2.0 * t * case["seq"] * d  # the two products of one forward pass, causal
    if case["kind"] == "eval":
        n = layers * (proj + 2 * d) + v * d + d
        return {"bytes": 2.0 * n + 2.0 * t * d + 2.0 * t * v + 8.0 * t, "flops": 2.0 * t * (layers * proj + v * d) + attn}
    if case["kind"] == "layer":
        n = proj + 2 * d
        return {"bytes": 4.0 * n + 8.0 * t * d, "flops": 6.0 * t * proj + 3.5 * attn}
    t *= case["micro"]
    attn *= case["micro"]
    n = layers * (proj + 2 * d) + 2 * v * d + d
    again = 1.0 if case["checkpoint"] else 0.0
    return {"bytes": 30.0 * n + 8.0 * t, "flops": (6.0 + 2.0 * again) * t * layers * proj + 6.0 * t * v * d + (3.5 + again) * attn}


def tolerance(case: dict[str, Any]) -> dict[str, float]:
    """Every activation is rounded to bf16, so the errors of a whole pass grow with its depth.  Measured against the same math
    in fp32 (relative 2-norms): logits 0.011-0.012, tensors of a layer pass 0.005-0.016, flat gradients of a training step
    0.008 (toy widths) to 0.016 (one layer) and 0.018 (two; single tensors up to 0.031); the same math as bf16 PyTorch
    operations is 4-7 % further off.  Two correct implementations are up to 1.4 times these figures apart.  ``modules``: library kernels
    throughout, one bf16 rounding of the gradients on the way."""
    return {"rel": {"train": 0.03, "layer": 0.025, "eval": 0.02, "modules": 0.01}[case["kind"]]}


# ----------------------------------------------------------------------------------------- the same in 64 bits
def exact(case: dict[str, Any], seed: int) -> dict[str, Any]:
    """What the first ``run`` after ``prepare(case, seed)`` returns, in plain torch operations in 64 bits: the weights as the
    compute type holds them, nothing rounded on the way."""
    return _EXACT[case["kind"]](case, prepare(case, seed))


def _exact_norm(x: torch.Tensor, w: torch.Tensor, eps: float) -> torch.Tensor:
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _exact_head(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> torch.Tensor:
    """Causal attention of one sequence and head."""
    hidden = torch.ones(q.shape[0], q.shape[0], dtype=torch.bool, device=q.device).triu_(1)
    return (q @ k.T / math.sqrt(q.shape[1])).masked_fill_(hidden, -math.inf).softmax(-1) @ v


def _exact_layer(x: torch.Tensor, w: dict[str, torch.Tensor], cfg: LlamaConfig, batch: int, seq: int) -> torch.Tensor:
    hq, hkv, hd, half = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.head_dim // 2
    pos = torch.arange(seq, dtype=torch.float64, device=x.device)
    ang = pos[:, None] * cfg.rope_theta ** (torch.arange(half, dtype=torch.float64, device=x.device) * (-2.0 / hd))
    cos, sin = ang.cos()[None, :, None, :], ang.sin()[None, :, None, :]

    def heads(name: str, n: int, rotate: bool) -> torch.Tensor:
        t = (n1 @ w[f"self_attn.{name}_proj.weight"].T).view(batch, seq, n, hd)
        if rotate:
            a, b = t[..., :half], t[..., half:]
            t = torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)
        return t.transpose(1, 2)

    n1 = _exact_norm(x, w["input_layernorm.weight"], cfg.rms_norm_eps)
    q, k, v = heads("q", hq, True), heads("k", hkv, True), heads("v", hkv, False)
    att = torch.stack([checkpoint(_exact_head, q[b, h], k[b, h * hkv // hq], v[b, h * hkv // hq], use_reentrant=False)
                       for b in range(batch) for h in range(hq)])
    att = att.view(batch, hq, seq, hd).transpose(1, 2).reshape(batch * seq, hq * hd)
    x = x + att @ w["self_attn.o_proj.weight"].T
    n2 = _exact_norm(x, w["post_attention_layernorm.weight"], cfg.rms_norm_eps)
    return x + (F.silu(n2 @ w["mlp.gate_proj.weight"].T) * (n2 @ w["mlp.up_proj.weight"].T)) @ w["mlp.down_proj.weight"].T


def _exact_logits(ids: torch.Tensor, w: dict[str, torch.Tensor], cfg: LlamaConfig) -> torch.Tensor:
    x = w["model.embed_tokens.weight"][ids.reshape(-1)]
    for i in range(cfg.num_hidden_layers):
        pre = f"model.layers.{i}."
        x = _exact_layer(x, {n[len(pre) :]: t for n, t in w.items() if n.startswith(pre)}, cfg, *ids.shape)
    return _exact_norm(x, w["model.norm.weight"], cfg.rms_norm_eps) @ w["lm_head.weight"].T


def _exact_weights(model: nn.Module, groups: list[Any]) -> tuple[dict[str, torch.Tensor], list[list[str]]]:
    """The parameters of a sharded model (one rank) as its compute type holds them, and their names by group in flat order."""
    names = {p: n for n, p in model.named_parameters()}
    order = [[names[sp.sharded_param] for sp in g.params] for g in groups]
    w = {}
    for g, members in zip(groups, order):
        for name, sp in zip(members, g.params):
            at = sp.placement.shard_offset
            w[name] = g.master_flat[at : at + sp.numel].view(sp.orig_shape).bfloat16().double().requires_grad_(True)
    return w, order


def _exact_step(w: dict[str, torch.Tensor], order: list[list[str]], groups: list[Any], clip: float, clipped_grads: bool) -> dict[str, Any]:
    """The first AdamW step from the masters of ``groups`` with the gradients in ``w``."""
    norm = torch.stack([t.grad.norm() for t in w.values()]).norm()
    coef = float(torch.clamp(clip / (norm + 1e-6), max=1.0)) if clip else 1.0
    out: dict[str, Any] = {"weights": [], "grads": [], "exp_avg": [], "exp_avg_sq": []}
    for g, members in zip(groups, order):
        grad = torch.zeros(g.master_flat.numel(), dtype=torch.float64, device=g.master_flat.device)
        for name, sp in zip(members, g.params):
            at = sp.placement.shard_offset
            grad[at : at + sp.numel] = w[name].grad.reshape(-1)
            w[name].grad = None
        m, v = grad * (0.1 * coef), grad.pow(2).mul_(0.05 * coef * coef)
        p = g.master_flat.double().mul_(1 - 1e-5 * 0.1).addcdiv_(m, (v / 0.05).sqrt_().add_(1e-8), value=-1e-5 / 0.1)
        for key, value in (("weights", p), ("grads", grad.mul_(coef) if clipped_grads else grad), ("exp_avg", m), ("exp_avg_sq", v)):
            out[key].append(value)
    return out


def _exact_train(case: dict[str, Any], s: dict[str, Any]) -> dict[str, Any]:
    w, order = _exact_weights(s["model"], s["groups"])
    total = torch.zeros((), dtype=torch.float64, device=s["device"])
    for ids, labels in s["batches"][: case["micro"]]:
        target = torch.cat([labels[:, 1:], torch.full_like(labels[:, :1], -100)], dim=1).to(s["device"]).reshape(-1)
        loss = F.cross_entropy(_exact_logits(ids.to(s["device"]), w, _config(case)), target, ignore_index=-100, reduction="sum")
        loss = loss / (target >= 0).sum().clamp(min=1) / case["micro"]
        loss.backward()
        total += loss.detach()
    return {"loss": total, **_exact_step(w, order, s["groups"], case["clip"], clipped_grads=False)}


def _exact_eval(case: dict[str, Any], s: dict[str, Any]) -> dict[str, Any]:
    with torch.no_grad():
        w = {n: p.double() for n, p in s["model"].named_parameters()}
        return {"logits": _exact_logits(s["ids"], w, _config(case)).view(case["batch"], case["seq"], -1)}


def _exact_layer_pass(case: dict[str, Any], s: dict[str, Any]) -> dict[str, Any]:
    w = {n: p.detach().double().requires_grad_(True) for n, p in s["params"].items()}
    x = s["x"].detach().double().requires_grad_(True)
    out = _exact_layer(x, w, _config(case), case["batch"], case["seq"])
    out.backward(s["dout"].double())
    return {"out": out.detach(), "dx": x.grad, "grads": {n: t.grad for n, t in w.items()}}


def _exact_modules(case: dict[str, Any], s: dict[str, Any]) -> dict[str, Any]:
    w, order = _exact_weights(s["model"], s["groups"])
    x0 = s["x"].detach().double().requires_grad_(True)
    x = x0
    for i in range(case["layers"]):
        n = F.layer_norm(x, x.shape[-1:], w[f"{i}.norm.weight"], w[f"{i}.norm.bias"])
        h = F.gelu(F.linear(n, w[f"{i}.up.weight"], w[f"{i}.up.bias"]))
        x = x + F.linear(h, w[f"{i}.down.weight"], w[f"{i}.down.bias"])
    loss = F.mse_loss(x, s["y"].double())
    loss.backward()
    step = _exact_step(w, order, s["groups"], case["clip"], clipped_grads=True)
    return {"loss": loss.detach(), "dx": x0.grad, "weights": step["weights"], "grads": step["grads"]}


_EXACT = {"train": _exact_train, "eval": _exact_eval, "layer": _exact_layer_pass, "modules": _exact_modules}
