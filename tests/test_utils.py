"""Profiling / logging helpers (CPU)."""

import io
import json

import pytest
import torch


def test_step_timer_and_logger():
    from yafsdp_b200.utils.profiling import StepLogger, StepTimer

    timer = StepTimer(torch.device("cpu"))
    for _ in range(3):
        with timer.step():
            torch.randn(64, 64) @ torch.randn(64, 64)
    s = timer.summary()
    assert s["steps"] == 3 and s["host_ms_mean"] > 0
    buf = io.StringIO()
    log = StepLogger(tokens_per_step_per_gpu=2048, stream=buf)
    rec = log.log(loss=3.5, iter_time_s=0.1, grad_norm=1.25)
    assert rec["tokens_per_s_per_gpu"] == 20480.0 and log.step == 1
    assert json.loads(buf.getvalue())["grad_norm"] == 1.25


def test_profile_steps_writes_a_trace(tmp_path):
    from yafsdp_b200.utils.profiling import profile_steps

    path = tmp_path / "trace.json"
    with profile_steps(str(path), wait=1, warmup=1, active=1) as prof:
        for _ in range(4):
            torch.randn(32, 32).sum()
            prof.step()
    assert path.exists() and "traceEvents" in json.loads(path.read_text())


@pytest.mark.parametrize("observer", ["profiler", "execution trace"])
def test_phase_labels_reach_every_observer(tmp_path, observer):
    """Ranges of the schedule are recorded for whatever watches them, not only under the autograd profiler."""
    from yafsdp_b200.common import _NO_LABEL, phase_label

    path = tmp_path / "trace.json"
    assert phase_label("YaFSDP::idle") is _NO_LABEL
    if observer == "profiler":
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
            with phase_label("YaFSDP::pre_forward", "layers.0"):
                torch.ones(2).sum()
        prof.export_chrome_trace(str(path))
    else:
        trace = torch.profiler.ExecutionTraceObserver()
        trace.register_callback(str(path))
        trace.start()
        with phase_label("YaFSDP::pre_forward", "layers.0"):
            torch.ones(2).sum()
        trace.stop()
        trace.unregister_callback()
    assert "YaFSDP::pre_forward (layers.0)" in path.read_text()
    assert phase_label("YaFSDP::idle") is _NO_LABEL


def test_checkpoint_module_recomputes():
    from yafsdp_b200.utils.checkpointing import checkpoint_module

    calls = []

    class M(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.l = torch.nn.Linear(4, 4)

        def forward(self, x):
            calls.append(1)
            return torch.tanh(self.l(x))

    m = checkpoint_module(M())
    x = torch.randn(2, 4, requires_grad=True)
    m(x).sum().backward()
    assert len(calls) == 2 and m.l.weight.grad is not None  # forward ran again during backward


def test_trainer_config_file_provides_defaults_and_flags_override():
    import argparse
    import os

    from yafsdp_b200.train import parse_with_config

    def parser():
        ap = argparse.ArgumentParser()
        ap.add_argument("--model", default="llama2-7b")
        ap.add_argument("--seq-len", type=int, default=2048)
        ap.add_argument("--checkpoint-layers", type=int, default=0)
        ap.add_argument("--steps", type=int, default=10)
        ap.add_argument("--batch", type=int, default=1)
        ap.add_argument("--lr", type=float, default=3e-4)
        ap.add_argument("--max-grad-norm", type=float, default=1.0)
        ap.add_argument("--comm-backend", default="auto")
        ap.add_argument("--config", default=None)
        return ap

    cfg = os.path.join(os.path.dirname(__file__), "..", "examples", "shard_config.yaml")
    args = parse_with_config(parser(), ["--config", cfg, "--seq-len", "4096"])
    assert args.steps == 100 and args.seq_len == 4096 and args.model == "llama2-7b" and args.checkpoint_layers == 0


def test_memory_plan_matches_a_measured_run_and_ranks_the_large_configs():
    from yafsdp_b200.models.llama import CONFIGS
    from yafsdp_b200.utils.memory import estimate_memory

    # Llama-2-7B, one GPU, 2048 tokens: 121.2 GiB peak allocated was measured on a B200
    one = estimate_memory(CONFIGS["llama2-7b"], world=1, seq_len=2048)
    assert abs(one["total"] / 2**30 - 121.2) < 3.0 and one["buffers"] == 0 and one["fits"]
    eight = estimate_memory(CONFIGS["llama2-7b"], world=8, seq_len=2048)
    assert eight["state"] * 8 == one["state"] and eight["buffers"] > 0 and eight["total"] < one["total"] / 3
    # 70B on 8 GPUs only fits with activation checkpointing... and not at all on 4
    big = CONFIGS["llama2-70b"]
    assert estimate_memory(big, 8, 2048, checkpoint_layers=80)["fits"]
    assert estimate_memory(big, 8, 2048, checkpoint_layers=80)["total"] < estimate_memory(big, 8, 2048)["total"]
    assert not estimate_memory(big, 4, 2048, checkpoint_layers=80)["fits"]
