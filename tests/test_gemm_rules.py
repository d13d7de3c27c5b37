"""Which GEMM kernels the native library chooses (host code alone: without a device it plans for 148 SMs)."""

import os
import subprocess
import sys

import pytest


def _pays(shapes, **env):
    """yf_gemm_swiglu_pays of every (tokens, F, K), in a process of its own: the library reads its switches once."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    # _native.py by its path: importing the package would import torch
    code = ("import importlib.util, sys; spec = importlib.util.spec_from_file_location('native', 'yafsdp_b200/_native.py'); "
            "n = importlib.util.module_from_spec(spec); sys.modules['native'] = n; spec.loader.exec_module(n); "
            f"print([n.lib().yf_gemm_swiglu_pays(*s) for s in {shapes!r}])")
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env={**os.environ, "CUDA_VISIBLE_DEVICES": "", **env}, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return eval(r.stdout)


@pytest.mark.parametrize("switch", ["0", "1"])
def test_switch_against_cta_pairs_covers_the_fused_activation(switch):
    want = 0 if switch == "1" else 1
    assert _pays([(8192, 11008, 4096), (2048, 28672, 8192)], YAFSDP_GEMM_CTA_GROUP=switch) == [want, want]
