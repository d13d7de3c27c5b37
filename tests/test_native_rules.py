"""Which kernels and splits the native library chooses (host code alone: without a device it plans for 148 SMs)."""

import os
import subprocess
import sys

import pytest


def _ask(function, arguments, **env):
    """``function`` of the library for every one of ``arguments``, in a process of its own: switches are read once."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    # _native.py by its path: importing the package would import torch
    code = ("import importlib.util, sys; spec = importlib.util.spec_from_file_location('native', 'yafsdp_b200/_native.py'); "
            "n = importlib.util.module_from_spec(spec); sys.modules['native'] = n; spec.loader.exec_module(n); "
            f"print([n.lib().{function}(*a) for a in {arguments!r}])")
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env={**os.environ, "CUDA_VISIBLE_DEVICES": "", **env}, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return eval(r.stdout)


@pytest.mark.parametrize("switch", ["0", "1"])
def test_switch_against_cta_pairs_covers_the_fused_activation(switch):
    want = 0 if switch == "1" else 1
    assert _ask("yf_gemm_swiglu_pays", [(8192, 11008, 4096), (2048, 28672, 8192)], YAFSDP_GEMM_CTA_GROUP=switch) == [want, want]


def test_parts_of_a_key_tile_where_they_were_measured():
    """The faster choice where the sides were at least 10 % apart (the figures stand at the rule)."""
    best = {(1, 777, 64, 8): 4, (1, 1024, 64, 8): 4, (1, 2048, 64, 8): 2, (1, 2048, 32, 8): 2, (2, 777, 32, 8): 2, (8, 300, 32, 8): 1,
            (4, 1024, 32, 8): 1, (1, 4096, 28, 4): 7, (1, 1337, 28, 4): 7, (1, 2048, 8, 1): 8, (6, 512, 16, 2): 4, (2, 64, 2, 2): 1}
    assert dict(zip(best, _ask("yf_attn_bwd_head_parts", list(best)))) == best


def test_fused_activation_where_it_was_measured():
    """The faster choice where the sides were at least 8 % apart (the figures stand at the rule): whole and ragged tiles, few tokens
    at large weights."""
    best = {(999, 11008, 4096): 1, (2048, 11008, 4096): 1, (2500, 11008, 4096): 1, (8192, 11008, 4096): 1, (2048, 14336, 4096): 1,
            (999, 13824, 5120): 1, (4096, 28672, 8192): 1, (45, 11008, 4096): 0, (300, 11008, 4096): 0, (777, 11008, 4096): 0,
            (300, 13824, 5120): 0, (777, 14336, 4096): 0, (45, 22016, 8192): 0, (128, 22016, 8192): 0, (777, 22016, 8192): 0,
            (128, 28672, 8192): 0, (777, 28672, 8192): 0}
    assert dict(zip(best, _ask("yf_gemm_swiglu_pays", list(best)))) == best


def test_tile_shapes_of_short_products():
    """Weight gradients of few tokens (fp32 output: kind 1, bf16: kind 2) and small outputs of many tokens: none of the shapes that
    were measured 10 % or more behind the best (the figures stand at the rule; 1, 2: 256 columns, pairs and single CTAs, 3, 4: 128 and
    64, 5: pairs of 128, 6: swapped)."""
    slow = {(57344, 8192, 100, 1): {1, 4, 5}, (57344, 8192, 200, 1): {4, 5}, (28672, 4096, 333, 1): {4, 5}, (11008, 4096, 333, 1): {4, 5},
            (57344, 8192, 100, 2): {1, 3, 4, 5}, (22016, 4096, 45, 2): {1, 3, 4, 5}, (6144, 4096, 512, 2): {1, 4, 5}, (28672, 4096, 777, 2): {3, 4, 5},
            (28672, 4096, 2048, 1): {2, 3, 4}, (8192, 512, 1408, 0): {1, 4, 6}, (8192, 1536, 512, 0): {4, 5, 6}}
    got = _ask("yf_gemm_plan", [(*k, 0, 0) for k in slow])
    assert {k: g % 16 for k, g in zip(slow, got) if g % 16 in slow[k]} == {}
