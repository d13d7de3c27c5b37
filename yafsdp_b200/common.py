"""Small shared definitions: mesh info, training states, the library logger.

Parity: ``ya_fsdp/_common.py:13-74``.
"""

from __future__ import annotations

import contextlib
import ctypes
import enum
import logging
import os
import traceback
from dataclasses import dataclass
from typing import Any, Callable

import torch
import torch.distributed as dist
from torch.distributed.device_mesh import DeviceMesh

logger = logging.getLogger("yafsdp_b200")

_NO_LABEL = contextlib.nullcontext()


def _observers() -> "Callable[[], bool]":
    """``at::hasCallbacks``: whether anything observes ``record_function`` ranges on this thread (a profiler, an execution-trace
    observer, an on-demand trace).  PyTorch exports it from its C++ library only; without it the answer is always yes."""
    try:
        has = ctypes.CDLL(os.path.join(os.path.dirname(torch.__file__), "lib", "libtorch_cpu.so"))._ZN2at12hasCallbacksEv
    except (OSError, AttributeError):
        return lambda: True
    has.restype, has.argtypes = ctypes.c_bool, []
    return has  # type: ignore[no-any-return]


_observed = _observers()


def phase_label(name: str, of: str = "") -> Any:
    """``record_function`` range ``name (of)`` where something would see it, nothing otherwise: entering and leaving a range
    costs 4 to 12 us of host time, 35 times in a step of a two-layer model; the question 0.4 us."""
    if not _observed():
        return _NO_LABEL
    return torch.profiler.record_function(f"{name} ({of})" if of else name)


class TrainingState(enum.Enum):
    """State of one ``fully_shard`` group inside a training step."""

    FORWARD = enum.auto()
    PRE_BACKWARD = enum.auto()
    POST_BACKWARD = enum.auto()
    IDLE = enum.auto()


@dataclass
class ShardMeshInfo:
    """The 1-D mesh a group is sharded over."""

    mesh: DeviceMesh
    shard_mesh_dim: int = 0

    def __post_init__(self) -> None:
        self.shard_process_group: dist.ProcessGroup = self.mesh.get_group(self.shard_mesh_dim)
        self.shard_mesh_size: int = self.mesh.size(self.shard_mesh_dim)
        self.shard_mesh_rank: int = self.shard_process_group.rank()


def raise_assert_with_print(*args: Any, **kwargs: Any) -> None:
    rank = dist.get_rank() if dist.is_initialized() else 0
    print(f"[Rank {rank}] ", end="")
    print(*args, **kwargs)
    traceback.print_stack()
    raise AssertionError(*args, **kwargs)


def cast_fp_tensor(dtype: torch.dtype, x: Any) -> Any:
    if not isinstance(x, torch.Tensor) or not torch.is_floating_point(x) or x.dtype == dtype:
        return x
    return x.to(dtype)


def is_backward_running() -> bool:
    """True while the autograd engine is executing a backward pass on this thread."""
    return torch._C._current_graph_task_id() != -1
