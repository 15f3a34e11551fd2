"""Loads the torch extension with the training-step operators (``csrc/torch/ops.cpp``)."""
from __future__ import annotations

import importlib.machinery
import importlib.util
from pathlib import Path

import torch
import torch.distributed as dist
from torch.autograd import forward_ad
from torch.nn.modules import module as _modules
from torch.utils._device import DeviceContext

_module = None


def ops():
    """The extension module. It is built in-tree; a missing one is built now, and a broken one is an error."""
    global _module
    if _module is None:
        from .. import _native  # noqa: F401  (loads libhylink_b200.so first)

        path = Path(__file__).resolve().parent.parent / "lib" / "_hylink_ops.so"
        if not path.exists():
            from .. import _build

            _build.build_torch_ext()
        loader = importlib.machinery.ExtensionFileLoader("_hylink_ops", str(path))
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_hylink_ops", loader))
        loader.exec_module(module)
        _module = module
    return _module


def check_products(device: int | None = None) -> None:
    """Raises, once, if a wait inside one of this library's matrix products on ``device`` (default: the current one) has run out
    since the last call: results that came after it are not valid. To be called where the host has waited for results;
    ``DDPTrainer.step`` does. Launches of further products raise too until then."""
    ops().check_products(-1 if device is None else device)


def alone() -> bool:
    """Whether this process is a job by itself: with several ranks, collectives hold multiprocessors beside the products."""
    return not (dist.is_available() and dist.is_initialized() and dist.get_world_size() > 1)


def overridden(m) -> bool:
    """Whether calling module ``m`` does anything besides its class's ``forward``: hooks, or a ``forward`` of its own."""
    return bool(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks or "forward" in m.__dict__)


def traced() -> bool:
    return torch.compiler.is_compiling() or torch.jit.is_tracing()


def plain_eager(*tensors) -> bool:
    """Whether ordinary eager autograd is all that looks at a call on these tensors. The operators work on addresses and have
    one backward: under tracing and compilation, function transforms (vmap, torch.func), forward-mode differentiation and
    modes that watch every call, and for tensor subclasses, the plain modules run."""
    if any(type(t) is not torch.Tensor and type(t) is not torch.nn.Parameter for t in tensors):
        return False
    if traced() or forward_ad._current_level >= 0:
        return False
    if torch._C._functorch.peek_interpreter_stack() is not None or torch._C._len_torch_dispatch_stack():
        return False
    # a default device is a mode too, one that the operators need not see
    return all(type(torch._C._get_function_stack_at(i)) is DeviceContext for i in range(torch._C._len_torch_function_stack()))


def global_module_hooks() -> bool:
    """Whether hooks on every module's calls are registered."""
    g = _modules
    return bool(g._global_forward_hooks or g._global_forward_pre_hooks or g._global_backward_hooks or g._global_backward_pre_hooks)
