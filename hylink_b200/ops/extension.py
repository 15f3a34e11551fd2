"""Loads the torch extension with the training-step operators (``csrc/torch/ops.cpp``)."""
from __future__ import annotations

import importlib.machinery
import importlib.util
from pathlib import Path

_module = None


def ops():
    """The extension module. It is built in-tree; a missing one is built now, and a broken one is an error."""
    global _module
    if _module is None:
        import torch  # noqa: F401  (the extension links against it)

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


def is_half_cuda(*tensors) -> bool:
    """Whether all tensors are CUDA tensors of one 16-bit float type."""
    import torch

    dt = tensors[0].dtype
    return dt in (torch.bfloat16, torch.float16) and all(t.is_cuda and t.dtype == dt for t in tensors)


def overridden(m) -> bool:
    """Whether calling module ``m`` does anything besides its class's ``forward``: hooks, or a ``forward`` of its own."""
    return bool(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks or "forward" in m.__dict__)
