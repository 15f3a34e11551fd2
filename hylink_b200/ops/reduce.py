"""Landing reduce: ``dst = scale * op(src_0..src_{k-1})`` in one pass."""
from __future__ import annotations

from typing import Sequence

import torch

from .._native import OPS, check
from .extension import ops


def reduce_landing(dst: torch.Tensor, srcs: Sequence[torch.Tensor], op: str = "sum", scale: float = 1.0,
                   accumulate: bool = False, blocks: int = 0) -> torch.Tensor:
    """Reduce up to eight same-typed sources into ``dst`` with the sm_100a kernel.

    Sources may be CUDA tensors or pinned host tensors (read over PCIe by the
    kernel itself). With ``accumulate`` the previous content of ``dst`` is the
    first operand.
    """
    code = ops().reduce_landing(dst, srcs, OPS[op], scale, accumulate, blocks)
    if code:
        check(code, "hlReduceLanding")
    return dst
