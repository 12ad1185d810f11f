"""Fused decode attention over a compressed cache plus the dense recent window.

``attention`` keeps the reference signature and checks
(reskv/_attention.py:10-144).  The dense window is folded into the same two
launches as the compressed tokens (partial kernel + merge kernel) instead of the
reference's extra ``bmm`` + ``mul_`` + merge kernel, and read where it lies: the
leading tokens of a longer buffer need no copy.  The tensor checks, allocations
and launches are native (``csrc/host.cpp``).
"""

from __future__ import annotations

import torch

from ._extension import LAYOUT_IDS, host, require_device
from .config import _reference_schedule
from .tensors import CompressedKV


def attention(
    query: torch.Tensor,
    cache: CompressedKV,
    *,
    position: int,
    start_position: int = 0,
    rope_theta: float = 500000.0,
    inv_freq: torch.Tensor | None = None,
    scaling: float | None = None,
    recent: tuple[torch.Tensor, torch.Tensor, torch.Tensor] | None = None,
):
    """Decode raw Q against compressed pre-RoPE K and V.

    ``query`` is FP16 ``[B,H,1,128]`` before RoPE; ``recent`` is ``(rotated Q,
    rotated K, V)`` of the dense window; ``inv_freq`` holds the model's 64 RoPE
    frequencies (omit it to derive them from ``rope_theta``).  Returns FP16
    ``[B,H,1,128]``.
    """
    key, value = cache.key, cache.value
    plan = key.plan
    if plan is not value.plan and plan != value.plan:
        raise ValueError("K and V plans differ")
    if isinstance(query, torch.Tensor) and query.is_cuda:
        require_device(query.get_device())
    # A plan from ``resolve()`` carries the split count of the reference's schedule table, which was tuned
    # for other kernels on another GPU: such a plan gets this library's own schedule (0).  A split count that
    # differs from the table entry was chosen by the caller and is passed on.
    splits = plan.splits
    if splits and plan.layout != "compact" and splits == _reference_schedule(
            plan.layout, plan.centroid_fusion, plan.bits, query.shape[0])[1]:
        splits = 0
    return host().attention(query, key.centroids, key._native, value._native, LAYOUT_IDS[plan.layout], plan.bits, position,
                            start_position, rope_theta, inv_freq, scaling, recent, splits)
