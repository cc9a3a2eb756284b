"""Unpad / pad glue for padded batches, computed on the device with no host read-back.

Mirrors `_get_unpad_data`, `index_first_axis`, `_upad_input` and `pad_input` of
src/turbot5/model/padding.py (:79-88, :46-76, :113-150, :30-44).  The reference
reads the longest length back to the host (`.item()`, padding.py:82); here the
packed buffers are sized for the worst case (B*L rows) and the kernels take the
lengths from the device, so a forward pass never synchronises.
"""
from typing import NamedTuple

import torch

from . import _native as nat

_host = nat.host


class UnpadPlan(NamedTuple):
    seqlens: torch.Tensor      # int32 (B,)
    cu_seqlens: torch.Tensor   # int32 (B+1,)
    dest: torch.Tensor         # int32 (B*L,): packed row of each kept token, negative for padding
    batch: int
    seqlen: int


def get_unpad_plan(attention_mask: torch.Tensor) -> UnpadPlan:
    """mask (B, L), non-zero = keep -> lengths, cumulative lengths, destination rows."""
    return UnpadPlan(*_host.unpad_plan(attention_mask), *attention_mask.shape)


def unpad_rows(x: torch.Tensor, plan: UnpadPlan) -> torch.Tensor:
    """(B, L, ...) -> packed (B*L, ...): kept tokens first, in order; the unused tail is zero.
    Differentiable: the gradient is the scatter back (`pad_rows`)."""
    return _host.rows(x, plan.dest, plan.batch, plan.seqlen, True)


def pad_rows(packed: torch.Tensor, plan: UnpadPlan) -> torch.Tensor:
    """packed (>= total kept rows, ...) -> (B, L, ...) with zeros at padded positions.
    Differentiable: the gradient is the gather (`unpad_rows`)."""
    return _host.rows(packed, plan.dest, plan.batch, plan.seqlen, False)
