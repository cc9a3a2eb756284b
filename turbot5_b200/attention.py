"""Fused relative-position-bias attention: the functional surface.

Same names, argument meaning and error behaviour as the TurboT5 operators they
replace:

* `flash_attention_with_fusing_bias`         src/turbot5/ops/fused_bias_attention.py:876
* `flash_attention_with_fusing_bias_varlen`  src/turbot5/ops/varlen_fused_bias_attn.py:870

plus the split-KV decoding operator the reference only sketches
(src/turbot5/ops/flash_decoding.py) and a bucket-index check.  Argument checks, allocation, the
launches and the autograd nodes are native (csrc/host/ops.cpp).
"""
from typing import Optional

import torch

from . import _native as nat

_host = nat.host


def device_status(device) -> torch.Tensor:
    """Per-device int32 word the kernels write to when a bounded wait runs out."""
    dev = torch.device(device)
    return _host.device_status(dev.index if dev.index is not None else torch.cuda.current_device())


def check_device_status(device="cuda") -> None:
    """Synchronising check of the status word through the library's `t5b_check_status`: raises
    if a kernel's bounded wait ran out since the last check (and clears the word)."""
    word = device_status(device)
    code = nat.C.c_int32(0)
    with torch.cuda.device(word.device):
        st = nat.lib().t5b_check_status(word.data_ptr(), nat.C.byref(code), nat.stream_ptr(word.device))
    if st == nat.ERR_DEVICE_TIMEOUT:
        raise RuntimeError(f"turbot5_b200 kernel gave up waiting on the device (code {code.value})")
    nat.check(st, "check_device_status")


class _Workspaces:
    """The per-stream scratch buffers kept by the host extension: zero-initialised, one per (kind, device,
    stream); the kernels leave them ready for the next call."""

    @staticmethod
    def items():
        return _host.scratch_items()


_workspaces = _Workspaces()


def flash_attention_with_fusing_bias(q, k, v, bias, causal=False, sm_scale=None,
                                     NUM_BUCKETS=32, MAX_DISTANCE=128, *, q_pos_offset=None,
                                     return_lse=False, kernel="auto", balance_last_wave=True, local_block=None,
                                     window=None):
    """softmax(sm_scale * Q K^T + T5 bias(n - m) [+ causal mask]) V without an L x L tensor; differentiable
    in q, k, v and the bias table (through a node that mirrors `FlashAttentionBias`,
    src/turbot5/ops/fused_bias_attention.py:822-873).

    q (B,H,M,D), k/v (B,H,N,D), any batch/head/row strides (last dim contiguous);
    bias is the [NUM_BUCKETS, H] relative-attention table or None.  `causal`
    selects the mask and unidirectional buckets together, as in the reference.
    `sm_scale=None` means 1/sqrt(D); T5 modules pass 1.0.  The query at row m sits
    at key position `q_pos_offset + m` (default N - M, the cached-decoding
    alignment of the reference's `basic` path; sequence parallel callers pass
    their shard offset).  Returns a tensor with q's shape, dtype and strides.
    `balance_last_wave` lets the kernel split the key range of the query tiles of a partially
    filled last wave of blocks (scratch comes from a per-stream cache).
    `local_block` turns the call into block-local attention (T5LocalAttention: the keys of the three
    neighbouring blocks); `window` into a sliding window |n - query position| < window (tensor-core
    kernels only: bf16/fp16, not causal)."""
    return _host.attention(q, k, v, bias, causal, sm_scale, NUM_BUCKETS, MAX_DISTANCE, q_pos_offset, return_lse,
                           nat.KERNELS[kernel], balance_last_wave, local_block, window, False)


def flash_attention_partial(q, k, v, bias, causal=False, sm_scale=None, NUM_BUCKETS=32, MAX_DISTANCE=128, *,
                            q_pos_offset=0, kernel="auto"):
    """Attention of q over a SLICE of the keys: returns (out, lse) with `out` in float32, for
    `merge_attention_partials`.  `q_pos_offset` is the position of query row 0 relative to the
    slice's first key (absolute query position minus the slice's first key position; may be
    negative).  Forward only."""
    with torch.no_grad():
        try:
            return _host.attention(q, k, v, bias, causal, sm_scale, NUM_BUCKETS, MAX_DISTANCE, q_pos_offset, True,
                                   nat.KERNELS[kernel], True, None, None, True)
        except NotImplementedError:
            # shapes the tensor-core kernels do not take: the partial is rounded to the element type first
            out, lse = _host.attention(q, k, v, bias, causal, sm_scale, NUM_BUCKETS, MAX_DISTANCE, q_pos_offset, True,
                                       nat.KERNELS[kernel], True, None, None, False)
            return out.float(), lse


def merge_attention_partials(parts, dtype, return_lse=False):
    """Combine `(out float32 (B,H,M,D), lse float32 (B,H,M))` pairs computed over disjoint key
    slices into the attention over all of them (one rounding to `dtype`).  The result has the
    layout of the first partial."""
    with torch.no_grad():
        return _host.merge([o for o, _ in parts], [l for _, l in parts], dtype, return_lse)


def flash_attention_with_fusing_bias_varlen(q, k, v, bias, cu_seqlens_q, cu_seqlens_k,
                                            max_seqlen_q, max_seqlen_k, causal=False, sm_scale=None,
                                            NUM_BUCKETS=32, MAX_DISTANCE=128, *, return_lse=False,
                                            kernel="auto", window=None):
    """Packed-sequence variant: q (Tq,H,D), k/v (Tk,H,D), int32 cu_seqlens on the device; differentiable in
    q, k, v and the bias table.  Positions are relative to each sequence.  Tiles are scheduled on the
    device from cu_seqlens: no host loop, no host read of the lengths.  `max_seqlen_*` are accepted for
    signature compatibility (bounds for scheduling only).  `window`: sliding window
    |n - query position| < window inside every sequence (tensor-core kernels only).

    q, k and v may have more rows than `cu_seqlens[-1]` (buffers sized for the worst case): those rows
    are never attended and the matching output rows are not written, but the rows of k and v must
    hold finite numbers -- the last tile of the last sequence can load them, a masked key has
    probability 0, and 0 x NaN is NaN."""
    return _host.attention_packed(q, k, v, bias, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, causal, sm_scale,
                                  NUM_BUCKETS, MAX_DISTANCE, return_lse, nat.KERNELS[kernel], window)


def flash_decoding_with_fusing_bias(q, k, v, bias, causal=False, sm_scale=None, NUM_BUCKETS=32,
                                    MAX_DISTANCE=128, *, kv_len=None, seqlens_k=None,
                                    q_pos_offset=None, num_splits=0, workspace=None):
    """Split-KV decoding step: q (B,H,M,D) with small M against a K/V cache (B,H,cap,D).

    Only the first `kv_len` keys (default: all) -- or `seqlens_k[b]` keys per batch
    row, an int32 device tensor -- are attended.  Query row m sits at key position
    kv_len - M + m unless `q_pos_offset` is given; `causal` gives the decoder
    self-attention mask and unidirectional buckets, cross attention passes
    bias=None, causal=False.  One launch: the last block per (batch, head) merges
    the splits.  Scratch comes from a per-stream cache unless `workspace` is given.
    """
    return _host.decode(q, k, v, bias, causal, sm_scale, NUM_BUCKETS, MAX_DISTANCE, kv_len, seqlens_k, q_pos_offset,
                        num_splits, workspace)


def relative_position_bucket_table(num_buckets=32, max_distance=128, bidirectional=True,
                                   lo=None, hi=None) -> torch.Tensor:
    """bucket(delta) for delta in [lo, hi] as an int32 CPU tensor (host table of the library)."""
    lo = -max_distance - 1 if lo is None else int(lo)
    hi = max_distance + 1 if hi is None else int(hi)
    out = torch.empty(hi - lo + 1, dtype=torch.int32)
    nat.check(nat.lib().t5b_bucket_table_host(int(num_buckets), int(max_distance), int(bool(bidirectional)),
                                              lo, hi, out.data_ptr()), "relative_position_bucket_table")
    return out


def relative_position_bucket_grid(M, N, q_pos_offset=0, bidirectional=True, num_buckets=32,
                                  max_distance=128, device="cuda") -> torch.Tensor:
    """(M, N) int32 bucket indices computed by the device lookup the kernels use."""
    out = torch.empty((M, N), dtype=torch.int32, device=device)
    with torch.cuda.device(out.device):
        nat.check(nat.lib().t5b_bucket_indices(out.data_ptr(), M, N, int(q_pos_offset), int(bool(bidirectional)),
                                               int(num_buckets), int(max_distance), nat.stream_ptr(out.device)),
                  "relative_position_bucket_grid")
    return out
