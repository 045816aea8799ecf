"""Segmented decode attention and the decode KV-cache update on sm_100a, behind the
reference's call signatures (src/modeling/models/utils/decode_attention.py and
decode_attention_fast.py).  All compute happens in libspsattn.so; there is no fallback.
"""

from __future__ import annotations

from dataclasses import dataclass
from typing import Optional, Sequence

import torch
from torch import Tensor

from . import _lib


@dataclass
class KVSegment:
    """A block of keys/values with per-element validity lengths
    (same fields as decode_attention.py:21-32).

    k, v: [B, H, max_T, D]; lengths: [B, H] (per head) or [B]; max_len_cap: optional host cap
    on the rows scanned.
    """
    k: Tensor
    v: Tensor
    lengths: Tensor
    max_len_cap: Optional[int] = None


@dataclass
class PackedKVSegment:
    """A cache that is not a dense [B, H, max_T, D] block: row r of (sequence s, head h) is at
    element offset ``seq_offset[s] + h * head_stride + r * row_stride`` of ``k`` / ``v``.
    ``lengths`` is [S] or [S, H] int64; ``max_rows`` caps the rows scanned (host int).
    """
    k: Tensor
    v: Tensor
    seq_offset: Tensor
    head_stride: int
    row_stride: int
    lengths: Tensor
    max_rows: int


def decode_attention(
    q: Tensor,                                   # [S, nq, H, D]
    segments: Sequence,                          # KVSegment | PackedKVSegment, with query masks
    extras: Sequence[tuple],                     # (k [S,H,D], v [S,H,D], query_mask)
    *,
    segment_query_masks: Optional[Sequence[int]] = None,
    sm_scale: Optional[float] = None,
) -> Tensor:
    """nq (1 or 2) queries per (sequence, head) over the live rows of every segment plus the
    extra single-token entries; returns fp32 [S, nq, H, D].  Bit i of a query mask says whether
    query slot i sees that segment / entry."""
    return _lib.native().decode(q, segments, extras, segment_query_masks, sm_scale)


def segmented_q2_attention(
    q_Bx2xHxD: Tensor,
    segments: list,
    *,
    current_normal_k_BxHxD: Tensor,
    current_normal_v_BxHxD: Tensor,
    current_predict_k_BxHxD: Tensor,
    current_predict_v_BxHxD: Tensor,
    attn_dtype: torch.dtype,
) -> Tensor:
    """q=2 segmented decode attention for SPS-family generation (decode_attention.py:483-594).

    Slot 0 attends over the segments plus the current normal key; slot 1 over the same
    segments plus current normal and current predict.  Fail-fast like the reference.
    """
    return _lib.native().decode_q2(q_Bx2xHxD, segments, current_normal_k_BxHxD, current_normal_v_BxHxD,
                                   current_predict_k_BxHxD, current_predict_v_BxHxD, attn_dtype)


# the name the reference binds (src/modeling/models/reverse_sps/inference.py:354)
triton_segmented_q2_attention = segmented_q2_attention


def segmented_q1_attention(q_BxHxD: Tensor, segments: list, *, extra_kv=None,
                           attn_dtype: torch.dtype) -> Tensor:
    """q=1 variant: up to 3 segments and 2 always-valid extra entries (decode_attention.py:393-480)."""
    return _lib.native().decode_q1(q_BxHxD, segments, extra_kv, attn_dtype)


def masked_kv_attention(q_BxHxD: Tensor, segments: list, *, extra_kv=None, attn_dtype: torch.dtype,
                        check_finite: bool = False, error_context: str = "",
                        prefer_triton: bool = False, require_triton: bool = False) -> Tensor:
    """Attention of one query per (batch, head) over variable-length KV segments
    (decode_attention.py:597-704).  Always runs the CUDA kernel; ``prefer_triton`` /
    ``require_triton`` are accepted for signature compatibility."""
    out = _lib.native().decode_q1(q_BxHxD, segments, extra_kv, attn_dtype)
    if check_finite and not torch.isfinite(out).all():
        raise RuntimeError(f"Non-finite attention output{error_context}")
    return out


def fused_sps_kv_update(*, nw_k: Tensor, nw_v: Tensor, nw_len: Tensor, nw_pos: Tensor,
                        br_k: Tensor, br_v: Tensor, br_len: Tensor,
                        k_window_BxHxD: Tensor, v_window_BxHxD: Tensor,
                        k_retained_BxHxD: Tensor, v_retained_BxHxD: Tensor,
                        active_mask_B: Tensor, window_tokens: int) -> None:
    """Single-launch in-place KV update for SPS-family decode (decode_attention_fast.py:139-221)."""
    _lib.native().kv_update(nw_k, nw_v, nw_len, nw_pos, br_k, br_v, br_len, k_window_BxHxD, v_window_BxHxD,
                            k_retained_BxHxD, v_retained_BxHxD, active_mask_B, window_tokens)


def fill_decode_caches(k_Bx2TxHxD: Tensor, v_Bx2TxHxD: Tensor, current_doc_mask_BxT: Tensor, *,
                       br_k: Tensor, br_v: Tensor, br_len: Tensor,
                       nw_k: Optional[Tensor] = None, nw_v: Optional[Tensor] = None,
                       nw_len: Optional[Tensor] = None, nw_pos: Optional[Tensor] = None,
                       window_tokens: int = 0, retained_slot: int = 0, window_slot: int = 1) -> None:
    """Fill one layer's decode caches from the prefill K/V in one launch, no host sync
    (what reverse_sps/inference.py:568-613 does with a Python loop over batch rows).

    ``retained_slot`` / ``window_slot``: parity of the doubled-sequence row that feeds the retained
    cache / the ring (SPS: 0 and 1; Reverse-SPS and Delayed-State: 1 and 0).
    """
    lib = _lib.load()
    B, two_t, H, D = k_Bx2TxHxD.shape
    T = two_t // 2
    k = k_Bx2TxHxD.to(br_k.dtype)
    v = v_Bx2TxHxD.to(br_v.dtype)
    if k.stride(3) != 1 or any(s % 8 for s in k.stride()[:3]):
        k = k.contiguous()
    if v.stride() != k.stride():
        v = v.contiguous()
        k = k.contiguous()
    assert br_k.element_size() == 2, "caches hold 16-bit elements"
    assert br_k.is_contiguous() and br_v.is_contiguous() and br_len.is_contiguous()
    assert br_len.dtype == torch.int64 and tuple(br_len.shape) == (B, H)
    mask = current_doc_mask_BxT.to(torch.uint8).contiguous()
    assert tuple(mask.shape) == (B, T)
    ring = [None, None, None, None]
    window_storage = 0
    if window_tokens > 0:
        assert nw_k.is_contiguous() and nw_v.is_contiguous()
        assert nw_len.dtype == torch.int64 and nw_pos.dtype == torch.int64
        window_storage = int(nw_k.size(2))
        ring = [nw_k.data_ptr(), nw_v.data_ptr(), nw_len.data_ptr(), nw_pos.data_ptr()]
    with torch.cuda.device(k.device):
        rc = lib.spsattn_fill_decode_caches(
            k.data_ptr(), v.data_ptr(), k.stride(0), k.stride(1), k.stride(2), mask.data_ptr(),
            br_k.data_ptr(), br_v.data_ptr(), br_len.data_ptr(), ring[0], ring[1], ring[2], ring[3],
            B, T, H, D, int(br_k.size(2)), window_storage, int(window_tokens), int(retained_slot),
            int(window_slot), torch.cuda.current_stream().cuda_stream)
    _lib.check(rc, "spsattn_fill_decode_caches")
