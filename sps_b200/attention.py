"""Prefill attention of the SPS model family on sm_100a, behind the reference's call signatures.

``sps_sliding_attention``, ``reverse_sps_sliding_attention`` and ``full_attention`` take the
same arguments, in the same order and with the same meaning, as the reference's
src/modeling/models/attention/triton_sps_flash_attention.py:725-753,
triton_reverse_sps_flash_attention.py:827-853 and triton_full_flash_attention.py:679-709, so the
model classes can call them unchanged (see ``sps_b200.install``).  For head_dim 64 and 128 they
are differentiable like the reference's ``torch.autograd.Function``s (backward:
triton_sps_flash_attention.py:623-720); the other head dims are forward only.
All compute happens in libspsattn.so (tcgen05 / TMA kernels for every head_dim), the host path in
native code as well (csrc/native.cpp).
"""

from __future__ import annotations

from typing import Optional

import torch

from . import _lib

def _status(device: torch.device) -> torch.Tensor:
    """Per-device int32 word of STATUS bits: a bounded wait that expired, an input outside its range."""
    return _lib.native().status_word(device.index if device.index is not None else torch.cuda.current_device())


def check_device_status(device=None) -> None:
    """Synchronise and raise if any kernel reported a failure (a bounded wait that expired, a token id
    outside the vocabulary)."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    word = _status(dev)
    code = int(word.item())
    if code != 0:
        word.zero_()
        what = [text for bit, text in ((_lib.STATUS_WAIT_EXPIRED, "a bounded wait expired"),
                                       (_lib.STATUS_BAD_TOKEN, "a token id outside the vocabulary")) if code & bit]
        raise _lib.SpsAttnError(f"device reported status {code} ({', '.join(what)})")


def _dtype_code(t: torch.Tensor) -> int:
    if t.dtype == torch.bfloat16:
        return _lib.DTYPE_BF16
    if t.dtype == torch.float16:
        return _lib.DTYPE_FP16
    raise TypeError(f"sps_b200 attention computes in bf16 or fp16, got {t.dtype}")


def prefill_attention_backward(
    q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, o: torch.Tensor, lse: torch.Tensor,
    d_o: torch.Tensor, sm_scale: float, *, persistent_parity: int, temporary_window: int = 0,
    persistent_window: Optional[int] = None, documents_idx: Optional[torch.Tensor] = None,
    mask_flags: int = 0,
):
    """dQ, dK, dV of ``prefill_attention`` from dO, the forward output ``o`` and its ``lse``
    (the reference's backward: triton_sps_flash_attention.py:623-720).  head_dim 64 or 128."""
    return _lib.native().prefill_backward(q, k, v, o, lse, d_o, sm_scale, persistent_parity, int(temporary_window),
                                          persistent_window, mask_flags, documents_idx)


def prefill_attention(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    sm_scale: float,
    *,
    persistent_parity: int,
    temporary_window: int = 0,
    persistent_window: Optional[int] = None,
    documents_idx: Optional[torch.Tensor] = None,
    mask_flags: int = 0,
    return_lse: bool = False,
    out: Optional[torch.Tensor] = None,
):
    """Masked attention over [B, H, N, D] tensors; the general entry the three wrappers share.

    ``persistent_parity``: 0 (SPS), 1 (Reverse-SPS / Delayed-State) or -1 (Standard).
    Returns O (same dtype as q) and, with ``return_lse``, the base-2 log-sum-exp [B, H, N] fp32.
    When an input requires grad (head_dim 64 or 128) the result is differentiable.
    """
    return _lib.native().prefill(q, k, v, sm_scale, persistent_parity, int(temporary_window), persistent_window,
                                 mask_flags, documents_idx, return_lse, out)


def sps_sliding_attention(q, k, v, sm_scale, temporary_key_window, warp_specialize=True,
                          documents_idx_BxT=None, persistent_key_window=None):
    """SPS variant: the persistent (window-exempt) key is the even / input slot, the <predict>
    slot is windowed.  ``warp_specialize`` is accepted for signature compatibility and ignored.
    """
    return _lib.native().prefill(q, k, v, sm_scale, _lib.PARITY_EVEN, int(temporary_key_window),
                                 persistent_key_window, 0, documents_idx_BxT, False, None)


def reverse_sps_sliding_attention(q, k, v, sm_scale, temporary_key_window, warp_specialize=True,
                                  documents_idx_BxT=None, persistent_key_window=None):
    """Reverse-SPS / Delayed-State variant: the persistent key is the odd slot."""
    return _lib.native().prefill(q, k, v, sm_scale, _lib.PARITY_ODD, int(temporary_key_window),
                                 persistent_key_window, 0, documents_idx_BxT, False, None)


def full_attention(q, k, v, sm_scale, warp_specialize=True, documents_idx_BxT=None):
    """Standard model: causal attention with an optional same-document mask."""
    return _lib.native().prefill(q, k, v, sm_scale, _lib.PARITY_NONE, 0, None, 0, documents_idx_BxT, False, None)


def visibility(n_ctx: int, *, persistent_parity: int, temporary_window: int = 0,
               persistent_window: Optional[int] = None, documents_idx: Optional[torch.Tensor] = None,
               mask_flags: int = 0, batch: int = 1, device="cuda") -> torch.Tensor:
    """The boolean mask the kernels apply, evaluated on the device ([B, N, N] bool); test hook."""
    lib = _lib.load()
    dev = torch.device(device)
    B = batch if documents_idx is None else documents_idx.shape[0]
    vis = torch.empty((B, n_ctx, n_ctx), dtype=torch.uint8, device=dev)
    docs_ptr, docs_i64, sb, st, ws, ws_bytes = None, 0, 0, 0, None, 0
    if documents_idx is not None:
        docs = documents_idx.to(dev)
        if docs.dtype not in (torch.int64, torch.int32):
            docs = docs.to(torch.int64)
        docs_ptr, docs_i64 = docs.data_ptr(), int(docs.dtype == torch.int64)
        sb, st = docs.stride()
        ws_bytes = lib.spsattn_prefill_workspace_bytes(B, 1, n_ctx, 64)
        ws = torch.empty(ws_bytes, dtype=torch.uint8, device=dev)
    pw = _lib.NO_WINDOW if persistent_window is None else max(-1, min(int(persistent_window), n_ctx))
    with torch.cuda.device(dev):
        rc = lib.spsattn_debug_visibility(
            vis.data_ptr(), docs_ptr, docs_i64, sb, st, B, n_ctx, int(persistent_parity),
            max(-1, min(int(temporary_window), n_ctx)), pw, int(mask_flags),
            None if ws is None else ws.data_ptr(), ws_bytes, torch.cuda.current_stream().cuda_stream)
    _lib.check(rc, "spsattn_debug_visibility")
    return vis.bool()


_X_DTYPES = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}


def rope_cast(x_BxNxHxD: torch.Tensor, freqs_cis: Optional[torch.Tensor], *,
              out_dtype: torch.dtype = torch.bfloat16) -> torch.Tensor:
    """Rotary embedding (``freqs_cis`` complex64 [N, D/2] or [B, N, D/2]; None = cast only) and
    cast of one projection in a single pass.  Input: a [B, N, H, D] view (any of bf16 / fp16 /
    fp32, row strides free).  Returns the attention operand as a [B, H, N, D] view of a
    token-major buffer, which the prefill kernel reads in place.  One kernel instead of the
    float / complex / multiply / cast / transpose chain of model.py:201-230 and sps/core.py:45-55.
    """
    lib = _lib.load()
    x = x_BxNxHxD
    if not x.is_cuda:
        raise RuntimeError("rope_cast needs CUDA tensors")
    B, N, H, D = x.shape
    if x.dtype not in _X_DTYPES:
        raise TypeError(f"unsupported projection dtype {x.dtype}")
    align = 4 if x.dtype == torch.float32 else 8
    if x.stride(3) != 1 or any(s % align for s in x.stride()[:3]) or x.data_ptr() % 16:
        x = x.contiguous()
    out = torch.empty((B, N, H, D), dtype=out_dtype, device=x.device)
    f_ptr, f_sb = None, 0
    if freqs_cis is not None:
        f = torch.view_as_real(freqs_cis.to(torch.complex64)).contiguous()    # [.., N, D/2, 2] fp32
        assert f.shape[-3:] == (N, D // 2, 2), f"freqs_cis must be [N, D/2] or [B, N, D/2], got {tuple(freqs_cis.shape)}"
        if f.dim() == 4:
            assert f.shape[0] == B
            f_sb = N * (D // 2)
        f_ptr = f.data_ptr()
    with torch.cuda.device(x.device):
        rc = lib.spsattn_rope_cast(x.data_ptr(), _X_DTYPES[x.dtype], x.stride(0), x.stride(1), x.stride(2),
                                   f_ptr, f_sb, out.data_ptr(), _dtype_code(out), out.stride(0), out.stride(1),
                                   out.stride(2), B, N, H, D, int(freqs_cis is not None),
                                   torch.cuda.current_stream().cuda_stream)
    _lib.check(rc, "spsattn_rope_cast")
    return out.transpose(1, 2)
