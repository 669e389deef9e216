"""DS4 decode-side cache operators with the reference's names
(reference: src/moespresso/runtime/deepseek_v4/decode_attention_kernel.py).

``fp8_kv_prefix_rows``   E4M3FN round trip of the non-rotary prefix of 512-wide compressed-KV rows (:587-619)

``fused_decode_prep``    QAT of q, scores, exact top-k, and the prepared KV row (rope tail + FP8 round trip) (:669-730)
``fused_decode_sdpa``    rope on q, attention over the window (with the prepared row) and the selected rows, sink,
                         inverse rope (:733-786)

Each fused operator is one call of the library and a few launches (the reference runs each as one Metal launch);
``params`` is read on the device, so neither synchronises with the host and both can be captured in a CUDA graph.
"""
from __future__ import annotations

import ctypes as C

import torch

from .. import _abi
from .. import _torchabi as _t
from .._torchabi import native, ptr, require_cuda

_HEAD_DIM = 512


def fp8_kv_prefix_rows(x, *, replay: bool = False):
    """``x`` ``[..., 512]`` float32 -> float32 of the same shape: dims [0, 448) through DS4's E4M3FN round trip
    (power-of-two scale per 64-element block), dims [448, 512) unchanged.  ``replay=True`` evaluates the
    reference's NumPy replay form instead (compressor_diff.py:74-86: exact power-of-two scale, ties to even)."""
    if x.ndim < 1 or int(x.shape[-1]) != _HEAD_DIM:
        raise ValueError("fp8 rows expect 512-wide rows")
    if x.dtype != torch.float32:
        raise ValueError("fp8 rows must be float32")
    dev = require_cuda(x)
    rows2d = x.reshape(-1, _HEAD_DIM).contiguous()
    n_rows = int(rows2d.shape[0])
    if n_rows == 0:
        raise ValueError("fp8 rows expect at least one row")
    out = torch.empty((n_rows, _HEAD_DIM), dtype=torch.float32, device=dev)
    a = _abi.Fp8KvRowsArgs()
    a.x, a.out, a.n_rows, a.width, a.mode = ptr(rows2d), ptr(out), n_rows, _HEAD_DIM, 1 if replay else 0
    _abi.check(_t.launch("fp8_kv_rows", _abi.load().mxb_fp8_kv_rows, a))
    return out.reshape(x.shape)


_INDEX_HEAD_DIM = 128
_MAX_HEADS = 64
_ROPE_DIM = 64


def _token_operands(inv_freq, params, need):
    """inv_freq float32 [32] and params int32 / int64 [>= need], contiguous, with the int64 flag."""
    if int(inv_freq.numel()) != _ROPE_DIM // 2:
        raise ValueError("inv_freq must hold rope_dim / 2 values")
    if int(params.numel()) < need:
        raise ValueError("params must hold the token position and the write index")
    if params.dtype not in (torch.int32, torch.int64):
        params = params.to(torch.int64)
    return inv_freq.contiguous(), params.contiguous(), 1 if params.dtype == torch.int64 else 0


def fused_decode_prep(q_idx, pooled_qat, weights, kv_row, inv_freq, params, *, scale, topk):
    """Score, select, and prepare the KV row for one ratio-4 decode token (reference: :669-730).

    q_idx ``[n_heads, 128]`` (float32 / float16 / bfloat16, post-rope, pre-QAT), pooled_qat float32
    ``[n_rows, 128]``, weights float32 ``[n_heads]`` (already times ``n_heads ** -0.5``), kv_row float16 ``[512]``
    (post-norm, pre-rope), inv_freq float32 ``[32]``, params int32 with the token position first.
    Returns ``(sel int32 [topk], row float16 [512], scores float32 [n_rows])``: the selected pool rows (the exact
    top-k with ties to the lower row; ids ASCENDING here, where the reference emits the strictly-above rows first
    and the boundary ties after them — the same set), the roped and FP8-rounded KV row, and the scores.
    Three launches: everything that precedes the scan, the exact fp32 scores, the top-k."""
    r = native("fused_decode_prep", q_idx, pooled_qat, weights, kv_row, inv_freq, params, scale, topk)
    if r is not None:
        return r
    if q_idx.ndim != 2 or int(q_idx.shape[1]) != _INDEX_HEAD_DIM:
        raise ValueError("q_idx must have shape [n_heads, 128]")
    n_heads = int(q_idx.shape[0])
    if n_heads <= 0 or n_heads > _MAX_HEADS:
        raise ValueError("q_idx must carry between 1 and 64 heads")
    if q_idx.dtype not in (torch.float32, torch.float16, torch.bfloat16):
        raise ValueError("q_idx must be float32, float16, or bfloat16")
    if pooled_qat.ndim != 2 or int(pooled_qat.shape[1]) != _INDEX_HEAD_DIM or pooled_qat.dtype != torch.float32:
        raise ValueError("pooled_qat must be float32 [n_rows, 128]")
    n_rows = int(pooled_qat.shape[0])
    topk = int(topk)
    if not 0 < topk < n_rows:
        raise ValueError("topk must be positive and smaller than n_rows")
    if tuple(int(v) for v in weights.shape) != (n_heads,) or weights.dtype != torch.float32:
        raise ValueError("weights must be float32 [n_heads]")
    if tuple(int(v) for v in kv_row.shape) != (_HEAD_DIM,) or kv_row.dtype != torch.float16:
        raise ValueError("kv_row must be float16 [512]")
    if int(inv_freq.shape[-1]) != _ROPE_DIM // 2 or inv_freq.dtype != torch.float32:
        raise ValueError("inv_freq must be float32 [32]")
    dev = require_cuda(q_idx, pooled_qat, weights, kv_row, inv_freq, params)
    inv_freq, params, wide = _token_operands(inv_freq, params, 1)
    q_idx, pooled_qat, weights, kv_row = (t.contiguous() for t in (q_idx, pooled_qat, weights, kv_row))
    lib = _abi.load()
    a = _abi.FusedDecodePrepArgs()
    a.q_idx, a.q_dtype, a.pooled_qat, a.weights = ptr(q_idx), _t.dtype_code(q_idx), ptr(pooled_qat), ptr(weights)
    a.kv_row, a.inv_freq, a.params, a.params_int64 = ptr(kv_row), ptr(inv_freq), ptr(params), wide
    a.scale, a.n_heads, a.topk, a.n_rows = float(scale), n_heads, topk, n_rows
    sel = torch.empty((topk,), dtype=torch.int32, device=dev)
    row = torch.empty((_HEAD_DIM,), dtype=torch.float16, device=dev)
    scores = torch.empty((n_rows,), dtype=torch.float32, device=dev)
    ws = _t.workspace(lib.mxb_fused_decode_prep_workspace_bytes(C.byref(a)), dev)
    a.sel, a.row, a.scores, a.workspace, a.workspace_bytes = ptr(sel), ptr(row), ptr(scores), ptr(ws), ws.numel()
    _abi.check(_t.launch("fused_decode_prep", lib.mxb_fused_decode_prep, a))
    return sel, row, scores


def fused_decode_sdpa(q, window, row, pooled, sel, sinks, inv_freq, params, *, scale):
    """Attend one decode token over the window and the selected pooled rows (reference: :733-786).

    q float16 ``[n_heads, 512]`` (post-norm, pre-rope), window float16 ``[window_rows, 512]`` (pre-update), row
    float16 ``[512]`` (from ``fused_decode_prep``; replaces ``window[write_idx]``), pooled float16 ``[n_rows, 512]``,
    sel int32 ``[topk]``, sinks float16 ``[n_heads]``, inv_freq float32 ``[32]``, params int32
    ``[position, write_idx]``.  Every window row and every selected row is a key and a value; the sink joins the
    maximum and the denominator once.  Returns float16 ``[n_heads, 512]`` after the inverse rope.
    Launches: the operands (rope, window, sinks), the attention (and its merge, where its splits are not one cluster), the
    inverse rope."""
    r = native("fused_decode_sdpa", q, window, row, pooled, sel, sinks, inv_freq, params, scale)
    if r is not None:
        return r
    if q.ndim != 2 or int(q.shape[1]) != _HEAD_DIM or q.dtype != torch.float16:
        raise ValueError("q must be float16 [n_heads, 512]")
    n_heads = int(q.shape[0])
    if n_heads <= 0:
        raise ValueError("q must carry at least one head")
    if window.ndim != 2 or int(window.shape[1]) != _HEAD_DIM or window.dtype != torch.float16:
        raise ValueError("window must be float16 [window_rows, 512]")
    if tuple(int(v) for v in row.shape) != (_HEAD_DIM,) or row.dtype != torch.float16:
        raise ValueError("row must be float16 [512]")
    if pooled.ndim != 2 or int(pooled.shape[1]) != _HEAD_DIM or pooled.dtype != torch.float16:
        raise ValueError("pooled must be float16 [n_rows, 512]")
    if sel.ndim != 1 or sel.dtype != torch.int32:
        raise ValueError("sel must be int32 [topk]")
    if tuple(int(v) for v in sinks.shape) != (n_heads,) or sinks.dtype != torch.float16:
        raise ValueError("sinks must be float16 [n_heads]")
    if int(inv_freq.shape[-1]) != _ROPE_DIM // 2 or inv_freq.dtype != torch.float32:
        raise ValueError("inv_freq must be float32 [32]")
    dev = require_cuda(q, window, row, pooled, sel, sinks, inv_freq, params)
    inv_freq, params, wide = _token_operands(inv_freq, params, 2)
    q, window, row, pooled, sel, sinks = (t.contiguous() for t in (q, window, row, pooled, sel, sinks))
    lib = _abi.load()
    a = _abi.FusedDecodeSdpaArgs()
    a.q, a.window, a.row, a.pooled, a.sel, a.sinks = ptr(q), ptr(window), ptr(row), ptr(pooled), ptr(sel), ptr(sinks)
    a.inv_freq, a.params, a.params_int64, a.scale = ptr(inv_freq), ptr(params), wide, float(scale)
    a.n_heads, a.window_rows, a.topk, a.n_rows = n_heads, int(window.shape[0]), int(sel.shape[0]), int(pooled.shape[0])
    out = torch.empty((n_heads, _HEAD_DIM), dtype=torch.float16, device=dev)
    ws = _t.workspace(lib.mxb_fused_decode_sdpa_workspace_bytes(C.byref(a)), dev)
    a.out, a.workspace, a.workspace_bytes = ptr(out), ptr(ws), ws.numel()
    _abi.check(_t.launch("fused_decode_sdpa", lib.mxb_fused_decode_sdpa, a))
    return out
