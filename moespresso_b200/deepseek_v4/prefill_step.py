"""Ratio-4 compressed-KV sparse prefill of one chunk: indexer scores -> per-token top-k ->
indexed sparse attention.

Operator-calling part of the reference's ``_Ratio4PrefillFastAttention.__call__``
(``src/moespresso/runtime/deepseek_v4/model.py:1320-1480``): scores by the tiled score
kernel with the causal compressed-row mask (:1434-1441), ``argpartition`` + ascending sort
(:1442-1451), then the indexed prefill consumer (:1453-1472); when the pool holds no more
than ``k`` rows every row is selected (:1393-1395).  Projections, RoPE and the QAT pre-op
are outside this operator.

The [tokens x rows] fp32 score matrix is never materialised: tokens are processed in
chunks whose scores (``token_chunk`` x rows x 4 bytes) are written to one reused buffer between the score
kernel and the selection kernel.  The default chunk is eight tokens per SM (1184 on a B200): with 16 index
heads that is one CTA of the score kernel per SM, which keeps its eight tokens and walks all rows.  The buffer
is bounded: four tokens per SM where eight would take more than 320 MB of scores.  Scores and selection of 4096
tokens, us at 592 / 888 / 1184 / 1480 / 4096 tokens per chunk (bf16, 16 heads of 64, k = 2048): 4096 rows 164 /
166 / 142 / 156 / 149, 16384 rows 459 / 470 / 408 / 487 / 434, 32768 rows 699 / 770 / 657 / 773 / 672, 33000 rows
722 / 779 / 669 / 786 / 687, 65536 rows (310 MB at 1184) 1468 / 1559 / 1350 / 1461 / 1346.
"""
from __future__ import annotations

import torch

from .attention import topk_select
from .indexed_attention_kernel import indexer_scores_tiled_live, sparse_attention

_SCORE_BYTES = 320_000_000


def sparse_prefill_step(q, comp_kv, idx_q, idx_keys, idx_w, *, pos0: int, ratio: int = 4, k: int = 512,
                        scale=None, d_v=None, sinks=None, raw_kv=None, window: int = 128, raw_start: int = 0,
                        token_chunk: int | None = None, return_ids: bool = False):
    """q [T,H,Dqk]; comp_kv [R,Dqk]; idx_q [T,Hi,Di]; idx_keys [R,Di]; idx_w [T,Hi] float32
    (all scale factors folded in); raw_kv [raw_cap,Dqk] or None.  Token t sits at ``pos0 + t``.
    Returns float32 [T,H,d_v] (and the int32 ids [T,k], ascending, -1 padded)."""
    T, H, Dqk = (int(x) for x in q.shape)
    R = int(comp_kv.shape[0])
    dev = q.device
    kk = min(int(k), R)
    if R <= int(k):
        # every pooled row is a candidate; visibility is still applied by the attention kernel's walk
        ids = torch.arange(R, dtype=torch.int32, device=dev).expand(T, R).contiguous()
    else:
        ids = torch.empty((T, kk), dtype=torch.int32, device=dev)
        if token_chunk is None:
            token_chunk = 8 * torch.cuda.get_device_properties(dev).multi_processor_count
            if token_chunk * R * 4 > _SCORE_BYTES:
                token_chunk //= 2
        chunk = max(1, min(int(token_chunk), T))
        buf = torch.empty((1, chunk, R), dtype=torch.float32, device=dev)
        iq = idx_q.permute(1, 0, 2)[None]            # [1,Hi,T,Di]
        for t0 in range(0, T, chunk):
            n = min(chunk, T - t0)
            scores = indexer_scores_tiled_live(iq[:, :, t0:t0 + n], idx_w[None, t0:t0 + n].contiguous(),
                                               idx_keys[None], pos0=pos0 + t0, ratio=ratio, out=buf[:, :n])
            topk_select(scores[0, :n], kk, out=ids[t0:t0 + n])
    out = sparse_attention(q.permute(1, 0, 2)[None], comp_kv, ids[None], sinks, pos0=pos0, window=window,
                           ratio=ratio, raw_kv=None if raw_kv is None else raw_kv[None], raw_start=raw_start,
                           scale=scale, d_v=d_v, n_comp=R, out_layout="bthd")[0]
    return (out, ids) if return_ids else out
