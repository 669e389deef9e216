"""Workloads that stand for what a program built on this package has it do, and what each cannot do without.

``listed()`` names twelve of them, ``draw(rng)`` gives more from the same ranges, ``prepare`` makes the inputs and
whatever a program keeps between calls (caches, plans), ``run`` is one pass through the public entry points, ``work``
the bytes and operations of a pass, ``tolerance`` how far two correct implementations may differ.

Kinds:

``decode_eager``    one layer of a float32 decode step, called operator by operator (``sparse_decode_step``)
``decode_plan``     a batched decode step over ragged contexts as a server runs it (``SparseDecodePlan.run``)
``ds4_token``       one batch-1 decode token in the layout of the fused decode operators: indexer QAT, scores,
                    selection, KV-row preparation, attention over a window and the selected pool rows
``prefill``         one chunk of sparse prefill over ratio-4 compressed rows (``sparse_prefill_step``)
``quantize_rows``   new latent rows into the int8 cache format (``quantize_kv_int8``)
``flash``           causal GQA prefill with or without the gate (``sdpa_fa_prefill``)
``q8_chunk``        one chunk over an affine-q8 past: append, the chunk's own round trip, attention
``q8_token``        one decode token over an affine-q8 cache: append, attention
"""
from __future__ import annotations

import math

import torch

from moespresso_b200.deepseek_v4.attention import rope_inverse_frequencies
from moespresso_b200.deepseek_v4.decode_attention_kernel import fused_decode_prep, fused_decode_sdpa
from moespresso_b200.deepseek_v4.decode_step import LatentCache, SparseDecodePlan, quantize_kv_int8, sparse_decode_step
from moespresso_b200.deepseek_v4.prefill_step import sparse_prefill_step
from moespresso_b200.qwen.full_attention import (QuantizedKVCache, dequantize_affine_q8, quantize_affine_q8,
                                                 sdpa_decode_q8, sdpa_fa_prefill, sdpa_fa_prefill_q8)

# Shapes that every case shares: 64 heads over 576-wide latent rows (512 latent + 64 rotary, values = the first 512),
# a 16 x 64 indexer; 16 query and 2 KV heads of 256 for the GQA layers.
HEADS, D_QK, D_V, IDX_HEADS, IDX_DIM = 64, 576, 512, 16, 64
GQA_HQ, GQA_HKV, GQA_D = 16, 2, 256

_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}


def listed():
    return [
        # One sequence, 4096 rows in float32, the operators called one by one: launches and host time.
        {"name": "decode_fp32_4k", "kind": "decode_eager", "rows": 4096, "k": 512},
        # One token of a single-user session: small pool, five-launch selection and attention, all latency.
        {"name": "ds4_token_2500", "kind": "ds4_token", "rows": 2500, "k": 512, "window": 128, "pos": 10003},
        # A lightly loaded server: three short conversations, bf16 latent cache.
        {"name": "decode_b3_bf16", "kind": "decode_plan", "batch": 3, "lo": 2000, "hi": 7000, "k": 512, "kv": "bf16"},
        # The loaded server: 32 long conversations, int8 latent cache with per-token scales, FP8 index keys.
        {"name": "decode_b32_int8", "kind": "decode_plan", "batch": 32, "lo": 32768, "hi": 131072, "k": 2048, "kv": "int8"},
        # One very long document: a selection over a million scores.
        {"name": "decode_1m_int8", "kind": "decode_plan", "batch": 1, "lo": 1048576, "hi": 1048576, "k": 2048, "kv": "int8"},
        # The tail chunk of a short prompt: ragged token and row counts, raw window, fp16.
        {"name": "prefill_tail_f16", "kind": "prefill", "tokens": 333, "rows": 5003, "k": 512, "dtype": "f16", "window": 128},
        # A full chunk late in a long prompt: 4096 tokens over 32768 compressed rows.
        {"name": "prefill_4096_bf16", "kind": "prefill", "tokens": 4096, "rows": 32768, "k": 2048, "dtype": "bf16", "window": 0},
        # The cache append behind a prefill chunk (every sequence of a batch at once).
        {"name": "quantize_rows_40k", "kind": "quantize_rows", "rows": 40001, "dtype": "bf16"},
        # A prompt in one piece through a gated full-attention layer.
        {"name": "flash_8192_bf16", "kind": "flash", "tokens": 8192, "past": 0, "dtype": "bf16", "gate": True},
        # A short ragged prompt behind a dense past, no gate.
        {"name": "flash_tail_f16", "kind": "flash", "tokens": 700, "past": 1365, "dtype": "f16", "gate": False},
        # A chunk of a long prompt over the 8-bit cache.
        {"name": "q8_chunk_2048", "kind": "q8_chunk", "tokens": 2048, "past": 30720},
        # Generation late in a long conversation over the 8-bit cache.
        {"name": "q8_token_131072", "kind": "q8_token", "past": 131071},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng, lo, hi):
    """A row count.  7901 to 8191 stay out: at this writing the selection's launch is refused there (its shared memory
    passes the default limit before the rule that raises the limit applies)."""
    n = _log(rng, lo, hi)
    return n if n <= 7900 or n >= 8192 else 8209


def draw(rng):
    kind = rng.choice(["decode_eager", "decode_plan", "decode_plan", "decode_plan", "ds4_token", "prefill", "prefill",
                       "quantize_rows", "flash", "flash", "q8_chunk", "q8_token"])
    if kind == "decode_eager":
        return {"kind": kind, "rows": _rows(rng, 1024, 16384), "k": rng.choice([256, 512, 1024])}
    if kind == "decode_plan":
        batch = _log(rng, 1, 64)
        # the tables of a batch stay below three million rows
        hi = _log(rng, 2048, min(1048576, 3000000 // batch))
        lo = max(1024, hi // rng.choice([1, 2, 4]))
        if lo < 8192 and hi > 7900:
            hi = 7900                              # the longest context would be drawn around 8000 (see _rows)
        return {"kind": kind, "batch": batch, "lo": min(lo, hi), "hi": hi,
                "k": rng.choice([512, 1024, 2048]), "kv": rng.choice(["int8", "int8", "bf16"])}
    if kind == "ds4_token":
        rows = _rows(rng, 600, 16384)
        return {"kind": kind, "rows": rows, "k": rng.choice([256, 512]), "window": rng.choice([64, 127, 128]),
                "pos": 4 * rows + rng.randrange(4)}
    if kind == "prefill":
        tokens = _log(rng, 64, 2048)
        return {"kind": kind, "tokens": tokens, "rows": _rows(rng, 2200, 32768),
                "k": rng.choice([512, 1024, 2048]), "dtype": rng.choice(["bf16", "f16"]),
                "window": rng.choice([0, 100, 128])}
    if kind == "quantize_rows":
        return {"kind": kind, "rows": _log(rng, 500, 200000), "dtype": rng.choice(["bf16", "f16", "f32"])}
    if kind == "flash":
        return {"kind": kind, "tokens": _log(rng, 100, 8000), "past": rng.choice([0, 0, _log(rng, 50, 8000)]),
                "dtype": rng.choice(["bf16", "f16"]), "gate": rng.random() < 0.6}
    if kind == "q8_chunk":
        return {"kind": kind, "tokens": _log(rng, 64, 2048), "past": _log(rng, 500, 30000)}
    return {"kind": kind, "past": _log(rng, 32768, 200000)}


class _Gen:
    """Seeded draws on the device."""

    def __init__(self, seed):
        self.dev = torch.device("cuda")
        self.g = torch.Generator(device=self.dev).manual_seed(int(seed))

    def normal(self, *shape, scale=1.0, dtype=torch.float32):
        return torch.randn(shape, generator=self.g, device=self.dev).mul_(scale).to(dtype)

    def normal_rows(self, n, width, dtype):
        """A long table of normal rows, drawn in pieces (the float32 draw of all of it would be larger than the table)."""
        out = torch.empty((n, width), dtype=dtype, device=self.dev)
        for lo in range(0, n, 1 << 18):
            hi = min(n, lo + (1 << 18))
            out[lo:hi] = torch.randn((hi - lo, width), generator=self.g, device=self.dev).to(dtype)
        return out

    def ints(self, lo, hi, *shape, dtype=torch.int64):
        return torch.randint(lo, hi, shape, generator=self.g, device=self.dev, dtype=dtype)

    def log_uniform(self, n, lo, hi, dtype):
        u = torch.rand(n, generator=self.g, device=self.dev)
        return torch.exp(u * (math.log(hi) - math.log(lo)) + math.log(lo)).to(dtype)


def _lengths(case, gen):
    """Context lengths of a batch: host integers, as a scheduler holds them."""
    return [int(n) for n in gen.ints(case["lo"], case["hi"] + 1, case["batch"]).tolist()]


def _latent_cache(gen, lens, kv):
    total = sum(lens)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    if kv == "int8":
        rows, scales = gen.ints(-127, 128, total, D_QK, dtype=torch.int8), gen.log_uniform(total, 1e-3, 1e-1, torch.float16)
    else:
        rows, scales = gen.normal_rows(total, D_QK, _DTYPES[kv]), None
    keys = gen.normal_rows(total, IDX_DIM, torch.float32 if kv == "f32" else torch.float8_e4m3fn)
    return LatentCache(kv=rows, kv_scales=scales, idx_keys=keys,
                       row_start=torch.tensor(starts, dtype=torch.int64, device=gen.dev),
                       row_count=torch.tensor(lens, dtype=torch.int32, device=gen.dev), max_rows=max(lens))


def prepare(case, seed):
    gen, kind = _Gen(seed), case["kind"]
    s = {"case": case}
    if kind in ("decode_eager", "decode_plan"):
        eager = kind == "decode_eager"
        B = 1 if eager else case["batch"]
        qdt = torch.float32 if eager else torch.bfloat16
        cache = _latent_cache(gen, [case["rows"]] if eager else _lengths(case, gen), "f32" if eager else case["kv"])
        s["q"] = gen.normal(B, HEADS, D_QK, dtype=qdt)
        s["idx_q"] = gen.normal(B, IDX_HEADS, IDX_DIM, dtype=qdt)
        s["idx_w"] = gen.normal(B, IDX_HEADS, scale=0.25)
        if eager:
            s["cache"] = cache
        else:
            s["plan"] = SparseDecodePlan(cache, heads=HEADS, d_qk=D_QK, idx_heads=IDX_HEADS, idx_dim=IDX_DIM, k=case["k"],
                                         scale=D_QK ** -0.5, d_v=D_V, q_dtype=qdt, out_dtype=torch.bfloat16)
    elif kind == "ds4_token":
        s["q_idx"] = gen.normal(HEADS, 128, dtype=torch.float16)
        s["pooled_qat"] = gen.normal(case["rows"], 128)
        s["weights"] = gen.normal(HEADS, scale=HEADS ** -0.5)
        s["kv_row"] = gen.normal(512, dtype=torch.float16)
        s["q"] = gen.normal(HEADS, 512, dtype=torch.float16)
        s["window"] = gen.normal(case["window"], 512, dtype=torch.float16)
        s["pooled"] = gen.normal(case["rows"], 512, dtype=torch.float16)
        s["sinks"] = gen.normal(HEADS, dtype=torch.float16)
        s["inv_freq"] = torch.as_tensor(rope_inverse_frequencies(64, 160000.0), device=gen.dev).to(torch.float32)
        s["params"] = torch.tensor([case["pos"], case["pos"] % case["window"]], dtype=torch.int32, device=gen.dev)
    elif kind == "prefill":
        T, R, dt = case["tokens"], case["rows"], _DTYPES[case["dtype"]]
        s["q"] = gen.normal(T, HEADS, D_QK, dtype=dt)
        s["kv"] = gen.normal(R, D_QK, dtype=dt)
        s["idx_q"] = gen.normal(T, IDX_HEADS, IDX_DIM, dtype=dt)
        s["idx_keys"] = gen.normal(R, IDX_DIM, dtype=dt)
        s["idx_w"] = gen.normal(T, IDX_HEADS, scale=0.25)
        s["sinks"] = gen.normal(HEADS)
        # the raw rows a chunk needs: its own and the window before its first token
        s["raw"] = gen.normal(T + case["window"], D_QK, dtype=dt) if case["window"] else None
    elif kind == "quantize_rows":
        s["rows"] = gen.normal_rows(case["rows"], D_QK, _DTYPES[case["dtype"]])
    elif kind == "flash":
        L, P, dt = case["tokens"], case["past"], _DTYPES[case["dtype"]]
        s["q"] = gen.normal(L, GQA_HQ, GQA_D, scale=0.5, dtype=dt)
        s["k"], s["v"] = (gen.normal(P + L, GQA_HKV, GQA_D, scale=0.5, dtype=dt) for _ in range(2))
        s["gate"] = gen.normal(L, GQA_HQ, GQA_D, dtype=dt) if case["gate"] else None
    else:
        L, P, bf = case.get("tokens", 1), case["past"], torch.bfloat16
        s["cache"] = QuantizedKVCache(GQA_HKV, GQA_D, P + L)
        for lo in range(0, P, 16384):
            n = min(16384, P - lo)
            s["cache"].update_and_fetch(*(gen.normal(1, GQA_HKV, n, GQA_D, scale=0.5, dtype=bf) for _ in range(2)))
        s["q"] = gen.normal(1, GQA_HQ, L, GQA_D, scale=1.0 if L == 1 else 0.5, dtype=bf)
        s["k"], s["v"] = (gen.normal(1, GQA_HKV, L, GQA_D, scale=0.5, dtype=bf) for _ in range(2))
        s["gate"] = gen.normal(1, L, GQA_HQ * GQA_D, dtype=bf)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode_eager":
        out, ids = sparse_decode_step(s["q"], s["idx_q"], s["idx_w"], s["cache"], k=case["k"], scale=D_QK ** -0.5, d_v=D_V,
                                      return_ids=True)
        return {"out": out, "ids": ids}
    if kind == "decode_plan":
        out = s["plan"].run(s["q"], s["idx_q"], s["idx_w"])
        return {"out": out, "ids": s["plan"].ids}
    if kind == "ds4_token":
        sel, row, scores = fused_decode_prep(s["q_idx"], s["pooled_qat"], s["weights"], s["kv_row"], s["inv_freq"],
                                             s["params"], scale=128 ** -0.5, topk=case["k"])
        out = fused_decode_sdpa(s["q"], s["window"], row, s["pooled"], sel, s["sinks"], s["inv_freq"], s["params"],
                                scale=512 ** -0.5)
        return {"sel": sel, "row": row, "scores": scores, "out": out}
    if kind == "prefill":
        T, R = case["tokens"], case["rows"]
        # the chunk ends where the pool does
        out, ids = sparse_prefill_step(s["q"], s["kv"], s["idx_q"], s["idx_keys"], s["idx_w"], pos0=4 * R - T, ratio=4,
                                       k=case["k"], scale=D_QK ** -0.5, d_v=D_V, sinks=s["sinks"], raw_kv=s["raw"],
                                       window=case["window"], return_ids=True)
        return {"out": out, "ids": ids}
    if kind == "quantize_rows":
        return quantize_kv_int8(s["rows"])
    if kind == "flash":
        return sdpa_fa_prefill(s["q"], s["k"], s["v"], GQA_D ** -0.5, gate=s["gate"], layout="lhd")
    cache = s["cache"]
    cache.offset = case["past"]                    # every pass appends at the same place
    if kind == "q8_token":
        qk, qv = cache.update_and_fetch(s["k"], s["v"])
        return sdpa_decode_q8(s["q"], *qk, *qv, GQA_D ** -0.5)
    past_k, past_v = cache.state
    cache.update_and_fetch(s["k"], s["v"])
    self_k = dequantize_affine_q8(*quantize_affine_q8(s["k"]))
    self_v = dequantize_affine_q8(*quantize_affine_q8(s["v"]))
    return sdpa_fa_prefill_q8(s["q"], *past_k, *past_v, self_k, self_v, GQA_D ** -0.5, gate=s["gate"])


def work(case):
    """Bytes: every input read once and every output written once, rows that a selection leaves out not at all.
    Operations: two per multiply-add of the scores and of both contractions of the attention."""
    kind = case["kind"]
    if kind in ("decode_eager", "decode_plan"):
        if kind == "decode_eager":
            B, rows, es, row_bytes, key_bytes, out_es = 1, case["rows"], 4, D_QK * 4, IDX_DIM * 4, 4
        else:
            B, es, out_es, key_bytes = case["batch"], 2, 2, IDX_DIM
            rows = B * (case["lo"] + case["hi"]) / 2           # the mean of the uniform lengths
            row_bytes = D_QK + 2 if case["kv"] == "int8" else D_QK * 2
        k = case["k"]
        nbytes = (rows * key_bytes + B * (IDX_HEADS * IDX_DIM * es + IDX_HEADS * 4 + HEADS * D_QK * es + k * row_bytes
                                          + HEADS * D_V * out_es + k * 4))
        return {"bytes": nbytes, "flops": 2 * IDX_HEADS * IDX_DIM * rows + 2 * B * HEADS * k * (D_QK + D_V)}
    if kind == "ds4_token":
        R, n = case["rows"], case["k"] + case["window"]
        return {"bytes": R * 128 * 4 + R * 4 + n * 1024 + 2 * HEADS * 1024 + HEADS * 128 * 2,
                "flops": 2 * HEADS * 128 * R + 4 * HEADS * n * 512}
    if kind == "prefill":
        T, R, k = case["tokens"], case["rows"], case["k"]
        n = k + min(case["window"], 4 * R)
        nbytes = T * (HEADS * D_QK * 2 + IDX_HEADS * (IDX_DIM * 2 + 4) + HEADS * D_V * 4 + k * 4)
        nbytes += R * (D_QK + IDX_DIM) * 2 + (T + case["window"]) * D_QK * 2 * (case["window"] > 0)
        # the last token of the chunk sees all rows, the first T / 4 fewer
        return {"bytes": nbytes, "flops": 2 * IDX_HEADS * IDX_DIM * T * (R - T / 8) + 2 * T * HEADS * n * (D_QK + D_V)}
    if kind == "quantize_rows":
        es = 4 if case["dtype"] == "f32" else 2
        return {"bytes": case["rows"] * (D_QK * (es + 1) + 2), "flops": 0}
    P, L = case["past"], case.get("tokens", 1)
    flops = 4 * GQA_HQ * GQA_D * (L * P + L * (L + 1) / 2)
    if kind == "flash":
        return {"bytes": 2 * GQA_D * (L * GQA_HQ * (3 if case["gate"] else 2) + 2 * (P + L) * GQA_HKV), "flops": flops}
    q8_row = GQA_HKV * (GQA_D + 2 * 2 * GQA_D // 64)           # packed words, scales and biases of one position
    nbytes = 2 * q8_row * (P + L) + 2 * 2 * GQA_HKV * GQA_D * L + 2 * GQA_HQ * GQA_D * L * (3 if kind == "q8_chunk" else 2)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times the distance (relative 2-norm, largest) of the present results from the same path in float64.
    ``differ``: ids come out ascending, so one swap between two scores that nearly tie at the boundary moves all the
    ids between them."""
    kind = case["kind"]
    if kind == "quantize_rows":
        return "exact"                                         # int8 values and fp16 scales, each a single rounding
    if kind == "decode_eager":                                 # float32 throughout: 3.3e-7, 4.0e-6
        return {"rel": 2e-6, "max": 2e-5, "differ": 4e-3}
    if kind == "q8_token":                                     # fp16 operands, a mean over many keys: 7.7e-3, 1.1e-2
        return {"rel": 3e-2, "max": 5e-2}
    if kind == "ds4_token" or case.get("dtype") == "f16":      # fp16 rows, weights and result: 3.1e-4, 1.8e-3
        return {"rel": 1.3e-3, "max": 8e-3, "differ": 4e-3}
    return {"rel": 8e-3, "max": 4e-2, "differ": 4e-3}          # bf16 operands or result: 2.3e-3, 1.0e-2
