"""Sparse attention of a few tokens (one cluster per token and 16 heads) against the CPU oracle, at the edges of its row
tiles, splits and head groups.  Tolerances (max-abs) as for the other tensor-core path: 2e-2, 2e-3 for fp16 tables."""
import numpy as np
import pytest
import torch

from moespresso_b200.deepseek_v4 import indexed_attention_kernel as iak
from oracle import ds4
from tests.gpu_util import bf16_round, dev, f16_round, max_abs, need_gpu

pytestmark = pytest.mark.gpu


def _tables(rng, kind, R, raw_cap, D):
    if kind == "int8":
        mk = lambda n: (rng.integers(-127, 128, size=(n, D), dtype=np.int8),
                        np.exp(rng.uniform(np.log(1e-3), np.log(1e-1), size=n)).astype(np.float16))
        (comp, cs), (raw, rs) = mk(R), mk(max(raw_cap, 1))
        return dict(comp=comp, raw=raw, cs=cs, rs=rs, ct=dev(comp), rt=dev(raw), cst=dev(cs), rst=dev(rs),
                    okw=dict(kv_scales=cs, raw_scales=rs))
    rnd, kt = {"f16": (f16_round, torch.float16), "bf16": (bf16_round, torch.bfloat16),
               "f32": (lambda x: x.astype(np.float32), torch.float32)}[kind]
    comp, raw = rnd(rng.standard_normal((R, D))), rnd(rng.standard_normal((max(raw_cap, 1), D)))
    return dict(comp=comp, raw=raw, ct=dev(comp, kt), rt=dev(raw, kt), cst=None, rst=None, okw={})


@pytest.mark.parametrize("kind", ["f16", "bf16", "int8"])
@pytest.mark.parametrize("D,H,k,window,raw_cap", [
    (576, 64, 1, 0, 0),        # one row
    (512, 16, 63, 0, 0),       # one split, one head group, a row short of a tile
    (576, 64, 64, 0, 0),       # a full tile
    (512, 17, 65, 0, 0),       # a second split of one row, a second group of one head
    (576, 1, 512, 128, 128),   # ten splits: blocks of features that one CTA owns twice
    (512, 64, 515, 101, 128),  # a ragged window before the list
    (576, 40, 1023, 0, 0),     # sixteen splits of 64 rows
    (576, 64, 1025, 0, 0),     # nine of 128
    (512, 64, 1900, 100, 128), # sixteen of 128, window included
    (576, 64, 2048, 0, 0),
])
def test_one_token(kind, D, H, k, window, raw_cap):
    need_gpu()
    rng = np.random.default_rng(k * 131 + D + H)
    R = max(2 * k, 40)
    t = _tables(rng, kind, R, raw_cap, D)
    qr, qt = (f16_round, torch.float16) if kind == "f16" else (bf16_round, torch.bfloat16)
    q = qr(rng.standard_normal((H, D)))
    sinks = rng.standard_normal(H).astype(np.float32)
    ids = np.sort(rng.choice(R, size=k, replace=False)).astype(np.int32)
    if k > 60:
        ids[[0, 5, 59]] = -1            # skipped
        ids[-2] = R + 7                 # ends the walk: the last entry is not visited
    scale = D ** -0.5 * (20.0 if kind == "int8" else 1.0)
    pos0 = 128 + R * 4 - 1
    raw = t["raw"] if raw_cap else None
    ref = ds4.indexed_mixed_attention_decode(q, raw, t["comp"], ids, sinks, pos0=pos0, window=window, ratio=4,
                                             raw_start=11 if raw_cap else 0, scale=scale, d_v=512, **t["okw"])
    out = iak.sparse_attention(dev(q, qt)[None, :, None, :], t["ct"], dev(ids)[None, None], dev(sinks), pos0=pos0, window=window,
                               ratio=4, raw_kv=t["rt"][None] if raw_cap else None, raw_start=11 if raw_cap else 0, scale=scale,
                               d_v=512, kv_scales=t["cst"], raw_scales=t["rst"] if raw_cap else None, check=True)[0, :, 0]
    assert max_abs(out, ref) <= (2e-3 if kind == "f16" else 2e-2)


@pytest.mark.parametrize("kind,qkind", [("f16", "f16"), ("f16", "f32"), ("bf16", "bf16"), ("bf16", "f32"), ("int8", "bf16"),
                                        ("int8", "f16")])
@pytest.mark.parametrize("B,T,k", [(3, 1, 512), (2, 2, 512), (7, 1, 300), (3, 1, 2048), (1, 1, 4000)])
def test_batches_and_strided_q(kind, qkind, B, T, k):
    """Splits of 64, 128 and (int8) 256 rows, ragged sequences, q with a head axis that is not the second slowest, q whose
    rows are not 16-byte aligned, all output types."""
    need_gpu()
    D, H = 576, 64
    rng = np.random.default_rng(B * 7 + T + k)
    lens = rng.integers(max(k - 40, 1), 2 * k, size=B)
    starts = np.concatenate([[0], np.cumsum(lens)[:-1]])
    t = _tables(rng, kind, int(lens.sum()), 0, D)
    rnd, qt = {"f32": (lambda x: x.astype(np.float32), torch.float32), "f16": (f16_round, torch.float16),
               "bf16": (bf16_round, torch.bfloat16)}[qkind]
    q = rnd(rng.standard_normal((B, H, T, D)))
    ids = np.full((B, T, k), -1, np.int32)
    for b in range(B):
        for x in range(T):
            n = min(k, int(lens[b]))
            ids[b, x, :n] = np.sort(rng.choice(int(lens[b]), size=n, replace=False))
    scale = D ** -0.5 * (20.0 if kind == "int8" else 1.0)
    kw = dict(pos0=0, window=0, ratio=0, scale=scale, d_v=512, kv_scales=t["cst"], comp_row_start=dev(starts.astype(np.int64)),
              comp_row_count=dev(lens.astype(np.int32)), n_comp=int(lens.max()), check=True)
    qd = dev(q, qt)
    bthd = qd.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
    store = torch.zeros(q.size + 1, dtype=qt, device="cuda")
    odd = store[1:].view(B, H, T, D)
    odd.copy_(qd)
    out = iak.sparse_attention(qd, t["ct"], dev(ids), None, **kw)
    for other in (bthd, odd):
        assert torch.equal(iak.sparse_attention(other, t["ct"], dev(ids), None, **kw), out)
    tol = 2e-3 if kind == "f16" else 2e-2
    for b in range(B):
        s, n = int(starts[b]), int(lens[b])
        okw = dict(kv_scales=t["cs"][s:s + n]) if kind == "int8" else {}
        for x in range(T):
            ref = ds4.indexed_mixed_attention_decode(q[b, :, x], None, t["comp"][s:s + n], ids[b, x], None, pos0=0, window=0,
                                                     ratio=0, scale=scale, d_v=512, **okw)
            assert max_abs(out[b, :, x], ref) <= tol
    for od in (torch.bfloat16, torch.float16):
        half = iak.sparse_attention(qd, t["ct"], dev(ids), None, out_dtype=od, **kw)
        assert torch.equal(half, out.to(od))


def test_q_of_any_magnitude_over_int8_rows():
    """q is scaled by a power of two per head: the softmax of a q that is 2^20 or 2^-20 times another, over a scale that undoes
    it, is the same to the bit; a head of zeros averages its rows."""
    need_gpu()
    rng = np.random.default_rng(4)
    D, H, R, k = 576, 64, 900, 512
    t = _tables(rng, "int8", R, 0, D)
    q = bf16_round(rng.standard_normal((H, D)))
    q[3] = 0.0
    ids = dev(np.sort(rng.choice(R, size=k, replace=False)).astype(np.int32))[None, None]
    f = lambda e: iak.sparse_attention(dev(np.ldexp(q, e), torch.bfloat16)[None, :, None, :], t["ct"], ids, None, pos0=0, window=0,
                                       ratio=0, scale=float(np.ldexp(0.5, -e)), d_v=512, kv_scales=t["cst"], n_comp=R, check=True)
    base = f(0)
    assert torch.equal(f(20), base) and torch.equal(f(-20), base)
    sel = ids[0, 0].cpu().numpy()
    mean = (t["comp"][sel].astype(np.float64) * t["cs"][sel].astype(np.float64)[:, None])[:, :512].mean(0)
    assert max_abs(base[0, 3, 0], mean) <= 2e-2


@pytest.mark.parametrize("e", [-126, -112, 99, 116, 125])
def test_int8_tables_take_any_finite_q(e):
    """q is scaled by a power of two into fp16's range: over all of bfloat16's range the same bits as for q of 1."""
    need_gpu()
    rng = np.random.default_rng(5)
    D, H, k, R = 576, 20, 300, 900
    t = _tables(rng, "int8", R, 0, D)
    q = np.round(8 * rng.standard_normal((H, D)).clip(-3.9, 3.9)) / 8       # times 2^e exactly a bfloat16
    ids = np.sort(rng.choice(R, size=k, replace=False)).astype(np.int32)

    def f(e):
        x = dev((q * 2.0 ** e).astype(np.float32), torch.bfloat16)[None, :, None, :]
        return iak.sparse_attention(x, t["ct"], dev(ids)[None, None], None, pos0=0, window=0, ratio=0, scale=0.7 * 2.0 ** -e, d_v=512,
                                    kv_scales=t["cst"], n_comp=R)
    base = f(0)
    assert bool(base.isfinite().all()) and torch.equal(f(e), base)
    ref = ds4.indexed_mixed_attention_decode(q.astype(np.float32), None, t["comp"], ids, None, pos0=0, window=0, ratio=0, scale=0.7,
                                             d_v=512, kv_scales=t["cs"])
    assert max_abs(base[0, :, 0], ref) <= 2e-2


@pytest.mark.parametrize("kind", ["bf16", "int8"])
@pytest.mark.parametrize("k", [64, 700, 2048])
def test_partials_of_list_halves_merge_to_the_whole(kind, k):
    """Partial output: un-normalised O and (m, l) of two halves of a list, merged on the host, against the whole list's output;
    a half without rows carries (-inf, 0)."""
    need_gpu()
    rng = np.random.default_rng(k)
    D, H, R = 576, 40, 3000
    t = _tables(rng, kind, R, 0, D)
    q = dev(bf16_round(rng.standard_normal((H, D))), torch.bfloat16)[None, :, None, :]
    ids = np.sort(rng.choice(R, size=k, replace=False)).astype(np.int32)
    kw = dict(pos0=0, window=0, ratio=0, scale=D ** -0.5, d_v=512, kv_scales=t["cst"], n_comp=R, check=True)
    whole = iak.sparse_attention(q, t["ct"], dev(ids)[None, None], None, **kw)[0, :, 0].double()
    for cut in (0, k // 3):
        parts = []
        for half in (np.where(np.arange(k) < cut, ids, -1), np.where(np.arange(k) >= cut, ids, -1)):
            o, ml = iak.sparse_attention(q, t["ct"], dev(half.astype(np.int32))[None, None], None, partial=True, **kw)
            parts.append((o[0, :, 0].double(), ml[0, 0, :, 0].double(), ml[0, 0, :, 1].double()))
        if cut == 0:
            assert bool((parts[0][1] == -np.inf).all()) and float(parts[0][2].abs().max()) == 0.0
        m = torch.maximum(parts[0][1], parts[1][1])
        w = [torch.exp(x[1] - m) for x in parts]
        out = sum(x[0] * y[:, None] for x, y in zip(parts, w)) / sum(x[2] * y for x, y in zip(parts, w))[:, None]
        # the weights of either side are rounded to 16 bits (2^-9, fp16 2^-12) relative to another maximum
        assert float((out - whole).abs().max()) <= (2 ** -8 if kind == "bf16" else 2 ** -11) * float(np.abs(whole.cpu().numpy()).max() * 4)


@pytest.mark.parametrize("D,H,k,window,raw_cap,B", [
    (576, 64, 1, 0, 0, 1),
    (512, 3, 65, 0, 0, 1),        # three of a group's four heads, a second split of one row
    (576, 64, 512, 0, 0, 1),      # eight splits: more than four heads per CTA, the last group not full
    (576, 40, 1024, 0, 0, 1),     # sixteen splits
    (512, 64, 400, 101, 128, 1),  # a ragged window before the list
    (576, 16, 256, 0, 0, 7),      # a batch
])
def test_float32_tables(D, H, k, window, raw_cap, B):
    """1e-4 as for the other float32 kernel, which exact_fp32 with a fixed number of splits still takes."""
    need_gpu()
    rng = np.random.default_rng(k * 7 + D + H)
    R = max(2 * k, 40)
    t = _tables(rng, "f32", R, raw_cap, D)
    q = rng.standard_normal((B, H, 1, D)).astype(np.float32)
    sinks = rng.standard_normal(H).astype(np.float32)
    ids = np.stack([np.sort(rng.choice(R, size=k, replace=False)) for _ in range(B)]).astype(np.int32)[:, None]
    if k > 60:
        ids[:, 0, [0, 5, 59]] = -1
        ids[:, 0, -2] = R + 7
    pos0 = 128 + R * 4 - 1
    kw = dict(pos0=pos0, window=window, ratio=4, raw_kv=t["rt"][None] if raw_cap else None, raw_start=11 if raw_cap else 0,
              scale=D ** -0.5, d_v=512, comp_row_start=torch.zeros(B, dtype=torch.int64, device="cuda"), n_comp=R, check=True)
    out = iak.sparse_attention(dev(q), t["ct"], dev(ids), dev(sinks), **kw)
    other = iak.sparse_attention(dev(q), t["ct"], dev(ids), dev(sinks), n_splits=2, **kw)
    for b in range(B):
        ref = ds4.indexed_mixed_attention_decode(q[b, :, 0], t["raw"] if raw_cap else None, t["comp"], ids[b, 0], sinks, pos0=pos0,
                                                 window=window, ratio=4, raw_start=11 if raw_cap else 0, scale=D ** -0.5, d_v=512)
        assert max_abs(out[b, :, 0], ref) <= 1e-4 and max_abs(other[b, :, 0], ref) <= 1e-4
    half = iak.sparse_attention(dev(q), t["ct"], dev(ids), dev(sinks), out_dtype=torch.bfloat16, **kw)
    assert torch.equal(half, out.to(torch.bfloat16))
    o, ml = iak.sparse_attention(dev(q), t["ct"], dev(ids), None, partial=True, **kw)
    plain = iak.sparse_attention(dev(q), t["ct"], dev(ids), None, **kw)
    assert max_abs(o / ml[:, 0, :, 1][:, :, None, None], plain) <= 1e-5
