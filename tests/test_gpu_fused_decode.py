"""The reference-named fused decode operators (composed here from the package's operators) against the oracle."""
import numpy as np
import pytest
import torch

from moespresso_b200.deepseek_v4 import attention as att
from moespresso_b200.deepseek_v4.decode_attention_kernel import fused_decode_prep, fused_decode_sdpa
from oracle import ds4
from tests.gpu_util import dev, need_gpu

pytestmark = pytest.mark.gpu


def _inv_freq():
    return att.rope_inverse_frequencies(64, att.DS4_COMPRESS_ROPE_BASE, att.DS4_YARN).astype(np.float32)


@pytest.mark.parametrize("n_heads,n_rows,topk,pos,qdtype", [(64, 961, 512, 3843, torch.float32),
                                                             (64, 4000, 512, 65535, torch.bfloat16),
                                                             (16, 300, 64, 7, torch.float16)])
def test_fused_decode_prep(n_heads, n_rows, topk, pos, qdtype):
    need_gpu()
    rng = np.random.default_rng(n_rows + pos)
    q = dev(rng.standard_normal((n_heads, 128), dtype=np.float32)).to(qdtype)
    pooled = ds4.indexer_qat(rng.standard_normal((n_rows, 128), dtype=np.float32))
    weights = (rng.standard_normal(n_heads, dtype=np.float32) * n_heads ** -0.5).astype(np.float32)
    kv_row = (rng.standard_normal(512) * 2).astype(np.float16)
    inv = _inv_freq()
    params = torch.tensor([pos, 5], dtype=torch.int32, device="cuda")
    sel, row, scores = fused_decode_prep(q, dev(pooled), dev(weights), dev(kv_row), dev(inv), params,
                                         scale=128 ** -0.5, topk=topk)
    assert sel.dtype == torch.int32 and tuple(sel.shape) == (topk,)
    assert row.dtype == torch.float16 and tuple(row.shape) == (512,)
    exp_scores = ds4.fused_qat_indexer_scores(q.float().cpu().numpy(), pooled, weights, 128 ** -0.5)
    np.testing.assert_allclose(scores.cpu().numpy(), exp_scores, rtol=1e-5, atol=1e-5)
    # the selection is the exact top-k of the scores the device produced (ties to the lower row), ascending
    np.testing.assert_array_equal(sel.cpu().numpy(), ds4.topk_ids(scores.cpu().numpy(), topk)[0])
    np.testing.assert_array_equal(row.cpu().numpy().view(np.uint16),
                                  ds4.fused_decode_prep_row(kv_row, pos, inv).view(np.uint16))


@pytest.mark.parametrize("n_heads,window_rows,n_rows,topk,pos", [(64, 128, 961, 512, 3843), (8, 128, 200, 16, 130),
                                                                  (64, 128, 5000, 512, 20000)])
def test_fused_decode_sdpa(n_heads, window_rows, n_rows, topk, pos):
    need_gpu()
    rng = np.random.default_rng(n_rows * 7 + n_heads)
    q = rng.standard_normal((n_heads, 512)).astype(np.float16)
    window = rng.standard_normal((window_rows, 512)).astype(np.float16)
    row = rng.standard_normal(512).astype(np.float16)
    pooled = rng.standard_normal((n_rows, 512)).astype(np.float16)
    sel = np.sort(rng.choice(n_rows, size=topk, replace=False)).astype(np.int32)
    sinks = rng.standard_normal(n_heads).astype(np.float16)
    inv = _inv_freq()
    write_idx = pos % window_rows
    params = torch.tensor([pos, write_idx], dtype=torch.int32, device="cuda")
    got = fused_decode_sdpa(dev(q), dev(window), dev(row), dev(pooled), dev(sel), dev(sinks), dev(inv), params,
                            scale=512 ** -0.5)
    assert got.dtype == torch.float16 and tuple(got.shape) == (n_heads, 512)
    exp = ds4.fused_decode_sdpa(q, window, row, pooled, sel, sinks, inv, pos, write_idx, 512 ** -0.5)
    # the reference's own tolerance for its float16 attention kernels
    assert np.abs(got.float().cpu().numpy() - exp.astype(np.float32)).max() <= 2e-3


def test_fused_decode_rejects_bad_inputs():
    need_gpu()
    z = lambda *s, dt=torch.float32: torch.zeros(s, device="cuda", dtype=dt)  # noqa: E731
    params = torch.tensor([3, 1], dtype=torch.int32, device="cuda")
    with pytest.raises(ValueError, match="smaller than n_rows"):
        fused_decode_prep(z(8, 128), z(16, 128), z(8), z(512, dt=torch.float16), z(32), params, scale=0.1, topk=16)
    with pytest.raises(ValueError, match=r"float16 \[512\]"):
        fused_decode_prep(z(8, 128), z(16, 128), z(8), z(512), z(32), params, scale=0.1, topk=4)
    with pytest.raises(ValueError, match="between 1 and 64 heads"):
        fused_decode_prep(z(65, 128), z(16, 128), z(65), z(512, dt=torch.float16), z(32), params, scale=0.1, topk=4)
    with pytest.raises(ValueError, match=r"q must be float16"):
        fused_decode_sdpa(z(8, 512), z(128, 512, dt=torch.float16), z(512, dt=torch.float16),
                          z(16, 512, dt=torch.float16), torch.zeros(4, dtype=torch.int32, device="cuda"),
                          z(8, dt=torch.float16), z(32), params, scale=0.1)


@pytest.mark.parametrize("n_heads,window_rows,n_rows,topk,pos,write_idx,pdtype", [
    (64, 128, 961, 512, 3843, 3, torch.int32),     # replaced row inside the window
    (1, 1, 5, 4, 0, 0, torch.int64),               # the smallest of everything; the window is older than the position
    (7, 127, 300, 64, 60, 127, torch.int32),       # position before the window's end, write index outside it
    (64, 0, 961, 512, 3843, 0, torch.int32),       # no window
])
def test_fused_operators_equal_the_single_operators(n_heads, window_rows, n_rows, topk, pos, write_idx, pdtype):
    """Bit for bit what the QAT, score, top-k, FP8 round-trip, rope and attention operators give one by one; operands
    that are views of larger tensors, bases that are not 16-byte aligned included."""
    need_gpu()
    from moespresso_b200.deepseek_v4.decode_attention_kernel import fp8_kv_prefix_rows
    from moespresso_b200.deepseek_v4.indexed_attention_kernel import sparse_attention
    from moespresso_b200.deepseek_v4.indexer_score_kernel import fused_qat_indexer_scores
    g = torch.Generator(device="cuda").manual_seed(n_rows + pos)
    mk = lambda *s, dt=torch.float16: torch.randn(s, generator=g, device="cuda").to(dt)  # noqa: E731
    h16 = torch.float16
    inv = dev(_inv_freq())
    params = torch.tensor([pos, write_idx], dtype=pdtype, device="cuda")
    q_idx, weights = mk(n_heads, 2, 128)[:, 0], mk(n_heads, dt=torch.float32)
    pooled_qat, kv_row = mk(n_rows, 128, dt=torch.float32), mk(513)[1:]
    sel, row, scores = fused_decode_prep(q_idx, pooled_qat, weights, kv_row, inv, params, scale=0.09, topk=topk)
    ref_scores = fused_qat_indexer_scores(q_idx.reshape(1, n_heads, 1, 128), pooled_qat[None],
                                          weights.reshape(1, 1, n_heads), 0.09)
    p64 = params[0:1].to(torch.int64)
    rope = lambda x, **kw: att.apply_rope_tail(x, p64, inv_freq=inv, half_chain=True, **kw)  # noqa: E731
    ref_row = fp8_kv_prefix_rows(kv_row.float()[None])[0].to(h16)
    ref_row[448:] = rope(kv_row.reshape(1, 1, 512)).reshape(-1)[448:]
    assert torch.equal(scores, ref_scores) and torch.equal(sel, att.topk_select(ref_scores[None], topk)[0])
    assert torch.equal(row.view(torch.int16), ref_row.view(torch.int16))

    q, sinks = mk(n_heads * 512 + 1)[1:].reshape(n_heads, 512), mk(n_heads)
    window, pooled = mk(window_rows, 512), mk(n_rows, 512)
    got = fused_decode_sdpa(q, window, row, pooled, sel, sinks, inv, params, scale=512 ** -0.5)
    win = window.clone()
    if write_idx < window_rows:
        win[write_idx] = row
    out = sparse_attention(rope(q.reshape(n_heads, 1, 512)).reshape(1, n_heads, 1, 512), pooled, sel.reshape(1, 1, -1),
                           sinks.float(), pos0=max(pos, window_rows - 1), window=0, ratio=0,
                           raw_kv=win[None] if window_rows else None, scale=512 ** -0.5, d_v=512, out_dtype=h16)
    ref = rope(out.reshape(n_heads, 1, 512), inverse=True).reshape(n_heads, 512)
    assert torch.equal(got.view(torch.int16), ref.view(torch.int16))
