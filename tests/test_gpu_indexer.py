"""Indexer score kernels against the CPU oracle (float64)."""
import numpy as np
import pytest
import torch

from moespresso_b200 import synth
from moespresso_b200.deepseek_v4 import indexed_attention_kernel as iak
from oracle import ds4
from tests.gpu_util import bf16_round, dev, f16_round, fp8_from_bits, need_gpu

pytestmark = pytest.mark.gpu


def _case(rng, B, H, T, D, R):
    q = rng.standard_normal((B, H, T, D)).astype(np.float32)
    keys = rng.standard_normal((B, R, D)).astype(np.float32)
    w = (rng.standard_normal((B, T, H)) / 4).astype(np.float32)
    return q, keys, w


def _oracle(q, keys, w, pos0, ratio):
    return np.stack([ds4.indexer_scores(q[b].transpose(1, 0, 2), keys[b], w[b], pos0=pos0, ratio=ratio)
                     for b in range(q.shape[0])])


@pytest.mark.parametrize("B,H,T,D,R,pos0,ratio", [
    (1, 16, 1, 64, 4096, 0, 0),          # config-1 shape
    (2, 64, 5, 128, 333, 1200, 4),       # reference head shape, ragged tile, causal mask
    (1, 3, 2, 64, 1, 7, 4),              # single row, odd head count
    (1, 8, 9, 64, 130, 300, 4),          # masked tail inside the chunk
])
def test_exact_fp32_matches_oracle(B, H, T, D, R, pos0, ratio):
    need_gpu()
    rng = np.random.default_rng(5)
    q, keys, w = _case(rng, B, H, T, D, R)
    got = iak.indexer_scores_tiled_live(dev(q), dev(w), dev(keys), pos0=pos0, ratio=ratio).cpu().numpy()
    ref = _oracle(q, keys, w, pos0, ratio)
    assert np.array_equal(np.isneginf(got), np.isneginf(ref))
    fin = np.isfinite(ref)
    np.testing.assert_allclose(got[fin], ref[fin], rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("form", ["bf16", "f16", "fp8_bf16", "fp8_f16"])
@pytest.mark.parametrize("B,H,T,D,R,pos0,ratio", [
    (1, 16, 1, 64, 4096, 0, 0),
    (2, 16, 40, 64, 1000, 3000, 4),      # token tiles x 16 heads: 16 tokens and a ragged last tile for FP8 keys, 8 for 16-bit ones
    (1, 64, 7, 128, 700, 2500, 4),       # D = 128 (two swizzle slabs), 64 heads
    (3, 32, 1, 64, 129, 0, 0),
    (2, 16, 1, 64, 1000, 1500, 4),       # one token WITH the causal row mask: rows >= (1500 + 1) // 4 are -inf
])
def test_tensor_core_path_matches_oracle(form, B, H, T, D, R, pos0, ratio):
    need_gpu()
    rng = np.random.default_rng(11)
    q, keys, w = _case(rng, B, H, T, D, R)
    if form.startswith("fp8"):
        bits = synth.to_e4m3_bits(keys)
        keys_r = synth.e4m3_bits_to_f32(bits)
        kt = fp8_from_bits(bits)
        qdt = torch.bfloat16 if form.endswith("bf16") else torch.float16
    else:
        qdt = torch.bfloat16 if form == "bf16" else torch.float16
        keys_r = bf16_round(keys) if form == "bf16" else f16_round(keys)
        kt = dev(keys_r, qdt)
    q_r = bf16_round(q) if qdt == torch.bfloat16 else f16_round(q)
    before = iak.indexer_scores_call_counts()
    got = iak.indexer_scores_tiled_live(dev(q_r, qdt), dev(w), kt, pos0=pos0, ratio=ratio, check=True).cpu().numpy()
    ref = _oracle(q_r, keys_r, w, pos0, ratio)
    assert np.array_equal(np.isneginf(got), np.isneginf(ref))
    fin = np.isfinite(ref)
    np.testing.assert_allclose(got[fin], ref[fin], rtol=2e-4, atol=2e-3)
    if form.startswith("fp8"):   # the direct FP8 tensor-core mode: reduced-precision accumulation
        got3 = iak.indexer_scores_tiled_live(dev(q_r, qdt), dev(w), kt, pos0=pos0, ratio=ratio, fp8_mma=True,
                                             check=True).cpu().numpy()
        np.testing.assert_allclose(got3[fin], ref[fin], rtol=5e-3, atol=5e-2)
        before["fp8"] += 1
    # the explicit fp32 mode agrees as well
    got2 = iak.indexer_scores_tiled_live(dev(q_r, qdt), dev(w), kt, pos0=pos0, ratio=ratio,
                                         exact_fp32=True).cpu().numpy()
    np.testing.assert_allclose(got2[fin], ref[fin], rtol=1e-5, atol=1e-4)
    after = iak.indexer_scores_call_counts()
    assert sum(after.values()) == sum(before.values()) + 2


def test_ragged_batch_fp8_scores():
    need_gpu()
    c = synth.config3(seed=3, lens=[700, 129, 4096, 1, 2500])
    keys_r = synth.e4m3_bits_to_f32(c["idx_key_bits"])
    rs = dev(c["row_start"]); rc = dev(c["lens"].astype(np.int32))
    got = iak.indexer_scores(dev(c["idx_q"], torch.bfloat16)[:, :, None, :], dev(c["idx_w"])[:, None, :].contiguous(),
                             fp8_from_bits(c["idx_key_bits"]), n_rows=int(c["lens"].max()), row_start=rs,
                             row_count=rc, check=True).cpu().numpy()
    for b, (s, n) in enumerate(zip(c["row_start"], c["lens"])):
        ref = ds4.indexer_scores(c["idx_q"][b][None], keys_r[s:s + n], c["idx_w"][b][None])[0]
        np.testing.assert_allclose(got[s:s + n], ref, rtol=2e-4, atol=2e-3)


def test_scan_counts_the_first_digit_of_the_selection():
    """The decode scan leaves, per sequence, the histogram of the top 11 bits of the selection keys of exactly the
    scores it wrote; a call the scan does not take refuses the histogram."""
    need_gpu()
    from tests.gpu_util import first_digit_hist
    c = synth.config3(seed=4, lens=[70000, 129, 33000, 1, 2500, 5000])
    B = int(c["lens"].size)
    rs = dev(c["row_start"]); rc = dev(c["lens"].astype(np.int32))
    q = dev(c["idx_q"], torch.bfloat16)[:, :, None, :]
    w = dev(c["idx_w"])[:, None, :].contiguous()
    keys = fp8_from_bits(c["idx_key_bits"])
    assert iak.scan_counts_digits(q, keys, n_tokens=1, ratio=0)
    hist = torch.zeros((B, iak.DIGIT_BINS), dtype=torch.int32, device="cuda")
    got = iak.indexer_scores(q, w, keys, n_rows=int(c["lens"].max()), row_start=rs, row_count=rc, digit_hist=hist)
    plain = iak.indexer_scores(q, w, keys, n_rows=int(c["lens"].max()), row_start=rs, row_count=rc)
    assert torch.equal(got, plain)                         # the same score bits with and without the counting
    sc, h = got.cpu().numpy(), hist.cpu().numpy()
    for b, (s, n) in enumerate(zip(c["row_start"], c["lens"])):
        np.testing.assert_array_equal(h[b], first_digit_hist(sc[s:s + n]))
        assert int(h[b].sum()) == int(n)
    # a second call adds on top (the selection is what clears the counters)
    iak.indexer_scores(q, w, keys, n_rows=int(c["lens"].max()), row_start=rs, row_count=rc, digit_hist=hist)
    np.testing.assert_array_equal(hist.cpu().numpy(), 2 * h)
    with pytest.raises(ValueError):                        # wrong shape
        iak.indexer_scores(q, w, keys, n_rows=int(c["lens"].max()), row_start=rs, row_count=rc, digit_hist=hist[:, :100])
    from moespresso_b200 import _abi
    with pytest.raises((_abi.MxbError, RuntimeError)):     # float32 keys: not the scan
        iak.indexer_scores(q.float(), w, dev(synth.e4m3_bits_to_f32(c["idx_key_bits"])), n_rows=int(c["lens"].max()),
                           row_start=rs, row_count=rc, digit_hist=hist)


def test_score_is_independent_of_row_partition():
    """A row's score bits do not depend on where the row sits in the table
    (needed for bit-exact top-k under KV-range sharding)."""
    need_gpu()
    rng = np.random.default_rng(2)
    q, keys, w = _case(rng, 1, 16, 1, 64, 5000)
    bits = synth.to_e4m3_bits(keys[0])
    qd, wd = dev(bf16_round(q), torch.bfloat16), dev(w)
    full = iak.indexer_scores_tiled_live(qd, wd, fp8_from_bits(bits)[None], pos0=0, ratio=0)[0, 0]
    for lo, hi in [(0, 1000), (1000, 1777), (1777, 5000)]:
        part = iak.indexer_scores_tiled_live(qd, wd, fp8_from_bits(bits[lo:hi])[None], pos0=0, ratio=0)[0, 0]
        assert torch.equal(part, full[lo:hi])


@pytest.mark.parametrize("D,H,rows", [(64, 1, 1), (64, 16, 33), (64, 17, 128 * 296 + 5), (128, 33, 31), (128, 64, 2500),
                                      (128, 64, 128 * 296 + 1), (64, 14, 128 * 296 + 7), (128, 29, 128 * 296 + 127)])
@pytest.mark.parametrize("qdt,kdt", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_exact_scores_of_one_token_have_the_bits_of_a_chunk(D, H, rows, qdt, kdt):
    """The kernel for one token splits the heads over warps; a chunk of two equal tokens takes the kernel that walks
    them in one thread.  Edges of the row tiles (32 and 128), both row widths, heads that do not fill the warps; calls
    of few heads and many rows, which go to the kernel for chunks, among them."""
    need_gpu()
    g = torch.Generator(device="cuda").manual_seed(rows + H)
    q = torch.randn(1, H, 1, D, generator=g, device="cuda").to(qdt)
    w = torch.randn(1, 1, H, generator=g, device="cuda")
    keys = torch.randn(rows, D, generator=g, device="cuda").to(kdt)
    one = iak.indexer_scores(q, w, keys, n_rows=rows, exact_fp32=True)
    two = iak.indexer_scores(q.expand(1, H, 2, D).contiguous(), w.expand(1, 2, H).contiguous(), keys, n_rows=rows,
                             exact_fp32=True)
    assert torch.equal(one.reshape(-1), two.reshape(2, rows)[0])


@pytest.mark.parametrize("form", ["bf16", "f16"])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("H,T,R", [
    (16, 9, 2049),    # 8 + 1 tokens: the second tile's drain groups 1-3 have none, group 0 has one
    (16, 13, 700),    # a group with one token of its two between full and empty groups
    (16, 15, 2049),   # the last group has one; 17 row tiles wrap the ring of four accumulators, the last holds one row
    (16, 41, 4096),
    (32, 7, 2049),    # four tokens of 32 heads per tile, the last tile ragged
    (64, 3, 1025),    # two tokens of 64 heads
    (32, 333, 5003),  # tiles of 256 columns, shared by two drain groups: eight tokens, the last tile has five
    (48, 333, 5003),  # five tokens of 48 heads (two and three), the last tile has three
    (64, 331, 5003),  # four tokens, the last tile has three
])
def test_partial_token_tiles_of_16bit_keys(form, H, T, R, D):
    """Tiles that are not full, for the drain with the weights in registers (16 heads) and the one that reads them:
    against the fp32 kernel on the same operands; nothing is written behind the last token or row."""
    need_gpu()
    dt = torch.bfloat16 if form == "bf16" else torch.float16
    g = torch.Generator(device="cuda").manual_seed(H + T + R)
    mk = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    q, w, keys = mk(1, H, T, D).to(dt), mk(1, T, H) / 4, mk(1, R, D).to(dt)
    kw = dict(pos0=2 * R, ratio=4)
    ref = iak.indexer_scores_tiled_live(q, w, keys, exact_fp32=True, **kw)
    store = torch.full((1, T + 3, R + 5), 12345.0, device="cuda")
    iak.indexer_scores_tiled_live(q, w, keys, out=store[:, :T, :R], check=True, **kw)
    got = store[:, :T, :R]
    assert torch.equal(torch.isneginf(got), torch.isneginf(ref))
    fin = torch.isfinite(ref)
    np.testing.assert_allclose(got[fin].cpu().numpy(), ref[fin].cpu().numpy(), rtol=2e-4, atol=2e-3)
    store[:, :T, :R] = 12345.0
    assert bool((store == 12345.0).all())


def test_more_token_tiles_than_a_grid_holds():
    """65,535 tiles of eight tokens (16 heads) and two more: the second launch continues where the first ended."""
    need_gpu()
    first = 8 * 65535
    T, H, D, R = first + 13, 16, 64, 33
    g = torch.Generator(device="cuda").manual_seed(1)
    q = torch.randn(1, H, T, D, generator=g, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(1, T, H, generator=g, device="cuda")
    keys = torch.randn(1, R, D, generator=g, device="cuda").bfloat16()
    got = iak.indexer_scores_tiled_live(q, w, keys, pos0=4 * R, ratio=4, check=True)
    for lo in (0, first - 8, first):
        part = iak.indexer_scores_tiled_live(q[:, :, lo:lo + 13], w[:, lo:lo + 13], keys, pos0=4 * R, ratio=4)
        assert torch.equal(got[:, lo:lo + 13], part)
    assert bool(torch.isfinite(got).all())
