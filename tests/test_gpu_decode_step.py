"""Whole sparse decode step (indexer score -> top-k -> sparse attention) against the oracle."""
import numpy as np
import pytest
import torch

from moespresso_b200 import synth
from moespresso_b200.deepseek_v4.decode_step import LatentCache, sparse_decode_step
from oracle import ds4
from tests.gpu_util import dev, fp8_from_bits, max_abs, need_gpu

pytestmark = pytest.mark.gpu


def boundary_exact(ids_gpu, scores_gpu, scores_ref, k):
    """Top-k parity when the two sides computed scores with different rounding: the GPU
    selection must be the exact top-k of the GPU's own score bits, and every row on which
    it differs from the oracle's selection must sit within rounding distance of the k-th
    boundary of the oracle's scores."""
    own = ds4.topk_ids(scores_gpu, k)[0]
    np.testing.assert_array_equal(ids_gpu, own)
    ref = ds4.topk_ids(scores_ref, k)[0]
    diff = np.setxor1d(ids_gpu[ids_gpu >= 0], ref[ref >= 0])
    if diff.size:
        kth = np.sort(scores_ref[np.isfinite(scores_ref)])[::-1][min(k, np.isfinite(scores_ref).sum()) - 1]
        assert np.all(np.abs(scores_ref[diff] - kth) <= 1e-3 * max(1.0, abs(kth)))
    return diff.size


def test_config1_step_fp32():
    need_gpu()
    c = synth.config1()
    cache = LatentCache(kv=dev(c["kv"]), kv_scales=None, idx_keys=dev(c["idx_keys"]),
                        row_start=dev(np.zeros(1, np.int64)), row_count=dev(np.array([4096], np.int32)),
                        max_rows=4096)
    out, ids, scores = sparse_decode_step(dev(c["q"])[None], dev(c["idx_q"])[None], dev(c["idx_w"])[None], cache,
                                          k=c["k"], scale=c["scale"], d_v=c["d_v"], return_ids=True,
                                          return_scores=True)
    ref_scores, ref_ids, ref_out = ds4.sparse_decode_step(c["q"], c["kv"], c["idx_q"], c["idx_keys"], c["idx_w"],
                                                          k=c["k"], scale=c["scale"], d_v=c["d_v"])
    np.testing.assert_allclose(scores.cpu().numpy(), ref_scores, rtol=1e-5, atol=1e-5)
    ndiff = boundary_exact(ids[0].cpu().numpy(), scores.cpu().numpy(), ref_scores, c["k"])
    if ndiff == 0:
        assert max_abs(out[0], ref_out) <= 1e-4
    else:  # attention over the GPU's own selection
        ref2 = ds4.indexed_mixed_attention_decode(c["q"], None, c["kv"], ids[0].cpu().numpy(), None, pos0=0,
                                                  window=0, ratio=0, scale=c["scale"], d_v=c["d_v"])
        assert max_abs(out[0], ref2) <= 1e-4


@pytest.mark.parametrize("lens", [[5000, 2049, 40000, 300], [50000, 47000]])
def test_config3_shaped_step(lens):
    need_gpu()
    c = synth.config3(seed=1, lens=lens)
    cache = LatentCache(kv=dev(c["kv"]), kv_scales=dev(c["kv_scales"]), idx_keys=fp8_from_bits(c["idx_key_bits"]),
                        row_start=dev(c["row_start"]), row_count=dev(c["lens"].astype(np.int32)),
                        max_rows=int(max(lens)))
    out, ids, scores = sparse_decode_step(dev(c["q"], torch.bfloat16), dev(c["idx_q"], torch.bfloat16),
                                          dev(c["idx_w"]), cache, k=c["k"], scale=c["scale"], d_v=c["d_v"],
                                          return_ids=True, return_scores=True)
    keys = synth.e4m3_bits_to_f32(c["idx_key_bits"])
    scores = scores.cpu().numpy(); ids = ids.cpu().numpy()
    for b, n in enumerate(lens):
        s = int(c["row_start"][b])
        ref_scores = ds4.indexer_scores(c["idx_q"][b][None], keys[s:s + n], c["idx_w"][b][None])[0]
        np.testing.assert_allclose(scores[s:s + n], ref_scores, rtol=2e-4, atol=2e-3)
        boundary_exact(ids[b], scores[s:s + n], ref_scores, c["k"])
        ref = ds4.indexed_mixed_attention_decode(c["q"][b], None, c["kv"][s:s + n], ids[b], None, pos0=0, window=0,
                                                 ratio=0, scale=c["scale"], d_v=c["d_v"],
                                                 kv_scales=c["kv_scales"][s:s + n])
        assert max_abs(out[b], ref) <= 2e-2


@pytest.mark.parametrize("graph", [True, False])
def test_plan_matches_eager_step(graph):
    """The CUDA-graph plan returns the bits of the eager step, from device or pinned-host inputs."""
    need_gpu()
    from moespresso_b200.deepseek_v4.decode_step import SparseDecodePlan
    c = synth.config3(seed=3, lens=[3000, 2500, 6000])
    cache = LatentCache(kv=dev(c["kv"]), kv_scales=dev(c["kv_scales"]), idx_keys=fp8_from_bits(c["idx_key_bits"]),
                        row_start=dev(c["row_start"]), row_count=dev(c["lens"].astype(np.int32)), max_rows=6000)
    q, iq, iw = dev(c["q"], torch.bfloat16), dev(c["idx_q"], torch.bfloat16), dev(c["idx_w"])
    eager = sparse_decode_step(q, iq, iw, cache, k=c["k"], scale=c["scale"], d_v=c["d_v"], out_dtype=torch.bfloat16)
    plan = SparseDecodePlan(cache, heads=64, d_qk=576, idx_heads=16, idx_dim=64, k=c["k"], scale=c["scale"],
                            d_v=c["d_v"], q_dtype=torch.bfloat16, out_dtype=torch.bfloat16, graph=graph)
    out = plan.run(q, iq, iw)
    torch.cuda.synchronize()
    assert torch.equal(out, eager)
    plan.q.zero_()
    out = plan.run(q.cpu().pin_memory(), iq.cpu().pin_memory(), iw.cpu().pin_memory())
    torch.cuda.synchronize()
    assert torch.equal(out, eager)
    plan.packed.zero_()
    host, (qv, iqv, iwv) = plan.host_buffer()
    qv.copy_(q.cpu())
    iqv.copy_(iq.cpu())
    iwv.copy_(iw.cpu())
    out = plan.run_packed(host)
    torch.cuda.synchronize()
    assert torch.equal(out, eager)


def test_plan_with_16bit_cache():
    """bf16 latent cache: the attention kernel gathers rows by TMA (tensor maps passed as kernel parameters); the
    captured graph must replay to the eager step's bits and stay within the 16-bit bound of the oracle."""
    need_gpu()
    from moespresso_b200.deepseek_v4.decode_step import SparseDecodePlan
    lens = [3000, 2500, 6000]
    c = synth.config3(seed=4, lens=lens)
    kv = synth.to_bf16_f32(c["kv"].astype(np.float32) * c["kv_scales"].astype(np.float32)[:, None])   # dequantised rows
    cache = LatentCache(kv=dev(kv, torch.bfloat16), kv_scales=None, idx_keys=fp8_from_bits(c["idx_key_bits"]),
                        row_start=dev(c["row_start"]), row_count=dev(c["lens"].astype(np.int32)), max_rows=6000)
    q, iq, iw = dev(c["q"], torch.bfloat16), dev(c["idx_q"], torch.bfloat16), dev(c["idx_w"])
    eager, ids = sparse_decode_step(q, iq, iw, cache, k=c["k"], scale=c["scale"], d_v=c["d_v"], return_ids=True)
    plan = SparseDecodePlan(cache, heads=64, d_qk=576, idx_heads=16, idx_dim=64, k=c["k"], scale=c["scale"],
                            d_v=c["d_v"], q_dtype=torch.bfloat16)
    for _ in range(2):
        out = plan.run(q, iq, iw)
        torch.cuda.synchronize()
        assert torch.equal(out, eager)
    ids = ids.cpu().numpy()
    # The 2e-2 bound is stated for unit-scale values.  These rows reach |v| = 12.7 (int8 x scale), where bf16 itself
    # resolves 0.0625 and the bf16 softmax weights (8 significant bits) move an output by up to |v| * 2^-9: the
    # bound scales with the table's magnitude.
    tol = 2e-2 * max(1.0, float(np.abs(kv).max()) / 4.0)
    for b, n in enumerate(lens):
        s = int(c["row_start"][b])
        ref = ds4.indexed_mixed_attention_decode(c["q"][b], None, kv[s:s + n], ids[b], None, pos0=0, window=0, ratio=0,
                                                 scale=c["scale"], d_v=c["d_v"])
        assert max_abs(eager[b], ref) <= tol


@pytest.mark.parametrize("sizes", [(0, 1, 15), (16, 17, 4097), (8192, 8191, (3 << 20) + 5)])
@pytest.mark.parametrize("offset", [0, 2])
def test_copy_buffers(sizes, offset):
    """Bytes on and off 16-byte boundaries, nothing copied behind them."""
    need_gpu()
    from moespresso_b200 import _abi
    from moespresso_b200 import _torchabi as _t
    a = _abi.CopyBuffersArgs()
    src = [torch.randint(1, 256, (n + 32,), dtype=torch.uint8, device="cuda") for n in sizes]
    dst = [torch.zeros(n + 32, dtype=torch.uint8, device="cuda") for n in sizes]
    for i, n in enumerate(sizes):
        a.dst[i], a.src[i], a.bytes[i] = dst[i].data_ptr() + offset, src[i].data_ptr() + 16, n
    _abi.check(_t.launch("copy_buffers", _abi.load().mxb_copy_buffers, a))
    for i, n in enumerate(sizes):
        assert torch.equal(dst[i][offset:offset + n], src[i][16:16 + n])
        assert int(dst[i].sum()) == int(src[i][16:16 + n].sum())


def test_plan_takes_inputs_of_every_layout():
    """Contiguous device inputs are copied together, strided or otherwise typed ones one by one: the same step."""
    need_gpu()
    from moespresso_b200.deepseek_v4.decode_step import SparseDecodePlan
    g = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    lens = [1500, 1100]
    cache = LatentCache(kv=mk(2600, 576).bfloat16(), kv_scales=None, idx_keys=mk(2600, 64).to(torch.float8_e4m3fn),
                        row_start=torch.tensor([0, 1500], device="cuda"),
                        row_count=torch.tensor(lens, dtype=torch.int32, device="cuda"), max_rows=1500)
    plan = SparseDecodePlan(cache, heads=64, d_qk=576, idx_heads=16, idx_dim=64, k=256, scale=576 ** -0.5, d_v=512)
    q, iq, iw = mk(2, 64, 576).bfloat16(), mk(2, 16, 64).bfloat16(), mk(2, 16)
    want = plan.run(q, iq, iw).clone()
    for args in ((q.float(), iq, iw), (q.transpose(1, 2).contiguous().transpose(1, 2), iq, iw), (q.cpu(), iq, iw.cpu())):
        plan.packed.zero_()
        assert torch.equal(plan.run(*args), want)


def _plan_over(batch, rows, k, kv):
    from moespresso_b200.deepseek_v4.decode_step import SparseDecodePlan
    g = torch.Generator(device="cuda").manual_seed(batch + rows)
    mk = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    n = batch * rows
    lens = torch.full((batch,), rows, dtype=torch.int32, device="cuda")
    cache = LatentCache(kv=mk(n, 576).mul(30).clamp(-127, 127).to(torch.int8) if kv == "int8" else mk(n, 576).to(torch.bfloat16),
                        kv_scales=(0.01 + 0.02 * torch.rand(n, generator=g, device="cuda")).half() if kv == "int8" else None,
                        idx_keys=mk(n, 64).to(torch.float8_e4m3fn), row_count=lens, max_rows=rows,
                        row_start=torch.arange(batch, dtype=torch.int64, device="cuda") * rows)
    plan = SparseDecodePlan(cache, heads=64, d_qk=576, idx_heads=16, idx_dim=64, k=k, scale=576 ** -0.5, d_v=512)
    inputs = [(mk(batch, 64, 576).bfloat16(), mk(batch, 16, 64).bfloat16(), mk(batch, 16)) for _ in range(4)]
    return cache, plan, inputs


@pytest.mark.parametrize("batch,rows,k,kv", [
    (1, 3000, 512, "int8"),        # selection of one CTA, most SMs free for the attention to set up on
    (1, 3000, 512, "bf16"),
    (3, 20000, 512, "bf16"),       # clusters
    (40, 20000, 2048, "int8"),     # a partial selection wave, splits in clusters
    (150, 3000, 512, "bf16"),      # more tokens than SMs
])
def test_early_start_behind_the_selection_gives_the_same_bits(batch, rows, k, kv):
    """The attention may start while the selection finishes.  Steps with changing inputs, one after another without a
    wait, against the selection and an attention that waits: the ids and outputs of every step."""
    need_gpu()
    from moespresso_b200.deepseek_v4.attention import topk_select
    from moespresso_b200.deepseek_v4.indexed_attention_kernel import indexer_scores, sparse_attention
    cache, plan, inputs = _plan_over(batch, rows, k, kv)
    want = []
    for q, iq, iw in inputs:
        scores = indexer_scores(iq[:, :, None], iw[:, None], cache.idx_keys, n_rows=rows, row_start=cache.row_start,
                                row_count=cache.row_count)
        ids = topk_select(scores, k, valid=cache.row_count, row_start=cache.row_start, n=rows)
        torch.cuda.synchronize()
        out = sparse_attention(q[:, :, None], cache.kv, ids[:, None], None, pos0=0, window=0, ratio=0, scale=576 ** -0.5,
                               d_v=512, kv_scales=cache.kv_scales, comp_row_start=cache.row_start,
                               comp_row_count=cache.row_count, n_comp=rows)
        want.append((ids, out[:, :, 0]))
    bad = torch.zeros((), dtype=torch.int64, device="cuda")
    for step in range(200):
        i = (step * 7 + step // 5) % len(inputs)
        if step % 2:
            out, ids = plan.run(*inputs[i]), plan.ids
        else:
            out, ids = sparse_decode_step(*inputs[i], cache, k=k, scale=576 ** -0.5, d_v=512, return_ids=True)
        bad += (ids != want[i][0]).sum() + (out != want[i][1]).sum()
    assert int(bad) == 0


def test_host_fed_steps_between_others():
    """run(), load_inputs() and run_packed() in turn without a wait: every step's output is its own inputs'."""
    need_gpu()
    _, plan, inputs = _plan_over(32, 30000, 512, "bf16")
    want = []
    for x in inputs:
        want.append(plan.run(*x).clone())
        torch.cuda.synchronize()
    host = []
    for x in inputs:
        buf, views = plan.host_buffer()
        for v, t in zip(views, x):
            v.copy_(t.cpu())
        host.append(buf)
    outs = []
    for step in range(60):
        i, j = step % 4, (step + 1 + step // 4) % 4
        outs.append((j, plan.run(*inputs[j]).clone()) if step % 3 else (j, None))
        if not step % 3:
            plan.load_inputs(*inputs[j])
        outs.append((i, plan.run_packed(host[i]).clone()))
    torch.cuda.synchronize()
    for i, out in outs:
        assert out is None or torch.equal(out, want[i])
