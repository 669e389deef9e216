"""Kernels that are launched while the one before them runs: back to back over changing inputs they give the bits that they
give with the device idle between the calls, and what a reference gives whose stages cannot overlap: the single operators with
an idle device between them, or the sums in float64."""
import pytest
import torch

from moespresso_b200.deepseek_v4.attention import apply_rope_tail, rope_inverse_frequencies, topk_select
from moespresso_b200.deepseek_v4.decode_attention_kernel import fp8_kv_prefix_rows, fused_decode_prep, fused_decode_sdpa
from moespresso_b200.deepseek_v4.decode_step import LatentCache, sparse_decode_step
from moespresso_b200.deepseek_v4.indexed_attention_kernel import indexer_scores, sparse_attention
from moespresso_b200.deepseek_v4.indexer_score_kernel import fused_qat_indexer_scores
from moespresso_b200.qwen.full_attention import QuantizedKVCache, dequantize_affine_q8, sdpa_decode_q8
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu
STEPS = 60


def _both(step, apart=None, tol=0.0):
    """step(i) -> tensors; all steps in a row, then one at a time; then some of them against ``apart(i)``, within ``tol``."""
    torch.cuda.synchronize()
    row = [step(i) for i in range(STEPS)]
    torch.cuda.synchronize()
    for i in range(STEPS):
        one = step(i)
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(row[i], one)), i
    for i in (0, 1, STEPS // 2, STEPS - 1) if apart else ():
        ref = apart(i)
        assert len(ref) == len(row[i])
        for x, y in zip(row[i], ref):
            assert torch.equal(x, y) if tol == 0.0 else float((x.double() - y).abs().max()) <= tol, i


def _idle(x):
    torch.cuda.synchronize()
    return x


def _n(gen, *s, dt=torch.float32):
    return torch.randn(s, generator=gen, device="cuda").to(dt)


def test_ratio4_token():
    need_gpu()
    gen, h = torch.Generator(device="cuda").manual_seed(1), torch.float16
    inv = torch.as_tensor(rope_inverse_frequencies(64, 160000.0), device="cuda").float()
    q, qi, kv, w = _n(gen, STEPS, 64, 512, dt=h), _n(gen, STEPS, 64, 128, dt=h), _n(gen, STEPS, 512, dt=h), _n(gen, STEPS, 64)
    pool, rows, window, sinks = _n(gen, 1700, 128), _n(gen, 1700, 512, dt=h), _n(gen, 127, 512, dt=h), _n(gen, 64, dt=h)
    pos = torch.stack([torch.arange(STEPS) + 6800, torch.arange(STEPS) % 127], 1).int().cuda()

    def step(i):
        sel, row, scores = fused_decode_prep(qi[i], pool, w[i], kv[i], inv, pos[i], scale=0.1, topk=256)
        return sel, row, scores, fused_decode_sdpa(q[i], window, row, rows, sel, sinks, inv, pos[i], scale=0.05)

    def apart(i):
        at = pos[i, 0:1].long()
        rope = lambda x, **kw: _idle(apply_rope_tail(x, at, inv_freq=inv, half_chain=True, **kw))  # noqa: E731
        scores = _idle(fused_qat_indexer_scores(qi[i].reshape(1, 64, 1, 128), pool[None], w[i].reshape(1, 1, 64), 0.1))
        sel = _idle(topk_select(scores.reshape(1, -1), 256))[0]
        row = _idle(fp8_kv_prefix_rows(kv[i].float()[None]))[0].to(h)
        row[448:] = rope(kv[i].reshape(1, 1, 512)).reshape(-1)[448:]
        win = window.clone()
        win[int(pos[i, 1])] = row
        out = _idle(sparse_attention(rope(q[i].reshape(64, 1, 512)).reshape(1, 64, 1, 512), rows, sel.reshape(1, 1, -1), sinks.float(),
                                     pos0=int(pos[i, 0]), window=0, ratio=0, raw_kv=win[None], scale=0.05, d_v=512, out_dtype=h))
        return sel, row, scores.reshape(-1), rope(out.reshape(64, 1, 512), inverse=True).reshape(64, 512)
    _both(step, apart)


@pytest.mark.parametrize("kv,lens", [(torch.float32, [4000]), (torch.bfloat16, [1200, 3000, 700]), (torch.bfloat16, [60000])])
def test_decode_step(kv, lens):
    need_gpu()
    gen = torch.Generator(device="cuda").manual_seed(2)
    B, dt = len(lens), torch.float32 if kv == torch.float32 else torch.bfloat16
    keys = _n(gen, sum(lens), 64)
    cache = LatentCache(kv=_n(gen, sum(lens), 576, dt=kv), kv_scales=None,
                        idx_keys=keys if kv == torch.float32 else keys.to(torch.float8_e4m3fn),
                        row_start=torch.tensor([sum(lens[:i]) for i in range(B)], device="cuda"),
                        row_count=torch.tensor(lens, dtype=torch.int32, device="cuda"), max_rows=max(lens))
    q, iq, w = _n(gen, STEPS, B, 64, 576, dt=dt), _n(gen, STEPS, B, 16, 64, dt=dt), _n(gen, STEPS, B, 16)

    def apart(i):
        kw = dict(row_start=cache.row_start, row_count=cache.row_count)
        scores = _idle(indexer_scores(iq[i][:, :, None], w[i][:, None], cache.idx_keys, n_rows=cache.max_rows, **kw))
        ids = _idle(topk_select(scores, 300, valid=cache.row_count, row_start=cache.row_start, n=cache.max_rows))
        out = _idle(sparse_attention(q[i][:, :, None], cache.kv, ids[:, None], None, pos0=0, window=0, ratio=0, scale=0.05, d_v=512,
                                     comp_row_start=cache.row_start, comp_row_count=cache.row_count, n_comp=cache.max_rows))
        return out[:, :, 0], ids, scores
    _both(lambda i: sparse_decode_step(q[i], iq[i], w[i], cache, k=300, scale=0.05, d_v=512, return_ids=True, return_scores=True),
          apart)


def test_q8_token():
    need_gpu()
    gen, b = torch.Generator(device="cuda").manual_seed(3), torch.bfloat16
    cache = QuantizedKVCache(2, 256, 5000)
    cache.update_and_fetch(_n(gen, 1, 2, 4999, 256, dt=b), _n(gen, 1, 2, 4999, 256, dt=b))
    k, v, q = (_n(gen, STEPS, 1, h, 1, 256, dt=b) for h in (2, 2, 16))

    def step(i):
        cache.offset = 4999
        pre = cache.update_and_fetch(k[i], v[i])
        return (sdpa_decode_q8(q[i], *pre[0], *pre[1], 0.0625),)

    def apart(i):
        cache.offset = 4999
        pre = _idle(cache.update_and_fetch(k[i], v[i]))
        kd, vd = (dequantize_affine_q8(*t, dtype=torch.float32).double().repeat_interleave(8, 1) for t in pre)
        p = torch.softmax(q[i].double() @ kd.transpose(2, 3) * 0.0625, -1)
        return (p @ vd,)
    _both(step, apart, tol=2e-2)     # as for the composed path: fp16 operands, bf16 result


def test_operands_written_by_the_launch_before():
    """Scores and lists from kernels of torch, which let nothing start early, and a selection in between."""
    need_gpu()
    gen = torch.Generator(device="cuda").manual_seed(4)
    rows = _n(gen, 3000, 512, dt=torch.float16)
    base, q = _n(gen, 2, 3000), _n(gen, 2, 64, 1, 512, dt=torch.float16)

    def step(i):
        ids = topk_select(base * float(1 + i) + base.flip(1), 200)
        out = sparse_attention(q * (1.0 + 0.01 * i), rows, (ids // 2 * 2)[:, None, :].contiguous(), None, pos0=0, window=0, ratio=0,
                               scale=0.05, comp_row_start=torch.zeros(2, dtype=torch.int64, device="cuda"), n_comp=3000)
        return ids, out
    _both(step)
