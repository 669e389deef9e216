"""Kernels that are launched while the one before them runs: back to back over changing inputs they give the bits that they
give with the device idle between the calls."""
import pytest
import torch

from moespresso_b200.deepseek_v4.attention import rope_inverse_frequencies, topk_select
from moespresso_b200.deepseek_v4.decode_attention_kernel import fused_decode_prep, fused_decode_sdpa
from moespresso_b200.deepseek_v4.decode_step import LatentCache, sparse_decode_step
from moespresso_b200.deepseek_v4.indexed_attention_kernel import sparse_attention
from moespresso_b200.qwen.full_attention import QuantizedKVCache, sdpa_decode_q8
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu
STEPS = 60


def _both(step):
    """step(i) -> tensors; all steps in a row, then one at a time."""
    torch.cuda.synchronize()
    row = [step(i) for i in range(STEPS)]
    torch.cuda.synchronize()
    for i in range(STEPS):
        one = step(i)
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(row[i], one)), i


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
    _both(step)


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
    _both(lambda i: sparse_decode_step(q[i], iq[i], w[i], cache, k=300, scale=0.05, d_v=512, return_ids=True, return_scores=True))


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
    _both(step)


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
