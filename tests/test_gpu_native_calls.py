"""The native host calls against the Python operators they stand in for: the same bits in the plain case, and everything
else (conversions, copies, errors) left to Python."""
import numpy as np
import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

from moespresso_b200 import _abi
from moespresso_b200 import _torchabi as _t
from moespresso_b200.deepseek_v4.attention import rope_inverse_frequencies
from moespresso_b200.deepseek_v4.decode_attention_kernel import fused_decode_prep, fused_decode_sdpa
from moespresso_b200.deepseek_v4.decode_step import LatentCache, sparse_decode_step
from moespresso_b200.qwen.full_attention import QuantizedKVCache, sdpa_decode_q8
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture
def taken(monkeypatch):
    """Names of the native calls that took their case."""
    need_gpu()
    names = []
    real = _t.native

    def spy(name, *args):
        r = real(name, *args)
        if r is not None:
            names.append(name)
        return r
    for mod in ("deepseek_v4.decode_step", "deepseek_v4.decode_attention_kernel", "qwen.full_attention"):
        monkeypatch.setattr(f"moespresso_b200.{mod}.native", spy)
    return names


def _python(f):
    """The same call through the Python operators: a timed launch is one that the native calls leave alone."""
    _t.TIMER = {}
    try:
        return f()
    finally:
        _t.TIMER = None


def _cache(kind, lens, gen):
    total, D = sum(lens), 576
    if kind == "int8":
        kv = torch.randint(-127, 128, (total, D), generator=gen, device="cuda").to(torch.int8)
        scales = (torch.rand(total, generator=gen, device="cuda") * 0.1 + 1e-3).half()
    else:
        kv, scales = torch.randn(total, D, generator=gen, device="cuda").to(kind), None
    keys = torch.randn(total, 64, generator=gen, device="cuda")
    starts = np.concatenate([[0], np.cumsum(lens)[:-1]])
    return LatentCache(kv=kv, kv_scales=scales, idx_keys=keys if kind == torch.float32 else keys.to(torch.float8_e4m3fn),
                       row_start=torch.tensor(starts, dtype=torch.int64, device="cuda"),
                       row_count=torch.tensor(lens, dtype=torch.int32, device="cuda"), max_rows=max(lens))


@pytest.mark.parametrize("kind,qdt", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), ("int8", torch.bfloat16),
                                      (torch.float16, torch.float16)])
def test_decode_step(kind, qdt, taken):
    gen = torch.Generator(device="cuda").manual_seed(3)
    lens = [1500, 700]
    cache = _cache(kind, lens, gen)
    B, H = len(lens), 64
    q = torch.randn(H, B, 576, generator=gen, device="cuda").to(qdt).permute(1, 0, 2)        # any strides on batch and heads
    iq, w = torch.randn(B, 16, 64, generator=gen, device="cuda").to(qdt), torch.randn(B, 16, generator=gen, device="cuda")
    sinks = torch.randn(H, generator=gen, device="cuda")
    f = lambda **kw: sparse_decode_step(q, iq, w, cache, k=300, scale=0.05, d_v=512, return_ids=True, return_scores=True, **kw)
    for kw in ({}, {"sinks": sinks, "out_dtype": torch.bfloat16}, {"exact_fp32": True}):
        del taken[:]
        got = f(**kw)
        assert taken == ["decode_step"]
        ref = _python(lambda: f(**kw))
        assert len(got) == len(ref) == 3
        for x, y in zip(got, ref):
            assert x.dtype == y.dtype and x.shape == y.shape and x.stride() == y.stride() and torch.equal(x, y)
    # left to Python: head weights that need a copy, counts of another type, a k that is not a plain int, a partial
    del taken[:]
    ww = torch.stack([w, w], -1)[..., 0]
    assert torch.equal(sparse_decode_step(q, iq, ww, cache, k=300, scale=0.05, d_v=512),
                       sparse_decode_step(q, iq, w, cache, k=np.int64(300), scale=0.05, d_v=512))
    sparse_decode_step(q, iq, w, cache, k=300, scale=0.05, d_v=512, partial=True)
    assert taken == []
    with pytest.raises(ValueError):
        sparse_decode_step(q, iq, w, cache, k=0, scale=0.05, d_v=512)
    with pytest.raises(RuntimeError):
        sparse_decode_step(q.cpu(), iq, w, cache, k=300, scale=0.05, d_v=512)


def test_decode_step_on_a_side_stream(taken):
    """The launches go to the current stream, the outputs belong to it."""
    gen = torch.Generator(device="cuda").manual_seed(4)
    cache = _cache(torch.bfloat16, [2000], gen)
    q, iq = (torch.randn(1, h, d, generator=gen, device="cuda").bfloat16() for h, d in ((64, 576), (16, 64)))
    w = torch.randn(1, 16, generator=gen, device="cuda")
    f = lambda: sparse_decode_step(q, iq, w, cache, k=256, scale=0.05, d_v=512)
    ref = f()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        late = torch.zeros_like(q)
        torch.cuda._sleep(2_000_000)
        late.copy_(q)
        out = sparse_decode_step(late, iq, w, cache, k=256, scale=0.05, d_v=512)
    side.synchronize()
    assert torch.equal(out, ref) and taken == ["decode_step"] * 2


@pytest.mark.parametrize("wide", [False, True])
def test_token_operators(wide, taken):
    gen = torch.Generator(device="cuda").manual_seed(5)
    n = lambda *s, dt=torch.float16: torch.randn(s, generator=gen, device="cuda").to(dt)
    inv = torch.as_tensor(rope_inverse_frequencies(64, 160000.0), device="cuda").float()
    params = torch.tensor([4003, 3], dtype=torch.int64 if wide else torch.int32, device="cuda")
    prep = (n(64, 128), n(900, 128, dt=torch.float32), n(64, dt=torch.float32), n(512), inv, params)
    f = lambda *p: fused_decode_prep(*p, scale=0.1, topk=256)
    got, ref = f(*prep), _python(lambda: f(*prep))
    assert all(torch.equal(x, y) and x.dtype == y.dtype for x, y in zip(got, ref))
    sdpa = (n(64, 512), n(128, 512), got[1], n(900, 512), got[0], n(64), inv, params)
    g = lambda *p: fused_decode_sdpa(*p, scale=0.05)
    assert torch.equal(g(*sdpa), _python(lambda: g(*sdpa)))
    assert taken == ["fused_decode_prep", "fused_decode_sdpa"]
    # a window of another stride is copied by the Python operator; errors are its own
    del taken[:]
    strided = torch.cat([sdpa[1], sdpa[1]], 1)[:, :512]
    assert torch.equal(g(sdpa[0], strided, *sdpa[2:]), _python(lambda: g(*sdpa)))
    assert taken == []
    with pytest.raises(ValueError):
        fused_decode_prep(*prep, scale=0.1, topk=900)
    with pytest.raises(ValueError):
        g(sdpa[0].float(), *sdpa[1:])


def test_q8_token(taken):
    gen = torch.Generator(device="cuda").manual_seed(6)
    n = lambda *s: torch.randn(s, generator=gen, device="cuda").bfloat16()
    caches = [QuantizedKVCache(2, 256, 600) for _ in range(2)]
    k, v = n(1, 2, 500, 256), n(1, 2, 500, 256)
    steps = [(n(1, 2, 1, 256), n(1, 2, 1, 256)) for _ in range(3)]
    steps.append((n(1, 2, 3, 512)[..., :256], n(1, 2, 3, 512)[..., :256]))                   # row strides of their own
    q = n(1, 16, 1, 256)
    outs = []
    for i, c in enumerate(caches):
        def walk():
            for x, y in [(k, v), *steps]:
                pre = c.update_and_fetch(x, y)
            return [*pre[0], *pre[1], sdpa_decode_q8(q, *pre[0], *pre[1], 0.0625)]
        outs.append(walk() if i == 0 else _python(walk))
    assert taken == ["q8_append"] * 5 + ["q8_decode"]
    assert caches[0].offset == caches[1].offset == 506
    for x, y in zip(*outs):
        assert x.shape == y.shape and x.stride() == y.stride() and x.dtype == y.dtype and torch.equal(x, y)
    del taken[:]
    c = caches[0]
    c.update_and_fetch(steps[0][0].float(), steps[0][1].float())                             # another type: converted in Python
    c.update_and_fetch(steps[0][0], steps[3][1][:, :, :1])                                   # keys and values of two layouts
    assert taken == [] and c.offset == 508
    with pytest.raises(ValueError):
        c.update_and_fetch(k, v)                                                             # capacity
    assert c.offset == 508
    # rows of another width than the kernel's 256 features: not the native call's, and refused before any launch
    del taken[:]
    narrow = QuantizedKVCache(2, 128, 600)
    narrow.offset = 500
    before = _abi.load().mxb_kernel_launches()
    with pytest.raises(ValueError):
        sdpa_decode_q8(q, *narrow.state[0], *narrow.state[1], 0.0625)
    assert taken == [] and _abi.load().mxb_kernel_launches() == before


class _Plain(torch.Tensor):
    pass


def test_modes_and_wrappers_are_left_to_python(taken):
    """Function and dispatch modes, tensor subclasses and the wrappers of torch.func: the native calls see none of them."""
    gen = torch.Generator(device="cuda").manual_seed(7)
    cache = _cache(torch.bfloat16, [1500], gen)
    q, iq = (torch.randn(1, h, d, generator=gen, device="cuda").bfloat16() for h, d in ((64, 576), (16, 64)))
    w = torch.randn(1, 16, generator=gen, device="cuda")
    f = lambda x=q: sparse_decode_step(x, iq, w, cache, k=256, scale=0.05, d_v=512)
    ref = f()
    assert taken == ["decode_step"]
    del taken[:]
    seen = []

    class Functions(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append("function")
            return func(*args, **(kwargs or {}))

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append("dispatch")
            return func(*args, **(kwargs or {}))
    for mode, name in ((Functions, "function"), (Dispatch, "dispatch")):
        del seen[:]
        with mode():
            out = f()
        assert torch.equal(out, ref) and taken == [] and name in seen       # the operator's own tensor calls went through it
    assert torch.equal(f(q.as_subclass(_Plain)).as_subclass(torch.Tensor), ref)
    assert torch.equal(f(torch.nn.Parameter(q)), ref) and taken == ["decode_step"]       # (a parameter is a plain tensor)
    args = lambda x: (x, iq, w, cache.kv, None, cache.idx_keys, cache.row_start, cache.row_count, cache.max_rows, 256, 0.05, 512, None,
                      torch.float32, False)

    def inside(x):
        seen.append(_t.native("decode_step", *args(x)))
        return x.float().sum()
    del seen[:]
    torch.func.vmap(inside)(torch.stack([q, q]))
    torch.func.grad(inside)(q.float())
    assert seen == [None, None] and _t.native("decode_step", *args(q)) is not None


def test_native_calls_in_a_graph(taken):
    """Under capture the outputs and scratch come from the graph's pool, and a replay computes from what the inputs hold then."""
    gen = torch.Generator(device="cuda").manual_seed(8)
    cache = _cache(torch.float32, [1800], gen)
    q, iq = (torch.randn(1, h, d, generator=gen, device="cuda") for h, d in ((64, 576), (16, 64)))
    w = torch.randn(1, 16, generator=gen, device="cuda")
    f = lambda: sparse_decode_step(q, iq, w, cache, k=256, scale=0.05, d_v=512, return_ids=True)
    f()
    graph = torch.cuda.CUDAGraph()
    del taken[:]
    with torch.cuda.graph(graph):
        out, ids = f()
    assert taken == ["decode_step"]
    for _ in range(3):
        q.copy_(torch.randn(q.shape, generator=gen, device="cuda"))
        iq.copy_(torch.randn(iq.shape, generator=gen, device="cuda"))
        graph.replay()
        ref = f()
        assert torch.equal(out, ref[0]) and torch.equal(ids, ref[1])
