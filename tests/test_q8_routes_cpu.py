"""Which calls of the affine-q8 cache reach the paired kernels, which take raw pointers, strides and widths on trust:
routing and refusals on the CPU, with the launches replaced."""
import ctypes as C

import pytest
import torch

from moespresso_b200.qwen import full_attention as fa

BF = torch.bfloat16


def _past(Hkv, P, words, groups):
    one = lambda: (torch.zeros(1, Hkv, P, words, dtype=torch.int32), *(torch.zeros(1, Hkv, P, groups, dtype=BF) for _ in range(2)))  # noqa: E731
    return (*one(), *one())


def _no_launch(monkeypatch):
    monkeypatch.setattr(fa, "require_cuda", lambda *tensors: torch.device("cpu"))
    for name in ("_q8_pair", "_q8_call"):
        monkeypatch.setattr(fa, name, lambda *a, **k: pytest.fail("a kernel would have been launched"))


@pytest.mark.parametrize("words,groups", [(32, 2), (128, 8), (64, 2), (64, 8)])
def test_past_of_another_width_is_refused(monkeypatch, words, groups):
    """A head of the [past + chunk] operand is 256 wide: rows of 128 or 512 features, or of 256 with scales for another
    width, must not be expanded into it."""
    _no_launch(monkeypatch)
    chunk = torch.zeros(1, 2, 3, 256, dtype=BF)
    with pytest.raises(ValueError):
        fa.sdpa_fa_prefill_q8(torch.zeros(1, 4, 3, 256, dtype=BF), *_past(2, 5, words, groups), chunk, chunk, 1 / 16)


@pytest.mark.parametrize("P", [0, 5])
def test_empty_past_and_chunk_that_broadcasts(monkeypatch, P):
    """Of an empty past nothing is read, so its tensors may be anywhere ("cpu" stands for the device here, "meta" for
    another place); values of one head for both are copied like any others."""
    operand = {}
    monkeypatch.setattr(fa, "dequantize_affine_q8", lambda *q8, out: out.fill_(7))
    monkeypatch.setattr(fa, "_q8_pair", lambda *a, **k: pytest.fail("the paired kernel needs whole rows on one device"))
    monkeypatch.setattr(fa, "sdpa_fa_prefill", lambda q, k, v, scale, **kw: operand.update(k=k, v=v) or q)

    def require(*tensors):
        assert all(t.device.type == "cpu" for t in tensors)
        return torch.device("cpu")
    monkeypatch.setattr(fa, "require_cuda", require)
    chunk = torch.arange(2 * 3 * 256).reshape(1, 2, 3, 256).remainder(9).to(BF)
    past = _past(2, P, 64, 4)
    out = fa.sdpa_fa_prefill_q8(torch.zeros(1, 4, 3, 256, dtype=BF), past[0], *(t if P else t.to("meta") for t in past[1:]),
                                chunk, chunk[:, :1] if P else chunk, 1 / 16)
    assert tuple(out.shape) == (1, 4, 3, 256) and tuple(operand["k"].shape) == (P + 3, 2, 256)
    assert torch.equal(operand["k"][P:], chunk[0].transpose(0, 1)) and bool((operand["k"][:P] == 7).all())
    assert torch.equal(operand["v"][P:, 1], chunk[0, 0 if P else 1])


def test_expansion_refuses_output_rows_that_overlap():
    from moespresso_b200 import _abi
    lib = _abi.load()
    a = _abi.AffineQ8PairArgs()
    for i in range(2):
        for field in (a.x, a.packed, a.scales, a.biases):
            field[i] = 4096
    a.x_dtype = a.sb_dtype = _abi.BF16
    a.head_rows, a.n_rows, a.heads, a.width = 5, 5, 2, 512
    a.x_head_stride, a.x_row_stride = 5 * 256, 256
    assert lib.mxb_affine_q8_expand(C.byref(a), None) == -1
    assert b"must not overlap" in lib.mxb_last_error()


def _wide(stores):       # views of the first rows of longer buffers
    out = []
    for t in stores:
        big = torch.zeros(1, t.shape[1], 50, t.shape[3], dtype=t.dtype)
        out.append(big[:, :, :t.shape[2]])
    return out


@pytest.mark.parametrize("layout,head_rows", [
    (lambda six: six, 20),                                                           # as allocated
    (lambda six: _wide(six), 50),
    (lambda six: [t[:, :, :9].clone() for t in six], 9),                              # compact copies of fewer rows
    (lambda six: [t.transpose(1, 2).contiguous().transpose(1, 2) for t in six], 0),   # rows outside heads
    (lambda six: [*six[:3], *_wide(six[3:])], 0),                                    # values laid out unlike the keys
    (lambda six: [*six[:4], *(t.float() for t in six[4:])], 0),                      # scales of two types
    (lambda six: [torch.cat([t, t]) for t in six], 0),                               # two batch entries: rows broadcast
])
def test_append_follows_the_stores(monkeypatch, layout, head_rows):
    """``keys`` and ``values`` are public: the paired append must go by what they are, and leave to the copies what it
    cannot address."""
    def quantize(x):      # any three values of the right shapes and types
        return x[..., ::4].to(torch.int32), x[..., ::64], -x[..., ::64]
    launches = []
    monkeypatch.setattr(fa, "quantize_affine_q8", quantize)
    monkeypatch.setattr(fa, "require_cuda", lambda *tensors: torch.device("cpu"))
    monkeypatch.setattr(fa, "_q8_pair", lambda *a: launches.append(a[6:9]))
    cache = fa.QuantizedKVCache(2, 256, 20, device="cpu")
    six = layout([*cache.keys, *cache.values])
    cache.keys, cache.values, cache.offset = tuple(six[:3]), tuple(six[3:]), 4
    rows = [torch.randint(1, 100, (1, 2, 5, 256)).float() for _ in range(2)]
    cache.update_and_fetch(*rows)
    assert cache.offset == 9 and launches == ([(head_rows, 4, 5)] if head_rows else [])
    if not head_rows:
        for store, x in zip((cache.keys, cache.values), rows):
            for got, want in zip(store, quantize(x.to(store[1].dtype))):
                assert torch.equal(got[:, :, 4:9], want.expand(got.shape[0], -1, -1, -1))
                assert not got[:, :, :4].any() and not got[:, :, 9:].any()


def test_state_of_an_offset_past_the_stores_clips():
    """A program that trims the stores and keeps counting gets the rows there are, as from any slice."""
    cache = fa.QuantizedKVCache(2, 256, 20, device="cpu")
    cache.keys, cache.values = (tuple(t[:, :, :9] for t in six) for six in (cache.keys, cache.values))
    cache.offset = 12
    assert all(t.shape[2] == 9 for six in cache.state for t in six)


def test_native_calls_leave_cpu_tensors_to_python():
    """Without a device the native calls take nothing: the Python operators raise their own error."""
    import torch
    from moespresso_b200 import _torchabi
    x = torch.zeros(1, 2, 1, 256)
    assert _torchabi.native("q8_decode", x, x, x, x, x, x, x, 0.1, 4) is None
    assert _torchabi.native("decode_step") is None


def _narrow(i, n):       # tensor i of the six with rows of n values
    return lambda six: [t[..., :n].contiguous() if j == i else t for j, t in enumerate(six)]


@pytest.mark.parametrize("cache", [
    lambda six: _past(2, 5, 32, 2), lambda six: _past(2, 5, 128, 8), lambda six: _past(2, 5, 64, 2), lambda six: _past(2, 5, 16, 1),
    _narrow(0, 32), _narrow(3, 16), _narrow(1, 2), _narrow(2, 1), _narrow(5, 3),
    lambda six: [*six[:3], *(t[:, :, :4] for t in six[3:])],                         # fewer values than keys
    lambda six: [*six[:3], *(t[:, :1] for t in six[3:])],                            # values of fewer heads
    lambda six: [*six[:4], six[4].float(), six[5]],                                  # scales of two types
    lambda six: [six[0].to(torch.int16), *six[1:]],
    lambda six: [torch.zeros(1, 2, 5 * 64 + 32, dtype=torch.int32).as_strided((1, 2, 5, 64), (0, 5 * 64 + 32, 64, 1)), *six[1:]],
    lambda six: [t[:0] for t in six],
])
def test_decode_refuses_rows_that_the_kernel_would_misread(monkeypatch, cache):
    """The decode kernel is told head_dim 256, the rows of a head and one type of scales, and reads by them."""
    monkeypatch.setattr(fa, "require_cuda", lambda *tensors: torch.device("cpu"))
    monkeypatch.setattr(fa._t, "launch", lambda *a: pytest.fail("a kernel would have been launched"))
    with pytest.raises(ValueError):
        fa.sdpa_decode_q8(torch.zeros(1, 4, 1, 256, dtype=BF), *cache(_past(2, 5, 64, 4)), 1 / 16)


@pytest.mark.parametrize("layout,head_rows", [
    (lambda six: six, 5), (_wide, 50),
    (lambda six: [*(t[:, :, :3] for t in six[:3]), *six[3:]], 5),                    # values of keys to come
    (lambda six: [torch.cat([t, t]) for t in six], 5),                               # the first entry of a batch
])
def test_decode_takes_the_caches_that_it_can_address(monkeypatch, layout, head_rows):
    seen = []
    monkeypatch.setattr(fa, "require_cuda", lambda *tensors: torch.device("cpu"))
    monkeypatch.setattr(fa._t, "launch", lambda name, fn, a: seen.append(a) or 0)
    monkeypatch.setattr("moespresso_b200.deepseek_v4.indexed_attention_kernel.require_cuda", lambda *t: torch.device("cpu"))
    six = layout(_past(2, 5, 64, 4))
    fa.sdpa_decode_q8(torch.zeros(1, 4, 1, 256, dtype=BF), *six, 1 / 16)
    assert (seen[0].P, seen[0].head_stride_rows) == (six[0].shape[2], head_rows)
