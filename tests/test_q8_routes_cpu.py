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
