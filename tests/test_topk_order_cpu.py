"""The score order of a selection with the launch replaced: the ids that a caller's buffer and the result hold."""
import torch

from moespresso_b200.deepseek_v4 import attention as att


def test_score_order_reaches_the_callers_buffer(monkeypatch):
    scores = torch.tensor([[1.0, 5.0, float("-inf"), 3.0], [float("-inf"), 2.0, 2.0, 7.0]])
    out = torch.zeros(2, 3, dtype=torch.int32)

    def launch(name, fn, args):
        assert args.out_ids == out.data_ptr()
        out.copy_(torch.tensor([[0, 1, 3], [1, 2, 3]]))
        return 0
    monkeypatch.setattr(att, "require_cuda", lambda *tensors: torch.device("cpu"))
    monkeypatch.setattr(att._t, "launch", launch)
    got = att.topk_select(scores, 3, order="score", out=out)
    assert got.tolist() == out.tolist() == [[1, 3, 0], [3, 1, 2]]
    assert got.data_ptr() == out.data_ptr()
