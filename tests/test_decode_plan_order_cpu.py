"""Order of a decode plan's work on its two streams, with graphs, copies, events and streams replaced by a record of
what waits for what: q is written on the side stream, read (and by ``load_inputs`` written) on the main one."""
import pytest
import torch

from moespresso_b200 import _abi
from moespresso_b200.deepseek_v4 import decode_step
from moespresso_b200.deepseek_v4.decode_step import SparseDecodePlan


class _Stream:
    cuda_stream = 0

    def __init__(self):
        self.seen = set()                  # what has finished when the next thing on this stream starts

    def do(self, what):
        self.seen.add(what)

    def wait_event(self, event):
        self.seen |= event.seen


class _Event:
    seen = frozenset()

    def record(self, stream):
        self.seen = frozenset(stream.seen)


class _Graph:
    def __init__(self, stream, name):
        self.stream, self.name, self.n = stream, name, 0

    def replay(self):
        self.n += 1
        self.stream.do(f"{self.name} {self.n}")


def _plan(monkeypatch):
    main, side = _Stream(), _Stream()
    plan = SparseDecodePlan.__new__(SparseDecodePlan)
    plan._offs, plan._sizes, plan._shapes = (0, 256, 512), (256, 256, 256), ((1, 2, 32), (1, 2, 32), (1, 64))
    plan._dtypes = (torch.float32,) * 3
    plan.packed = torch.zeros(768, dtype=torch.uint8)
    plan.q, plan.idx_q, plan.idx_w = plan._views(plan.packed)
    plan.out = plan._out2 = None
    plan.graph, plan._graph_select, plan._graph_attend = (_Graph(main, n) for n in ("step", "select", "attend"))
    plan._copy_stream, plan._q_copied, plan._attend_done, plan._q_on_main = side, _Event(), _Event(), False
    copies = []

    class _Lib:
        @staticmethod
        def mxb_copy_h2d_async(*args):
            copies.append(set(side.seen))
            side.do(f"copy {len(copies)}")
            return 0
    monkeypatch.setattr(_abi, "load", lambda: _Lib)
    monkeypatch.setattr(decode_step.torch.cuda, "current_stream", lambda *a: main)
    monkeypatch.setattr(decode_step.torch.cuda, "current_device", lambda: -1)
    return plan, main, copies


@pytest.mark.parametrize("before", ["run", "launch", "load_inputs"])
def test_host_fed_step_waits_for_the_steps_before_it(monkeypatch, before):
    plan, main, copies = _plan(monkeypatch)
    host = torch.zeros(768, dtype=torch.uint8)
    plan.run_packed(host)
    if before == "launch":
        plan.launch()
    else:
        main.do("inputs")
        getattr(plan, before)(*plan._views(host))
    plan.run_packed(host)
    plan.run_packed(host)
    wanted = {"launch": {"step 1"}, "load_inputs": {"inputs"}, "run": {"inputs", "step 1"}}[before]
    assert wanted | {"attend 1"} <= copies[1] and "attend 2" in copies[2]
    assert not {"select 2", "attend 2"} & copies[1]      # and still travels while its own step's selection runs
    assert "copy 3" in main.seen                         # the attention waits for its q
