"""Digit products without memory for their scratch: the plan's steps run on the FP64
kernels instead of failing, and the scratch makes room for everything else (host logic,
with an allocator that runs out)."""
import pytest
import torch

from pytreenet_gb300 import _lib
from pytreenet_gb300 import engine as E


class _Memory:
    """torch.empty with `left` entries to give."""

    def __init__(self, monkeypatch, left):
        self.left, real = left, torch.empty

        def empty(n, *a, **k):
            if n > self.left:
                raise torch.OutOfMemoryError("no memory")
            return real(n, *a, **k)
        monkeypatch.setattr(E.torch, "empty", empty)


def _plan(ws):
    cb = E.ChainBuilder(ws)
    x = E.Operand.contiguous(("in",), ["m", "k"], [4, 3])
    t = cb.contract(x, E.Operand.contiguous(("fixed", torch.zeros(3, 2, dtype=E.CDT)), ["k", "l"], [3, 2]), ["k"])
    cb.contract(t, E.Operand.contiguous(("fixed", torch.zeros(2, 5, dtype=E.CDT)), ["l", "n"], [2, 5]), ["l"],
                out=E.Operand.contiguous(("out",), ["m", "n"], [4, 5]))
    return cb.plan()


def _kinds(plan):
    ops = plan.native_ops()
    ops.bind(plan.ws)
    return [ops.ops[i].kind for i in range(ops.n)]


@pytest.fixture
def sizes(monkeypatch):
    want = iter([16 * 1000, 16 * 50])                   # bytes of the two steps of a plan
    monkeypatch.setattr(E, "contract_work_bytes", lambda desc, device: next(want))


def test_steps_without_scratch_run_on_the_fp64_kernels(monkeypatch, sizes):
    plan = _plan(E.Workspace(torch.device("cpu")))
    mem = _Memory(monkeypatch, 100)
    assert _kinds(plan) == [_lib.OP_ZCONTRACT, _lib.OP_ZCONTRACT_WS]
    mem.left = 10 ** 6                                  # what did not fit is not tried on every run
    plan.ws.get("other", 60)
    assert _kinds(plan) == [_lib.OP_ZCONTRACT, _lib.OP_ZCONTRACT_WS]


def test_scratch_makes_room_for_other_buffers(monkeypatch, sizes):
    ws = E.Workspace(torch.device("cpu"))
    plan = _plan(ws)
    assert _kinds(plan) == [_lib.OP_ZCONTRACT_WS, _lib.OP_ZCONTRACT_WS]
    real, failed = torch.empty, []

    def empty(n, *a, **k):
        if ws.SPARE in ws.bufs:
            failed.append(n)
            raise torch.OutOfMemoryError("no memory")
        return real(n, *a, **k)
    monkeypatch.setattr(E.torch, "empty", empty)
    assert ws.get("basis", 5000).numel() == 5000
    assert failed == [5000] and ws.SPARE not in ws.bufs
    assert _kinds(plan) == [_lib.OP_ZCONTRACT, _lib.OP_ZCONTRACT]
    with pytest.raises(torch.OutOfMemoryError):         # nothing left to give up
        monkeypatch.setattr(E.torch, "empty", lambda *a, **k: (_ for _ in ()).throw(torch.OutOfMemoryError("no")))
        ws.get("basis", 9000)
