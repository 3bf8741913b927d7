"""A plan times its candidates on a stream of its own: the operands' stream is
waited for first, except while that stream is capturing."""
import types

import pytest
import torch

from finchgb import _lib as L
from finchgb import device as dev
from finchgb.plan import Plan


@pytest.mark.parametrize("capturing", [False, True])
def test_operands_are_ready_before_the_plan_is_tuned(monkeypatch, capturing):
    order = []
    stream = types.SimpleNamespace(synchronize=lambda: order.append("wait"))
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: stream)
    monkeypatch.setattr(dev, "context", lambda: None)
    monkeypatch.setattr(L, "call", lambda name, *a: order.append(name))
    A = types.SimpleNamespace(desc=L.FgbSparse)
    Plan(L.FgbPlanDesc(), A, (), 1)
    assert order == (["fgb_plan_create"] if capturing else ["wait", "fgb_plan_create"])
