"""Who gives a DecodePlan's recorded launches back, without a device."""
import contextlib
import copy
import gc
import pickle

import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import cuda_dense as D


@pytest.fixture
def freed(monkeypatch):
    out = []

    def call(name, *args):
        if name == "ill_chain_new":
            args[-1]._obj.value = 5
    monkeypatch.setattr(D._lib, "call", call)

    def status(name, *args):
        if name == "ill_chain_free":
            out.append((name, args[0].value))
        return 0
    monkeypatch.setattr(D._lib, "status", status)
    monkeypatch.setattr(D, "_stream", lambda: 0)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    return out


def test_copies_of_a_plan_share_its_launches(freed):
    plan = D.DecodePlan([_lib.DecodeOp()], device="cpu")
    others = [copy.copy(plan), copy.deepcopy(plan)]
    del plan
    gc.collect()
    assert freed == []
    others.clear()
    gc.collect()
    assert freed == [("ill_chain_free", 5)]


def test_a_plan_does_not_outlive_its_process(freed):
    with pytest.raises(TypeError):
        pickle.dumps(D.DecodePlan([_lib.DecodeOp()], device="cpu"))


def test_scratch_is_held_for_a_stream_of_another_run(freed, monkeypatch):
    plan, held = D.DecodePlan([_lib.DecodeOp()], device="cpu"), []

    class Scratch(torch.Tensor):
        def record_stream(self, stream):
            held.append(stream)
    plan.chain.scratch = plan.chain.scratch.as_subclass(Scratch)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: "another")
    plan.run()
    assert held == []
    monkeypatch.setattr(D, "_stream", lambda: 7)
    plan.run()
    assert held == ["another"]
