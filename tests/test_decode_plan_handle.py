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
    monkeypatch.setattr(D._lib, "status", lambda name, *args: out.append((name, args[0].value)))
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
