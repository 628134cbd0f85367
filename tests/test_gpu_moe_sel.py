"""The one-token expert products by the router's choice (ill_moe_glu_sel, ill_moe_mv_sel): the bits of the same products given a table
of the chosen experts' addresses; numbers from the end; a number out of range stays inside the pool and raises the status word."""
import dataclasses

import numpy as np
import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D
from illatio_b200 import cuda_ds4f as M

from gpu_util import dev_act

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def layer(cuda_lib):
    d, ff, ne = 512, 256, 5
    pool = M.make_expert_pool(B.synth_matrix(B.IQ2_XXS, ne * ff, d, seed=1), B.synth_matrix(B.IQ2_XXS, ne * ff, d, seed=2),
                              B.synth_matrix(B.Q2_K, ne * d, ff, seed=3), d, ff, ne)
    return pool, dev_act(B.IQ2_XXS, np.random.default_rng(0).standard_normal(d).astype(np.float32))


def _run(pool, act, sel, table):
    k = sel.numel()
    w = torch.linspace(0.5, 1.5, k, device="cuda")
    mid, down = torch.zeros(k * pool.ff, device="cuda"), torch.zeros(k * pool.d, device="cuda")
    head = (_lib.stream(),)
    if table is None:
        ptrs = (pool.ptrs_all.data_ptr(), pool.n_expert, sel.data_ptr(), k)
        glu, mv = "ill_moe_glu_sel", "ill_moe_mv_sel"
    else:
        ptrs = (table.data_ptr(), k)
        glu, mv = "ill_moe_glu", "ill_moe_mv"
    _lib.call(glu, pool.gate_fmt, pool.d, pool.ff, 0, pool.gate_bytes, *ptrs, act.xq.data_ptr(), act.xs.data_ptr(), act.xsum.data_ptr(), 0, 10.0,
              w.data_ptr(), mid.data_ptr(), pool.ff, *head)
    midq = D.quant_q8(mid, D.make_qact(mid.numel(), "q8k"))
    _lib.call(mv, pool.down_fmt, pool.ff, pool.d, 2 * pool.gate_bytes, *ptrs, midq.xq.data_ptr(), midq.xs.data_ptr(), midq.xsum.data_ptr(), 1,
              down.data_ptr(), pool.d, *head)
    return mid, down


@pytest.mark.parametrize("sel", [[0], [4, 4, 0], [-1, 2, -5], [3, 1, 0, 2, 4, 1]])
def test_chosen_experts_are_those_of_the_table(layer, sel):
    pool, act = layer
    s = torch.tensor(sel, dtype=torch.int32, device="cuda")
    got, want = _run(pool, act, s, None), _run(pool, act, s, pool.slot_ptrs(s))
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert D.device_status() == 0


@pytest.mark.parametrize("bad", [5, -6, 2 ** 31 - 1])
def test_an_expert_out_of_range_raises_the_status_word(layer, bad):
    pool, act = layer
    got = _run(pool, act, torch.tensor([bad, 2], dtype=torch.int32, device="cuda"), None)
    zero = torch.tensor([0, 2], dtype=torch.int32, device="cuda")
    want = _run(pool, act, zero, pool.slot_ptrs(zero))
    assert all(torch.equal(a, b) for a, b in zip(got, want))  # expert 0 was read
    assert D.device_status() == 0x600
    assert D.device_status() == 0


def test_native_operators_leave_other_forms_to_python(layer):
    pool, _ = layer
    x = torch.randn(pool.d, device="cuda")
    w = torch.tensor([0.25, 0.75], device="cuda")
    sel = torch.tensor([1, 3], dtype=torch.int32, device="cuda")
    moe, mid = M.dk_ffn_tail(pool, x, sel, w, 10.0)
    for other in (sel.long(), torch.stack([sel, sel], dim=1)[:, 0]):  # 64-bit numbers, numbers apart
        m2, mid2 = M.dk_ffn_tail(pool, x, other, w, 10.0)
        assert torch.equal(moe, m2) and torch.equal(mid, mid2)


class Reversed(M.ExpertPool):
    def slot_ptrs(self, experts):
        return self.ptrs_all.flip(0)[experts.long()]


class Slots:
    """A caller's own pool: the experts' addresses by slot_ptrs() alone."""

    def __init__(self, pool):
        self.d, self.ff, self.gate_fmt, self.down_fmt, self.gate_bytes = pool.d, pool.ff, pool.gate_fmt, pool.down_fmt, pool.gate_bytes
        self.slot_ptrs = lambda experts: pool.slot_ptrs(experts)


@pytest.mark.parametrize("kind", ["subclass", "object", "instance", "longer table", "table apart"])
def test_a_pool_of_the_callers_own(layer, kind):
    """The experts' addresses are those that the pool's slot_ptrs() gives."""
    pool, _ = layer
    x = torch.randn(pool.d, device="cuda")
    w = torch.tensor([0.25, 0.75], device="cuda")
    sel = torch.tensor([1, 3], dtype=torch.int32, device="cuda")
    own, as_pool = dataclasses.replace(pool), sel
    if kind == "subclass":
        own, as_pool = Reversed(**vars(pool)), 4 - sel
    elif kind == "object":
        own = Slots(pool)
    elif kind == "instance":
        own.slot_ptrs, as_pool = (lambda experts: pool.slot_ptrs(4 - experts)), 4 - sel
    elif kind == "longer table":
        own.n_expert = 2
    else:
        own.ptrs_all = torch.stack([pool.ptrs_all, pool.ptrs_all + 1], dim=1)[:, 0]
    want, got = M.dk_ffn_tail(pool, x, as_pool, w, 10.0), M.dk_ffn_tail(own, x, sel, w, 10.0)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert D.device_status() == 0
