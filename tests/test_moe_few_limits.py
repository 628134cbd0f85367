"""The launches of a chunk whose experts of a few rows are taken apart, without a device: every expert's rows by one of the two products."""
from types import SimpleNamespace as NS

import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_ds4f_prefill as P


@pytest.mark.parametrize("gate,d,ff,limits", [(B.IQ2_XXS, 7168, 2048, (8, 16)), (B.Q2_K, 4096, 9216, (16, 8)), (B.Q2_K, 5120, 1536, (16, 16))])
@pytest.mark.parametrize("n", [17, 64])
def test_each_product_leaves_the_other_what_it_does_not_take(monkeypatch, gate, d, ff, limits, n):
    most = _lib.lib().ill_moe_few_most
    assert (most(gate, d), most(B.Q2_K, ff)) == limits
    nu, ne, seen = 4, 64, []
    pool = NS(d=d, ff=ff, n_expert=ne, gate_fmt=gate, down_fmt=B.Q2_K, gate_bytes=4096, ptrs_all=torch.zeros(ne, dtype=torch.int64))
    t = torch.zeros(16)
    act = NS(xq=t, xs=t, xsum=t)
    sc = NS(rows=n * nu, xq=act, midq=act, **{k: t for k in "counts bases rmap smap wrow g u mid xh xe mh me down moe".split()})
    monkeypatch.setattr(P._lib, "call", lambda name, *a: seen.append((name, a)))
    P._few_rows_chunk(pool, n, nu, 10.0, sc, None, P.few_rows(pool, n, nu), 0)
    few = [(a[0], a[1], most(a[0], a[1])) for name, a in seen if name.startswith("ill_moe_few")]
    over = [(a[0], a[1], a[-2]) for name, a in seen if name == "ill_moe_mm_id_over"]
    assert few == over == [(gate, d, limits[0]), (B.Q2_K, ff, limits[1])]
    assert [a[-2] for name, a in seen if name == "ill_act_f16_over"] == [limits[0]]


@pytest.mark.parametrize("fmt,step", [(B.Q2_K, 4), (B.IQ2_XXS, 2)])
def test_a_matrix_off_its_boundary_is_refused(fmt, step):
    """(A matrix on its boundary gets past the checks: no rows, no launch.)"""
    P_ = 0x10000
    who, x = (P_, P_, P_, 4, 0), (P_, P_, P_, P_)
    for add, rc in ((0, 0), (step, 0), (step // 2, 2), (1, 2), (step + 1, 2)):
        for form in ("ill_moe_few", "ill_moe_few_all"):
            assert _lib.status(form, fmt, 512, 16, add, *who, *x, P_, 16, 0) == rc, (form, add)
        for a, b in ((add, 0), (0, add)):
            assert _lib.status("ill_moe_few2", fmt, 512, 16, a, b, *who, *x, P_, P_, 16, 0) == rc
            for form in ("ill_moe_few_glu", "ill_moe_few_glu_all"):
                assert _lib.status(form, fmt, 512, 16, a, b, *who, *x, 1.0, P_, P_, 16, 0) == rc
