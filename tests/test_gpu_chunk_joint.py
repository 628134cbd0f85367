"""Chunk products of two or three matrices in one launch (ill_mv_3n of more than sixteen tokens) have the bits of one launch each; what one
launch does not take is done one by one."""
import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D

pytestmark = pytest.mark.gpu


def _p(t):
    return 0 if t is None else t.data_ptr()


@pytest.mark.parametrize("fmts,rows,cols,n,off,one", [
    ((B.Q8_0, B.Q8_0, B.Q8_0), (896, 128, 128), 896, 777, 0, True),     # rows of 16-byte boundaries two by two
    ((B.Q8_0, B.Q8_0, B.Q8_0), (1, 257, 130), 128, 17, 2, True),        # a matrix of one row; blocks at another alignment
    ((B.Q8_0, B.Q8_0), (300, 127), 512, 65, 6, True),
    ((B.Q8_0, B.Q8_0), (5000, 5000), 128, 2048, 0, True),               # several rounds, tiles of 128 tokens
    ((B.Q4_K, B.Q6_K), (130, 77), 512, 33, 0, True),
    ((B.Q4_K, B.Q4_K, B.Q6_K), (16, 256, 1), 256, 17, 2, True),
    ((B.Q6_K, B.Q6_K), (1024, 1024), 768, 65, 2, True),
    ((B.Q6_K, B.Q4_K), (1024, 1040), 512, 1024, 0, True),               # tiles of 64 tokens, two CTAs an SM
    ((B.Q4_K, B.Q6_K), (1024, 1024), 256, 500, 0, True),                # four CTAs an SM
    ((B.Q4_K, B.Q6_K), (1024, 1024), 256, 2048, 0, False),              # more CTAs than run side by side
    ((B.Q2_K, B.Q2_K), (64, 64), 256, 20, 0, False),
])
def test_matrices_of_a_chunk_in_one_launch(cuda_lib, fmts, rows, cols, n, off, one):
    g = torch.Generator(device="cuda").manual_seed(n + cols)
    kind = D.matrix_act_kind(D.CMat("", fmts[0], 1, cols, None))
    act = D.quant_q8(torch.randn(n * cols, device="cuda", generator=g), D.make_qact(n * cols, kind))
    mats = []
    for i, (f, r) in enumerate(zip(fmts, rows)):
        w = B.synth_matrix_torch(f, r, cols, seed=i + r)
        buf = torch.zeros(w.numel() + 16, dtype=torch.uint8, device="cuda")
        buf[off:off + w.numel()] = w
        mats.append((buf, torch.randn(r, device="cuda", generator=g) if i != 1 else None))
    third = len(fmts) == 3
    got = [torch.full((n * r + 8,), 7.0, device="cuda") for r in rows]

    def three(values, none=0):
        return values if third else [*values, none]
    rc = _lib.status("ill_mv_3n", *three(list(fmts)), *three([_p(b) + off for b, _ in mats]), *three(list(rows)), cols, _p(act.xq), _p(act.xs),
                     0 if kind == "q8" else _p(act.xsum), *three([_p(y) for y in got]), *three([_p(b) for _, b in mats]), n, _lib.stream())
    assert rc == (0 if one else 3)
    if one:
        for (buf, bias), f, r, y in zip(mats, fmts, rows, got):
            want = torch.empty(n * r, device="cuda")
            _lib.call("ill_mv", f, _p(buf) + off, r, cols, _p(act.xq), _p(act.xs), 0 if kind == "q8" else _p(act.xsum), _p(want), _p(bias), 0, n, _lib.stream())
            assert torch.equal(y[:n * r], want) and (y[n * r:] == 7.0).all()
    assert D.device_status() == 0


@pytest.mark.parametrize("fmts,rows,cols,n", [((B.Q8_0,) * 3, (896, 128, 128), 896, 100), ((B.Q4_K, B.Q4_K, B.Q6_K), (2048, 256, 256), 512, 64),
                                              ((B.Q4_K, B.Q4_K, B.Q6_K), (256, 256, 256), 512, 20), ((B.Q2_K,) * 3, (64, 64, 64), 256, 40)])
def test_qkv_of_a_chunk(cuda_lib, fmts, rows, cols, n):
    """Q, K and V of a chunk: Q by the tcgen05 kernel of the K formats where it is large, the others in one launch."""
    g = torch.Generator(device="cuda").manual_seed(n)
    ws = [D.upload_gmat(B.synth_matrix_torch(f, r, cols, seed=r + i), f, r, cols) for i, (f, r) in enumerate(zip(fmts, rows))]
    act = D.quant_q8(torch.randn(n * cols, device="cuda", generator=g), D.make_qact(n * cols, D.matrix_act_kind(ws[0])))
    bias = torch.randn(rows[1], device="cuda", generator=g)
    got, want = ([torch.zeros(n * r, device="cuda") for r in rows] for _ in range(2))
    D.qkv_mul(*ws, act, *got, bk=bias, n=n)
    for w, y, b in zip(ws, want, (None, bias, None)):
        D.cmat_mul(w, act, y, n, bias=b)
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and D.device_status() == 0
