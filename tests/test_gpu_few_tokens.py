"""Products of two to sixteen tokens: two or three matrices in one launch (ill_mv_3n) give each matrix's own bits, whatever groups and
sums the launch deals out; ragged rows, rows at every alignment, Q4_K beside Q6_K; and the product itself against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D

from gpu_util import act_to_host, dev_act, rel_errors

pytestmark = pytest.mark.gpu


def _mat(fmt, rows, cols, seed, off):
    w = B.synth_matrix(fmt, rows, cols, seed=seed)
    buf = torch.zeros(w.size + 16, dtype=torch.uint8, device="cuda")
    buf[off:off + w.size] = torch.as_tensor(np.ascontiguousarray(w)).cuda().reshape(-1)
    return w, buf, buf.data_ptr() + off


@pytest.mark.parametrize("fmts,rows,cols,n,off", [
    ((B.Q8_0, B.Q8_0, B.Q8_0), (896, 128, 130), 896, 2, 2),
    ((B.Q8_0, B.Q8_0), (17, 1), 32, 16, 0),            # one block a row: one partial sum
    ((B.Q8_0, B.Q8_0), (128, 128), 128, 2, 0),
    ((B.Q8_0, B.Q8_0), (300, 300), 4864, 9, 0),
    ((B.Q4_K, B.Q4_K, B.Q4_K), (257, 16, 15), 256, 3, 0),
    ((B.Q4_K, B.Q4_K), (2000, 2000), 2560, 16, 0),     # five partial sums
    ((B.Q4_K, B.Q4_K), (40, 33), 1792, 7, 2),          # blocks that start in the middle of a word
    ((B.Q6_K, B.Q6_K, B.Q6_K), (513, 100, 64), 5120, 4, 0),
    ((B.Q6_K, B.Q6_K), (65, 65), 768, 16, 2),          # rows that start on words and between them in turn
    ((B.Q4_K, B.Q4_K, B.Q6_K), (4096, 1024, 1024), 2560, 16, 0),
    ((B.Q4_K, B.Q4_K, B.Q6_K), (33, 47, 5), 2048, 8, 2),
    ((B.Q6_K, B.Q4_K), (31, 100), 512, 5, 0),
    ((B.Q4_K, B.Q6_K, B.Q4_K), (3000, 2500, 20), 3072, 12, 0),
])
def test_matrices_in_one_launch_give_each_ones_bits(cuda_lib, fmts, rows, cols, n, off):
    x = np.random.default_rng(rows[0] + cols).standard_normal(n * cols).astype(np.float32)
    act = dev_act(fmts[0], x)
    mats = [_mat(f, r, cols, 11 + i, off) for i, (f, r) in enumerate(zip(fmts, rows))]
    bias = [torch.randn(r, device="cuda") if i != 1 else None for i, r in enumerate(rows)]
    xsum = 0 if act.kind == "q8" else act.xsum.data_ptr()
    want, got = [], []
    for (w, keep, ptr), f, r, b in zip(mats, fmts, rows, bias):
        y = torch.zeros(n * r, device="cuda")
        _lib.call("ill_mv", f, ptr, r, cols, act.xq.data_ptr(), act.xs.data_ptr(), xsum, y.data_ptr(), b.data_ptr() if b is not None else 0, 0, n,
                  _lib.stream())
        want.append(y)
        got.append(torch.full((n * r + 8,), 7.0, device="cuda"))
    third = len(fmts) == 3
    _lib.call("ill_mv_3n", fmts[0], fmts[1], fmts[2] if third else 0, mats[0][2], mats[1][2], mats[2][2] if third else 0, rows[0], rows[1],
              rows[2] if third else 0, cols, act.xq.data_ptr(), act.xs.data_ptr(), xsum, got[0].data_ptr(), got[1].data_ptr(),
              got[2].data_ptr() if third else 0, bias[0].data_ptr(), 0, bias[2].data_ptr() if third else 0, n, _lib.stream())
    for g, w, r in zip(got, want, rows):
        assert torch.equal(g[:n * r], w)
        assert (g[n * r:] == 7.0).all()
    assert D.device_status() == 0


@pytest.mark.parametrize("fmt,rows,cols,n,groups", [(B.Q4_K, 36000, 768, 4, 4), (B.Q4_K, 35520, 256, 16, 15), (B.Q6_K, 35520, 256, 3, 15),
                                                    (B.Q6_K, 36000, 768, 3, 4), (B.Q8_0, 36001, 576, 8, 8)])
def test_short_rows_of_many(cuda_lib, fmt, rows, cols, n, groups):
    """Short rows whose tiles nearly fill the rounds: many groups a CTA, up to fifteen of one warp, one for each barrier; the bits of
    launches of some of the rows, which have other groups."""
    out = (ctypes.c_int * 8)()
    assert _lib.status("ill_test_few_tokens_plan", 1, fmt, 0, 0, rows, 0, 0, cols, n, 148, out) == 0 and out[1] == out[2] == groups
    act = dev_act(fmt, np.random.default_rng(rows).standard_normal(n * cols).astype(np.float32))
    w, keep, ptr = _mat(fmt, rows, cols, 5, 0)
    xsum = 0 if act.kind == "q8" else act.xsum.data_ptr()

    def mul(row0, count):
        y = torch.full((n * count + 8,), 7.0, device="cuda")
        _lib.call("ill_mv", fmt, ptr + row0 * B.row_bytes(fmt, cols), count, cols, act.xq.data_ptr(), act.xs.data_ptr(), xsum, y.data_ptr(), 0, 0, n,
                  _lib.stream())
        assert (y[n * count:] == 7.0).all()
        return y[:n * count].view(n, count)

    got = mul(0, rows)
    for row0, count in ((0, 1600), (17760, 333), (rows - 1000, 1000)):
        _lib.call("ill_test_few_tokens_plan", 1, fmt, 0, 0, count, 0, 0, cols, n, 148, out)
        assert out[1] != groups
        assert torch.equal(got[:, row0:row0 + count], mul(row0, count))
    assert D.device_status() == 0


@pytest.mark.parametrize("fmt,cols,n", [(B.Q4_K, 256, 2), (B.Q4_K, 2560, 16), (B.Q6_K, 768, 9), (B.Q4_K, 17408, 5), (B.Q6_K, 17408, 16)])
def test_sums_of_16_that_lie_on_eight_bytes(cuda_lib, fmt, cols, n):
    """The sums of 16 need lie on eight bytes only: the bits of sums on sixteen, of one matrix and of two in a launch, and through the
    operators given an activation of the caller's own."""
    rows = 33
    act = dev_act(fmt, np.random.default_rng(cols + n).standard_normal(n * cols).astype(np.float32))
    buf = torch.empty(act.xsum.numel() + 4, dtype=torch.int16, device="cuda")
    off = buf[4:]
    off.copy_(act.xsum)
    assert act.xsum.data_ptr() % 16 == 0 and off.data_ptr() % 16 == 8
    mats = [D.upload_gmat(B.synth_matrix(fmt, rows, cols, seed=s), fmt, rows, cols) for s in (1, 2, 3)]
    other = D.QAct(act.kind, act.xq, act.xs, off)
    got, want = ([torch.zeros(n * rows, device="cuda") for _ in mats] for _ in range(2))
    for m, y in zip(mats, want):
        D.cmat_mul(m, act, y, n)
    D.cmat_mul(mats[0], other, got[0], n)
    assert torch.allclose(got[0], want[0], rtol=0, atol=1e-5 * want[0].abs().max().item())
    if cols < 17408:  # (longer rows' kernel wants Q4_K's sums on sixteen bytes: the product is another's, in another order)
        assert torch.equal(got[0], want[0])
        D.qkv_mul(*mats, other, *got, n=n)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        fa = D.glu_mul(mats[0], mats[1], act, torch.empty_like(want[0]), n, fb=torch.empty_like(want[0]))
        fo = D.glu_mul(mats[0], mats[1], other, torch.empty_like(want[0]), n, fb=torch.empty_like(want[0]))
        assert torch.equal(fa, fo)
    assert D.device_status() == 0


@pytest.mark.parametrize("fmt,rows,cols,n", [(B.Q8_0, 50, 1152, 16), (B.Q4_K, 40, 2560, 16), (B.Q4_K, 19, 1280, 3), (B.Q6_K, 40, 5120, 16),
                                             (B.Q6_K, 23, 2304, 2), (B.Q8_0, 4864, 896, 16), (B.Q4_K, 2560, 4096, 4),
                                             (B.Q6_K, 1024, 2560, 9), (B.Q4_K, 2400, 17408, 3), (B.Q6_K, 176, 17408, 16)])
def test_few_tokens_against_the_oracle(oracle, cuda_lib, fmt, rows, cols, n):
    x = np.random.default_rng(cols).standard_normal(n * cols).astype(np.float32)
    act = dev_act(fmt, x)
    w, keep, ptr = _mat(fmt, rows, cols, 3, 0)
    y = torch.zeros(n * rows, device="cuda")
    _lib.call("ill_mv", fmt, ptr, rows, cols, act.xq.data_ptr(), act.xs.data_ptr(), 0 if act.kind == "q8" else act.xsum.data_ptr(),
              y.data_ptr(), 0, 0, n, _lib.stream())
    xq, xs, bs = act_to_host(act)
    want = []
    for t in range(n):
        per = 32 if fmt == B.Q8_0 else 256
        h = (xq[t * cols:(t + 1) * cols], xs[t * (cols // per):(t + 1) * (cols // per)])
        h = h + ((bs[t * (cols // 16):(t + 1) * (cols // 16)],) if bs is not None else (None,))
        want.append(oracle.matvec(fmt, w, rows, cols, h)[0])
    # whole-number block sums: what differs is the order of at most 152 32-bit additions
    err, _ = rel_errors(y.cpu().numpy().reshape(n, rows), np.stack(want))
    assert err <= 1e-5


@pytest.mark.parametrize("fmt", [B.Q8_0, B.Q4_K])
def test_a_third_matrix_of_no_rows_is_refused(cuda_lib, fmt):
    """The entry point takes two matrices when the third has neither rows nor an address; the operator's three are three."""
    cols, n = 256, 4
    act = dev_act(fmt, np.ones(n * cols, np.float32))
    m = D.upload_gmat(B.synth_matrix(fmt, 16, cols, seed=1), fmt, 16, cols)
    none = D.CMat("", fmt, 0, cols, torch.empty(0, dtype=torch.uint8, device="cuda"))
    y = [torch.zeros(n * 16, device="cuda") for _ in range(3)]
    with pytest.raises(_lib.IllatioError) as e:
        D.qkv_mul(m, m, none, act, *y, n=n)
    assert e.value.code == 1


@pytest.mark.parametrize("fmts", [(B.Q8_0,), (B.Q4_K,), (B.Q6_K,), (B.Q4_K, B.Q6_K)])
@pytest.mark.parametrize("n", [8, 16])
def test_registers_are_what_the_choice_of_ctas_takes_them_for(cuda_lib, fmts, n):
    out = (ctypes.c_int * 8)()
    assert _lib.status("ill_test_few_tokens_plan", len(fmts), fmts[0], fmts[-1], 0, 64, 64 if len(fmts) > 1 else 0, 0, 1024, n, 0, out) == 0
    assert 0 < out[7] <= out[6]  # (registers are given out eight a thread at a time)


@pytest.mark.parametrize("fmt", [B.Q8_0, B.Q4_K, B.Q6_K])
@pytest.mark.parametrize("n", [4, 16])
def test_long_rows_in_one_cta_and_in_a_cluster(cuda_lib, fmt, n):
    """Rows too long for their activations to stay in shared memory: a tile of sixteen rows in one CTA (100 tiles: a round of the SMs more
    than half full; 250) or in a cluster of four (10 tiles; 160), the same bits."""
    cols, rows = (17408 if n == 4 else 11008), 4000
    out = (ctypes.c_int * 8)()
    assert _lib.status("ill_test_few_tokens_plan", 1, fmt, 0, 0, rows, 0, 0, cols, n, 148, out) == 3
    act = dev_act(fmt, np.random.default_rng(n).standard_normal(n * cols).astype(np.float32))
    w, keep, ptr = _mat(fmt, rows, cols, 5, 0)

    def mul(row0, count):
        y = torch.full((n * count + 8,), 7.0, device="cuda")
        _lib.call("ill_mv", fmt, ptr + row0 * B.row_bytes(fmt, cols), count, cols, act.xq.data_ptr(), act.xs.data_ptr(),
                  0 if act.kind == "q8" else act.xsum.data_ptr(), y.data_ptr(), 0, 0, n, _lib.stream())
        assert (y[n * count:] == 7.0).all()
        return y[:n * count].view(n, count)

    got = mul(0, rows)
    for row0, count in ((0, 160), (160, 1600), (1440, 2560), (3999, 1)):
        assert torch.equal(got[:, row0:row0 + count], mul(row0, count))
    assert D.device_status() == 0
