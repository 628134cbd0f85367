"""ill_mm_chunk_exact: two matrices of few rows against a chunk, bit for bit what ill_mv (int32 sums) gives, also where a block's sum
passes 2^24; and the chunks of Q, K and V that take it."""
import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D

pytestmark = pytest.mark.gpu

Q4, Q6 = B.Q4_K, B.Q6_K


def _matrix(fmt, rows, cols, kind, seed):
    w = B.synth_matrix_torch(fmt, rows, cols, seed=seed)
    if kind:   # every field at its largest (Q6_K: the scales 127, or -128), the block's scales as they are
        v = w.view(-1, B.matrix_bytes(fmt, 1, 256))
        if fmt == Q4:
            v[:, 4:] = 0xff
        else:
            v[:, :192], v[:, 192:208] = (0xff, 0x7f) if kind == 1 else (0, 0x80)
    return D.CMat("w", fmt, rows, cols, w)


def _chunk(n, cols, kind):
    g = torch.Generator(device="cuda").manual_seed(n + cols)
    x = torch.randn(n * cols, device="cuda", generator=g)
    if kind:
        x = 1.0 + 1e-4 * x
    return D.quant_q8(x, D.make_qact(n * cols, "q8k"))


def _mv(w, act, n):
    y = torch.empty(n * w.rows, device="cuda")
    _lib.call("ill_mv", w.type, w.qs.data_ptr(), w.rows, w.cols, act.xq.data_ptr(), act.xs.data_ptr(), act.xsum.data_ptr(), y.data_ptr(), 0, 0, n, _lib.stream())
    return y


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("fmts", [(Q4, Q4), (Q6, Q6), (Q4, Q6), (Q6, Q4)])
@pytest.mark.parametrize("rows,cols,n", [(4, 256, 17), (124, 512, 33), (132, 768, 17), (128, 256, 65), (1024, 2560, 512), (260, 1280, 129), (2044, 512, 1000), (1024, 256, 777)])
def test_bits_of_int32_sums(cuda_lib, fmts, rows, cols, n, kind):
    act = _chunk(n, cols, kind)
    ws = [_matrix(f, rows, cols, kind, seed=rows + i) for i, f in enumerate(fmts)]
    cf = D.ChunkF16(n, cols).fill(act)
    ys = [torch.full((n * rows + 8,), 7.0, device="cuda") for _ in ws]
    _lib.call("ill_mm_chunk_exact", ws[0].type, ws[0].qs.data_ptr(), ws[1].type, ws[1].qs.data_ptr(), rows, cols, cf.xh.data_ptr(),
              cf.xe.data_ptr(), cf.xd.data_ptr(), n, ys[0].data_ptr(), ys[1].data_ptr(), _lib.stream())
    for w, y in zip(ws, ys):
        assert torch.equal(y[:n * rows], _mv(w, act, n)) and (y[n * rows:] == 7.0).all()
    assert D.device_status() == 0


@pytest.mark.parametrize("fmts,krows,n,off,bias", [((Q4, Q4, Q6), 1024, 512, 0, False), ((Q4, Q6, Q6), 512, 512, 0, False),
                                                   ((Q4, Q6, Q4), 508, 520, 0, False), ((Q6, Q4, Q4), 252, 100, 0, False),
                                                   ((Q4, Q4, Q4), 254, 100, 0, False),    # rows that are not whole 16-byte pieces of Y
                                                   ((Q4, Q4, Q6), 256, 100, 1, False),    # Y off its 16-byte boundary
                                                   ((Q4, Q4, Q6), 256, 100, 0, True), ((Q4, Q6, Q6), 256, 63, 0, False)])
def test_qkv_chunks(cuda_lib, fmts, krows, n, off, bias):
    """K and V beside a Q of the tcgen05 kernel have the bits of a product by itself, whichever kernel takes them."""
    cols, rows = 512, (2048, krows, krows)
    act = _chunk(n, cols, 0)
    ws = [_matrix(f, r, cols, 0, seed=r + i) for i, (f, r) in enumerate(zip(fmts, rows))]
    b = torch.randn(krows, device="cuda") if bias else None
    got, want = ([torch.zeros(n * r + off, device="cuda")[off:] for r in rows] for _ in range(2))
    if off:
        got[0] = torch.zeros(n * rows[0], device="cuda")   # (Q itself needs the boundary)
        want[0] = torch.zeros(n * rows[0], device="cuda")
    D.qkv_mul(*ws, act, *got, bk=b, n=n)
    for w, y, bb in zip(ws, want, (None, b, None)):
        D.cmat_mul(w, act, y, n, bias=bb)
    assert all(torch.equal(a, c) for a, c in zip(got, want)) and D.device_status() == 0


@pytest.mark.parametrize("fmts", [(Q4, Q6), (Q6, Q6)])
def test_the_same_bits_every_time(cuda_lib, fmts):
    """Many tiles a CTA, so that raw blocks, slots and accumulators are reused all the time: sixty launches agree."""
    rows, cols, n = 1024, 8192, 2048
    act = _chunk(n, cols, 0)
    ws = [_matrix(f, rows, cols, 0, seed=i) for i, f in enumerate(fmts)]
    cf = D.ChunkF16(n, cols).fill(act)
    want = [_mv(w, act, n) for w in ws]
    bad = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(60):
        ys = [torch.full((n * rows,), 7.0, device="cuda") for _ in ws]
        _lib.call("ill_mm_chunk_exact", fmts[0], ws[0].qs.data_ptr(), fmts[1], ws[1].qs.data_ptr(), rows, cols, cf.xh.data_ptr(), cf.xe.data_ptr(),
                  cf.xd.data_ptr(), n, ys[0].data_ptr(), ys[1].data_ptr(), _lib.stream())
        for y, w in zip(ys, want):
            bad += (y != w).sum()
    assert bad.item() == 0 and D.device_status() == 0
