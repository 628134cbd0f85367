"""A dense Q4_K or Q6_K matrix (its blocks brought 128 rows at a time, Q6_K's where four rows are whole 16-byte pieces) has the bits of the
same matrix as an expert, whose blocks are brought piece by piece."""
import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("rows,cols,n,off", [(4, 256, 1, 0), (124, 512, 17, 16), (132, 768, 64, 0), (300, 1280, 65, 48), (640, 256, 128, 0),
                                             (1000, 512, 129, 16), (384, 2560, 256, 0), (2572, 1024, 700, 0), (17408, 512, 512, 0)])
@pytest.mark.parametrize("fmt", [B.Q4_K, B.Q6_K])
def test_dense_matrix_as_an_expert(cuda_lib, fmt, rows, cols, n, off, two):
    if fmt == B.Q6_K and rows == 124:
        off = 4   # (not a boundary a load can start from)
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    w = B.synth_matrix_torch(fmt, (2 if two else 1) * rows, cols, seed=rows)
    buf = torch.zeros(w.numel() + off, dtype=torch.uint8, device="cuda")
    buf[off:] = w
    base, gap = buf.data_ptr() + off, w.numel() // 2
    cf = D.ChunkF16(n, cols).fill(D.quant_q8(torch.randn(n * cols, device="cuda", generator=g), D.make_qact(n * cols, "q8k")))
    x = (cf.xh.data_ptr(), cf.xe.data_ptr(), cf.xd.data_ptr())
    got, want = ([torch.full((n * rows + 8,), 7.0, device="cuda") for _ in range(2)] for _ in range(2))
    ptrs, counts, bases = (torch.tensor([v], dtype=t, device="cuda") for v, t in ((base, torch.int64), (n, torch.int32), (0, torch.int32)))
    table = (ptrs.data_ptr(), counts.data_ptr(), bases.data_ptr(), 1, n, *x, 0)
    if two:
        _lib.call("ill_mm_chunk2", fmt, base, base + gap, rows, cols, *x, n, got[0].data_ptr(), got[1].data_ptr(), _lib.stream())
        _lib.call("ill_moe_mm_id2", fmt, cols, rows, 0, gap, *table, want[0].data_ptr(), want[1].data_ptr(), rows, _lib.stream())
    else:
        _lib.call("ill_mm_chunk", fmt, base, rows, cols, *x, n, got[0].data_ptr(), 0, _lib.stream())
        _lib.call("ill_moe_mm_id", fmt, cols, rows, 0, *table, 0, want[0].data_ptr(), rows, _lib.stream())
    for y, e in zip(got, want):
        assert torch.equal(y, e) and (y[n * rows:] == 7.0).all()
    assert D.device_status() == 0
