"""Q8_0 chunk products (ill_mv of more than 16 tokens; on tcgen05, some on mma.sync): tiles, ragged edges and rows at every alignment, bit for
bit against the same sums taken block by block in plain PyTorch: y = y + float(isum) * (d_w * d_x), a rounding a step."""
import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import cuda_dense as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,n,off,acc,bias", [
    (1, 128, 17, 0, False, False),      # one row, in a map of its own
    (2, 128, 31, 0, True, False),
    (127, 384, 33, 0, False, True),     # rows 408 bytes long: the even and the odd ones in two maps
    (129, 256, 64, 0, True, True),      # rows 272 bytes long: one map; a second tile of one row
    (300, 896, 129, 2, True, False),    # blocks that start in the middle of a word
    (257, 896, 65, 8, False, False),
    (130, 640, 48, 4, False, True),
    (896, 1152, 777, 0, False, False),  # tiles of 48
    (384, 512, 1000, 14, True, True),
    (2048, 1024, 300, 0, False, False),
    (5120, 128, 3900, 0, False, False),  # many rounds of tiles of 128
    (9728, 128, 512, 0, False, False),  # even shares, tiles that end where a tile of rows or a share does
    (9700, 128, 505, 2, True, True),
    (17300, 256, 399, 0, False, True),
    (1536, 128, 8190, 0, True, False),
    (151936, 128, 17, 0, False, False),  # many tiles of rows of few tokens
    (127, 384, 29, 0, False, True),
    (129, 256, 32, 0, True, True),
    # chunks of the kernel on mma.sync (as the third and fourth, and 128 x 128 below)
    (128, 128, 64, 0, False, False),
    (1024, 128, 33, 0, True, True),
    (20001, 256, 80, 2, False, True),
    (4864, 896, 511, 4, True, False),
    (5120, 1536, 301, 10, False, False),
])
def test_q8_0_chunk_bits(cuda_lib, rows, cols, n, off, acc, bias):
    g = torch.Generator(device="cuda")
    g.manual_seed(rows * 7 + cols * 3 + n)
    nb = cols // 32
    d = torch.randn(rows, nb, device="cuda", generator=g).abs().to(torch.float16)
    q = torch.randint(-128, 128, (rows, nb, 32), dtype=torch.int8, device="cuda", generator=g)
    raw = torch.cat([d.view(torch.uint8).reshape(rows, nb, 2), q.view(torch.uint8)], dim=2).reshape(-1)
    buf = torch.empty(raw.numel() + 16, dtype=torch.uint8, device="cuda")
    w = buf[off:off + raw.numel()]
    w.copy_(raw)
    x = torch.randint(-127, 128, (n, nb, 32), dtype=torch.int8, device="cuda", generator=g)
    xs = torch.rand(n, nb, device="cuda", generator=g) * 0.03
    b = torch.randn(rows, device="cuda", generator=g) if bias else None
    y0 = torch.randn(n * rows + 32, device="cuda", generator=g)
    want = torch.zeros(n, rows, device="cuda")
    for k in range(nb):
        isum = x[:, k].float() @ q[:, k].float().T  # whole numbers below 2^24: exact
        want += isum * (xs[:, k, None] * d[None, :, k].float())
    if bias:
        want += b
    if acc:
        want += y0[:n * rows].view(n, rows)
    y = y0.clone()
    _lib.call("ill_mv", 0, w.data_ptr(), rows, cols, x.data_ptr(), xs.data_ptr(), 0, y.data_ptr(), b.data_ptr() if bias else 0, int(acc), n,
              _lib.stream())
    assert torch.equal(y[:n * rows].view(n, rows), want)
    assert torch.equal(y[n * rows:], y0[n * rows:])
    assert D.device_status() == 0
