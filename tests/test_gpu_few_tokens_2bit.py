"""Products of two to sixteen tokens in the 2-bit formats (ill_mv on mma.sync) against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D

from gpu_util import act_to_host, dev_act, rel_errors, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(cuda_lib):
    yield
    assert D.device_status() == 0


def _p(t):
    return t.data_ptr()


@pytest.mark.parametrize("fmt,rows,cols,n,off", [(B.Q2_K, 40, 2560, 16, 0), (B.Q2_K, 19, 256, 3, 0), (B.Q2_K, 300, 5120, 8, 2), (B.Q2_K, 33, 1792, 9, 4),
                                                 (B.IQ2_XXS, 40, 2560, 16, 0), (B.IQ2_XXS, 19, 256, 2, 2), (B.IQ2_XXS, 300, 4096, 8, 0),
                                                 (B.IQ2_XXS, 33, 1792, 9, 6), (B.IQ2_XXS, 2400, 1024, 5, 0), (B.Q2_K, 20, 17408, 4, 0), (B.Q2_K, 36, 17408, 9, 0),
                                                 (B.IQ2_XXS, 36, 17408, 15, 0)])
def test_few_tokens_of_the_two_bit_formats(oracle, fmt, rows, cols, n, off):
    x = np.random.default_rng(cols).standard_normal(n * cols).astype(np.float32)
    act = dev_act(fmt, x)
    w = B.synth_matrix(fmt, rows, cols, seed=3)
    buf = torch.zeros(w.size + 16, dtype=torch.uint8, device="cuda")
    buf[off:off + w.size] = to_dev(w).reshape(-1)
    y, bias = torch.full((n * rows + 8,), 7.0, device="cuda"), torch.randn(rows, device="cuda")
    _lib.call("ill_mv", fmt, _p(buf) + off, rows, cols, _p(act.xq), _p(act.xs), _p(act.xsum), _p(y), _p(bias), 0, n, _lib.stream())
    xq, xs, bs = act_to_host(act)
    want = np.stack([oracle.matvec(fmt, w, rows, cols, (xq[t * cols:(t + 1) * cols], xs[t * (cols // 256):(t + 1) * (cols // 256)],
                                                        bs[t * (cols // 16):(t + 1) * (cols // 16)]))[0] for t in range(n)])
    # whole-number block sums: what differs is the order of at most 136 32-bit additions
    err, _ = rel_errors(y[:n * rows].cpu().numpy().reshape(n, rows) - bias.cpu().numpy(), want)
    assert err <= 1e-5 and (y[n * rows:] == 7.0).all()


@pytest.mark.parametrize("fmt", [B.Q2_K, B.IQ2_XXS])
@pytest.mark.parametrize("n", [8, 16])
def test_registers_of_the_two_bit_formats(fmt, n):
    out = (ctypes.c_int * 8)()
    assert _lib.status("ill_test_few_tokens_plan", 1, fmt, 0, 0, 64, 0, 0, 1024, n, 0, out) == 0
    assert 0 < out[7] <= out[6]
