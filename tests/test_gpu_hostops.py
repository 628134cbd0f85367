"""The native host side of the decode operators (csrc/hostops.cpp) and the kernel behind its several-token gated product."""
import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,off", [(1, 0), (3, 0), (1023, 0), (1024, 0), (1025, 0), (4096, 1)])
def test_silu_mul(cuda_lib, n, off):
    """ill_silu_mul at the edges of its four values a thread, 16-byte aligned or not, in place; against the same
    formula in torch, a rounding of each of its four steps apart (4 * 2^-24)."""
    g = torch.Generator(device="cuda").manual_seed(n)
    a, b = (torch.randn(n + off + 8, device="cuda", generator=g) * 4 for _ in range(2))
    x, y = a[off:off + n], b[off:off + n]
    want = (x.double() / (1.0 + torch.exp(-x.double()))) * y.double()
    tail = a[off + n:].clone()
    _lib.call("ill_silu_mul", n, x.data_ptr(), y.data_ptr(), x.data_ptr(), _lib.stream())
    # exp is a 2-ulp function; its relative error reaches the quotient at most whole
    assert ((x.double() - want).abs() <= 6 * 2.0 ** -24 * want.abs() + 1e-30).all()
    assert torch.equal(a[off + n:], tail)


def test_arguments_and_errors(cuda_lib):
    """Positional and keyword arguments, what comes back, and the exceptions the Python forms raise."""
    w = D.upload_gmat(B.synth_matrix(B.Q4_K, 64, 512, seed=1), B.Q4_K, 64, 512)
    x = torch.randn(4 * 512, device="cuda")
    act, y, z = D.make_qact(4 * 512, "q8k"), torch.zeros(4 * 64, device="cuda"), torch.ones(4 * 64, device="cuda")
    assert D.quant_q8(x, act=act) is act
    assert D.cmat_mul(w, act, y, n=4) is y
    D.cmat_mul(w, act, z, 4, acc=True)
    assert torch.equal(z, y + 1.0)
    with pytest.raises(TypeError):
        D.cmat_mul(w, act)
    with pytest.raises(TypeError):
        D.quant_q8(x, act, scale=1)
    with pytest.raises(TypeError):
        D.cmat_mul(w, act, 5)
    bad = D.QAct("q8k", act.xq[1:], act.xs, act.xsum)
    with pytest.raises(_lib.IllatioError) as e:
        D.cmat_mul(w, bad, y)
    assert e.value.code == 2
    assert D.device_status() == 0
