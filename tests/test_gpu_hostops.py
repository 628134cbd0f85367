"""The native host side of the decode operators (csrc/hostops.cpp) and the kernel behind its several-token gated product."""
import threading
import time

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


def _mat(fmt, rows, cols, seed):
    return D.upload_gmat(B.synth_matrix(fmt, rows, cols, seed=seed), fmt, rows, cols)


@pytest.mark.parametrize("n", [1, 2, 16, 17])
@pytest.mark.parametrize("fmts", [(B.Q4_K, B.Q4_K), (B.Q4_K, B.Q6_K), (B.Q8_0, B.Q8_0)])
@pytest.mark.parametrize("extra", [None, 0, 24])
def test_glu_mul_of_several_tokens(cuda_lib, fmts, n, extra):
    """glu_mul without FB (EXTRA None), with one, and with buffers EXTRA rows longer than the N tokens take: two products and
    the formula, and nothing else of FA written."""
    rows, cols = 40, 512
    g, u = _mat(fmts[0], rows, cols, 1), _mat(fmts[1], rows, cols, 2)
    x = torch.randn(n * cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    act = D.quant_q8(x, D.make_qact(n * cols, D.matrix_act_kind(g)))
    a, b = (torch.empty(n * rows, device="cuda") for _ in range(2))
    D.cmat_mul(g, act, a, n)
    D.cmat_mul(u, act, b, n)
    want = a.double() / (1.0 + torch.exp(-a.double())) * b.double()
    fa = torch.full((n * rows + (extra or 0) * rows,), 7.0, device="cuda")
    fb = None if extra is None else torch.full_like(fa, 9.0)
    assert D.glu_mul(g, u, act, fa, n, fb=fb) is fa
    # one token of one format takes its products in one launch (float terms in another order: 2e-6 of the largest, as the
    # other products of two kernels here); else the same two products, six roundings of the formula apart
    tol = 4e-6 * (a.abs().max() * b.abs().max() + want.abs().max()) if n == 1 and fmts[0] == fmts[1] else 6 * 2.0 ** -24 * want.abs() + 1e-30
    assert ((fa[:n * rows].double() - want).abs() <= tol).all()
    assert (fa[n * rows:] == 7.0).all()


def test_other_threads_run_while_a_launch_waits(cuda_lib):
    """A launch into a full queue (thousands behind half a second's sleep on the device) leaves the interpreter to others."""
    x, act = torch.randn(256, device="cuda"), D.make_qact(256, "q8k")
    D.quant_q8(x, act)
    torch.cuda.synchronize()
    gap, stop = [0.0], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gap[0], last = max(gap[0], now - last), now

    t = threading.Thread(target=tick)
    t.start()
    start = time.perf_counter()
    torch.cuda._sleep(1_000_000_000)  # cycles
    for _ in range(4000):
        D.quant_q8(x, act)
    took = time.perf_counter() - start
    stop.set()
    t.join()
    torch.cuda.synchronize()
    assert took > 0.3, "the queue never filled"
    assert gap[0] < took / 3, (gap[0], took)


@pytest.mark.parametrize("n", [1, 3, 17])
@pytest.mark.parametrize("fmts", [(B.Q4_K, B.Q4_K, B.Q6_K), (B.Q4_K, B.Q4_K, B.Q4_K), (B.Q4_K, B.Q6_K, B.Q6_K)])
def test_qkv_mul_of_mixed_formats_eager_and_captured(cuda_lib, fmts, n):
    """Q, K and V with biases in one format, with V in another and with Q in another: three products' values, launched one by
    one and replayed from a graph (where V runs beside Q and K) with other activations each time."""
    cols, rows = 512, (96, 40, 24)
    w = [_mat(f, r, cols, 3 + i) for i, (f, r) in enumerate(zip(fmts, rows))]
    g = torch.Generator(device="cuda").manual_seed(n)
    b = [torch.randn(r, device="cuda", generator=g) for r in rows]
    x, act = torch.empty(n * cols, device="cuda"), D.make_qact(n * cols, "q8k")
    y, want = ([torch.full((n * r,), -1.0, device="cuda") for r in rows] for _ in range(2))

    def step():
        D.quant_q8(x, act)
        D.qkv_mul(*w, act, *y, bq=b[0], bk=b[1], bv=b[2], n=n)

    x.normal_(generator=g)
    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for run in (step, graph.replay, graph.replay):
        x.normal_(generator=g)
        for t in y:
            t.fill_(-1.0)
        run()
        other = D.quant_q8(x, D.make_qact(n * cols, "q8k"))
        for m, bias, t in zip(w, b, want):
            D.cmat_mul(m, other, t, n, bias=bias)
        for got, t in zip(y, want):  # (one launch for several matrices may add a row's float terms in another order)
            assert (got - t).abs().max() <= 2e-6 * t.abs().max()
