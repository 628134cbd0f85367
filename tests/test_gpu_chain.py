"""A token's chain as recorded launches (ill_chain_*, DecodePlan) and as the one cooperative launch (ill_decode_plan / ill_decode_run): the
same bits; into a recording of the caller's; lists that are refused."""
import ctypes

import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D

from gpu_util import one_launch

pytestmark = pytest.mark.gpu
EPS = 1e-6


@pytest.fixture(autouse=True)
def _need_gpu(cuda_lib):
    yield
    assert D.device_status() == 0


def _mat(fmt, rows, cols, seed):
    return D.CMat("m", fmt, rows, cols, B.synth_matrix_torch(fmt, rows, cols, seed=seed))


class Layer:
    """Products whose activations are shared by two, three and one of them, in one format and in two, with and without biases, sums into
    a vector that exists, norms and gated products; and products large enough (16 MB) that a launch of two of them would add a
    row's blocks in another order than one each."""

    def __init__(self, main, alt, hidden=512, kv=256, ffn=1024, big=0):
        g = torch.Generator(device="cuda").manual_seed(hidden + main)
        self.keep = [_mat(f, r, c, i + 1) for i, (f, r, c) in enumerate([
            (main, hidden, hidden), (main, kv, hidden), (alt, kv, hidden), (main, hidden, hidden), (main, ffn, hidden), (main, ffn, hidden),
            (alt, hidden, ffn), (main, big or 64, hidden), (main, big or 64, hidden)])]
        q, k, v, o, gate, up, down, b1, b2 = self.keep
        f = dict(dtype=torch.float32, device="cuda")
        self.x0 = torch.randn(hidden, device="cuda", generator=g)
        self.nw = torch.rand(hidden, device="cuda", generator=g) + 0.5
        self.bias = torch.randn(kv, device="cuda", generator=g)
        self.h = torch.empty(hidden, **f)
        self.out = [torch.empty(n, **f) for n in (hidden, kv, kv, ffn, big or 64, big or 64)]
        yq, yk, yv, fa, y1, y2 = self.out
        op = D.decode_op
        self.ops = [op(q, self.h, yq, norm_w=self.nw, eps=EPS), op(k, self.h, yk, norm_w=self.nw, eps=EPS, bias=self.bias, after=False),
                    op(v, self.h, yv, norm_w=self.nw, eps=EPS, after=False), op(o, yq, self.h, acc=True),
                    op(gate, self.h, fa, w2=up, norm_w=self.nw, eps=EPS), op(down, fa, self.h, acc=True),
                    op(b1, self.h, y1), op(b2, self.h, y2, after=False)]

    def state(self, run):
        self.h.copy_(self.x0)
        for t in self.out:
            t.fill_(-3.0)
        run()
        torch.cuda.synchronize()
        return [t.clone() for t in [self.h, *self.out]]


@pytest.mark.parametrize("main,alt,big", [(B.Q4_K, B.Q6_K, 0), (B.Q8_0, B.Q8_0, 0), (B.IQ2_XXS, B.Q2_K, 0), (B.Q6_K, B.Q4_K, 0), (B.Q4_K, B.Q6_K, 36000)])
def test_recorded_launches_are_the_one_launch(main, alt, big):
    m = Layer(main, alt, big=big)
    want = m.state(one_launch(m.ops))
    plan = D.DecodePlan(m.ops)
    for _ in range(2):
        for a, b in zip(m.state(plan.run), want):
            assert torch.isfinite(a).all() and torch.equal(a, b)


def test_into_a_recording_and_in_another_stream():
    m = Layer(B.Q4_K, B.Q6_K)
    plan = D.DecodePlan(m.ops)
    want = m.state(plan.run)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.run()
    assert all(torch.equal(a, b) for a, b in zip(m.state(graph.replay), want))
    side = torch.cuda.Stream()

    def aside():
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            plan.run()
        torch.cuda.current_stream().wait_stream(side)
    assert all(torch.equal(a, b) for a, b in zip(m.state(aside), want))
    plan.run()
    del plan            # a token may still be on its way
    torch.cuda.synchronize()


def test_scratch_of_a_plan_that_runs_in_another_stream():
    """The plan goes while a token waits in a stream that is not the one it was made in: its scratch is not given out meanwhile."""
    m = Layer(B.Q4_K, B.Q6_K)
    plan = D.DecodePlan(m.ops)
    want = m.state(plan.run)
    m.h.copy_(m.x0)
    torch.cuda.synchronize()
    side, busy = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)
        plan.run()
        busy.record()
    at, size = plan.chain.scratch.data_ptr(), plan.chain.scratch.numel()
    del plan
    others = [torch.empty(size, dtype=torch.uint8, device="cuda") for _ in range(3)]
    assert not busy.query() and all(t.data_ptr() != at for t in others)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip([m.h, *m.out], want))


def test_a_plan_is_made_beside_what_runs():
    """Without waiting for the stream, and with no memory but its scratch."""
    m = Layer(B.Q4_K, B.Q6_K)
    D.DecodePlan(m.ops)
    torch.cuda.synchronize()
    busy, before = torch.cuda.Event(), torch.cuda.memory_allocated()
    torch.cuda._sleep(200_000_000)
    busy.record()
    plan = D.DecodePlan(m.ops)
    assert not busy.query()
    assert torch.cuda.memory_allocated() - before <= (plan.chain.scratch.numel() + 511) // 512 * 512
    torch.cuda.synchronize()


@pytest.mark.parametrize("change", ["", "cols 500", "cols 32768", "cols 33024", "rows 0", "w 8", "kind 7", "fmt 9", "w2 16", "x 4", "y 2", "1024", "many"])
def test_the_check_refuses_what_the_one_launch_does(change):
    w = _mat(B.Q4_K, 16, 512, 1)
    op = D.decode_op(w, torch.zeros(512, device="cuda"), torch.zeros(16, device="cuda"))
    ops = [op]
    if change == "1024":
        ops = [op] * 1024
    elif change == "many":        # does not fit beside so many columns
        ops = [op] * 900
        op.cols = 32768
    elif change:
        k, v = change.split()
        setattr(op, k, getattr(op, k) + int(v) if k in ("w", "x", "y") else int(v))
    n = len(ops)
    arr, nbytes, launch = (_lib.DecodeOp * n)(*ops), _lib.lib().ill_decode_plan_bytes(n), (ctypes.c_int32 * 16)()
    buf = torch.zeros(nbytes + 128, dtype=torch.uint8, device="cuda")
    rc = _lib.status("ill_decode_plan", arr, n, (buf.data_ptr() + 127) // 128 * 128, nbytes, launch, _lib.stream())
    assert _lib.status("ill_decode_check", arr, n) == rc and (rc == 0) == (change in ("", "cols 32768", "1024")) and bool(launch[9]) == (rc == 0)
    if rc:
        with pytest.raises(_lib.IllatioError) as e:
            D.DecodePlan(ops)
        assert e.value.code == rc
    with pytest.raises(ValueError):
        D.DecodePlan([op] * 1025)


def test_what_a_chain_refuses():
    m = Layer(B.Q4_K, B.Q6_K)
    n = len(m.ops)
    arr, out = (_lib.DecodeOp * n)(*m.ops), ctypes.c_uint64(7)
    nbytes = _lib.lib().ill_chain_scratch_bytes(arr, n)
    buf = torch.empty(nbytes + 128, dtype=torch.uint8, device="cuda")
    base = (buf.data_ptr() + 127) // 128 * 128
    new = lambda a, k, s, b: _lib.status("ill_chain_new", a, k, s, b, ctypes.byref(out))  # noqa: E731
    assert new(arr, 0, base, nbytes) == 1 and out.value == 0
    assert new(arr, n, 0, nbytes) == 1 and new(arr, n, base + 16, nbytes) == 2 and new(arr, n, base, nbytes - 1) == 6
    arr[1].cols = 500
    assert new(arr, n, base, nbytes) == 1
    assert _lib.status("ill_chain_run", 0, _lib.stream()) == 1 and _lib.status("ill_chain_free", 0) == 0
