"""The native decode operators (csrc/hostops.cpp) where they raise before they launch anything: no GPU needed."""
import os
import subprocess
import sys
from types import SimpleNamespace

import pytest
import torch

from illatio_b200 import cuda_dense as D

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SPARSE = "torch.sparse_coo_tensor([[0]], [1.0], (32,))"
ACT = "D.make_qact(32, 'q8', device='cpu')"
MAT = "D.CMat('w', 0, 1, 32, torch.zeros(34, dtype=torch.uint8))"
NO_STORAGE = [
    "D.quant_q8(%s, %s)" % (SPARSE, ACT),
    "torch.func.vmap(lambda x: D.quant_q8(x, %s) and x)(torch.zeros(2, 32))" % ACT,
    "D.rmsnorm_q8(%s, torch.ones(32), %s, 32, 1e-6)" % (SPARSE, ACT),
    "D.cmat_mul(%s, %s, %s)" % (MAT, ACT, SPARSE),
    "D.qkv_mul(%s, %s, %s, %s, %s, None, None)" % (MAT, MAT, MAT, ACT, SPARSE),
    "D.glu_mul(%s, %s, %s, %s)" % (MAT, MAT, ACT, SPARSE),
    "D.embed(%s, torch.zeros(1, dtype=torch.int32), %s)" % (MAT, SPARSE),
]
NO_DRIVER = [
    "D.quant_q8(torch.zeros(32), %s)" % ACT,
    "D.rmsnorm_q8(torch.zeros(32), torch.ones(32), %s, 32, 1e-6)" % ACT,
    "D.cmat_mul(%s, %s, torch.zeros(1))" % (MAT, ACT),
    "D.qkv_mul(%s, %s, %s, %s, torch.zeros(1), torch.zeros(1), torch.zeros(1))" % (MAT, MAT, MAT, ACT),
    "D.glu_mul(%s, %s, %s, torch.zeros(1))" % (MAT, MAT, ACT),
    "D.glu_mul(%s, %s, %s, torch.zeros(2), 2, torch.zeros(2))" % (MAT, MAT, ACT),
    "D.embed(%s, torch.zeros(1, dtype=torch.int32), torch.zeros(32))" % MAT,
]
CODE = """
import torch
from illatio_b200 import cuda_dense as D
for expr in %r:
    try:
        eval(expr)
    except RuntimeError as e:
        print("raised", flush=True)
    else:
        raise SystemExit(expr)
"""


@pytest.mark.skipif(torch.cuda.is_available(), reason="host tensors: only where nothing can be launched")
@pytest.mark.parametrize("exprs", [NO_STORAGE, NO_DRIVER], ids=["no_storage", "no_driver"])
def test_an_exception_of_torch_is_a_python_exception(exprs):
    """In a process of its own: a C++ exception that is not caught ends the process."""
    r = subprocess.run([sys.executable, "-c", CODE % exprs], capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0 and r.stdout.count("raised") == len(exprs), (r.returncode, r.stdout, r.stderr[-500:])


@pytest.mark.parametrize("fa,fb,n", [((16, 8), (4, 8), 4), ((128,), (32,), 4), ((4, 8), (16, 8), 4), ((32,), (4, 8), 4), ((2, 8), (2, 8), 4),
                                     ((2, 8), None, 4), ((128,), (32,), 0)])
def test_glu_mul_refuses_buffers_that_do_not_agree(fa, fb, n):
    """FA and FB of different shapes, or shorter than the N tokens' rows: refused before anything is launched."""
    m = D.CMat("w", 0, 8, 32, torch.zeros(8 * 34, dtype=torch.uint8))
    act = D.make_qact(4 * 32, "q8", device="cpu")
    with pytest.raises(RuntimeError, match="do not agree|broadcast"):
        D.glu_mul(m, m, act, torch.zeros(fa), n, None if fb is None else torch.zeros(fb))


@pytest.mark.skipif(torch.cuda.is_available(), reason="host tensors: only where nothing can be launched")
def test_few_tokens_follow_tc_min_tokens(monkeypatch):
    """TC_MIN_TOKENS below 16: cmat_mul sends what tc_takes() says to the tcgen05 kernel."""
    sent = []
    monkeypatch.setattr(D, "TC_MIN_TOKENS", 4)
    monkeypatch.setattr(D, "TC_MIN_ROWS", 8)
    monkeypatch.setattr(D, "_chunk_f16_of", lambda act, n, cols: n)
    monkeypatch.setattr(D, "cmat_mul_tc", lambda w, cf, y, acc=False: sent.append((cf, acc)) or y)
    w = D.CMat("w", 1, 8, 256, torch.zeros(8 * 144, dtype=torch.uint8))
    for n in (4, 16):
        assert D.tc_takes(w, n)
        D.cmat_mul(w, D.make_qact(n * 256, "q8k", device="cpu"), torch.zeros(n * 8), n, acc=True)
    assert sent == [(4, True), (16, True)]
    with pytest.raises(RuntimeError):  # three tokens: a launch
        D.cmat_mul(w, D.make_qact(3 * 256, "q8k", device="cpu"), torch.zeros(24), 3)


@pytest.mark.skipif(torch.cuda.is_available(), reason="host tensors: only where nothing can be launched")
def test_activations_of_the_callers_own_class():
    """An object with a QAct's four attributes gets as far as the launch, and its fp16 form is made on it."""
    a = D.make_qact(256, "q8k", device="cpu")
    own = SimpleNamespace(kind=a.kind, xq=a.xq, xs=a.xs, xsum=a.xsum)
    w = D.CMat("w", 1, 1, 256, torch.zeros(144, dtype=torch.uint8))
    for call in (lambda: D.quant_q8(torch.zeros(256), own), lambda: D.rmsnorm_q8(torch.zeros(256), torch.ones(256), own, 256, 1e-6),
                 lambda: D.cmat_mul(w, own, torch.zeros(1)), lambda: D._chunk_f16_of(own, 1, 256)):
        with pytest.raises(RuntimeError):
            call()


@pytest.mark.parametrize("call", [lambda act: D.quant_q8(torch.sparse_coo_tensor([[0]], [1.0], (512,)), act),
                                  lambda act: D.rmsnorm_q8(torch.sparse_coo_tensor([[0]], [1.0], (512,)), torch.ones(512), act, 512, 1e-6)])
def test_an_activation_keeps_its_f16_buffers_past_an_exception(call):
    """A captured token may still use them."""
    act = D.make_qact(512, "q8k", device="cpu")
    cf = act._cf = SimpleNamespace(n=1, cols=256)
    act._cf_fresh = True
    with pytest.raises(RuntimeError):
        call(act)
    assert act._cf is cf and not act._cf_fresh
