"""Host side of the dense decode path: the reference's src/cuda-dense.lisp,
mirrored name for name over the C ABI.

The reference drives its kernels from Lisp (`launch`, src/cuda.lisp:323); no
Lisp implementation is available to run, so this module plays the part of the
Lisp caller: the same operators (UPLOAD-GMAT, QUANT-Q8, CMAT-MUL, QKV-MUL,
GLU-MUL, EMBED), the same argument meaning, over libillatio_b200.so.  torch is
used only to own device memory and streams.

Differences from the reference's device layout, all invisible to callers of
these operators: matrices stay as raw GGUF blocks (no repack_q8 / repack_q6k),
and K-quant products take Q8_K activations as the CPU path does (`xs` is then
one float per 256 and `xsum` one int16 per 16 quants).
"""
from dataclasses import dataclass

import numpy as np
import torch

from . import _lib
from .blocks import BLOCK_BYTES, BLOCK_WEIGHTS, NAMES, Q8_0, row_bytes


def _ptr(t):
    return 0 if t is None else t.data_ptr()


_stream = _lib.stream


@dataclass
class CMat:
    """A matrix on the device (CMAT, src/cuda-dense.lisp:13-16): raw blocks."""
    name: str
    type: int
    rows: int
    cols: int
    qs: torch.Tensor  # uint8, rows * row_bytes

    @property
    def row_bytes(self):
        return row_bytes(self.type, self.cols)

    @property
    def nbytes(self):
        return self.rows * self.row_bytes


def cmat_kquant_p(w):
    return w.type != Q8_0


def upload_gmat(blocks, fmt, rows, cols, name="", device="cuda"):
    """UPLOAD-GMAT (src/cuda-dense.lisp:75-100): a tensor's raw blocks (uint8
    numpy array or tensor) to the device, as they are."""
    if cols % BLOCK_WEIGHTS[fmt]:
        raise ValueError("%s: %d columns is not a whole number of blocks" % (name, cols))
    t = torch.as_tensor(blocks).reshape(-1)
    if t.dtype != torch.uint8 or t.numel() != rows * row_bytes(fmt, cols):
        raise ValueError("%s: expected %d bytes of %s blocks" % (name, rows * row_bytes(fmt, cols), NAMES[fmt]))
    return CMat(name, fmt, rows, cols, t.to(device, non_blocking=True).contiguous())


@dataclass
class QAct:
    """Quantized activations of N tokens (the cctx's xq / xs / xsum)."""
    kind: str            # "q8" (Q8_0 blocks) or "q8k" (Q8_K super-blocks)
    xq: torch.Tensor     # int8 [n * cols]
    xs: torch.Tensor     # float32 per 32 (q8) or per 256 (q8k)
    xsum: torch.Tensor   # q8: int32 per 32 (or None); q8k: int16 per 16
    _cf = None           # the fp16 form, once a tcgen05 product has used it (a ChunkF16)
    _cf_fresh = False    # it is that of the quants


def make_qact(n, kind, device="cuda", want_xsum=False):
    """Room for N activations in KIND (MAKE-QACT, src/kquant.lisp:506-510)."""
    if kind == "q8":
        return QAct(kind, torch.empty(n, dtype=torch.int8, device=device),
                    torch.empty(n // 32, dtype=torch.float32, device=device),
                    torch.empty(n // 32, dtype=torch.int32, device=device) if want_xsum else None)
    return QAct(kind, torch.empty(n, dtype=torch.int8, device=device),
                torch.empty(n // 256, dtype=torch.float32, device=device),
                torch.empty(n // 16, dtype=torch.int16, device=device))


def matrix_act_kind(w):
    """MATRIX-ACT-KIND (src/kquant.lisp:532-533)."""
    return "q8k" if cmat_kquant_p(w) else "q8"


# The operators of a decoded token are native (csrc/hostops.cpp: the signatures and docstrings are there); the
# functions below that begin with an underscore and share a name with one are what it leaves to Python.
_H = _lib.hostops()
quant_q8, rmsnorm_q8, cmat_mul, qkv_mul, glu_mul, embed = (getattr(_H, f) for f in (
    "quant_q8", "rmsnorm_q8", "cmat_mul", "qkv_mul", "glu_mul", "embed"))


def _quant_q8(x, act, f16_scale=True):
    """quant_q8 of an ACT whose fp16 form is in use by the tcgen05 products: renewed in the same launch."""
    n, cf = x.numel(), act._cf
    if act.kind == "q8k" and cf.n * cf.cols == n:
        _lib.call("ill_quant_q8_k_f16", _ptr(x), _ptr(act.xq), _ptr(act.xs), _ptr(act.xsum), _ptr(cf.xh), _ptr(cf.xe), n // 256,
                  _stream())
        cf.xd = act.xs
        act._cf_fresh = True
        return act
    act._cf, act._cf_fresh = None, False
    try:
        return quant_q8(x, act, f16_scale)
    finally:
        act._cf = cf


def _rmsnorm_q8(x, w, act, d, eps, n=1, h=None, f16_scale=True):
    """rmsnorm_q8 of an ACT whose fp16 form is in use by the tcgen05 products: renewed in the same launch."""
    cf = act._cf
    if act.kind == "q8k" and cf.n == n and cf.cols == d:
        _lib.call("ill_rmsnorm_q8k_f16", _ptr(x), _ptr(w), _ptr(h), _ptr(act.xq), _ptr(act.xs), _ptr(act.xsum), _ptr(cf.xh),
                  _ptr(cf.xe), d, float(eps), n, _stream())
        cf.xd = act.xs
        act._cf_fresh = True
        return act
    act._cf, act._cf_fresh = None, False
    try:
        return rmsnorm_q8(x, w, act, d, eps, n, h, f16_scale)
    finally:
        act._cf = cf


def _by_tc(w, act, n, bias):
    """Whether a product of a chunk goes to the tcgen05 kernel of the K formats."""
    return ((w.type == 1 or (w.type == 2 and TC_Q6K)) and act.kind == "q8k" and n >= TC_MIN_TOKENS and w.rows >= TC_MIN_ROWS and w.rows % 4 == 0 and bias is None
            and w.qs.data_ptr() % 16 == 0 and act.xq.numel() == n * w.cols)


def _cmat_mul(w, act, y, n=1, bias=None, acc=False):
    """cmat_mul of a chunk, or of a few tokens that have to be split."""
    if _by_tc(w, act, n, bias):
        # a prefill chunk of a Q4_K / Q6_K matrix: the tcgen05 kernel (the activations' fp16 form is made once per quantization)
        return cmat_mul_tc(w, _chunk_f16_of(act, n, w.cols), y, acc=acc)
    done = 0
    # Q8_0 / Q4_K / Q6_K take a whole chunk of tokens in one launch; the other formats up to 16 tokens --
    # fewer when their activations do not fit beside the stages
    kmax = n
    while done < n:
        k = min(kmax, n - done)
        sc = w.cols // (32 if act.kind == "q8" else 256)
        rc = _lib.status("ill_mv", w.type, _ptr(w.qs), w.rows, w.cols,
                         act.xq.data_ptr() + done * w.cols, act.xs.data_ptr() + 4 * done * sc,
                         0 if act.kind == "q8" else act.xsum.data_ptr() + 2 * done * (w.cols // 16),
                         y.data_ptr() + 4 * done * w.rows, _ptr(bias), 1 if acc else 0, k, _stream())
        if rc == 3 and k > 1:   # ILL_ERR_UNSUPPORTED: long rows, many tokens
            kmax = 16 if k > 16 else k // 2
            continue
        if rc:
            _lib.call("ill_mv", w.type, _ptr(w.qs), w.rows, w.cols, act.xq.data_ptr() + done * w.cols,
                      act.xs.data_ptr() + 4 * done * sc, 0 if act.kind == "q8" else act.xsum.data_ptr() + 2 * done * (w.cols // 16),
                      y.data_ptr() + 4 * done * w.rows, _ptr(bias), 1 if acc else 0, k, _stream())  # raises with the text
        done += k
    return y


_SIDE = {}


def _side_stream(device):
    """A second stream per device for products that may run beside the current stream's."""
    s = _SIDE.get(device)
    if s is None:
        s = _SIDE[device] = torch.cuda.Stream(device=device)
    return s


# Two matrices of few rows beside one of the tcgen05 kernel (which wants the activations' fp16 form in this stream in any case) go to the
# exact form of that kernel: its tiles are 64 rows of X at most, which a chunk's K and V make one round of, and it adds the same integers
# in the same steps as the int8 kernel.  us, int8 / exact, both of Q4_K | one of Q6_K: 1024 x 2560 of 64 tokens 23.5 / 17.3 | 23.5 / 21.5, of
# 256 30 / 17 | 32 / 23, of 512 44 / 19 | 48 / 23, of 2048 135 / 54 | 133 / 64; 1024 x 8192 of 64 53 / 34 | 54 / 48; 256 x 2048 of 64 19.4 / 15.4 |
# 19.4 / 18.5, of 2048 38 / 17 | 40 / 21; 128 x 4096 of 64 30 / 20 | 30 / 28.  Q6_K of an odd number of blocks, which a TMA load cannot
# bring: 1024 x 2304 of 64 21.5 / 21.6, of 128 21.5 / 23.5, of 256 29.7 / 23.5.
EXACT_MIN_Q6K = 1 << 18  # rows times tokens, there


def _exact_takes(w, y, bias, like, act, n):
    """Whether a matrix beside one of _by_tc's, and in one launch with LIKE, goes to ill_mm_chunk_exact."""
    return ((w.type == 1 or (w.type == 2 and TC_Q6K and (w.cols % 512 == 0 or w.rows * n >= EXACT_MIN_Q6K))) and 0 < w.rows == like.rows and w.rows % 4 == 0
            and w.cols == like.cols and bias is None and w.qs.data_ptr() % 16 == 0 and y.data_ptr() % 16 == 0 and act.xq.numel() == n * w.cols)


def chunk_mul_3(mats, act, n):
    """The products of a chunk of N tokens that share the activations ACT, MATS a list of (matrix, output, bias): two or three in one
    launch where that is to be had (ill_mm_chunk_exact, ill_mv_3n), else one by one; those of the tcgen05 kernel of the K formats by themselves."""
    joint = [m for m in mats if not _by_tc(m[0], act, n, m[2])]
    if len(joint) == 2 < len(mats) and all(_exact_takes(w, y, b, joint[0][0], act, n) for w, y, b in joint):
        cf, (w, y, _), (w2, y2, _) = _chunk_f16_of(act, n, joint[0][0].cols), *joint
        _lib.call("ill_mm_chunk_exact", w.type, _ptr(w.qs), w2.type, _ptr(w2.qs), w.rows, w.cols, _ptr(cf.xh), _ptr(cf.xe), _ptr(cf.xd), n, _ptr(y), _ptr(y2),
                  _stream())
        mats, joint = [m for m in mats if all(m is not j for j in joint)], []
    a = joint[0][0] if joint else None
    if 2 <= len(joint) <= 3 and n > 16 and all(w.cols == a.cols and (w.type == 0) == (a.type == 0) and w.rows > 0 for w, _, _ in joint) and (a.type == 0) == (act.kind == "q8"):
        w, y, b = ([m[i] for m in joint] + [None] * (3 - len(joint)) for i in range(3))
        rc = _lib.status("ill_mv_3n", *(m.type if m else 0 for m in w), *(_ptr(m.qs) if m else 0 for m in w), *(m.rows if m else 0 for m in w),
                         a.cols, _ptr(act.xq), _ptr(act.xs), 0 if act.kind == "q8" else _ptr(act.xsum), *map(_ptr, y), *map(_ptr, b), n, _stream())
        if rc == 0:
            mats = [m for m in mats if all(m is not j for j in joint)]
        elif rc != 3:
            _lib.fail("ill_mv_3n", rc)
    for w, y, b in mats:
        cmat_mul(w, act, y, n, bias=b)


def _qkv_mul(wq, wk, wv, act, q, k, v, bq=None, bk=None, bv=None, n=1):
    """qkv_mul of a chunk; or of one token with a V in a format of its own, in a stream that is being captured: Q and K in one
    launch, V in its own beside it (both read the same activations; in the graph this is a fork and a join)."""
    if n != 1:
        return chunk_mul_3([(wq, q, bq), (wk, k, bk), (wv, v, bv)], act, n)
    cur = torch.cuda.current_stream()
    side = _side_stream(cur.device)
    side.wait_stream(cur)
    with torch.cuda.stream(side):
        cmat_mul(wv, act, v, n, bias=bv)
    _lib.call("ill_mv_3", wq.type, _ptr(wq.qs), _ptr(wk.qs), 0, wq.rows, wk.rows, 0, wq.cols,
              _ptr(act.xq), _ptr(act.xs), _ptr(act.xsum) if act.kind == "q8k" else 0,
              _ptr(q), _ptr(k), 0, _ptr(bq), _ptr(bk), 0, _stream())
    cur.wait_stream(side)


def _glu_mul(g, u, act, fa, n=1, fb=None):
    """glu_mul of several tokens, or of two formats."""
    if fb is None:
        fb = torch.empty_like(fa)
    count = max(n, 0) * g.rows
    if torch.broadcast_shapes(fa.shape, fb.shape) != fa.shape or min(fa.numel(), fb.numel()) < count:
        raise RuntimeError("glu_mul(): FA of %d values and FB of %d do not agree, or hold fewer than N * ROWS = %d" % (fa.numel(), fb.numel(), count))
    cmat_mul(g, act, fa, n)
    cmat_mul(u, act, fb, n)
    _lib.call("ill_silu_mul", count, _ptr(fa), _ptr(fb), _ptr(fa), _stream())
    return fa


_SLOW = {"quant_q8": _quant_q8, "rmsnorm_q8": _rmsnorm_q8, "cmat_mul": _cmat_mul, "qkv_mul": _qkv_mul, "glu_mul": _glu_mul,
             "error": _lib.fail, "vars": globals()}
_H.set_slow(_SLOW)


class ChunkF16:
    """A chunk's Q8_K activations as the tcgen05 product takes them (ill_act_f16): XH [n, cols] the quants as fp16
    (exact), XE [n, cols / 256, 64] the sums of 16 as fp16 (exact; 48 of each 64 zero), XD the block scales."""

    def __init__(self, n, cols, device="cuda"):
        self.n, self.cols = n, cols
        self.xh = torch.empty(n, cols, dtype=torch.float16, device=device)
        self.xe = torch.empty(n, cols // 256, 64, dtype=torch.float16, device=device)
        self.xd = None

    def fill(self, act):
        _lib.call("ill_act_f16", self.n, self.cols, _ptr(act.xq), _ptr(act.xsum), 0, _ptr(self.xh), _ptr(self.xe), _stream())
        self.xd = act.xs
        return self


def cmat_mul_tc(w, cf, y, acc=False):
    """CMAT-MUL-N for a prefill chunk on the 5th-generation tensor cores (ill_mm_chunk): Y[t*rows + r] (+)= W[r] . X[t]
    for the chunk CF (a ChunkF16 filled from the chunk's Q8_K activations) and a Q4_K or Q6_K matrix W.  Replaces
    mm_q4k_mma / mm_q6k_mma (src/cuda/kquant.cu:316-466) behind CMAT-MUL-N (src/cuda-dense.lisp:250-255)."""
    _lib.call("ill_mm_chunk", w.type, _ptr(w.qs), w.rows, w.cols, _ptr(cf.xh), _ptr(cf.xe), _ptr(cf.xd), cf.n, _ptr(y),
              1 if acc else 0, _stream())
    return y


def glu_mul_tc(g, u, act, n, fa, fb):
    """The gate and up products of a gated FFN over a prefill chunk in one launch of the tcgen05 kernel
    (ill_mm_chunk2): FA = G X, FB = U X for the chunk's Q8_K activations ACT.  Both matrices of one format and
    shape, and large enough for tc_takes()."""
    cf = _chunk_f16_of(act, n, g.cols)
    _lib.call("ill_mm_chunk2", g.type, _ptr(g.qs), _ptr(u.qs), g.rows, g.cols, _ptr(cf.xh), _ptr(cf.xe), _ptr(cf.xd), n, _ptr(fa),
              _ptr(fb), _stream())
    return fa, fb


def swiglu_chunk_f16(g, u, cf, clamp=3.0e38):
    """silu(G) * U over a chunk's [n, ff] gate and up products, quantized to Q8_K and left in CF (a ChunkF16 of n x ff)
    in the form the tcgen05 product takes -- the swiglu, quant_q8 and fp16 steps between a prefill chunk's up and
    down products in one launch (ill_swiglu_q8k_f16: each step's arithmetic, bit for bit)."""
    n, ff = cf.n, cf.cols
    if cf.xd is None or cf.xd.numel() != n * ff // 256:
        cf.xd = torch.empty(n * ff // 256, dtype=torch.float32, device=cf.xh.device)
    _lib.call("ill_swiglu_q8k_f16", n, ff, float(clamp), _ptr(g), _ptr(u), 0, _ptr(cf.xh), _ptr(cf.xe), _ptr(cf.xd), 0, _stream())
    return cf


def tc_takes(w, n):
    """Whether cmat_mul sends N tokens of matrix W to the tcgen05 kernel."""
    return ((w.type == 1 or (w.type == 2 and TC_Q6K)) and n >= TC_MIN_TOKENS and w.rows >= TC_MIN_ROWS and w.rows % 4 == 0
            and w.qs.data_ptr() % 16 == 0)


# Matrices of fewer rows that are not K and V beside a larger Q (those: _exact_takes) go to the int8 mma.sync kernel, which is slower there
# (us, tcgen05 / int8, 512 tokens: 1024 x 2560 of Q4_K 14.0 / 21.6, 1024 x 5120 of Q6_K 37.5 / 45.1) but holds a block's sum in int32: in fp32, exact to 2^24, blocks
# of near-constant weights and activations lose bits (relative error against 64 bits, tcgen05 / int8: Q6_K 4.9e-7 / 4.3e-8, Q4_K
# 9.5e-8 / 4.5e-8; ordinary blocks 3.6e-8 both).  It also reads the quants themselves, in any stream and with Y at any float.
# Fewer tokens go there for the same reasons, not for speed: 17 / 63 tokens of 4096 x 2560 of Q4_K 13.2 / 13.6 us on tcgen05 and 19.0 /
# 21.7, of 5120 x 5120 of Q6_K 36.4 / 38.0 and 38.7 / 45.0, and 2 us for the activations' fp16 form once.
TC_MIN_TOKENS, TC_MIN_ROWS = 64, 2048
# Q6_K on the tcgen05 path: scale * (q - 32) reaches 4064 and fp16 holds only even integers above 2048, so the kernel
# multiplies an even part and an odd part of every product (both exact).  False keeps Q6_K chunks on the int8 kernel.
TC_Q6K = True


def _chunk_f16_of(act, n, cols):
    """ACT's fp16 form for the tcgen05 product, made once per quantization of ACT (quant_q8 / rmsnorm_q8 mark it stale)."""
    cf = getattr(act, "_cf", None)
    if cf is None or cf.n != n or cf.cols != cols:
        cf = act._cf = ChunkF16(n, cols, device=act.xq.device)
        act._cf_fresh = False
    if not getattr(act, "_cf_fresh", False):
        cf.fill(act)
        act._cf_fresh = True
    return cf


def swiglu(g, u, out, ff, clamp=3.0e38):
    """OUT = silu(G) * U over whole rows of FF values (the reference's swiglu launch between the gate / up and the
    down products of a prefill chunk, src/cuda-dense.lisp:326-339); CLAMP as d4_swiglu_w clamps, off by default."""
    _lib.call("ill_swiglu_w", g.numel(), ff, float(clamp), _ptr(g), _ptr(u), 0, _ptr(out), _stream())
    return out


OP_MV, OP_GLU = 0, 1


def decode_op(w, x, y, w2=None, norm_w=None, eps=1e-6, bias=None, acc=False, after=True, f16_scale=True):
    """One product of a token's chain for DecodePlan: Y (+)= W X' (+ BIAS), or Y = silu(W X') * (W2 X') when W2 is
    given; X' = X (floats on the device) after RMSNORM! by NORM_W (when given) and the quantizer W's format takes.
    AFTER: the product reads or adds into what an earlier one of the chain writes."""
    import ctypes
    op = _lib.DecodeOp()
    op.w, op.w2, op.x, op.norm_w, op.y, op.bias = _ptr(w.qs), _ptr(w2.qs) if w2 is not None else 0, _ptr(x), _ptr(norm_w), _ptr(y), _ptr(bias)
    op.fmt, op.kind, op.rows, op.cols = w.type, OP_GLU if w2 is not None else OP_MV, w.rows, w.cols
    op.acc, op.after, op.f16_scale, op.eps = int(bool(acc)), int(bool(after)), int(bool(f16_scale)), float(eps)
    if w2 is not None and (w2.type, w2.rows, w2.cols) != (w.type, w.rows, w.cols):
        raise ValueError("a gated product's two matrices must agree in format and shape")
    return op


class _Chain:
    """Recorded launches (ill_chain_new) and the scratch that they go through, given back with the last plan that has them: copies of a
    plan share them, and no other process can have them."""

    def __init__(self, arr, n, device):
        import ctypes
        self.handle = ctypes.c_uint64(0)  # (first: __del__ looks at it whatever fails)
        self.stream = _stream()
        nbytes = _lib.lib().ill_chain_scratch_bytes(arr, n)
        self.scratch = torch.empty(nbytes + 128, dtype=torch.uint8, device=device)
        _lib.call("ill_chain_new", arr, n, (self.scratch.data_ptr() + 127) // 128 * 128, nbytes, ctypes.byref(self.handle))

    def __del__(self):
        if self.handle and _lib is not None:
            _lib.status("ill_chain_free", self.handle)

    def run(self):
        st = _stream()
        _lib.call("ill_chain_run", self.handle, st)
        if st != self.stream:  # the scratch is this stream's too: not given out anew before what runs here is through
            self.scratch.record_stream(torch.cuda.current_stream())

    def __copy__(self):
        return self

    def __deepcopy__(self, memo):
        return self

    def __reduce__(self):
        raise TypeError("a plan's recorded launches belong to this process")


class DecodePlan:
    """A token's chain of products enqueued with one call: what CUDA-FORWARD-N (src/cuda-dense.lisp:380-432) issues as a
    launch per product and per quantization.  OPS: decode_op()s in order.  The plan owns its scratch and the recorded
    launches (ill_chain_new); run() enqueues one token on the current stream, any stream of the device.  It may go while a token is
    on its way, but not before a recording of the caller's that run() went into, nor before the buffers that OPS names."""

    def __init__(self, ops, device="cuda"):
        self.n = len(ops)
        arr = (_lib.DecodeOp * self.n)(*ops)
        if _lib.lib().ill_decode_plan_bytes(self.n) <= 0:
            raise ValueError("a chain holds 1 to 1024 products")
        with torch.cuda.device(device):
            # (what the one-launch form refuses is refused.  The code in an error is that of its entry point.)
            rc = _lib.status("ill_decode_check", arr, self.n)
            if rc:
                _lib.fail("ill_decode_plan", rc)
            self.chain = _Chain(arr, self.n, device)

    def run(self):
        self.chain.run()


def dequant_rows(w, first_row, nrows, out=None):
    """Rows FIRST_ROW.. of W as floats (the bit-exactness check point)."""
    if out is None:
        out = torch.empty(nrows, w.cols, dtype=torch.float32, device=w.qs.device)
    _lib.call("ill_dequant_rows", w.type, _ptr(w.qs), w.cols, 0, first_row, nrows, _ptr(out), _stream())
    return out


def device_status():
    """The device status word (0 = no kernel gave up a wait); synchronises."""
    import ctypes
    v = ctypes.c_uint(0)
    _lib.status("ill_device_status", ctypes.byref(v), _stream())
    return v.value
