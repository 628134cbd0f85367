"""Dense products for a chunk of tokens (CMAT-MUL-N with more than 16 tokens: src/cuda-dense.lisp:220-255) --
the tensor cores' int8 kernel against the one-token product, token by token (the one-token product is what the
other tests hold against the CPU oracle, bit for bit in its integer sums), and against the oracle directly."""
import numpy as np
import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D
from gpu_util import to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(cuda_lib):
    assert torch.cuda.is_available()
    yield
    assert D.device_status() == 0


def _case(fmt, rows, cols, n, seed=0):
    w = D.CMat("w", fmt, rows, cols, B.synth_matrix_torch(fmt, rows, cols, seed=seed))
    x = torch.randn(n * cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed + 1))
    act = D.quant_q8(x, D.make_qact(n * cols, D.matrix_act_kind(w)))
    return w, x, act


@pytest.mark.parametrize("fmt,rows,cols,n", [
    (B.Q4_K, 300, 512, 17), (B.Q4_K, 1000, 2560, 33), (B.Q4_K, 2560, 9728, 100), (B.Q4_K, 9728, 2560, 512),
    (B.Q6_K, 300, 768, 20), (B.Q6_K, 2560, 5120, 64), (B.Q6_K, 1031, 17408, 130), (B.Q6_K, 5120, 5120, 512),
    (B.Q8_0, 300, 896, 17), (B.Q8_0, 4864, 896, 96), (B.Q8_0, 896, 4864, 200), (B.Q8_0, 151936, 896, 40),
    # a few tokens of rows too long to keep their activations beside the weights: the columns dealt to a CTA's warps
    (B.Q6_K, 300, 17408, 4), (B.Q6_K, 1031, 17408, 16), (B.Q4_K, 250, 19456, 9), (B.Q8_0, 300, 17408, 16), (B.Q8_0, 40, 17280, 3),
])
def test_chunk_product_equals_token_by_token(fmt, rows, cols, n):
    w, x, act = _case(fmt, rows, cols, n)
    y = torch.full((n * rows,), -3.0, device="cuda")
    D.cmat_mul(w, act, y, n)
    want = torch.empty(n * rows, device="cuda")
    for t in range(n):   # one token at a time through the matvec kernel
        a1 = D.quant_q8(x[t * cols:(t + 1) * cols], D.make_qact(cols, D.matrix_act_kind(w)))
        D.cmat_mul(w, a1, want[t * rows:(t + 1) * rows], 1)
    torch.cuda.synchronize()
    assert torch.isfinite(y).all()
    # the integer sums are the same; the blocks' float terms are added in a different order (a row whole here,
    # lanes' partial sums in the one-token kernel)
    err = ((y - want).abs().max() / want.abs().max()).item()
    assert err < 2e-6, err


@pytest.mark.parametrize("rows,cols,n,base", [
    (1, 128, 17, 0), (129, 128, 33, 2), (64, 384, 81, 6), (31, 4864, 17, 14), (896, 896, 161, 0), (1000, 4864, 200, 2),
    (300, 640, 385, 10), (2048, 4096, 65, 0), (4864, 896, 777, 8), (5121, 256, 400, 4),
])
def test_q8_0_chunk_tiles(rows, cols, n, base):
    """Q8_0's chunk kernel at the edges of its tiles (32 to 80 tokens, 32 to 128 rows), blocks at even alignments, with a
    bias, adding to Y: against the one-token product."""
    nbytes = B.matrix_bytes(B.Q8_0, rows, cols)
    buf = torch.zeros(nbytes + 32, dtype=torch.uint8, device="cuda")
    buf[base:base + nbytes] = B.synth_matrix_torch(B.Q8_0, rows, cols, seed=rows)
    w = D.CMat("w", B.Q8_0, rows, cols, buf[base:base + nbytes])
    g = torch.Generator(device="cuda").manual_seed(n)
    x, y, bias = (torch.randn(k, device="cuda", generator=g) for k in (n * cols, n * rows, rows))
    want = y.clone()
    D.cmat_mul(w, D.quant_q8(x, D.make_qact(n * cols, "q8")), y, n, bias=bias, acc=True)
    one = torch.empty(rows, device="cuda")
    top = 0.0
    for t in range(n):
        D.cmat_mul(w, D.quant_q8(x[t * cols:(t + 1) * cols], D.make_qact(cols, "q8")), one, 1)
        top = max(top, one.abs().max().item())
        want[t * rows:(t + 1) * rows] += one + bias
    # the same integers; cols / 32 float terms added in another order: a few units of 2^-24 of the largest sum
    assert (y - want).abs().max().item() < 2e-6 * max(top, want.abs().max().item())


@pytest.mark.parametrize("rows,cols,n", [(40, 256, 33), (129, 384, 100), (300, 2048, 161)])
def test_q8_0_chunk_adds_a_rows_blocks_in_order(rows, cols, n):
    """Bit for bit: every block's float(sum) * (d_w * d_x), each step rounded, added in the row's order whatever the tile."""
    w, x, act = _case(B.Q8_0, rows, cols, n)
    y = torch.empty(n * rows, device="cuda")
    D.cmat_mul(w, act, y, n)
    nb = cols // 32
    blk = w.qs[:rows * nb * 34].cpu().numpy().reshape(rows, nb, 34)
    d = blk[:, :, :2].copy().view(np.float16)[:, :, 0].astype(np.float32)
    q = blk[:, :, 2:].copy().view(np.int8).astype(np.int32)
    xq, xs = act.xq.cpu().numpy()[:n * cols].reshape(n, nb, 32).astype(np.int32), act.xs.cpu().numpy()[:n * nb].reshape(n, nb)
    want = np.zeros((n, rows), np.float32)
    for b in range(nb):
        want += (xq[:, b] @ q[:, b].T).astype(np.float32) * (d[None, :, b] * xs[:, b, None])
    assert np.array_equal(y.cpu().numpy().reshape(n, rows).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("fmt", [B.Q8_0, B.Q4_K, B.Q6_K])
def test_chunk_product_against_the_oracle(oracle, fmt):
    rows, cols, n = 200, 1024, 70
    wb = B.synth_matrix(fmt, rows, cols, seed=4)
    w = D.upload_gmat(wb, fmt, rows, cols)
    rng = np.random.default_rng(6)
    xh = rng.standard_normal((n, cols)).astype(np.float32)
    act = D.quant_q8(to_dev(xh.reshape(-1)), D.make_qact(n * cols, D.matrix_act_kind(w)))
    bias = to_dev(rng.standard_normal(rows).astype(np.float32))
    y = torch.zeros(n * rows, device="cuda")
    D.cmat_mul(w, act, y, n, bias=bias)
    torch.cuda.synchronize()
    got = y.cpu().numpy().reshape(n, rows)
    for t in (0, 1, 37, n - 1):
        want = oracle.matvec(fmt, wb, rows, cols, oracle.quantize_act(fmt, xh[t]), bias=bias.cpu().numpy())[0]
        assert np.abs(got[t] - want).max() / np.abs(want).max() < 2e-6
    # added into Y when ACC
    y2 = y.clone()
    D.cmat_mul(w, act, y2, n, acc=True)
    torch.cuda.synchronize()
    assert ((y2 - 2 * y + bias.repeat(n)).abs().max() / y.abs().max()).item() < 1e-5


def test_ffn_head_chunk_against_the_oracle(oracle):
    """DK-FFN-HEAD-CHUNK: RMSNorm, the router's logits and the shared expert over a chunk, token by token against
    the CPU routines (RMSNORM!, F32MV! on the widened router, D4-SHARED!)."""
    from illatio_b200 import cuda_ds4f_prefill as P
    n, d, ff, ne, clamp, eps = 70, 1024, 512, 64, 10.0, 1e-6
    rng = np.random.default_rng(11)
    mats = [B.synth_matrix(B.Q8_0, r, c, seed=20 + i) for i, (r, c) in enumerate(((ff, d), (ff, d), (d, ff)))]
    ws = [D.upload_gmat(m, B.Q8_0, r, c) for m, (r, c) in zip(mats, ((ff, d), (ff, d), (d, ff)))]
    router = torch.as_tensor(rng.standard_normal((ne, d)).astype(np.float32) * 0.05).to(torch.float16)
    cur = rng.standard_normal((n, d)).astype(np.float32)
    nw = (rng.random(d) + 0.5).astype(np.float32)
    hs = P.HeadScratch(n + 3, d, ff, ne)
    norm2, logits, sout = P.dk_ffn_head_chunk(to_dev(cur), to_dev(nw), eps, router.cuda(), ws[0], ws[1], ws[2], clamp, hs)
    torch.cuda.synchronize()
    norm2, logits, sout = norm2.cpu().numpy(), logits.cpu().numpy(), sout.cpu().numpy()
    rf = router.to(torch.float32).numpy()
    for t in (0, 16, 33, n - 1):
        want_n = oracle.rmsnorm(cur[t], nw, eps)
        assert np.abs(norm2[t] - want_n).max() <= 1e-6 * np.abs(want_n).max()
        want_l = oracle.f32mv(rf, norm2[t])
        terms = np.abs(rf.astype(np.float64) * norm2[t].astype(np.float64)).sum(1)
        assert (np.abs(logits[t] - want_l) <= 1e-6 * terms + 1e-30).all()
        want_s = oracle.moe_shared(d, ff, mats[0], mats[1], mats[2], norm2[t], clamp, threads=2)
        assert np.abs(sout[t] - want_s).max() / np.abs(want_s).max() < 2e-3


@pytest.mark.parametrize("fmt,rows,cols,n", [(B.Q4_K, 300, 512, 40), (B.Q4_K, 1000, 2560, 130), (B.Q4_K, 9728, 2560, 512),
                                             (B.Q4_K, 2560, 9728, 200), (B.Q6_K, 300, 768, 40), (B.Q6_K, 1031 - 3, 2560, 130),
                                             (B.Q6_K, 2560, 9728, 512), (B.Q6_K, 5120, 5120, 200)])
def test_chunk_on_tcgen05_equals_token_by_token(fmt, rows, cols, n):
    """The same chunk product through the tcgen05 kernel (the expert product with the matrix as its one expert):
    integer operands exact in fp16 (Q6_K's products as an even and an odd part), fp32 accumulation in tensor memory,
    the blocks scaled as they are drained."""
    w, x, act = _case(fmt, rows, cols, n, seed=3)
    cf = D.ChunkF16(n, cols).fill(act)
    y = torch.full((n * rows,), -3.0, device="cuda")
    D.cmat_mul_tc(w, cf, y)
    want = torch.empty(n * rows, device="cuda")
    one = D.make_qact(cols, "q8k")
    for t in range(n):   # one token at a time through the matvec kernel
        D.cmat_mul(w, D.quant_q8(x[t * cols:(t + 1) * cols], one), want[t * rows:(t + 1) * rows], 1)
    torch.cuda.synchronize()
    assert torch.isfinite(y).all()
    err = ((y - want).abs().max() / want.abs().max()).item()
    assert err < 2e-6, err
    # added into Y when asked; and cmat_mul takes this path by itself for chunks of large matrices
    y2 = y.clone()
    D.cmat_mul_tc(w, cf, y2, acc=True)
    y3 = torch.empty_like(y)
    D.cmat_mul(w, act, y3, n)
    torch.cuda.synchronize()
    assert torch.equal(y2, y + y)
    if rows >= D.TC_MIN_ROWS and n >= D.TC_MIN_TOKENS:
        assert torch.equal(y3, y)


@pytest.mark.parametrize("fmt", [B.Q4_K, B.Q6_K])
def test_chunk_on_tcgen05_against_the_oracle(oracle, fmt):
    rows, cols, n = 200, 1024, 70
    wb = B.synth_matrix(fmt, rows, cols, seed=4)
    w = D.upload_gmat(wb, fmt, rows, cols)
    rng = np.random.default_rng(6)
    xh = rng.standard_normal((n, cols)).astype(np.float32)
    act = D.quant_q8(to_dev(xh.reshape(-1)), D.make_qact(n * cols, "q8k"))
    y = torch.zeros(n * rows, device="cuda")
    D.cmat_mul_tc(w, D.ChunkF16(n, cols).fill(act), y)
    torch.cuda.synchronize()
    got = y.cpu().numpy().reshape(n, rows)
    for t in (0, 1, 37, n - 1):
        want = oracle.matvec(fmt, wb, rows, cols, oracle.quantize_act(fmt, xh[t]))[0]
        assert np.abs(got[t] - want).max() / np.abs(want).max() < 2e-6


def test_fused_swiglu_into_the_down_product():
    """SwiGLU, Q8_K and the fp16 form in one launch (swiglu_chunk_f16) feed the tcgen05 down product with the same
    bits as the three steps apart."""
    n, ff, rows = 130, 2560, 2048
    g = torch.Generator(device="cuda").manual_seed(5)
    ga, ub = torch.randn(n * ff, device="cuda", generator=g), torch.randn(n * ff, device="cuda", generator=g)
    w = D.CMat("down", B.Q6_K, rows, ff, B.synth_matrix_torch(B.Q6_K, rows, ff, seed=2))
    assert D.tc_takes(w, n)
    y1 = torch.zeros(n * rows, device="cuda")
    D.cmat_mul_tc(w, D.swiglu_chunk_f16(ga, ub, D.ChunkF16(n, ff)), y1)
    mid = torch.empty_like(ga)
    D.swiglu(ga, ub, mid, ff)
    y2 = torch.zeros(n * rows, device="cuda")
    D.cmat_mul(w, D.quant_q8(mid, D.make_qact(n * ff, "q8k")), y2, n)
    torch.cuda.synchronize()
    assert torch.isfinite(y1).all() and torch.equal(y1, y2)


def test_vanishing_block_is_quantized_to_zeros(oracle):
    """A Q8_K block whose largest magnitude is below 3.8e-37 (-127 / max overflows: the reference's arithmetic is not
    defined there) is taken as zeros by the device quantizers and by the oracle alike -- and the fused SwiGLU step,
    where such blocks arise (silu of a very negative gate), hands the tcgen05 product finite operands."""
    x = np.zeros(768, np.float32)
    x[256:512] = np.float32(1e-40) * np.arange(1, 257, dtype=np.float32)   # denormals
    x[512:] = np.linspace(-1, 1, 256, dtype=np.float32)
    act = D.quant_q8(to_dev(x), D.make_qact(768, "q8k"))
    torch.cuda.synchronize()
    q, d, bs = oracle.quantize_q8k(x)
    assert np.array_equal(act.xq.cpu().numpy(), q) and np.array_equal(act.xs.cpu().numpy(), d)
    assert np.array_equal(act.xsum.cpu().numpy().astype(np.int32), bs)
    assert d[0] == 0 and d[1] == 0 and d[2] != 0 and not q[:512].any() and q[512:].any()
    # gates of -95 (e^-95 is a denormal) against ups of one: every middle value is a denormal
    n, ff = 64, 512
    g = torch.full((n * ff,), -95.0, device="cuda")
    u = torch.ones(n * ff, device="cuda")
    cf = D.swiglu_chunk_f16(g, u, D.ChunkF16(n, ff))
    torch.cuda.synchronize()
    assert torch.isfinite(cf.xh.float()).all() and (cf.xh == 0).all() and (cf.xd == 0).all()


@pytest.mark.parametrize("fmt", [B.Q4_K, B.Q6_K])
def test_gate_and_up_in_one_launch(fmt):
    """ill_mm_chunk2: two matrices against the same chunk in one launch give what two launches give, bit for bit."""
    rows, cols, n = 2048 + 128, 1024, 200
    wg, x, act = _case(fmt, rows, cols, n, seed=7)
    wu = D.CMat("u", fmt, rows, cols, B.synth_matrix_torch(fmt, rows, cols, seed=8))
    fa, fb = torch.empty(n * rows, device="cuda"), torch.empty(n * rows, device="cuda")
    D.glu_mul_tc(wg, wu, act, n, fa, fb)
    ya, yb = torch.empty_like(fa), torch.empty_like(fb)
    D.cmat_mul(wg, act, ya, n)
    D.cmat_mul(wu, act, yb, n)
    torch.cuda.synchronize()
    assert torch.equal(fa, ya) and torch.equal(fb, yb) and torch.isfinite(fa).all()


def test_quantizers_that_also_leave_the_fp16_forms():
    """Once an activation buffer's fp16 form is in use (a chunk went to the tcgen05 kernel), quant_q8 and rmsnorm_q8
    renew it in their own launch: the same bytes, the same halves as ill_act_f16 makes."""
    n, cols = 96, 2048
    g = torch.Generator(device="cuda").manual_seed(3)
    w = D.CMat("w", B.Q4_K, 2048, cols, B.synth_matrix_torch(B.Q4_K, 2048, cols, seed=1))
    nw = torch.rand(cols, device="cuda", generator=g) + 0.5
    for norm in (False, True):
        act, ref = D.make_qact(n * cols, "q8k"), D.make_qact(n * cols, "q8k")
        y = torch.empty(n * 2048, device="cuda")
        outs = []
        for it in range(2):   # first pass: the fp16 form is made by ill_act_f16; second: by the quantizer itself
            x = torch.randn(n * cols, device="cuda", generator=g)
            if norm:
                D.rmsnorm_q8(x, nw, act, cols, 1e-6, n=n)
                D.rmsnorm_q8(x, nw, ref, cols, 1e-6, n=n)
            else:
                D.quant_q8(x, act)
                D.quant_q8(x, ref)
            assert bool(getattr(act, "_cf_fresh", False)) == (it == 1)
            D.cmat_mul(w, act, y, n)
            fresh = D.ChunkF16(n, cols).fill(ref)     # ref never goes to the tensor-core path: plain quantizer + ill_act_f16
            torch.cuda.synchronize()
            assert torch.equal(act.xq, ref.xq) and torch.equal(act.xs, ref.xs) and torch.equal(act.xsum, ref.xsum)
            assert torch.equal(act._cf.xh, fresh.xh) and torch.equal(act._cf.xe, fresh.xe)
            outs.append(y.clone())
        assert torch.isfinite(outs[1]).all()


@pytest.mark.parametrize("fmt", [B.Q4_K, B.Q6_K])
@pytest.mark.parametrize("rows,cols,n", [(128, 256, 1), (132, 768, 97), (1024, 2560, 513), (384, 2816, 31), (2560, 1024, 130), (19456, 256, 512),
                                         # on 148 SMs Q6_K takes tiles of two jobs here: 144, 176, 256, 256 and 208 rows, the last ones 97, 160, 256, 250 and 153
                                         (5120, 256, 385), (5116, 768, 512), (17408, 256, 512), (18940, 256, 250), (4736, 512, 777)])
def test_chunk_on_tcgen05_tiles(fmt, rows, cols, n):
    """The tcgen05 chunk product at the edges of its tiles (16 to 128 tokens, Q6_K 16 to 256, by the number of tiles a matrix makes),
    with fewer blocks than are in flight and matrices of one tile: against the one-token product, and adding to Y."""
    w, x, act = _case(fmt, rows, cols, n, seed=n)
    cf = D.ChunkF16(n, cols).fill(act)
    y = torch.full((n * rows + 64,), -3.0, device="cuda")
    D.cmat_mul_tc(w, cf, y)
    want = torch.empty(n, rows, device="cuda")
    for t in range(n):
        D.cmat_mul(w, D.quant_q8(x[t * cols:(t + 1) * cols], D.make_qact(cols, "q8k")), want[t], 1)
    top = want.abs().max().item()
    assert (y[:n * rows].view(n, rows) - want).abs().max().item() < 2e-6 * top and (y[n * rows:] == -3.0).all()
    y[:n * rows] = 1.0
    D.cmat_mul_tc(w, cf, y, acc=True)
    assert (y[:n * rows].view(n, rows) - 1.0 - want).abs().max().item() < 2e-6 * max(top, 1.0) + 2.0 ** -23 * (1.0 + top)


@pytest.mark.parametrize("fmt", [B.Q4_K, B.Q6_K])
@pytest.mark.parametrize("rows,cols,n", [(9472, 256, 512), (17408, 512, 512), (2176, 1024, 200), (9468, 256, 257), (132, 256, 3)])
def test_gate_and_up_in_one_launch_tiles(fmt, rows, cols, n):
    """Two matrices against one chunk, in tiles of one and (Q6_K, 9472 and 17408 rows: 256 rows each) of two jobs: the bits of two
    launches, whatever tiles those take, and nothing past the last row."""
    g, x, act = _case(fmt, rows, cols, n, seed=n)
    u = D.CMat("u", fmt, rows, cols, B.synth_matrix_torch(fmt, rows, cols, seed=n + 7))
    fa, fb = (torch.full((n * rows + 64,), -3.0, device="cuda") for _ in range(2))
    D.glu_mul_tc(g, u, act, n, fa, fb)
    cf = D.ChunkF16(n, cols).fill(act)
    for w, y in ((g, fa), (u, fb)):
        want = torch.empty(n * rows, device="cuda")
        D.cmat_mul_tc(w, cf, want)
        assert torch.equal(y[:n * rows], want) and (y[n * rows:] == -3.0).all()


@pytest.mark.parametrize("fmt", [B.Q4_K, B.Q6_K])
@pytest.mark.parametrize("rows", [256, 1024, 2044])
def test_chunk_of_a_small_matrix(fmt, rows):
    """Chunks of 64 tokens through matrices of fewer than 2048 rows (a layer's K and V): block sums past 2^24 are whole numbers
    as in the one-token product, Y may lie at any float, and the quants count as they are when the product is enqueued."""
    cols, n = 256, 64
    g = torch.Generator(device="cuda").manual_seed(rows)
    wb = torch.randint(0, 256, (rows, B.BLOCK_BYTES[fmt]), dtype=torch.uint8, device="cuda", generator=g)
    if fmt == B.Q6_K:   # quants 56 .. 63, scales 112 .. 127: sums up to 6.2 * 2^24
        wb[:, :128] |= 0x88
        wb[:, 128:192] = 0xff
        wb[:, 192:208] = wb[:, 192:208] & 0x0f | 0x70
    else:               # quants 12 .. 15, scales 48 .. 63, no mins: up to 1.6 * 2^24
        wb[:, 4:8] |= 0xf0
        wb[:, 8:12] = 0
        wb[:, 12:16] &= 0x0f
        wb[:, 16:] |= 0xcc
    for off in B.SCALE_OFFSETS[fmt]:
        wb[:, off:off + 2] = (torch.rand(rows, device="cuda", generator=g) + 0.5).to(torch.float16).view(torch.uint8).view(rows, 2)
    w = D.CMat("w", fmt, rows, cols, wb.reshape(-1))
    x = 1.0 + 0.03 * torch.randn(2, n * cols, device="cuda", generator=g).clamp(-2.0, 2.0)
    act, one = D.make_qact(n * cols, "q8k"), D.make_qact(cols, "q8k")
    y, want = torch.empty(n * rows + 1, device="cuda")[1:], torch.empty(n * rows, device="cuda")
    for i in range(2):  # the second time the quants are written by the library's own entry point
        _lib.call("ill_quant_q8_k", x[i].data_ptr(), act.xq.data_ptr(), act.xs.data_ptr(), act.xsum.data_ptr(), n, _lib.stream())
        D.cmat_mul(w, act, y, n)
        for t in range(n):
            D.cmat_mul(w, D.quant_q8(x[i, t * cols:(t + 1) * cols], one), want[t * rows:(t + 1) * rows], 1)
        # one block a row: the same whole number, rounded to the same float, times two scales -- two roundings of 2^-24 on either side
        assert ((y - want).abs() <= 4.00001 * 2.0 ** -24 * want.abs()).all()
        # the tcgen05 kernel, which larger matrices take, adds in fp32: 16 columns at a time, Q6_K's even and odd parts apart, each addition
        # cut off at 2^-23 of the sum (measured: 1.1e-6 and 3.6e-7 in all)
        yt = torch.empty(n * rows, device="cuda")
        D.cmat_mul_tc(w, D.ChunkF16(n, cols).fill(act), yt)
        assert ((yt - want).abs() <= ((32 if fmt == B.Q6_K else 16) + 2) * 2.0 ** -23 * want.abs()).all()
