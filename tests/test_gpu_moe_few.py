"""The experts' products for a few rows an expert (ill_moe_few, ill_moe_few2, ill_moe_few_glu): the bits of the chunk product, experts of
more rows left to it (ill_moe_mm_id_over)."""
import numpy as np
import pytest
import torch

from illatio_b200 import _lib
from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D
from illatio_b200 import cuda_ds4f as M
from illatio_b200 import cuda_ds4f_prefill as P

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(cuda_lib):
    yield
    assert D.device_status() == 0


def _p(t):
    return t.data_ptr()


@pytest.mark.parametrize("fmt,base", [(B.IQ2_XXS, 0), (B.IQ2_XXS, 2), (B.Q2_K, 4)])
@pytest.mark.parametrize("rows,cols", [(200, 768), (18, 256), (260, 2304), (64, 9216 - 512)])
@pytest.mark.parametrize("counts", [(0, 1, 8, 9, 3, 0, 16), (17, 15, 16, 2000, 1), (16,), (0, 0, 5)])
def test_few_rows_have_the_chunk_products_bits(fmt, base, rows, cols, counts):
    """At the edges of a tile of eight and of the sixteen rows an expert may have, rows that are no multiple of sixteen, one block, an odd
    number of them, and so many that eight tokens fit only; rows read through a map; nothing written past a row's end."""
    ne, n = len(counts), sum(counts)
    most = _lib.lib().ill_moe_few_most(fmt, cols)
    assert most == (8 if fmt == B.IQ2_XXS and cols > 8192 else 16)
    nbytes = B.matrix_bytes(fmt, rows, cols)
    step = (2 * nbytes + 64) // 16 * 16
    buf = torch.zeros(ne * step + 32, dtype=torch.uint8, device="cuda")
    for e in range(ne):
        buf[base + e * step:base + e * step + 2 * nbytes] = B.synth_matrix_torch(fmt, 2 * rows, cols, seed=e + rows)
    g = torch.Generator(device="cuda").manual_seed(n + cols)
    tokens = n // 2 + 1
    act = D.quant_q8(torch.randn(tokens * cols, device="cuda", generator=g), D.make_qact(tokens * cols, "q8k"))
    tmap = torch.randint(0, tokens, (n,), dtype=torch.int32, device="cuda", generator=g)
    xh = torch.empty(n, cols, dtype=torch.float16, device="cuda")
    xe = torch.empty(n, cols // 256, 64, dtype=torch.float16, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    ptrs = torch.tensor([_p(buf) + base + e * step for e in range(ne)], dtype=torch.int64, device="cuda")
    cnt, bases = torch.tensor(counts, **i32), torch.tensor([sum(counts[:e]) for e in range(ne)], **i32)
    who = (_p(ptrs), _p(cnt), _p(bases), ne, n)
    stride = (rows + 3) // 4 * 4 + 4
    _lib.call("ill_act_f16", n, cols, _p(act.xq), _p(act.xsum), _p(tmap), _p(xh), _p(xe), _lib.stream())
    want = [torch.full((n, stride), 5.0, device="cuda") for _ in range(2)]
    _lib.call("ill_moe_mm_id2", fmt, cols, rows, 0, nbytes, *who, _p(xh), _p(xe), _p(act.xs), _p(tmap), _p(want[0]), _p(want[1]), stride, _lib.stream())
    few = torch.repeat_interleave(cnt <= most, cnt.long())[:, None]
    x = (_p(act.xq), _p(act.xs), _p(act.xsum), _p(tmap))
    one, two = torch.full((n, stride), 5.0, device="cuda"), [torch.full((n, stride), 5.0, device="cuda") for _ in range(2)]
    _lib.call("ill_moe_few", fmt, cols, rows, nbytes, *who, *x, _p(one), stride, _lib.stream())
    _lib.call("ill_moe_few2", fmt, cols, rows, 0, nbytes, *who, *x, _p(two[0]), _p(two[1]), stride, _lib.stream())
    assert torch.equal(one, torch.where(few, want[1], 5.0))
    for a, b in zip(two, want):
        assert torch.equal(a, torch.where(few, b, 5.0))
    w = torch.rand(n, device="cuda", generator=g)
    mid, ref = torch.full((n, stride), 5.0, device="cuda"), torch.empty(n, rows, device="cuda")
    _lib.call("ill_moe_few_glu", fmt, cols, rows, 0, nbytes, *who, *x, 1.5, _p(w), _p(mid), stride, _lib.stream())
    if n:
        a, b = (t[:, :rows].contiguous() for t in want)
        _lib.call("ill_swiglu_w", n * rows, rows, 1.5, _p(a), _p(b), _p(w), _p(ref), _lib.stream())
    assert torch.equal(mid[:, :rows], torch.where(few, ref, 5.0)) and (mid[:, rows:] == 5.0).all()
    # the experts that are left: the operands first as ill_act_f16_over has them, over what was there
    any_over = max(counts) > most
    xh2, xe2 = torch.zeros_like(xh), torch.zeros_like(xe)
    _lib.call("ill_act_f16_over", n, cols, _p(act.xq), _p(act.xsum), _p(tmap), _p(xh2), _p(xe2), _p(cnt), ne, most, _lib.stream())
    assert torch.equal(xh2, xh if any_over else torch.zeros_like(xh)) and (not any_over or torch.equal(xe2, xe))
    _lib.call("ill_moe_mm_id_over", fmt, cols, rows, 0, nbytes, *who, _p(xh2), _p(xe2), _p(act.xs), _p(tmap), _p(two[0]), _p(two[1]), stride, most,
              _lib.stream())
    assert torch.equal(two[0], want[0]) and torch.equal(two[1], want[1])


def test_counts_that_are_not_the_routers_stay_inside_the_buffers():
    """Numbers of rows past the last row there is, and negative ones: such an expert is left out, or its rows that are there."""
    fmt, rows, cols, n = B.Q2_K, 48, 512, 10
    w = B.synth_matrix_torch(fmt, rows, cols, seed=1)
    act = D.quant_q8(torch.randn(n * cols, device="cuda"), D.make_qact(n * cols, "q8k"))
    i32 = dict(dtype=torch.int32, device="cuda")
    ptrs = torch.full((4,), _p(w), dtype=torch.int64, device="cuda")
    cnt, bases = torch.tensor([4, -3, 9, 16], **i32), torch.tensor([0, 4, 8, 2 ** 31 - 1], **i32)
    y = torch.full((n + 16, rows), 5.0, device="cuda")
    _lib.call("ill_moe_few", fmt, cols, rows, 0, _p(ptrs), _p(cnt), _p(bases), 4, n, _p(act.xq), _p(act.xs), _p(act.xsum), 0, _p(y), rows, _lib.stream())
    assert (y[4:] == 5.0).all() and (y[:4] != 5.0).any(1).all()


@pytest.mark.parametrize("n,gate", [(16, B.IQ2_XXS), (17, B.Q2_K), (90, B.IQ2_XXS), (90, B.Q2_K)])
def test_chunk_driver_with_and_without(n, gate):
    """The chunk driver with its experts of a few rows apart and with all of them on the chunk product: the same bits.  Twelve experts of
    which one is chosen by every token."""
    d, ff, ne, nu = 512, 256, 12, 3
    pool = M.make_expert_pool(B.synth_matrix(gate, ne * ff, d, seed=1), B.synth_matrix(gate, ne * ff, d, seed=2),
                              B.synth_matrix(B.Q2_K, ne * d, ff, seed=3), d, ff, ne, gate_fmt=gate)
    g = torch.Generator(device="cuda").manual_seed(n)
    norms, logits = torch.randn(n, d, device="cuda", generator=g), torch.randn(n, ne, device="cuda", generator=g)
    logits[:, 4] += 30.0
    sc = P.make_chunk_scratch(pool, n, nu)
    assert P.few_rows(pool, n, nu) == 16
    got = P.dk_ffn_routed_chunk(pool, norms, logits, nu, 10.0, sc).clone()
    if n > 16:
        assert sc.counts.max() > 16 and sc.counts.min() <= 16
    want = P.dk_ffn_routed_chunk(pool, norms, logits, nu, 10.0, sc, fused=False)
    assert torch.equal(got, want)


@pytest.mark.parametrize("n,d", [(4, 512), (16, 512), (4, 7168)])
@pytest.mark.parametrize("masked", [False, True])
def test_a_router_that_gives_a_token_one_expert_again(n, d, masked):
    """Scores that are NaN, or -inf by a mask that leaves fewer than NU experts: the router takes expert 0 for each of the slots that are
    left, which then has more rows than a launch for a few takes at a time.  The other tokens' rows are theirs, bit for bit, and none
    is what the scratch held before.  (7168 columns of IQ2_XXS: eight rows at a time.)"""
    ff, ne, nu = 256, 12, 8
    pool = M.make_expert_pool(B.synth_matrix(B.IQ2_XXS, ne * ff, d, seed=1), B.synth_matrix(B.IQ2_XXS, ne * ff, d, seed=2),
                              B.synth_matrix(B.Q2_K, ne * d, ff, seed=3), d, ff, ne, gate_fmt=B.IQ2_XXS)
    g = torch.Generator(device="cuda").manual_seed(n)
    norms, logits = torch.randn(n, d, device="cuda", generator=g), torch.randn(n, ne, device="cuda", generator=g)
    healthy, bias = torch.ones(n, dtype=torch.bool, device="cuda"), None
    if masked:
        bias = torch.full((ne,), float("-inf"), device="cuda")
        bias[[2, 5, 7]] = 0.0
    else:
        logits[:, 0] += 30.0     # the healthy ones choose expert 0 too
        logits[1] = logits[n - 1] = float("nan")
        healthy[1] = healthy[n - 1] = False
    sc = P.make_chunk_scratch(pool, n, nu)
    most = P.few_rows(pool, n, nu)
    assert most == (16 if d == 512 else 8)
    want = P.dk_ffn_routed_chunk(pool, norms, logits, nu, 10.0, sc, bias=bias, fused=False).clone()
    assert int(sc.counts[0]) > most
    for t in (sc.mid, sc.down, sc.g, sc.u, sc.moe):
        t.fill_(1e30)
    got = P.dk_ffn_routed_chunk(pool, norms, logits, nu, 10.0, sc, bias=bias)
    assert torch.isfinite(want[healthy]).all() and torch.equal(got[healthy], want[healthy])


@pytest.mark.parametrize("fmt,cols", [(B.IQ2_XXS, 512), (B.Q2_K, 768), (B.Q2_K, 9216)])
@pytest.mark.parametrize("counts", [(17, 0, 16, 33, 1), (40,), (0, 8, 9, 64, 0, 25)])
def test_all_experts_in_passes(fmt, cols, counts):
    """ill_moe_few_all and ill_moe_few_glu_all: experts of more rows than a pass has (16; 8 of 9216 columns), at the edges of a pass and
    beside experts of few and of none: the chunk product's bits."""
    rows, ne, n = 200, len(counts), sum(counts)
    nbytes = B.matrix_bytes(fmt, rows, cols)
    step = (2 * nbytes + 15) // 16 * 16
    buf = torch.zeros(ne * step, dtype=torch.uint8, device="cuda")
    for e in range(ne):
        buf[e * step:e * step + 2 * nbytes] = B.synth_matrix_torch(fmt, 2 * rows, cols, seed=e + rows)
    g = torch.Generator(device="cuda").manual_seed(n + cols)
    act = D.quant_q8(torch.randn(n * cols, device="cuda", generator=g), D.make_qact(n * cols, "q8k"))
    tmap = torch.randint(0, n, (n,), dtype=torch.int32, device="cuda", generator=g)
    xh, xe = torch.empty(n, cols, dtype=torch.float16, device="cuda"), torch.empty(n, cols // 256, 64, dtype=torch.float16, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    ptrs = torch.tensor([_p(buf) + e * step for e in range(ne)], dtype=torch.int64, device="cuda")
    cnt, bases = torch.tensor(counts, **i32), torch.tensor([sum(counts[:e]) for e in range(ne)], **i32)
    who, x = (_p(ptrs), _p(cnt), _p(bases), ne, n), (_p(act.xq), _p(act.xs), _p(act.xsum), _p(tmap))
    _lib.call("ill_act_f16", n, cols, x[0], x[2], _p(tmap), _p(xh), _p(xe), _lib.stream())
    want = [torch.empty(n, rows, device="cuda") for _ in range(2)]
    _lib.call("ill_moe_mm_id2", fmt, cols, rows, 0, nbytes, *who, _p(xh), _p(xe), x[1], _p(tmap), _p(want[0]), _p(want[1]), rows, _lib.stream())
    w = torch.rand(n, device="cuda", generator=g)
    got, mid, ref = (torch.full((n, rows), 5.0, device="cuda") for _ in range(3))
    _lib.call("ill_moe_few_all", fmt, cols, rows, nbytes, *who, *x, _p(got), rows, _lib.stream())
    _lib.call("ill_moe_few_glu_all", fmt, cols, rows, 0, nbytes, *who, *x, 1.5, _p(w), _p(mid), rows, _lib.stream())
    _lib.call("ill_swiglu_w", n * rows, rows, 1.5, _p(want[0]), _p(want[1]), _p(w), _p(ref), _lib.stream())
    assert torch.equal(got, want[1]) and torch.equal(mid, ref)


def test_counts_past_the_rows_there_are_in_passes():
    """Counts that add up to more rows than there are (experts that share rows): each expert's results, in some order, and nothing else."""
    fmt, rows, cols, n, ne = B.Q2_K, 48, 512, 40, 3
    w = B.synth_matrix_torch(fmt, rows, cols, seed=1)
    act = D.quant_q8(torch.randn(n * cols, device="cuda"), D.make_qact(n * cols, "q8k"))
    i32 = dict(dtype=torch.int32, device="cuda")
    ptrs = torch.full((ne,), _p(w), dtype=torch.int64, device="cuda")
    cnt, bases = torch.tensor([40, 40, 41], **i32), torch.zeros(ne, **i32)
    y, one = torch.full((n + 16, rows), 5.0, device="cuda"), torch.empty(n, rows, device="cuda")
    _lib.call("ill_moe_few_all", fmt, cols, rows, 0, _p(ptrs), _p(cnt), _p(bases), ne, n, _p(act.xq), _p(act.xs), _p(act.xsum), 0, _p(y), rows, _lib.stream())
    eight = torch.tensor([8], **i32)
    for t in range(0, n, 8):
        _lib.call("ill_moe_few", fmt, cols, rows, 0, _p(ptrs), _p(eight), _p(bases), 1, 8, _p(act.xq) + t * cols, _p(act.xs) + 4 * t * (cols // 256),
                  _p(act.xsum) + 2 * t * (cols // 16), 0, _p(one) + 4 * t * rows, rows, _lib.stream())
    assert torch.equal(y[:n], one) and (y[n:] == 5.0).all()


def test_chunk_driver_with_limits_that_differ():
    """Eight rows of 7168 columns of IQ2_XXS for gate and up, sixteen for down: experts between them, and of fewer and more."""
    d, ff, ne, nu, n = 7168, 256, 12, 3, 40
    pool = M.make_expert_pool(B.synth_matrix(B.IQ2_XXS, ne * ff, d, seed=1), B.synth_matrix(B.IQ2_XXS, ne * ff, d, seed=2),
                              B.synth_matrix(B.Q2_K, ne * d, ff, seed=3), d, ff, ne, gate_fmt=B.IQ2_XXS)
    g = torch.Generator(device="cuda").manual_seed(n)
    norms, logits = torch.randn(n, d, device="cuda", generator=g), torch.randn(n, ne, device="cuda", generator=g)
    logits[:, 4] += 30.0
    sc = P.make_chunk_scratch(pool, n, nu)
    want = P.dk_ffn_routed_chunk(pool, norms, logits, nu, 10.0, sc, fused=False).clone()
    c = sc.counts
    assert ((c > 8) & (c <= 16)).any() and (c > 16).any() and (c <= 8).any()
    for t in (sc.down, sc.g, sc.u, sc.moe):
        t.fill_(1e30)
    assert torch.equal(P.dk_ffn_routed_chunk(pool, norms, logits, nu, 10.0, sc), want)


def test_block_sums_past_24_bits(oracle):
    """IQ2_XXS's block sums reach 2.6 times 2^24: whole numbers of 32 bits here, each sum rounded once (three roundings a block: the sum, the
    product of the scales, theirs), where the chunk product adds in fp32.  One block a row of the largest scale and codebook entry."""
    fmt, rows, cols, n = B.IQ2_XXS, 32, 256, 5
    rng = np.random.default_rng(1)
    base = B.synth_matrix(fmt, 256, cols, seed=1).reshape(256, 66).copy()
    base[:, :2] = np.frombuffer(np.float16(1.0).tobytes(), np.uint8)
    base[:, 2:].reshape(256, 8, 8)[:, :, 4:] = np.frombuffer(np.uint32(0xf0000000).tobytes(), np.uint8)  # no signs, the scale 31
    base[:, 2:].reshape(256, 8, 8)[:, :, :4] = np.arange(256, dtype=np.uint8)[:, None, None]
    sums = oracle.dequant(fmt, base.reshape(-1), 256, cols).astype(np.float64).sum(1)
    block = base[sums.argmax()].copy()
    w = np.repeat(block[None], rows, 0)
    w[:, 2:].reshape(rows, 8, 8)[:, :, 4] ^= rng.integers(0, 4, (rows, 8), dtype=np.uint8)  # some signs
    wf = oracle.dequant(fmt, w.reshape(-1), rows, cols).astype(np.float64)
    act = D.quant_q8(torch.full((n * cols,), 0.7, device="cuda") * (1 + torch.rand(n * cols, device="cuda") / 64), D.make_qact(n * cols, "q8k"))
    q, d = act.xq.cpu().numpy().astype(np.float64).reshape(n, cols), act.xs.cpu().numpy().astype(np.float64)
    want = (q @ wf.T) * d[:, None]
    assert np.abs(q @ wf.T).max() * 8 > 2 ** 24
    i32 = dict(dtype=torch.int32, device="cuda")
    dw = torch.as_tensor(w.reshape(-1)).cuda()
    ptrs, cnt, bases = torch.tensor([_p(dw)], dtype=torch.int64, device="cuda"), torch.tensor([n], **i32), torch.tensor([0], **i32)
    who = (_p(ptrs), _p(cnt), _p(bases), 1, n)
    y, chunk = torch.empty(n, rows, device="cuda"), torch.empty(n, rows, device="cuda")
    xh = torch.empty(n, cols, dtype=torch.float16, device="cuda")
    _lib.call("ill_moe_few", fmt, cols, rows, 0, *who, _p(act.xq), _p(act.xs), _p(act.xsum), 0, _p(y), rows, _lib.stream())
    _lib.call("ill_act_f16", n, cols, _p(act.xq), _p(act.xsum), 0, _p(xh), 0, _lib.stream())
    _lib.call("ill_moe_mm_id", fmt, cols, rows, 0, *who, _p(xh), 0, _p(act.xs), 0, 0, _p(chunk), rows, _lib.stream())
    err, err_chunk = (np.abs(t.cpu().numpy() - want).max() / np.abs(want).max() for t in (y, chunk))
    assert err <= 3 * 2.0 ** -24, err
    assert err <= err_chunk <= (3 + 16 * 2) * 2.0 ** -24, err_chunk  # sixteen additions of 16 columns, each off by up to 2 past 2^24
