"""The work a user has this framework do, as cases that can be timed: decoded tokens, small batches and prefill chunks
through the dense products of a model, one product in every format, and a mixture-of-experts layer for one token, a
few sequences and a chunk.

Attention and the other steps between the products are not part of the framework: an attention output is an input here,
the queries, keys and values are outputs.  Weights are seeded random blocks scaled as a trained model's are (a row's
product with unit-variance activations has a variance near one), so the residual stream and the middle values keep the
magnitudes that they have in use.
"""
import math

import numpy as np
import torch

from illatio_b200 import blocks as B
from illatio_b200 import cuda_dense as D
from illatio_b200 import cuda_ds4f as M
from illatio_b200 import cuda_ds4f_prefill as P

EPS = 1e-6
CLAMP = 10.0
FMT = B.BY_NAME

# hidden size, rows of Q, rows of K and of V, FFN width, vocabulary; the format of the products, and that of V, the down
# product and the output head (which is the embedding too); whether Q, K and V have biases
MODELS = {
    "qwen2_0.5b_q8_0": (896, 896, 128, 4864, 151936, "q8_0", "q8_0", True),
    "qwen3_4b_q4_k_m": (2560, 4096, 1024, 9728, 151936, "q4_k", "q6_k", False),
    "qwen3.5_27b_q6_k": (5120, 5120, 1024, 17408, 151936, "q6_k", "q6_k", False),
}
LAYERS = {"qwen2_0.5b_q8_0": 24, "qwen3_4b_q4_k_m": 36, "qwen3.5_27b_q6_k": 8}

# hidden size, expert FFN width, experts, experts a token, format of gate and up (down is Q2_K), Zipf exponent of the
# experts' popularity
MOES = {
    "ds4_flash": (4096, 2048, 256, 6, "iq2_xxs", 0.0),
    "glm": (5120, 1536, 288, 8, "q2_k", 1.1),
}


def listed():
    return [
        # one token of a small model, every product launched by itself: latency and launches count
        dict(name="token_0.5b_q8_0", path="token", model="qwen2_0.5b_q8_0", layers=24, n=1, graph=False),
        # one token of the usual mixed-format file, the token kept as a CUDA graph as a serving loop keeps it
        dict(name="token_4b_q4_k_m_graph", path="token", model="qwen3_4b_q4_k_m", layers=36, n=1, graph=True),
        # the same token through the framework's own plan of a token (one launch)
        dict(name="plan_4b_q4_k_m", path="plan", model="qwen3_4b_q4_k_m", layers=36),
        # four and sixteen sequences decoded together: a large model's layers (an eighth of them), and a whole 4B one
        dict(name="batch4_27b_q6_k", path="token", model="qwen3.5_27b_q6_k", layers=8, n=4, graph=False),
        dict(name="batch16_4b_q4_k_m", path="token", model="qwen3_4b_q4_k_m", layers=36, n=16, graph=False),
        # prompts: the usual chunk of a 4B model, and a ragged one of a small model
        dict(name="prefill512_4b_q4_k_m", path="prefill", model="qwen3_4b_q4_k_m", layers=36, n=512),
        dict(name="prefill777_0.5b_q8_0", path="prefill", model="qwen2_0.5b_q8_0", layers=24, n=777),
        # one matrix of an output head's size in each of the formats, one token
        dict(name="matvec_5_formats", path="matvec", formats="q8_0,q4_k,q6_k,q2_k,iq2_xxs", rows=151936, cols=2560, n=1),
        # a mixture-of-experts layer: one decoded token, 64 sequences with skewed experts, and a prompt's chunk each
        dict(name="moe_token_iq2_xxs", path="moe", moe="ds4_flash", n=1),
        dict(name="moe_batch64_q2_k", path="moe", moe="glm", n=64),
        dict(name="moe_prefill4096_iq2_xxs", path="moe", moe="ds4_flash", n=4096),
        dict(name="moe_prefill8192_q2_k", path="moe", moe="glm", n=8192),
    ]


def _log(rng, lo, hi):
    """A whole number from LO to HI, even over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(["token", "token", "plan", "prefill", "prefill", "matvec", "matvec", "moe", "moe", "moe"])
    model = rng.choice(sorted(MODELS))
    if path == "token":
        return dict(path=path, model=model, layers=rng.randint(1, LAYERS[model]), n=_log(rng, 1, 16), graph=rng.random() < 0.5)
    if path == "plan":
        return dict(path=path, model=rng.choice(["qwen2_0.5b_q8_0", "qwen3_4b_q4_k_m"]), layers=rng.randint(1, 24))
    if path == "prefill":
        n = _log(rng, 17, 2048)
        hidden, q, kv, ffn = MODELS[model][:4]
        most = int(3.5e12 / (2.0 * n * (hidden * (2 * q + 2 * kv) + 3 * hidden * ffn)))
        return dict(path=path, model=model, layers=rng.randint(1, max(1, min(LAYERS[model], most))), n=n)
    if path == "matvec":
        fmts = sorted(FMT)
        names = ",".join(sorted(rng.sample(fmts, rng.randint(1, len(fmts)))))
        cols = 256 * _log(rng, 2, 68)
        return dict(path=path, formats=names, rows=_log(rng, 512, min(151936, 151936 * 5120 // cols)), cols=cols,
                    n=rng.choice([1, 1, 1, _log(rng, 2, 16)]))
    return dict(path=path, moe=rng.choice(sorted(MOES)), n=_log(rng, 1, 4096))


# ---------------------------------------------------------------- inputs

# root mean square of a random block's weights, for a scale of one (SCALE_OFFSETS' first field drawn from |N(0, 1)|)
_RMS = {B.Q8_0: 73.3, B.Q4_K: 380.0, B.Q6_K: 1367.0, B.Q2_K: 20.0, B.IQ2_XXS: 64.0}
# the second scale field over the first, so that the mins centre the weights as they do in a quantized model
_MIN = {B.Q4_K: 7.5, B.Q2_K: 1.5}


def _blocks(fmt, rows, cols, g, gain=1.0):
    """Raw blocks of a rows x cols matrix whose weights have a root mean square of GAIN / sqrt(cols)."""
    nb = rows * (cols // B.BLOCK_WEIGHTS[fmt])
    blk = torch.randint(0, 256, (nb, B.BLOCK_BYTES[fmt]), dtype=torch.uint8, device="cuda", generator=g)
    if fmt == B.Q8_0:
        blk[:, 2:34] = torch.randint(-127, 128, (nb, 32), dtype=torch.int8, device="cuda", generator=g).view(torch.uint8)
    sigma = gain / math.sqrt(cols) / _RMS[fmt]
    for i, off in enumerate(B.SCALE_OFFSETS[fmt]):
        d = torch.randn(nb, device="cuda", generator=g).abs() * (sigma * (_MIN[fmt] if i else 1.0))
        blk[:, off:off + 2] = d.to(torch.float16).view(torch.uint8).reshape(nb, 2)
    return blk.reshape(-1)


def _mat(fmt, rows, cols, g, gain=1.0):
    return D.upload_gmat(_blocks(fmt, rows, cols, g, gain), fmt, rows, cols)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _f32(*shape):
    return torch.empty(*shape, dtype=torch.float32, device="cuda")


class Dense:
    """A model's weights and the buffers that a program keeps for N tokens at a time."""

    def __init__(self, case, g, n):
        hidden, qd, kv, ffn, vocab, main, alt, bias = MODELS[case["model"]]
        main, alt, nl = FMT[main], FMT[alt], case["layers"]
        self.hidden, self.ffn, self.n = hidden, ffn, n
        self.layers = []
        for _ in range(nl):
            # the products that add to the residual stream are scaled down, as trained ones are
            L = dict(q=_mat(main, qd, hidden, g), k=_mat(main, kv, hidden, g), v=_mat(alt, kv, hidden, g), o=_mat(main, hidden, qd, g, 0.25),
                     gate=_mat(main, ffn, hidden, g), up=_mat(main, ffn, hidden, g), down=_mat(alt, hidden, ffn, g, 0.25))
            L["nw1"], L["nw2"] = (torch.rand(hidden, device="cuda", generator=g) + 0.5 for _ in range(2))
            L["bq"], L["bk"], L["bv"] = ((torch.randn(r, device="cuda", generator=g) * 0.1 if bias else None) for r in (qd, kv, kv))
            self.layers.append(L)
        self.head = _mat(alt, vocab, hidden, g)
        self.nwf = torch.rand(hidden, device="cuda", generator=g) + 0.5
        self.tokens = torch.randint(0, vocab, (n,), dtype=torch.int32, device="cuda", generator=g)
        self.att = torch.randn(n * qd, device="cuda", generator=g)
        self.h, self.q = _f32(n * hidden), _f32(n * qd)
        self.k, self.v = _f32(nl, n * kv), _f32(nl, n * kv)
        self.fa, self.fb = _f32(n * ffn), _f32(n * ffn)
        kind = D.matrix_act_kind(self.head)
        self.act_h, self.act_q, self.act_f = (D.make_qact(n * w, kind) for w in (hidden, qd, ffn))
        self.act_last = D.make_qact(hidden, kind)


def _qkv_o(s, L, i):
    """The products around a layer's attention."""
    a = D.rmsnorm_q8(s.h, L["nw1"], s.act_h, s.hidden, EPS, n=s.n)
    D.qkv_mul(L["q"], L["k"], L["v"], a, s.q, s.k[i], s.v[i], bq=L["bq"], bk=L["bk"], bv=L["bv"], n=s.n)
    D.cmat_mul(L["o"], D.quant_q8(s.att, s.act_q), s.h, s.n, acc=True)


def _token(s):
    """One token of each of N sequences: embedding, every layer, the output head."""
    D.embed(s.head, s.tokens, s.h)
    for i, L in enumerate(s.layers):
        _qkv_o(s, L, i)
        a = D.rmsnorm_q8(s.h, L["nw2"], s.act_h, s.hidden, EPS, n=s.n)
        D.glu_mul(L["gate"], L["up"], a, s.fa, s.n, fb=s.fb)
        D.cmat_mul(L["down"], D.quant_q8(s.fa, s.act_f), s.h, s.n, acc=True)
    D.cmat_mul(s.head, D.rmsnorm_q8(s.h, s.nwf, s.act_h, s.hidden, EPS, n=s.n), s.logits, s.n)


def _prefill(s):
    """A prompt's chunk: embedding, every layer, the output head for the last token."""
    D.embed(s.head, s.tokens, s.h)
    for i, L in enumerate(s.layers):
        _qkv_o(s, L, i)
        a = D.rmsnorm_q8(s.h, L["nw2"], s.act_h, s.hidden, EPS, n=s.n)
        if s.mid is not None:
            D.glu_mul_tc(L["gate"], L["up"], a, s.n, s.fa, s.fb)
            D.cmat_mul_tc(L["down"], D.swiglu_chunk_f16(s.fa, s.fb, s.mid), s.h, acc=True)
        else:
            D.cmat_mul(L["gate"], a, s.fa, s.n)
            D.cmat_mul(L["up"], a, s.fb, s.n)
            D.swiglu(s.fa, s.fb, s.fa, s.ffn)
            D.cmat_mul(L["down"], D.quant_q8(s.fa, s.act_f), s.h, s.n, acc=True)
    D.cmat_mul(s.head, D.rmsnorm_q8(s.h[(s.n - 1) * s.hidden:], s.nwf, s.act_last, s.hidden, EPS), s.logits, 1)


def _plan(s):
    D.embed(s.head, s.tokens, s.h)
    s.plan.run()


class Moe:
    """A mixture-of-experts layer with a shared expert, and the buffers for N tokens."""

    def __init__(self, case, g):
        d, ff, ne, nu, gate, zipf = MOES[case["moe"]]
        n, gate = case["n"], FMT[gate]
        self.n, self.d, self.ff, self.nu = n, d, ff, nu
        self.pool = M.make_expert_pool(_blocks(gate, ne * ff, d, g), _blocks(gate, ne * ff, d, g), _blocks(B.Q2_K, ne * d, ff, g), d, ff, ne,
                                       gate_fmt=gate)
        self.router = (torch.randn(ne, d, device="cuda", generator=g) / math.sqrt(d)).to(torch.float16)
        self.bias = torch.from_numpy(_popularity(ne, zipf)).cuda() if zipf else None
        self.shared = [_mat(B.Q8_0, r, c, g) for r, c in ((ff, d), (ff, d), (d, ff))]
        self.nw = torch.rand(d, device="cuda", generator=g) + 0.5
        self.cur = torch.randn(n, d, device="cuda", generator=g)
        if n > 1:
            self.hs = P.HeadScratch(n, d, ff, ne)
            self.sc = P.make_chunk_scratch(self.pool, n, nu)
        else:
            self.norm2, self.logits, self.sout, self.moe = _f32(d), _f32(1, ne), _f32(d), _f32(d)
            self.act = D.make_qact(d, "q8")


def _popularity(ne, zipf):
    """What a router adds to its scores to choose expert e about as often as 1 / (e + 1)^ZIPF."""
    p = 1.0 / np.arange(1, ne + 1) ** zipf
    return (0.06 * (np.log(p) - np.log(p).mean())).astype(np.float32)


def _moe_token(s):
    D.rmsnorm_q8(s.cur, s.nw, s.act, s.d, EPS, h=s.norm2, f16_scale=False)
    M.dk_mv16(s.router, s.norm2, s.logits)
    sel, w = M.route(s.logits, s.nu, bias=s.bias)
    M.dk_shared(*s.shared, s.norm2, CLAMP, s.sout)
    M.dk_ffn_tail(s.pool, s.norm2, sel[0], w[0], CLAMP, shared=s.sout, moe=s.moe)
    return {"moe": s.moe, "logits": s.logits}


def _moe_chunk(s):
    norms, logits, shared = P.dk_ffn_head_chunk(s.cur, s.nw, EPS, s.router, *s.shared, CLAMP, s.hs)
    ffn = P.dk_ffn_small if s.n <= 64 else P.dk_ffn_routed_chunk
    return {"moe": ffn(s.pool, norms, logits, s.nu, CLAMP, s.sc, bias=s.bias, shared=shared), "logits": logits}


def prepare(case, seed):
    g = _generator(seed)
    path = case["path"]
    if path == "matvec":
        rows, cols, n = case["rows"], case["cols"], case["n"]
        mats = [_mat(FMT[f], rows, cols, g) for f in case["formats"].split(",")]
        x = torch.randn(n * cols, device="cuda", generator=g)
        return dict(path=path, n=n, x=x, mats=mats, acts=[D.make_qact(n * cols, D.matrix_act_kind(w)) for w in mats],
                    ys=[_f32(n * rows) for _ in mats])
    if path == "moe":
        return dict(path=path, s=Moe(case, g))
    s = Dense(case, g, case.get("n", 1))
    vocab = s.head.rows
    s.logits = _f32((1 if path == "prefill" else s.n) * vocab)
    state = dict(path=path, s=s)
    if path == "prefill":
        one = s.layers[0]
        tc = D.tc_takes(one["gate"], s.n) and D.tc_takes(one["down"], s.n)
        s.mid = D.ChunkF16(s.n, s.ffn) if tc else None
    elif path == "plan":
        ops = []
        for i, L in enumerate(s.layers):
            ops += [D.decode_op(L["q"], s.h, s.q, norm_w=L["nw1"], eps=EPS, bias=L["bq"], after=True),
                    D.decode_op(L["k"], s.h, s.k[i], norm_w=L["nw1"], eps=EPS, bias=L["bk"], after=False),
                    D.decode_op(L["v"], s.h, s.v[i], norm_w=L["nw1"], eps=EPS, bias=L["bv"], after=False),
                    D.decode_op(L["o"], s.att, s.h, acc=True, after=True),
                    D.decode_op(L["gate"], s.h, s.fa, w2=L["up"], norm_w=L["nw2"], eps=EPS, after=True),
                    D.decode_op(L["down"], s.fa, s.h, acc=True, after=True)]
        ops.append(D.decode_op(s.head, s.h, s.logits, norm_w=s.nwf, eps=EPS, after=True))
        s.plan = D.DecodePlan(ops)
    elif case["graph"]:
        _token(s)  # the first pass is not captured: it sets up what is set up once
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            _token(s)
        state["graph"] = True
    return state


def run(state):
    path, s = state["path"], state.get("s")
    if path == "matvec":
        for w, act, y in zip(state["mats"], state["acts"], state["ys"]):
            D.cmat_mul(w, D.quant_q8(state["x"], act), y, state["n"])
        return state["ys"]
    if path == "moe":
        return _moe_token(s) if s.n == 1 else _moe_chunk(s)
    if path == "prefill":
        _prefill(s)
    elif path == "plan":
        _plan(s)
    elif state.get("graph"):
        s.graph.replay()
    else:
        _token(s)
    return {"h": s.h, "k": s.k, "v": s.v, "logits": s.logits}


# ---------------------------------------------------------------- what a pass cannot do without

def _distinct_experts(moe, n):
    """Experts that N tokens choose, expected over the router's scores."""
    d, ff, ne, nu, gate, zipf = MOES[moe]
    score = 1.0 / (1.0 + np.exp(-np.random.default_rng(0).standard_normal((4096, ne))))
    score += _popularity(ne, zipf) if zipf else 0.0
    chosen = np.argpartition(-score, nu, axis=1)[:, :nu]
    share = np.bincount(chosen.reshape(-1), minlength=ne) / 4096.0
    return float((1.0 - (1.0 - share) ** n).sum())


def work(case):
    path = case["path"]
    if path == "matvec":
        rows, cols, n = case["rows"], case["cols"], case["n"]
        fmts = [FMT[f] for f in case["formats"].split(",")]
        return {"bytes": sum(B.matrix_bytes(f, rows, cols) for f in fmts) + 4 * n * cols + 4 * n * rows * len(fmts),
                "flops": 2.0 * rows * cols * n * len(fmts)}
    if path == "moe":
        d, ff, ne, nu, gate, _ = MOES[case["moe"]]
        n = case["n"]
        expert = 2 * B.matrix_bytes(FMT[gate], ff, d) + B.matrix_bytes(B.Q2_K, d, ff)
        shared = 3 * B.matrix_bytes(B.Q8_0, ff, d)
        return {"bytes": _distinct_experts(case["moe"], n) * expert + shared + 2 * ne * d + 4 * n * (2 * d + ne),
                "flops": 2.0 * n * (3.0 * d * ff * (nu + 1) + ne * d)}
    hidden, qd, kv, ffn, vocab, main, alt, _ = MODELS[case["model"]]
    main, alt, n, nl = FMT[main], FMT[alt], case.get("n", 1), case["layers"]
    layer = sum(B.matrix_bytes(f, r, c) for f, r, c in ((main, qd, hidden), (main, kv, hidden), (alt, kv, hidden), (main, hidden, qd),
                                                        (main, ffn, hidden), (main, ffn, hidden), (alt, hidden, ffn)))
    heads = 1 if path == "prefill" else n
    weights = hidden * (2 * qd + 2 * kv) + 3 * hidden * ffn
    return {"bytes": nl * layer + B.matrix_bytes(alt, vocab, hidden) + n * B.row_bytes(alt, hidden) + 4 * n * (hidden + qd + 2 * nl * kv)
            + 4 * heads * vocab,
            "flops": 2.0 * (nl * weights * n + vocab * hidden * heads)}


def tolerance(case):
    if case["path"] == "matvec":
        return {"rel": 1e-5, "max": 1e-4}  # whole-number block sums, 32-bit floats between them
    # the activations between two products are rounded to 8 bits: a difference in the last bit of a 32-bit sum moves one of
    # them to the next value now and then, and every later layer rounds again; a near tie can choose another expert
    return {"rel": 1e-2, "max": 0.9}
