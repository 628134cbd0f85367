// chain.cu -- a token's chain of products as a CUDA graph: a launch a product and a quantization, recorded once and launched as one.
//
// The chain kernel (decode.cu) runs the token as one cooperative launch whose CTAs meet between dependent products; 145 meetings at
// five to six microseconds are most of a 4B token's time.  Launches one behind the other, each of which brings its weights before the one
// before it ends (programmatic dependent launch, which a graph keeps), take three to four: us a token, that kernel / this: 36 layers
// of a 4B model (Q4_K, Q6_K) and its head 2360 / 1515, 24 of a 0.5B one (Q8_0) 1120 / 463, one layer and the head 101 / 55.
// The products and quantizers are the stand-alone ones (ill_mv, ill_mv_3, ill_mv_glu, ill_quant_q8_*, ill_rmsnorm_q8), so the results are
// theirs, bit for bit, and the chain kernel's where that takes a row whole (decode.cu).
// In a recording of the caller's, products of two formats go one behind the other: the fork (issue's SIDE) needs a stream and events that
// would be that recording's.
//
// Replaces the launches of CUDA-FORWARD-N (src/cuda-dense.lisp:380-432).
#include <new>
#include <vector>

#include "formats.cuh"
#include "host.h"

using namespace ill;

namespace {

// what the products of one set of activations read: quants, scales, sums of 16
struct Scratch {
  ill_dptr xq, xs, xsum;
  int64_t bytes;
};
Scratch layout(const ill_decode_op* ops, int nops, ill_dptr base) {
  int64_t cols = 0;
  for (int i = 0; i < nops; ++i)
    if (ops[i].cols > cols) cols = ops[i].cols;
  cols = (cols + 255) / 256 * 256;
  Scratch s;
  s.xq = base;
  s.xs = s.xq + cols;
  s.xsum = s.xs + cols / 32 * 4;
  s.bytes = cols + cols / 32 * 4 + cols / 16 * 2;
  return s;
}

int check_ops(const ill_decode_op* ops, int nops, ill_dptr scratch, int64_t bytes) {
  if (!ops || nops < 1 || !scratch) return ILL_ERR_ARG;
  for (int i = 0; i < nops; ++i) {
    const ill_decode_op& o = ops[i];
    const int bw = fmt_block_weights(o.fmt);
    if (!bw || (o.kind != ILL_OP_MV && o.kind != ILL_OP_GLU) || o.rows <= 0 || o.cols <= 0 || o.cols % (bw == 32 ? 32 : 256) || !o.w || !o.x ||
        !o.y || (o.kind == ILL_OP_GLU && (!o.w2 || o.acc || o.bias)) || (o.kind == ILL_OP_MV && o.w2))
      return ILL_ERR_ARG;
    if ((o.w & 15) || (o.w2 & 15) || (o.x & 15) || (o.norm_w & 15) || (o.y & 3) || (o.bias & 3)) return ILL_ERR_ALIGN;
  }
  if (scratch & 127) return ILL_ERR_ALIGN;
  return bytes < layout(ops, nops, 0).bytes ? ILL_ERR_TOO_LARGE : ILL_OK;
}

// The launches, in order, on ST.  SIDE (a recording): products of one set of activations whose formats differ go beside each other, the
// second format's in that stream (a file's V in Q6_K beside Q and K: 3 us of a layer's 39).
int issue(const ill_decode_op* ops, int nops, const Scratch& s, cudaStream_t st, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join) {
  for (int i = 0; i < nops;) {
    const ill_decode_op& a = ops[i];
    const bool q8 = a.fmt == ILL_Q8_0;
    const ill_dptr xsum = q8 ? 0 : s.xsum;
    int rc;
    if (a.norm_w)
      rc = ill_rmsnorm_q8(q8 ? 0 : 1, a.x, a.norm_w, 0, s.xq, s.xs, xsum, a.cols, a.eps, 1, a.f16_scale ? 1 : 0, st);
    else if (q8)
      rc = ill_quant_q8_0(a.x, s.xq, s.xs, 0, a.cols / 32, a.f16_scale ? 1 : 0, st);
    else
      rc = ill_quant_q8_k(a.x, s.xq, s.xs, s.xsum, a.cols / 256, st);
    if (rc) return rc;
    // the products of these activations: until one that an earlier product's results go into, or other activations
    int end = i + 1;
    while (end < nops && !ops[end].after && ops[end].x == a.x && ops[end].norm_w == a.norm_w && (!a.norm_w || ops[end].eps == a.eps) &&
           ops[end].cols == a.cols && (ops[end].fmt == ILL_Q8_0) == q8 && (!q8 || (ops[end].f16_scale != 0) == (a.f16_scale != 0)))
      ++end;
    // (forked where the activations are there, not behind the products of the first format)
    bool forked = false;
    for (int k = i; side && k < end; ++k) forked = forked || (ops[k].fmt != a.fmt && !ops[k].acc);
    if (forked) {
      cudaError_t e = cudaEventRecord(fork, st);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(side, fork, 0);
      if (e != cudaSuccess) return cuda_fail(e);
    }
    while (i < end) {
      const ill_decode_op& o = ops[i];
      // up to three plain products of one format in a launch, where each alone would add a row's blocks in the same order: that
      // follows from whether the launch moves 16 MB
      const int bw = fmt_block_weights(o.fmt);
      auto small = [&](long long rows) { return rows * (o.cols / bw * fmt_block_bytes(o.fmt)) < (16ll << 20); };
      int m = 1;
      long long rows = o.rows;
      while (o.kind == ILL_OP_MV && !o.acc && m < 3 && i + m < end && ops[i + m].kind == ILL_OP_MV && !ops[i + m].acc && ops[i + m].fmt == o.fmt &&
             small(rows + ops[i + m].rows)) {
        rows += ops[i + m].rows;
        ++m;
      }
      const cudaStream_t on = forked && o.fmt != a.fmt && !o.acc ? side : st;
      if (o.kind == ILL_OP_GLU)
        rc = ill_mv_glu(o.fmt, o.w, o.w2, o.rows, o.cols, s.xq, s.xs, xsum, o.y, on);
      else if (m == 1)
        rc = ill_mv(o.fmt, o.w, o.rows, o.cols, s.xq, s.xs, xsum, o.y, o.bias, o.acc ? 1 : 0, 1, on);
      else {
        const ill_decode_op &p = ops[i + 1], *q = m > 2 ? &ops[i + 2] : nullptr;
        rc = ill_mv_3(o.fmt, o.w, p.w, q ? q->w : 0, o.rows, p.rows, q ? q->rows : 0, o.cols, s.xq, s.xs, xsum, o.y, p.y, q ? q->y : 0, o.bias,
                      p.bias, q ? q->bias : 0, on);
      }
      if (rc) return rc;
      i += m;
    }
    if (forked) {
      cudaError_t e = cudaEventRecord(join, side);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(st, join, 0);
      if (e != cudaSuccess) return cuda_fail(e);
    }
  }
  return ILL_OK;
}

struct Chain {
  std::vector<ill_decode_op> ops;
  Scratch s;
  cudaGraphExec_t exec;
};

}  // namespace

extern "C" int64_t ill_chain_scratch_bytes(const ill_decode_op* ops, int nops) { return !ops || nops < 1 ? 0 : layout(ops, nops, 0).bytes; }

extern "C" int ill_chain_new(const ill_decode_op* ops, int nops, ill_dptr scratch, int64_t scratch_bytes, uint64_t* chain) {
  if (!chain) return ILL_ERR_ARG;
  *chain = 0;
  int rc = check_ops(ops, nops, scratch, scratch_bytes);
  if (rc) return rc;
  Chain* c = new (std::nothrow) Chain();
  if (!c) return ILL_ERR_TOO_LARGE;
  try {
    c->ops.assign(ops, ops + nops);
  } catch (...) {
    delete c;
    return ILL_ERR_TOO_LARGE;
  }
  c->s = layout(ops, nops, scratch);
  cudaStream_t st = nullptr, side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  cudaGraph_t graph = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&join, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaStreamBeginCapture(st, cudaStreamCaptureModeRelaxed);
  if (e == cudaSuccess) {
    rc = issue(c->ops.data(), nops, c->s, st, side, fork, join);
    e = cudaStreamEndCapture(st, &graph);  // (after a launch that failed too: the recording ends)
    if (!rc && e == cudaSuccess) e = cudaGraphInstantiate(&c->exec, graph, 0);
  }
  if (rc || e != cudaSuccess) (void)cudaGetLastError();
  if (graph) cudaGraphDestroy(graph);
  if (fork) cudaEventDestroy(fork);
  if (join) cudaEventDestroy(join);
  if (side) cudaStreamDestroy(side);
  if (st) cudaStreamDestroy(st);
  if (!rc && e != cudaSuccess) rc = cuda_fail(e);
  if (rc) {
    delete c;
    return rc;
  }
  *chain = (uint64_t)(uintptr_t)c;
  return ILL_OK;
}

extern "C" int ill_chain_run(uint64_t chain, ill_stream stream) {
  Chain* c = (Chain*)(uintptr_t)chain;
  if (!c) return ILL_ERR_ARG;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing((cudaStream_t)stream, &cap);
  if (e != cudaSuccess) return cuda_fail(e);
  // a recording of the caller's gets the launches themselves
  if (cap != cudaStreamCaptureStatusNone) return issue(c->ops.data(), (int)c->ops.size(), c->s, (cudaStream_t)stream, nullptr, nullptr, nullptr);
  e = cudaGraphLaunch(c->exec, (cudaStream_t)stream);
  return e == cudaSuccess ? ILL_OK : cuda_fail(e);
}

extern "C" int ill_chain_free(uint64_t chain) {
  Chain* c = (Chain*)(uintptr_t)chain;
  if (!c) return ILL_OK;
  // (a launch that is still running keeps what it needs)
  const cudaError_t e = cudaGraphExecDestroy(c->exec);
  delete c;
  return e == cudaSuccess ? ILL_OK : cuda_fail(e);
}
