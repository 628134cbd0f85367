// mm_q8.cu -- Q8_0 products of a chunk of tokens (more than 16) on the 5th-generation tensor cores.
//
//   Y[token, row] (+)= sum over blocks b of 32 columns of  float(W_b[row] . X_b[token]) * (d_w * d_x)   (+ bias[row])
//
// Q8_0 has a scale for every 32 columns on both sides, so every 32-wide product of integers has to leave the tensor core and meet
// its scales: tcgen05.mma.kind::i8 takes the int8 quants of both as they are (128 x N x 32, int32 accumulators: one instruction a
// block, no conversion of either operand) and the drain turns the int32 sums into floats.  A row's blocks are added in order and each
// step is rounded as the CPU path rounds it (Q8-ROW-DOT-AT, src/tensor.lisp:321-336: sum += float(isum) * (d_w * d_x)), so the bits do
// not depend on the tile.
//
// A persistent CTA an SM walks tiles of 128 weight rows x BM (a multiple of 16, at most 128) tokens; columns go by in steps of 128.
//   warp 0       brings X by TMA: a step of the tile's tokens, 128 bytes a token (128-byte swizzle), the MMA's B operand
//   warp 1       allocates tensor memory; one lane issues the products
//   warp 2       brings the weights' raw blocks by TMA: 176 bytes of each row, from the 16-byte boundary at or before the step's 136
//   warp 3       brings the activations' scales (cp.async), transposed to [block][token]
//   warps 4-19   drain: four warps for each 32 weight rows, a quarter of the tokens each
//   warps 20-27  take the 34-byte blocks apart and store the quants to tensor memory, where they are the MMA's A operand: four warps,
//                a row a lane, every second step
// Tensor memory: three accumulators of 128 columns (a block of 128 tokens, two of 64 or four of 32 a job, so that a hand-over is
// always about 128 columns' worth), four stages of A.
//
// What bounds it: the drain.  A sum takes a conversion, a multiplication d_w * d_x, one with the sum and an addition.  The three are
// packed, two sums an instruction: no faster by themselves, but the schedulers have a slot in two left, which the conversions and the
// rest take (cycles of a scheduler, measured: two scalar multiply-adds and a conversion 3.2, a packed one and a conversion 2.5).  With the
// loads of the scales, the hand-overs and the unpacking about 1000 cycles for 128 x 128 x 32, where the product itself takes 64.  us,
// scalar / packed: 896 x 896 x 777 tokens 10.8 / 10.5, 896 x 4864 x 777 43.4 / 41.1, 4864 x 896 x 777 36.1 / 34.2, 2048 x 4096 x 64 20.7 / 20.1, x
// 200 27.0 / 25.5, x 4096 296 / 274, 4096 x 2048 x 4096 287 / 267, 1536 x 5120 x 8192 561 / 522, 5120 x 1536 x 8192 519 / 484.  (The same with
// int8 mma.sync, mm_q8_i8.cu: 896 x 4864 x 777 67, 2048 x 4096 x 200 60.)
// Measured and taken back: eight drain warps with the next half on its way while one is scaled (NT 128: 309 -> 398); 16 x 256-bit
// loads of tensor memory, a quarter of the shared memory's traffic (309 -> 319: it was no bound); raw blocks by cp.async of the
// warps that take them apart (a step 0.5 -> 1.1 us); even shares whatever the rounds (4864 x 896 x 200 13.6 -> 16.3).
//
// Every mbarrier wait is bounded; on a time-out the kernel records a code in the status word, skips what depends on the wait, lets
// copies and products in flight end, frees its tensor memory and returns.
//
// Replaces mm_q8_mma2 behind CMAT-MUL-N for prefill chunks (src/cuda-dense.lisp:220-255; src/cuda/dense.cu:885-1100).
#include <string.h>

#include "formats.cuh"
#include "tc05.cuh"
#include "host.h"

namespace ill {

constexpr int MQ_ROWS = 128;                        // weight rows a tile (the MMA's M)
constexpr int MQ_STEP = 128, MQ_WSTEP = 136;        // columns a step; a row's bytes of one (four blocks of 34)
constexpr int MQ_NS = 4, MQ_NACC = 3, MQ_NRAW = 4;  // stages of X, A and scales; accumulators; stages of raw blocks
constexpr int MQ_DRAIN = 16, MQ_UNPACK = 8, MQ_THREADS = 32 * (4 + MQ_DRAIN + MQ_UNPACK);
constexpr int MQ_PITCH = 176;                       // bytes of a row in a raw stage: an odd number of 16-byte pieces
constexpr uint32_t MQ_RAW_BYTES = MQ_ROWS * MQ_PITCH, MQ_A_COL = 128 * MQ_NACC;
constexpr int MQ_REGS_AUX = 32, MQ_REGS_DRAIN = 88, MQ_REGS_UNPACK = 56;
constexpr int MQ_REGS_SUM = 128 * MQ_REGS_AUX + 32 * (MQ_DRAIN * MQ_REGS_DRAIN + MQ_UNPACK * MQ_REGS_UNPACK);

constexpr int MQ_MATS = 3;
struct MqMat {         // one of up to three matrices that share the activations
  float* y;
  const float* bias;
  int rows, rt_end;    // tiles of rows of this one and those before it
  int off[2];          // where the first row's bytes start in the (even, odd) map
};
struct MqParams {
  MqMat m[MQ_MATS];
  int nsteps;
  int split;           // rows are a multiple of 16 bytes apart only two by two: the even ones and the odd ones have a map each
  int cols;
  const float* xs;
  int acc, n;
  int bm;              // tokens a tile, a multiple of 16; a CTA takes every gridDim.x-th tile -- or, SHARE not 0,
  int early;           // the next kernel may start before this one ends
  int ncol, share;     // SHARE of the NCOL columns of 16 tokens of all the tiles of rows one after another, in tiles of up to BM
  uint32_t zero;
  uint64_t neg_zero;   // two of them (mul2_rn)
  unsigned* status;
};
struct MqMaps {
  CUtensorMap x, w[MQ_MATS][2];
};

template <int NT> struct MqGeom {
  static constexpr int G = 128 / NT, JOBS = 4 / G;  // blocks a job; jobs a step
  static constexpr int TW = NT / 4;                 // tokens a drain warp
  static constexpr uint32_t X_BYTES = NT * MQ_STEP;
  static constexpr uint32_t RAW = MQ_NS * X_BYTES, WSC = RAW + MQ_NRAW * MQ_RAW_BYTES, XSC = WSC + MQ_NS * 4 * MQ_ROWS * 4,
                            BARS = XSC + MQ_NS * 4 * NT * 4, SLOT = BARS + 8 * (2 * MQ_NS + 2 * MQ_NACC + 2 * MQ_NRAW + 1);
  // at least what keeps a second CTA, which would wait for tensor memory, off the SM
  static constexpr size_t NEED = SLOT + 16 + 1024 /* alignment */, SMEM = NEED > 118 * 1024 ? NEED : 118 * 1024;
};

// D[tmem] = A[tmem] * B[smem]^T, 128 x N x 32, int8 operands, int32 accumulators.  A: 128 lanes x 8 columns (four quants a column).
__device__ __forceinline__ void umma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc)
      : "memory");
}
__device__ __forceinline__ void mq_cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// A CTA's tiles, in order
struct MqWalk {
  int pos, end, ntr;         // the tile, or column, next; past the last
  int mi, row0, tok0, nvalid;  // the tile: of which matrix, where
  __device__ __forceinline__ explicit MqWalk(const MqParams& p) {
    ntr = p.m[MQ_MATS - 1].rt_end;
    pos = p.share ? blockIdx.x * p.share : blockIdx.x;
    end = p.share ? min(pos + p.share, ntr * p.ncol) : ntr * ((p.n + p.bm - 1) / p.bm);
  }
  __device__ __forceinline__ void at_row_tile(const MqParams& p, int rt) {
    mi = (rt >= p.m[0].rt_end) + (rt >= p.m[1].rt_end);
    row0 = (rt - (mi ? p.m[mi - 1].rt_end : 0)) * MQ_ROWS;
  }
  __device__ __forceinline__ bool next(const MqParams& p) {
    if (pos >= end) return false;
    if (p.share) {
      const int rt = pos / p.ncol, col = pos - rt * p.ncol, take = min(min(p.bm / 16, end - pos), p.ncol - col);
      at_row_tile(p, rt);
      tok0 = 16 * col;
      nvalid = min(16 * take, p.n - tok0);
      pos += take;
    } else {                 // tiles of rows vary fastest: CTAs running together share X
      const int tt = pos / ntr;
      at_row_tile(p, pos - tt * ntr);
      tok0 = tt * p.bm;
      nvalid = min(p.bm, p.n - tok0);
      pos += gridDim.x;
    }
    return true;
  }
};

template <int NT>
__global__ void __launch_bounds__(MQ_THREADS, 1) mm_q8_kernel(const __grid_constant__ MqMaps maps, const MqParams p) {
  typedef MqGeom<NT> G;
  constexpr int JOBS = G::JOBS, GB = G::G, TW = G::TW;
  extern __shared__ __align__(1024) u8 smem_raw[];
  u8* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  u8* x_tiles = smem;                                // [MQ_NS][NT tokens][128 bytes], swizzled
  u8* raw = smem + G::RAW;                           // [MQ_NRAW][128 rows][MQ_PITCH] (SPLIT: the even rows, then the odd ones)
  float* wsc = (float*)(smem + G::WSC);              // [MQ_NS][4 blocks][128 weight rows]
  float* xsc = (float*)(smem + G::XSC);              // [MQ_NS][4 blocks][NT tokens]
  uint64_t* bars = (uint64_t*)(smem + G::BARS);
  uint64_t *full = bars,                             // the step's X landed (TMA), its quants of the weights are in tensor memory (4 warps),
                                                     // its scales in shared memory (those warps' and 32 lanes' copies)
      *free = bars + MQ_NS,                          // the drain is through with the step (16 warps): so are the products
      *acc_full = bars + 2 * MQ_NS,                  // a job's products completed
      *acc_free = acc_full + MQ_NACC,                // the drain has read them (16 warps)
      *raw_full = acc_free + MQ_NACC,                // the step's raw blocks landed (TMA)
      *raw_free = raw_full + MQ_NRAW,                // they have been read (4 warps)
      *fin = raw_free + MQ_NRAW;                     // after a time-out: the products issued so far completed
  uint32_t* tmem_slot = (uint32_t*)(smem + G::SLOT);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

  if (p.early) pdl_launch_dependents();
  if (tid == 32) {
    for (int s = 0; s < MQ_NS; ++s) { mbar_init(&full[s], 1 + 4 + 32); mbar_init(&free[s], MQ_DRAIN); }
    for (int b = 0; b < MQ_NACC; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_free[b], MQ_DRAIN); }
    for (int r = 0; r < MQ_NRAW; ++r) { mbar_init(&raw_full[r], 1); mbar_init(&raw_free[r], 4); }
    mbar_init(fin, 1);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  const int nsteps = p.nsteps;
  MqWalk tile(p);
  bool ok = true;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(MQ_REGS_AUX));
    if (warp == 0) {
      // ---- X by TMA
      pdl_wait();
      int k = 0;  // steps so far
      while (ok && tile.next(p)) {
        for (int st = 0; st < nsteps; ++st, ++k) {
          const int s = k % MQ_NS;
          ok = __all_sync(0xffffffffu, mbar_wait(&free[s], ((uint32_t)(k / MQ_NS) & 1u) ^ 1u, p.status, ST_MQ_WAIT));
          if (!ok) break;
          if (elect_one()) {
            mbar_expect_tx(&full[s], p.bm * MQ_STEP);
            tma_load_2d(x_tiles + s * G::X_BYTES, &maps.x, st * MQ_STEP, tile.tok0, &full[s]);
          }
          __syncwarp();
        }
      }
      if (!ok)  // a wait ran out: the copies in flight land before the CTA goes
        for (int j = max(0, k - MQ_NS); j < k; ++j) mbar_wait(&full[j % MQ_NS], (uint32_t)(j / MQ_NS) & 1u, nullptr, 0, 0, ILL_WAIT_NS / 20);
    } else if (warp == 1) {
      // ---- the products: the whole warp walks the loop, one elected lane issues.  Lane 0 watches the step, lane
      // 1 the job's accumulator: one poll looks at both.
      const uint64_t xdesc0 = umma_desc(x_tiles);
      const unsigned code = ST_MQ_WAIT + 1 + (lane ? 1 : 0);
      int k = 0, b = 0;
      uint32_t bph = 1;  // parity that a free accumulator's barrier has completed (a fresh barrier: 1)
      while (ok && tile.next(p)) {
        // int32 accumulate, int8 A and B, both K-major, M = 128 weight rows, N = the tile's tokens up to 16
        const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((tile.nvalid + 15) >> 4) << 18) | ((uint32_t)(MQ_ROWS >> 4) << 24);
        for (int st = 0; st < nsteps && ok; ++st, ++k) {
          const int s = k % MQ_NS;
#pragma unroll
          for (int j = 0; j < JOBS; ++j) {
            BarPoll poll(p.status, code);
            uint64_t* bar = lane == 0 ? &full[s] : &acc_free[b];
            if (!(ok = poll.until(bar, lane == 0 ? (uint32_t)(k / MQ_NS) & 1u : bph, j == 0 ? 3u : 2u))) break;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
              for (int g = 0; g < GB; ++g)
                umma_i8_ts(tmem_base + b * 128 + g * NT, tmem_base + MQ_A_COL + s * 32 + (j * GB + g) * 8,
                           xdesc0 + (uint32_t)(s * (int)(G::X_BYTES >> 4)) + 2 * (j * GB + g), idesc);
              umma_commit(&acc_full[b]);
            }
            __syncwarp();
            if (++b == MQ_NACC) { b = 0; bph ^= 1; }
          }
        }
      }
      if (!ok) {
        // a wait ran out: the products issued so far end before tensor memory is freed
        if (elect_one()) umma_commit(fin);
        __syncwarp();
        mbar_wait(fin, 0, nullptr, 0, 0, ILL_WAIT_NS / 20);
      }
    } else if (warp == 2) {
      // ---- the weights' raw blocks by TMA (they do not depend on the kernel before)
      int k = 0;
      while (ok && tile.next(p)) {
        const int off0 = p.m[tile.mi].off[0], off1 = p.m[tile.mi].off[1];
        const CUtensorMap* maps_w = maps.w[tile.mi];
        for (int st = 0; st < nsteps; ++st, ++k) {
          const int r = k % MQ_NRAW;
          ok = __all_sync(0xffffffffu, mbar_wait(&raw_free[r], ((uint32_t)(k / MQ_NRAW) & 1u) ^ 1u, p.status, ST_MQ_WAIT + 7));
          if (!ok) break;
          if (elect_one()) {
            u8* dst = raw + r * MQ_RAW_BYTES;
            mbar_expect_tx(&raw_full[r], MQ_RAW_BYTES);
            if (p.split) {
              tma_load_2d(dst, &maps_w[0], (off0 + st * MQ_WSTEP) & ~15, tile.row0 / 2, &raw_full[r]);
              tma_load_2d(dst + MQ_RAW_BYTES / 2, &maps_w[1], (off1 + st * MQ_WSTEP) & ~15, tile.row0 / 2, &raw_full[r]);
            } else {
              tma_load_2d(dst, &maps_w[0], (off0 + st * MQ_WSTEP) & ~15, tile.row0, &raw_full[r]);
            }
          }
          __syncwarp();
        }
      }
      if (!ok)
        for (int j = max(0, k - MQ_NRAW); j < k; ++j)
          mbar_wait(&raw_full[j % MQ_NRAW], (uint32_t)(j / MQ_NRAW) & 1u, nullptr, 0, 0, ILL_WAIT_NS / 20);
    } else {
      // ---- the activations' scales, [token][block] in memory, [block][token] in shared memory
      pdl_wait();
      const int nb = p.cols / 32;
      int k = 0;
      while (ok && tile.next(p)) {
        const float* src0 = p.xs + (long long)(tile.tok0 + lane) * nb;
        for (int st = 0; st < nsteps; ++st, ++k) {
          const int s = k % MQ_NS;
          ok = __all_sync(0xffffffffu, mbar_wait(&free[s], ((uint32_t)(k / MQ_NS) & 1u) ^ 1u, p.status, ST_MQ_WAIT + 4));
          if (!ok) break;
#pragma unroll
          for (int t = 0; t < NT; t += 32)
            if (t + lane < tile.nvalid) {
              const float* src = src0 + (long long)t * nb + 4 * st;
              float* dst = xsc + s * 4 * NT + t + lane;
#pragma unroll
              for (int b = 0; b < 4; ++b) mq_cp_async4(dst + b * NT, src + b);
            }
          cp_async_arrive(&full[s]);
        }
      }
      cp_async_wait_all();
    }
  } else if (warp < 4 + MQ_DRAIN) {
    // ---- drain.  A warp reads the 32 lanes of tensor memory that its number gives it (warp % 4: 32 weight rows) and a quarter of
    // the tokens of every block: 32 columns a job.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(MQ_REGS_DRAIN));
    pdl_wait();
    const int q = warp & 3, c0 = ((warp - 4) >> 2) * TW, m = q * 32 + lane;
    const uint32_t t0 = tmem_base + ((uint32_t)(q * 32) << 16) + c0;
    int s = 0, b = 0;
    uint32_t sph = 0, bph = 0;
    while (ok && tile.next(p)) {
      const int nvalid = tile.nvalid;
      uint64_t out[TW / 2];    // pairs of fp32
#pragma unroll
      for (int i = 0; i < TW / 2; ++i) out[i] = 0ull;
      for (int st = 0; st < nsteps; ++st) {
        // (complete as soon as the step's first products are: what makes the scales visible here)
        bool lane_ok = mbar_wait(&full[s], sph, p.status, ST_MQ_WAIT + 5);
        const float *ws = wsc + s * 4 * MQ_ROWS + m, *xs = xsc + s * 4 * NT + c0;
#pragma unroll
        for (int j = 0; j < JOBS; ++j) {
          lane_ok = lane_ok && mbar_wait(&acc_full[b], bph, p.status, ST_MQ_WAIT + 6);
          __syncwarp();
          tc_fence_after();
          uint32_t v[4][8];
          if (c0 < nvalid) {
#pragma unroll
            for (int r = 0; r < 4; ++r) tmem_ld(t0 + b * 128 + (8 * r / TW) * NT + 8 * r % TW, v[r]);
            tmem_ld_wait(v[0]);
            tmem_ld_done(v[1]); tmem_ld_done(v[2]); tmem_ld_done(v[3]);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_free[b]);
          if (++b == MQ_NACC) { b = 0; bph ^= 1; }
          if (c0 < nvalid) {  // (columns past the tile's last token: whatever lies there; they are not stored)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              const int blk = j * GB + 8 * r / TW, c = 8 * r % TW;
              const float dw = ws[blk * MQ_ROWS];
              const uint64_t dw2 = pack2(dw, dw);
#pragma unroll
              for (int i = 0; i < 8; i += 4) {
                const ulonglong2 dx = *(const ulonglong2*)(xs + blk * NT + c + i);
                uint64_t* o = out + (c + i) / 2;
                o[0] = add2(o[0], mul2_rn(pack2((float)(int)v[r][i], (float)(int)v[r][i + 1]), mul2(dw2, dx.x), p.neg_zero));
                o[1] = add2(o[1], mul2_rn(pack2((float)(int)v[r][i + 2], (float)(int)v[r][i + 3]), mul2(dw2, dx.y), p.neg_zero));
              }
            }
          }
        }
        if (!(ok = __all_sync(0xffffffffu, lane_ok))) break;
        // (ZERO is none that the compiler knows: the step's last scales have been used, not only asked for, when it is given back)
        if (lane == 0) mbar_arrive(free + s + ((uint32_t)(out[TW / 2 - 1] >> 32) & p.zero));
        if (++s == MQ_NS) { s = 0; sph ^= 1; }
      }
      const MqMat& mat = p.m[tile.mi];
      const int row = tile.row0 + m, rows = mat.rows;
      if (ok && row < rows) {
        const float bias = mat.bias ? mat.bias[row] : 0.0f;
        float* yp = mat.y + (long long)(tile.tok0 + c0) * rows + row;
#pragma unroll
        for (int i0 = 0; i0 < TW; i0 += 8) {
          if (c0 + i0 < nvalid) {
            float old[8];
            if (p.acc) {
#pragma unroll
              for (int i = 0; i < 8; ++i) old[i] = c0 + i0 + i < nvalid ? yp[(long long)(i0 + i) * rows] : 0.0f;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              float r = __uint_as_float((uint32_t)(out[(i0 + i) >> 1] >> (32 * (i & 1))));
              if (mat.bias) r += bias;
              if (p.acc) r = old[i] + r;
              if (c0 + i0 + i < nvalid) yp[(long long)(i0 + i) * rows] = r;
            }
          }
        }
      }
    }
  } else {
    // ---- the weights: a warp has 32 rows of every second step, a lane one of them
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(MQ_REGS_UNPACK));
    const int q = warp & 3, set = (warp - 4 - MQ_DRAIN) >> 2, row = 32 * q + lane, odd = p.split & row & 1;
    const uint32_t a0 = tmem_base + ((uint32_t)(q * 32) << 16) + MQ_A_COL;
    const u8* mine = raw + (p.split ? odd * (MQ_RAW_BYTES / 2) + (row >> 1) * MQ_PITCH : row * MQ_PITCH);
    int k = 0;
    while (ok && tile.next(p)) {
      const int off = p.m[tile.mi].off[odd ? 1 : 0];
      const bool by8 = (off & 7) == 0;               // (the same for all rows of a matrix: they lie a multiple of eight bytes apart)
      for (int st = 0; st < nsteps; ++st, ++k) {
        if ((k & 1) != set) continue;
        const int s = k % MQ_NS, r = k % MQ_NRAW;
        const uint32_t free_par = ((uint32_t)(k / MQ_NS) & 1u) ^ 1u;
        ok = __all_sync(0xffffffffu, mbar_wait(&raw_full[r], (uint32_t)(k / MQ_NRAW) & 1u, p.status, ST_MQ_WAIT + 8));
        if (!ok) break;
        // the step's 34 words: four blocks of a half and 32 quants, 34 bytes apart
        const uint32_t o16 = (uint32_t)(off + st * MQ_WSTEP) & 15u, sh = 8 * (o16 & 2u);
        const u8* src = mine + r * MQ_RAW_BYTES + (o16 & ~3u);
        auto words = [&](int w0, int n, uint32_t* w) {
          if (by8) {
#pragma unroll
            for (int i = 0; i < 18; i += 2)
              if (i < n) {
                const uint2 v = *(const uint2*)(src + 4 * (w0 + i));
                w[i] = v.x;
                w[i + 1] = v.y;
              }
          } else {                                   // a row may start in the middle of a word
#pragma unroll
            for (int i = 0; i < 18; ++i)
              if (i < n) w[i] = __funnelshift_r(*(const uint32_t*)(src + 4 * (w0 + i)), *(const uint32_t*)(src + 4 * (w0 + i) + 4), sh);
          }
        };
        uint32_t w[18], a[16], d[4];
        words(0, 18, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          a[i] = __funnelshift_r(w[i], w[i + 1], 16);
          a[8 + i] = w[9 + i];
        }
        d[0] = w[0] & 0xffffu;
        d[1] = w[8] >> 16;
        const uint32_t w17 = w[17];
        ok = __all_sync(0xffffffffu, mbar_wait(&free[s], free_par, p.status, ST_MQ_WAIT + 3));
        if (!ok) break;
        tc_fence_after();
        tmem_st16(a0 + s * 32, a);
        words(18, 16, w);
        d[2] = w17 & 0xffffu;
        d[3] = w[7] >> 16;
        a[0] = __funnelshift_r(w17, w[0], 16);
#pragma unroll
        for (int i = 1; i < 8; ++i) a[i] = __funnelshift_r(w[i - 1], w[i], 16);
#pragma unroll
        for (int i = 0; i < 8; ++i) a[8 + i] = w[8 + i];
        tmem_st16(a0 + s * 32 + 16, a);
#pragma unroll
        for (int i = 0; i < 4; ++i) wsc[(s * 4 + i) * MQ_ROWS + row] = h2f(d[i]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        // (the raw words have been stored by now, not only asked for)
        if (lane == 0) { mbar_arrive(&full[s]); mbar_arrive(&raw_free[r]); }
      }
    }
    tmem_st_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

template <int NT>
static int mq_launch(const MqMaps& maps, const MqParams& p, int grid, cudaStream_t st) {
  const void* k = (const void*)mm_q8_kernel<NT>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MqGeom<NT>::SMEM);
  if (e != cudaSuccess) return cuda_fail(e);
  // the warp groups trade registers after launch: what they ask for together must fit in what the CTA was given.  (Asked for at each
  // launch, 0.35 us with the attribute above: an answer kept from the first launch would be one device's, and a failure's for good.)
  cudaFuncAttributes fa;
  e = cudaFuncGetAttributes(&fa, k);
  if (e != cudaSuccess) return cuda_fail(e);
  if (fa.numRegs / 8 * 8 * MQ_THREADS < MQ_REGS_SUM) return ILL_ERR_UNSUPPORTED;
  MqMaps m = maps;
  MqParams pp = p;
  void* args[] = {&m, &pp};
  return launch_kernel(k, dim3((unsigned)grid), dim3(MQ_THREADS), MqGeom<NT>::SMEM, args, st);
}

// A map of ROWS rows of BYTES bytes, STRIDE apart (a multiple of 16, as BASE), read in boxes of BOX_BYTES x BOX_ROWS
static bool byte_map(CUtensorMap* map, uint64_t base, uint64_t bytes, uint64_t rows, uint64_t stride, uint32_t box_bytes, uint32_t box_rows,
                     bool swizzle) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {bytes, rows}, strides[1] = {stride};
  const cuuint32_t box[2] = {box_bytes, box_rows}, estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)(uintptr_t)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Which tiles: BM tokens each, one after another or (SHARE not 0) in even shares of SHARE columns of 16 tokens; a step's time, us
struct MqDeal {
  int bm, share, grid;
  float us;
};
static MqDeal mq_deal(long long ntr, int n, int sms) {  // NTR tiles of rows
  MqDeal d = {};
  // Tokens a tile: the rounds of tiles on the SMs times a tile's time a step, us, over 21 matrices at 17 to 8192 tokens.  A step's
  // hand-overs cost 16 tokens as much as its arithmetic; above 64 tokens a block is a job of its own.  The choice takes the
  // fastest of them or one that is 0.3 % slower on average, 9 % at most.
  static const float step_us[8] = {0.63f, 0.79f, 1.14f, 1.27f, 2.02f, 2.10f, 2.34f, 2.38f};
  float best = 1e30f;
  long long tiles = 0, rounds = 0;
  for (int bm = 16; bm <= 128; bm += 16) {
    const long long count = ntr * ((n + bm - 1) / bm), r = (count + sms - 1) / sms;
    const float us = (float)r * step_us[bm / 16 - 1];
    if (us < best) { best = us; d.bm = bm; tiles = count; rounds = r; }
  }
  d.grid = (int)(tiles < sms ? tiles : sms);
  d.us = best;
  // Even shares instead of a last round that is half empty, for tiles of 64 tokens, three a share at least: the tile more at a share's
  // ends costs what less than 13 % off the rounds saves, or 4 % where a share is a third of a tile of rows at most.  us, rounds /
  // shares: 9728 x 2560 x 512 tokens (4.1 rounds) 130 / 123, x 400 (3.6) 104 / 97, 17408 x 5120 x 400 (6.4) 352 / 340; 896 x 4864 x
  // 8192 (6.1) 335 / 322, 1536 x 5120 x 8192 (10.4) 570 / 557; where less is to be saved 36000 x 1024 x 300 (9.5) 109 / 115, 5120 x 1536
  // x 2048 (8.6) 143 / 150.  Other tiles gain nothing (128 tokens: 5120 x 1536 x 4096 259 / 273; 32: 151936 x 896 x 32 61 / 61).
  const long long ncol = (n + 15) / 16, share = (ntr * ncol + sms - 1) / sms;
  if (d.bm == 64 && share >= 12 && 100 * share < 4 * rounds * (3 * share <= ncol ? 96 : 87)) {
    d.share = (int)share;
    d.us = 1.10f * step_us[3] * (float)share / 4.0f;
    d.grid = (int)((ntr * ncol + share - 1) / share);
  }
  return d;
}

// Whether the kernel on mma.sync is the faster one: by the two estimates, with 0.3 us for this kernel's start, and well enough for the
// estimates' error.  Over 393 products of 21 matrices at 17 to 8192 tokens the choice takes the faster kernel or one within 3 % of it
// for 358; of rows of 256 columns and more, 25 are slower by more, the most by 15 %.  Up to 32 tokens a tile holds all of them and this
// kernel has it.  us, this kernel / that: 36000 x 1024 x 80 tokens 39.4 / 29.2, x 160 63.8 / 54.5, 17408 x 5120 x 160 147 / 130, 5120 x
// 1536 x 512 42.4 / 39.4, 4864 x 896 x 512 26.1 / 24.2, x 777 36 / 38, 896 x 4864 x 777 43 / 67, 2048 x 4096 x 200 26 / 60.
static bool mq_i8_is_faster(const MqDeal& d, int rows, int cols, int n, int sms) {
  const float nsteps = (float)(cols / MQ_STEP);
  return n > 32 && nsteps * mm_q8_i8_step_us(rows, n, sms) < 0.92f * (nsteps * d.us + 0.3f);
}

static long long mq_row_tiles(int rows) { return (rows + MQ_ROWS - 1) / MQ_ROWS; }

// Whether one launch of several matrices is faster than one each: by the estimates, with the two microseconds that a launch behind
// another costs beside its steps.  us, a launch each / one: 896 x 896 and 128 x 896, 17 tokens 11.2 / 5.9, 777 17.7 / 11.2,
// 2048 26.7 / 19.4; 2 x 1536 x 5120, 64 tokens 49 / 26, 256 62 / 46.
static bool mq_joint_is_faster(const MqDeal& d, int nmat, const int* rows, int cols, int n, int sms) {
  const float nsteps = (float)(cols / MQ_STEP);
  float apart = 0.0f;
  for (int i = 0; i < nmat; ++i) {
    const MqDeal one = mq_deal(mq_row_tiles(rows[i]), n, sms);
    const float us = mq_i8_is_faster(one, rows[i], cols, n, sms) ? mm_q8_i8_step_us(rows[i], n, sms) : one.us;
    apart += nsteps * us + 2.0f;
  }
  return nsteps * d.us + 2.0f < apart;
}

// N tokens of up to three Q8_0 matrices that share the activations; ILL_ERR_UNSUPPORTED for what it is not written for, and where
// several are faster one by one.
int mm_q8_try(int nmat, const uint64_t* w, const int* rows, int cols, uint64_t xq, uint64_t xs, const uint64_t* y, const uint64_t* bias, int acc,
              int n, void* stream) {
  if (n < 2 || cols % MQ_STEP || (xq & 15) || (xs & 15) || nmat < 1 || nmat > MQ_MATS) return ILL_ERR_UNSUPPORTED;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  MqParams p = {};
  long long ntr = 0;
  for (int i = 0; i < MQ_MATS; ++i) {
    if (i < nmat) {
      if (w[i] & 1) return ILL_ERR_UNSUPPORTED;
      p.m[i].rows = rows[i];
      p.m[i].y = (float*)(uintptr_t)y[i];
      p.m[i].bias = bias ? (const float*)(uintptr_t)bias[i] : nullptr;
      ntr += mq_row_tiles(rows[i]);
    }
    if (ntr * ((n + 15) / 16) > 0x7fffffffll) return ILL_ERR_TOO_LARGE;
    p.m[i].rt_end = (int)ntr;
  }
  p.cols = cols;
  p.nsteps = cols / MQ_STEP;
  p.xs = (const float*)(uintptr_t)xs;
  p.acc = acc;
  p.n = n;
  p.neg_zero = 0x8000000080000000ull;
  p.status = device_status_word();
  const MqDeal d = mq_deal(ntr, n, sms);
  if (nmat > 1) {
    if (!mq_joint_is_faster(d, nmat, rows, cols, n, sms)) return ILL_ERR_UNSUPPORTED;
  } else if (mq_i8_is_faster(d, rows[0], cols, n, sms)) {
    return mm_q8_i8(w[0], rows[0], cols, xq, xs, y[0], bias ? bias[0] : 0, acc, n, sms, stream);
  }
  p.bm = d.bm;
  p.ncol = (n + 15) / 16;
  p.share = d.share;
  // What the next kernel's early start gives is a microsecond or two: 896 x 4864 x 777 (43 us) and its like lose 1 % of a chunk
  // without.  After a long launch, whose CTAs end a tile apart, it costs more: the CTAs of the chain behind it go to whichever SM is
  // free, not in order, and the large expert products at its end take longer (down product of a shared expert, 5120 x 1536 x 8192 tokens,
  // 513 us: the layer 8673 us with the early start, 8530 without).
  p.early = (float)p.nsteps * d.us < 100.0f;
  const int grid = d.grid;
  MqMaps maps;
  const uint64_t row_bytes = (uint64_t)cols / 32 * 34;
  if (!byte_map(&maps.x, xq, cols, n, cols, MQ_STEP, p.bm, true)) return cuda_fail(cudaErrorInvalidValue);
  // Rows lie a multiple of eight bytes apart; a map's have to lie a multiple of 16.  A row starts OFF bytes after a 16-byte boundary.
  p.split = row_bytes % 16 != 0;
  for (int mi = 0; mi < MQ_MATS; ++mi) {
    if (mi >= nmat) {
      memcpy(maps.w[mi], maps.w[0], sizeof maps.w[mi]);
      continue;
    }
    for (int i = 0; i < 2; ++i) {
      const uint64_t base = w[mi] + (p.split && i && rows[mi] > 1 ? row_bytes : 0),
                     count = p.split ? (rows[mi] > 1 ? (rows[mi] + 1 - i) / 2 : 1) : rows[mi];
      p.m[mi].off[i] = (int)(base & 15);
      if (!byte_map(&maps.w[mi][i], base & ~15ull, p.m[mi].off[i] + row_bytes, count, p.split ? 2 * row_bytes : row_bytes, MQ_PITCH,
                    p.split ? MQ_ROWS / 2 : MQ_ROWS, false))
        return cuda_fail(cudaErrorInvalidValue);
    }
  }
  cudaStream_t st = (cudaStream_t)stream;
  if (p.bm <= 32) return mq_launch<32>(maps, p, grid, st);
  if (p.bm <= 64) return mq_launch<64>(maps, p, grid, st);
  return mq_launch<128>(maps, p, grid, st);
}

}  // namespace ill

using namespace ill;

extern "C" int ill_test_q8_chunk_plan(int rows, int cols, int n, int sms, int* out) {
  if (!out || rows < 1 || cols < MQ_STEP || n < 2 || sms < 1) return ILL_ERR_ARG;
  const MqDeal d = mq_deal(mq_row_tiles(rows), n, sms);
  out[0] = d.bm;
  out[1] = d.share;
  out[2] = d.grid;
  out[3] = mq_i8_is_faster(d, rows, cols, n, sms);
  return ILL_OK;
}
