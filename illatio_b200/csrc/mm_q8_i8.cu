// mm_q8_i8.cu -- Q8_0 products of a chunk of tokens on the tensor cores' int8 path (mma.sync): the tiles and CTAs are smaller than those of
// the kernel on tcgen05 (mm_q8.cu), several an SM, and fill the SMs better where many rows and tokens make rounds of tiles that
// the other leaves half empty, and for rows of a step or two, whose products do not pay for the other's start.  mm_q8_try weighs the
// two.
//
// What bounds a Q8_0 chunk is not the tensor pipe but what every m16n8k32 product needs after it: its four integers
// become floats and meet d_w * d_x, because Q8_0's scales are per 32 columns on both sides.  So the kernel is built
// around those instructions -- four conversions, four packed multiplies and two packed additions (f32x2) a product -- and
// keeps everything else off the issue slots:
//   * columns in steps of 128 (four blocks; a row's step is 136 bytes), weights and activations both by 16-byte
//     cp.async into a ring of three stages, one __syncthreads a step;
//   * what a thread copies lies at fixed distances from one step to the next: a step's copies are an add and a few
//     predicates beside the copies themselves;
//   * the activations' scales are staged in the order a lane reads them: the four of a token pair's two blocks are one
//     16-byte load for two products;
//   * two blocks of weights sit in registers at a time (mmd_kernel holds a step's): 80 tokens a CTA fit 128 registers, and
//     sixteen warps an SM.
// A CTA of RW warps takes 16 RW rows x 8 NT8 tokens; few rows of many columns take small CTAs, several an SM.  A row's
// blocks are added in order, each step rounded as the CPU path rounds it (Q8-ROW-DOT-AT, src/tensor.lisp:321-336): the bits of
// mm_q8.cu, whatever the tile.
//
// Measured against mmd_kernel (mmd.cu), which took Q8_0 first: 2048 x 4096 x 4096 tokens 412 -> 295 us (233 int8 TOPS), 5120 x 1536
// x 8192 728 -> 529, 4864 x 896 x 777 58 -> 37, 896 x 4864 x 777 129 -> 66, 2048 x 4096 x 64 62 -> 25.  What is left (the
// first of these shapes): about 40 cycles a product and scheduler, 18.5 instructions of it at 50 % issue, where the packed
// arithmetic alone takes 12 and the int8 mma.sync 8.2; the largest stalls are the shared-memory loads and the products'
// results (1.2 warps an issue), fixed latencies (0.9) and the arithmetic pipe (0.9).  Measured and dropped: 32 rows a warp
// (half the ldmatrix traffic, the same time); the integers turned into floats by adding 1.5 * 2^23 in the product (4 %
// slower); the columns dealt to groups of a CTA's warps (896 x 4864 x 777 in 40 us, but sums in another order: after a few
// layers' 8-bit activations that is a difference of 1 % in a model's output); fused multiply-adds (5 % faster, other bits).
//
// Replaces mm_q8_mma2 behind CMAT-MUL-N for prefill chunks (src/cuda-dense.lisp:220-255; src/cuda/dense.cu:885-1100).
#include "formats.cuh"
#include "host.h"
#include "mma_i8.cuh"

namespace ill {

struct MiParams {
  const u8* w;
  int rows, cols, row_bytes, nsteps;
  const i8* xq;
  const float* xs;
  float* y;
  const float* bias;
  int acc, n;
  uint64_t neg_zeros;    // two floats -0.0
};

template <int NT8, int RW>
struct MiGeom {
  static constexpr int TN = 8 * NT8, THREADS = 32 * RW;
  static constexpr int WPITCH = 176;  // ten chunks of 16 bytes a row's step; 44 words: eight rows x four words on 32 banks
  static constexpr int XPITCH = 144;  // 36 words: ldmatrix's eight rows on 32 banks
  static constexpr int W_BYTES = RW * 16 * WPITCH, X_BYTES = TN * XPITCH, S_BYTES = TN * 16;
  static constexpr int STAGE = W_BYTES + X_BYTES + S_BYTES;
  // CTAs an SM: sixteen warps of 128 registers, or what its shared memory holds
  static constexpr int FIT = 233472 / (3 * STAGE + 1024), PER_SM = FIT < 16 / RW ? FIT : 16 / RW;
};

__device__ __forceinline__ uint64_t mi_mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// A product rounded by itself: a * b + -0.0, with a -0.0 that the compiler does not know.  (It joins a mul.rn.f32x2 and the
// add.rn.f32x2 after it into one fused instruction, .rn or not: other bits than the CPU's two roundings.)
__device__ __forceinline__ uint64_t mi_mul2_rounded(uint64_t a, uint64_t b, uint64_t neg_zeros) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(neg_zeros));
  return d;
}
__device__ __forceinline__ void mi_add2(uint64_t& d, uint64_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ uint64_t mi_pack(float a, float b) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}

template <int NT8, int RW>
__global__ void __launch_bounds__(MiGeom<NT8, RW>::THREADS, MiGeom<NT8, RW>::PER_SM) mm_q8_i8_kernel(const MiParams p) {
  extern __shared__ __align__(128) u8 smem[];
  using C = MiGeom<NT8, RW>;
  constexpr int TN = C::TN;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int ntt = (p.n + TN - 1) / TN;
  const int tok0 = (int)(blockIdx.x % ntt) * TN, row_base = (int)(blockIdx.x / ntt) * (16 * RW) + warp * 16;
  const int nsteps = p.nsteps;
  const bool live = row_base < p.rows;  // a warp whose rows are all past the end only helps to bring the activations
  const u8* wrow0 = p.w + (long long)row_base * p.row_bytes;

  // Weights: four lanes a row, chunks lane % 4, + 4 and + 8 of its 16-byte aligned span (nine or ten chunks).
  const u8* wsrc = wrow0 + (long long)g * p.row_bytes;  // row g's bytes of the step copied next
  const long long w8 = 8ll * p.row_bytes;
  const bool in0 = live && row_base + g < p.rows, in8 = live && row_base + g + 8 < p.rows;
  const uint32_t wdst = (uint32_t)((warp * 16 + g) * C::WPITCH + 16 * t);
  // Activations: eight threads a token's 128 quants, XT tokens at a time; a thread a scale, ST tokens at a time.
  constexpr int XT = C::THREADS / 8, ST = C::THREADS / 4, XJ = (TN + XT - 1) / XT, SJ = (TN + ST - 1) / ST;
  const int xtk = tid >> 3, stk = tid >> 2;
  const i8* xsrc = p.xq + (long long)(tok0 + xtk) * p.cols + 16 * (tid & 7);
  const float* ssrc = p.xs + (long long)(tok0 + stk) * (p.cols / 32) + (tid & 3);
  const uint32_t xdst = (uint32_t)(C::W_BYTES + xtk * C::XPITCH + 16 * (tid & 7));
  // scale of token 2 j + h, block 2 b + o of the step -> float [b][j][o][h]
  const uint32_t sdst = (uint32_t)(C::W_BYTES + C::X_BYTES + 4 * ((((tid & 3) >> 1) * (TN / 2) + (stk >> 1)) * 4 + 2 * (tid & 1) + (stk & 1)));
  int w_step = 0, x_step = 0;  // the steps copied next
  auto fill_w = [&](u8* st) {
    if (w_step < nsteps) {
      auto row = [&](const u8* src, u8* dst) {
        const u8* a = (const u8*)((uintptr_t)src & ~(uintptr_t)15) + 16 * t;
        cp_async16(dst, a);
        cp_async16(dst + 64, a + 64);
        if (t == 0 || (t == 1 && ((uintptr_t)src & 15) > 8)) cp_async16(dst + 128, a + 128);
      };
      if (in0) row(wsrc, st + wdst);
      if (in8) row(wsrc + w8, st + wdst + 8 * C::WPITCH);
    }
    wsrc += 136;
    ++w_step;
  };
  auto fill_x = [&](u8* st) {
    if (x_step < nsteps) {
#pragma unroll
      for (int j = 0; j < XJ; ++j)
        if ((TN % XT == 0 || XT * j + xtk < TN) && tok0 + XT * j + xtk < p.n)
          cp_async16(st + xdst + XT * j * C::XPITCH, xsrc + (long long)XT * j * p.cols);
#pragma unroll
      for (int j = 0; j < SJ; ++j)
        if ((TN % ST == 0 || ST * j + stk < TN) && tok0 + ST * j + stk < p.n)
          cp_async4(st + sdst + 8 * ST * j, ssrc + (long long)ST * j * (p.cols / 32));
    }
    xsrc += 128;
    ssrc += 4;
    ++x_step;
  };

  fill_w(smem);  // the weights do not depend on the previous kernel
  fill_w(smem + C::STAGE);
  pdl_launch_dependents();
  pdl_wait();
  fill_x(smem);
  cp_async_commit();
  fill_x(smem + C::STAGE);
  cp_async_commit();

  uint64_t acc[NT8][2];  // [tile of eight tokens][row g / g + 8]: tokens 2 t and 2 t + 1
#pragma unroll
  for (int nt = 0; nt < NT8; ++nt) acc[nt][0] = acc[nt][1] = 0ull;
  const bool even_off = ((uintptr_t)p.w & 2) == 0;  // a row is a multiple of four bytes: which blocks' quants are word-aligned
  constexpr uint32_t last = 2 * C::STAGE;
  uint32_t use_at = 0, fill_at = last, w_off = (uint32_t)(uintptr_t)wrow0 + (uint32_t)g * p.row_bytes;
  for (int step = 0; step < nsteps; ++step) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // all but the newest: this step's copies are in
    __syncthreads();  // ... everyone's; and everyone is through with the stage refilled next
    fill_w(smem + fill_at);
    fill_x(smem + fill_at);
    cp_async_commit();
    const u8* st = smem + use_at;
    use_at = use_at == last ? 0 : use_at + C::STAGE;
    fill_at = fill_at == last ? 0 : fill_at + C::STAGE;
    const uint32_t o0 = w_off;
    w_off += 136;
    if (!live) continue;
    const u8* r0 = st + (warp * 16 + g) * C::WPITCH + (o0 & 15);
    const u8* r8 = st + (warp * 16 + g + 8) * C::WPITCH + ((o0 + 8u * p.row_bytes) & 15);
    const u8* xl = st + C::W_BYTES + (lane & 7) * C::XPITCH + 16 * (lane >> 3);
    const u8* sl = st + C::W_BYTES + C::X_BYTES + 16 * t;
#pragma unroll
    for (int b2 = 0; b2 < 2; ++b2) {  // blocks 2 b2 and 2 b2 + 1 of the step
      uint32_t a[2][4];
      uint64_t d0[2], d8[2];
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const u8 *q0 = r0 + 34 * (2 * b2 + o) + 2 + 4 * t, *q8 = r8 + 34 * (2 * b2 + o) + 2 + 4 * t;
        if ((o == 1) == even_off) {
          a[o][0] = *(const uint32_t*)q0; a[o][1] = *(const uint32_t*)q8;
          a[o][2] = *(const uint32_t*)(q0 + 16); a[o][3] = *(const uint32_t*)(q8 + 16);
        } else {
          a[o][0] = __funnelshift_r(*(const uint32_t*)(q0 - 2), *(const uint32_t*)(q0 + 2), 16);
          a[o][1] = __funnelshift_r(*(const uint32_t*)(q8 - 2), *(const uint32_t*)(q8 + 2), 16);
          a[o][2] = __funnelshift_r(*(const uint32_t*)(q0 + 14), *(const uint32_t*)(q0 + 18), 16);
          a[o][3] = __funnelshift_r(*(const uint32_t*)(q8 + 14), *(const uint32_t*)(q8 + 18), 16);
        }
        const float f0 = ldh(q0 - 2 - 4 * t), f8 = ldh(q8 - 2 - 4 * t);
        d0[o] = mi_pack(f0, f0);
        d8[o] = mi_pack(f8, f8);
      }
#pragma unroll
      for (int nt = 0; nt < NT8; ++nt) {
        uint32_t x[4];
        ldsm4(x, xl + 8 * nt * C::XPITCH + 64 * b2);
        const ulonglong2 s = *(const ulonglong2*)(sl + (b2 * (TN / 2) + 4 * nt) * 16);
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          const uint64_t xs = o ? s.y : s.x;
          int c[4];
          mma_k32_s8(c, a[o], x[2 * o], x[2 * o + 1]);
          // Q8-ROW-DOT-AT: sum += float(isum) * (d_w * d_x)
          mi_add2(acc[nt][0], mi_mul2_rounded(mi_pack((float)c[0], (float)c[1]), mi_mul2(d0[o], xs), p.neg_zeros));
          mi_add2(acc[nt][1], mi_mul2_rounded(mi_pack((float)c[2], (float)c[3]), mi_mul2(d8[o], xs), p.neg_zeros));
        }
      }
    }
  }
  float v[NT8][4];
#pragma unroll
  for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
    for (int i = 0; i < 2; ++i) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[nt][2 * i]), "=f"(v[nt][2 * i + 1]) : "l"(acc[nt][i]));
  if (!live) return;
#pragma unroll
  for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const long long row = row_base + g + 8 * (i >> 1);
      const int tok = tok0 + 8 * nt + 2 * t + (i & 1);
      if (row < p.rows && tok < p.n) {
        float r = v[nt][i];
        if (p.bias) r += p.bias[row];
        float* yp = p.y + (long long)tok * p.rows + row;
        *yp = p.acc ? *yp + r : r;
      }
    }
}

// Which tile: the one with the least estimated time, steps x (time a step) x (how often the
// SMs are filled).  STEP is the time in us of a step with every SM full, measured on 2048 x 4096 x 4096 tokens.  CTAs that do
// not fill the SMs take less of it, but not in proportion: what counts, over every tile, is how many warps the GPU holds --
// 0.4 of STEP up to 256 warps, 0.55 at 512, 0.8 at 640, all of it at 2368 (sixteen on each of a B200's 148 SMs).  Over eight
// matrices of 128 to 5120 rows at 17, 64, 200, 777 and 4096 tokens it takes the fastest tile or one within 5 % of it for 34
// of the 40; it is furthest off at 200 tokens of 896 rows (x 4864: 51 us against 39, x 896: 9.6 against 7.3), then 128 x 896 x
// 4096 (14.8 against 12.2), 2048 x 4096 x 200 (64 against 54), 5120 x 1536 x 17 and 1536 x 5120 x 200 (15 and 11 %).
struct MiTile {
  float step;
  int rn, tn, threads, per_sm;
  uint32_t smem;
  const void* kernel;
};
template <int NT8, int RW>
static MiTile mi_tile(float step) {
  using C = MiGeom<NT8, RW>;
  return {step, 16 * RW, C::TN, C::THREADS, C::PER_SM, 3u * C::STAGE, (const void*)mm_q8_i8_kernel<NT8, RW>};
}

// The tile for N tokens, its CTAs, and a step's estimated time, us
static const MiTile* mi_pick(int rows, int n, int sms, long long* grid, float* step_us) {
  static const MiTile tiles[] = {
      mi_tile<4, 4>(1.78f), mi_tile<4, 2>(1.66f), mi_tile<6, 4>(2.19f), mi_tile<6, 2>(1.70f),
      mi_tile<8, 4>(2.17f), mi_tile<10, 8>(3.13f), mi_tile<10, 4>(2.49f),
  };
  const MiTile* best = nullptr;
  double best_us = 0.0;
  for (const MiTile& t : tiles) {
    const long long ctas = (long long)((rows + t.rn - 1) / t.rn) * ((n + t.tn - 1) / t.tn), fit = (long long)t.per_sm * sms;
    const double warps = (double)(ctas % fit) * (t.threads / 32);  // of the last, partial filling
    double last = 0.0;
    if (warps > 640.0) last = warps < 2368.0 ? 0.8 + 0.2 * (warps - 640.0) / 1728.0 : 1.0;
    else if (warps > 512.0) last = 0.55 + 0.25 * (warps - 512.0) / 128.0;
    else if (warps > 0.0) last = warps > 256.0 ? 0.4 + 0.15 * (warps - 256.0) / 256.0 : 0.4;
    const double us = t.step * ((double)(ctas / fit) + last);
    if (!best || us < best_us) { best = &t; best_us = us; *grid = ctas; }
  }
  *step_us = (float)best_us;
  return best;
}

float mm_q8_i8_step_us(int rows, int n, int sms) {
  long long grid;
  float us;
  mi_pick(rows, n, sms, &grid, &us);
  return us;
}

int mm_q8_i8(uint64_t w, int rows, int cols, uint64_t xq, uint64_t xs, uint64_t y, uint64_t bias, int acc, int n, int sms, void* stream) {
  MiParams p = {};
  p.w = (const u8*)(uintptr_t)w;
  p.rows = rows;
  p.cols = cols;
  p.row_bytes = cols / 32 * 34;
  p.nsteps = cols / 128;
  p.xq = (const i8*)(uintptr_t)xq;
  p.xs = (const float*)(uintptr_t)xs;
  p.y = (float*)(uintptr_t)y;
  p.bias = (const float*)(uintptr_t)bias;
  p.acc = acc;
  p.n = n;
  p.neg_zeros = 0x8000000080000000ull;
  long long grid;
  float us;
  const MiTile* t = mi_pick(rows, n, sms, &grid, &us);
  if (grid > 0x7fffffffll) return ILL_ERR_TOO_LARGE;
  cudaError_t e = cudaFuncSetAttribute(t->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)t->smem);
  if (e != cudaSuccess) return cuda_fail(e);
  void* args[] = {&p};
  return launch_kernel(t->kernel, dim3((unsigned)grid), dim3((unsigned)t->threads), t->smem, args, (cudaStream_t)stream);
}

}  // namespace ill
