// Dense products for a chunk of tokens (prefill): Y[token][row] = W[row] . X[token] for more than 16 tokens,
// W in Q8_0 / Q4_K / Q6_K blocks, X quantized to Q8_0 (for Q8_0) or Q8_K (for the K formats) -- the same integer
// arithmetic a row of the one-token product does, 16 rows x 8 tokens at a time on the tensor cores' int8 path
// (mma.sync m16n8k32 / m16n8k16), each group's integer sum scaled as the CPU path scales it.
//
// Design.  A CTA of eight warps takes 128 rows x TN tokens (TN = 32, 64 or 128); warp w owns rows 16 w .. 16 w + 15
// against all TN tokens, so a block of weights is unpacked into tensor-core fragments once and used TN / 8 times
// from registers.  The columns go by in steps of 256:
//   * weights: every warp brings its own sixteen rows' blocks (144 / 210 bytes, widened to 16-byte boundaries) by cp.async, four
//     lanes a row;
//   * activations: the step's TN x 256 quants and their scales are brought by all threads with cp.async; a token tile's quants
//     reach the registers as B fragments through ldmatrix.
// Both go through a ring of two to four stages, one __syncthreads a step.  (With a bulk copy a row segment, sixteen a warp and step, the
// copy unit took 2.7 us a step of eight warps whatever the tokens.  us, bulk copies / now: 1024 x 2560 of Q4_K, 17 tokens 26.8 / 18.8, 128
// 33.6 / 19.7, 512 28.4 / 21.9, 2048 65.8 / 62.6; of Q6_K, 512 28.9 / 23.4; 1024 x 5120 of Q6_K, 512 56.3 / 45.1; 9728 x 2560 of Q4_K, 63
// 56.1 / 45.3.)  Bound now by the chain of one warp's step where few rows and tokens leave a warp or two an SM (1.8 us a step: a
// block's fragments, then its products), by instruction issue where they do not.
// This is mmd_kernel, for Q4_K and Q6_K; Q8_0 has kernels of its own (mm_q8.cu, mm_q8_i8.cu).
// Token tiles are the fastest-varying CTA index: the CTAs that share a tile of rows run together and the weights
// come from HBM once.
//
// Replaces mm_q8_mma2 / mm_q4k_mma / mm_q6k_mma behind CMAT-MUL-N for prefill chunks
// (src/cuda-dense.lisp:220-255; src/cuda/dense.cu:885-1100, src/cuda/kquant.cu:316-466).
#include "formats.cuh"
#include "host.h"
#include "mma_i8.cuh"

namespace ill {

constexpr int MD_WARPS = 8, MD_THREADS = 32 * MD_WARPS, MD_MAX_STAGES = 3 /* of mmk_kernel */;
constexpr int MD_XPITCH = 272;  // bytes between the tokens' 256 quants of a step: 68 words, so eight tokens x four words hit 32 banks

struct MdParams {
  const u8* w;
  int rows, cols, row_bytes, nsteps;
  const i8* xq;
  const float* xs;
  const int16_t* xsum;
  float* y;
  const float* bias;
  int acc, n;
  int warps;             // warps a CTA (16 rows each)
  int stages;            // mmd_kernel: stages of weights and activations (2 to 4)
  int pitch;             // bytes between the rows of a staged piece
  uint32_t stage_bytes;
  uint32_t xbuf_bytes, xs_off, xsum_off;  // one activation buffer: its size, where its scales and (Q4_K) sums start
  uint32_t ring_off, part_off;
};

// ---- a step's block(s) of 16 rows as tensor-core fragments, and their use against eight tokens ---------------
// load(): ROW0 / ROW8 = the staged bytes of rows g and g + 8 (g = lane / 4), NB = valid blocks in the step.
// apply(): B = the tile's eight tokens' 256 quants as B fragments (ldsm4 of 64 bytes each); YA / YB the Q8_K scales
// of tokens 8 nt + 2 (lane % 4) and + 1 (Q8_0: SA / SB their eight scales); ACC the lane's four outputs:
// i -> row g + 8 (i / 2), token 8 nt + 2 (lane % 4) + i % 2.
//
// The integer sums are the CPU path's, exactly.  Q6_K's 0..63 quants go in as signed q - 32 (no sums of activations
// needed), each group of 16 a k16 product scaled by its signed scale; Q4_K's mins meet the activations' sums of 16.
// (Carrying Q4_K's scales on the tensor core -- (s & 7) q and (s >> 3) q both fit a byte, so a block is c1 + 8 c2 of
// two accumulating chains, the mins a third -- was measured slower: an int8 mma.sync costs about seven issue slots
// here, so fewer of them with an integer multiply-add a group wins.)
template <int FMT> struct MdFrag;

template <> struct MdFrag<ILL_Q8_0> {
  static constexpr int SB = 272;  // eight blocks of 34 bytes
  static constexpr int SPITCH = 32;  // bytes between the tokens' eight scales of a step
  uint32_t a[8][4];
  float d0[8], d8[8];
  __device__ __forceinline__ void load(const u8* row0, const u8* row8, int lane, int nb) {
    const int t4 = 4 * (lane & 3);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const u8 *r0 = row0 + 34 * b, *r8 = row8 + 34 * b;
      const bool in = b < nb;  // past the row's last block: zeros
      a[b][0] = in ? lds32u(r0 + 2 + t4) : 0u;
      a[b][1] = in ? lds32u(r8 + 2 + t4) : 0u;
      a[b][2] = in ? lds32u(r0 + 18 + t4) : 0u;
      a[b][3] = in ? lds32u(r8 + 18 + t4) : 0u;
      d0[b] = in ? ldh(r0) : 0.0f;
      d8[b] = in ? ldh(r8) : 0.0f;
    }
  }
  __device__ __forceinline__ void apply(const uint32_t (&x)[4][4], const u8* sa, const u8* sb, float, float, float (&acc)[4]) const {
    const float4 xa0 = *(const float4*)sa, xa1 = *(const float4*)(sa + 16), xb0 = *(const float4*)sb, xb1 = *(const float4*)(sb + 16);
    const float da[8] = {xa0.x, xa0.y, xa0.z, xa0.w, xa1.x, xa1.y, xa1.z, xa1.w};
    const float db[8] = {xb0.x, xb0.y, xb0.z, xb0.w, xb1.x, xb1.y, xb1.z, xb1.w};
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const uint32_t bb[2] = {x[b >> 1][2 * (b & 1)], x[b >> 1][2 * (b & 1) + 1]};
      int c[4] = {0, 0, 0, 0};
      mma_k32(c, a[b], bb, false);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        // Q8-ROW-DOT-AT: sum += float(isum) * (d_w * d_x)
        acc[i] = __fadd_rn(acc[i], __fmul_rn((float)c[i], __fmul_rn(i < 2 ? d0[b] : d8[b], (i & 1) ? db[b] : da[b])));
    }
  }
};

template <> struct MdFrag<ILL_Q4_K> {
  static constexpr int SB = 144;
  static constexpr int SPITCH = 48;  // bytes between the tokens' sixteen sums of a step: four tokens' 16-byte reads on different banks
  uint32_t lo[4][4], hi[4][4];
  int sc0[8], sc8[8];
  int mn0[4], mn8[4];  // the mins of groups 2 j and 2 j + 1, each in two bytes: dp2a against the group's two sums of 16
  float d0, m0, d8, m8;
  __device__ __forceinline__ void load(const u8* row0, const u8* row8, int lane, int) {
    const int t4 = 4 * (lane & 3);
    const LdsWords q0(row0 + t4), q8(row8 + t4);
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // 64 weights: groups 2k (low nibbles) and 2k + 1 (high)
      const uint32_t w0 = q0(16 + 32 * k), w1 = q8(16 + 32 * k);
      const uint32_t w2 = q0(32 + 32 * k), w3 = q8(32 + 32 * k);
      lo[k][0] = w0 & 0x0F0F0F0Fu; lo[k][1] = w1 & 0x0F0F0F0Fu; lo[k][2] = w2 & 0x0F0F0F0Fu; lo[k][3] = w3 & 0x0F0F0F0Fu;
      hi[k][0] = (w0 >> 4) & 0x0F0F0F0Fu; hi[k][1] = (w1 >> 4) & 0x0F0F0F0Fu;
      hi[k][2] = (w2 >> 4) & 0x0F0F0F0Fu; hi[k][3] = (w3 >> 4) & 0x0F0F0F0Fu;
      int a, b, ma, mb;
      scale_min_k4(row0 + 4, 2 * k, a, ma); scale_min_k4(row0 + 4, 2 * k + 1, b, mb);
      sc0[2 * k] = a; sc0[2 * k + 1] = b;
      mn0[k] = ma * 0x0101 | (mb * 0x0101) << 16;
      scale_min_k4(row8 + 4, 2 * k, a, ma); scale_min_k4(row8 + 4, 2 * k + 1, b, mb);
      sc8[2 * k] = a; sc8[2 * k + 1] = b;
      mn8[k] = ma * 0x0101 | (mb * 0x0101) << 16;
    }
    d0 = ldh(row0); m0 = ldh(row0 + 2); d8 = ldh(row8); m8 = ldh(row8 + 2);
  }
  // SA / SB: the sixteen sums of 16 (int16) of the two tokens' step
  __device__ __forceinline__ void apply(const uint32_t (&x)[4][4], const u8* sa, const u8* sb, float ya, float yb, float (&acc)[4]) const {
    int isum[4] = {0, 0, 0, 0}, imin[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t b0[2] = {x[k][0], x[k][1]}, b1[2] = {x[k][2], x[k][3]};
      int c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
      mma_k32(c0, lo[k], b0, true);
      mma_k32(c1, hi[k], b1, true);
#pragma unroll
      for (int i = 0; i < 4; ++i) isum[i] += c0[i] * (i < 2 ? sc0[2 * k] : sc8[2 * k]) + c1[i] * (i < 2 ? sc0[2 * k + 1] : sc8[2 * k + 1]);
    }
    // the mins' side: sum over the groups of min * (the group's two sums of 16)
    const int4 a0 = *(const int4*)sa, a1 = *(const int4*)(sa + 16), c0 = *(const int4*)sb, c1 = *(const int4*)(sb + 16);
    const int pa[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const int pb[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int m = i < 2 ? mn0[k] : mn8[k];
        imin[i] = dp2a_hi((i & 1) ? pb[2 * k + 1] : pa[2 * k + 1], m, dp2a_lo((i & 1) ? pb[2 * k] : pa[2 * k], m, imin[i]));
      }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float yd = (i & 1) ? yb : ya;
      // Q4K-ROW-DOT: sum -= (yd * dmin) * imin; sum += (yd * d) * isum
      const float s = __fsub_rn(acc[i], __fmul_rn(__fmul_rn(yd, i < 2 ? m0 : m8), (float)imin[i]));
      acc[i] = __fadd_rn(s, __fmul_rn(__fmul_rn(yd, i < 2 ? d0 : d8), (float)isum[i]));
    }
  }
};

// four 6-bit values 0..63, a byte each -> the signed bytes value - 32
__device__ __forceinline__ uint32_t q6_signed(uint32_t v) {
  const uint32_t t = v ^ 0x20202020u, s = t & 0x20202020u;  // t = value - 32 modulo 64; s: its sign (bit 5)
  return t | (s << 1) | (s << 2);
}

template <> struct MdFrag<ILL_Q6_K> {
  static constexpr int SB = 210;
  static constexpr int SPITCH = 0;
  uint32_t q[16][2];  // [group of 16][row g / g + 8]: the lane's four quants as signed bytes -32..31
  int sc0[16], sc8[16];
  float d0, d8;
  // every second block starts on a word, in all rows alike where they lie a multiple of four bytes apart
  __device__ __forceinline__ void load(const u8* row0, const u8* row8, int lane, int) {
    if (__all_sync(0xffffffffu, (((uintptr_t)row0 | (uintptr_t)row8) & 3) == 0)) load_al<true>(row0, row8, lane);
    else load_al<false>(row0, row8, lane);
  }
  template <bool W>
  __device__ __forceinline__ void load_al(const u8* row0, const u8* row8, int lane) {
    const RowWords<W> w0s(row0), w8s(row8), q0(row0 + 4 * (lane & 3)), q8(row8 + 4 * (lane & 3));
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int is = 0; is < 2; ++is) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const RowWords<W>& row = r ? q8 : q0;
          const uint32_t A = row(64 * c + 16 * is), B = row(64 * c + 32 + 16 * is), H = row(128 + 32 * c + 16 * is);
          // run RUN of the half covers weights 128 c + 32 run ..: its group of 16 is 8 c + 2 run + is
          q[8 * c + 0 + is][r] = q6_signed((A & 0x0F0F0F0Fu) | ((H << 4) & 0x30303030u));
          q[8 * c + 2 + is][r] = q6_signed((B & 0x0F0F0F0Fu) | ((H << 2) & 0x30303030u));
          q[8 * c + 4 + is][r] = q6_signed(((A >> 4) & 0x0F0F0F0Fu) | (H & 0x30303030u));
          q[8 * c + 6 + is][r] = q6_signed(((B >> 4) & 0x0F0F0F0Fu) | ((H >> 2) & 0x30303030u));
        }
      }
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint32_t w0 = w0s(192 + 4 * w), w8 = w8s(192 + 4 * w);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sc0[4 * w + j] = (int)(signed char)(w0 >> (8 * j));
        sc8[4 * w + j] = (int)(signed char)(w8 >> (8 * j));
      }
    }
    d0 = ldh(row0 + 208); d8 = ldh(row8 + 208);
  }
  __device__ __forceinline__ void apply(const uint32_t (&x)[4][4], const u8*, const u8*, float ya, float yb, float (&acc)[4]) const {
    int isum[4] = {0, 0, 0, 0};
#pragma unroll
    for (int grp = 0; grp < 16; ++grp) {  // group GRP's 16 weights face the token's 16 quants at 16 grp
      int cc[4] = {0, 0, 0, 0};
      mma_k16_s8(cc, q[grp][0], q[grp][1], x[grp >> 2][grp & 3], false);
#pragma unroll
      for (int i = 0; i < 4; ++i) isum[i] += cc[i] * (i < 2 ? sc0[grp] : sc8[grp]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      // Q6K-ROW-DOT: sum += (d * yd) * float(sum over the groups of scale * dot(q - 32, x))
      acc[i] = __fadd_rn(acc[i], __fmul_rn(__fmul_rn(i < 2 ? d0 : d8, (i & 1) ? yb : ya), (float)isum[i]));
  }
};

// A CTA's tile BLOCK of a matrix
template <int FMT, int NT8>
__device__ __forceinline__ void md_tile(const MdParams& p, int block, u8* smem) {
  constexpr int TN = 8 * NT8, SB = MdFrag<FMT>::SB, MD_SPITCH = MdFrag<FMT>::SPITCH;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int ntt = (p.n + TN - 1) / TN, nthreads = blockDim.x;  // eight warps, or fewer when the matrix has few rows
  const int tok0 = block % ntt * TN, row_base = block / ntt * (nthreads / 2) + warp * 16;
  const int nsteps = p.nsteps, stages = p.stages;
  const bool live = row_base < p.rows;  // a warp whose rows are all past the end only helps to bring the activations
  u8* ring = smem + p.ring_off + (size_t)warp * stages * p.stage_bytes;

  int w_step = 0, w_at = 0, x_step = 0, x_at = 0;  // the steps brought next, their stages
  auto fill_w = [&]() {  // the warp's sixteen rows, four lanes a row segment
    if (live && w_step < nsteps) {
      u8* st = ring + (size_t)w_at * p.stage_bytes;
      const u8* src = p.w + (long long)(row_base + g) * p.row_bytes + (long long)w_step * SB;
#pragma unroll
      for (int h = 0; h < 16; h += 8)
        if (row_base + h + g < p.rows)
          copy_segment<(SB + 30) / 16>(st + (size_t)(h + g) * p.pitch, src + (long long)h * p.row_bytes, SB, t);
    }
    ++w_step;
    w_at = w_at + 1 == stages ? 0 : w_at + 1;
  };
  auto fill_x = [&]() {  // all threads
    if (x_step < nsteps) {
      u8* xb = smem + (size_t)x_at * p.xbuf_bytes;
      const int c0 = 256 * x_step;
      for (int i = tid; i < TN * 16; i += nthreads) {
        const int tk = i >> 4, ch = i & 15;
        if (tok0 + tk < p.n) cp_async16(xb + tk * MD_XPITCH + 16 * ch, p.xq + (long long)(tok0 + tk) * p.cols + c0 + 16 * ch);
      }
      for (int i = tid; i < TN; i += nthreads)
        if (tok0 + i < p.n) cp_async4(xb + p.xs_off + 4 * i, p.xs + (long long)(tok0 + i) * nsteps + x_step);
      if constexpr (FMT == ILL_Q4_K) {
        for (int i = tid; i < TN * 2; i += nthreads) {
          const int tk = i >> 1, ch = i & 1;
          if (tok0 + tk < p.n)
            cp_async16(xb + p.xsum_off + tk * MD_SPITCH + 16 * ch, p.xsum + (long long)(tok0 + tk) * (p.cols / 16) + 16 * x_step + 8 * ch);
        }
      }
    }
    ++x_step;
    x_at = x_at + 1 == stages ? 0 : x_at + 1;
  };

  // the activation buffers start as zeros: the tokens past the last stay so
  for (uint32_t i = 16u * tid; i < stages * p.xbuf_bytes; i += 16u * nthreads) *(uint4*)(smem + i) = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (int s = 0; s < stages - 1; ++s) fill_w();  // the weights do not depend on the previous kernel
  pdl_launch_dependents();
  pdl_wait();
  for (int s = 0; s < stages - 1; ++s) {          // a group a step (the weights are in the first)
    fill_x();
    cp_async_commit();
  }

  float acc[NT8][4];
#pragma unroll
  for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[nt][i] = 0.0f;
  int at = 0;
  for (int step = 0; step < nsteps; ++step) {
    // all but the newer steps' copies: this step's are in
    if (stages == 4) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else if (stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else cp_async_wait_all();
    __syncthreads();  // ... everyone's; and everyone is through with the stages of the step before, which are filled next
    fill_w();
    fill_x();
    cp_async_commit();
    const u8* piece = ring + (size_t)at * p.stage_bytes;
    const u8* xb = smem + (size_t)at * p.xbuf_bytes;
    at = at + 1 == stages ? 0 : at + 1;
    if (!live) continue;
    MdFrag<FMT> f;
    {
      // a row's bytes start where its block starts inside the 16-byte aligned span that was copied
      const long long o0 = (long long)(row_base + g) * p.row_bytes + (long long)step * SB;
      const long long o8 = o0 + 8ll * p.row_bytes;
      const u8* row0 = piece + (size_t)g * p.pitch + (((uintptr_t)p.w + o0) & 15);
      const u8* row8 = piece + (size_t)(g + 8) * p.pitch + (((uintptr_t)p.w + o8) & 15);
      f.load(row0, row8, lane, 8);
    }
    const u8* xl = xb + (lane & 7) * MD_XPITCH + 16 * (lane >> 3);  // this lane's row of the four matrices ldsm4 reads
    const u8* scl = xb + p.xsum_off + 2 * t * MD_SPITCH;  // Q4_K: the sixteen sums of 16 of token 2 t (+ 8 nt)
    const float* ys = (const float*)(xb + p.xs_off) + 2 * t;
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt) {
      uint32_t x[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) ldsm4(x[j], xl + 8 * nt * MD_XPITCH + 64 * j);
      f.apply(x, scl + 8 * nt * MD_SPITCH, scl + (8 * nt + 1) * MD_SPITCH, ys[8 * nt], ys[8 * nt + 1], acc[nt]);
    }
  }
  if (!live) return;
#pragma unroll
  for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const long long row = row_base + g + 8 * (i >> 1);
      const int tok = tok0 + 8 * nt + 2 * t + (i & 1);
      if (row < p.rows && tok < p.n) {
        float v = acc[nt][i];
        if (p.bias) v += p.bias[row];
        float* yp = p.y + (long long)tok * p.rows + row;
        *yp = p.acc ? *yp + v : v;
      }
    }
}

// MINB = 2 (token tiles of 64): a thread stays within 128 registers and two CTAs share an SM
template <int FMT, int NT8, int MINB>
__global__ void __launch_bounds__(MD_THREADS, MINB) mmd_kernel(const MdParams p) {
  extern __shared__ __align__(128) u8 smem[];
  md_tile<FMT, NT8>(p, (int)blockIdx.x, smem);
}

// Two or three matrices that share the activations (a chunk's K and V), their tiles one matrix after another: alone, 1024 rows of 512
// tokens are a CTA or two of four warps an SM.  us, a launch each / one, 1024 x 2560
// of Q4_K and of Q6_K: 17 tokens 31.8 / 16.6, 64 33.8 / 17.4, 256 40.1 / 25.7, 1024 96 / 66.
constexpr int MD_MATS = 3;
struct MdJoint {
  MdParams m[MD_MATS];
  int first[MD_MATS];   // its first CTA (of matrices that are not there: beyond the last)
  int q6[MD_MATS];      // Q6_K, not Q4_K
};
template <int NT8, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) mmd_joint_kernel(const __grid_constant__ MdJoint j) {
  extern __shared__ __align__(128) u8 smem[];
  const int block = (int)blockIdx.x, i = (block >= j.first[1]) + (block >= j.first[2]);
  if (j.q6[i]) md_tile<ILL_Q6_K, NT8>(j.m[i], block - j.first[i], smem);
  else md_tile<ILL_Q4_K, NT8>(j.m[i], block - j.first[i], smem);
}

// ---- up to sixteen tokens of rows too long for mvt.cu to keep the activations resident ------------------------
// A 16-row tile's column steps are dealt to eight warps (warp w takes steps w, w + 8, ...), in one CTA or, two each, in the four CTAs of a
// cluster: each warp streams its own steps' weights (its ring of three stages) AND its own steps' activations (two buffers of its own), all
// by 16-byte cp.async of its lanes (Q6_K 5120 x 17408, 4 tokens: 40 us; 59 with a bulk copy a row segment), so the warps
// never wait for one another until the end, where their partial sums are read, from the four CTAs' shared memory, in warp order.  A matrix
// of few rows and many columns (5120 x 17408) thus fills the machine where the chunk kernel above would run two warps a CTA
// through all 68 steps.  Eight warps in one CTA take most of an SM's shared memory, so 160 tiles are two rounds on 148
// SMs and 320 three; CTAs of two warps spread over the SMs to a quarter of a tile, but meet through the cluster (mk_cluster says which).
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// the float that CTA RANK of the cluster has at P of its shared memory
__device__ __forceinline__ float ld_cluster(const float* p, int rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

constexpr int MK_PP = 20;  // floats between the tokens of a partial sum: a fragment's stores lie on different banks

template <int FMT, int NT8, int CTAS /* of a tile: a cluster, where more than one */>
__global__ void __launch_bounds__(MD_THREADS / CTAS, CTAS == 1 ? 1 : NT8 == 1 ? 8 : 0) mmk_kernel(const MdParams p) {
  extern __shared__ __align__(128) u8 smem[];
  constexpr int WARPS = MD_WARPS / CTAS;
  constexpr int TN = 8 * NT8, SB = MdFrag<FMT>::SB, SP = MdFrag<FMT>::SPITCH;
  constexpr bool KQ = FMT != ILL_Q8_0;
  const int tid = threadIdx.x, lane = tid & 31, cwarp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int rank = (int)(blockIdx.x % CTAS), warp = rank * WARPS + cwarp;
  const int ntt = (p.n + TN - 1) / TN;
  const int tok0 = (int)(blockIdx.x / CTAS % ntt) * TN, row_base = (int)(blockIdx.x / CTAS / ntt) * 16;
  const int nsteps = p.nsteps;
  u8* xw = smem + (size_t)cwarp * 2 * p.xbuf_bytes;  // this warp's two activation buffers
  u8* ring = smem + p.ring_off + (size_t)cwarp * MD_MAX_STAGES * p.stage_bytes;
  float* part = (float*)(smem + p.part_off);        // [this CTA's warps][TN][MK_PP: 16 rows]

  auto fill_w = [&](int k) {  // this warp's K-th step's weights -> stage k % 3 (a group of cp.async, possibly empty)
    const int step = warp + MD_WARPS * k;
    if (step < nsteps) {
      const uint32_t len = (uint32_t)min(SB, p.row_bytes - step * SB);
      u8* st = ring + (size_t)(k % MD_MAX_STAGES) * p.stage_bytes;
#pragma unroll
      for (int h = 0; h < 16; h += 8)
        if (row_base + h + g < p.rows)
          copy_segment<(SB + 30) / 16>(st + (size_t)(h + g) * p.pitch,
                                       p.w + (long long)(row_base + h + g) * p.row_bytes + (long long)step * SB, len, t);
    }
    cp_async_commit();
  };
  auto fill_x = [&](int k) {  // this warp's K-th step -> its buffer k % 2 (a group of cp.async, possibly empty)
    const int step = warp + MD_WARPS * k;
    if (step < nsteps) {
      u8* xb = xw + (size_t)(k & 1) * p.xbuf_bytes;
      const int c0 = 256 * step;
      for (int i = lane; i < TN * 16; i += 32) {
        const int tk = i >> 4, ch = i & 15;
        if (tok0 + tk < p.n && c0 + 16 * ch < p.cols)
          cp_async16(xb + tk * MD_XPITCH + 16 * ch, p.xq + (long long)(tok0 + tk) * p.cols + c0 + 16 * ch);
      }
      if constexpr (KQ) {
        for (int i = lane; i < TN; i += 32)
          if (tok0 + i < p.n) cp_async4(xb + p.xs_off + 4 * i, p.xs + (long long)(tok0 + i) * nsteps + step);
        if constexpr (FMT == ILL_Q4_K) {
          for (int i = lane; i < TN * 2; i += 32) {
            const int tk = i >> 1, ch = i & 1;
            if (tok0 + tk < p.n)
              cp_async16(xb + p.xsum_off + tk * SP + 16 * ch, p.xsum + (long long)(tok0 + tk) * (p.cols / 16) + 16 * step + 8 * ch);
          }
        }
      } else {
        for (int i = lane; i < TN * 2; i += 32) {
          const int tk = i >> 1, ch = i & 1;
          if (tok0 + tk < p.n && c0 + 128 * ch < p.cols)
            cp_async16(xb + p.xs_off + tk * SP + 16 * ch, p.xs + (long long)(tok0 + tk) * (p.cols / 32) + 8 * step + 4 * ch);
        }
      }
    }
    cp_async_commit();
  };

  // the warp's activation buffers start as zeros (tokens past the last, columns past a Q8_0 row's end)
  for (uint32_t i = 16u * lane; i < 2u * p.xbuf_bytes; i += 16u * 32u) *(uint4*)(xw + i) = make_uint4(0, 0, 0, 0);
  __syncwarp();
  for (int s = 0; s < MD_MAX_STAGES; ++s) fill_w(s);  // the weights do not depend on the previous kernel
  pdl_launch_dependents();
  pdl_wait();
  fill_x(0);

  float acc[NT8][4];
#pragma unroll
  for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[nt][i] = 0.0f;
  for (int k = 0; warp + MD_WARPS * k < nsteps; ++k) {
    const int step = warp + MD_WARPS * k;
    fill_x(k + 1);                                          // the other buffer: its readers are through (the __syncwarp below)
    // step k is in: all but that group and, after the first step, the weights asked for at the end of the last one
    if (k == 0) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncwarp();
    const int s = k % MD_MAX_STAGES;
    MdFrag<FMT> f;
    {
      const u8* piece = ring + (size_t)s * p.stage_bytes;
      const long long o0 = (long long)(row_base + g) * p.row_bytes + (long long)step * SB;
      const long long o8 = o0 + 8ll * p.row_bytes;
      const u8* row0 = piece + (size_t)g * p.pitch + (((uintptr_t)p.w + o0) & 15);
      const u8* row8 = piece + (size_t)(g + 8) * p.pitch + (((uintptr_t)p.w + o8) & 15);
      f.load(row0, row8, lane, min(8, (p.cols - 256 * step) / 32));
    }
    __syncwarp();
    fill_w(k + MD_MAX_STAGES);
    const u8* xb = xw + (size_t)(k & 1) * p.xbuf_bytes;
    const u8* xl = xb + (lane & 7) * MD_XPITCH + 16 * (lane >> 3);
    const u8* scl = xb + (FMT == ILL_Q4_K ? p.xsum_off : p.xs_off) + 2 * t * SP;
    const float* ys = (const float*)(xb + p.xs_off) + 2 * t;
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt) {
      uint32_t x[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) ldsm4(x[j], xl + 8 * nt * MD_XPITCH + 64 * j);
      float ya = 0.0f, yb = 0.0f;
      if constexpr (KQ) { ya = ys[8 * nt]; yb = ys[8 * nt + 1]; }
      f.apply(x, scl + 8 * nt * SP, scl + (8 * nt + 1) * SP, ya, yb, acc[nt]);
    }
    __syncwarp();  // every lane is through with buffer k % 2 before the next iteration's copies into it are issued
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // the warps' partial sums meet: thread (row, token) adds them in warp order, a quarter of the tile's in each CTA
#pragma unroll
  for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) part[(cwarp * TN + 8 * nt + 2 * t + (i & 1)) * MK_PP + g + 8 * (i >> 1)] = acc[nt][i];
  if constexpr (CTAS > 1) cluster_sync(); else __syncthreads();
#pragma unroll
  for (int o = rank * (16 * TN / CTAS) + tid; o < (rank + 1) * (16 * TN / CTAS); o += 32 * WARPS) {
    const long long row = row_base + (o & 15);
    const int tok = tok0 + (o >> 4), at = (o >> 4) * MK_PP + (o & 15);
    if (row < p.rows && tok < p.n) {
      float v = 0.0f;
#pragma unroll
      for (int w = 0; w < MD_WARPS; ++w) v = __fadd_rn(v, CTAS > 1 ? ld_cluster(part + w % WARPS * TN * MK_PP + at, w / WARPS) : part[w * TN * MK_PP + at]);
      if (p.bias) v += p.bias[row];
      float* yp = p.y + (long long)tok * p.rows + row;
      *yp = p.acc ? *yp + v : v;
    }
  }
  if constexpr (CTAS > 1) cluster_sync();  // nobody's partial sums go before everyone has read them
}
constexpr int MK_CTAS = 4;

template <int FMT>
static int mmd_launch(const MdParams& p, int tn, size_t smem, int grid, cudaStream_t st) {
  const void* k = tn == 32 ? (const void*)mmd_kernel<FMT, 4, 1> : tn == 64 ? (const void*)mmd_kernel<FMT, 8, 2> : (const void*)mmd_kernel<FMT, 16, 1>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e);
  MdParams pp = p;
  void* args[] = {&pp};
  return launch_kernel(k, dim3(grid), dim3(32 * p.warps), smem, args, st);
}

// The chunk product on the tensor cores of up to three matrices that share the activations, for the formats and layouts it is written
// for; ILL_ERR_UNSUPPORTED otherwise (the caller then takes the products one by one, one by the token loop of the CUDA-core kernel).
int mmd_try(int nmat, const int* fmts, const uint64_t* w, const int* rows, int cols, uint64_t xq, uint64_t xs, uint64_t xsum, const uint64_t* y,
            const uint64_t* bias, int acc, int n, void* stream) {
  if (fmts[0] == ILL_Q8_0) {
    for (int i = 1; i < nmat; ++i)
      if (fmts[i] != ILL_Q8_0) return ILL_ERR_UNSUPPORTED;
    return mm_q8_try(nmat, w, rows, cols, xq, xs, y, bias, acc, n, stream);
  }
  bool q4 = false;
  for (int i = 0; i < nmat; ++i) {
    if (fmts[i] != ILL_Q4_K && fmts[i] != ILL_Q6_K) return ILL_ERR_UNSUPPORTED;
    q4 = q4 || fmts[i] == ILL_Q4_K;
  }
  if (n < 2) return ILL_ERR_UNSUPPORTED;
  // 16-byte pieces of the activations are copied as they lie: the quants of a step, Q4_K's sixteen sums
  if ((xq & 15) || cols % 256) return ILL_ERR_UNSUPPORTED;
  if (q4 && (xsum & 15)) return ILL_ERR_UNSUPPORTED;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  // Tokens a CTA: 128 amortize a block's unpacking best (one CTA of eight warps an SM, up to 255 registers); tiles
  // of 64 keep a thread within 128 registers so that two CTAs share an SM -- measured equal to slower where both
  // fill the machine, so they are for chunks of up to 64 tokens and for matrices with so few rows that tiles of 128
  // would leave the SMs with fewer than eight warps each; 32 below that.
  long long tiles16 = 0;
  for (int i = 0; i < nmat; ++i) tiles16 += (rows[i] + 15) / 16;
  int tn = n <= 32 ? 32 : n <= 64 ? 64 : 128;
  while (tn > 32 && tiles16 * ((n + tn - 1) / tn) < 8ll * sms) tn >>= 1;
  // Warps a CTA: eight (128 rows), or four when that would leave SMs without a CTA (few rows of many columns).  (Fewer than four bring
  // the activations too slowly, 64 to 1536 rows of 1024 to 17408 columns at 17 to 512 tokens: 256 x 2560 x 64 tokens of Q4_K with one, two,
  // four, eight warps 18.4 / 16.1 / 15.6 / 22.4 us, 1024 x 5120 x 128 35.6 / 33.0 / 30.2 / 43.4, 64 x 17408 x 17 112 / 99 / 97 / 97; four the
  // fastest of them or within 2 %.)
  const int ntt = (n + tn - 1) / tn;
  int warps = MD_WARPS;
  auto ctas = [&](int m) { return (long long)((rows[m] + 16 * warps - 1) / (16 * warps)) * ntt; };
  auto all_ctas = [&] {
    long long c = 0;
    for (int i = 0; i < nmat; ++i) c += ctas(i);
    return c;
  };
  while (warps > 4 && all_ctas() < sms) warps >>= 1;
  // Several matrices go in one launch where its CTAs run side by side: two of four warps, or of 64 tokens, fit an SM, and with two
  // stages and 128 registers four of four warps (a launch each / two CTAs an SM / four, us: 1024 x 2560 of Q4_K and of Q6_K, 256 tokens
  // 43 / 25.7 / 34, 512 45.0 / 47.2 / 42.6; 2 x 1024 x 5120 of Q6_K, 512 91 / 91 / 79).  Beyond that the SMs are full with a launch each.
  if (nmat > 1 && tn == 32 && all_ctas() > sms) warps = 4;
  const bool four = nmat > 1 && tn == 32 && warps == 4 && all_ctas() > 2ll * sms;
  if (nmat > 1 && all_ctas() > (long long)sms * (four ? 4 : warps <= 4 || tn == 64 ? 2 : 1)) return ILL_ERR_UNSUPPORTED;
  MdJoint jt = {};
  size_t smem = 0;
  for (int i = 0; i < nmat; ++i) {
    const int bw = fmt_block_weights(fmts[i]), bb = fmt_block_bytes(fmts[i]);
    MdParams& p = jt.m[i];
    p.w = (const u8*)(uintptr_t)w[i];
    p.rows = rows[i];
    p.cols = cols;
    p.row_bytes = cols / bw * bb;
    p.nsteps = cols / 256;
    p.xq = (const i8*)(uintptr_t)xq;
    p.xs = (const float*)(uintptr_t)xs;
    p.xsum = (const int16_t*)(uintptr_t)xsum;
    p.y = (float*)(uintptr_t)y[i];
    p.bias = bias ? (const float*)(uintptr_t)bias[i] : nullptr;
    p.acc = acc;
    p.n = n;
    p.warps = warps;
    // a row's step: its 16-byte aligned span (a block is read from its stage once a step, so the rows' pitch need not
    // spread them over the banks); 16 bytes after the last row for the unaligned loads' second word
    p.pitch = (bb + 15 + 15) / 16 * 16;
    p.stage_bytes = (uint32_t)(16 * p.pitch + 16);
    uint32_t off = (uint32_t)tn * MD_XPITCH;
    p.xs_off = off;
    off += 4u * tn;
    off = (off + 15) / 16 * 16;
    p.xsum_off = off;
    if (fmts[i] == ILL_Q4_K) off += (uint32_t)tn * MdFrag<ILL_Q4_K>::SPITCH;
    p.xbuf_bytes = (off + 127) / 128 * 128;
    // stages of weights and activations: four, three where that is all that fits, two where two CTAs share an SM
    const uint32_t stage = (uint32_t)p.warps * p.stage_bytes + p.xbuf_bytes;
    p.stages = tn == 64 || four ? 2 : 226 * 1024 / stage < 4 ? 226 * 1024 / stage : 4;
    p.ring_off = p.stages * p.xbuf_bytes;
    if (p.stages * (size_t)stage > smem) smem = p.stages * (size_t)stage;
    jt.q6[i] = fmts[i] == ILL_Q6_K;
  }
  if (smem > 226 * 1024) return ILL_ERR_UNSUPPORTED;
  const long long grid = all_ctas();
  if (grid > 0x7fffffffll) return ILL_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  if (nmat == 1) return fmts[0] == ILL_Q4_K ? mmd_launch<ILL_Q4_K>(jt.m[0], tn, smem, (int)grid, st) : mmd_launch<ILL_Q6_K>(jt.m[0], tn, smem, (int)grid, st);
  for (int i = 1; i < MD_MATS; ++i) jt.first[i] = i < nmat ? jt.first[i - 1] + (int)ctas(i - 1) : 0x7fffffff;
  const void* k = four ? (const void*)mmd_joint_kernel<4, 128, 4> : tn == 32 ? (const void*)mmd_joint_kernel<4, MD_THREADS, 1>
                  : tn == 64 ? (const void*)mmd_joint_kernel<8, MD_THREADS, 2> : (const void*)mmd_joint_kernel<16, MD_THREADS, 1>;
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e);
  void* args[] = {&jt};
  return launch_kernel(k, dim3((unsigned)grid), dim3(32 * warps), smem, args, st);
}

template <int FMT>
static int mmk_launch(const MdParams& p, int tn, int ctas, size_t smem, int grid, cudaStream_t st) {
  const void* k = ctas == 1 ? tn == 8 ? (const void*)mmk_kernel<FMT, 1, 1> : (const void*)mmk_kernel<FMT, 2, 1>
                            : tn == 8 ? (const void*)mmk_kernel<FMT, 1, MK_CTAS> : (const void*)mmk_kernel<FMT, 2, MK_CTAS>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e);
  MdParams pp = p;
  void* args[] = {&pp};
  return launch_kernel(k, dim3(grid), dim3(32 * MD_WARPS / ctas), smem, args, st, ctas);
}

// Whether a tile goes to a cluster of four CTAs and not to one.  Four SMs work on a tile where there are few, up to two sevenths of the
// SMs, and quarters of a tile fill a last round that is less than 45 % full; else the cluster's meeting, and SMs with CTAs of several
// tiles, cost more than they give.  Two CTAs a tile of Q4_K fit an SM with up to eight tokens, and with more Q8_0's cluster kernel is the
// slower: those take clusters for few tiles only.  us, one CTA / a cluster, 17408 columns, weights cold: Q6_K, 16 tokens, 16 tiles
// 15.2 / 10.6, 36 15.4 / 13.2, 64 15.6 / 18.8, 148 17.8 / 23.5, 149 30.3 / 23.6, 200 32.5 / 31.2, 280 34.3 / 38.1, 310 48.7 / 41.4;
// Q4_K, 4 tokens, 16 tiles 12.4 / 9.6, 148 12.9 / 19.6, 280 20.6 / 23.1; Q8_0, 16 tokens, 11008 columns, 16 tiles 19.8 / 18.0, 148
// 22.6 / 40.5, 280 44.2 / 47.1.
static bool mk_cluster(int fmt, int tn, long long tiles, int sms) {
  if (tiles <= sms) return 7 * tiles <= 2 * sms;
  if (fmt == ILL_Q4_K ? tn == 8 : fmt == ILL_Q8_0 && tn == 16) return false;
  const long long last = (tiles - 1) % sms + 1;
  return 20 * last <= 9 * sms;
}

// Up to sixteen tokens with the columns dealt to a CTA's warps (mmk_kernel): for rows of many columns.
int mmk_try(int fmt, uint64_t w, int rows, int cols, uint64_t xq, uint64_t xs, uint64_t xsum, uint64_t y, uint64_t bias, int acc,
            int n, void* stream) {
  if (fmt != ILL_Q8_0 && fmt != ILL_Q4_K && fmt != ILL_Q6_K) return ILL_ERR_UNSUPPORTED;
  if (n < 2 || n > 16) return ILL_ERR_UNSUPPORTED;
  const bool kq = fmt != ILL_Q8_0;
  if (xq & 15) return ILL_ERR_UNSUPPORTED;
  if (kq ? cols % 256 != 0 : ((xs & 15) || cols % 128)) return ILL_ERR_UNSUPPORTED;
  if (fmt == ILL_Q4_K && (xsum & 15)) return ILL_ERR_UNSUPPORTED;
  const int bw = fmt_block_weights(fmt), bb = fmt_block_bytes(fmt);
  MdParams p = {};
  p.w = (const u8*)(uintptr_t)w;
  p.rows = rows;
  p.cols = cols;
  p.row_bytes = cols / bw * bb;
  p.nsteps = (cols + 255) / 256;
  if (p.nsteps < 2 * MD_WARPS) return ILL_ERR_UNSUPPORTED;  // too few steps to deal out
  p.xq = (const i8*)(uintptr_t)xq;
  p.xs = (const float*)(uintptr_t)xs;
  p.xsum = (const int16_t*)(uintptr_t)xsum;
  p.y = (float*)(uintptr_t)y;
  p.bias = (const float*)(uintptr_t)bias;
  p.acc = acc;
  p.n = n;
  p.warps = MD_WARPS;
  const int tn = n <= 8 ? 8 : 16;
  const int sb = fmt == ILL_Q8_0 ? 272 : bb;
  p.pitch = (sb + 15 + 15) / 16 * 16;
  p.stage_bytes = (uint32_t)(16 * p.pitch + 16);
  uint32_t off = (uint32_t)tn * MD_XPITCH;
  p.xs_off = off;
  off += kq ? 4u * tn : (uint32_t)tn * MdFrag<ILL_Q8_0>::SPITCH;
  off = (off + 15) / 16 * 16;
  p.xsum_off = off;
  if (fmt == ILL_Q4_K) off += (uint32_t)tn * MdFrag<ILL_Q4_K>::SPITCH;
  p.xbuf_bytes = (off + 127) / 128 * 128;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  const int ctas = mk_cluster(fmt, tn, (rows + 15) / 16, sms) ? MK_CTAS : 1, warps = MD_WARPS / ctas;
  p.ring_off = 2 * warps * p.xbuf_bytes;
  p.part_off = (uint32_t)((p.ring_off + (size_t)warps * MD_MAX_STAGES * p.stage_bytes + 127) / 128 * 128);
  const size_t smem = p.part_off + (size_t)warps * MK_PP * tn * 4;
  const long long grid = ctas * (long long)((rows + 15) / 16) * ((n + tn - 1) / tn);
  if (grid > 0x7fffffffll) return ILL_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  switch (fmt) {
    case ILL_Q8_0: return mmk_launch<ILL_Q8_0>(p, tn, ctas, smem, (int)grid, st);
    case ILL_Q4_K: return mmk_launch<ILL_Q4_K>(p, tn, ctas, smem, (int)grid, st);
    default: return mmk_launch<ILL_Q6_K>(p, tn, ctas, smem, (int)grid, st);
  }
}

}  // namespace ill
