// mtblock.cuh -- one block of sixteen weight rows against a few tokens on the tensor cores' int8 path (mma.sync): the tokens'
// activations in shared memory, and the 2-bit formats' blocks.  Shared by the several-token product (mvt.cu, which has the other
// formats' blocks) and the experts' (mve.cu).
#pragma once
#include "formats.cuh"
#include "mma_i8.cuh"

namespace ill {

// The tokens' activations in shared memory.
struct MtX {
  const i8* q;        // token t's quants at q + t * stride
  int stride;
  const float* s;     // [t][scales a token]
  const u8* bs;       // K formats, [t][block][32]: the block's sixteen sums of 16 in two bytes each: sum >> 4 (signed), then sum & 15
  int nsc, nb;
};
// Bytes between the tokens' quants: the eight tokens of a fragment's request lie on different banks (rows of 16 bytes that ldmatrix
// reads; IQ2_XXS: eight bytes a lane, half a warp at a time).
__host__ __device__ constexpr int mt_x_stride(int fmt, int cols) { return cols + (fmt == ILL_IQ2_XXS ? 32 : 16); }
// B fragments of 64 columns from K on against tokens 8 NT .. 8 NT + 7: r[0], r[1] the first 32 columns', r[2], r[3] the others'; of k16
// products one each
__device__ __forceinline__ void xfrag(uint32_t (&r)[4], const MtX& x, int nt, int k, int lane) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(x.q + (size_t)(8 * nt + (lane & 7)) * x.stride + k + 16 * (lane >> 3))));
}
// Eight sums of 16 (V: two a word) as they are staged: the sums' high parts (sum >> 4, signed), a byte each, and their low parts.
__device__ __forceinline__ void split_sums(const uint4& v, uint2& hi, uint2& lo) {
  // bits 4..11 of the four 16-bit sums, a byte each; bits 0..3
  hi = make_uint2(__byte_perm(v.x >> 4, v.y >> 4, 0x6420), __byte_perm(v.z >> 4, v.w >> 4, 0x6420));
  lo = make_uint2(__byte_perm(v.x, v.y, 0x6420) & 0x0f0f0f0fu, __byte_perm(v.z, v.w, 0x6420) & 0x0f0f0f0fu);
}

// 16 / 4 bytes global -> shared, asynchronously, or zeros
__device__ __forceinline__ void cp_async16_or_zero(void* dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4_or_zero(void* dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 4 : 0) : "memory");
}

// ---- the 2-bit formats: addresses in shared memory as 32-bit numbers, worked out once a lane ---------------
template <class T> __device__ __forceinline__ T lds(uint32_t a) { return *(const T*)__cvta_shared_to_generic(a); }

// Words of a row at multiples of four bytes from an address: one that lies on a word (AL4), or on any byte.
template <bool AL4> struct SWords {
  uint32_t a, sh;
  __device__ __forceinline__ explicit SWords(uint32_t p) : a(AL4 ? p : p & ~3u), sh(AL4 ? 0u : 8u * (p & 3u)) {}
  __device__ __forceinline__ uint32_t operator()(int off) const {
    if (AL4) return lds<uint32_t>(a + off);
    return __funnelshift_r(lds<uint32_t>(a + off), lds<uint32_t>(a + off + 4), sh);
  }
};

// The tokens' activations as a lane reads them (g = lane / 4, t = lane % 4); a block is 256 (Q, IQ), 32 (BS) and 4 (S) bytes on
struct MtLane {
  uint32_t q;         // what the lane gives ldmatrix: token lane % 8, 16-byte piece lane / 8; IQ2_XXS: token g's bytes 8 t ..
  uint32_t bs, s;     // token g's split sums 4 t ..; token 2 t's scales
  uint32_t q8, bs8, s8, s1;  // to the tokens eight on; to the scales of the next token
  uint32_t iq;        // IQ2_XXS: this lane's copy of the tables (iq_tables_fill's), the grid and then the signs
  // FMT's activations: token k's quants at XQ + k XSTRIDE, its NB scales and (BSA) split sums after those of the tokens before
  template <int FMT> __device__ __forceinline__ void set(uint32_t xq, int xstride, uint32_t xs, uint32_t bsa, int nb, uint32_t tables, int lane) {
    const int g = lane >> 2, t = lane & 3;
    q = FMT == ILL_IQ2_XXS ? xq + g * xstride + 8 * t : xq + (lane & 7) * xstride + 16 * (lane >> 3);
    bs = bsa + 32 * g * nb + 4 * t;
    s = xs + 8 * t * nb;
    q8 = 8 * xstride; bs8 = 256 * nb; s8 = 32 * nb; s1 = 4 * nb;
    iq = tables + 8 * (lane & (IQ_COPIES - 1));
  }
};

// ---- one block of 16 rows against the tokens: ACC[nt][i] += ... --------------------------------------
// The block's bytes of rows g and g + 8 of the tile in the staged piece; its number in the row; NT8 tiles of eight tokens.  Output i of a
// tile: row g + 8 (i / 2), token 8 nt + 2 t + i % 2.  A token past the last has whatever lies in its place: a column of its own, that
// nobody reads.
template <int FMT, int NT8, bool AL4> struct MtBlock;

// Q2_K: scale * q is at most 45, 180 for the field four times too large where it lies, so the scales go in with the weights as
// unsigned bytes and a block is two chains of products (fields 0 and 2, fields 1 and 3), the mins a third: sixteen times the
// mins against the sums' high parts, the mins against their low parts.
template <int NT8, bool AL4> struct MtBlock<ILL_Q2_K, NT8, AL4> {
  __device__ __forceinline__ static void run(uint32_t row0, uint32_t row8, int blk, const MtLane& x, int lane, float (&acc)[NT8][4]) {
    const uint32_t t4 = 4 * (lane & 3);
    const SWords<AL4> h0(row0), h8(row8), q0(row0 + t4), q8(row8 + t4);
    const uint32_t xq = x.q + 256 * blk, xb = x.bs + 32 * blk, xs = x.s + 4 * blk;
    int c[2][NT8][4];
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) c[0][nt][i] = c[1][nt][i] = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {        // half of the block: 128 weights, four runs of 32 at shifts 0, 2, 4, 6 of 32 bytes
      const uint32_t w[4] = {q0(16 + 32 * h), q8(16 + 32 * h), q0(32 + 32 * h), q8(32 + 32 * h)};
#pragma unroll
      for (int k = 0; k < 2; ++k) {      // runs 2 k and 2 k + 1: bytes 0, 1 and 2, 3 of a word of scales
        const uint32_t s0 = h0(8 * h + 4 * k) & 0x0f0f0f0fu, s8 = h8(8 * h + 4 * k) & 0x0f0f0f0fu;
        uint32_t a[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            a[j][i] = ((k ? w[i] >> 4 : w[i]) & (0x03030303u << (2 * j))) * __byte_perm(i & 1 ? s8 : s0, 0, 0x4440 + 2 * j + (i >> 1));
#pragma unroll
        for (int nt = 0; nt < NT8; ++nt) {
          uint32_t b[4];
          ldsm4_at(b, xq + nt * x.q8 + 128 * h + 64 * k);
          const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
          mma_k32(c[0][nt], a[0], b0, true);
          mma_k32(c[1][nt], a[1], b1, true);
        }
      }
    }
    const uint32_t m0 = q0(0), m8 = q8(0), e0 = h0(80), e8 = h8(80);
    const uint32_t am[4] = {m0 & 0xf0f0f0f0u, m8 & 0xf0f0f0f0u, (m0 >> 4) & 0x0f0f0f0fu, (m8 >> 4) & 0x0f0f0f0fu};
    const float d0 = h2f(e0 & 0xffffu), n0 = -h2f(e0 >> 16), d8 = h2f(e8 & 0xffffu), n8 = -h2f(e8 >> 16);
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt) {
      const uint32_t bm[2] = {lds<uint32_t>(xb + nt * x.bs8), lds<uint32_t>(xb + nt * x.bs8 + 16)};
      int cm[4] = {0, 0, 0, 0};
      mma_k32(cm, am, bm, true);
      const float y[2] = {lds<float>(xs + nt * x.s8), lds<float>(xs + nt * x.s8 + x.s1)};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // Q2K-DOT-AVX2 (src/avx2.lisp:147-150): y.d * d * sum - y.d * dmin * mins
        const float v = __fmaf_rn(__fmul_rn(y[i & 1], i < 2 ? n0 : n8), (float)cm[i], acc[nt][i]);
        acc[nt][i] = __fmaf_rn(__fmul_rn(i < 2 ? d0 : d8, y[i & 1]), (float)(c[0][nt][i] + (c[1][nt][i] >> 2)), v);
      }
    }
  }
};

// IQ2_XXS: a sub-block of 32 is the codebook's bytes with their signs, a product, whose sum meets the sub-block's scale.  A lane takes
// whole groups of eight weights (its four columns of a fragment are 8 t .. 8 t + 3, the other four 8 t + 4 ..), so a group costs one
// look-up of the codebook and one of the signs.  ACC comes out eight times too large (the caller's 1/8 at the end, as IQ2XXS-DOT-AVX2
// has it, src/avx2.lisp:107-110).
template <int NT8, bool AL4> struct MtBlock<ILL_IQ2_XXS, NT8, AL4> {
  // every second block's sub-blocks start on a word, in all rows alike where they lie a multiple of four bytes apart
  __device__ __forceinline__ static void run(uint32_t row0, uint32_t row8, int blk, const MtLane& x, int lane, float (&acc)[NT8][4]) {
    if (__all_sync(0xffffffffu, (((row0 + 2) | (row8 + 2)) & 3) == 0)) run_al<true>(row0, row8, blk, x, lane, acc);
    else run_al<false>(row0, row8, blk, x, lane, acc);
  }
  template <bool W>
  __device__ __forceinline__ static void run_al(uint32_t row0, uint32_t row8, int blk, const MtLane& x, int lane, float (&acc)[NT8][4]) {
    const uint32_t t = lane & 3;
    const SWords<W> q0(row0 + 2), q8(row8 + 2);
    // byte T of a sub-block's indices and field T of its signs times the tables' 128 bytes an entry: rotations by these
    const uint32_t ri = (8u * t + 25u) & 31u, rs = (7u * t + 25u) & 31u;
    auto group = [&](uint32_t idx, uint32_t aux, uint32_t& lo, uint32_t& hi) {
      const uint2 v = lds<uint2>(x.iq + (__funnelshift_r(idx, idx, ri) & 0x7f80u));
      const uint2 m = lds<uint2>(x.iq + (__funnelshift_r(aux, aux, rs) & 0x3f80u) + 8 * IQ_COPIES * 256);
      // (v ^ m) - m per byte; v is 8, 25 or 43, never 0, so adding 1 to a flipped byte never carries
      lo = (v.x ^ m.x) + (m.x & 0x01010101u);
      hi = (v.y ^ m.y) + (m.y & 0x01010101u);
    };
    int isum[NT8][4];
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) isum[nt][i] = 0;
    const uint32_t xq = x.q + 256 * blk, xs = x.s + 4 * blk;
#pragma unroll
    for (int ib = 0; ib < 8; ++ib) {
      const uint32_t x0 = q0(8 * ib + 4), x8 = q8(8 * ib + 4);
      uint32_t a[4];
      group(q0(8 * ib), x0, a[0], a[2]);
      group(q8(8 * ib), x8, a[1], a[3]);
      const int s0 = (int)((x0 >> 27) | 1u), s8 = (int)((x8 >> 27) | 1u);  // 2 LS + 1 (bit 27 is a sign's)
#pragma unroll
      for (int nt = 0; nt < NT8; ++nt) {
        const uint2 b = lds<uint2>(xq + nt * x.q8 + 32 * ib);
        int c[4];
        mma_k32_s8(c, a, b.x, b.y);
#pragma unroll
        for (int i = 0; i < 4; ++i) isum[nt][i] += c[i] * (i < 2 ? s0 : s8);
      }
    }
    const float d0 = h2f(lds<u16>(row0)), d8 = h2f(lds<u16>(row8));
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt) {
      const float y[2] = {lds<float>(xs + nt * x.s8), lds<float>(xs + nt * x.s8 + x.s1)};
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[nt][i] = __fmaf_rn(__fmul_rn(i < 2 ? d0 : d8, y[i & 1]), (float)isum[nt][i], acc[nt][i]);
    }
  }
};

}  // namespace ill
