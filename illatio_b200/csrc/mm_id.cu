// mm_id.cu -- the routed experts' product for a chunk of tokens, on the 5th-generation
// tensor cores (tcgen05, operands and accumulators in tensor memory).
//
//   Y[place, n] = sum_k X[place, k] * W_e[n, k]      for every expert e and every row
//                                                    `place` in [bases[e], bases[e] + counts[e])
//
// X is the chunk's activations already grouped by expert (ill_moe_group), as fp16
// (ill_act_f16: the Q8_K quants, exact in fp16).  W_e is expert e's matrix of raw IQ2_XXS
// or Q2_K blocks at ptrs[e] + add -- or of Q4_K / Q6_K blocks: the dense prefill products run through the same
// kernel with the matrix as its one expert (ill_mm_chunk; mm_q4k_mma / mm_q6k_mma, src/cuda/kquant.cu:316-466).
//
// A persistent grid (a CTA per SM) walks tiles of 128 weight rows x up to NT (64, 128 or 256) rows of X, picked on the host by the
// sizes of a dense matrix and on the device by the rows of the experts.  The
// weights are the tensor core's A operand and live in tensor memory: the dequantizing warps write
// their integer parts (exact in fp16) there with tcgen05.st, so they never pass through shared
// memory; X is the B operand, brought by TMA (128-byte swizzle).  The accumulator
// D[weight row, row of X] is drained once per 256-wide block of K and scaled by the block's two
// float scales.
//   warp 0      brings the X tiles by TMA, no more rows than the tile has (to the next 32)
//   warp 1      allocates tensor memory; one lane issues tcgen05.mma (128 x N x 16, fp16 in,
//               fp32 accumulate) and commits each step back to the producers
//   warps 4-..  drain the accumulators block by block (tcgen05.ld), scaling each block's integer
//               sums by the block's float scales; then store the tile (a lane = a weight row, so
//               the 32 lanes of a warp write 128 contiguous bytes of a row of Y)
//   the others  bring W_e's raw blocks into shared memory (cp.async; or warps 2 and 3 do: LOADERS, MM_TMA_W) and turn them into the A operand
// The roles' register needs differ widely, so the warp groups trade registers (setmaxnreg).
// What bounds it: the drain beside the unpacking, by instructions and latency, not the tensor pipe or memory.  Left out for
// timing: the drain's arithmetic 14-23 % of a launch, its stores 10 %, IQ2_XXS's unpacking 21 %, the X loads, the raw copies
// and the products' width nothing.  us, with four drain warps, two raw-load warps and 128-row tiles throughout / now, timed in turn:
// gate and up of 512 tokens x 2 x 9728 x 2560 (Q4_K) 153 / 83, 2560 x 9728 (Q6_K) 123 / 74; 64 tokens on 288 experts (Q2_K), gate and
// up of 1536 x 5120 1146 / 660, down 671 / 378; 96 rows each on 256 experts, down of 4096 x 2048 (Q2_K) 774 / 682, gate and up of 2048 x
// 4096 (IQ2_XXS) 1292 / 1274.  (Since, by who brings the raw blocks and how Q6_K is unpacked: Q4_K 7 % less, Q6_K 20 %; MM_TMA_W, w_q6k.)
// Every mbarrier wait is bounded; on a time-out the kernel records a code in the status
// word, skips what depends on the wait, lets copies and products in flight end, frees its tensor memory and returns.
//
// Replaces d4_mm_id_iq2_xxs / d4_mm_id_q2_k (src/cuda/ds4f_mm.cu:229-257: mma.sync
// m16n8k16, 64x64 tiles) behind DK-FFN-ROUTED-CHUNK (src/cuda-ds4f-prefill.lisp:315-356).
#include <string.h>

#include "formats.cuh"
#include "iq2xxs_tables.cuh"
#include "quantdev.cuh"
#include "tc05.cuh"
#include "host.h"

namespace ill {

constexpr int MM_BN = 128;                             // weight rows a tile (the MMA's M)
constexpr int MM_BK = 64;                              // K step: one 128-byte row of the swizzled X tile
constexpr int MM_XBOX = 32;                            // rows of X a load brings, or two, three or four times as many

struct MmParams {
  int ncols, nrows;            // K and N of every expert matrix
  int row_bytes;
  long long add, add2;         // a second matrix of every expert (gate and up in one launch) when Y2 is given
  const unsigned long long* ptrs;
  const unsigned* counts;
  const unsigned* bases;
  const float* xd;             // the activations' block scales, [token][K/256]
  const unsigned* map;         // token of each row of X (null: the row itself)
  const unsigned* ymap;        // row of Y each row of X is written to (null: the same row)
  const unsigned long long* ypeers;  // with YMAP: Y of every rank (peer memory); YMAP[place] = rank << 24 | row there
  long long total_rows;
  float* y;
  float* y2;
  long long y_stride;          // floats between rows of Y
  int ne;
  unsigned int* status;
  // a dense product (ill_mm_chunk): no tables on the device -- PTRS is null, the one "expert" is the matrix at
  // ONE_PTR with all ONE_COUNT rows of X; ACC: add into Y
  unsigned long long one_ptr;
  unsigned one_count;
  int acc;
  int bm;                      // rows of X a tile of a dense matrix, at most the kernel's NT
  int over;                    // experts of no more rows than this are left out
  float neg_zero;              // -0, for mul2_rn
  int tma;                     // the raw blocks come by TMA (mm_tma), of MmMaps::w[WMAP], [WMAP + 1]
  int wmap;
};
// (DENSE is a template argument of the kernel, so that the experts' launches compile to what they were without it)
template <int FMT, bool DENSE> __device__ __forceinline__ bool mm_tma(const MmParams& p) {
  if constexpr (!DENSE) return false; else return FMT == ILL_Q4_K || (FMT == ILL_Q6_K && p.tma);
}
template <bool DENSE> __device__ __forceinline__ unsigned long long mm_ptr(const MmParams& p, int e) {
  if constexpr (DENSE) return p.one_ptr; else return p.ptrs[e];
}
template <bool DENSE> __device__ __forceinline__ int mm_count(const MmParams& p, int e) {
  if constexpr (DENSE) return (int)p.one_count; else return (int)p.counts[e];
}
template <bool DENSE> __device__ __forceinline__ int mm_base(const MmParams& p, int e) {
  if constexpr (DENSE) return 0; else return (int)p.bases[e];
}

// two unsigned bytes (byte positions B0, B1 of V) as the halves 1024 + byte
__device__ __forceinline__ uint32_t bytes_to_h2_1024(uint32_t v, uint32_t sel) {
  return __byte_perm(v, 0x64646464u, sel);
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// the small integer N (twice, as two halves) without a conversion: 1024 + N has the bits 0x6400 | N
__device__ __forceinline__ uint32_t small_h2(uint32_t n) {
  uint32_t v = 0x64006400u | (n * 0x10001u);
  asm("add.rn.f16x2 %0, %0, %1;" : "+r"(v) : "r"(0xe400e400u));  // - 1024
  return v;
}

// ---- the weights' integer parts, 32 at a time, as 16 words of two halves -----------------
// IQ2_XXS: one sub-block (IDX: four grid indices; AUX: four groups of seven signs, and the scale):
// the 32 integers grid * sign * (2 LS + 1) (at most 43 * 31: exact in fp16).  The block's float
// part is d / 8 (src/avx2.lisp:77-110 takes the products this way).  GRID points at this lane's copy
// of the grid as halves (16 bytes an entry, eight interleaved copies: entry e of copy c at [8 e + c],
// so the eight lanes of a 128-bit request's quarter never share a bank).  SGN points at this lane's copy of the
// signs (a word an entry, 32 copies: one wavefront a request): for the seven stored bits, the eight sign bits s (the
// eighth is the parity of the seven: ksigns_iq2xs[i] = i | parity(i) << 7) as s << 9 | s << 24, so that a shift by
// 6 - 2 k brings signs 2 k and 2 k + 1 to the sign bits of the k-th pair of halves.  (A table of the eight halves' sign
// bits, 16 bytes an entry, costs four wavefronts a look-up.)
__device__ __forceinline__ void w_iq2xxs(uint32_t idx, uint32_t aux, const uint4* grid, const uint32_t* sgn, uint32_t* out) {
  const uint32_t s2 = small_h2(2 * (aux >> 28) + 1);
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const uint4 g = grid[8 * ((idx >> (8 * l)) & 0xff)];
    const uint32_t m = sgn[32 * ((aux >> (7 * l)) & 127u)];
    out[4 * l] = hmul2(g.x, s2) ^ ((m << 6) & 0x80008000u);
    out[4 * l + 1] = hmul2(g.y, s2) ^ ((m << 4) & 0x80008000u);
    out[4 * l + 2] = hmul2(g.z, s2) ^ ((m << 2) & 0x80008000u);
    out[4 * l + 3] = hmul2(g.w, s2) ^ (m & 0x80008000u);
  }
}

// byte I of V as the half 1024 + byte, twice
__device__ __forceinline__ uint32_t byte_h2_1024(uint32_t v, int i) { return __byte_perm(v, 0x64646464u, 0x4040u + 0x0101u * i); }
// 4 NW weights from the NW words Q: their fields under MASK, 2^SH too large where they lie, times the scale in byte I of SC.
// 1024 + 2^SH q has the byte's bits under the exponent of 1024; times s / 2^SH, less 1024 s / 2^SH, it is s q exactly (Q2_K: at
// most 45, Q4_K: 945; the fused multiply-add rounds once): no shift, no conversion.
template <int NW, int SH>
__device__ __forceinline__ void w_fields(const uint32_t* q, uint32_t mask, uint32_t sc, int i, uint32_t* out) {
  constexpr uint32_t inv = (uint32_t)(15 - SH) << 10, inv2 = inv | inv << 16;             // 2^-SH, twice
  constexpr uint32_t off = 0x8000u | (uint32_t)(25 - SH) << 10, off2 = off | off << 16;  // -1024 / 2^SH, twice
  const uint32_t s2 = hfma2(byte_h2_1024(sc, i), inv2, off2), bias = hmul2(s2, 0xe400e400u /* -1024 */);
#pragma unroll
  for (int k = 0; k < NW; ++k) {
    const uint32_t v = q[k] & mask;
    out[2 * k] = hfma2(bytes_to_h2_1024(v, 0x4140), s2, bias);
    out[2 * k + 1] = hfma2(bytes_to_h2_1024(v, 0x4342), s2, bias);
  }
}
// Q2_K: eight mins (scale bytes M0, M1 >> 4) as four words
__device__ __forceinline__ void w_q2k_mins(uint32_t m0, uint32_t m1, uint32_t* v) {
  const uint32_t lo = (m0 >> 4) & 0x0f0f0f0fu, hi = (m1 >> 4) & 0x0f0f0f0fu;
  const uint32_t k1024 = 0xe400e400u;  // -1024 twice
  v[0] = bytes_to_h2_1024(lo, 0x4140); v[1] = bytes_to_h2_1024(lo, 0x4342);
  v[2] = bytes_to_h2_1024(hi, 0x4140); v[3] = bytes_to_h2_1024(hi, 0x4342);
#pragma unroll
  for (int i = 0; i < 4; ++i) asm("add.rn.f16x2 %0, %0, %1;" : "+r"(v[i]) : "r"(k1024));
}

// Q4_K: the four 6-bit scales and the four mins of half H of a block, a byte each, from the twelve packed bytes S
// (get_scale_min_k4, src/kquant.lisp:64-72, four at a time)
__device__ __forceinline__ void q4k_scales_mins(const uint32_t* s, int h, uint32_t& sc, uint32_t& mn) {
  sc = h ? (s[2] & 0x0f0f0f0fu) | ((s[0] >> 2) & 0x30303030u) : s[0] & 0x3f3f3f3fu;
  mn = h ? ((s[2] >> 4) & 0x0f0f0f0fu) | ((s[1] >> 2) & 0x30303030u) : s[1] & 0x3f3f3f3fu;
}
// Q4_K: four groups' mins, each twice (a group of 32 faces two of the activations' sums of 16), as four words
__device__ __forceinline__ void w_q4k_mins(uint32_t mn, uint32_t* v) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = byte_h2_1024(mn, i);
    asm("add.rn.f16x2 %0, %0, %1;" : "+r"(v[i]) : "r"(0xe400e400u));  // - 1024
  }
}

// N words at RW of a row whose block starts SH / 8 (0 or 2) bytes into its first word
template <int N>
__device__ __forceinline__ void raw_words(const uint32_t* rw, uint32_t sh, uint32_t* out) {
  uint32_t prev = rw[0];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t next = rw[i + 1];
    out[i] = __funnelshift_r(prev, next, sh);
    prev = next;
  }
}
// Q6_K: 16 weights of a K step -- the low (ODD 0) or high nibbles of the four words QL, the 2-bit fields at shift QSH of the
// four words QH -- times their group's signed scale.  |scale * (q - 32)| reaches 4064 and fp16 holds only even
// integers above 2048, so the product goes to the tensor core in two exact parts: EVEN = (scale - scale % 2) * (q - 32), an
// even integer of at most 4096, and ODD = (scale % 2) * (q - 32); both are multiplied with the same activations into
// the same accumulator.  EX: of the scale's upper four bits (-8 .. 7) and lower four.
// A nibble in the upper half of its byte, and its 2-bit field in the lower bits of 0x64, are the bits of 1024 + 16 q; times part / 16, less
// 96 parts, is part * (q - 32) exactly (one rounding).  SE and SO: part / 16, twice (q6k_parts).  (Put together at bit 0,
// less 1056 and then multiplied, and the half's two K steps stored together: 2560 x 9728, 512 tokens 83 us, now 75; 5120 x 17408 220, now 185.)
__device__ __forceinline__ void w_q6k(const uint32_t* ql, const uint32_t* qh, int odd, int qsh, uint32_t se, uint32_t so, uint32_t* even, uint32_t* oddp) {
  const uint32_t be = hmul2(se, 0xe600e600u /* -1536 */), bo = hmul2(so, 0xe600e600u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t lo = (odd ? ql[i] : ql[i] << 4) & 0xf0f0f0f0u, hi = ((qh[i] >> qsh) & 0x03030303u) | 0x64646464u;
    const uint32_t a = __byte_perm(lo, hi, 0x5140), b = __byte_perm(lo, hi, 0x7362);
    even[2 * i] = hfma2(a, se, be);
    even[2 * i + 1] = hfma2(b, se, be);
    oddp[2 * i] = hfma2(a, so, bo);
    oddp[2 * i + 1] = hfma2(b, so, bo);
  }
}
// The two parts of four scales, a byte each, the even or upper ones plus 128 or 8
template <bool EX> __device__ __forceinline__ void q6k_parts(uint32_t sc, uint32_t& e, uint32_t& o) {
  const uint32_t t = sc ^ 0x80808080u;
  e = EX ? (t >> 4) & 0x0f0f0f0fu : t & 0xfefefefeu;
  o = sc & (EX ? 0x0f0f0f0fu : 0x01010101u);
}

// The tensor maps of X (rows of 64 halves, two K steps a load) and of its sums of 16 for loads of 32, 64, 96 and 128 rows
struct MmMaps {
  CUtensorMap x[4], e[4];
  CUtensorMap w[2];  // MM_TMA_W: a dense matrix, and the one beside it, as rows of bytes
};
// Whether the raw blocks may come by TMA, 128 rows of a block at a time: of a dense matrix (an expert's address is the device's to look
// up, so it has no map).  Q4_K blocks start on 16-byte boundaries: one load.  Q6_K (MmParams::tma: where four rows are a whole number of
// 16-byte pieces, an even number of blocks a row): the map's rows are four of the matrix's, so that rows 4 i + k start 16-byte aligned up
// to what k and the block decide; four loads of 32 rows' windows.  Asked for by the lanes that unpack them, the 16-byte pieces took 590 of
// Q4_K's 3300 cycles a block that bound the kernel.  us, 512 tokens, before / now: Q4_K 2 x 9728 x 2560 98 / 91, 4096 x 2560 32 / 30,
// 2560 x 4096 38.4 / 35.0; 64 tokens x 4096 x 2560 25.2 / 23.6; 2048 x 9728 x 2560 159 / 149.  Q6_K 2560 x 9728 75 / 67, 5120 x 17408
// 185 / 181, 5120 x 5120 of 1024 tokens 111 / 99 (also without bank conflicts where the four rows' windows start at four words).
template <int FMT, bool DENSE> constexpr bool MM_TMA_W = DENSE && (FMT == ILL_Q4_K || FMT == ILL_Q6_K);
__device__ __forceinline__ int mm_boxes(int rows) { return max(1, (rows + MM_XBOX - 1) / MM_XBOX); }

// Geometry per format and per NT, the most rows of X a tile has (64, 128 or 256).  A 256-wide block is four K steps; the
// formats with mins (KM) have a second, small product a block: the mins against the activations' sums of 16 (one K = 16 MMA).
// A tile of up to 128 rows is one job a block (one accumulator); a tile of up to 256 is two, its halves, against the same
// A operand: a block's weights are then unpacked once for twice the rows.
// Tensor memory, 512 columns (an accumulator's column = a row of X):
//   D[2] at 0, two accumulators that alternate job by job; KM: the mins' accumulator (two when NT is 64); then the ring
//   of A slots, a K step each, to the end
// EX (tiles of up to 64): two accumulators a job, each an integer that fp32 holds, for sums that round once, as int32 would (mm_exact_kernel):
// Q4_K the block's first and second half of K (at most 128 * 945 * 128 < 2^24), Q6_K the scales' upper and lower four bits (at most
// 256 * 480 * 128; a block's whole sum reaches 2^27).
template <int FMT, int NT, bool EX = false> struct MmGeom {
  static_assert(!EX || (NT == 64 && (FMT == ILL_Q4_K || FMT == ILL_Q6_K)), "tensor memory");
  static constexpr bool KM = FMT == ILL_Q2_K || FMT == ILL_Q4_K;
  static constexpr int BB = FMT == ILL_Q2_K ? 84 : FMT == ILL_Q4_K ? 144 : FMT == ILL_Q6_K ? 210 : 66;
  static constexpr int HALVES = NT > 128 ? 2 : 1;
  static constexpr int DC = NT < 128 ? NT : 128;            // columns of an accumulator
  // Dequantizing warps: a set of eight makes a block -- four (32 weight rows each) its first half of K, four the second --
  // and two sets take the CTA's blocks in turn.  In wide tiles, and in tiles of 128 with two accumulators a block, the way out
  // of tensor memory takes longer than the way in, and a second set's registers go to it.
  static constexpr int SETS = NT < 128 || (NT == 128 && !KM) ? 2 : 1, DQ_WARPS = 8 * SETS;
  // Drain warps: DR_GROUPS times four (32 weight rows each); a group takes every DR_GROUPS-th eight columns
  static constexpr int DR_GROUPS = NT == 128 && KM ? 4 : 2, DR_WARPS = 4 * DR_GROUPS;
  static constexpr int THREADS = 32 * (4 + DR_WARPS + DQ_WARPS);
  // registers a thread after the roles part (the sum must fit in what the CTA was launched with: checked by the host)
  static constexpr int REGS_AUX = 40, REGS_DRAIN = FMT == ILL_Q6_K ? (NT > 128 ? 152 : 104) : DR_GROUPS == 4 ? 88 : 120,
                       REGS_DQ = FMT == ILL_Q6_K ? 64 : 56;
  static constexpr int REGS_SUM = 128 * REGS_AUX + 32 * (DR_WARPS * REGS_DRAIN + DQ_WARPS * REGS_DQ);
  static constexpr uint32_t SLOTW = FMT == ILL_Q6_K ? 64 : 32;  // columns of an A slot (Q6_K: the even and the odd part)
  static constexpr int NDM = !KM ? 0 : NT < 128 ? 2 : 1;
  static constexpr uint32_t DB = EX ? 2 * DC : DC;          // columns of a job's accumulators
  static constexpr uint32_t DM_COL = 2 * DB, A_COL = KM && (EX || NT == 128) ? 384 : 256;
  static_assert(!(NT > 128 && KM) && DM_COL + NDM * DC <= A_COL, "accumulators and the A ring overlap");
  static constexpr int NSLOT = (512 - A_COL) / SLOTW;       // a block or two
  static_assert(NSLOT == 4 || NSLOT == 8, "a block's slots are consecutive");
  // Raw blocks: the two warps that unpack them (a block's halves, the same 32 rows) bring their rows' windows -- or, LOADERS,
  // where the unpacking bounds the kernel: IQ2_XXS (gate and up of 24576 rows on 256 experts 1360 -> 1301 us) and tiles of 128 of
  // Q2_K (2 x 1536 x 5120 on 64 experts of 128 rows 357 -> 346; tiles of 64 were 15 % slower, Q6_K and Q4_K 7 %), the two warps that
  // have no other role, for all -- the CPR 16-byte pieces from the
  // boundary at or before the block, PITCH bytes apart (an odd number of 16-byte pieces: 32 rows' words lie in at most four
  // lanes a bank), RPI rows a request, a block of theirs ahead
  static constexpr bool LOADERS = FMT == ILL_IQ2_XXS || (FMT == ILL_Q2_K && NT == 128);
  static constexpr int CPR = FMT == ILL_Q2_K ? 6 : FMT == ILL_Q4_K ? 9 : FMT == ILL_Q6_K ? 14 : 5;
  static constexpr int PITCH = FMT == ILL_Q2_K ? 112 : FMT == ILL_Q4_K ? 144 : FMT == ILL_Q6_K ? 240 : 80;
  static constexpr int RPI = 32 / CPR;
  static constexpr uint32_t RAW_BYTES = 32 * PITCH;         // 32 rows'; there are DQ_WARPS of these
  static constexpr uint32_t X_BYTES = 2 * DC * MM_BK * 2, E_BYTES = KM ? DC * 32 : 0, M_BYTES = KM ? 128 * 32 : 0;
  static constexpr int NX = FMT == ILL_Q6_K && NT == 128 ? 3 : 4;  // stages of the ring of X tiles, two K steps each
  static constexpr uint32_t BODY = NX * X_BYTES + 2 * E_BYTES + 2 * M_BYTES + DQ_WARPS * RAW_BYTES + 4 * 256 * 4 /* weight scales */ +
                                   16 * NT /* X scales */;
};
// Shared memory of a kernel for tiles of up to NT rows of X or, when NT2 is not 0, of up to NT or of up to NT2
constexpr uint32_t MM_BARS = 768;  // the barriers of one of them
constexpr int MM_MAX_NE = 512;     // experts a launch
template <int FMT, int NT, int NT2> struct MmSmem {
  static constexpr uint32_t BODY2 = MmGeom<FMT, NT2 ? NT2 : NT>::BODY, BODY = MmGeom<FMT, NT>::BODY > BODY2 ? MmGeom<FMT, NT>::BODY : BODY2;
  static constexpr uint32_t FIRST = BODY + (NT2 ? 2 : 1) * MM_BARS, SLOTS = FIRST + 4 * (MM_MAX_NE + 1) /* experts' first tiles */,
                            TABLES = (SLOTS + 8 + 255) / 256 * 256;
  static constexpr size_t SMEM = TABLES + (FMT == ILL_IQ2_XXS ? 8 * 4096 + 32 * 512 : 0) + 1024 /* alignment */;
  static_assert(SMEM <= 227 * 1024, "shared memory of a CTA");
};

template <int FMT, int FMT2> struct MmExactSmem {
  static constexpr uint32_t BODY2 = MmGeom<FMT2, 64, true>::BODY, BODY = MmGeom<FMT, 64, true>::BODY > BODY2 ? MmGeom<FMT, 64, true>::BODY : BODY2;
  static constexpr size_t SMEM = BODY + MM_BARS + 16 + 1024 /* alignment */;
  static_assert(SMEM <= 227 * 1024, "shared memory of a CTA");
};

// One of two warps' (H) requests for the windows of a block of ROWS <= 32 rows (the first row's block at SRC) into the buffer DST;
// FULL gets this warp's 32 arrivals once they have landed.
template <int FMT, int NT>
__device__ __forceinline__ void mm_fetch(const u8* src, int row_bytes, int rows, int h, int lane, u8* dst, uint64_t* full) {
  typedef MmGeom<FMT, NT> G;
  const int r0 = lane / G::CPR + h * G::RPI, ch = lane % G::CPR;
  if (lane < G::CPR * G::RPI) {
    src += (long long)r0 * row_bytes;
    dst += r0 * G::PITCH + 16 * ch;
    const long long step = 2ll * G::RPI * row_bytes;
#pragma unroll
    for (int r = 0; r < 32; r += 2 * G::RPI, src += step)
      if (r + r0 < rows) cp_async16(dst + r * G::PITCH, (const void*)(((uintptr_t)src & ~(uintptr_t)15) + 16 * ch));
  }
  cp_async_arrive(full);
}

// The mbarriers of a kernel for tiles of up to NT rows of X
template <int FMT, int NT, bool EX = false> struct MmBars {
  typedef MmGeom<FMT, NT, EX> G;
  uint64_t xfull[G::NX];      // the X tile landed (TMA)
  uint64_t xempty[G::NX];     // the MMAs that read it completed
  uint64_t afull[G::NSLOT];   // the K step of A is in tensor memory (4 warps)
  // [2][4] the MMAs that read block n's K steps completed, at n % 2: a barrier for each block that may be waited for, since
  // a warp two blocks ahead could not tell a slot's phases apart by their parity
  uint64_t aempty[8];
  uint64_t efull[2];          // KM: the job's sums of 16 landed
  uint64_t eempty[2];
  uint64_t mfull[2];          // KM: the block's mins are in their tile (8 warps)
  uint64_t mempty[2];
  uint64_t acc_full[2];       // a job's MMAs completed
  uint64_t acc_free[2];       // the drain warps have read the job's accumulators
  uint64_t raw_full[G::DQ_WARPS];   // both warps' copies into a raw buffer landed
  uint64_t raw_empty[G::DQ_WARPS];  // both warps have read it
  uint64_t fin;               // after a time-out: the MMAs issued so far completed
  // TMA: a raw buffer is a block's 128 rows, at [2 set + buffer], filled by one warp and read by a set's eight warps
  __device__ __forceinline__ void init(bool tma_w) {
    for (int s = 0; s < G::NX; ++s) { mbar_init(&xfull[s], 1); mbar_init(&xempty[s], 1); }
    for (int s = 0; s < G::NSLOT; ++s) mbar_init(&afull[s], 4);
    for (int s = 0; s < 8; ++s) mbar_init(&aempty[s], 1);
    for (int s = 0; s < G::DQ_WARPS; ++s) { mbar_init(&raw_full[s], tma_w ? 1 : 64); mbar_init(&raw_empty[s], tma_w ? 8 : 2); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&efull[s], 1); mbar_init(&eempty[s], 1);
      mbar_init(&mfull[s], 8); mbar_init(&mempty[s], 1);
      mbar_init(&acc_full[s], 1); mbar_init(&acc_free[s], G::DR_WARPS);
    }
    mbar_init(&fin, 1);
  }
};

// What a CTA does once its barriers, tables and tensor memory are there and the experts' tiles of up to BM rows of X are counted
// (TILE_FIRST): tiles CTA, + CTAS, ...
template <int FMT, bool DENSE, int NT, bool EX = false>
__device__ __forceinline__ void mm_tiles(const MmMaps& maps, const MmParams& p, int bm, u8* smem, MmBars<FMT, NT, EX>* bars, const int* tile_first,
                                         const uint4* iq_grid, const uint32_t* iq_sgn, uint32_t tmem_base, int warp, int lane, int cta, int ctas) {
  typedef MmGeom<FMT, NT, EX> G;
  constexpr int BB = G::BB, NSLOT = G::NSLOT, NX = G::NX, PITCH = G::PITCH, HALVES = G::HALVES, DC = G::DC;
  constexpr bool KM = G::KM, TMA_W = MM_TMA_W<FMT, DENSE>;
  constexpr uint32_t W_BYTES = 4 * G::RAW_BYTES;  // a block's 128 rows
  static_assert(!TMA_W || ((PITCH == BB || FMT == ILL_Q6_K) && (NX * G::X_BYTES + 2 * G::E_BYTES + 2 * G::M_BYTES) % 128 == 0 && G::RAW_BYTES % 128 == 0), "where TMA writes");
  const bool tma = mm_tma<FMT, DENSE>(p);
  // [X ring][KM: sums of 16 x 2, mins x 2] (the X tiles 1024-byte aligned, as the 128-byte swizzle needs), the
  // dequantizing warps' raw blocks, scales
  u8* x_tiles = smem;
  u8* e_tiles = smem + NX * G::X_BYTES;          // KM: the sums of 16 of the job's rows of X
  u8* m_tiles = e_tiles + 2 * G::E_BYTES;        // KM: the mins
  u8* raw = m_tiles + 2 * G::M_BYTES;
  float* wsc = (float*)(raw + G::DQ_WARPS * G::RAW_BYTES);  // [4 blocks in flight][2: d, dmin][128 weight rows]
  float* xsc = wsc + 4 * 256;                    // [drain warps][HALVES * DC / DR_GROUPS] the block's scales of the warp's rows of X
  uint64_t *xfull = bars->xfull, *xempty = bars->xempty, *afull = bars->afull, *aempty = bars->aempty, *efull = bars->efull,
           *eempty = bars->eempty, *mfull = bars->mfull, *mempty = bars->mempty, *acc_full = bars->acc_full, *acc_free = bars->acc_free,
           *raw_full = bars->raw_full, *raw_empty = bars->raw_empty, *fin = &bars->fin;

  const int nkb = p.ncols / 256;
  const int ntn1 = (p.nrows + MM_BN - 1) / MM_BN;
  const int ntn = p.y2 ? 2 * ntn1 : ntn1;     // the second matrix's weight-row tiles follow the first's
  const int ntiles = tile_first[p.ne] * ntn;  // weight-row tiles vary fastest: CTAs running together share X
  bool ok = true;

  // tile index -> expert, first row of X, valid rows, weight-row tile
  // (NT >= ntn1: tile NT - ntn1 of the second matrix)
  auto locate = [&](int tile, int& expert, int& row0, int& nvalid, int& nt) {
    const int mt = tile / ntn;
    nt = tile - mt * ntn;
    int lo = 0, hi = p.ne - 1;  // the last expert whose first tile is <= mt and that has tiles
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (tile_first[mid] <= mt) lo = mid; else hi = mid - 1;
    }
    expert = lo;
    const int m_in = mt - tile_first[lo];
    row0 = mm_base<DENSE>(p, lo) + m_in * bm;
    nvalid = min(bm, mm_count<DENSE>(p, lo) - m_in * bm);
    // counts / bases come from the caller: a tile never reaches past the TOTAL_ROWS rows X and Y have
    if ((long long)row0 >= p.total_rows) { row0 = 0; nvalid = 0; }
    else nvalid = min(nvalid, (int)(p.total_rows - row0));
  };

  if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(G::REGS_AUX));
  if (warp == 0) {
    // ---- TMA producer of the X tiles: a load brings two K steps of the job's rows of X (up to 32, 64, 96 or 128).  Lanes 0
    // and 1 watch a job's two stages, lane 2 (KM) the tile for its sums of 16: one poll looks at all of them.
    int s = 0, g = 0;                              // stage of the ring; jobs so far
    uint32_t ph = 1;                               // parity that a free stage's barrier has completed (a fresh barrier: 1)
    for (int tile = cta; tile < ntiles && ok; tile += ctas) {
      int expert, row0, nvalid, nt;
      locate(tile, expert, row0, nvalid, nt);
      for (int kb = 0; kb < nkb && ok; ++kb) {
        for (int half = 0; half == 0 || (half < HALVES && 128 * half < nvalid); ++half, ++g) {
          const int boxes = mm_boxes(min(DC, nvalid - 128 * half)), hrow = row0 + 128 * half, b = g & 1;
          const bool wrap = s + lane >= NX;
          uint64_t* bar = lane == 2 && KM ? &eempty[b] : &xempty[lane < 2 ? (wrap ? s + lane - NX : s + lane) : s];
          const uint32_t par = lane == 2 && KM ? ((uint32_t)(g >> 1) & 1u) ^ 1u : ph ^ (wrap && lane < 2 ? 1u : 0u);
          BarPoll poll(p.status, lane == 2 ? ST_MM_WAIT_EMPTY + 4 : ST_MM_WAIT_EMPTY);
#pragma unroll
          for (int i = 0; i < (KM ? 3 : 2); ++i) {
            if (!(ok = poll.until(bar, par, 1u << i))) break;
            if (i < 2) {
              if (elect_one()) {
                mbar_expect_tx(&xfull[s], boxes * (2 * MM_XBOX * MM_BK * 2));
                tma_load_3d(x_tiles + s * G::X_BYTES, &maps.x[boxes - 1], 0, hrow, kb * 4 + 2 * i, &xfull[s]);
              }
              __syncwarp();
              if (++s == NX) { s = 0; ph ^= 1; }
            } else {
              if (elect_one()) {
                mbar_expect_tx(&efull[b], boxes * (MM_XBOX * 32));
                tma_load_2d(e_tiles + b * G::E_BYTES, &maps.e[boxes - 1], kb * MM_BK, hrow, &efull[b]);
              }
              __syncwarp();
            }
          }
          if (!ok) break;
        }
      }
    }
    if (!ok) {
      // a wait ran out: the copies that are in flight land before the CTA goes (a stage's last phase, if it had one)
      for (int i = 0; i < NX; ++i) mbar_wait(&xfull[i], i < s ? ph ^ 1u : ph, nullptr, 0, 0, ILL_WAIT_NS / 20);
      if (KM)
        for (int j = max(0, g - 2); j < g; ++j) mbar_wait(&efull[j & 1], (uint32_t)(j >> 1) & 1u, nullptr, 0, 0, ILL_WAIT_NS / 20);
    }
  } else if (warp == 1) {
    // ---- MMA issuer: the whole warp walks the loop (so that addresses and descriptors stay in uniform
    // registers) and one elected lane issues.  A barrier costs 60 to 90 cycles to look at, so each lane watches one of a
    // job's: 0 and 1 its X stages, 4..7 its K steps of A, 8 its accumulator; KM: 9 its sums of 16, 10 the block's mins, 11 the
    // mins' accumulator (when there is one, the job before must have been drained).
    uint64_t* ring = lane < 2 ? xfull : lane < 4 ? acc_free : lane < 8 ? afull : lane == 9 ? efull : lane == 10 ? mfull : acc_free;
    const int len = lane < 2 ? NX : lane < 4 ? 2 : lane < 8 ? NSLOT : 2, step = lane < 2 ? 2 : lane < 4 ? 1 : lane < 8 ? 4 : 1;
    int idx = lane < 2 ? lane : lane < 4 ? 0 : lane < 8 ? lane - 4 : lane == 11 ? 1 : 0;
    uint32_t par = lane == 8 || lane == 11 ? 1u : 0u;
    const bool per_block = (lane >= 4 && lane < 8) || lane == 10;  // shared by a block's jobs
    const unsigned code = lane < 4 ? ST_MM_WAIT_FULL : lane < 8 ? ST_MM_WAIT_FULL + 1 : lane == 8 ? ST_MM_WAIT_EPI
                          : lane == 9 ? ST_MM_WAIT_FULL + 4 : lane == 10 ? ST_MM_WAIT_FULL + 3 : ST_MM_WAIT_EPI + 2;
    const uint64_t xdesc0 = umma_desc(x_tiles);
    int s = 0, slot = 0, g = 0, g_kb = 0;          // X stage; first A slot of the block; jobs and blocks so far
    for (int tile = cta; tile < ntiles && ok; tile += ctas) {
      int expert, row0, nvalid, nt;
      locate(tile, expert, row0, nvalid, nt);
      nvalid = __shfl_sync(0xffffffffu, nvalid, 0);
      const bool two = HALVES > 1 && nvalid > 128;
      for (int kb = 0; kb < nkb && ok; ++kb, ++g_kb) {
        for (int half = 0; half <= (two ? 1 : 0); ++half, ++g) {
          const int b = g & 1, rows = min(DC, nvalid - 128 * half);
          const bool last = half == (two ? 1 : 0);
          // fp32 accumulate, fp16 A and B, both K-major, M = 128 weight rows, N = the job's rows of X up to 16
          const int nmma = max(16, (rows + 15) & ~15);
          const uint32_t idesc = (1u << 4) | ((uint32_t)(nmma >> 3) << 17) | ((uint32_t)(MM_BN >> 4) << 24);
          const uint32_t d1 = tmem_base + (uint32_t)b * G::DB;
          const uint32_t xstep = mm_boxes(rows) * (MM_XBOX * MM_BK * 2 / 16);  // a K step's tile in a stage
          uint64_t* aem = aempty + 4 * (g_kb & 1);
          BarPoll poll(p.status, code);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (!(ok = poll.until(ring + idx, par, (i ? 0u : 0x100u) | (1u << (i >> 1)) | (0x10u << i)))) break;
            tc_fence_after();
            const uint64_t xdsc = xdesc0 + (uint32_t)(s * (int)(G::X_BYTES >> 4)) + (i & 1 ? xstep : 0u);
            const uint32_t a0 = tmem_base + G::A_COL + G::SLOTW * (slot + i);
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < MM_BK / 16; ++k)  // 16 of K: 8 columns of A, 32 bytes inside X's swizzle atom
                umma_f16_ts(EX && FMT == ILL_Q4_K ? d1 + (i >> 1) * DC : d1, a0 + 8 * k, xdsc + 2 * k, idesc,
                            ((EX && FMT == ILL_Q4_K ? i & 1 : i) | k) ? 1u : 0u);
              if constexpr (FMT == ILL_Q6_K) {  // the weights' odd parts (EX: their other parts) against the same activations
#pragma unroll
                for (int k = 0; k < MM_BK / 16; ++k)
                  umma_f16_ts(EX ? d1 + DC : d1, a0 + 32 + 8 * k, xdsc + 2 * k, idesc, EX && !(i | k) ? 0u : 1u);
              }
              if (i & 1) umma_commit(&xempty[s]);
              if (last) umma_commit(&aem[i]);
              if (!KM && i == 3) umma_commit(&acc_full[b]);
            }
            __syncwarp();
            if ((i & 1) && ++s == NX) s = 0;
          }
          if (!ok) break;
          if constexpr (KM) {
            const int mb = g_kb & 1;
            if (!(ok = poll.until(ring + idx, par, G::NDM == 1 ? 0xe00u : 0x600u))) break;
            tc_fence_after();
            // mins x sums of 16: one K = 16 product into the mins' accumulator
            if (elect_one()) {
              umma_f16_ss(tmem_base + G::DM_COL + (G::NDM == 2 ? b * DC : 0), umma_desc32(m_tiles + mb * G::M_BYTES),
                          umma_desc32(e_tiles + b * G::E_BYTES), idesc, 0u);
              umma_commit(&eempty[b]);
              if (last) umma_commit(&mempty[mb]);
              umma_commit(&acc_full[b]);
            }
            __syncwarp();
          }
          if (last || !per_block) {
            idx += step;
            if (idx >= len) { idx -= len; par ^= 1; }
          }
        }
        slot += 4;
        if (slot == NSLOT) slot = 0;
      }
    }
    if (!ok) {
      // a wait ran out: the products issued so far end before tensor memory is freed
      if (elect_one()) umma_commit(fin);
      __syncwarp();
      mbar_wait(fin, 0, nullptr, 0, 0, ILL_WAIT_NS / 20);
    }
  } else if (warp < 4) {
    // ---- warps 2, 3 (LOADERS) bring the raw windows of every block, half of each 32 rows' requests a warp; TMA: warp 2 its rows
    if constexpr (TMA_W) {
      int g_kb = 0;
      for (int tile = warp == 2 && tma ? cta : ntiles; tile < ntiles && ok; tile += ctas) {
        int expert, row0, nvalid, nt;
        locate(tile, expert, row0, nvalid, nt);
        const bool second = nt >= ntn1;
        if (second) nt -= ntn1;
        for (int kb = 0; kb < nkb; ++kb, ++g_kb) {
          const int it = g_kb / G::SETS, at = 2 * (g_kb % G::SETS) + (it & 1);
          ok = __all_sync(0xffffffffu, mbar_wait(&raw_empty[at], ((uint32_t)(it >> 1) & 1u) ^ 1u, p.status, ST_MM_WAIT_EMPTY + 2));
          if (!ok) break;
          if (elect_one()) {
            mbar_expect_tx(&raw_full[at], W_BYTES);
            const CUtensorMap* map = &maps.w[p.wmap + (second ? 1 : 0)];
            if constexpr (FMT == ILL_Q4_K) {
              tma_load_2d(raw + at * W_BYTES, map, kb * BB, nt * MM_BN, &raw_full[at]);
            } else {
#pragma unroll 1
              for (int k = 0; k < 4; ++k)
                tma_load_2d(raw + at * W_BYTES + k * G::RAW_BYTES, map, (k * p.row_bytes + kb * BB) & ~15, nt * (MM_BN / 4), &raw_full[at]);
            }
          }
          __syncwarp();
        }
      }
      if (!ok)  // a wait ran out: the copies that are in flight land before the CTA goes
        for (int k = max(0, g_kb - 2 * G::SETS); k < g_kb; ++k)
          mbar_wait(&raw_full[2 * (k % G::SETS) + (k / G::SETS & 1)], (uint32_t)(k / G::SETS >> 1) & 1u, nullptr, 0, 0, ILL_WAIT_NS / 20);
    }
    if constexpr (G::LOADERS) {
      int g_kb = 0;
      for (int tile = cta; tile < ntiles && ok; tile += ctas) {
        int expert, row0, nvalid, nt;
        locate(tile, expert, row0, nvalid, nt);
        const bool second = nt >= ntn1;
        if (second) nt -= ntn1;
        const u8* w0 = (const u8*)(uintptr_t)mm_ptr<DENSE>(p, expert) + (second ? p.add2 : p.add) + (long long)nt * MM_BN * p.row_bytes;
        const int rows_here = p.nrows - nt * MM_BN;
        for (int kb = 0; kb < nkb && ok; ++kb, ++g_kb) {
          const int set = g_kb % G::SETS, it = g_kb / G::SETS, buf = it & 1;
          // lane WQ < 4 watches the four warp pairs' buffers: the block two back must have been read from them
          uint64_t* bar = raw_empty + (set * 4 + (lane & 3)) * 2 + buf;
          BarPoll poll(p.status, ST_MM_WAIT_EMPTY + 2);
#pragma unroll 1
          for (int wq = 0; wq < 4; ++wq) {
            if (!(ok = poll.until(bar, ((uint32_t)(it >> 1) & 1u) ^ 1u, 1u << wq))) break;
            mm_fetch<FMT, NT>(w0 + (long long)(32 * wq) * p.row_bytes + (long long)kb * BB, p.row_bytes, min(32, rows_here - 32 * wq), warp & 1,
                              lane, raw + ((set * 4 + wq) * 2 + buf) * G::RAW_BYTES, raw_full + (set * 4 + wq) * 2 + buf);
          }
        }
      }
      cp_async_wait_all();
    }
  } else if (warp < 4 + G::DR_WARPS) {
    // ---- warps 4.. drain the accumulators job by job, scaling each block's integer sums by the
    // block's float scales, and store the finished tile.  A warp reads the 32 tensor-memory lanes
    // its number gives it (warp % 4: 32 weight rows) and every DR_GROUPS-th eight columns (rows of X), so that
    // the warps have the same share whatever the tile's rows.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(G::REGS_DRAIN));
    const int q = warp & 3, hh = (warp - 4) >> 2;
    const int m = q * 32 + lane;                   // accumulator lane = weight row in the tile
    constexpr int STRIDE = 8 * G::DR_GROUPS, NP = DC / (32 * G::DR_GROUPS);  // a warp's eights of columns lie STRIDE apart; it has 32 NP columns of a job
    constexpr bool PIPE = NT <= 128;
    const uint32_t t0 = tmem_base + ((uint32_t)(q * 32) << 16) + 8 * hh;
    int g = 0, d_kb = 0;                           // jobs and blocks drained so far by this CTA
    float* xsw = xsc + (warp - 4) * (HALVES * NP * 32);
    const uint64_t nz2 = EX ? pack2(p.neg_zero, p.neg_zero) : 0ull;
    for (int tile = cta; tile < ntiles && ok; tile += ctas) {
      int expert, row0, nvalid, nt;
      locate(tile, expert, row0, nvalid, nt);
      // pairs of fp32: this weight row against the tile's rows of X 128 half + column(0 .. 32 NP - 1)
      uint64_t out[HALVES * NP * 16];
      auto column = [&](int i) { return STRIDE * (i >> 3) + 8 * hh + (i & 7); };
#pragma unroll
      for (int i = 0; i < HALVES * NP * 16; ++i) out[i] = 0ull;
      // a lane fetches the scales of one row of X of 32 (a row past the tile's last: the first row's), a block ahead
      int tok[HALVES * NP];
      float dxn[HALVES * NP];
#pragma unroll
      for (int i = 0; i < HALVES * NP; ++i) {
        const int c = 128 * (i / NP) + column(32 * (i % NP) + lane);
        const long long place = (long long)row0 + (c < nvalid ? c : 0);
        tok[i] = !DENSE && p.map ? (int)p.map[place] : (int)place;
        dxn[i] = p.xd[(long long)tok[i] * nkb];
      }
      for (int kb = 0; kb < nkb && ok; ++kb, ++d_kb) {
#pragma unroll
        for (int i = 0; i < HALVES * NP; ++i) {
          xsw[32 * i + lane] = dxn[i];
          if (kb + 1 < nkb) dxn[i] = p.xd[(long long)tok[i] * nkb + kb + 1];
        }
        __syncwarp();
#pragma unroll
        for (int half = 0; half < HALVES; ++half) {
          if (half > 0 && (nvalid <= 128 * half || !ok)) break;
          const int b = g & 1;
          const bool e_ok = mbar_wait(&acc_full[b], (uint32_t)(g >> 1) & 1u, p.status, ST_MM_WAIT_ACC);
          if (!__all_sync(0xffffffffu, e_ok)) { ok = false; break; }
          tc_fence_after();
          // Two fp32 at a time (each half of a packed instruction rounds as the scalar one does).
          // IQ2XXS-DOT-AVX2 (src/avx2.lisp:107-110): total += d * y.d * sum, the 1/8 at the end;
          // Q2K-DOT-AVX2 (src/avx2.lisp:147-150): y.d * d * sum - y.d * dmin * mins
          const float dw = wsc[(d_kb & 3) * 256 + m];
          const uint64_t dw2 = pack2(dw, dw);
          uint64_t dm2 = 0;
          if constexpr (KM) {
            const float dm = -wsc[(d_kb & 3) * 256 + 128 + m];
            dm2 = pack2(dm, dm);
          }
          const float* xp = xsw + half * NP * 32;
          const int nv = nvalid - 128 * half - 8 * hh;  // columns past the tile's last row of X were not computed
          const uint32_t td = t0 + b * G::DB, tm = t0 + G::DM_COL + (G::NDM == 2 ? b * DC : 0);
          // eight columns at a time; in narrow tiles, where the registers allow it, the next eight are on their way meanwhile
          uint32_t v[PIPE ? 2 : 1][8], w[PIPE ? 2 : 1][8], u[PIPE ? 2 : 1][8];
          if (PIPE && nv > 0) {
            tmem_ld(td, v[0]);
            if constexpr (EX) tmem_ld(td + DC, u[0]);
            if constexpr (KM) tmem_ld(tm, w[0]);
          }
#pragma unroll
          for (int c = 0; c < NP * 32; c += 8) {
            const int cur = PIPE ? (c >> 3) & 1 : 0, col = STRIDE * (c >> 3), nxt = col + STRIDE;
            if (col < nv) {
              if (!PIPE) {
                tmem_ld(td + col, v[0]);
                if constexpr (KM) tmem_ld(tm + col, w[0]);
              }
              tmem_ld_wait(v[cur]);
              if constexpr (EX) tmem_ld_done(u[cur]);
              if constexpr (KM) tmem_ld_done(w[cur]);
              if (PIPE && c + 8 < NP * 32 && nxt < nv) {
                tmem_ld(td + nxt, v[PIPE ? cur ^ 1 : 0]);
                if constexpr (EX) tmem_ld(td + DC + nxt, u[PIPE ? cur ^ 1 : 0]);
                if constexpr (KM) tmem_ld(tm + nxt, w[PIPE ? cur ^ 1 : 0]);
              }
#pragma unroll
              for (int i = 0; i < 8; i += 4) {
                const ulonglong2 dx = *(const ulonglong2*)(xp + c + i);
                uint64_t* o = out + half * NP * 16 + (c + i) / 2;
                if constexpr (EX) {                // the steps of the int8 kernels, each rounded
#pragma unroll
                  for (int k = 0; k < 2; ++k) {
                    const uint64_t d = k ? dx.y : dx.x, v2 = pack2u(v[cur][i + 2 * k], v[cur][i + 2 * k + 1]), u2 = pack2u(u[cur][i + 2 * k], u[cur][i + 2 * k + 1]);
                    if constexpr (KM) o[k] = add2(o[k], mul2_rn(mul2(d, dm2), pack2u(w[cur][i + 2 * k], w[cur][i + 2 * k + 1]), nz2));
                    o[k] = add2(o[k], mul2_rn(mul2(dw2, d), KM ? add2(v2, u2) : fma2(v2, pack2(16.0f, 16.0f), u2), nz2));
                  }
                  continue;
                }
                if constexpr (KM) {
                  o[0] = fma2(mul2(dx.x, dm2), pack2u(w[cur][i], w[cur][i + 1]), o[0]);
                  o[1] = fma2(mul2(dx.y, dm2), pack2u(w[cur][i + 2], w[cur][i + 3]), o[1]);
                }
                o[0] = fma2(mul2(dw2, dx.x), pack2u(v[cur][i], v[cur][i + 1]), o[0]);
                o[1] = fma2(mul2(dw2, dx.y), pack2u(v[cur][i + 2], v[cur][i + 3]), o[1]);
              }
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_free[b]);
          ++g;
        }
        __syncwarp();                              // the scales of this block have been read
      }
      const bool second = nt >= ntn1;
      if (second) nt -= ntn1;
      const int n = nt * MM_BN + m;
      if (ok && n < p.nrows) {
        const float fin_scale = FMT == ILL_IQ2_XXS ? 0.125f : 1.0f;
        float* ycol = (second ? p.y2 : p.y) + n;
        const unsigned ys = (unsigned)p.y_stride;
        // eight rows of X at a time: the rows of Y (or what is added to) first, then the stores: a load does not wait
        // for the store before it
#pragma unroll
        for (int i0 = 0; i0 < HALVES * NP * 32; i0 += 8) {
          const int c0 = 128 * (i0 / (32 * NP)) + column(i0 % (32 * NP));
          if (c0 < nvalid) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float((uint32_t)(out[(i0 + i) >> 1] >> (32 * (i & 1)))) * fin_scale;
            if (!DENSE && p.ymap) {
              unsigned yr[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) yr[i] = c0 + i < nvalid ? __ldg(p.ymap + row0 + c0 + i) : 0u;
              if (p.ypeers) {
                // the combine of an expert-parallel chunk, fused: the row goes straight into the memory of the
                // rank that owns its token (a plain store over NVLink), tile by tile as the products finish
#pragma unroll
                for (int i = 0; i < 8; ++i)
                  if (c0 + i < nvalid)
                    *((float*)(uintptr_t)__ldg(p.ypeers + (yr[i] >> 24)) + (size_t)(yr[i] & 0xffffffu) * ys + n) = v[i];
              } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                  if (c0 + i < nvalid) ycol[(size_t)yr[i] * ys] = v[i];
              }
            } else {
              float* yp = ycol + (size_t)(row0 + c0) * ys;
              if (DENSE && p.acc) {
                float old[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) old[i] = c0 + i < nvalid ? yp[(size_t)i * ys] : 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = old[i] + v[i];
              }
              if (c0 + 8 <= nvalid) {
#pragma unroll
                for (int i = 0; i < 8; ++i, yp += ys) *yp = v[i];
              } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                  if (c0 + i < nvalid) yp[(size_t)i * ys] = v[i];
              }
            }
          }
        }
      }
    }
  } else {
    // ---- the other warps turn the raw blocks into the A operand in tensor memory: a thread makes two K steps (half H) of its
    // weight row in every SETS-th block of the CTA, so the tensor core can start on a K step while the others are still being
    // made.  The two warps with the same rows bring their raw windows (cp.async) a block of theirs ahead.  (Rows past the
    // matrix's last: whatever lies in shared memory; they are not stored.)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(G::REGS_DQ));
    const int wi = warp - (4 + G::DR_WARPS), wq = wi & 3, h = (wi >> 2) & 1, set = wi >> 3, row = 32 * wq + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(wq * 32) << 16) + G::A_COL;  // this warp's lanes
    // this lane's row in the two warps' two buffers (TMA: in the set's two)
    const uint32_t buf_bytes = tma ? W_BYTES : G::RAW_BYTES;
    const u8* praw = !tma ? raw + (set * 4 + wq) * 2 * G::RAW_BYTES + lane * PITCH
                     : FMT == ILL_Q4_K ? raw + set * 2 * W_BYTES + row * PITCH : raw + set * 2 * W_BYTES + (lane & 3) * G::RAW_BYTES + (row >> 2) * PITCH;
    uint64_t* rfull = raw_full + (tma ? set : set * 4 + wq) * 2;
    uint64_t* rempty = raw_empty + (tma ? set : set * 4 + wq) * 2;
    const uint4* grid = iq_grid + (lane & 7);
    const uint32_t* sgn = iq_sgn + lane;
    int tile = cta, kb = set;               // the block that is fetched next: of the CTA's blocks, every SETS-th
    const u8* wrow0 = nullptr;                     // the warp's first row of the tile's matrix
    int rows_here = 0;
    auto at_tile = [&]() {
      if (tile >= ntiles) return;
      int expert, row0, nvalid, nt;
      locate(tile, expert, row0, nvalid, nt);
      const bool second = nt >= ntn1;
      if (second) nt -= ntn1;
      wrow0 = (const u8*)(uintptr_t)mm_ptr<DENSE>(p, expert) + (second ? p.add2 : p.add) + (long long)(nt * MM_BN + 32 * wq) * p.row_bytes;
      rows_here = min(32, p.nrows - nt * MM_BN - 32 * wq);
    };
    auto to_block = [&]() {                        // on to the tile that block kb falls in
      while (kb >= nkb && tile < ntiles) { kb -= nkb; tile += ctas; if (kb < nkb) at_tile(); }
    };
    auto start = [&]() { return ((uint32_t)(uintptr_t)wrow0 + (uint32_t)lane * (uint32_t)p.row_bytes + (uint32_t)kb * BB) & 15u; };
    auto fetch = [&](int buf) -> uint32_t {        // this warp's part of block kb's windows; where the lane's row starts in its own
      if (!G::LOADERS && !tma)
        mm_fetch<FMT, NT>(wrow0 + (long long)kb * BB, p.row_bytes, rows_here, h, lane, raw + ((set * 4 + wq) * 2 + buf) * G::RAW_BYTES, &rfull[buf]);
      return start();
    };
    at_tile();
    to_block();
    uint32_t o16n = 0;
    bool more = tile < ntiles;
    if (more) o16n = fetch(0);
    for (int g_kb = set, it = 0; more; g_kb += G::SETS, ++it) {
      const int buf = it & 1;
      const uint32_t o16 = o16n;
      // the next block into the other buffer, once both warps have read the block before from it
      kb += G::SETS;
      to_block();
      more = tile < ntiles;
      if (more) {
        if (!G::LOADERS && !tma && !__all_sync(0xffffffffu, mbar_wait(&rempty[buf ^ 1], ((uint32_t)(it + 1) >> 1 & 1u) ^ 1u, p.status, ST_MM_WAIT_EMPTY + 2))) { ok = false; break; }
        o16n = fetch(buf ^ 1);
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&rfull[buf], (uint32_t)(it >> 1) & 1u, p.status, ST_MM_WAIT_FULL + 2))) { ok = false; break; }
      const uint32_t sh = (o16 & 2u) * 8u;         // IQ2_XXS, Q6_K: the block may start in the middle of a word
      const uint32_t* mine = (const uint32_t*)(praw + (buf ? buf_bytes : 0u));
      const uint32_t* rw = mine + (o16 >> 2);
      uint32_t dd, m4[2] = {0, 0};                 // d, dmin; Q4_K: the half's scales and mins, Q2_K: its eight scale bytes
      if constexpr (FMT == ILL_IQ2_XXS) dd = rw[0] >> sh;
      else if constexpr (FMT == ILL_Q6_K) dd = rw[52] >> sh;
      else if constexpr (FMT == ILL_Q4_K) {        // (a Q4_K block is 16-byte aligned)
        const uint4 hd = *(const uint4*)mine;
        dd = hd.x;
        const uint32_t s12[3] = {hd.y, hd.z, hd.w};
        q4k_scales_mins(s12, h, m4[0], m4[1]);
      } else {
        dd = rw[20];
        m4[0] = rw[2 * h]; m4[1] = rw[2 * h + 1];
      }
      const int slot = (4 * g_kb) % NSLOT;
      const int prev = g_kb - NSLOT / 4;           // the block that was in the slots before
      auto slot_free = [&](int j) {                // its MMAs of the K step must be done
        if (prev >= 0)
          ok = __all_sync(0xffffffffu, mbar_wait(&aempty[4 * (prev & 1) + j], (uint32_t)(prev >> 1) & 1u, p.status, ST_MM_WAIT_EMPTY + 1));
        tc_fence_after();
        if (j == 0) {
          // The drain of four blocks back is over: the MMAs that freed this slot were issued after it.
          wsc[(g_kb & 3) * 256 + row] = h2f(dd & 0xffff);
          if (KM) wsc[(g_kb & 3) * 256 + 128 + row] = h2f(dd >> 16);
        }
        return ok;
      };
      const uint32_t a0 = lane_base + G::SLOTW * (slot + 2 * h);
      if constexpr (FMT == ILL_Q6_K) {
        // Left out for timing, 2560 x 9728 x 64 tokens of 62 us: what follows 19, its second stores 4, the raw copies 6 where these warps
        // ask for them (one after the other in a warp; five or six slots in place of four gave nothing, reading the words in pairs neither).
        // Step jj of the half has the nibbles at shift 4 jj of ql[0 .. 63]; columns 32 sb .. of it go with the 2-bit fields at shift
        // 2 (2 jj + sb) of qh.  Sixteen weights (a group) at a time.
        uint32_t sc[2], se[2], so[2], ql[16], qh[8];
        raw_words<2>(rw + 48 + 2 * h, sh, sc);
        raw_words<16>(rw + 16 * h, sh, ql);
        raw_words<8>(rw + 32 + 8 * h, sh, qh);
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) q6k_parts<EX>(sc[jj], se[jj], so[jj]);
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
#pragma unroll
          for (int gr = 0; gr < 4; ++gr) {         // 16 weights: columns 32 sb + 16 hf
            const int sb = gr >> 1, hf = gr & 1;
            uint32_t ev[8], od[8];
            // (1024 + part, plus its offset) / 16, less the rest
            w_q6k(ql + 8 * sb + 4 * hf, qh + 4 * hf, jj, 2 * (2 * jj + sb), hfma2(byte_h2_1024(se[jj], 2 * sb + hf), 0x2c002c00u, EX ? 0xd408d408u : 0xd480d480u),
                  hfma2(byte_h2_1024(so[jj], 2 * sb + hf), 0x2c002c00u, 0xd400d400u), ev, od);
            if (gr == 0 && !slot_free(2 * h + jj)) break;
            tmem_st8(a0 + G::SLOTW * jj + 16 * sb + 8 * hf, ev);
            tmem_st8(a0 + G::SLOTW * jj + 32 + 16 * sb + 8 * hf, od);
          }
          if (!ok) break;
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&afull[slot + 2 * h + jj]);
            if (jj == 1) mbar_arrive(&rempty[buf]);  // every word has been used: a load that is only asked for may still be under way
          }
        }
      } else {
        uint32_t w[8];
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {           // K step j = 2 h + jj
          const int j = 2 * h + jj;
#pragma unroll
          for (int sb = 0; sb < 2; ++sb) {         // 32 weights = 16 columns at a time
            uint32_t v[16];
            if constexpr (FMT == ILL_IQ2_XXS) {    // sub-block 2 j + sb
              if (sb == 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = __funnelshift_rc(rw[4 * j + i], rw[4 * j + i + 1], 16 + sh);
              }
              w_iq2xxs(w[2 * sb], w[2 * sb + 1], grid, sgn, v);
            } else if constexpr (FMT == ILL_Q4_K) {  // group 2 j + sb: the low or the high nibbles of chunk j
              if (sb == 0) {
                const uint4 a = *(const uint4*)(mine + 4 + 8 * j), c = *(const uint4*)(mine + 8 + 8 * j);
                w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = c.x; w[5] = c.y; w[6] = c.z; w[7] = c.w;
              }
              if (sb == 0) w_fields<8, 0>(w, 0x0f0f0f0fu, m4[0], 2 * jj, v);
              else w_fields<8, 4>(w, 0xf0f0f0f0u, m4[0], 2 * jj + 1, v);
            } else {                               // shift 2 (2 jj + sb) of the half's quants; scale bytes 4 j + 2 sb, + 1
              if (jj == 0 && sb == 0) {
#pragma unroll
                for (int i = 0; i < 8; ++i) w[i] = rw[4 + 8 * h + i];
              }
              const uint32_t sc = m4[jj] & 0x0f0f0f0fu;
              if (jj == 0 && sb == 0) { w_fields<4, 0>(w, 0x03030303u, sc, 0, v); w_fields<4, 0>(w + 4, 0x03030303u, sc, 1, v + 8); }
              else if (jj == 0) { w_fields<4, 2>(w, 0x0c0c0c0cu, sc, 2, v); w_fields<4, 2>(w + 4, 0x0c0c0c0cu, sc, 3, v + 8); }
              else if (sb == 0) { w_fields<4, 4>(w, 0x30303030u, sc, 0, v); w_fields<4, 4>(w + 4, 0x30303030u, sc, 1, v + 8); }
              else { w_fields<4, 6>(w, 0xc0c0c0c0u, sc, 2, v); w_fields<4, 6>(w + 4, 0xc0c0c0c0u, sc, 3, v + 8); }
            }
            if (sb == 0 && !slot_free(j)) break;   // (the first 32 weights are made before the slot is waited for)
            tmem_st16(a0 + G::SLOTW * jj + 16 * sb, v);
          }
          if (!ok) break;
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&afull[slot + j]);
            if (jj == 1) mbar_arrive(&rempty[buf]);  // both K steps' words have been read
          }
        }
      }
      if (!ok) break;
      if constexpr (KM) {
        const int mb = g_kb & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(&mempty[mb], ((uint32_t)(g_kb >> 1) & 1u) ^ 1u, p.status, ST_MM_WAIT_EMPTY + 3))) { ok = false; break; }
        uint32_t v[4];
        // half h's eight mins: K = 8 h .. 8 h + 7 of the 16, chunk h of the row (Q4_K: groups 4 h .. 4 h + 3, each twice)
        if constexpr (FMT == ILL_Q4_K) w_q4k_mins(m4[1], v);
        else w_q2k_mins(m4[0], m4[1], v);
        store_chunk32(m_tiles + mb * G::M_BYTES, row, h, make_uint4(v[0], v[1], v[2], v[3]));
        fence_async_smem();  // the tensor core reads the tile through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(&mfull[mb]);
      }
    }
    cp_async_wait_all();
  }
}

// What an expert of C rows costs in tiles of up to 64 and of up to 128 rows of X (Q2_K, Q4_K), in hundredths of a tile of 64 with
// 16 rows.  Measured on Q2_K, a tile an expert: of 64 with 16, 32, 48, 64 rows 100, 106, 114, 131; of 128 with 16, 64, 96, 128 rows
// 142, 158, 168, 190.
__device__ __forceinline__ int mm_cost64(int c) { return c / 64 * 131 + (c % 64 ? 92 + 6 * (c % 64) / 10 : 0); }
__device__ __forceinline__ int mm_cost128(int c) { return c / 128 * 190 + (c % 128 ? 134 + 4 * (c % 128) / 10 : 0); }

// NT2: tiles of up to NT2 rows of X in place of NT where the experts' rows ask for them.  Only the device knows the rows, and a mean
// of what the host knows misleads where the tokens meet in few experts (or where TOTAL_ROWS is a capacity): every tile unpacks its
// expert's weights again.  us, all tiles of 128 / of 64 / picked here, 288 experts, Q2_K, gate and up of 1536 x 5120: 64 tokens
// 1000 / 665 / 660; 512 that all choose the same eight 193 / 251 / 190; 1400 skewed by 1 / rank^0.4 1241 / - / 1044, 4096 1756 / - / 1788.
// Where the two are close tiles of 128 are taken: many small tiles of few columns cost more than the sum says (model 0.93, measured 1.03).
template <int FMT, bool DENSE, int NT, int NT2>
__global__ void __launch_bounds__(MmGeom<FMT, NT>::THREADS, 1) mm_id_kernel(const __grid_constant__ MmMaps maps, const MmParams p) {
  typedef MmGeom<FMT, NT> G;
  typedef MmSmem<FMT, NT, NT2> S;
  constexpr uint32_t TMEM_COLS = 512;
  static_assert(!NT2 || MmGeom<FMT, NT2 ? NT2 : NT>::THREADS == G::THREADS, "one launch for both");
  static_assert(sizeof(MmBars<FMT, NT>) <= MM_BARS && sizeof(MmBars<FMT, NT2 ? NT2 : NT>) <= MM_BARS, "barriers");
  extern __shared__ __align__(1024) u8 smem_raw[];
  u8* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  MmBars<FMT, NT>* bars = (MmBars<FMT, NT>*)(smem + S::BODY);
  MmBars<FMT, NT2 ? NT2 : NT>* bars2 = (MmBars<FMT, NT2 ? NT2 : NT>*)(smem + S::BODY + MM_BARS);
  int* tile_first = (int*)(smem + S::FIRST);          // [ne + 1] first row tile of each expert; the total
  uint32_t* tmem_slot = (uint32_t*)(smem + S::SLOTS);
  uint32_t* narrow = tmem_slot + 1;                   // NT2: tiles of up to NT2 rows
  uint4* iq_grid = (uint4*)(smem + S::TABLES);        // [256 entries][8 copies] the grid as halves
  uint32_t* iq_sgn = (uint32_t*)(iq_grid + 8 * 256);  // [128 entries][32 copies] the eight signs (w_iq2xxs)

  // the warp number through a shuffle: the compiler then knows that the role branches are warp-uniform
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

  // ---- once per CTA: barriers, tables, tensor memory; then, after the kernel before, the experts' row tiles counted
  // (first tile of each expert, in shared memory).
  pdl_launch_dependents();
  if (tid == 32) {
    bars->init(mm_tma<FMT, DENSE>(p));
    if constexpr (NT2 != 0) bars2->init(mm_tma<FMT, DENSE>(p));
    mbar_fence_init();
  }
  if (FMT == ILL_IQ2_XXS) {
    for (int i = tid; i < 8 * 256; i += G::THREADS) {
      const uint64_t g = ill_iq2xxs_grid[i >> 3];
      uint32_t h[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const __half2 hh = __floats2half2_rn((float)((g >> (16 * k)) & 0xff), (float)((g >> (16 * k + 8)) & 0xff));
        h[k] = *(const uint32_t*)&hh;
      }
      iq_grid[i] = make_uint4(h[0], h[1], h[2], h[3]);
    }
    for (int i = tid; i < 32 * 128; i += G::THREADS) {
      const uint32_t s7 = (uint32_t)i >> 5, sg = s7 | ((__popc(s7) & 1u) << 7);
      iq_sgn[i] = (sg << 9) | (sg << 24);
    }
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  pdl_wait();
  int bm = DENSE ? p.bm : NT;
  if constexpr (NT2 != 0) {  // every expert's rows, all loads at once
    for (int e = tid; e < p.ne; e += G::THREADS) {
      const int c = mm_count<DENSE>(p, e);
      tile_first[e] = c > p.over ? min(c, 1 << 22) : 0;
    }
    __syncthreads();
  }
  if (warp == 0) {
    if constexpr (NT2 != 0) {
      float more = 0.0f;                         // what tiles of NT2 cost more, for a margin of a tenth
      for (int e = lane; e < p.ne; e += 32) {
        const int c = tile_first[e];
        more += 1.1f * (float)mm_cost64(c) - (float)mm_cost128(c);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) more += __shfl_xor_sync(0xffffffffu, more, o);
      if (more <= 0.0f) bm = NT2;
      if (lane == 0) *narrow = bm == NT2;
    }
    int before = 0;
    for (int e0 = 0; e0 < p.ne; e0 += 32) {
      const int e = e0 + lane;
      int c = e >= p.ne ? 0 : NT2 ? tile_first[e] : mm_count<DENSE>(p, e);
      if (!NT2 && !DENSE && c <= p.over) c = 0;
      const int tiles = (c + bm - 1) / bm;
      int incl = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (e < p.ne) tile_first[e] = before + incl - tiles;
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) tile_first[p.ne] = before;  // row tiles in all
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  if constexpr (NT2 != 0) {
    if (__shfl_sync(0xffffffffu, *narrow, 0)) mm_tiles<FMT, DENSE, NT2>(maps, p, NT2, smem, bars2, tile_first, iq_grid, iq_sgn, tmem_base, warp, lane, blockIdx.x, gridDim.x);
    else mm_tiles<FMT, DENSE, NT>(maps, p, NT, smem, bars, tile_first, iq_grid, iq_sgn, tmem_base, warp, lane, blockIdx.x, gridDim.x);
  } else {
    mm_tiles<FMT, DENSE, NT>(maps, p, DENSE ? p.bm : NT, smem, bars, tile_first, iq_grid, iq_sgn, tmem_base, warp, lane, blockIdx.x, gridDim.x);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// Two dense matrices of few rows (K and V) against a chunk, with the bits of the int8 kernel of mma.sync: EX's accumulators hold a
// block's sum exactly, and the drain takes that kernel's float steps.  FMT2 other than FMT: the second matrix (P2) is of another format,
// and CTAs SPLIT and up take its tiles.  Bound by the unpacking of one block after the other in a CTA (0.75 us a block of Q4_K, 1.13
// of Q6_K, and 0.004 a row of X).  us, the int8 kernel's joint launch / this: K and V of 1024 x 2560, 512 tokens, both Q4_K 44 / 19.4, one of
// Q6_K 48 / 23.4; of 1024 x 5120, both Q6_K 86 / 38.
template <int FMT, int FMT2>
__global__ void __launch_bounds__(MmGeom<FMT, 64, true>::THREADS, 1)
    mm_exact_kernel(const __grid_constant__ MmMaps maps, const MmParams p, const MmParams p2, int split) {
  typedef MmGeom<FMT, 64, true> G;
  typedef MmExactSmem<FMT, FMT2> S;
  constexpr uint32_t TMEM_COLS = 512;
  static_assert(MmGeom<FMT2, 64, true>::THREADS == G::THREADS, "one launch for both");
  static_assert(sizeof(MmBars<FMT, 64, true>) <= MM_BARS && sizeof(MmBars<FMT2, 64, true>) <= MM_BARS, "barriers");
  extern __shared__ __align__(1024) u8 smem_raw[];
  u8* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  MmBars<FMT, 64, true>* bars = (MmBars<FMT, 64, true>*)(smem + S::BODY);
  MmBars<FMT2, 64, true>* bars2 = (MmBars<FMT2, 64, true>*)(smem + S::BODY);
  int* tile_first = (int*)(smem + S::BODY + MM_BARS);
  uint32_t* tmem_slot = (uint32_t*)(tile_first + 2);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const bool second = FMT2 != FMT && (int)blockIdx.x >= split;
  pdl_launch_dependents();
  if (tid == 32) {
    if (second) bars2->init(mm_tma<FMT2, true>(p2));
    else bars->init(mm_tma<FMT, true>(p));
    mbar_fence_init();
    tile_first[0] = 0;
    tile_first[1] = (int)((p.one_count + p.bm - 1) / p.bm);
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  if constexpr (FMT2 != FMT) {
    if (second) mm_tiles<FMT2, true, 64, true>(maps, p2, p2.bm, smem, bars2, tile_first, nullptr, nullptr, tmem_base, warp, lane, blockIdx.x - split, gridDim.x - split);
    else mm_tiles<FMT, true, 64, true>(maps, p, p.bm, smem, bars, tile_first, nullptr, nullptr, tmem_base, warp, lane, blockIdx.x, split);
  } else {
    mm_tiles<FMT, true, 64, true>(maps, p, p.bm, smem, bars, tile_first, nullptr, nullptr, tmem_base, warp, lane, blockIdx.x, gridDim.x);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// The Q8_K activations as the tensor cores take them, in expert order: XH[place, k] = fp16(q[t, k])
// (exact), t = MAP[place] (or place when MAP is null); and, when XE is given, the sums of 16 as
// XE[place, kb, 0..15] = fp16(bsums[t, 16 kb ..]) (exact: at most 2032), the other 48 of each 64 zero.
// Row t's quants are at XQ + t * XQ_STRIDE bytes and its sums at BSUMS + t * BS_STRIDE bytes.  With XD_OUT,
// the row also carries its block scales (SC + t * XQ_STRIDE) and a weight (WT + t * XQ_STRIDE), copied
// to XD_OUT[place, kb] and W_OUT[place]: the rows of an expert-parallel exchange, unpacked.
__global__ void __launch_bounds__(256) act_f16_kernel(long long rows, int cols, const u8* __restrict__ xq, long long xq_stride,
                                                      const u8* __restrict__ bsums, long long bs_stride,
                                                      const unsigned* __restrict__ map, __half* __restrict__ xh,
                                                      __half* __restrict__ xe, const u8* __restrict__ sc,
                                                      const u8* __restrict__ wt, float* __restrict__ xd_out,
                                                      float* __restrict__ w_out, const unsigned* __restrict__ rows_dev,
                                                      const unsigned* __restrict__ counts, int ne, int over) {
  pdl_launch_dependents();
  pdl_wait();
  if (counts) {  // nothing to do unless some expert has more than OVER rows
    bool any = false;
    for (int e = threadIdx.x; e < ne; e += blockDim.x) any = any || (int)counts[e] > over;
    if (!__syncthreads_or(any)) return;
  }
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // one thread: 16 values
  const int per_row = cols / 16;
  if (gid >= rows * per_row) return;
  const long long place = gid / per_row;
  if (rows_dev && place >= (long long)*rows_dev) return;  // the rows in use, known on the device only
  const int j = (int)(gid - place * per_row);
  const long long t = map ? (long long)map[place] : place;
  const uint4 q = *(const uint4*)(xq + t * xq_stride + 16 * j);
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  uint32_t h[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int b0 = (int)(signed char)((w[i >> 1] >> (16 * (i & 1))) & 0xff);
    const int b1 = (int)(signed char)((w[i >> 1] >> (16 * (i & 1) + 8)) & 0xff);
    const __half2 hh = __floats2half2_rn((float)b0, (float)b1);
    h[i] = *(const uint32_t*)&hh;
  }
  uint4* dst = (uint4*)(xh + place * cols + 16 * j);
  dst[0] = make_uint4(h[0], h[1], h[2], h[3]);
  dst[1] = make_uint4(h[4], h[5], h[6], h[7]);
  if (xe) {
    // this thread's 16 quants are one sum of 16: element j%16 of block j/16; it also clears 3 of the 48 zeros
    const int kb = j >> 4, g = j & 15;
    __half* e = xe + (place * (cols / 256) + kb) * 64;
    e[g] = __float2half_rn((float)((const int16_t*)(bsums + t * bs_stride))[j]);
    e[16 + 3 * g] = __float2half_rn(0.0f);
    e[16 + 3 * g + 1] = __float2half_rn(0.0f);
    e[16 + 3 * g + 2] = __float2half_rn(0.0f);
  }
  if (xd_out) {
    if (j < cols / 256) xd_out[place * (cols / 256) + j] = ((const float*)(sc + t * xq_stride))[j];
    if (j == per_row - 1) w_out[place] = *(const float*)(wt + t * xq_stride);
  }
}

// A row of an expert-parallel exchange: the token's Q8_K form and its routing weight in one piece,
//   [cols int8 quants][cols/256 float scales][cols/16 int16 sums][float weight][pad to 16 bytes]
// PACKED[place] from token MAP[place]'s quantized activations and W[place].  One block a row.
__global__ void __launch_bounds__(128) ep_pack_kernel(int cols, long long row_bytes, const uint32_t* __restrict__ xq,
                                                      const uint32_t* __restrict__ xs, const uint32_t* __restrict__ xsum,
                                                      const uint32_t* __restrict__ w, const unsigned* __restrict__ map,
                                                      uint32_t* __restrict__ packed) {
  pdl_launch_dependents();
  pdl_wait();
  const long long place = blockIdx.x;
  const long long t = map[place];
  const int nq = cols / 4, ns = cols / 256, nb = cols / 32;  // words of quants, scales, sums
  uint32_t* dst = packed + place * (row_bytes / 4);
  for (int i = threadIdx.x; i < nq + ns + nb + 1; i += blockDim.x) {
    uint32_t v;
    if (i < nq) v = xq[t * nq + i];
    else if (i < nq + ns) v = xs[t * ns + (i - nq)];
    else if (i < nq + ns + nb) v = xsum[t * nb + (i - nq - ns)];
    else v = w[place];
    dst[i] = v;
  }
}

// ep_pack_kernel for exchanges of a fixed size: rank g's rows go to slab g of PACKED, CAP rows a slab, in the
// order of their places; PSLOT[place] = the row's slot (g * cap + index in the slab).  BASES[e] = first place
// of expert e on this rank (ill_moe_group), so destination g's rows are places [bases[g * per], bases[(g + 1) *
// per]).  A slab that would overflow sets *OVERFLOW and drops the rows past CAP.
__global__ void __launch_bounds__(128) ep_pack_cap_kernel(int cols, long long row_bytes, const uint32_t* __restrict__ xq,
                                                          const uint32_t* __restrict__ xs, const uint32_t* __restrict__ xsum,
                                                          const uint32_t* __restrict__ w, const unsigned* __restrict__ map,
                                                          const unsigned* __restrict__ bases, int per, int world, int cap,
                                                          long long rows, uint32_t* __restrict__ packed,
                                                          unsigned* __restrict__ pslot, unsigned* __restrict__ overflow,
                                                          const unsigned long long* __restrict__ peers, int rank) {
  pdl_launch_dependents();
  pdl_wait();
  const long long place = blockIdx.x;
  __shared__ long long slot_s;
  __shared__ int dest_s;
  if (threadIdx.x == 0) {
    int g = 0;
    while (g + 1 < world && (long long)bases[(g + 1) * per] <= place) ++g;
    const long long idx = place - (long long)bases[g * per];
    dest_s = g;
    if (idx >= cap) { atomicOr(overflow, 1u); slot_s = -1; pslot[place] = 0; }
    else { slot_s = (long long)g * cap + idx; pslot[place] = (unsigned)slot_s; }
  }
  __syncthreads();
  long long slot = slot_s;
  if (slot < 0) return;
  if (peers) {
    // the dispatch without a collective: the row is stored into slab RANK of the receiving rank's buffer
    packed = (uint32_t*)(uintptr_t)peers[dest_s];
    slot = (long long)rank * cap + (slot - (long long)dest_s * cap);
  }
  const long long t = map[place];
  const int nq = cols / 4, ns = cols / 256, nb = cols / 32;  // words of quants, scales, sums
  uint32_t* dst = packed + slot * (row_bytes / 4);
  // the quants 16 bytes at a time (a token's quants and a packed row both start on 16-byte boundaries), the rest by words
  for (int i = threadIdx.x; i < nq / 4; i += blockDim.x) ((uint4*)dst)[i] = ((const uint4*)(xq + t * nq))[i];
  for (int i = nq + threadIdx.x; i < nq + ns + nb + 1; i += blockDim.x) {
    uint32_t v;
    if (i < nq + ns) v = xs[t * ns + (i - nq)];
    else if (i < nq + ns + nb) v = xsum[t * nb + (i - nq - ns)];
    else v = w[place];
    dst[i] = v;
  }
}

// The whole dispatch of an expert-parallel chunk in one launch: block T quantizes token T's activations once (Q8_K,
// the arithmetic of quant_q8_k_kernel: the same bits) into a packed row in shared memory and stores it, for each of
// the token's NU slots, into slab RANK of that expert's rank (peer memory) with the slot's weight appended -- the
// quantized token never passes through this rank's memory, and what ep_pack_cap_kernel, quant_q8_k_kernel and
// ep_put_counts_kernel do in three launches is done in one; the first blocks also store this rank's rows-per-expert
// into row RANK of every rank's table.  A slab that would overflow raises *OVERFLOW to EPOCH (never cleared: the
// chunk with that number overflowed) and drops the rows past CAP.
constexpr int EP_MAX_NU = 32;
__global__ void __launch_bounds__(128) ep_dispatch_kernel(int cols, int nu, long long row_bytes, const float* __restrict__ x,
                                                          const uint32_t* __restrict__ w, const unsigned* __restrict__ smap,
                                                          const unsigned* __restrict__ bases, const unsigned* __restrict__ counts,
                                                          int per, int world, int cap, unsigned* __restrict__ pslot,
                                                          unsigned* __restrict__ overflow, unsigned epoch,
                                                          const unsigned long long* __restrict__ peers_rows,
                                                          const unsigned long long* __restrict__ peers_rc, int rank) {
  extern __shared__ __align__(16) u8 srow[];  // the token's packed row (without the weight)
  __shared__ unsigned long long dst_s[EP_MAX_NU];  // where slot s's row goes (0: dropped)
  __shared__ uint32_t w_s[EP_MAX_NU];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  {
    const int i = blockIdx.x * 128 + tid;
    if (i < world * per) ((unsigned*)(uintptr_t)peers_rc[i / per])[rank * per + (i % per)] = counts[i];
  }
  const long long t = blockIdx.x;
  if (tid < nu) {
    const long long place = smap[t * nu + tid];
    int g = 0;
    while (g + 1 < world && (long long)bases[(g + 1) * per] <= place) ++g;
    const long long idx = place - (long long)bases[g * per];
    if (idx >= cap) { atomicMax(overflow, epoch); dst_s[tid] = 0; pslot[place] = 0; }
    else {
      pslot[place] = (unsigned)((long long)g * cap + idx);
      dst_s[tid] = peers_rows[g] + (unsigned long long)(((long long)rank * cap + idx) * row_bytes);
    }
    w_s[tid] = w[place];
  }
  const float* xr = x + t * cols;
  const int nb = cols / 256;
  float* dscale = (float*)(srow + cols);
  int16_t* dsum = (int16_t*)(srow + cols + nb * 4);
  for (int b = warp; b < nb; b += 4) {
    const float4 v0 = ((const float4*)(xr + b * 256))[2 * lane], v1 = ((const float4*)(xr + b * 256))[2 * lane + 1];
    const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    int q[8];
    float d;
    q8k_values(v, lane, q, d);
    uint32_t w0, w1;
    int sum = q8k_pack(q, w0, w1);
    ((uint2*)(srow + b * 256))[lane] = make_uint2(w0, w1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    if (!(lane & 1)) dsum[b * 16 + (lane >> 1)] = (int16_t)sum;
    if (lane == 0) dscale[b] = d;
  }
  __syncthreads();
  // the packed row to each of its destinations, 16 bytes a thread at a time (rows and slabs are 16-byte aligned);
  // the last word, after the sums, is the slot's weight
  const int body = cols + nb * 4 + cols / 8, nv = body / 16;
  for (int s = 0; s < nu; ++s) {
    u8* dst = (u8*)(uintptr_t)dst_s[s];
    if (!dst) continue;
    for (int i = tid; i < nv; i += 128) ((uint4*)dst)[i] = ((const uint4*)srow)[i];
    for (int i = nv * 4 + tid; i < body / 4; i += 128) ((uint32_t*)dst)[i] = ((const uint32_t*)srow)[i];
    if (tid == 0) *(uint32_t*)(dst + body) = w_s[s];
  }
}

// The receiving rank's plan, on the device, for exchanges of a fixed size: RC[s * per + e] = rows source s counted
// for local expert e.  The sender keeps, per destination, only the first CAP rows of its expert order, so of
// those RC rows the ones that arrived are GOT = min(RC, max(0, cap - rows of s's earlier experts)), at slots
// s * cap + (rows of s's earlier experts) ...  Everything below is built from GOT, never from RC, so that the rows
// planned are at most WORLD * CAP whatever the counts say: COUNTS / BASES of the local experts (what ill_moe_mm_id
// reads), P2R[place] = slot of the row placed there (expert by expert, source after source), R2P its inverse on the
// slots in use, P2R of the places past the last row = 0 (a row that exists, so that element-wise steps over all
// CAP * WORLD places read valid memory), TOTAL[0] = rows in all, and *OVERFLOW |= 1 when some source's rows were
// cut (its own flag is up too: that chunk's result is void).  One CTA.
__global__ void __launch_bounds__(256) ep_plan_dev_kernel(int world, int per, int cap, int rank, const unsigned* __restrict__ rc,
                                                          unsigned* __restrict__ counts, unsigned* __restrict__ bases,
                                                          unsigned* __restrict__ p2r, unsigned* __restrict__ r2p,
                                                          unsigned* __restrict__ pdst, unsigned* __restrict__ total,
                                                          unsigned* __restrict__ overflow, const unsigned long long* flag_peers,
                                                          unsigned* flags, unsigned epoch, unsigned long long wait_ns,
                                                          unsigned* status) {
  extern __shared__ unsigned plan_s[];
  unsigned* in_src = plan_s;                 // [world][per] rows of the source's earlier experts (as counted)
  unsigned* before = plan_s + world * per;   // [world][per] rows of the expert that arrived from earlier sources
  unsigned* got = before + world * per;      // [world][per] rows of the segment that arrived
  unsigned* lb = got + world * per;          // [per + 1] first place of each local expert; the total
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x;
  if (flag_peers) {
    // the ranks meet first (slot 0): this rank's rows and counts are in its peers' buffers (the kernels before this
    // one in the stream stored them), and what RC and the slabs hold is complete once every peer has said the same.
    // A meeting that times out leaves a plan of no rows at all.
    const bool ok = ep_meet(flag_peers, flags, world, rank, 0, epoch, true, wait_ns, status);
    if (!__syncthreads_and(ok)) {
      for (int e = tid; e < per; e += blockDim.x) { counts[e] = 0; bases[e] = 0; }
      for (unsigned p = tid; p < (unsigned)(world * cap); p += blockDim.x) {
        p2r[p] = 0;
        if (pdst) pdst[p] = (unsigned)rank << 24 | ((unsigned)rank * cap);
      }
      if (tid == 0) total[0] = 0;
      return;
    }
  }
  for (int s = tid; s < world; s += blockDim.x) {
    unsigned a = 0;
    bool cut = false;
    for (int e = 0; e < per; ++e) {
      const unsigned n = rc[s * per + e];
      const unsigned room = a < (unsigned)cap ? (unsigned)cap - a : 0u;
      in_src[s * per + e] = a;
      got[s * per + e] = n < room ? n : room;
      cut |= n > room;
      a = a + n < a ? 0xffffffffu : a + n;   // saturate: counts are the caller's, not trusted
    }
    if (cut && overflow) { if (flag_peers) atomicMax(overflow, epoch); else atomicOr(overflow, 1u); }
  }
  __syncthreads();
  for (int e = tid; e < per; e += blockDim.x) {
    unsigned a = 0;
    for (int s = 0; s < world; ++s) { before[s * per + e] = a; a += got[s * per + e]; }
    counts[e] = a;
  }
  __syncthreads();
  if (tid == 0) {
    unsigned a = 0;
    for (int e = 0; e < per; ++e) { lb[e] = a; bases[e] = a; a += counts[e]; }
    lb[per] = a;                             // <= world * cap: every source contributes at most cap rows
    total[0] = a;
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  for (int seg = warp; seg < world * per; seg += nw) {
    const int s = seg / per, e = seg - s * per;
    const unsigned n = got[seg], a0 = (unsigned)s * cap + in_src[seg], p0 = lb[e] + before[seg];
    for (unsigned i = lane; i < n; i += 32) {  // in_src + i < cap for every i < got
      p2r[p0 + i] = a0 + i;
      r2p[a0 + i] = p0 + i;
      // where the row's result goes: rank s, row (this rank's slab there) * cap + its index in the slab
      if (pdst) pdst[p0 + i] = ((unsigned)s << 24) | ((unsigned)rank * cap + in_src[seg] + i);
    }
  }
  for (unsigned p = lb[per] + tid; p < (unsigned)(world * cap); p += blockDim.x) {
    p2r[p] = 0;
    if (pdst) pdst[p] = (unsigned)rank << 24 | ((unsigned)rank * cap);
  }
}

// This rank's rows per expert to the experts' ranks, without a collective: COUNTS[g * per + e] into row RANK of
// rank g's [world, per] table (peer memory).
__global__ void __launch_bounds__(256) ep_put_counts_kernel(int world, int per, int rank, const unsigned* __restrict__ counts,
                                                            const unsigned long long* __restrict__ peers,
                                                            unsigned* __restrict__ overflow) {
  pdl_launch_dependents();
  pdl_wait();
  if (overflow && blockIdx.x == 0 && threadIdx.x == 0) *overflow = 0;  // for the pack that follows in the stream
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < world * per; i += gridDim.x * blockDim.x) {
    const int g = i / per, e = i - g * per;
    ((unsigned*)(uintptr_t)peers[g])[rank * per + e] = counts[i];
  }
}

}  // namespace ill

using namespace ill;

static int act_f16_launch(int64_t rows, int cols, const u8* qp, long long qs, const u8* bp, long long bs, ill_dptr map,
                          ill_dptr xh, ill_dptr xe, const u8* sc, const u8* wt, ill_dptr xd_out, ill_dptr w_out,
                          ill_stream stream, ill_dptr rows_dev = 0, ill_dptr counts = 0, int ne = 0, int over = 0) {
  long long nrows = rows;
  const unsigned* mp = (const unsigned*)(uintptr_t)map;
  __half* hp = (__half*)(uintptr_t)xh;
  __half* ep = (__half*)(uintptr_t)xe;
  float* xo = (float*)(uintptr_t)xd_out;
  float* wo = (float*)(uintptr_t)w_out;
  const unsigned* rd = (const unsigned*)(uintptr_t)rows_dev;
  const unsigned* cn = (const unsigned*)(uintptr_t)counts;
  void* args[] = {&nrows, &cols, &qp, &qs, &bp, &bs, &mp, &hp, &ep, &sc, &wt, &xo, &wo, &rd, &cn, &ne, &over};
  const long long threads = rows * (cols / 16);
  return launch_kernel((const void*)act_f16_kernel, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, args,
                       (cudaStream_t)stream);
}

extern "C" int ill_act_f16(int64_t rows, int cols, ill_dptr xq, ill_dptr bsums, ill_dptr map, ill_dptr xh, ill_dptr xe,
                           ill_stream stream) {
  if (rows < 0 || cols <= 0 || cols % 256 || !xq || !xh || (xe && !bsums)) return ILL_ERR_ARG;
  if ((xq & 15) || (bsums & 1) || (map & 3) || (xh & 15) || (xe & 15)) return ILL_ERR_ALIGN;
  if (rows == 0) return ILL_OK;
  return act_f16_launch(rows, cols, (const u8*)(uintptr_t)xq, cols, (const u8*)(uintptr_t)bsums, cols / 8, map, xh, xe, nullptr,
                        nullptr, 0, 0, stream);
}

extern "C" int ill_act_f16_over(int64_t rows, int cols, ill_dptr xq, ill_dptr bsums, ill_dptr map, ill_dptr xh, ill_dptr xe, ill_dptr counts,
                                int ne, int over, ill_stream stream) {
  if (rows < 0 || cols <= 0 || cols % 256 || !xq || !xh || (xe && !bsums) || !counts || ne < 1 || over < 0) return ILL_ERR_ARG;
  if ((xq & 15) || (bsums & 1) || (map & 3) || (xh & 15) || (xe & 15) || (counts & 3)) return ILL_ERR_ALIGN;
  if (rows == 0) return ILL_OK;
  return act_f16_launch(rows, cols, (const u8*)(uintptr_t)xq, cols, (const u8*)(uintptr_t)bsums, cols / 8, map, xh, xe, nullptr,
                        nullptr, 0, 0, stream, 0, counts, ne, over);
}

extern "C" int64_t ill_ep_row_bytes(int cols) {
  if (cols <= 0 || cols % 256) return 0;
  return ((int64_t)cols + cols / 256 * 4 + cols / 16 * 2 + 4 + 15) / 16 * 16;
}

extern "C" int ill_ep_pack(int64_t rows, int cols, ill_dptr xq, ill_dptr xs, ill_dptr xsum, ill_dptr w, ill_dptr map,
                           ill_dptr packed, ill_stream stream) {
  if (rows < 0 || cols <= 0 || cols % 256 || !xq || !xs || !xsum || !w || !map || !packed) return ILL_ERR_ARG;
  if ((xq & 3) || (xs & 3) || (xsum & 3) || (w & 3) || (map & 3) || (packed & 15)) return ILL_ERR_ALIGN;
  if (rows == 0) return ILL_OK;
  long long rb = ill_ep_row_bytes(cols);
  const uint32_t* qp = (const uint32_t*)(uintptr_t)xq;
  const uint32_t* sp = (const uint32_t*)(uintptr_t)xs;
  const uint32_t* bp = (const uint32_t*)(uintptr_t)xsum;
  const uint32_t* wp = (const uint32_t*)(uintptr_t)w;
  const unsigned* mp = (const unsigned*)(uintptr_t)map;
  uint32_t* pp = (uint32_t*)(uintptr_t)packed;
  void* args[] = {&cols, &rb, &qp, &sp, &bp, &wp, &mp, &pp};
  return launch_kernel((const void*)ep_pack_kernel, dim3((unsigned)rows), dim3(128), 0, args, (cudaStream_t)stream);
}

extern "C" int ill_ep_pack_cap(int64_t rows, int cols, ill_dptr xq, ill_dptr xs, ill_dptr xsum, ill_dptr w, ill_dptr map,
                               ill_dptr bases, int per, int world, int cap, ill_dptr packed, ill_dptr pslot, ill_dptr overflow,
                               ill_dptr peers, int rank, ill_stream stream) {
  if (rows < 0 || cols <= 0 || cols % 256 || per < 1 || world < 1 || cap < 1 || !xq || !xs || !xsum || !w || !map || !bases ||
      (!packed && !peers) || !pslot || !overflow || rank < 0 || rank >= world)
    return ILL_ERR_ARG;
  if ((xq & 15) || (xs & 3) || (xsum & 3) || (w & 3) || (map & 3) || (bases & 3) || (packed & 15) || (pslot & 3) || (overflow & 3) ||
      (peers & 7))
    return ILL_ERR_ALIGN;
  if (rows == 0) return ILL_OK;
  long long rb = ill_ep_row_bytes(cols), nrows = rows;
  const uint32_t* qp = (const uint32_t*)(uintptr_t)xq;
  const uint32_t* sp = (const uint32_t*)(uintptr_t)xs;
  const uint32_t* bp = (const uint32_t*)(uintptr_t)xsum;
  const uint32_t* wp = (const uint32_t*)(uintptr_t)w;
  const unsigned* mp = (const unsigned*)(uintptr_t)map;
  const unsigned* bs = (const unsigned*)(uintptr_t)bases;
  uint32_t* pp = (uint32_t*)(uintptr_t)packed;
  unsigned* ps = (unsigned*)(uintptr_t)pslot;
  unsigned* ov = (unsigned*)(uintptr_t)overflow;
  const unsigned long long* pr = (const unsigned long long*)(uintptr_t)peers;
  void* args[] = {&cols, &rb, &qp, &sp, &bp, &wp, &mp, &bs, &per, &world, &cap, &nrows, &pp, &ps, &ov, &pr, &rank};
  return launch_kernel((const void*)ep_pack_cap_kernel, dim3((unsigned)rows), dim3(128), 0, args, (cudaStream_t)stream);
}

extern "C" int ill_ep_dispatch(int64_t ntok, int nu, int cols, ill_dptr x, ill_dptr w, ill_dptr smap, ill_dptr bases, ill_dptr counts,
                               int per, int world, int cap, int rank, ill_dptr peers_rows, ill_dptr peers_rc, ill_dptr pslot,
                               ill_dptr overflow, uint32_t epoch, ill_stream stream) {
  if (ntok < 0 || nu < 1 || nu > EP_MAX_NU || cols <= 0 || cols % 256 || per < 1 || world < 1 || cap < 1 || !x || !w || !smap || !bases ||
      !counts || !peers_rows || !peers_rc || !pslot || !overflow || rank < 0 || rank >= world || epoch == 0)
    return ILL_ERR_ARG;
  if ((x & 15) || (w & 3) || (smap & 3) || (bases & 3) || (counts & 3) || (pslot & 3) || (overflow & 3) || (peers_rows & 7) || (peers_rc & 7))
    return ILL_ERR_ALIGN;
  long long rb = ill_ep_row_bytes(cols);
  if (rb % 16 || rb > 64 * 1024) return ILL_ERR_UNSUPPORTED;
  const float* xp = (const float*)(uintptr_t)x;
  const uint32_t* wp = (const uint32_t*)(uintptr_t)w;
  const unsigned* mp = (const unsigned*)(uintptr_t)smap;
  const unsigned* bs = (const unsigned*)(uintptr_t)bases;
  const unsigned* cp = (const unsigned*)(uintptr_t)counts;
  unsigned* ps = (unsigned*)(uintptr_t)pslot;
  unsigned* ov = (unsigned*)(uintptr_t)overflow;
  const unsigned long long* pr = (const unsigned long long*)(uintptr_t)peers_rows;
  const unsigned long long* pc = (const unsigned long long*)(uintptr_t)peers_rc;
  void* args[] = {&cols, &nu, &rb, &xp, &wp, &mp, &bs, &cp, &per, &world, &cap, &ps, &ov, &epoch, &pr, &pc, &rank};
  const long long need = ((long long)world * per + 127) / 128;  // blocks that carry the counts
  if (ntok < need) return ILL_ERR_UNSUPPORTED;  // fewer tokens than that: use ill_ep_put_counts and ill_ep_pack_cap
  if (rb > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute((const void*)ep_dispatch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rb);
    if (e != cudaSuccess) return cuda_fail(e);
  }
  return launch_kernel((const void*)ep_dispatch_kernel, dim3((unsigned)ntok), dim3(128), (size_t)rb, args, (cudaStream_t)stream);
}

extern "C" int ill_ep_put_counts(int world, int per, int rank, ill_dptr counts, ill_dptr peers, ill_dptr overflow,
                                 ill_stream stream) {
  if (world < 1 || per < 1 || rank < 0 || rank >= world || !counts || !peers) return ILL_ERR_ARG;
  if ((counts & 3) || (peers & 7) || (overflow & 3)) return ILL_ERR_ALIGN;
  const unsigned* cp = (const unsigned*)(uintptr_t)counts;
  const unsigned long long* pr = (const unsigned long long*)(uintptr_t)peers;
  unsigned* ov = (unsigned*)(uintptr_t)overflow;
  void* args[] = {&world, &per, &rank, &cp, &pr, &ov};
  return launch_kernel((const void*)ep_put_counts_kernel, dim3((unsigned)((world * per + 255) / 256)), dim3(256), 0, args,
                       (cudaStream_t)stream);
}

static int ep_plan_dev_launch(int world, int per, int cap, int rank, ill_dptr rc, ill_dptr counts, ill_dptr bases, ill_dptr p2r,
                              ill_dptr r2p, ill_dptr pdst, ill_dptr total, ill_dptr overflow, ill_dptr flag_peers, ill_dptr flags,
                              uint32_t epoch, int64_t wait_ns, ill_stream stream);

extern "C" int ill_ep_plan_dev(int world, int per, int cap, int rank, ill_dptr rc, ill_dptr counts, ill_dptr bases, ill_dptr p2r,
                               ill_dptr r2p, ill_dptr pdst, ill_dptr total, ill_dptr overflow, ill_stream stream) {
  return ep_plan_dev_launch(world, per, cap, rank, rc, counts, bases, p2r, r2p, pdst, total, overflow, 0, 0, 0, 0, stream);
}

extern "C" int ill_ep_plan_dev_sync(int world, int per, int cap, int rank, ill_dptr rc, ill_dptr counts, ill_dptr bases, ill_dptr p2r,
                                    ill_dptr r2p, ill_dptr pdst, ill_dptr total, ill_dptr overflow, ill_dptr flag_peers,
                                    ill_dptr flags, uint32_t epoch, int64_t wait_ns, ill_stream stream) {
  if (!flag_peers || !flags || (flag_peers & 7) || (flags & 3) || world > EP_MAX_RANKS || wait_ns < 0) return ILL_ERR_ARG;
  return ep_plan_dev_launch(world, per, cap, rank, rc, counts, bases, p2r, r2p, pdst, total, overflow, flag_peers, flags, epoch,
                            wait_ns, stream);
}

static int ep_plan_dev_launch(int world, int per, int cap, int rank, ill_dptr rc, ill_dptr counts, ill_dptr bases, ill_dptr p2r,
                              ill_dptr r2p, ill_dptr pdst, ill_dptr total, ill_dptr overflow, ill_dptr flag_peers, ill_dptr flags,
                              uint32_t epoch, int64_t wait_ns, ill_stream stream) {
  if (world < 1 || world > 255 || per < 1 || cap < 1 || (long long)world * cap > 0xffffff || rank < 0 || rank >= world ||
      (long long)world * per > 8192 || !rc || !counts || !bases || !p2r || !r2p || !total)
    return ILL_ERR_ARG;
  if ((rc & 3) || (counts & 3) || (bases & 3) || (p2r & 3) || (r2p & 3) || (pdst & 3) || (total & 3) || (overflow & 3)) return ILL_ERR_ALIGN;
  const unsigned* rp = (const unsigned*)(uintptr_t)rc;
  unsigned* cp = (unsigned*)(uintptr_t)counts;
  unsigned* bp = (unsigned*)(uintptr_t)bases;
  unsigned* pp = (unsigned*)(uintptr_t)p2r;
  unsigned* ip = (unsigned*)(uintptr_t)r2p;
  unsigned* tp = (unsigned*)(uintptr_t)total;
  unsigned* dp = (unsigned*)(uintptr_t)pdst;
  unsigned* ov = (unsigned*)(uintptr_t)overflow;
  const unsigned long long* fp = (const unsigned long long*)(uintptr_t)flag_peers;
  unsigned* fl = (unsigned*)(uintptr_t)flags;
  unsigned long long wn = (unsigned long long)wait_ns;
  unsigned* stw = device_status_word();
  void* args[] = {&world, &per, &cap, &rank, &rp, &cp, &bp, &pp, &ip, &dp, &tp, &ov, &fp, &fl, &epoch, &wn, &stw};
  const size_t smem = ((size_t)3 * world * per + per + 1) * 4;
  const void* k = (const void*)ep_plan_dev_kernel;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e);
  }
  return launch_kernel(k, dim3(1), dim3(256), smem, args, (cudaStream_t)stream);
}

extern "C" int ill_ep_unpack(int64_t rows, int cols, ill_dptr packed, ill_dptr map, ill_dptr xh, ill_dptr xe, ill_dptr xd,
                             ill_dptr w, ill_dptr rows_dev, ill_stream stream) {
  if (rows < 0 || cols <= 0 || cols % 256 || !packed || !xh || !xd || !w) return ILL_ERR_ARG;
  if ((packed & 15) || (map & 3) || (xh & 15) || (xe & 15) || (xd & 3) || (w & 3) || (rows_dev & 3)) return ILL_ERR_ALIGN;
  if (rows == 0) return ILL_OK;
  const long long rb = ill_ep_row_bytes(cols);
  const u8* base = (const u8*)(uintptr_t)packed;
  return act_f16_launch(rows, cols, base, rb, base + cols + cols / 256 * 4, rb, map, xh, xe, base + cols,
                        base + cols + cols / 256 * 4 + cols / 16 * 2, xd, w, stream, rows_dev);
}

// Rows of 64 K halves (X: a load brings two K steps of BOX_ROWS rows) or, SUMS, the first 16 of each 64 (a block's sums of 16)
static int encode_map(CUtensorMap* map, ill_dptr base, int64_t cols, int64_t rows, bool sums, cuuint32_t box_rows) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return cuda_fail(cudaErrorNotSupported);
  const cuuint64_t dims[3] = {sums ? (cuuint64_t)cols : MM_BK, (cuuint64_t)rows, (cuuint64_t)cols / MM_BK};
  const cuuint64_t strides[2] = {(cuuint64_t)cols * 2, MM_BK * 2};
  const cuuint32_t box[3] = {sums ? 16u : MM_BK, box_rows, 2};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, sums ? 2 : 3, (void*)(uintptr_t)base, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, sums ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? ILL_OK : cuda_fail(cudaErrorInvalidValue);
}

// A matrix's bytes, 128 rows of a block a load, or (Q6_K) a window of 32 of every fourth row (rows past the last: zeros)
static int encode_raw_map(CUtensorMap* map, int fmt, ill_dptr base, int ncols, int rows) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return cuda_fail(cudaErrorNotSupported);
  const int each = fmt == ILL_Q4_K ? 1 : 4;
  const cuuint64_t bytes = (cuuint64_t)ncols / 256 * fmt_block_bytes(fmt) * each;
  const cuuint64_t dims[2] = {bytes, (cuuint64_t)(rows / each)}, strides[1] = {bytes};
  const cuuint32_t box[2] = {fmt == ILL_Q4_K ? 144u : 240u, (cuuint32_t)(MM_BN / each)}, estr[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)(uintptr_t)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? ILL_OK : cuda_fail(cudaErrorInvalidValue);
}
// Whether encode_raw_map takes a matrix: Q4_K's are 16-byte aligned by contract
static bool raw_map_takes(int fmt, ill_dptr base, int ncols, int rows) {
  return fmt == ILL_Q4_K || (fmt == ILL_Q6_K && !(base & 15) && rows % 4 == 0 && ncols % 512 == 0);
}

static int mm_id_launch(int fmt, int ncols, int nrows, int64_t add, ill_dptr ptrs, ill_dptr counts, ill_dptr bases, int ne,
                        int64_t total_rows, ill_dptr xh, ill_dptr xe, ill_dptr xd, ill_dptr map, ill_dptr ymap, ill_dptr ypeers,
                        ill_dptr y, int64_t y_stride, ill_stream stream, int64_t add2 = 0, ill_dptr y2 = 0, ill_dptr one_ptr = 0,
                        int acc = 0, int over = 0);

extern "C" int ill_moe_mm_id2(int fmt, int ncols, int nrows, int64_t add, int64_t add2, ill_dptr ptrs, ill_dptr counts,
                              ill_dptr bases, int ne, int64_t total_rows, ill_dptr xh, ill_dptr xe, ill_dptr xd, ill_dptr map,
                              ill_dptr y, ill_dptr y2, int64_t y_stride, ill_stream stream) {
  if (!y || !y2 || (y2 & 15) || (add2 & 3)) return ILL_ERR_ARG;
  return mm_id_launch(fmt, ncols, nrows, add, ptrs, counts, bases, ne, total_rows, xh, xe, xd, map, 0, 0, y, y_stride, stream, add2,
                      y2);
}

extern "C" int ill_moe_mm_id(int fmt, int ncols, int nrows, int64_t add, ill_dptr ptrs, ill_dptr counts, ill_dptr bases,
                             int ne, int64_t total_rows, ill_dptr xh, ill_dptr xe, ill_dptr xd, ill_dptr map, ill_dptr ymap,
                             ill_dptr y, int64_t y_stride, ill_stream stream) {
  if (!y) return ILL_ERR_ARG;
  return mm_id_launch(fmt, ncols, nrows, add, ptrs, counts, bases, ne, total_rows, xh, xe, xd, map, ymap, 0, y, y_stride, stream);
}

extern "C" int ill_moe_mm_id_over(int fmt, int ncols, int nrows, int64_t add, int64_t add2, ill_dptr ptrs, ill_dptr counts, ill_dptr bases,
                                  int ne, int64_t total_rows, ill_dptr xh, ill_dptr xe, ill_dptr xd, ill_dptr map, ill_dptr y, ill_dptr y2,
                                  int64_t y_stride, int over, ill_stream stream) {
  if (!y || (y2 & 15) || (add2 & 3) || over < 0) return ILL_ERR_ARG;
  return mm_id_launch(fmt, ncols, nrows, add, ptrs, counts, bases, ne, total_rows, xh, xe, xd, map, 0, 0, y, y_stride, stream, add2, y2, 0, 0,
                      over);
}

extern "C" int ill_moe_mm_id_peers(int fmt, int ncols, int nrows, int64_t add, ill_dptr ptrs, ill_dptr counts, ill_dptr bases,
                                   int ne, int64_t total_rows, ill_dptr xh, ill_dptr xe, ill_dptr xd, ill_dptr map, ill_dptr ydst,
                                   ill_dptr ypeers, int64_t y_stride, ill_stream stream) {
  if (!ydst || !ypeers || (ypeers & 7)) return ILL_ERR_ARG;
  // Y is only named through YPEERS; any aligned non-null value keeps the common checks happy
  return mm_id_launch(fmt, ncols, nrows, add, ptrs, counts, bases, ne, total_rows, xh, xe, xd, map, ydst, ypeers, 16, y_stride,
                      stream);
}

extern "C" int ill_mm_chunk(int fmt, ill_dptr w, int rows, int cols, ill_dptr xh, ill_dptr xe, ill_dptr xd, int64_t n, ill_dptr y,
                            int acc, ill_stream stream) {
  if (!w || !y || n < 0 || n > 0x7fffffffll) return ILL_ERR_ARG;
  if (fmt != ILL_Q4_K && fmt != ILL_Q6_K) return ILL_ERR_UNSUPPORTED;
  return mm_id_launch(fmt, cols, rows, 0, 0, 0, 0, 1, n, xh, xe, xd, 0, 0, 0, y, rows, stream, 0, 0, w, acc ? 1 : 0);
}

// two matrices of one shape against the same chunk in one launch (a gated FFN's gate and up): twice the tiles for
// the persistent CTAs to share, so the last round of tiles is fuller than in two launches
extern "C" int ill_mm_chunk2(int fmt, ill_dptr w, ill_dptr w2, int rows, int cols, ill_dptr xh, ill_dptr xe, ill_dptr xd, int64_t n,
                             ill_dptr y, ill_dptr y2, ill_stream stream) {
  if (!w || !w2 || !y || !y2 || (y2 & 15) || n < 0 || n > 0x7fffffffll) return ILL_ERR_ARG;
  if (fmt != ILL_Q4_K && fmt != ILL_Q6_K) return ILL_ERR_UNSUPPORTED;
  const int64_t add2 = (int64_t)(w2 - w);  // the second matrix, relative to the first (unsigned wrap-around is intended)
  if (add2 & (fmt == ILL_Q4_K ? 15 : 3)) return ILL_ERR_ALIGN;
  return mm_id_launch(fmt, cols, rows, 0, 0, 0, 0, 1, n, xh, xe, xd, 0, 0, 0, y, rows, stream, add2, y2, w, 0);
}

struct MmVariant {
  const void* k;
  size_t smem;
  int threads, regs_sum;
};
template <int FMT, bool DENSE, int NT, int NT2 = 0>
static MmVariant mm_one() {
  typedef MmGeom<FMT, NT> G;
  constexpr int sum2 = MmGeom<FMT, NT2 ? NT2 : NT>::REGS_SUM;
  return MmVariant{(const void*)mm_id_kernel<FMT, DENSE, NT, NT2>, MmSmem<FMT, NT, NT2>::SMEM, G::THREADS, G::REGS_SUM > sum2 ? G::REGS_SUM : sum2};
}
// The kernel for tiles of up to NT rows of X of a dense matrix; for experts (NT 0) the formats with mins pick on the device between
// tiles of 64, whose A ring holds two blocks, and of 128.  IQ2_XXS and Q6_K, bound by their unpacking, gain 0 to 2 % from tiles of
// 64 where no expert has more rows and lose up to 90 % elsewhere: always 128.  (A kernel of both made IQ2_XXS's tiles of 128 10 % slower.)
template <int FMT>
static MmVariant mm_variant(int nt) {
  if constexpr (FMT == ILL_Q6_K)
    if (nt == 256) return mm_one<FMT, true, 256>();
  if constexpr (FMT == ILL_Q4_K || FMT == ILL_Q6_K)
    if (nt) return nt == 64 ? mm_one<FMT, true, 64>() : mm_one<FMT, true, 128>();
  if constexpr (FMT == ILL_Q2_K || FMT == ILL_Q4_K) return mm_one<FMT, false, 128, 64>();
  else return mm_one<FMT, false, 128>();
}

static int mm_ready(const MmVariant& v) {
  cudaError_t e = cudaFuncSetAttribute(v.k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem);
  if (e != cudaSuccess) return cuda_fail(e);
  // The warp groups trade registers after launch; what they ask for together must fit in what the
  // CTA was given, or the drain warps would wait for registers for ever.
  cudaFuncAttributes fa;
  e = cudaFuncGetAttributes(&fa, v.k);
  if (e != cudaSuccess) return cuda_fail(e);
  if (fa.numRegs / 8 * 8 * v.threads < v.regs_sum) return ILL_ERR_UNSUPPORTED;
  return ILL_OK;
}

// Rows of X a tile of a dense matrix: the rounds of tiles on the SMs times a tile's measured time a block of 256 columns, us; tiles
// of up to 64, of up to 128, and (Q6_K, which has one accumulator a block: with two, draining 256 columns takes longer than it
// saves) 256 rows.
static int mm_pick_tile(int fmt, long long rows, long long ntn, int sms) {
  const bool q6 = fmt == ILL_Q6_K;
  double best = 1e30;
  int bm = 16;
  for (int b = 16; b <= (q6 ? 256 : 128); b += 16) {
    const long long tiles = (rows + b - 1) / b * ntn, rounds = (tiles + sms - 1) / sms;
    const double us = b <= 64 ? (q6 ? 1.27 + 0.001 * b : 0.82 + 0.0045 * b) : b <= 128 ? (q6 ? 1.13 + 0.0032 * b : 1.05 + 0.0043 * b) : 1.75 + 0.0043 * b;
    if (rounds * us < best) { best = rounds * us; bm = b; }
  }
  return bm;
}

static int mm_id_launch(int fmt, int ncols, int nrows, int64_t add, ill_dptr ptrs, ill_dptr counts, ill_dptr bases, int ne,
                        int64_t total_rows, ill_dptr xh, ill_dptr xe, ill_dptr xd, ill_dptr map, ill_dptr ymap, ill_dptr ypeers,
                        ill_dptr y, int64_t y_stride, ill_stream stream, int64_t add2, ill_dptr y2, ill_dptr one_ptr, int acc,
                        int over) {
  if (fmt != ILL_IQ2_XXS && fmt != ILL_Q2_K && fmt != ILL_Q4_K && fmt != ILL_Q6_K) return ILL_ERR_UNSUPPORTED;
  const bool km = fmt == ILL_Q2_K || fmt == ILL_Q4_K;  // formats with mins: the sums of 16 of X come along
  if (ncols <= 0 || ncols % 256 || nrows <= 0 || ne <= 0 || ne > 65535 || total_rows < 0 || y_stride < nrows ||
      y_stride > 0xffffffffll)
    return ILL_ERR_ARG;
  if (!one_ptr && (!ptrs || !counts || !bases)) return ILL_ERR_ARG;
  if (!xh || !xd || !y || (km && !xe)) return ILL_ERR_ARG;
  if (fmt == ILL_Q4_K && (one_ptr & 15)) return ILL_ERR_ALIGN;
  if ((ptrs & 7) || (counts & 3) || (bases & 3) || (xh & 15) || (xe & 15) || (xd & 3) || (map & 3) || (ymap & 3) || (y & 15) ||
      (y_stride & 3) || (add & 3))
    return ILL_ERR_ALIGN;
  if (fmt == ILL_Q4_K && ((add | add2) & 15)) return ILL_ERR_ALIGN;  // (and every PTRS[e]: the kernel copies 16-byte pieces of the rows as they lie)
  if (total_rows == 0) return ILL_OK;
  MmMaps maps;
  for (int i = 0; i < 4; ++i) {
    int rc = encode_map(&maps.x[i], xh, ncols, total_rows, false, MM_XBOX * (i + 1));
    if (rc == ILL_OK && km) rc = encode_map(&maps.e[i], xe, (int64_t)(ncols / 256) * 64, total_rows, true, MM_XBOX * (i + 1));
    if (rc) return rc;
  }
  if (!km) memcpy(maps.e, maps.x, sizeof maps.e);
  const ill_dptr other = one_ptr + (y2 ? add2 : 0);
  const bool tma = one_ptr && raw_map_takes(fmt, one_ptr, ncols, nrows) && raw_map_takes(fmt, other, ncols, nrows);
  for (int i = 0; i < 2; ++i) {
    maps.w[i] = maps.x[0];  // (not read)
    const int rc = tma ? encode_raw_map(&maps.w[i], fmt, i ? other : one_ptr, ncols, nrows) : ILL_OK;
    if (rc) return rc;
  }
  MmParams p;
  p.neg_zero = -0.0f;
  p.tma = tma;
  p.wmap = 0;
  p.ncols = ncols;
  p.nrows = nrows;
  p.row_bytes = ncols / 256 * fmt_block_bytes(fmt);
  p.add = add;
  p.add2 = add2;
  p.ptrs = (const unsigned long long*)(uintptr_t)ptrs;
  p.counts = (const unsigned*)(uintptr_t)counts;
  p.bases = (const unsigned*)(uintptr_t)bases;
  p.xd = (const float*)(uintptr_t)xd;
  p.map = (const unsigned*)(uintptr_t)map;
  p.ymap = (const unsigned*)(uintptr_t)ymap;
  p.ypeers = (const unsigned long long*)(uintptr_t)ypeers;
  p.total_rows = total_rows;
  p.y = (float*)(uintptr_t)y;
  p.y2 = (float*)(uintptr_t)y2;
  p.y_stride = y_stride;
  p.ne = ne;
  p.one_ptr = one_ptr;
  p.one_count = (unsigned)total_rows;
  p.acc = acc;
  p.over = over;
  p.status = device_status_word();
  if (ne > MM_MAX_NE) return ILL_ERR_TOO_LARGE;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  const long long ntn = (nrows + MM_BN - 1) / MM_BN * (y2 ? 2 : 1);
  int nt = 0;
  p.bm = MM_BN;
  if (one_ptr) {
    p.bm = mm_pick_tile(fmt, total_rows, ntn, sms);
    nt = p.bm <= 64 ? 64 : p.bm <= 128 ? 128 : 256;
  }
  const int least = one_ptr ? p.bm : 64;         // rows of X a tile
  const long long max_tiles = ((total_rows + least - 1) / least + ne) * ntn;  // an upper bound
  const MmVariant v = fmt == ILL_IQ2_XXS ? mm_variant<ILL_IQ2_XXS>(nt) : fmt == ILL_Q2_K ? mm_variant<ILL_Q2_K>(nt)
                      : fmt == ILL_Q4_K ? mm_variant<ILL_Q4_K>(nt) : mm_variant<ILL_Q6_K>(nt);
  const int ready = mm_ready(v);
  if (ready) return ready;
  void* args[] = {&maps, &p};
  // persistent: a CTA an SM, each walks tiles
  return launch_kernel(v.k, dim3((unsigned)(max_tiles < sms ? max_tiles : sms)), dim3((unsigned)v.threads), v.smem, args, (cudaStream_t)stream);
}

extern "C" int ill_mm_chunk_exact(int fmt, ill_dptr w, int fmt2, ill_dptr w2, int rows, int cols, ill_dptr xh, ill_dptr xe, ill_dptr xd, int64_t n,
                                  ill_dptr y, ill_dptr y2, ill_stream stream) {
  if (fmt == ILL_Q6_K && fmt2 == ILL_Q4_K) {  // the other way round
    const int f = fmt; fmt = fmt2; fmt2 = f;
    ill_dptr t = w; w = w2; w2 = t;
    t = y; y = y2; y2 = t;
  }
  if ((fmt != ILL_Q4_K && fmt != ILL_Q6_K) || (fmt2 != ILL_Q4_K && fmt2 != ILL_Q6_K)) return ILL_ERR_UNSUPPORTED;
  if (!w || !w2 || !y || !y2 || !xh || !xd || (fmt == ILL_Q4_K && !xe) || rows <= 0 || rows % 4 || cols <= 0 || cols % 256 || n < 0 || n > 0x7fffffffll)
    return ILL_ERR_ARG;
  if ((xh & 15) || (xe & 15) || (xd & 3) || (y & 15) || (y2 & 15) || (w & (fmt == ILL_Q4_K ? 15 : 3)) || (w2 & (fmt2 == ILL_Q4_K ? 15 : 3)))
    return ILL_ERR_ALIGN;
  if (n == 0) return ILL_OK;
  const bool mixed = fmt != fmt2;
  MmMaps maps;
  for (int i = 0; i < 4; ++i) {
    int rc = encode_map(&maps.x[i], xh, cols, n, false, MM_XBOX * (i + 1));
    if (rc == ILL_OK && fmt == ILL_Q4_K) rc = encode_map(&maps.e[i], xe, (int64_t)(cols / 256) * 64, n, true, MM_XBOX * (i + 1));
    if (rc) return rc;
  }
  if (fmt != ILL_Q4_K) memcpy(maps.e, maps.x, sizeof maps.e);
  const bool tma = raw_map_takes(fmt, w, cols, rows) && (mixed || raw_map_takes(fmt2, w2, cols, rows)), tma2 = mixed && raw_map_takes(fmt2, w2, cols, rows);
  for (int i = 0; i < 2; ++i) {
    maps.w[i] = maps.x[0];  // (not read)
    const int rc = (i && mixed ? tma2 : tma) ? encode_raw_map(&maps.w[i], i ? fmt2 : fmt, i ? w2 : w, cols, rows) : ILL_OK;
    if (rc) return rc;
  }
  MmParams p = {}, p2;
  p.ncols = cols;
  p.nrows = rows;
  p.row_bytes = cols / 256 * fmt_block_bytes(fmt);
  p.xd = (const float*)(uintptr_t)xd;
  p.total_rows = n;
  p.y = (float*)(uintptr_t)y;
  p.y_stride = rows;
  p.ne = 1;
  p.one_ptr = w;
  p.one_count = (unsigned)n;
  p.neg_zero = -0.0f;
  p.tma = tma;
  p.status = device_status_word();
  p2 = p;
  if (mixed) {
    p2.tma = tma2;
    p2.wmap = 1;
    p2.row_bytes = cols / 256 * fmt_block_bytes(fmt2);
    p2.y = (float*)(uintptr_t)y2;
    p2.one_ptr = w2;
  } else {
    p.y2 = (float*)(uintptr_t)y2;
    p.add2 = (long long)(w2 - w);
  }
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 1) sms = 148;
  const long long ntn = (rows + MM_BN - 1) / MM_BN;
  // Rows of X a tile, and the SMs that Q4_K's tiles get beside Q6_K's: the rounds of tiles times a tile's measured time a block, us
  double best = 1e30;
  long long grid = 1;
  int split = 0;
  for (int b = 16; b <= 64; b += 16) {
    const long long tiles = (n + b - 1) / b * ntn, all = 2 * tiles, g = all < sms ? all : sms, rounds = (all + g - 1) / g;
    const double t4 = 0.75 + 0.0044 * b, t6 = 1.13 + 0.0035 * b;
    // (mixed: Q6_K, the slower, in at least its share of the rounds; a round more of its own leaves Q4_K more SMs)
    for (long long r = mixed ? 1 : rounds; r <= rounds; ++r) {
      const long long sp = mixed ? g - (tiles + r - 1) / r : 0;
      if (mixed && sp < 1) continue;
      const double a = mixed ? (double)((tiles + sp - 1) / sp) * t4 : 0.0, c = (double)r * (mixed || fmt == ILL_Q6_K ? t6 : t4), us = a > c ? a : c;
      if (us < best) { best = us; p.bm = p2.bm = b; grid = g; split = (int)sp; }
    }
  }
  typedef MmGeom<ILL_Q4_K, 64, true> G4;
  typedef MmGeom<ILL_Q6_K, 64, true> G6;
  const MmVariant v = mixed ? MmVariant{(const void*)mm_exact_kernel<ILL_Q4_K, ILL_Q6_K>, MmExactSmem<ILL_Q4_K, ILL_Q6_K>::SMEM, G4::THREADS,
                                        G4::REGS_SUM > G6::REGS_SUM ? G4::REGS_SUM : G6::REGS_SUM}
                      : fmt == ILL_Q4_K ? MmVariant{(const void*)mm_exact_kernel<ILL_Q4_K, ILL_Q4_K>, MmExactSmem<ILL_Q4_K, ILL_Q4_K>::SMEM, G4::THREADS, G4::REGS_SUM}
                                        : MmVariant{(const void*)mm_exact_kernel<ILL_Q6_K, ILL_Q6_K>, MmExactSmem<ILL_Q6_K, ILL_Q6_K>::SMEM, G6::THREADS, G6::REGS_SUM};
  const int ready = mm_ready(v);
  if (ready) return ready;
  void* args[] = {&maps, &p, &p2, &split};
  return launch_kernel(v.k, dim3((unsigned)grid), dim3((unsigned)v.threads), v.smem, args, (cudaStream_t)stream);
}
