// mvt.cu -- a quantized matrix times a few tokens (2 .. 16) with the weights read once: the integer
// block dots on the tensor cores' int8 path instead of one dp4a pass per token.
//
// At 2-16 tokens the product is still bound by the weights' bytes, but on CUDA cores every token costs a full
// pass of dp4a over the unpacked weights (mvn_kernel: batch 16 took 22-30 times the time of batch 1).  Here a warp
// holds 16 weight rows x one block of columns as the A operand of mma.sync (m16n8k32 / m16n8k16, u8 or s8
// weights, s8 activations, s32 accumulate) and the tokens as B, eight a tile: the weights are unpacked once
// whatever the number of tokens.  The integers are the CPU kernels' (exact); each block's sum meets its float
// scales as in the reference's portable loops (src/tensor.lisp:321-336, src/kquant.lisp:171-236).
//
//   * A persistent CTA stages the tokens' quantized activations in shared memory once (token stride padded by 16 bytes, so that the
//     eight tokens of a B fragment sit on different banks), then walks tiles of 16 rows, of one matrix or of up to three that share
//     the activations (Q, K and V; gate and up).  A tile's pieces -- 16 row segments of one or more blocks -- make up to eight partial
//     sums (piece I goes to sum I % 8), dealt to the warps of a group so that they have as many pieces each: five warps for rows
//     of ten Q4_K blocks, four for twenty of Q6_K; a CTA holds as many groups as its warps and shared memory allow.  Each warp
//     streams its pieces by 16-byte cp.async, four lanes a segment, through its own ring of stages, across tile boundaries.
//   * The partial sums (a float per row and token) meet in shared memory and are added in order: the bits do not depend on the groups.
//
// Bound by the chain from one launch to the next where the matrix is small (activations, one or two pieces a warp, the meeting), by
// instruction issue where it is large: 48 % of cycles, then the shared-memory queue (Q6_K's blocks, every second of which starts in the
// middle of a word).  us, weights cold and launches one behind the other, eight warps a tile and a launch a matrix / now: Q, K (Q4_K)
// and V (Q6_K) of 4096 + 2 x 1024 x 2560, 16 tokens 20.6 / 7.3; gate and up of 2 x 9728 x 2560 (Q4_K), 16 tokens 25.4 / 14.0, 4 tokens - / 12.0;
// of 2 x 17408 x 5120 (Q6_K), 4 tokens 66 / 42; 5120 x 5120 (Q6_K), 16 tokens 28.7 / 22.5; a head of 151936 x 2560 (Q6_K), 16 tokens
// 142 / 117.  What gave it: one launch; activations that are all asked for before anything is waited for (4 us a launch); the deal;
// Q4_K's mins against the sums of 16 by two products, its scales four at a time (half the instructions); ldmatrix.
//
// The 2-bit formats' blocks are in mtblock.cuh.  us, the token loop of mv.cu (a pass of dp4a a token) / now: Q2_K 151936 x 2560, 4 tokens 236 / 57,
// 16 tokens 923 / 70; IQ2_XXS 232 / 80 and 768 / 93; 4096 x 4096, 4 tokens 29.5 / 4.5 and 27.2 / 6.1; 512 x 512, 2 tokens 2.9 / 2.1 and 3.1 / 3.1.
//
// mma.sync is the legacy tensor path: right here, where N is 8 or 16 and the bound is HBM; the chunk-sized
// products (hundreds of rows of X an expert) use tcgen05 (mm_id.cu).
//
// Replaces mv_q8_n / mm_q8_mma's small-batch use and mv_k's token loop behind CMAT-MUL-N
// (src/cuda-dense.lisp:220-255; src/cuda/dense.cu:643-885, src/cuda/kquant.cu:169-466).
#include "host.h"
#include "iq2xxs_tables.cuh"
#include "mtblock.cuh"

namespace ill {

// A tile's pieces are dealt to eight partial sums (piece I to sum I % 8), and the sums to a group's warps; a CTA holds as many groups (a
// tile each at a time) as make up to sixteen warps, which share the staged activations, and each warp a ring of two to four stages.
constexpr int MT_SUMS = 8, MT_MAX_WARPS = 16, MT_ROWS = 16, MT_MAX_STAGES = 4, MT_MATS = 3;

// The named barrier at which the warps of group GRP meet.  A CTA has barriers 0 (that of __syncthreads) to 15, so fifteen groups at most.
// (Sixteen, those of one warp with __syncwarp instead: the branch cost every launch 1 %.)
__host__ __device__ constexpr int mt_barrier(int grp) { return 1 + grp; }
constexpr int MT_MAX_GROUPS = 15;
static_assert(mt_barrier(MT_MAX_GROUPS - 1) <= 15, "a CTA has no more barriers");

struct MtMat {
  const u8* w;
  float* y;
  const float* bias;
  int rows, tile_end;   // tiles of 16 rows of this matrix and those before it
  int alt;              // in the kernel's second format
};
// a format's pieces
struct MtFmt {
  int row_bytes;
  int cb, npieces;      // blocks a staged piece (a warp's unit of copying); pieces a row
  uint32_t piece_bytes; // of a row
  int pitch;            // bytes between the rows of a staged piece
  u8 sums[MT_SUMS];     // the partial sums of a group's warp (bits)
};
struct MtParams {
  MtMat m[MT_MATS];     // matrices that share the activations; the last ones may be empty
  MtFmt f[2];           // the kernel's formats
  int cols, nblocks;    // blocks a row
  const i8* xq;
  const float* xs;
  const int16_t* xsum;
  int acc, n;
  int nsums;            // partial sums a row, at most
  uint32_t stage_bytes;
  int stages, groups;   // stages a warp's ring; groups of warps a CTA
  int gw;               // warps a group
  int x_stride;         // bytes between the tokens' quants in shared memory
  uint32_t xs_off, bs_off, ring_off, part_off;
};

// sums of 16 times sixteen bytes of the rows' (S0, S8: row g's and g + 8's bytes 4 t ..), each sum split in two int8 halves
__device__ __forceinline__ void mul_sums(int (&c)[4], uint32_t s0, uint32_t s8, const MtX& x, int nt, int blk, int lane) {
  const u8* b = x.bs + ((size_t)(8 * nt + (lane >> 2)) * x.nb + blk) * 32 + 4 * (lane & 3);
  int hi[4] = {0, 0, 0, 0}, lo[4] = {0, 0, 0, 0};
  mma_k16_s8(hi, s0, s8, *(const uint32_t*)b, false);
  mma_k16_s8(lo, s0, s8, *(const uint32_t*)(b + 16), true);
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] = 16 * hi[i] + lo[i];
}

template <int NT8, bool AL4> struct MtBlock<ILL_Q8_0, NT8, AL4> {
  __device__ static void run(const u8* row0, const u8* row8, int blk, const MtX& x, int lane, float (&acc)[NT8][4]) {
    const int g = lane >> 2, t4 = 4 * (lane & 3);
    uint32_t a[4];
    const LdsWords q0(row0 + 2 + t4), q8(row8 + 2 + t4);
    a[0] = q0(0); a[1] = q8(0); a[2] = q0(16); a[3] = q8(16);
    const float d0 = ldh(row0), d8 = ldh(row8);
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt) {
      const i8* xw = x.q + (size_t)(8 * nt + g) * x.stride + 32 * blk + t4;
      const uint32_t b[2] = {*(const uint32_t*)xw, *(const uint32_t*)(xw + 16)};
      int c[4] = {0, 0, 0, 0};
      mma_k32(c, a, b, false);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int tok = 8 * nt + 2 * (lane & 3) + (i & 1);
        const float xs = x.s[tok * x.nsc + blk];
        // Q8-ROW-DOT-AT: sum += float(isum) * (d_w * d_x)
        acc[nt][i] = __fadd_rn(acc[nt][i], __fmul_rn((float)c[i], __fmul_rn(i < 2 ? d0 : d8, xs)));
      }
    }
  }
};

template <int NT8, bool AL4> struct MtBlock<ILL_Q4_K, NT8, AL4> {
  __device__ static void run(const u8* row0, const u8* row8, int blk, const MtX& x, int lane, float (&acc)[NT8][4]) {
    const int t = lane & 3, t4 = 4 * t;
    const RowWords<AL4> h0(row0), h8(row8), q0(row0 + t4), q8(row8 + t4);
    // the 6-bit scales and mins of the eight groups, a byte each (get_scale_min_k4, src/kquant.lisp:64-72, four at a time)
    uint32_t sc[2][2], mn[2][2];  // [row g / g + 8][groups 0-3 / 4-7]
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint32_t a = (r ? h8 : h0)(4), b = (r ? h8 : h0)(8), c = (r ? h8 : h0)(12);
      sc[r][0] = a & 0x3f3f3f3fu;
      sc[r][1] = (c & 0x0f0f0f0fu) | ((a >> 2) & 0x30303030u);
      mn[r][0] = b & 0x3f3f3f3fu;
      mn[r][1] = ((c >> 4) & 0x0f0f0f0fu) | ((b >> 2) & 0x30303030u);
    }
    int isum[NT8][4];
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) isum[nt][i] = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // 64 weights: groups 2k (low nibbles) and 2k + 1 (high)
      const uint32_t w[4] = {q0(16 + 32 * k), q8(16 + 32 * k), q0(32 + 32 * k), q8(32 + 32 * k)};
      uint32_t lo[4], hi[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { lo[i] = w[i] & 0x0F0F0F0Fu; hi[i] = (w[i] >> 4) & 0x0F0F0F0Fu; }
      int s[2][2];  // [row][group]
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int j = 0; j < 2; ++j) s[r][j] = (int)(sc[r][k >> 1] >> (16 * (k & 1) + 8 * j) & 0xffu);
#pragma unroll
      for (int nt = 0; nt < NT8; ++nt) {
        uint32_t b[4];
        xfrag(b, x, nt, 256 * blk + 64 * k, lane);
        const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
        int c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
        mma_k32(c0, lo, b0, true);
        mma_k32(c1, hi, b1, true);
#pragma unroll
        for (int i = 0; i < 4; ++i) isum[nt][i] += c0[i] * s[i >> 1][0] + c1[i] * s[i >> 1][1];
      }
    }
    const uint32_t e0 = h0(0), e8 = h8(0);
    const float d0 = h2f(e0 & 0xffffu), m0 = h2f(e0 >> 16), d8 = h2f(e8 & 0xffffu), m8 = h2f(e8 >> 16);
    // the mins against the sums of 16: a group of 32 faces two of them, so bytes 4 t .. are mins 2 t, 2 t, 2 t + 1, 2 t + 1
    const uint32_t sel = t & 1 ? 0x3322u : 0x1100u;
    const uint32_t a0 = __byte_perm(t >> 1 ? mn[0][1] : mn[0][0], 0, sel), a8 = __byte_perm(t >> 1 ? mn[1][1] : mn[1][0], 0, sel);
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt) {
      int imin[4];
      mul_sums(imin, a0, a8, x, nt, blk, lane);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int tok = 8 * nt + 2 * t + (i & 1);
        const float yd = x.s[tok * x.nsc + blk];
        // Q4K-ROW-DOT: sum -= (yd * dmin) * imin; sum += (yd * d) * isum
        const float v = __fsub_rn(acc[nt][i], __fmul_rn(__fmul_rn(yd, i < 2 ? m0 : m8), (float)imin[i]));
        acc[nt][i] = __fadd_rn(v, __fmul_rn(__fmul_rn(yd, i < 2 ? d0 : d8), (float)isum[nt][i]));
      }
    }
  }
};

template <int NT8, bool AL4> struct MtBlock<ILL_Q6_K, NT8, AL4> {
  // every second block starts on a word, in all rows alike where they lie a multiple of four bytes apart
  __device__ static void run(const u8* row0, const u8* row8, int blk, const MtX& x, int lane, float (&acc)[NT8][4]) {
    if (__all_sync(0xffffffffu, (((uintptr_t)row0 | (uintptr_t)row8) & 3) == 0)) run_al<true>(row0, row8, blk, x, lane, acc);
    else run_al<false>(row0, row8, blk, x, lane, acc);
  }
  template <bool W>
  __device__ __forceinline__ static void run_al(const u8* row0, const u8* row8, int blk, const MtX& x, int lane, float (&acc)[NT8][4]) {
    const int t4 = 4 * (lane & 3);
    int isum[NT8][4];
    const RowWords<W> q0(row0 + t4), q8(row8 + t4), h0(row0), h8(row8);
    uint32_t sc[2][4];  // [row g / g + 8]: the sixteen scales
#pragma unroll
    for (int j = 0; j < 4; ++j) { sc[0][j] = h0(192 + 4 * j); sc[1][j] = h8(192 + 4 * j); }
    {
      // The quants are 0..63: their -32 comes off as 32 * sum over the groups of scale * (the activations' sum of
      // the group) -- itself a product of the block's 16 x 16 scales with the tokens' sums
      const uint32_t s0 = q0(192), s8 = q8(192);
#pragma unroll
      for (int nt = 0; nt < NT8; ++nt) {
        mul_sums(isum[nt], s0, s8, x, nt, blk, lane);
#pragma unroll
        for (int i = 0; i < 4; ++i) isum[nt][i] *= -32;
      }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {    // half of the block: 128 weights, two groups of 16 of each of the half's four runs of 32
      uint32_t b[NT8][2][4];         // the tokens' quants of runs 0 and 1, 2 and 3: [run & 1][group]
#pragma unroll
      for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
        for (int r2 = 0; r2 < 2; ++r2) xfrag(b[nt][r2], x, nt, 256 * blk + 128 * c + 64 * r2, lane);
#pragma unroll
      for (int is = 0; is < 2; ++is) {
        uint32_t q[2][4];  // [row g / g + 8][run]: the lane's four 6-bit quants of each run
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const RowWords<W>& row = r ? q8 : q0;
          const uint32_t A = row(64 * c + 16 * is), B = row(64 * c + 32 + 16 * is), H = row(128 + 32 * c + 16 * is);
          q[r][0] = (A & 0x0F0F0F0Fu) | ((H << 4) & 0x30303030u);
          q[r][1] = (B & 0x0F0F0F0Fu) | ((H << 2) & 0x30303030u);
          q[r][2] = ((A >> 4) & 0x0F0F0F0Fu) | (H & 0x30303030u);
          q[r][3] = ((B >> 4) & 0x0F0F0F0Fu) | ((H >> 2) & 0x30303030u);
        }
#pragma unroll
        for (int run = 0; run < 4; ++run) {
          const int grp = 8 * c + 2 * run + is;  // the group of 16 and its scale
          const int s0 = (int)(signed char)(sc[0][grp >> 2] >> (8 * (grp & 3))), s8 = (int)(signed char)(sc[1][grp >> 2] >> (8 * (grp & 3)));
#pragma unroll
          for (int nt = 0; nt < NT8; ++nt) {
            int cc[4] = {0, 0, 0, 0};
            mma_k16_u8(cc, q[0][run], q[1][run], b[nt][run >> 1][2 * (run & 1) + is]);
#pragma unroll
            for (int i = 0; i < 4; ++i) isum[nt][i] += cc[i] * (i < 2 ? s0 : s8);
          }
        }
      }
    }
    const float d0 = ldh(row0 + 208), d8 = ldh(row8 + 208);
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int tok = 8 * nt + 2 * (lane & 3) + (i & 1);
        const float yd = x.s[tok * x.nsc + blk];
        // Q6K-ROW-DOT: sum += (d * yd) * float(isum - 32 imins)
        acc[nt][i] = __fadd_rn(acc[nt][i], __fmul_rn(__fmul_rn(i < 2 ? d0 : d8, yd), (float)isum[nt][i]));
      }
  }
};

// the meeting of one group's warps
__device__ __forceinline__ void group_sync(int grp, int gw) {
  asm volatile("barrier.cta.sync %0, %1;" ::"r"(mt_barrier(grp)), "r"(32 * gw) : "memory");
}

template <int N> struct IntC { static constexpr int value = N; };

// FMT2: the format of the matrices marked ALT (a file's V in Q6_K beside Q and K in Q4_K), or FMT
template <int FMT, int FMT2, int NT8, bool AL4>
__global__ void __launch_bounds__(32 * MT_MAX_WARPS, 1) mvt_kernel(const __grid_constant__ MtParams p) {
  extern __shared__ __align__(128) u8 smem[];
  constexpr int BW = Fmt<FMT>::BW, NTOK = 8 * NT8, PP = 20 /* floats a token's 16 rows of a partial sum are apart */;
  constexpr bool TWO = FMT != FMT2;
  const int tid = threadIdx.x, lane = tid & 31, cwarp = tid >> 5;  // the warp's number in the CTA
  const int gw = p.gw, grp = cwarp / gw, wg = cwarp - gw * grp, gtid = tid - 32 * gw * grp;
  const int nthreads = blockDim.x, stages = p.stages;
  const int tile0 = grp * gridDim.x + blockIdx.x, tile_step = gridDim.x * p.groups;
  i8* xq_s = (i8*)smem;
  float* xs_s = (float*)(smem + p.xs_off);
  const uint32_t ring = smem_u32(smem) + p.ring_off + cwarp * stages * p.stage_bytes;
  const int nb = p.nblocks;
  float* part = (float*)(smem + p.part_off) + (size_t)grp * 2 * p.nsums * NTOK * PP;  // [group][2][sums][tokens][PP]
  const int ntiles = p.m[MT_MATS - 1].tile_end;

  auto matrix = [&](int tile) { return (tile >= p.m[0].tile_end) + (tile >= p.m[1].tile_end); };
  auto format = [&](int mi) { return TWO ? p.m[mi].alt : 0; };
  // this warp's pieces in order: its group's tiles tile0, + tile_step, ...; of each, sum after sum, the pieces of its sums.  What a
  // tile's pieces share is worked out once a tile: 32-bit offsets from the lane's row are left for a piece.  (722 instructions a block of
  // Q6_K, 555 now, of which 355 take it apart and multiply it.  A head of 151936 x 2560, 16 tokens 121.8 / 117.4 us, of Q2_K, 4 tokens 60.5 /
  // 56.6; where latencies bound it nothing: gate and up of 2 x 17408 x 5120, 4 tokens 46.7 / 45.9.)
  const int g = lane >> 2, t = lane & 3;
  int n_tile = tile0, n_pc = 0;
  unsigned n_left = 0;
  const u8* n_src = nullptr;   // the lane's row g of the tile; row g + 8 is N_ROW8 bytes on
  uint32_t n_row8 = 0, n_dst = ring, n_end = 0;  // where the next stage starts; the end of the ring
  int n_rows = 0, n_alt = 0;   // rows of the matrix from row g on
  auto at_tile = [&]() {  // on to the first tile from n_tile on that this warp has a sum of
    while (n_tile < ntiles) {
      const int mi = matrix(n_tile);
      const MtFmt& f = p.f[format(mi)];
      n_left = f.sums[wg];
      if (n_left) {
        const int row = (n_tile - (mi ? p.m[mi - 1].tile_end : 0)) * MT_ROWS + g;
        n_pc = __ffs(n_left) - 1;
        n_src = p.m[mi].w + (long long)row * f.row_bytes;
        n_row8 = 8u * (uint32_t)f.row_bytes;
        n_rows = p.m[mi].rows - row;
        n_alt = format(mi);
        return;
      }
      n_tile += tile_step;
    }
  };
  at_tile();
  n_end = ring + stages * p.stage_bytes;
  auto issue_next = [&]() {  // all lanes: four a row segment, eight rows at a time; a group of cp.async, possibly empty
    if (n_tile < ntiles) {
      auto copy = [&](auto fmt_) {
        constexpr int F = decltype(fmt_)::value, BB = Fmt<F>::BB, MAXB = F == ILL_Q8_0 ? 8 : F == ILL_Q6_K ? 1 : 2;  // most blocks a piece
        const MtFmt& f = p.f[F != FMT];
        const uint32_t off = (uint32_t)n_pc * f.piece_bytes, len = min(f.piece_bytes, (uint32_t)f.row_bytes - off);
        const uint32_t dst = n_dst + g * f.pitch + 16 * t;
        const u8* src = n_src + off;
        if (n_rows > 0) copy_segment_at<(MAXB * BB + 30) / 16>(dst, src, len, t);
        if (n_rows > 8) copy_segment_at<(MAXB * BB + 30) / 16>(dst + 8 * f.pitch, src + n_row8, len, t);
        n_pc += MT_SUMS;
        if (n_pc >= f.npieces) {
          n_left &= n_left - 1;
          if (n_left) n_pc = __ffs(n_left) - 1;
          else { n_tile += tile_step; at_tile(); }
        }
      };
      if (TWO && n_alt) copy(IntC<FMT2>()); else copy(IntC<FMT>());
      n_dst += p.stage_bytes;
      if (n_dst == n_end) n_dst = ring;
    }
    cp_async_commit();
  };
  for (int s = 0; s < stages; ++s) issue_next();  // the weights do not depend on the previous kernel
  __shared__ uint2 iq_grid[FMT == ILL_IQ2_XXS ? IQ_TABLE_BYTES / 8 : 1];  // (static: the look-ups' addresses start at a constant)
  if constexpr (FMT == ILL_IQ2_XXS) iq_tables_fill(iq_grid, iq_grid + IQ_COPIES * 256, ill_iq2xxs_grid, ill_ksigns_iq2xs);
  pdl_launch_dependents();
  pdl_wait();

  // The tokens' activations -> shared memory, the tokens past the last (up to a whole tile of eight) as zeros: all asked for before
  // anything is waited for.  (A load, a store and the next load a thread took 12 latencies of L2 one after another: four of the 15 us
  // of gate and up, 2 x 9728 x 2560, of 16 tokens.)
  const int nsc = p.cols / BW, per_tok = p.cols / 16;
  uint4 sum8[2];            // K formats: eight sums of 16 a load; two loads a thread hold 16 tokens of 8192 columns
  constexpr bool SUMS = FMT != ILL_Q8_0 && FMT != ILL_IQ2_XXS;
  const int nsum8 = SUMS ? NTOK * per_tok / 8 : 0;
  auto load_sums = [&](int i) {
    if (i >= nsum8 || 8 * i >= p.n * per_tok) return make_uint4(0, 0, 0, 0);
    const uint2 a = ((const uint2*)p.xsum)[2 * i], b = ((const uint2*)p.xsum)[2 * i + 1];
    return make_uint4(a.x, a.y, b.x, b.y);  // (the sums lie on eight bytes, if not on sixteen)
  };
#pragma unroll
  for (int k = 0; k < 2; ++k) sum8[k] = load_sums(tid + k * nthreads);
  for (int tk = cwarp; tk < NTOK; tk += nthreads / 32)  // a warp a token
    for (int j = lane; j < per_tok; j += 32) {
      const bool in = tk < p.n;
      cp_async16_or_zero(xq_s + (size_t)tk * p.x_stride + 16 * j, in ? p.xq + (size_t)tk * p.cols + 16 * j : p.xq, in);
    }
  for (int i = tid; i < NTOK * nsc; i += nthreads) {
    const bool in = i < p.n * nsc;
    cp_async4_or_zero(xs_s + i, in ? p.xs + i : p.xs, in);
  }
  cp_async_commit();
  if constexpr (SUMS) {
    // per block 32 bytes: the sixteen sums' high parts (sum >> 4, signed), then their low parts (sum & 15)
    auto store_sums = [&](int i, const uint4& v) {
      u8* b = smem + p.bs_off + (i >> 1) * 32 + 8 * (i & 1);
      split_sums(v, *(uint2*)b, *(uint2*)(b + 16));
    };
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (tid + k * nthreads < nsum8) store_sums(tid + k * nthreads, sum8[k]);
    for (int i = tid + 2 * nthreads; i < nsum8; i += nthreads) store_sums(i, load_sums(i));
  }
  cp_async_wait_all();
  __syncthreads();
  MtX x;
  x.q = xq_s; x.stride = p.x_stride; x.s = xs_s; x.bs = smem + p.bs_off; x.nsc = nsc; x.nb = nb;
  MtLane xl;  // (the 2-bit formats')
  xl.set<FMT>(smem_u32(smem), p.x_stride, smem_u32(smem) + p.xs_off, smem_u32(smem) + p.bs_off, nb, FMT == ILL_IQ2_XXS ? smem_u32(iq_grid) : 0u, lane);

  uint32_t at = ring;          // the stage used next
  int it = 0;
  for (int tile = tile0; tile < ntiles; tile += tile_step, ++it) {
    const int mi = matrix(tile), row0 = (tile - (mi ? p.m[mi - 1].tile_end : 0)) * MT_ROWS;
    float* sums = part + (size_t)(it & 1) * p.nsums * NTOK * PP;
    const MtFmt& f = p.f[format(mi)];
    // where the lane's rows start, modulo 16
    const uint32_t o0 = (uint32_t)(uintptr_t)p.m[mi].w + (uint32_t)(row0 + g) * (uint32_t)f.row_bytes, o8 = o0 + 8u * (uint32_t)f.row_bytes;
    for (unsigned left = f.sums[wg]; left; left &= left - 1) {
      const int sum = __ffs(left) - 1;
      float acc[NT8][4];
#pragma unroll
      for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[nt][i] = 0.0f;
      for (int pc = sum; pc < f.npieces; pc += MT_SUMS) {
        // all but the newer stages' groups: this piece is in
        if (stages == 4) asm volatile("cp.async.wait_group 3;" ::: "memory");
        else if (stages == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        auto use = [&](auto fmt_) {
          constexpr int F = decltype(fmt_)::value, BB = Fmt<F>::BB;
          // a row's segment starts where its block starts inside the 16-byte aligned span that was copied
          const uint32_t off = (uint32_t)pc * f.piece_bytes;
          uint32_t s0 = at + g * f.pitch + ((o0 + off) & 15u), s8 = at + (g + 8) * f.pitch + ((o8 + off) & 15u);
          const int b0 = pc * f.cb, nhere = min(f.cb, nb - b0);
          for (int j = 0; j < nhere; ++j, s0 += BB, s8 += BB) {
            if constexpr (F == ILL_Q2_K || F == ILL_IQ2_XXS) MtBlock<F, NT8, AL4>::run(s0, s8, b0 + j, xl, lane, acc);
            else MtBlock<F, NT8, AL4>::run((const u8*)__cvta_shared_to_generic(s0), (const u8*)__cvta_shared_to_generic(s8), b0 + j, x, lane, acc);
          }
        };
        if (TWO && p.m[mi].alt) use(IntC<FMT2>()); else use(IntC<FMT>());
        at += p.stage_bytes;
        if (at == n_end) at = ring;
        __syncwarp();
        issue_next();
      }
#pragma unroll
      for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) sums[(sum * NTOK + 8 * nt + 2 * t + (i & 1)) * PP + g + 8 * (i >> 1)] = acc[nt][i];
    }
    // the partial sums meet: thread (token, row) adds them in order
    group_sync(grp, gw);
    const int nsums = min(MT_SUMS, f.npieces);
    for (int o = gtid; o < MT_ROWS * p.n; o += 32 * gw) {
      const int r = o & 15, tk = o >> 4, row = row0 + r;
      if (row < p.m[mi].rows) {
        float v = 0.0f;
#pragma unroll
        for (int k = 0; k < MT_SUMS; ++k)
          if (k < nsums) v = __fadd_rn(v, sums[(k * NTOK + tk) * PP + r]);
        if (FMT == ILL_IQ2_XXS) v *= 0.125f;
        if (p.m[mi].bias) v += p.m[mi].bias[row];
        float* yp = p.m[mi].y + (long long)tk * p.m[mi].rows + row;
        *yp = p.acc ? *yp + v : v;
      }
    }
  }
}

// Registers a thread of the kernel, at most: what decides whether an SM holds two CTAs
static int mt_regs(int fmt, int n) { return fmt == ILL_Q8_0 ? 96 : n <= 8 && fmt != ILL_IQ2_XXS ? 112 : 128; }

static const void* mt_kernel(int fmt, bool two, bool al4, int n) {
#define MT_PICK(F, F2, A) (n <= 8 ? (const void*)mvt_kernel<F, F2, 1, A> : (const void*)mvt_kernel<F, F2, 2, A>)
  if (fmt == ILL_Q8_0) return MT_PICK(ILL_Q8_0, ILL_Q8_0, false);
  if (fmt == ILL_Q6_K) return MT_PICK(ILL_Q6_K, ILL_Q6_K, false);
  if (fmt == ILL_IQ2_XXS) return MT_PICK(ILL_IQ2_XXS, ILL_IQ2_XXS, false);
  if (fmt == ILL_Q2_K) return al4 ? MT_PICK(ILL_Q2_K, ILL_Q2_K, true) : MT_PICK(ILL_Q2_K, ILL_Q2_K, false);
  if (two) return al4 ? MT_PICK(ILL_Q4_K, ILL_Q6_K, true) : MT_PICK(ILL_Q4_K, ILL_Q6_K, false);
  return al4 ? MT_PICK(ILL_Q4_K, ILL_Q4_K, true) : MT_PICK(ILL_Q4_K, ILL_Q4_K, false);
#undef MT_PICK
}

static int mvt_launch(const void* k, const MtParams& p, size_t smem, int grid, cudaStream_t st) {
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e);
  }
  MtParams pp = p;
  void* args[] = {&pp};
  return launch_kernel(k, dim3(grid), dim3(32 * p.gw * p.groups), smem, args, st);
}

// Deals the eight sums of NP pieces to GW warps, the longest first to the warp with the fewest pieces; returns the most a warp gets.
static int mt_deal(int np, int gw, u8* sums) {
  int load[MT_SUMS] = {}, most = 0;
  for (int i = 0; i < MT_SUMS; ++i) sums[i] = 0;
  for (int k = 0; k < MT_SUMS && k < np; ++k) {  // (earlier sums have as many pieces or one more)
    int w = 0;
    for (int i = 1; i < gw; ++i)
      if (load[i] < load[w]) w = i;
    load[w] += (np - k + MT_SUMS - 1) / MT_SUMS;
    sums[w] |= (u8)(1u << k);
    if (load[w] > most) most = load[w];
  }
  return most;
}

// A launch of mvt_kernel: everything but the pointers.
struct MtPlan {
  MtParams p;
  int fmt;              // the kernel's (first) format
  bool two;             // Q4_K and Q6_K
  int grid;
  size_t smem;
};

// The launch for NMAT matrices that share the activations -- of one format, or (FMTS) of Q4_K and Q6_K -- and N tokens on SMS SMs;
// ILL_ERR_UNSUPPORTED where the kernel is not written for them.
static int mvt_plan(int nmat, const int* fmts, const int* rows, int cols, int n, int sms, MtPlan* plan) {
  if (n < 2 || n > 16 || nmat < 1 || nmat > MT_MATS) return ILL_ERR_UNSUPPORTED;
  MtParams& p = plan->p;
  p = {};
  long long ntiles = 0, tiles[2] = {};
  bool two = false;
  for (int i = 0; i < nmat; ++i) two = two || fmts[i] != fmts[0];
  const int fmt = two ? ILL_Q4_K : fmts[0];
  for (int i = 0; i < MT_MATS; ++i) {
    if (i < nmat) {
      if (two && fmts[i] != ILL_Q4_K && fmts[i] != ILL_Q6_K) return ILL_ERR_UNSUPPORTED;
      p.m[i].rows = rows[i];
      p.m[i].alt = fmts[i] != fmt;
      const int t = (rows[i] + MT_ROWS - 1) / MT_ROWS;
      ntiles += t;
      tiles[p.m[i].alt] += t;
    }
    if (ntiles > 0x3fffffff) return ILL_ERR_TOO_LARGE;
    p.m[i].tile_end = (int)ntiles;
  }
  const int bw = fmt_block_weights(fmt), nsc = cols / bw;
  const uint32_t tables = fmt == ILL_IQ2_XXS ? IQ_TABLE_BYTES : 0u;  // static shared memory
  p.cols = cols;
  p.nblocks = nsc;
  p.n = n;
  p.x_stride = mt_x_stride(fmt, cols);
  const uint32_t ntok = n <= 8 ? 8 : 16;  // staged tokens: whole tiles of eight
  uint32_t off = ntok * (uint32_t)p.x_stride;
  off = (off + 15) / 16 * 16;
  p.xs_off = off;
  off += 4u * ntok * nsc;
  off = (off + 15) / 16 * 16;
  p.bs_off = off;
  for (int i = 0; i < (two ? 2 : 1); ++i) {
    const int ft = i ? ILL_Q6_K : fmt, bb = fmt_block_bytes(ft);
    MtFmt& f = p.f[i];
    f.row_bytes = p.nblocks * bb;
    // a row's segment: its block's 16-byte aligned span, rows a multiple of 16 bytes apart that is an odd multiple
    // of 16 mod 128 (eight rows x four words then sit on 32 different banks)
    // blocks a piece: about 200-300 bytes a row segment (four lanes' copies), but every sum should get a piece
    int cb = ft == ILL_Q8_0 ? 8 : ft == ILL_Q6_K ? 1 : 2;
    while (cb > 1 && (p.nblocks + cb - 1) / cb < MT_SUMS) cb >>= 1;
    // Too many tokens of too many columns (no room for eight warps with two stages each): mmd.cu's form, which brings the
    // activations step by step, is the faster one, and adds a row's blocks in another order.  The 2-bit formats, which have no such form, go
    // on with a block a piece and six warps (else the token loop of mv.cu; us, 5120 x 17408, 8 tokens: Q2_K 224 / 21, IQ2_XXS 252 / 42).
    const bool two_bit = ft == ILL_Q2_K || ft == ILL_IQ2_XXS;
    uint32_t stage;
    for (;; cb = 1) {
      f.cb = cb;
      f.npieces = (p.nblocks + cb - 1) / cb;
      f.pitch = (cb * bb + 15 + 15) / 16 * 16;
      while ((f.pitch / 16) % 8 % 2 == 0) f.pitch += 16;
      stage = (uint32_t)(MT_ROWS * f.pitch + 16 + 127) / 128 * 128;
      const uint32_t room = off + (ft == ILL_Q8_0 || ft == ILL_IQ2_XXS ? 0u : ft == ILL_Q4_K ? 16u : 32u) * ntok * (cols / 256) +
                            (two_bit ? 12288u : 16384u) + 2u * (two_bit && cb == 1 ? 6 : MT_SUMS) * stage + tables;
      if (room <= (two_bit ? 226u : 220u) * 1024u) break;
      if (!two_bit || cb == 1) return ILL_ERR_UNSUPPORTED;
    }
    f.piece_bytes = (uint32_t)(f.cb * bb);
    if (stage > p.stage_bytes) p.stage_bytes = stage;
    const int ns = f.npieces < MT_SUMS ? f.npieces : MT_SUMS;
    if (ns > p.nsums) p.nsums = ns;
  }
  if (fmt != ILL_Q8_0 && fmt != ILL_IQ2_XXS) off += 32u * ntok * (cols / 256);
  off = (off + 127) / 128 * 128;
  p.ring_off = off;
  // Warps a group and groups a CTA, for the least time: the tiles a group takes one after another, times the blocks of its busiest
  // warp, times what a block takes with that many warps an SM (a latency of 24, and 1 a warp).  The rings are as deep as fits (four
  // stages at most, two at least).  Swept over every pair on nine launches of a 0.5B, a 4B and a 27B model at 2, 4 and 16 tokens: the
  // fastest pair or one within 5 % of it but for a head of 151936 x 2560 at two tokens (10 %).  Short rows have few warps a group: such
  // a CTA takes groups without a tile up to eight warps, for the activations' sake (1024 x 256, 16 tokens, a warp / eight: Q6_K 4.9 / 3.4
  // us, Q4_K 4.6 / 3.1; over 1050 shapes of up to 1280 columns 6 % on average, 11 % slower at most, of 2.6 us).
  const uint32_t budget = 226u * 1024u - tables, part_bytes = 2u * p.nsums * ntok * 20 * 4;
  double best = 0;
  for (int gw = p.nsums; gw >= 1; --gw) {
    u8 sums[2][MT_SUMS];
    int most[2] = {};
    for (int i = 0; i < (two ? 2 : 1); ++i) most[i] = mt_deal(p.f[i].npieces, gw, sums[i]) * p.f[i].cb;
    const uint32_t ring1 = (uint32_t)gw * p.stage_bytes;
    for (int g = min(MT_MAX_WARPS / gw, MT_MAX_GROUPS); g >= 1; --g) {
      // (fewer groups have a tile each already, and with eight warps there are enough to bring the activations)
      if (g > 1 && (g - 1) * sms >= ntiles && (g - 1) * gw >= 8) continue;
      if (off + g * (part_bytes + 2 * ring1) > budget) continue;
      const long long rounds = (ntiles + (long long)g * sms - 1) / ((long long)g * sms);
      const long long busy = (ntiles + sms - 1) / sms;     // groups of a CTA that have a tile, at most
      const double a_tile = (double)(tiles[0] * most[0] + tiles[1] * most[1]) / ntiles, cost = rounds * a_tile * (24 + (g < busy ? g : busy) * gw);
      if (p.groups && cost >= best) continue;
      best = cost;
      p.groups = g;
      p.gw = gw;
      for (int i = 0; i < 2; ++i)
        for (int k = 0; k < MT_SUMS; ++k) p.f[i].sums[k] = sums[i][k];
      p.stages = (int)((budget - off - g * part_bytes) / (g * ring1));
      if (p.stages > MT_MAX_STAGES) p.stages = MT_MAX_STAGES;
    }
  }
  if (!p.groups) return ILL_ERR_UNSUPPORTED;
  off += (uint32_t)(p.groups * p.gw * p.stages) * p.stage_bytes;
  p.part_off = off;
  off += (uint32_t)p.groups * part_bytes;
  // Two CTAs an SM where their shared memory and registers fit: a grid of two an SM that holds one runs in two rounds, each with its
  // activations to bring (Q8_0 of 16 warps a CTA, 4 tokens: 4096 x 256 4.5 us, 2.7 with one; 17408 x 256 7.6 / 6.4)
  const int regs = 32 * p.gw * p.groups * mt_regs(fmt, n);
  const int per_sm = (int)((227u * 1024u) / (off + tables + 1024u)) >= 2 && 2 * regs <= 65536 ? 2 : 1;
  plan->grid = (int)((long long)sms * per_sm < ntiles ? (long long)sms * per_sm : ntiles);
  plan->smem = off;
  plan->fmt = fmt;
  plan->two = two;
  return ILL_OK;
}

// The several-token product on the tensor cores, for the formats it is written for; ILL_ERR_UNSUPPORTED otherwise (the caller then
// takes the CUDA-core kernel).
int mvt_try(int nmat, const int* fmts, const uint64_t* w, const int* rows, int cols, uint64_t xq, uint64_t xs, uint64_t xsum,
            const uint64_t* y, const uint64_t* bias, int acc, int n, void* stream) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  MtPlan plan;
  const int rc = mvt_plan(nmat, fmts, rows, cols, n, sms, &plan);
  if (rc) return rc;
  MtParams& p = plan.p;
  bool al4 = true;
  for (int i = 0; i < nmat; ++i) {
    p.m[i].w = (const u8*)(uintptr_t)w[i];
    p.m[i].y = (float*)(uintptr_t)y[i];
    p.m[i].bias = bias ? (const float*)(uintptr_t)bias[i] : nullptr;
    if (fmts[i] == ILL_Q4_K || fmts[i] == ILL_Q2_K) al4 = al4 && (w[i] & 3) == 0;
  }
  p.xq = (const i8*)(uintptr_t)xq;
  p.xs = (const float*)(uintptr_t)xs;
  p.xsum = (const int16_t*)(uintptr_t)xsum;
  p.acc = acc;
  return mvt_launch(mt_kernel(plan.fmt, plan.two, al4, n), p, plan.smem, plan.grid, (cudaStream_t)stream);
}

}  // namespace ill

using namespace ill;

extern "C" int ill_test_few_tokens_plan(int nmat, int fmt0, int fmt1, int fmt2, int rows0, int rows1, int rows2, int cols, int n, int sms,
                                        int* out) {
  const int fmts[3] = {fmt0, fmt1, fmt2}, rows[3] = {rows0, rows1, rows2};
  if (!out || nmat < 1 || nmat > MT_MATS || cols <= 0 || sms < 0) return ILL_ERR_ARG;
  for (int i = 0; i < nmat; ++i) {
    const int bw = fmt_block_weights(fmts[i]);
    if (!bw || rows[i] <= 0 || cols % bw) return ILL_ERR_ARG;
  }
  MtPlan plan;
  const int rc = mvt_plan(nmat, fmts, rows, cols, n, sms ? sms : 148, &plan);
  if (rc) return rc;
  const MtParams& p = plan.p;
  out[0] = p.gw;
  out[1] = p.groups;
  out[2] = mt_barrier(p.groups - 1);
  out[3] = p.stages;
  out[4] = plan.grid;
  out[5] = (int)plan.smem + (plan.fmt == ILL_IQ2_XXS ? IQ_TABLE_BYTES : 0);
  out[6] = mt_regs(plan.fmt, n);
  out[7] = 0;
  if (!sms) {
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, mt_kernel(plan.fmt, plan.two, true, n));
    if (e != cudaSuccess) return cuda_fail(e);
    out[7] = fa.numRegs;
  }
  return ILL_OK;
}
