// mve.cu -- the experts' products for the rows of a few tokens, Q2_K and IQ2_XXS: the weights of an expert that has up to sixteen rows
// are read and unpacked once for all of them, the integer block dots on the tensor cores' int8 path (mma.sync, mtblock.cuh).
//
// A persistent CTA of sixteen warps an SM.  The experts' tiles of 16 weight rows (or of gate's and up's) lie one after another on a line,
// a tile as long as it takes (me_cost), and every CTA has an even share of the line.  It stages an expert's activations, read where the
// tokens' quants lie, and its warps take that expert's tiles, all blocks of a row in order: the chunk kernel's order (mm_id.cu), and
// its bits while a block's sum stays under 2^24 (IQ2_XXS's can reach 2.6 times that: int32 holds it, the chunk kernel's fp32 rounds).  Weights: 16-byte cp.async into a ring a warp, four lanes a row segment, on across tiles and experts.
//
// Why not the chunk kernel: its block of 128 weight rows goes through raw bytes, fp16 operands in tensor memory, a product and a drain, a
// chain of about 1700 cycles whatever the rows of X; here a block of 128 x 256 weights takes 970 (Q2_K) and 1370 (IQ2_XXS) cycles an SM
// for up to eight rows and 1180 and 1580 for sixteen, and HBM would take 460 and 360.  Beyond sixteen rows the chunk kernel's tile of 64
// costs less than a second pass.  Bound by instruction issue: about 300 (Q2_K) and 540 (IQ2_XXS) a block of sixteen weight rows, the
// logic (unpacking, look-ups) at half rate, 57 % and 67 % of the issue slots taken by the sixteen warps that 128 registers allow (twenty
// of 96 registers: slower).  An expert of more rows is left to the chunk kernel, or (ALL: no other launch follows) taken in passes of
// sixteen.  us of the routed experts, before / now: 64 tokens on 288 experts of Q2_K 757 / 467 (gate and up 475 / 268),
// on 256 of IQ2_XXS and Q2_K 1275 / 686; 2 tokens 153 / 123 and 145 / 115.
//
// Replaces d4_mv_iq2_xxs / d4_mv_q2_k with COUNTS / BASES (src/cuda/ds4f.cu:769-902) behind DK-FFN-SMALL
// (src/cuda-ds4f-spec.lisp:31-132).
#include "host.h"
#include "iq2xxs_tables.cuh"
#include "mtblock.cuh"
#include "quantdev.cuh"

namespace ill {

constexpr int ME_WARPS = 16, ME_ROWS = 16, ME_MAX_STAGES = 4, ME_CB = 4 /* blocks a staged piece, at most */, ME_MAX_NE = 1024,
              ME_LINE = 0x3fffffff;  // the line's length, at most

struct MeParams {
  const unsigned long long* ptrs;
  int ne;                    // experts
  const unsigned* counts;      // rows of each expert, the first of them, the tokens they are
  const unsigned* bases;
  const unsigned* map;
  long long total_rows;
  long long add, up_add;       // the matrix within an expert; that of up beyond it
  int cols, rows, row_bytes, nb;
  int cb, npieces;             // blocks a staged piece (a warp's unit of copying); pieces a row
  const i8* xq;
  const float* xs;
  const int16_t* xsum;
  float* y;
  long long y_stride;          // floats between the rows' results
  float* y2;                   // two matrices, results apart: that of up
  const float* weights;        // ... or gated: a row's weight
  float clamp;
  int most;                    // rows that are taken at a time: 8 or 16
  int all;                     // an expert with more rows is taken in passes of that many, not left out
  int pitch, stages;           // bytes between the rows of a staged piece; stages a warp
  uint32_t stage_bytes, xs_off, bs_off, ring_off, first_off /* where each expert's tiles start on the line; its end */;
  int x_stride;
};

// What a tile of a segment of N tokens takes: two tiles of eight tokens about half as much again as one
__device__ __forceinline__ int me_cost(int n) { return n > 8 ? 3 : 2; }

// 16 bytes global -> shared, asynchronously
__device__ __forceinline__ void cp_async16_at(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

template <int N> struct MeN { static constexpr int value = N; };

template <int FMT, bool TWO>
__global__ void __launch_bounds__(32 * ME_WARPS, 1) mve_kernel(const __grid_constant__ MeParams p) {
  extern __shared__ __align__(128) u8 smem[];
  constexpr int BB = Fmt<FMT>::BB, MATS = TWO ? 2 : 1;
  constexpr bool SUMS = FMT == ILL_Q2_K, AL4 = FMT == ILL_Q2_K;  // (Q2_K: 84-byte blocks from a word on; IQ2_XXS: 66-byte ones, on two bytes)
  int* first = (int*)(smem + p.first_off);  // where each expert's tiles start on the line; its end
  __shared__ uint2 iq_grid[FMT == ILL_IQ2_XXS ? IQ_TABLE_BYTES / 8 : 1];  // (static: the look-ups' addresses start at a constant)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  constexpr int nwarps = ME_WARPS, nthreads = 32 * ME_WARPS;
  const int ntr = (p.rows + ME_ROWS - 1) / ME_ROWS;
  if constexpr (FMT == ILL_IQ2_XXS) iq_tables_fill(iq_grid, iq_grid + IQ_COPIES * 256, ill_iq2xxs_grid, ill_ksigns_iq2xs);
  pdl_launch_dependents();
  pdl_wait();  // the tables of experts may come from the kernel before

  // rows of an expert that is this launch's, and all of whose rows are there
  auto count = [&](int e) {
    const unsigned c = p.counts[e];
    return (p.all || c <= (unsigned)p.most) && (long long)p.bases[e] + c <= p.total_rows ? (int)c : 0;
  };
  const int pass_cost = ntr * me_cost(p.most);  // of a pass that is not an expert's last
  for (int e = tid; e < p.ne; e += nthreads) {
    const int c = count(e), passes = max(c - 1, 0) >> (p.most == 16 ? 4 : 3);
    first[e] = c ? passes * pass_cost + ntr * me_cost(c - passes * p.most) : 0;
  }
  __syncthreads();
  if (warp == 0) {
    int before = 0;
    for (int e0 = 0; e0 < p.ne; e0 += 32) {
      const int e = e0 + lane;
      int incl = e < p.ne ? first[e] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {  // (what passes ME_LINE is of counts that add up to more rows than there are)
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl = min(incl + v, ME_LINE);
      }
      const int excl = __shfl_up_sync(0xffffffffu, incl, 1);
      if (e < p.ne) first[e] = min(before + (lane ? excl : 0), ME_LINE);
      before = min(before + __shfl_sync(0xffffffffu, incl, 31), ME_LINE);
    }
    if (lane == 0) first[p.ne] = before;
  }
  __syncthreads();  // (and IQ2_XXS's tables)
  const long long line = first[p.ne];
  const int lo = (int)(line * blockIdx.x / gridDim.x), hi = (int)(line * (blockIdx.x + 1) / gridDim.x);

  // The CTA's experts in order, pass by pass: of each, the tiles that start in LO .. HI
  struct Seg {
    int e, pass, row0, n;  // the expert, the pass, its first row, its rows
    int t0, t1;            // the CTA's tiles of it
    int end;               // where it ends on the line
    const u8* w;
  };
  auto fill = [&](Seg& s) {
    const int done = s.pass * p.most;
    s.row0 = (int)p.bases[s.e] + done;
    s.n = min(count(s.e) - done, p.most);
    const int cost = me_cost(s.n), at = first[s.e] + s.pass * pass_cost;
    s.t0 = at >= lo ? 0 : (lo - at + cost - 1) / cost;
    s.t1 = min(ntr, (hi - at + cost - 1) / cost);
    s.end = at + ntr * cost;
    s.w = (const u8*)(uintptr_t)after_wait(p.ptrs)[s.e] + p.add;
  };
  auto begin = [&](Seg& s) -> bool {  // the one that LO lies in: the last that starts there or before (one without rows ends where it starts)
    if (lo >= hi) return false;
    int a = 0, b = p.ne - 1;
    while (a < b) {
      const int m = (a + b + 1) >> 1;
      if (first[m] <= lo) a = m; else b = m - 1;
    }
    s.e = a;
    s.pass = p.all ? (lo - first[a]) / pass_cost : 0;
    fill(s);
    return true;
  };
  auto next = [&](Seg& s) -> bool {
    const int end = s.end;
    if (end >= hi) return false;
    ++s.pass;
    if (first[s.e + 1] <= end) {
      do ++s.e; while (first[s.e + 1] <= end);  // (the line's end is beyond END)
      s.pass = 0;
    }
    fill(s);
    return true;
  };

  const uint32_t ring = smem_u32(smem) + p.ring_off + warp * p.stages * p.stage_bytes;
  Seg is;                        // the pieces brought next: segment, tile, matrix, piece; the stage they go to
  int i_tile = 0, i_mat = 0, i_pc = 0, i_slot = 0;
  bool i_more = begin(is);
  auto settle = [&]() {          // on to the first segment from IS on that this warp has a tile of
    i_tile = is.t0 + warp;
    while (i_more && i_tile >= is.t1) {
      i_more = next(is);
      i_tile = is.t0 + warp;
    }
  };
  if (i_more) settle();
  auto issue_next = [&]() {      // all lanes: four a row segment, eight rows at a time; a group of cp.async, possibly empty
    if (i_more) {
      const int row0 = i_tile * ME_ROWS + g;
      const uint32_t dst = ring + i_slot * p.stage_bytes + g * p.pitch + 16 * t, len = (uint32_t)min(p.cb, p.nb - i_pc * p.cb) * BB;
      const u8* src = is.w + (i_mat ? p.up_add : 0) + (long long)row0 * p.row_bytes + i_pc * (p.cb * BB);
#pragma unroll
      for (int h = 0; h < ME_ROWS; h += 8) {
        if (row0 + h < p.rows) {
          // the 16-byte pieces that cover the segment, from the boundary at or before it: the quad's lanes take one each
          const uint32_t off = (uint32_t)(uintptr_t)src & 15u, end = off + len;
          const u8* from = src - off + 16 * t;
#pragma unroll
          for (int k = 0; k < (ME_CB * BB + 30) / 16; k += 4)
            if (16u * (t + k) < end) cp_async16_at(dst + h * p.pitch + 16 * k, from + 16 * k);
        }
        src += 8ll * p.row_bytes;
      }
      if (++i_pc == p.npieces) {
        i_pc = 0;
        if (++i_mat == MATS) {
          i_mat = 0;
          i_tile += nwarps;
          if (i_tile >= is.t1) {
            i_more = next(is);
            settle();
          }
        }
      }
      i_slot = i_slot + 1 == p.stages ? 0 : i_slot + 1;
    }
    cp_async_commit();
  };
  for (int i = 0; i < p.stages; ++i) issue_next();

  MtLane x;
  x.set<FMT>(smem_u32(smem), p.x_stride, smem_u32(smem) + p.xs_off, smem_u32(smem) + p.bs_off, p.nb, FMT == ILL_IQ2_XXS ? smem_u32(iq_grid) : 0u, lane);
  auto stage_x = [&](const Seg& s) {
    const int per_tok = p.cols / 16;
    auto token = [&](int i) -> long long {
      return p.map ? (long long)p.map[s.row0 + i] : s.row0 + i;
    };
    for (int tk = warp; tk < s.n; tk += nwarps) {
      const long long tok = token(tk);
      for (int j = lane; j < per_tok; j += 32) cp_async16(smem + (size_t)tk * p.x_stride + 16 * j, p.xq + tok * p.cols + 16 * j);
    }
    for (int tk = nwarps - 1 - warp; tk < s.n; tk += nwarps) {
      const long long tok = token(tk);
      for (int j = lane; j < p.nb; j += 32) cp_async4((float*)(smem + p.xs_off) + tk * p.nb + j, p.xs + tok * p.nb + j);
      if constexpr (SUMS) {
        for (int j = lane; j < 2 * p.nb; j += 32) {
          const uint2* src = (const uint2*)(p.xsum + tok * per_tok) + 2 * j;
          const uint2 a = src[0], b = src[1];  // (the sums lie on eight bytes, if not on sixteen)
          u8* d = smem + p.bs_off + ((size_t)tk * p.nb + (j >> 1)) * 32 + 8 * (j & 1);
          split_sums(make_uint4(a.x, a.y, b.x, b.y), *(uint2*)d, *(uint2*)(d + 16));
        }
      }
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
  };

  int slot = 0;
  Seg seg;
  bool staged = false;
  for (bool more = begin(seg); more; more = next(seg)) {
    if (staged) __syncthreads();  // every warp is through with the segment before
    stage_x(seg);
    staged = true;
    auto tiles = [&](auto nt8) {
      constexpr int NT8 = decltype(nt8)::value;
      for (int tile = seg.t0 + warp; tile < seg.t1; tile += nwarps) {
        float acc[MATS][NT8][4];
#pragma unroll
        for (int m = 0; m < MATS; ++m) {
#pragma unroll
          for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[m][nt][i] = 0.0f;
          const u8* w = seg.w + (m ? p.up_add : 0);
          for (int pc = 0; pc < p.npieces; ++pc) {
            // all but the newer stages' groups: this piece is in
            if (p.stages == 4) asm volatile("cp.async.wait_group 3;" ::: "memory");
            else if (p.stages == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            const uint32_t piece = ring + slot * p.stage_bytes;
            slot = slot + 1 == p.stages ? 0 : slot + 1;
            // a row's segment starts where its block starts inside the 16-byte aligned span that was copied
            const uint32_t o0 = (uint32_t)(uintptr_t)w + (uint32_t)(tile * ME_ROWS + g) * (uint32_t)p.row_bytes + (uint32_t)(pc * p.cb * BB);
            uint32_t s0 = piece + g * p.pitch + (o0 & 15u), s8 = piece + (g + 8) * p.pitch + ((o0 + 8u * (uint32_t)p.row_bytes) & 15u);
            const int nhere = min(p.cb, p.nb - pc * p.cb);
            for (int j = 0; j < nhere; ++j, s0 += BB, s8 += BB) MtBlock<FMT, NT8, AL4>::run(s0, s8, pc * p.cb + j, x, lane, acc[m]);
            __syncwarp();
            issue_next();
          }
        }
        const float fin = FMT == ILL_IQ2_XXS ? 0.125f : 1.0f;
#pragma unroll
        for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = tile * ME_ROWS + g + 8 * (i >> 1), tk = 8 * nt + 2 * t + (i & 1);
            if (row < p.rows && tk < seg.n) {
              float v = acc[0][nt][i] * fin;
              const long long at = (long long)(seg.row0 + tk) * p.y_stride + row;
              if constexpr (TWO) {
                const float u = acc[MATS - 1][nt][i] * fin;
                if (p.weights) v = d4_middle(v, u, p.weights[seg.row0 + tk], p.clamp);
                else p.y2[at] = u;
              }
              p.y[at] = v;
            }
          }
      }
    };
    if (seg.n <= 8) tiles(MeN<1>());
    else tiles(MeN<2>());
  }
  cp_async_wait_all();
}

// Sizes of a launch for experts of up to 16 rows, or 8 where the activations of 16 do not fit in shared memory; ILL_ERR_UNSUPPORTED
// where those of 8 do not.
static int me_plan(int fmt, int cols, int rows, MeParams* pp, size_t* smem) {
  MeParams& p = *pp;
  const int bb = fmt_block_bytes(fmt);
  p.cols = cols;
  p.rows = rows;
  p.nb = cols / 256;
  p.row_bytes = p.nb * bb;
  p.x_stride = mt_x_stride(fmt, cols);
  const uint32_t budget = 226u * 1024u - (fmt == ILL_IQ2_XXS ? IQ_TABLE_BYTES : 0);
  for (p.most = 16; p.most >= 8; p.most -= 8) {
    uint32_t off = p.most * (uint32_t)p.x_stride;
    p.xs_off = off;
    off += (4u * p.most * p.nb + 15) / 16 * 16;
    p.bs_off = off;
    if (fmt == ILL_Q2_K) off += 32u * p.most * p.nb;
    p.first_off = off;
    off += 4u * (ME_MAX_NE + 1);
    off = (off + 127) / 128 * 128;
    p.ring_off = off;
    // the longest pieces that leave room for two stages a warp
    for (p.cb = ME_CB; p.cb; --p.cb) {
      p.npieces = (p.nb + p.cb - 1) / p.cb;
      p.pitch = (p.cb * bb + 15 + 15) / 16 * 16;
      while ((p.pitch / 16) % 8 % 2 == 0) p.pitch += 16;
      p.stage_bytes = (uint32_t)(ME_ROWS * p.pitch + 16 + 127) / 128 * 128;
      const uint32_t ring = (uint32_t)ME_WARPS * p.stage_bytes;
      if (off + 2 * ring > budget) continue;
      p.stages = (int)((budget - off) / ring);
      if (p.stages > ME_MAX_STAGES) p.stages = ME_MAX_STAGES;
      *smem = off + p.stages * ring;
      return ILL_OK;
    }
  }
  return ILL_ERR_UNSUPPORTED;
}

}  // namespace ill

using namespace ill;

extern "C" int ill_moe_few_most(int fmt, int ncols) {
  MeParams p = {};
  size_t smem = 0;
  if ((fmt != ILL_Q2_K && fmt != ILL_IQ2_XXS) || ncols <= 0 || ncols % 256 || ncols > 65536) return 0;
  return me_plan(fmt, ncols, 1, &p, &smem) == ILL_OK ? p.most : 0;
}

static int moe_few(bool all, int fmt, int ncols, int nrows, int64_t add, int64_t add2, ill_dptr ptrs, ill_dptr counts, ill_dptr bases, int ne,
                   int64_t total_rows, ill_dptr xq, ill_dptr xs, ill_dptr xsum, ill_dptr map, float clamp, ill_dptr weights, ill_dptr y,
                   ill_dptr y2, int64_t y_stride, ill_stream stream) {
  if (fmt != ILL_Q2_K && fmt != ILL_IQ2_XXS) return ILL_ERR_UNSUPPORTED;
  if (ncols <= 0 || ncols % 256 || ncols > 65536 || nrows <= 0 || ne <= 0 || total_rows < 0 || total_rows > 0x7fffffffll || y_stride < nrows)
    return ILL_ERR_ARG;
  if (!ptrs || !counts || !bases || !xq || !xs || !y || (fmt == ILL_Q2_K && !xsum)) return ILL_ERR_ARG;
  if ((ptrs & 7) || (counts & 3) || (bases & 3) || (xq & 15) || (xs & 3) || (xsum & 7) || (map & 3) || (weights & 3) || (y & 3) || (y2 & 3))
    return ILL_ERR_ALIGN;
  if ((add | add2) & (fmt == ILL_Q2_K ? 3 : 1)) return ILL_ERR_ALIGN;
  const long long ntr = (nrows + ME_ROWS - 1) / ME_ROWS, experts = ne < total_rows ? ne : total_rows;  // with rows, at most
  if (ne > ME_MAX_NE || 3 * ntr * ne > ME_LINE || (all && total_rows > 8 * (ME_LINE / (3 * ntr) - ne))) return ILL_ERR_TOO_LARGE;
  if (total_rows == 0) return ILL_OK;
  MeParams p = {};
  size_t smem = 0;
  const int rc = me_plan(fmt, ncols, nrows, &p, &smem);
  if (rc) return rc;
  p.ptrs = (const unsigned long long*)(uintptr_t)ptrs;
  p.counts = (const unsigned*)(uintptr_t)counts;
  p.bases = (const unsigned*)(uintptr_t)bases;
  p.map = (const unsigned*)(uintptr_t)map;
  p.ne = ne;
  p.all = all;
  p.total_rows = total_rows;
  p.add = add;
  p.up_add = add2 - add;
  p.xq = (const i8*)(uintptr_t)xq;
  p.xs = (const float*)(uintptr_t)xs;
  p.xsum = (const int16_t*)(uintptr_t)xsum;
  p.y = (float*)(uintptr_t)y;
  p.y2 = (float*)(uintptr_t)y2;
  p.y_stride = y_stride;
  p.weights = (const float*)(uintptr_t)weights;
  p.clamp = clamp;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  const bool two = weights || y2;
  const void* k = fmt == ILL_IQ2_XXS ? (two ? (const void*)mve_kernel<ILL_IQ2_XXS, true> : (const void*)mve_kernel<ILL_IQ2_XXS, false>)
                                     : (two ? (const void*)mve_kernel<ILL_Q2_K, true> : (const void*)mve_kernel<ILL_Q2_K, false>);
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e);
  void* args[] = {&p};
  return launch_kernel(k, dim3((unsigned)(experts * ntr < sms ? experts * ntr : sms)), dim3(32 * ME_WARPS), smem, args, (cudaStream_t)stream);
}

extern "C" int ill_moe_few(int fmt, int ncols, int nrows, int64_t add, ill_dptr ptrs, ill_dptr counts, ill_dptr bases, int ne,
                           int64_t total_rows, ill_dptr xq, ill_dptr xs, ill_dptr xsum, ill_dptr map, ill_dptr y, int64_t y_stride,
                           ill_stream stream) {
  return moe_few(false, fmt, ncols, nrows, add, add, ptrs, counts, bases, ne, total_rows, xq, xs, xsum, map, 0.0f, 0, y, 0, y_stride, stream);
}

extern "C" int ill_moe_few2(int fmt, int ncols, int nrows, int64_t add, int64_t add2, ill_dptr ptrs, ill_dptr counts, ill_dptr bases, int ne,
                            int64_t total_rows, ill_dptr xq, ill_dptr xs, ill_dptr xsum, ill_dptr map, ill_dptr y, ill_dptr y2,
                            int64_t y_stride, ill_stream stream) {
  if (!y2) return ILL_ERR_ARG;
  return moe_few(false, fmt, ncols, nrows, add, add2, ptrs, counts, bases, ne, total_rows, xq, xs, xsum, map, 0.0f, 0, y, y2, y_stride, stream);
}

extern "C" int ill_moe_few_glu(int fmt, int ncols, int nrows, int64_t gate_add, int64_t up_add, ill_dptr ptrs, ill_dptr counts,
                               ill_dptr bases, int ne, int64_t total_rows, ill_dptr xq, ill_dptr xs, ill_dptr xsum, ill_dptr map,
                               float clamp, ill_dptr weights, ill_dptr mid, int64_t mid_stride, ill_stream stream) {
  if (!weights) return ILL_ERR_ARG;
  return moe_few(false, fmt, ncols, nrows, gate_add, up_add, ptrs, counts, bases, ne, total_rows, xq, xs, xsum, map, clamp, weights, mid, 0, mid_stride,
                 stream);
}

extern "C" int ill_moe_few_all(int fmt, int ncols, int nrows, int64_t add, ill_dptr ptrs, ill_dptr counts, ill_dptr bases, int ne,
                               int64_t total_rows, ill_dptr xq, ill_dptr xs, ill_dptr xsum, ill_dptr map, ill_dptr y, int64_t y_stride,
                               ill_stream stream) {
  return moe_few(true, fmt, ncols, nrows, add, add, ptrs, counts, bases, ne, total_rows, xq, xs, xsum, map, 0.0f, 0, y, 0, y_stride, stream);
}

extern "C" int ill_moe_few_glu_all(int fmt, int ncols, int nrows, int64_t gate_add, int64_t up_add, ill_dptr ptrs, ill_dptr counts,
                                   ill_dptr bases, int ne, int64_t total_rows, ill_dptr xq, ill_dptr xs, ill_dptr xsum, ill_dptr map,
                                   float clamp, ill_dptr weights, ill_dptr mid, int64_t mid_stride, ill_stream stream) {
  if (!weights) return ILL_ERR_ARG;
  return moe_few(true, fmt, ncols, nrows, gate_add, up_add, ptrs, counts, bases, ne, total_rows, xq, xs, xsum, map, clamp, weights, mid, 0,
                 mid_stride, stream);
}
