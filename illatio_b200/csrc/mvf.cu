// mvf.cu -- small dense products with unquantized weights: the router's logits and the other F16 /
// BF16 / F32 tensors that sit between the quantized products (DK-MV16, src/cuda-ds4f.lisp:767-771:
// d4_mv_f16 src/cuda/ds4f.cu:145-165, g53_mv_bf16 src/cuda/glm53.cu:11, d41_mv_f32
// src/cuda/ds4f_v41.cu:204, and their several-token forms d4_mv_f16n / d41_mv_f32n).  The CPU path is
// F32MV! (src/ds4f.lisp:256-276) on the weights widened to float: a float dot a row.
//
// A token, or two to four: pure bandwidth and small (the router of a 256-expert layer is 2 MB), a warp a row, 16-byte
// loads of the row, the tokens' activations from L1/L2, fp32 accumulate, one shuffle reduction a (row, token).  More
// tokens: tiles staged in shared memory (mm_dense_kernel).  A sum is taken in the same order by all of them.
#include <cuda_bf16.h>

#include "common.cuh"
#include "host.h"

namespace ill {

template <int TYPE> struct DenseElt;
template <> struct DenseElt<ILL_F32> { static constexpr int BYTES = 4; };
template <> struct DenseElt<ILL_F16> { static constexpr int BYTES = 2; };
template <> struct DenseElt<ILL_BF16> { static constexpr int BYTES = 2; };

template <int TYPE>
__device__ __forceinline__ float dense_at(const u8* row, int j) {
  if constexpr (TYPE == ILL_F32) return ((const float*)row)[j];
  else if constexpr (TYPE == ILL_F16) return __half2float(((const __half*)row)[j]);
  else return __bfloat162float(((const __nv_bfloat16*)row)[j]);
}
// eight (four for F32) consecutive weights from a 16-byte load, as floats
template <int TYPE>
__device__ __forceinline__ void dense_vec(const uint4 v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  if constexpr (TYPE == ILL_F32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = __uint_as_float(w[i]);
  } else if constexpr (TYPE == ILL_F16) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 p = __half22float2(*(const __half2*)&w[i]);
      f[2 * i] = p.x; f[2 * i + 1] = p.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // a bfloat16 is the top half of a float
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
}

constexpr int MVF_MAXN = 16;

// Y[t * y_stride + r] = W[r] . X[t], r < rows, t < n: blockIdx.y takes the tokens sixteen at a time (a chunk's
// router logits: the matrix is small and stays in L2 between the token batches).  A warp takes RW rows against the
// batch's tokens: one row for a token or a few (more warps in flight), four for a chunk (an activation vector
// loaded once serves four rows).
template <int TYPE, int RW>
__global__ void __launch_bounds__(256) mv_dense_kernel(const u8* __restrict__ w, int rows, int cols, const float* __restrict__ x,
                                                       float* __restrict__ y, int n, long long y_stride, int vec_ok) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int r0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * RW;
  if (r0 >= rows) return;
  {
    const long long t0 = (long long)blockIdx.y * MVF_MAXN;
    x += t0 * cols;
    y += t0 * y_stride;
    n = min(n - (int)t0, MVF_MAXN);
  }
  constexpr int EB = DenseElt<TYPE>::BYTES, VE = 16 / EB;  // elements a 16-byte load
  const u8* row[RW];
#pragma unroll
  for (int q = 0; q < RW; ++q) row[q] = w + (long long)min(r0 + q, rows - 1) * cols * EB;  // rows past the end repeat the last: not stored
  float sum[RW][MVF_MAXN];
#pragma unroll
  for (int q = 0; q < RW; ++q)
#pragma unroll
    for (int t = 0; t < MVF_MAXN; ++t) sum[q][t] = 0.0f;
  int j0 = 0;
  if (vec_ok) {  // rows and activations 16-byte aligned, cols a whole number of vectors
    const int nv = cols / VE;
    for (int i = lane; i < nv; i += 32) {
      float f[RW][8];
#pragma unroll
      for (int q = 0; q < RW; ++q) dense_vec<TYPE>(__ldg((const uint4*)row[q] + i), f[q]);
#pragma unroll
      for (int t = 0; t < MVF_MAXN; ++t) {
        if (t < n) {
          const float4* xv = (const float4*)(x + (long long)t * cols + (long long)i * VE);
          const float4 a = xv[0];
          float4 b = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if constexpr (VE == 8) b = xv[1];
#pragma unroll
          for (int q = 0; q < RW; ++q) {
            float s = sum[q][t];
            s = fmaf(f[q][0], a.x, s); s = fmaf(f[q][1], a.y, s); s = fmaf(f[q][2], a.z, s); s = fmaf(f[q][3], a.w, s);
            if constexpr (VE == 8) {
              s = fmaf(f[q][4], b.x, s); s = fmaf(f[q][5], b.y, s); s = fmaf(f[q][6], b.z, s); s = fmaf(f[q][7], b.w, s);
            }
            sum[q][t] = s;
          }
        }
      }
    }
    j0 = nv * VE;
  }
  for (int j = j0 + lane; j < cols; j += 32) {
#pragma unroll
    for (int q = 0; q < RW; ++q) {
      const float wv = dense_at<TYPE>(row[q], j);
#pragma unroll
      for (int t = 0; t < MVF_MAXN; ++t)
        if (t < n) sum[q][t] = fmaf(wv, x[(long long)t * cols + j], sum[q][t]);
    }
  }
#pragma unroll
  for (int q = 0; q < RW; ++q)
#pragma unroll
    for (int t = 0; t < MVF_MAXN; ++t) {
      if (t < n) {
        const float v = warp_sum(sum[q][t]);
        if (lane == 0 && r0 + q < rows) y[(long long)t * y_stride + r0 + q] = v;
      }
    }
}

// One token: a warp a row, as above (the same bits), the row on its way to L2 before the kernel waits for the one before it
// (which may have written it), then in registers whole; two-warp CTAs reach 128 SMs.  The 2 MB of a 256-expert router come from
// HBM while the kernel before this one ends, where a loop that has four loads in flight paid their latency four times after it:
// a norm and this kernel of F16 [256, 4096] in a graph take 6.1 us together, 18.6 with that loop, 7.4 without the prefetch.
constexpr int MVF_AHEAD = 20;  // 5120 two-byte columns in one go
template <int TYPE>
__global__ void __launch_bounds__(64) mv_dense_one_kernel(const u8* __restrict__ w, int rows, int cols, const float* __restrict__ x,
                                                          float* __restrict__ y) {
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, r = blockIdx.x * 2 + (threadIdx.x >> 5);
  constexpr int EB = DenseElt<TYPE>::BYTES, VE = 16 / EB;
  const int nv = cols / VE;
  const uint4* row = (const uint4*)(w + (long long)min(r, rows - 1) * cols * EB);
  for (int i = 2 * lane; i < nv; i += 64) prefetch_l2(row + i);
  pdl_wait();
  row = after_wait(row);
  x = after_wait(x);
  float sum = 0.0f;
  for (int base = 0; base < nv; base += 32 * MVF_AHEAD) {
    uint4 v[MVF_AHEAD];
#pragma unroll
    for (int j = 0; j < MVF_AHEAD; ++j) {
      const int i = base + 32 * j + lane;
      if (i < nv) v[j] = __ldg(row + i);
    }
#pragma unroll
    for (int j = 0; j < MVF_AHEAD; ++j) {
      const int i = base + 32 * j + lane;
      if (i < nv) {
        float f[8];
        dense_vec<TYPE>(v[j], f);
        const float4* xv = (const float4*)(x + (long long)i * VE);
        const float4 a = xv[0];
        sum = fmaf(f[0], a.x, sum); sum = fmaf(f[1], a.y, sum); sum = fmaf(f[2], a.z, sum); sum = fmaf(f[3], a.w, sum);
        if constexpr (VE == 8) {
          const float4 b = xv[1];
          sum = fmaf(f[4], b.x, sum); sum = fmaf(f[5], b.y, sum); sum = fmaf(f[6], b.z, sum); sum = fmaf(f[7], b.w, sum);
        }
      }
    }
  }
  sum = warp_sum(sum);
  if (lane == 0 && r < rows) y[r] = sum;
}

__device__ __forceinline__ void mvf_cp16(void* dst, const void* src, bool there) {  // 16 bytes, or zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// The same products for a chunk of tokens, tiled: a CTA of WR x WT warps takes WR * RW rows against WT * NT tokens, a
// warp RW x NT of them with K dealt to its lanes as above (so the sums are the same bits).  Bound by the fp32 pipe:
// a vector of K is RW * NT * 8 multiply-adds for RW + 2 NT 16-byte shared loads and RW conversions, against one row's
// 4 x 8 for as many loads of x from L1 in mv_dense_kernel.  K comes in slabs of 32 vectors (a vector a lane) through a
// ring of MVF_STAGES cp.async stages; a token's slab is stored even 16-byte chunks first, so that the lanes'
// two loads of it are contiguous.  The lanes meet by halves (each exchange sends half of the sums that are
// left): the pairs that a shuffle per sum would add, in a quarter of the shuffles.
// 4096 tokens x F16 [256, 4096] on one B200: 305 us (28 TFLOP/s; 995 with mv_dense_kernel), 8192 x [288, 5120] 860 (2866),
// 64 x [288, 5120] 36 (114): two warps a scheduler leave the fp32 pipe at 40%, but twelve warps of 8 x 8 were no faster.
constexpr int MVF_STAGES = 3;
template <int TYPE, int RW, int NT, int WR, int WT>
struct MvfTile {
  static constexpr int VE = 16 / DenseElt<TYPE>::BYTES, ROWS = RW * WR, TOKS = NT * WT, XB = 32 * VE * 4;  // bytes of a token's slab
  static constexpr int STAGE = ROWS * 512 + TOKS * XB;
  static constexpr size_t SMEM = (size_t)MVF_STAGES * STAGE;
};
template <int TYPE, int RW, int NT, int WR, int WT>
__global__ void __launch_bounds__(32 * WR * WT) mm_dense_kernel(const u8* __restrict__ w, int rows, int cols, const float* __restrict__ x,
                                                                float* __restrict__ y, int n, long long y_stride) {
  typedef MvfTile<TYPE, RW, NT, WR, WT> T;
  constexpr int VE = T::VE, EB = DenseElt<TYPE>::BYTES, XC = T::XB / 16, THREADS = 32 * WR * WT;
  extern __shared__ __align__(128) u8 smem[];
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wr = warp % WR, wt = warp / WR;
  const int r0 = blockIdx.x * T::ROWS;
  const long long t0 = (long long)blockIdx.y * T::TOKS;
  const int nv = cols / VE, nslab = (nv + 31) / 32;
  pdl_wait();
  // this thread's chunks of a slab: rows a constant distance apart, so an address is an addition (rows and tokens past the
  // last, and vectors past a row's end, are zeros that nothing is read for)
  constexpr int WSTEP = THREADS / 32, XSTEP = THREADS / XC, WCH = (T::ROWS + WSTEP - 1) / WSTEP, XCH = (T::TOKS + XSTEP - 1) / XSTEP;
  static_assert(THREADS % XC == 0, "a token's chunks are shared by whole threads");
  const int cw = tid & 31, cx = tid % XC, rw0 = tid >> 5, rx0 = tid / XC;
  const u8* wsrc = w + ((long long)(r0 + rw0) * cols + cw * VE) * EB;
  const float* xsrc = x + (t0 + rx0) * cols + 4 * cx;
  const long long wstep = (long long)WSTEP * cols * EB, xstep = (long long)XSTEP * cols;
  u8* wdst = smem + rw0 * 512 + 16 * cw;
  u8* xdst = smem + T::ROWS * 512 + rx0 * T::XB + 16 * (XC == 64 ? (cx & 1) * 32 + (cx >> 1) : cx);
  auto stage = [&](int slab) {
    const int off = (slab % MVF_STAGES) * T::STAGE;
    const bool win = slab * 32 + cw < nv, xin = slab * 32 + cx / (XC / 32) < nv;
    const u8* ws = wsrc + (long long)slab * (32 * VE * EB);
    const float* xp = xsrc + (long long)slab * (32 * VE);
#pragma unroll
    for (int i = 0; i < WCH; ++i) {
      if (T::ROWS % WSTEP && rw0 + i * WSTEP >= T::ROWS) break;
      const bool in = win && r0 + rw0 + i * WSTEP < rows;
      mvf_cp16(wdst + off + i * WSTEP * 512, in ? ws + i * wstep : w, in);
    }
#pragma unroll
    for (int i = 0; i < XCH; ++i) {
      if (T::TOKS % XSTEP && rx0 + i * XSTEP >= T::TOKS) break;
      const bool in = xin && t0 + rx0 + i * XSTEP < n;
      mvf_cp16(xdst + off + i * XSTEP * T::XB, in ? xp + i * xstep : x, in);
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
  for (int s = 0; s < MVF_STAGES - 1; ++s) {
    if (s < nslab) stage(s);
    commit();
  }
  uint64_t acc[RW * NT / 2];  // pairs of fp32: [token][pair of rows]
#pragma unroll
  for (int i = 0; i < RW * NT / 2; ++i) acc[i] = 0ull;
  for (int slab = 0; slab < nslab; ++slab) {
    asm volatile("cp.async.wait_group %0;" ::"n"(MVF_STAGES - 2) : "memory");
    __syncthreads();  // the slab is there for every thread, and the stage refilled next was read by all
    if (slab + MVF_STAGES - 1 < nslab) stage(slab + MVF_STAGES - 1);
    commit();
    const u8* s = smem + (slab % MVF_STAGES) * T::STAGE;
    const u8* sw = s + wr * RW * 512 + 16 * lane;
    const u8* sx = s + T::ROWS * 512 + wt * NT * T::XB + 16 * lane;
    uint64_t f[RW / 2][VE];  // rows 2q and 2q + 1 side by side
#pragma unroll
    for (int q = 0; q < RW / 2; ++q) {
      float f0[8], f1[8];
      dense_vec<TYPE>(*(const uint4*)(sw + 2 * q * 512), f0);
      dense_vec<TYPE>(*(const uint4*)(sw + (2 * q + 1) * 512), f1);
#pragma unroll
      for (int k = 0; k < VE; ++k) asm("mov.b64 %0, {%1, %2};" : "=l"(f[q][k]) : "f"(f0[k]), "f"(f1[k]));
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      float xv[8];
      *(float4*)xv = *(const float4*)(sx + t * T::XB);
      if constexpr (VE == 8) *(float4*)(xv + 4) = *(const float4*)(sx + t * T::XB + 512);
#pragma unroll
      for (int k = 0; k < VE; ++k) {
        uint64_t x2;
        asm("mov.b64 %0, {%1, %1};" : "=l"(x2) : "f"(xv[k]));
#pragma unroll
        for (int q = 0; q < RW / 2; ++q)  // each half rounds as the scalar instruction does
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[t * (RW / 2) + q]) : "l"(f[q][k]), "l"(x2));
      }
    }
  }
  float sum[RW * NT];  // [token][row]
#pragma unroll
  for (int i = 0; i < RW * NT / 2; ++i) asm("mov.b64 {%0, %1}, %2;" : "=f"(sum[2 * i]), "=f"(sum[2 * i + 1]) : "l"(acc[i]));
  // lanes meet: after the exchange at distance O a lane holds the sums whose index has its bit O's value in that place
#pragma unroll
  for (int o = 16, half = RW * NT / 2; o > 0; o >>= 1, half >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float give = up ? sum[i] : sum[i + half], keep = up ? sum[i + half] : sum[i];
      sum[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  constexpr int PER = RW * NT / 32;  // sums a lane is left with: those at PER * LANE ..
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int at = PER * lane + i, q = at % RW;
    const long long t = t0 + wt * NT + at / RW;
    const int r = r0 + wr * RW + q;
    if (t < n && r < rows) y[t * y_stride + r] = sum[i];
  }
}

template <int TYPE, int RW, int NT, int WR, int WT>
static int mm_dense_launch(const u8* w, int rows, int cols, const float* x, float* y, int n, long long ys, cudaStream_t st) {
  typedef MvfTile<TYPE, RW, NT, WR, WT> T;
  const void* k = (const void*)mm_dense_kernel<TYPE, RW, NT, WR, WT>;
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM);
  if (e != cudaSuccess) return cuda_fail(e);
  void* args[] = {&w, &rows, &cols, &x, &y, &n, &ys};
  return launch_kernel(k, dim3((unsigned)((rows + T::ROWS - 1) / T::ROWS), (unsigned)((n + T::TOKS - 1) / T::TOKS)), dim3(32 * WR * WT), T::SMEM,
                       args, st);
}
// Tiles of 32 x 32 once they fill the SMs; before that 8 x 16 of two warps, which is where a small chunk still reaches every SM.
template <int TYPE>
static int mm_dense(const u8* w, int rows, int cols, const float* x, float* y, int n, long long ys, cudaStream_t st) {
  if ((long long)((rows + 31) / 32) * ((n + 31) / 32) >= 148) return mm_dense_launch<TYPE, 8, 16, 4, 2>(w, rows, cols, x, y, n, ys, st);
  return mm_dense_launch<TYPE, 8, 8, 1, 2>(w, rows, cols, x, y, n, ys, st);
}

template <int RW>
static const void* mv_dense_fn(int type) {
  return type == ILL_F32 ? (const void*)mv_dense_kernel<ILL_F32, RW>
         : type == ILL_F16 ? (const void*)mv_dense_kernel<ILL_F16, RW> : (const void*)mv_dense_kernel<ILL_BF16, RW>;
}

}  // namespace ill

using namespace ill;

extern "C" int ill_mv_dense(int type, ill_dptr w, int rows, int cols, ill_dptr x, ill_dptr y, int n, int64_t y_stride,
                            ill_stream stream) {
  if ((type != ILL_F32 && type != ILL_F16 && type != ILL_BF16) || rows <= 0 || cols <= 0 || n < 1 || n > 65535 * MVF_MAXN || !w || !x ||
      !y || y_stride < rows)
    return ILL_ERR_ARG;
  const int eb = type == ILL_F32 ? 4 : 2;
  if ((w & (eb - 1)) || (x & 3) || (y & 3)) return ILL_ERR_ALIGN;
  const int ve = 16 / eb;
  int vec_ok = !(w & 15) && !(x & 15) && cols % ve == 0 && ((long long)cols * eb) % 16 == 0 && ((long long)cols * 4) % 16 == 0;
  const u8* wp = (const u8*)(uintptr_t)w;
  const float* xp = (const float*)(uintptr_t)x;
  float* yp = (float*)(uintptr_t)y;
  long long ys = y_stride;
  void* args[] = {&wp, &rows, &cols, &xp, &yp, &n, &ys, &vec_ok};
  if (n == 1 && vec_ok) {
    void* one[] = {&wp, &rows, &cols, &xp, &yp};
    const void* k = type == ILL_F32 ? (const void*)mv_dense_one_kernel<ILL_F32> : type == ILL_F16 ? (const void*)mv_dense_one_kernel<ILL_F16>
                                                                                                  : (const void*)mv_dense_one_kernel<ILL_BF16>;
    return launch_kernel(k, dim3((unsigned)((rows + 1) / 2)), dim3(64), 0, one, (cudaStream_t)stream);
  }
  if (n > 4 && vec_ok && (n + 7) / 8 <= 65535) {
    cudaStream_t st = (cudaStream_t)stream;
    return type == ILL_F32 ? mm_dense<ILL_F32>(wp, rows, cols, xp, yp, n, ys, st)
           : type == ILL_F16 ? mm_dense<ILL_F16>(wp, rows, cols, xp, yp, n, ys, st) : mm_dense<ILL_BF16>(wp, rows, cols, xp, yp, n, ys, st);
  }
  const int rw = n > MVF_MAXN ? 4 : 1;  // (two to four tokens; rows or activations that 16-byte loads cannot take)
  const void* k = rw == 4 ? mv_dense_fn<4>(type) : mv_dense_fn<1>(type);
  return launch_kernel(k, dim3((unsigned)((rows + 8 * rw - 1) / (8 * rw)), (unsigned)((n + MVF_MAXN - 1) / MVF_MAXN)), dim3(256), 0, args,
                       (cudaStream_t)stream);
}
