// quant.cu -- activation quantizers and rows-as-floats.
//
// The quantizers reproduce the reference's CPU routines bit for bit
// (QUANTIZE-Q8! src/tensor.lisp:245-262, QUANTIZE-Q8K! src/kquant.lisp:130-167):
// IEEE division and round-half-even conversion, no fused multiply-add, the
// first of equal maxima wins.  They are what lets the products on the device
// follow the CPU kernels instead of the reference's own CUDA kernels, which feed
// K-quants Q8_0 blocks (src/cuda/kquant.cu:3-14).
#include "formats.cuh"
#include "iq2xxs_tables.cuh"
#include "quantdev.cuh"
#include "host.h"

namespace ill {

__global__ void __launch_bounds__(256) quant_q8_0_kernel(const float* __restrict__ x, i8* __restrict__ xq,
                                                         float* __restrict__ xs, int* __restrict__ xsum,
                                                         long long nblocks, int f16_scale) {
  pdl_launch_dependents();
  pdl_wait();
  const long long b = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (b >= nblocks) return;
  quant_block_q8_0(x[b * 32 + lane], lane, b, xq, xs, xsum, f16_scale);
}

// Four values of a Q8_0 block in each of its eight lanes (all 32 lanes take part; IN: the lane has values): the block's
// maximum takes three shuffles for four blocks where a value a lane takes five for one, its bytes leave as a word a lane.
// The same bits (a maximum and a sum of whole numbers do not depend on the order).  I4 numbers the fours from XQ's start.
__device__ __forceinline__ void quant_four_q8_0(float4 v, bool in, long long i4, uint32_t* xq, float* xs, int* xsum, int f16_scale) {
  float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float d = __fdiv_rn(amax, 127.0f);
  const float id = d == 0.0f ? 0.0f : __fdiv_rn(1.0f, d);
  const int q[4] = {__float2int_rn(__fmul_rn(v.x, id)), __float2int_rn(__fmul_rn(v.y, id)), __float2int_rn(__fmul_rn(v.z, id)),
                    __float2int_rn(__fmul_rn(v.w, id))};
  int t = q[0] + q[1] + q[2] + q[3];
  if (xsum) {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  if (!in) return;
  xq[i4] = (uint32_t)(q[0] & 0xff) | (uint32_t)(q[1] & 0xff) << 8 | (uint32_t)(q[2] & 0xff) << 16 | (uint32_t)(q[3] & 0xff) << 24;
  if ((threadIdx.x & 7) == 0) {
    xs[i4 >> 3] = f16_scale ? __half2float(__float2half_rn(d)) : d;
    if (xsum) xsum[i4 >> 3] = t;
  }
}

// quant_q8_0_kernel where X and XQ lie on 16- and 4-byte boundaries.  A value a lane was bound by the issue of its divisions
// and shuffles (777 x 4864 values 15.6 us, 4096 x 4096 68); four a lane are bound by memory (4.6 and 18 us).
__global__ void __launch_bounds__(256) quant_q8_0_vec_kernel(const float4* __restrict__ x, uint32_t* __restrict__ xq,
                                                             float* __restrict__ xs, int* __restrict__ xsum,
                                                             long long nblocks, int f16_scale) {
  pdl_launch_dependents();
  pdl_wait();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const bool in = i < 8 * nblocks;
  const float4 v = in ? x[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  quant_four_q8_0(v, in, i, xq, xs, xsum, f16_scale);
}

// A warp a super-block; lane l holds elements 8l .. 8l+7.  F16: also the block's fp16 forms (XH, XE).
template <bool F16>
__global__ void __launch_bounds__(256) quant_q8_k_kernel(const float* __restrict__ x, i8* __restrict__ xq,
                                                         float* __restrict__ xd, int16_t* __restrict__ bsums,
                                                         long long nblocks, __half* __restrict__ xh, __half* __restrict__ xe) {
  pdl_launch_dependents();
  pdl_wait();
  const long long b = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (b >= nblocks) return;
  const float4 v0 = ((const float4*)(x + b * 256))[2 * lane], v1 = ((const float4*)(x + b * 256))[2 * lane + 1];
  const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
  if constexpr (F16) quant_block_q8_k_f16(v, lane, b, xq, xd, bsums, xh, xe);
  else quant_block_q8_k(v, lane, b, xq, xd, bsums);
}

// RMSNORM! (src/model.lisp:205-216) fused with the activation quantizer, as the reference's rmsnorm_q8
// launch is (src/cuda/dense.cu:144-160, RMSNORM-Q8 src/cuda-dense.lisp:260-264): the squares (rounded to
// float) summed in double, scale = 1 / sqrt(float(sum / d + eps)), value = (x * scale) * w, then the
// blocks quantized as the stand-alone quantizers do.  Grid (slices, rows): every CTA of a row works the
// row's scale out for itself (the row comes from L2) and takes a slice of its blocks, so that one token's
// norm is not one CTA's serial work.  The double sum is taken in the order quantdev.cuh fixes, not in the
// CPU loop's; the two agree until the float the sum is rounded to sits within 1e-16 of a rounding boundary.
// Bound by latency: the norm's weights are on their way to L2 before the kernel waits for the one before it (which may have
// written them; more rows than SMs find them there), a warp asks for four of its groups and its first block's values at once,
// and a few rows are spread over their blocks too (in a graph of norms, before and now: 16 rows of 2560 3.8 -> 2.6 us, 4 of
// 5120 5.1 -> 2.8, one of 2560 3.0 -> 2.4, 512 of 5120 13.9 -> 6.8).  VEC: Q8_0 blocks by four values a lane (X, W, H and XQ
// aligned for it).
template <int K8K, bool F16, bool VEC>
__global__ void __launch_bounds__(256) rmsnorm_q8_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                         float* __restrict__ h, i8* __restrict__ xq, float* __restrict__ xs,
                                                         void* __restrict__ xsum, int d, float eps, int f16_scale,
                                                         __half* __restrict__ xh, __half* __restrict__ xe) {
  __shared__ double group_s[RMS_MAX_GROUPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // a unit is a warp's turn: a Q8_K block, a Q8_0 block, or (VEC) four Q8_0 blocks, the last unit perhaps fewer
  constexpr int BW = K8K ? 256 : VEC ? 128 : 32, VL = BW / 32;  // a unit's values, a lane's
  const int nb = (d + BW - 1) / BW, b0 = blockIdx.x * 8 + warp;
  float wv[VL], x0[VL];  // of the warp's first block
  auto load = [&](const float* src, int b, float (&v)[VL]) {
    if constexpr (K8K) rms_load8<false>(src, d, b * 256 + 8 * lane, v);
    else if constexpr (VEC) {
      const float4 f = b * 128 + 4 * lane < d ? ((const float4*)src)[b * 32 + lane] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else v[0] = src[b * 32 + lane];
  };
  if (gridDim.y <= 148 && b0 < nb && b0 * BW + VL * lane < d) prefetch_l2(w + b0 * BW + VL * lane);
  pdl_launch_dependents();
  pdl_wait();
  w = after_wait(w);
  const long long base = (long long)blockIdx.y * d;
  const float* xr = after_wait(x + base);
  if (!K8K && b0 < nb) load(w, b0, wv);
  if (b0 < nb) load(xr, b0, x0);
  const int ng = (d + 255) / 256;
  for (int g0 = warp; g0 < ng; g0 += 32) {
    float v[4][8];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (g0 + 8 * k < ng) rms_load8<false>(xr, d, (g0 + 8 * k) * 256 + 8 * lane, v[k]);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (g0 + 8 * k < ng) {
        const double s = rms_group_sum(v[k]);
        if (lane == 0) group_s[g0 + 8 * k] = s;
      }
  }
  if (K8K && b0 < nb) load(w, b0, wv);  // (eight registers a lane less while the row's sum is taken)
  __syncthreads();
  const float sc = rms_scale(rms_total(group_s, ng, lane), d, eps);
  for (int b = b0; b < nb; b += gridDim.x * 8) {
    if (b != b0) { load(w, b, wv); load(xr, b, x0); }
    float v[VL];
#pragma unroll
    for (int j = 0; j < VL; ++j) v[j] = __fmul_rn(__fmul_rn(x0[j], sc), wv[j]);
    const long long at = base + (long long)b * BW + VL * lane;  // the lane's first value
    if constexpr (VEC) {
      const bool in = b * 128 + 4 * lane < d;
      const float4 f = make_float4(v[0], v[1], v[2], v[3]);
      if (h && in) *(float4*)(h + at) = f;
      quant_four_q8_0(f, in, at / 4, (uint32_t*)xq, xs, (int*)xsum, f16_scale);
    } else {
      if (h)
#pragma unroll
        for (int j = 0; j < VL; ++j) h[at + j] = v[j];
      const long long gb = base / BW + b;
      if constexpr (!K8K) quant_block_q8_0(v[0], lane, gb, xq, xs, (int*)xsum, f16_scale);
      else if constexpr (F16) quant_block_q8_k_f16(v, lane, gb, xq, xs, (int16_t*)xsum, xh, xe);
      else quant_block_q8_k(v, lane, gb, xq, xs, (int16_t*)xsum);
    }
  }
}

template <int FMT>
__global__ void __launch_bounds__(256) dequant_rows_kernel(const u8* __restrict__ w, int cols, long long row_bytes,
                                                           const int* __restrict__ row_ids, long long first_row,
                                                           float* __restrict__ out) {
  const int i = blockIdx.x;
  const long long row = row_ids ? (long long)row_ids[i] : first_row + i;
  const u8* rp = w + row * row_bytes;
  for (int c = blockIdx.y * 256 + threadIdx.x; c < cols; c += gridDim.y * 256)
    out[(long long)i * cols + c] = dequant_weight<FMT>(rp, c, ill_iq2xxs_grid, ill_ksigns_iq2xs);
}

}  // namespace ill

using namespace ill;

extern "C" int ill_quant_q8_0(ill_dptr x, ill_dptr xq, ill_dptr xs, ill_dptr xsum, int64_t nblocks, int f16_scale,
                              ill_stream stream) {
  if (nblocks < 0 || !x || !xq || !xs) return ILL_ERR_ARG;
  if ((x & 3) || (xs & 3) || (xsum & 3)) return ILL_ERR_ALIGN;
  if (nblocks == 0) return ILL_OK;
  const float* xp = (const float*)(uintptr_t)x;
  i8* qp = (i8*)(uintptr_t)xq;
  float* sp = (float*)(uintptr_t)xs;
  int* sump = (int*)(uintptr_t)xsum;
  long long nb = nblocks;
  void* args[] = {&xp, &qp, &sp, &sump, &nb, &f16_scale};
  if (((x & 15) | (xq & 3)) == 0)
    return launch_kernel((const void*)quant_q8_0_vec_kernel, dim3((unsigned)((nblocks + 31) / 32)), dim3(256), 0, args,
                         (cudaStream_t)stream);
  return launch_kernel((const void*)quant_q8_0_kernel, dim3((unsigned)((nblocks + 7) / 8)), dim3(256), 0, args,
                       (cudaStream_t)stream);
}

static int quant_q8_k_launch(ill_dptr x, ill_dptr xq, ill_dptr xd, ill_dptr bsums, int64_t nblocks, ill_dptr xh, ill_dptr xe,
                             ill_stream stream) {
  if (nblocks < 0 || !x || !xq || !xd || !bsums) return ILL_ERR_ARG;
  if ((x & 15) || (xq & 7) || (xd & 3) || (bsums & 1) || (xh & 15) || (xe & 15)) return ILL_ERR_ALIGN;
  if (nblocks == 0) return ILL_OK;
  const float* xp = (const float*)(uintptr_t)x;
  i8* qp = (i8*)(uintptr_t)xq;
  float* dp = (float*)(uintptr_t)xd;
  int16_t* bp = (int16_t*)(uintptr_t)bsums;
  __half *hp = (__half*)(uintptr_t)xh, *ep = (__half*)(uintptr_t)xe;
  long long nb = nblocks;
  void* args[] = {&xp, &qp, &dp, &bp, &nb, &hp, &ep};
  const void* k = xh ? (const void*)quant_q8_k_kernel<true> : (const void*)quant_q8_k_kernel<false>;
  return launch_kernel(k, dim3((unsigned)((nblocks + 7) / 8)), dim3(256), 0, args, (cudaStream_t)stream);
}

extern "C" int ill_quant_q8_k(ill_dptr x, ill_dptr xq, ill_dptr xd, ill_dptr bsums, int64_t nblocks,
                              ill_stream stream) {
  return quant_q8_k_launch(x, xq, xd, bsums, nblocks, 0, 0, stream);
}

extern "C" int ill_quant_q8_k_f16(ill_dptr x, ill_dptr xq, ill_dptr xd, ill_dptr bsums, ill_dptr xh, ill_dptr xe, int64_t nblocks,
                                  ill_stream stream) {
  if (!xh || !xe) return ILL_ERR_ARG;
  return quant_q8_k_launch(x, xq, xd, bsums, nblocks, xh, xe, stream);
}

static int rmsnorm_q8_launch(int kind, ill_dptr x, ill_dptr w, ill_dptr h, ill_dptr xq, ill_dptr xs, ill_dptr xsum, int d, float eps,
                             int64_t n, int f16_scale, ill_dptr xh, ill_dptr xe, ill_stream stream);

extern "C" int ill_rmsnorm_q8(int kind, ill_dptr x, ill_dptr w, ill_dptr h, ill_dptr xq, ill_dptr xs, ill_dptr xsum, int d,
                              float eps, int64_t n, int f16_scale, ill_stream stream) {
  return rmsnorm_q8_launch(kind, x, w, h, xq, xs, xsum, d, eps, n, f16_scale, 0, 0, stream);
}

extern "C" int ill_rmsnorm_q8k_f16(ill_dptr x, ill_dptr w, ill_dptr h, ill_dptr xq, ill_dptr xs, ill_dptr xsum, ill_dptr xh, ill_dptr xe,
                                   int d, float eps, int64_t n, ill_stream stream) {
  if (!xh || !xe || (xh & 15) || (xe & 15)) return ILL_ERR_ARG;
  return rmsnorm_q8_launch(1, x, w, h, xq, xs, xsum, d, eps, n, 0, xh, xe, stream);
}

static int rmsnorm_q8_launch(int kind, ill_dptr x, ill_dptr w, ill_dptr h, ill_dptr xq, ill_dptr xs, ill_dptr xsum, int d, float eps,
                             int64_t n, int f16_scale, ill_dptr xh, ill_dptr xe, ill_stream stream) {
  const int bw = kind == 1 ? 256 : 32;
  if ((kind != 0 && kind != 1) || d <= 0 || d % bw || n < 0 || n > 65535 || !x || !w || !xq || !xs || (kind == 1 && !xsum))
    return ILL_ERR_ARG;
  if (d > 256 * RMS_MAX_GROUPS) return ILL_ERR_TOO_LARGE;
  if ((x & 3) || (w & 3) || (h & 3) || (xs & 3) || (xsum & (kind == 1 ? 1 : 3)) || (kind == 1 && (xq & 7))) return ILL_ERR_ALIGN;
  if (n == 0) return ILL_OK;
  const float* xp = (const float*)(uintptr_t)x;
  const float* wp = (const float*)(uintptr_t)w;
  float* hp = (float*)(uintptr_t)h;
  i8* qp = (i8*)(uintptr_t)xq;
  float* sp = (float*)(uintptr_t)xs;
  void* bp = (void*)(uintptr_t)xsum;
  __half *fhp = (__half*)(uintptr_t)xh, *fep = (__half*)(uintptr_t)xe;
  void* args[] = {&xp, &wp, &hp, &qp, &sp, &bp, &d, &eps, &f16_scale, &fhp, &fep};
  // few rows are spread over their blocks, as far as two CTAs an SM (148) go; many rows take a CTA each, and so do rows that
  // are normalized in place: a CTA of a row that is shared would still be reading what another has written
  const bool vec = kind == 0 && ((x | w | h) & 15) == 0 && (xq & 3) == 0;
  const uint64_t bytes = 4ull * (uint64_t)d * (uint64_t)n;
  const bool in_place = h && h < x + bytes && x < h + bytes;
  const int nb = vec ? (d + 127) / 128 : d / bw, most = n < 296 && !in_place ? (int)(296 / n) : 1;
  const unsigned slices = (unsigned)((nb + 7) / 8 < most ? (nb + 7) / 8 : most);
  const void* k = kind == 1 ? (xh ? (const void*)rmsnorm_q8_kernel<1, true, false> : (const void*)rmsnorm_q8_kernel<1, false, false>)
                            : vec ? (const void*)rmsnorm_q8_kernel<0, false, true> : (const void*)rmsnorm_q8_kernel<0, false, false>;
  return launch_kernel(k, dim3(slices, (unsigned)n), dim3(256), 0, args, (cudaStream_t)stream);
}

extern "C" int ill_dequant_rows(int fmt, ill_dptr w, int cols, ill_dptr row_ids, int64_t first_row, int nrows,
                                ill_dptr out, ill_stream stream) {
  const int bw = fmt_block_weights(fmt);
  if (!bw || cols <= 0 || cols % bw || nrows < 0 || !w || !out || first_row < 0) return ILL_ERR_ARG;
  if ((out & 3) || (row_ids & 3)) return ILL_ERR_ALIGN;
  if (nrows == 0) return ILL_OK;
  const long long row_bytes = (long long)(cols / bw) * fmt_block_bytes(fmt);
  const u8* wp = (const u8*)(uintptr_t)w;
  const int* ids = (const int*)(uintptr_t)row_ids;
  float* op = (float*)(uintptr_t)out;
  dim3 grid(nrows, (cols + 2047) / 2048 > 0 ? (cols + 2047) / 2048 : 1);
  cudaStream_t st = (cudaStream_t)stream;
  switch (fmt) {
    case ILL_Q8_0: dequant_rows_kernel<ILL_Q8_0><<<grid, 256, 0, st>>>(wp, cols, row_bytes, ids, first_row, op); break;
    case ILL_Q4_K: dequant_rows_kernel<ILL_Q4_K><<<grid, 256, 0, st>>>(wp, cols, row_bytes, ids, first_row, op); break;
    case ILL_Q6_K: dequant_rows_kernel<ILL_Q6_K><<<grid, 256, 0, st>>>(wp, cols, row_bytes, ids, first_row, op); break;
    case ILL_Q2_K: dequant_rows_kernel<ILL_Q2_K><<<grid, 256, 0, st>>>(wp, cols, row_bytes, ids, first_row, op); break;
    case ILL_IQ2_XXS:
      dequant_rows_kernel<ILL_IQ2_XXS><<<grid, 256, 0, st>>>(wp, cols, row_bytes, ids, first_row, op);
      break;
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ILL_OK : cuda_fail(e);
}
