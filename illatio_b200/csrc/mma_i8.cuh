// The legacy tensor-core path for 8-bit integers (mma.sync m16n8k32 / m16n8k16) and the small loads around it,
// shared by the several-token product (mvt.cu) and the dense chunk products (mmd.cu, mm_q8_i8.cu).
//
// Fragment layout, lane = 4 g + t: A (16 rows x K): a0 = row g, k 4t..4t+3; a1 = row g + 8, same k; for k32 a2 / a3
// the same rows at k + 16.  B (K x 8 columns): b0 = column g, k 4t..4t+3; b1 (k32) at k + 16.  C: c0 / c1 = row g,
// columns 2t / 2t + 1; c2 / c3 = row g + 8.
#pragma once
#include "common.cuh"

namespace ill {

__device__ __forceinline__ void mma_k32(int (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2], bool a_unsigned) {
  if (a_unsigned)
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
  else
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// D = A B with D's registers free of initialization, and free to be scheduled
__device__ __forceinline__ void mma_k32_s8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_k16_u8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a0), "r"(a1), "r"(b0));
}

// four 8 x 16-byte matrices of shared memory -> each lane its four bytes of row lane / 4 of each: lane l gives the
// address of row l % 8 of matrix l / 8.  For a token tile's 64 bytes of quants this is the B fragment of two k32
// (or four k16) steps: r[0], r[1] = b0, b1 of the first k32 step, r[2], r[3] of the second.
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p)));
}

__device__ __forceinline__ void ldsm4_at(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// a 32-bit word at any byte address of shared memory
__device__ __forceinline__ uint32_t lds32u(const u8* p) {
  const uint32_t mis = (uint32_t)(uintptr_t)p & 3u;
  const uint32_t* b = (const uint32_t*)(p - mis);
  return __funnelshift_r(b[0], b[1], 8u * mis);
}
// The same for many words at distances of a multiple of four from one address: the alignment is looked at once.
struct LdsWords {
  const uint32_t* b;
  uint32_t sh;
  __device__ __forceinline__ explicit LdsWords(const u8* p) {
    const uint32_t mis = (uint32_t)(uintptr_t)p & 3u;
    b = (const uint32_t*)(p - mis);
    sh = 8u * mis;
  }
  __device__ __forceinline__ uint32_t operator()(int off) const { return __funnelshift_r(b[off / 4], b[off / 4 + 1], sh); }
};
// Words of a row at multiples of four bytes from an address: one that lies on a word (AL4), or on any two bytes.
template <bool AL4> struct RowWords;
template <> struct RowWords<false> : LdsWords {
  __device__ __forceinline__ explicit RowWords(const u8* p) : LdsWords(p) {}
};
template <> struct RowWords<true> {
  const u8* p;
  __device__ __forceinline__ explicit RowWords(const u8* q) : p(q) {}
  __device__ __forceinline__ uint32_t operator()(int off) const { return *(const uint32_t*)(p + off); }
};
__device__ __forceinline__ float ldh(const u8* p) { return h2f(*(const u16*)p); }  // p is 2-byte aligned

__device__ __forceinline__ void mma_k16_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0, bool b_unsigned) {
  if (b_unsigned)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0));
}

// 16 / 4 bytes global -> shared, asynchronously; a group of them is waited for with cp.async.wait_group
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// A row segment's bytes SRC .. SRC + LEN -> shared memory by the four lanes T = 0..3 of a quad: the 16-byte aligned span
// that covers them, NCH chunks at most (the segment starts SRC % 16 bytes into it).  One instruction brings 64 bytes of
// each of eight rows; a bulk copy a segment costs its lane a turn of its own through the copy unit.
template <int NCH>
__device__ __forceinline__ void copy_segment(u8* dst, const u8* src, uint32_t len, int t) {
  const u8* a = (const u8*)((uintptr_t)src & ~(uintptr_t)15) + 16 * t;
  const u8* end = src + len;
#pragma unroll
  for (int k = 0; k < (NCH + 3) / 4; ++k)
    if (a + 64 * k < end) cp_async16(dst + 16 * t + 64 * k, a + 64 * k);
}

// The same to the address DST in shared memory, this lane's first piece's (T's).
template <int NCH>
__device__ __forceinline__ void copy_segment_at(uint32_t dst, const u8* src, uint32_t len, int t) {
  const uint32_t lo = (uint32_t)(uintptr_t)src & 15u, end = lo + len;
  const u8* a = src - lo + 16 * t;
#pragma unroll
  for (int k = 0; k < (NCH + 3) / 4; ++k)
    if (16u * t + 64u * k < end) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 64 * k), "l"(a + 64 * k) : "memory");
}

// get_scale_min_k4 (src/kquant.lisp:64-72) for group J of the 12 packed bytes at Q
__device__ __forceinline__ void scale_min_k4(const u8* q, int j, int& sc, int& mn) {
  if (j < 4) { sc = q[j] & 63; mn = q[j + 4] & 63; }
  else { sc = (q[j + 4] & 0xF) | ((q[j - 4] >> 6) << 4); mn = (q[j + 4] >> 4) | ((q[j] >> 6) << 4); }
}

}  // namespace ill
