// float32 products on the bfloat16 tensor-core instruction (mma.sync m16n8k16) without a loss of precision.
//
// A float32 number has 24 bits of mantissa and a bfloat16 has 8, so x = hi + mid + lo with three bfloat16 numbers, each the
// nearest one to what the ones before it leave (the differences are exact).  A product of two such numbers is the sum of the
// six products of terms down to 2^-16 of the largest; the other three are below 2^-25 of it.  Where an operand is bfloat16
// as stored it is one term and the product three.
#pragma once

#include "common.cuh"

__device__ __forceinline__ unsigned ms_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ms_mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ms_ldm4(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ms_ldm4t(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ms_copy16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void ms_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ms_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ unsigned ms_pack(float x, float y) {      // x in the low half
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ float ms_lo(unsigned p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float ms_hi(unsigned p) { return __uint_as_float(p & 0xffff0000u); }

// two neighbours as three packed pairs of bfloat16
__device__ __forceinline__ void ms_split(float x, float y, unsigned& p0, unsigned& p1, unsigned& p2) {
  p0 = ms_pack(x, y);
  x -= ms_lo(p0);
  y -= ms_hi(p0);
  p1 = ms_pack(x, y);
  p2 = ms_pack(x - ms_lo(p1), y - ms_hi(p1));
}

// The instruction cuts its running sum off instead of rounding it, so a chain of such sums loses a bit of the last place a
// step (8 steps of 16: 1.2e-6 of the result where float32 multiply-adds lose 1.5e-7).  The leading products of a step are
// therefore summed from zero and added with a rounded addition.
//
// d[i] + small[i] += a b[i] for N tiles, a in NA (1 or 3) terms and the b's in NB: the leading products into d, the others,
// 2^-8 of them and less, into chains of their own.  Term by term over the tiles, so that no two neighbouring instructions
// wait for one another.  b[i][term][2].
template <int N, int NA, int NB>
__device__ __forceinline__ void ms_terms(float (*d)[4], float (*small)[4], const unsigned (&a)[NA][4],
                                         const unsigned (&b)[N][NB][2]) {
  constexpr int A1 = NA > 1 ? 1 : 0, A2 = NA - 1, B1 = NB > 1 ? 1 : 0, B2 = NB - 1;
  if (NB == 3) {
#pragma unroll
    for (int i = 0; i < N; ++i) ms_mma(small[i], a[0], b[i][B2][0], b[i][B2][1]);
  }
  if (NA == 3 && NB == 3) {
#pragma unroll
    for (int i = 0; i < N; ++i) ms_mma(small[i], a[A1], b[i][B1][0], b[i][B1][1]);
  }
  if (NA == 3) {
#pragma unroll
    for (int i = 0; i < N; ++i) ms_mma(small[i], a[A2], b[i][0][0], b[i][0][1]);
  }
  if (NB == 3) {
#pragma unroll
    for (int i = 0; i < N; ++i) ms_mma(small[i], a[0], b[i][B1][0], b[i][B1][1]);
  }
  if (NA == 3) {
#pragma unroll
    for (int i = 0; i < N; ++i) ms_mma(small[i], a[A1], b[i][0][0], b[i][0][1]);
  }
  float t[N][4];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    t[i][0] = t[i][1] = t[i][2] = t[i][3] = 0.f;
    ms_mma(t[i], a[0], b[i][0][0], b[i][0][1]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) d[i][j] += t[i][j];
}
// NB terms of two neighbouring tiles (16 columns) of a b operand: `plane` bytes from one term to the next
template <int NB, bool TRANS>
__device__ __forceinline__ void ms_load_b(unsigned (*b)[NB][2], unsigned addr, unsigned plane) {
#pragma unroll
  for (int p = 0; p < NB; ++p) {
    unsigned r[4];
    if (TRANS) ms_ldm4t(r, addr + p * plane);
    else ms_ldm4(r, addr + p * plane);
    b[0][p][0] = r[0];
    b[0][p][1] = r[1];
    b[1][p][0] = r[2];
    b[1][p][1] = r[3];
  }
}
