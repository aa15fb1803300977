// What the recurrences by chunks of 64 tokens share (chunk_scan.cu, delta_chunks.cu).
#pragma once

#include <atomic>

#include "mma_split.cuh"

#define CS_C 64
#define CS_THREADS 256

// the entry and the chunk of work item `item`; false: there is no such item.  Every warp asks for itself.
__device__ __forceinline__ bool cs_item(int item, const int* __restrict__ cu_q, int E, int& e, int& chunk) {
  const int lane = threadIdx.x & 31;
  int base = 0;
  for (int e0 = 0; e0 < E; e0 += 32) {
    const int j = e0 + lane;
    const int mine = j < E ? (cu_q[j + 1] - cu_q[j] + CS_C - 1) / CS_C : 0;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, base + incl > item);
    if (hit) {
      const int l = __ffs(hit) - 1;
      e = e0 + l;
      chunk = item - base - __shfl_sync(0xffffffffu, incl - mine, l);
      return true;
    }
    base += __shfl_sync(0xffffffffu, incl, 31);
  }
  return false;
}
// the first work item of entry e
__device__ __forceinline__ int cs_first_item(int e, const int* __restrict__ cu_q) {
  const int lane = threadIdx.x & 31;
  int n = 0;
  for (int j = lane; j < e; j += 32) n += (cu_q[j + 1] - cu_q[j] + CS_C - 1) / CS_C;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  return n;
}

// products of a chunk's decays, by one warp (lane l: tokens l and l + 32; tokens behind the end have decay 1):
// pre[t] = a_0 ... a_t, suf[t] = a_(t+1) ... a_63.  Returns pre[63].  Float64, rounded once: with one decay a head every chunk
// multiplies the state by the same number, and its error would add up over the chunks (6e-7 of the state after 32).
__device__ __forceinline__ float cs_products(float a_lo, float a_hi, float* pre, float* suf) {
  const int lane = threadIdx.x & 31;
  double f0 = a_lo, f1 = a_hi, b0 = a_lo, b1 = a_hi;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double u0 = __shfl_up_sync(0xffffffffu, f0, o), u1 = __shfl_up_sync(0xffffffffu, f1, o);
    const double d0 = __shfl_down_sync(0xffffffffu, b0, o), d1 = __shfl_down_sync(0xffffffffu, b1, o);
    if (lane >= o) {
      f0 *= u0;
      f1 *= u1;
    }
    if (lane + o < 32) {
      b0 *= d0;
      b1 *= d1;
    }
  }
  const double first = __shfl_sync(0xffffffffu, f0, 31), second = __shfl_sync(0xffffffffu, b1, 0);
  const double n0 = __shfl_down_sync(0xffffffffu, b0, 1), n1 = __shfl_down_sync(0xffffffffu, b1, 1);
  if (pre != nullptr) {
    pre[lane] = (float)f0;
    pre[lane + 32] = (float)(first * f1);
  }
  if (suf != nullptr) {
    suf[lane] = (float)(lane < 31 ? n0 * second : second);
    suf[lane + 32] = lane < 31 ? (float)n1 : 1.f;
  }
  return (float)(first * second);
}

// G(t, s) = a_(s+1) ... a_t for s <= t (0 behind): the product of a run is made of the products of runs of 1, 2, 4 ... 32
// tokens that end where the rest begins (`runs` [6][64], made by one warp; av[t] is token t's decay), in float64 and
// rounded once.
__device__ __forceinline__ void cs_runs(const float* av, double* runs) {
  const int lane = threadIdx.x & 31;           // (lane l keeps the runs that end at tokens l and l + 32)
  double r0 = av[lane], r1 = av[lane + 32];
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    runs[j * CS_C + lane] = r0;
    runs[j * CS_C + lane + 32] = r1;
    const int o = 1 << j;      // the run of 2^j tokens that ends 2^j tokens earlier
    if (o < 32) {
      const double u0 = __shfl_up_sync(0xffffffffu, r0, o), u1 = __shfl_up_sync(0xffffffffu, r1, o);
      const double w0 = __shfl_sync(0xffffffffu, r0, (lane - o) & 31);
      r1 *= lane >= o ? u1 : w0;
      if (lane >= o) r0 *= u0;
    }
  }
}
__device__ __forceinline__ float cs_gap(const double* runs, int t, int s) {
  const int gap = t - s;
  if (gap < 0) return 0.f;
  double p = 1.0;
  int end = t;
#pragma unroll
  for (int j = 0; j < 6; ++j)
    if ((gap >> j) & 1) {
      p *= runs[j * CS_C + end];
      end -= 1 << j;
    }
  return (float)p;
}

// n rows (the rest of 64: zeros) of W numbers at `src`, asked for (`ask`: all of a thread's loads are on their way at once)
// and later put into shared memory as bfloat16 terms (`put`: one as stored, or three of float32, 64 rows of PITCH numbers a term)
template <typename T, int W, int PITCH, int THREADS>
struct CsTile {
  static constexpr int N = 16 / (int)sizeof(T), PIECES = W / N, ALL = (CS_C * PIECES + THREADS - 1) / THREADS;
  uint4 v[ALL];
  __device__ __forceinline__ void ask(const T* __restrict__ src, long stride, int n) {
#pragma unroll
    for (int j = 0; j < ALL; ++j) {
      const int i = j * THREADS + threadIdx.x, t = i / PIECES, c = (i % PIECES) * N;
      v[j] = make_uint4(0, 0, 0, 0);
      if (t < n) v[j] = *reinterpret_cast<const uint4*>(src + (size_t)t * stride + c);
    }
  }
  __device__ __forceinline__ void put(bf16* dst) const {
#pragma unroll
    for (int j = 0; j < ALL; ++j) {
      const int i = j * THREADS + threadIdx.x, t = i / PIECES, c = (i % PIECES) * N;
      if (CS_C * PIECES % THREADS != 0 && t >= CS_C) break;
      bf16* d = dst + t * PITCH + c;
      if (sizeof(T) == 2) {
        *reinterpret_cast<uint4*>(d) = v[j];
      } else {
        uint2 p0, p1, p2;
        ms_split(__uint_as_float(v[j].x), __uint_as_float(v[j].y), p0.x, p1.x, p2.x);
        ms_split(__uint_as_float(v[j].z), __uint_as_float(v[j].w), p0.y, p1.y, p2.y);
        *reinterpret_cast<uint2*>(d) = p0;
        *reinterpret_cast<uint2*>(d + CS_C * PITCH) = p1;
        *reinterpret_cast<uint2*>(d + 2 * CS_C * PITCH) = p2;
      }
    }
  }
};
template <typename T> __device__ __forceinline__ float4 cs_load4(const T* p);
template <> __device__ __forceinline__ float4 cs_load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 cs_load4<bf16>(const bf16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// One number of the state behind token `last` of a chunk: S <- a S + k (w v) over the tokens 0 .. last, from S (`from` null: 0,
// without the first decay).  k and v point at the number's channel and column in the chunk's first row.
template <typename T, typename A, typename W>
__device__ __forceinline__ float cs_again(const float* from, const T* k, long k_stride, const T* v, long v_stride, int last, A decay,
                                          W scale) {
  float s = 0.f;
  for (int t = 0; t <= last && s == s; ++t) {
    const float x = to_f32<T>(k[(size_t)t * k_stride]) * (to_f32<T>(v[(size_t)t * v_stride]) * scale(t));
    s = t > 0 ? fmaf(decay(t), s, x) : from != nullptr ? fmaf(decay(0), *from, x) : x;
  }
  return s;
}

// lets KERNEL have `bytes` of dynamic shared memory: asked for once a device (the call takes the host about as long as a launch)
template <auto KERNEL> static cudaError_t cs_room(size_t bytes) {
  static std::atomic<unsigned long long> done{0};
  int device = 0;
  cudaError_t rc = cudaGetDevice(&device);
  if (rc != cudaSuccess || (device < 64 && ((done.load() >> device) & 1))) return rc;
  rc = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (rc == cudaSuccess && device < 64) done.fetch_or(1ull << device);
  return rc;
}
