// Matrix-state recurrences of prompt portions, 64 tokens at a time.
//
// A linear recurrence S_t = a_t S_(t-1) + k_t v_t^T, o_t = S_t^T q_t (linear attention with decay, retention, a
// state-space layer) or its delta-rule form (u_t = beta_t (v_t - (a_t S_(t-1))^T k_t) in the place of v_t) walked token by
// token is bound by its chain: 2,048 tokens took 320 us with 12 heads and 790 us as a delta rule, at 2 % of the chip's
// arithmetic.  Cut into chunks of 64 tokens (C), with G(t, s) = a_(s+1) ... a_t,
//     o_t     = G(t, -) S0^T q_t + sum over s <= t of G(t, s) (q_t . k_s) v_s         S0: the state before the chunk
//     S_end   = G(C, -) S0 + sum over s of k_s (G(C, s) v_s)^T
// the work between two chunks' states is matrix products, and chunks meet only in S0:
//   chunk_write    per (chunk, head, 64 value columns): sum of k_s (G(C, s) v_s)^T
//   chunk_prefix   per (entry, head, part of the state): the states before every chunk, and the record's new state
//   chunk_read     per (chunk, head): the read-outs
// For the delta rule the written values depend on S0.  With L(t, s) = beta_t G(t, s) (k_t . k_s), s < t,
//     (1 + L) U = [beta_t v_t],  (1 + L) W = [beta_t G(t, -) k_t],  u = U - W S0
//   delta_solve    per (chunk, head): U and W by forward substitution, a column a thread
//   delta_walk     per (entry, head, 16 value columns): the chunks in order, two products and no division a chunk; the
//                  state stays in registers (a warp holds an eighth of the key channels)
// and chunk_read takes u for v.  The chain of 2,048 tokens is then 32 products long.
//
// Everything is float32 as in the walk by tokens: decays are running products (a decay that underflows to 0 stays 0,
// nothing is divided), products of float32 numbers are made of bfloat16 terms that hold all 24 bits (mma_split.cuh), and
// operands that are stored as bfloat16 are taken as they are.  A chunk starts where the step's portion does, so the order
// of the sums depends on how a prompt was cut into portions, within rounding.  Infinities have no bfloat16 terms and a
// product with 0 makes NaN of them, so a number that is not finite would show in the chunk's tokens before it, too: a thread
// that finds a state or a read-out not finite makes that number again token by token (`cs_again`), as the walk does.  (The
// delta rule's walk over chunks has NaN in a state where the walk by tokens may still have an infinity.)
//
// Taken for longer portions, key heads of 64 or 128 channels and value heads of a multiple of 64 (delta rule: 64 or 128,
// one decay a head): see `ops.chunked_scan`.
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

// Where the rows of a chunk come from: q, k and v heads of a row a token, or (delta rule) v as blocks of 64 rows.
template <typename T> struct CsRows {
  const T* proj;
  long stride;
  int q_off, k_off, v_off;
  const float* decay;        // one a head, or
  const float* tok_decay;    // one a (token, head) [tokens, H]
  const float* tok_scale;    // a factor on a token's v, or null
  const float* skip;         // one a head: its own v added to a token's read-out, or null
  const float* k_rows;       // delta rule: k in rows of its own (then q in `proj`), same stride
  const float* u;            // delta rule: [items][H][64][dv] in the place of v
  int hpg;                   // heads that read the same q and k
};

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

// The numbers of a thread's that are not finite, again.  (Where operands are float32 as calls of their own: inlined, they took
// the registers of chunk_read from 176 to 255 and 3 us of a delta rule's 277; bfloat16 operands: called, 6 of 125 us.)
// chunk_write: the thread's part of the states, from channel `ch0` and value column `v0` (of all heads') on.
template <typename T, int DK>
__device__ __forceinline__ void cs_write_again(const CsRows<T>& in, float* dst, int base, int n, int h, int H, int ch0, size_t v0) {
  const T* row = in.proj + (size_t)base * in.stride;
  auto decay = [&](int t) { return in.tok_decay ? in.tok_decay[(size_t)(base + t) * H + h] : in.decay[h]; };
  auto scale = [&](int t) { return in.tok_scale ? in.tok_scale[(size_t)(base + t) * H + h] : 1.f; };
#pragma unroll 1
  for (int i = 0; i < DK / 4; ++i) {
    const int col = 8 * ((i >> 1) & 1), ch = (i >> 2) * 8 + (i & 1);
    float* d = dst + col * DK + ch;
    if (!(fabsf(*d) < INFINITY))
      *d = cs_again<T>(nullptr, row + in.k_off + (h / in.hpg) * DK + ch0 + ch, in.stride, row + in.v_off + v0 + col, in.stride, n - 1,
                       decay, scale);
  }
}
// chunk_read: rows t0 and t0 + 8, 16 of every 64 columns
template <typename T, int DK>
__device__ __forceinline__ void cs_read_again(float* out, long out_stride, const T* q, const T* k, long stride, const T* v, long v_stride,
                                           const float* state, const float* av, const float* sc, bool skipped, float skip, int n,
                                           int dv, int t0, int col0) {
  auto decay = [&](int t) { return av[t]; };
  auto scale = [&](int t) { return sc[t]; };
#pragma unroll 1
  for (int i = 0; i < dv / 4; ++i) {
    const int t = t0 + 8 * ((i >> 3) & 1), col = (i >> 4) * 64 + col0 + ((i >> 1) & 3) * 8 + (i & 1);
    if (t >= n) continue;
    float* d = out + (size_t)t * out_stride + col;
    if (fabsf(*d) < INFINITY) continue;
    float a = 0.f;
    for (int ch = 0; ch < DK && a == a; ++ch)
      a = fmaf(cs_again<T>(state + (size_t)col * DK + ch, k + ch, stride, v + col, v_stride, t, decay, scale),
               to_f32<T>(q[(size_t)t * stride + ch]), a);
    *d = skipped ? fmaf(skip, to_f32<T>(v[(size_t)t * v_stride + col]), a) : a;
  }
}

template <int DK, typename... A>
__device__ __noinline__ void cs_write_again_f32(A... a) { cs_write_again<float, DK>(a...); }
template <int DK, typename... A>
__device__ __noinline__ void cs_read_again_f32(A... a) { cs_read_again<float, DK>(a...); }

// ---------------------------------------------------------------------------------------------------------------
// ds[item][h][dv][dk] = sum over the chunk's tokens of (G(C, s) scale_s v_s) k_s^T; gam[item][h] = G(C, -).
// Value columns are the M side (16 of the CTA's 64 a warp, half of the key channels each), tokens the inner dimension.
// ---------------------------------------------------------------------------------------------------------------
template <typename T, int DK>
__global__ void __launch_bounds__(CS_THREADS)
chunk_write_kernel(CsRows<T> in, const int* __restrict__ cu_q, const int* __restrict__ req_slot, int E, int num_slots,
                   float* __restrict__ ds, float* __restrict__ gam, int H, int dv) {
  constexpr int NPL = sizeof(T) == 2 ? 1 : 3;
  constexpr int KP = DK + 8, VP = 72;
  extern __shared__ __align__(16) unsigned char cs_smem[];
  bf16* ks = reinterpret_cast<bf16*>(cs_smem);                 // [NPL][64][KP]
  bf16* vs = ks + NPL * CS_C * KP;                             // [3][64][VP]
  __shared__ float suf[CS_C];
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int item = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * 64;
  int e, chunk;
  if (!cs_item(item, cu_q, E, e, chunk)) return;
  const int slot = req_slot[e];
  if (slot < 0 || slot >= num_slots) return;
  const int base = cu_q[e] + chunk * CS_C, n = min(CS_C, cu_q[e + 1] - base);
  CsTile<T, DK, KP, CS_THREADS> kt_;
  kt_.ask(in.proj + (size_t)base * in.stride + in.k_off + (h / in.hpg) * DK, in.stride, n);
  float4 v[4];
  float w[4];
  {
    const T* src = in.proj + (size_t)base * in.stride + in.v_off + (size_t)h * dv + c0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = j * CS_THREADS + tid, t = i >> 4, c = (i & 15) * 4;
      v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      w[j] = 1.f;
      if (t < n) {
        v[j] = cs_load4<T>(src + (size_t)t * in.stride + c);
        if (in.tok_scale) w[j] = in.tok_scale[(size_t)(base + t) * H + h];
      }
    }
  }
  if (warp == 0) {
    float a[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = lane + 32 * i;
      a[i] = t >= n ? 1.f : in.tok_decay ? in.tok_decay[(size_t)(base + t) * H + h] : in.decay[h];
    }
    const float all = cs_products(a[0], a[1], nullptr, suf);
    if (lane == 0 && blockIdx.z == 0) gam[(size_t)item * H + h] = all;
  }
  kt_.put(ks);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = j * CS_THREADS + tid, t = i >> 4, c = (i & 15) * 4;
    const float f = suf[t];
    uint2 p0, p1, p2;
    ms_split((v[j].x * w[j]) * f, (v[j].y * w[j]) * f, p0.x, p1.x, p2.x);
    ms_split((v[j].z * w[j]) * f, (v[j].w * w[j]) * f, p0.y, p1.y, p2.y);
    bf16* d = vs + t * VP + c;
    *reinterpret_cast<uint2*>(d) = p0;
    *reinterpret_cast<uint2*>(d + CS_C * VP) = p1;
    *reinterpret_cast<uint2*>(d + 2 * CS_C * VP) = p2;
  }
  __syncthreads();
  const int m = lane >> 3, r = lane & 7, rt = (warp & 3) * 16, kc = (warp >> 2) * (DK / 2);
  const unsigned ks_b = ms_smem(ks), vs_b = ms_smem(vs);
  constexpr int NT = DK / 16;
  float acc[NT][4], low[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = low[i][j] = 0.f;
#pragma unroll
  for (int kt = 0; kt < CS_C / 16; ++kt) {
    unsigned a[3][4];
#pragma unroll
    for (int p = 0; p < 3; ++p)
      ms_ldm4t(a[p], vs_b + 2 * ((p * CS_C + kt * 16 + (m >> 1) * 8 + r) * VP + rt + (m & 1) * 8));
#pragma unroll
    for (int nt = 0; nt < NT; nt += 4) {
      unsigned b[4][NPL][2];
      const unsigned at = ks_b + 2 * ((kt * 16 + (m & 1) * 8 + r) * KP + kc + nt * 8 + (m >> 1) * 8);
      ms_load_b<NPL, true>(b, at, 2 * CS_C * KP);
      ms_load_b<NPL, true>(b + 2, at + 32, 2 * CS_C * KP);
      ms_terms<4, 3, NPL>(acc + nt, low + nt, a, b);
    }
  }
  const int g = lane >> 2, c = lane & 3;
  float* dst = ds + (((size_t)item * H + h) * dv + c0 + rt + g) * DK + kc + 2 * c;
  bool odd = false;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[nt][j] += low[nt][j];
      odd |= !(fabsf(acc[nt][j]) < INFINITY);
    }
    *reinterpret_cast<float2*>(dst + nt * 8) = make_float2(acc[nt][0], acc[nt][1]);
    *reinterpret_cast<float2*>(dst + 8 * DK + nt * 8) = make_float2(acc[nt][2], acc[nt][3]);
  }
  if (odd) {
    const size_t v0 = (size_t)h * dv + c0 + rt + g;
    if constexpr (sizeof(T) == 4) cs_write_again_f32<DK>(in, dst, base, n, h, H, kc + 2 * c, v0);
    else cs_write_again<T, DK>(in, dst, base, n, h, H, kc + 2 * c, v0);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// ds[item] <- the state before the item's chunk; the record <- the state after the entry's last one.
// Four numbers of one head's state a thread, the chunks in order, CS_AHEAD loads on their way: bound by the two passes
// over ds.
// ---------------------------------------------------------------------------------------------------------------
#define CS_AHEAD 8
#define CS_PREFIX_THREADS 128
__global__ void __launch_bounds__(CS_PREFIX_THREADS)
chunk_prefix_kernel(float* __restrict__ ds, const float* __restrict__ gam, float* __restrict__ state, long slot_stride,
                    int num_slots, const int* __restrict__ cu_q, const int* __restrict__ req_slot, int H, int head_floats,
                    int write_state, int* status) {
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int h = blockIdx.y, e = blockIdx.z;
  const int slot = req_slot[e];
  if (slot < 0 || slot >= num_slots) {
    if (slot >= num_slots && threadIdx.x == 0) set_status(status, LL_ERR_SLOT_RANGE);
    return;
  }
  const int at = (blockIdx.x * CS_PREFIX_THREADS + threadIdx.x) * 4;
  const int first = cs_first_item(e, cu_q), chunks = (cu_q[e + 1] - cu_q[e] + CS_C - 1) / CS_C;
  if (at >= head_floats) return;
  float* rec = state + (size_t)slot * slot_stride + (size_t)h * head_floats + at;
  float s[4] = {rec[0], rec[1], rec[2], rec[3]};
  float* d = ds + ((size_t)first * H + h) * head_floats + at;
  const size_t step = (size_t)H * head_floats;
  const float* gp = gam + (size_t)first * H + h;
  for (int c0 = 0; c0 < chunks; c0 += CS_AHEAD) {
    float4 w[CS_AHEAD];
    float g[CS_AHEAD];
#pragma unroll
    for (int i = 0; i < CS_AHEAD; ++i)
      if (c0 + i < chunks) {
        w[i] = *reinterpret_cast<const float4*>(d + (size_t)(c0 + i) * step);
        g[i] = gp[(size_t)(c0 + i) * H];
      }
#pragma unroll
    for (int i = 0; i < CS_AHEAD; ++i)
      if (c0 + i < chunks) {
        *reinterpret_cast<float4*>(d + (size_t)(c0 + i) * step) = make_float4(s[0], s[1], s[2], s[3]);
        s[0] = fmaf(g[i], s[0], w[i].x);
        s[1] = fmaf(g[i], s[1], w[i].y);
        s[2] = fmaf(g[i], s[2], w[i].z);
        s[3] = fmaf(g[i], s[3], w[i].w);
      }
  }
  if (write_state) {
    rec[0] = s[0]; rec[1] = s[1]; rec[2] = s[2]; rec[3] = s[3];
  }
}

// ---------------------------------------------------------------------------------------------------------------
// The read-outs: o_t = G(t, -) S0^T q_t + sum over s <= t of G(t, s) (q_t . k_s) scale_s v_s (+ skip_h v_t).
// Tokens are the M side (16 of the chunk's 64 a warp).  The scores of a row are made by two warps, half of the keys each,
// and go through shared memory (in k's place) as the second product's operand, so they are made once for all value
// columns; the columns come 64 at a time, 32 a warp, the next 64's state and values on their way meanwhile.  One CTA an
// SM (registers, shared memory): two warps a scheduler, bound by the latencies of their own instructions (tensor pipe 30 % active where
// q is float32, with six products a term of S0^T q_t, 18 % otherwise).
// ---------------------------------------------------------------------------------------------------------------
template <typename T, int DK>
__global__ void __launch_bounds__(CS_THREADS)
chunk_read_kernel(CsRows<T> in, const int* __restrict__ cu_q, const int* __restrict__ req_slot, int E, int num_slots,
                  const float* __restrict__ s0, float* __restrict__ o, int H, int dv) {
  constexpr int NPL = sizeof(T) == 2 ? 1 : 3;
  constexpr int KP = DK + 8, VP = 72;
  constexpr int KROWS = (NPL * KP > 3 * VP ? NPL * KP : 3 * VP);          // k's terms, later the scores' three
  extern __shared__ __align__(16) unsigned char cs_smem[];
  bf16* qs = reinterpret_cast<bf16*>(cs_smem);                 // [NPL][64][KP]
  bf16* ks = qs + NPL * CS_C * KP;                             // [NPL][64][KP], then the scores [3][64][VP]
  bf16* vs = ks + KROWS * CS_C;                                // [NPL][64][VP]
  bf16* ss = vs + NPL * CS_C * VP;                             // [3][64][KP]: row = value column
  __shared__ float av[CS_C], pre[CS_C], sc[CS_C];
  __shared__ double runs[6 * CS_C];
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int item = blockIdx.x, h = blockIdx.y;
  int e, chunk;
  if (!cs_item(item, cu_q, E, e, chunk)) return;
  const int slot = req_slot[e];
  const int base = cu_q[e] + chunk * CS_C, n = min(CS_C, cu_q[e + 1] - base);
  float* orow = o + (size_t)base * H * dv + (size_t)h * dv;
  if (slot < 0 || slot >= num_slots) {       // a padding entry: defined output, nothing read
    for (int i = tid; i < n * dv; i += CS_THREADS) orow[(size_t)(i / dv) * H * dv + i % dv] = 0.f;
    return;
  }
  const float* srow = s0 + ((size_t)item * H + h) * dv * DK;
  const T* prow = in.proj + (size_t)base * in.stride;
  const bool own_u = sizeof(T) == 4 && in.u != nullptr;
  const T* vrow = own_u ? reinterpret_cast<const T*>(in.u) + ((size_t)item * H + h) * CS_C * dv
                        : prow + in.v_off + (size_t)h * dv;
  const long vstride = own_u ? dv : in.stride;
  const T* krow = (sizeof(T) == 4 && in.k_rows != nullptr) ? reinterpret_cast<const T*>(in.k_rows) + (size_t)base * in.stride
                                                           : prow + in.k_off;
  if (tid < CS_C) {
    av[tid] = tid >= n ? 1.f : in.tok_decay ? in.tok_decay[(size_t)(base + tid) * H + h] : in.decay[h];
    sc[tid] = (in.tok_scale && tid < n) ? in.tok_scale[(size_t)(base + tid) * H + h] : 1.f;
  }
  CsTile<T, DK, KP, CS_THREADS> qt, kt_;
  CsTile<T, 64, VP, CS_THREADS> vt;
  CsTile<float, DK, KP, CS_THREADS> st;
  qt.ask(prow + in.q_off + (h / in.hpg) * DK, in.stride, n);
  kt_.ask(krow + (h / in.hpg) * DK, in.stride, n);
  qt.put(qs);
  st.ask(srow, DK, CS_C);
  kt_.put(ks);
  vt.ask(vrow, vstride, n);
  __syncthreads();
  if (warp == 0) cs_products(av[lane], av[lane + 32], pre, nullptr);
  if (warp == 1) cs_runs(av, runs);
  st.put(ss);
  vt.put(vs);
  __syncthreads();
  const int m = lane >> 3, r = lane & 7, g = lane >> 2, c = lane & 3;
  const unsigned qs_b = ms_smem(qs), ks_b = ms_smem(ks), vs_b = ms_smem(vs), ss_b = ms_smem(ss);
  const int rt = warp & 3, row = rt * 16, half = warp >> 2;
  float x[4][4], low[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) x[i][j] = low[i][j] = 0.f;
  if (half <= rt / 2) {                                 // (keys behind every row of the warp are not asked)
#pragma unroll
    for (int kt = 0; kt < DK / 16; ++kt) {
      unsigned a[NPL][4], b[4][NPL][2];
#pragma unroll
      for (int p = 0; p < NPL; ++p)
        ms_ldm4(a[p], qs_b + 2 * ((p * CS_C + row + (m & 1) * 8 + r) * KP + kt * 16 + (m >> 1) * 8));
      const unsigned at = ks_b + 2 * ((half * 32 + (m >> 1) * 8 + r) * KP + kt * 16 + (m & 1) * 8);
      ms_load_b<NPL, false>(b, at, 2 * CS_C * KP);
      ms_load_b<NPL, false>(b + 2, at + 2 * 16 * KP, 2 * CS_C * KP);
      ms_terms<4, NPL, NPL>(x, low, a, b);
    }
  }
  __syncthreads();                                      // k has been read
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int s = half * 32 + i * 8 + 2 * c;
    const float e0 = sc[s], e1 = sc[s + 1];
    unsigned p0, p1, p2;
    unsigned char* dst = reinterpret_cast<unsigned char*>(ks) + 2 * ((row + g) * VP + s);
    ms_split((x[i][0] + low[i][0]) * (cs_gap(runs, row + g, s) * e0), (x[i][1] + low[i][1]) * (cs_gap(runs, row + g, s + 1) * e1),
             p0, p1, p2);
    *reinterpret_cast<unsigned*>(dst) = p0;
    *reinterpret_cast<unsigned*>(dst + 2 * CS_C * VP) = p1;
    *reinterpret_cast<unsigned*>(dst + 4 * CS_C * VP) = p2;
    dst += 2 * 8 * VP;
    ms_split((x[i][2] + low[i][2]) * (cs_gap(runs, row + g + 8, s) * e0),
             (x[i][3] + low[i][3]) * (cs_gap(runs, row + g + 8, s + 1) * e1), p0, p1, p2);
    *reinterpret_cast<unsigned*>(dst) = p0;
    *reinterpret_cast<unsigned*>(dst + 2 * CS_C * VP) = p1;
    *reinterpret_cast<unsigned*>(dst + 4 * CS_C * VP) = p2;
  }
  const float f0 = pre[row + g], f1 = pre[row + g + 8];
  const float skip = in.skip ? in.skip[h] : 0.f;
  bool odd = false;
  for (int c0 = 0; c0 < dv; c0 += 64) {
    const bool more = c0 + 64 < dv;
    __syncthreads();                                    // the scores, this pass's state and values are there
    if (more) {
      st.ask(srow + (size_t)(c0 + 64) * DK, DK, CS_C);
      vt.ask(vrow + c0 + 64, vstride, n);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) x[i][j] = low[i][j] = 0.f;
#pragma unroll
    for (int kt = 0; kt < DK / 16; ++kt) {
      unsigned a[NPL][4], b[4][3][2];
#pragma unroll
      for (int p = 0; p < NPL; ++p)
        ms_ldm4(a[p], qs_b + 2 * ((p * CS_C + row + (m & 1) * 8 + r) * KP + kt * 16 + (m >> 1) * 8));
      const unsigned at = ss_b + 2 * ((half * 32 + (m >> 1) * 8 + r) * KP + kt * 16 + (m & 1) * 8);
      ms_load_b<3, false>(b, at, 2 * CS_C * KP);
      ms_load_b<3, false>(b + 2, at + 2 * 16 * KP, 2 * CS_C * KP);
      ms_terms<4, NPL, 3>(x, low, a, b);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[i][j] = (x[i][j] + low[i][j]) * (j < 2 ? f0 : f1);
        low[i][j] = 0.f;
      }
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
      if (kt <= rt) {
        unsigned a[3][4], b[4][NPL][2];
#pragma unroll
        for (int p = 0; p < 3; ++p)
          ms_ldm4(a[p], ks_b + 2 * ((p * CS_C + row + (m & 1) * 8 + r) * VP + kt * 16 + (m >> 1) * 8));
        const unsigned at = vs_b + 2 * ((kt * 16 + (m & 1) * 8 + r) * VP + half * 32 + (m >> 1) * 8);
        ms_load_b<NPL, true>(b, at, 2 * CS_C * VP);
        ms_load_b<NPL, true>(b + 2, at + 32, 2 * CS_C * VP);
        ms_terms<4, 3, NPL>(x, low, a, b);
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int t = row + g + 8 * q;
      if (t >= n) continue;
      const int col = c0 + half * 32 + 2 * c;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float u = x[i][2 * q] + low[i][2 * q], w = x[i][2 * q + 1] + low[i][2 * q + 1];
        if (in.skip) {
          u = fmaf(skip, to_f32<T>(vrow[(size_t)t * vstride + col + i * 8]), u);
          w = fmaf(skip, to_f32<T>(vrow[(size_t)t * vstride + col + i * 8 + 1]), w);
        }
        *reinterpret_cast<float2*>(orow + (size_t)t * H * dv + col + i * 8) = make_float2(u, w);
        odd |= !(fabsf(u) < INFINITY && fabsf(w) < INFINITY);
      }
    }
    if (more) {
      __syncthreads();                                  // this pass's state and values have been read
      st.put(ss);
      vt.put(vs);
    }
  }
  if (odd) {
    const T *qh = prow + in.q_off + (h / in.hpg) * DK, *kh = krow + (h / in.hpg) * DK;
    const float *a = av, *w = sc;
    if constexpr (sizeof(T) == 4)
      cs_read_again_f32<DK>(orow, (long)H * dv, qh, kh, in.stride, vrow, vstride, srow, a, w, in.skip != nullptr, skip, n, dv, row + g,
                            half * 32 + 2 * c);
    else
      cs_read_again<T, DK>(orow, (long)H * dv, qh, kh, in.stride, vrow, vstride, srow, a, w, in.skip != nullptr, skip, n, dv, row + g,
                           half * 32 + 2 * c);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Delta rule, before the walk: U = (1 + L)^-1 [beta v], float32 [items][H][64][dv], and W = (1 + L)^-1 [beta G(t, -) k],
// float32 [items][H][64][DK]; suf[items][H][64] = G(C, s), gam[items][H].  k_t . k_s on tensor cores, then every column of
// the right-hand sides is a thread's: 2,016 multiply-adds against L in shared memory (all threads read the same number),
// no inverse is formed.
// ---------------------------------------------------------------------------------------------------------------
template <int DK, int DV>
__global__ void __launch_bounds__(DK + DV)
delta_solve_kernel(const float* __restrict__ kn, const float* __restrict__ vc, const float* __restrict__ beta,
                   const float* __restrict__ g, const int* __restrict__ cu_q, const int* __restrict__ req_slot, int E,
                   float* __restrict__ u, float* __restrict__ w, float* __restrict__ suf_out, float* __restrict__ gam, int H,
                   int Hk) {
  constexpr int KP = DK + 8, THREADS = DK + DV, WARPS = THREADS / 32;
  extern __shared__ __align__(16) unsigned char cs_smem[];
  bf16* ks = reinterpret_cast<bf16*>(cs_smem);                   // [3][64][KP]
  float* L = reinterpret_cast<float*>(ks + 3 * CS_C * KP);       // [64][64]
  __shared__ float av[CS_C], bt[CS_C], pre[CS_C], suf[CS_C];
  __shared__ double runs[6 * CS_C];
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int item = blockIdx.x, h = blockIdx.y, hk = h / (H / Hk);
  int e, chunk;
  if (!cs_item(item, cu_q, E, e, chunk)) return;
  if (req_slot[e] < 0) return;
  const int base = cu_q[e] + chunk * CS_C, n = min(CS_C, cu_q[e + 1] - base);
  const long Cq = (long)Hk * DK, Cv = (long)H * DV;
  {
    CsTile<float, DK, KP, THREADS> kt_;
    kt_.ask(kn + (size_t)base * Cq + hk * DK, Cq, n);
    if (tid < CS_C) {
      av[tid] = tid < n ? g[(size_t)(base + tid) * H + h] : 1.f;
      bt[tid] = tid < n ? beta[(size_t)(base + tid) * H + h] : 0.f;
    }
    kt_.put(ks);
  }
  __syncthreads();
  if (warp == 0) {
    const float all = cs_products(av[lane], av[lane + 32], pre, suf);
    if (lane == 0) gam[(size_t)item * H + h] = all;
  }
  if (warp == 1) cs_runs(av, runs);
  __syncthreads();
  if (tid < CS_C) suf_out[((size_t)item * H + h) * CS_C + tid] = suf[tid];
  // scores of 16 rows by 16 columns at a time, the lower triangle of them
  {
    const int m = lane >> 3, r = lane & 7, gg = lane >> 2, c = lane & 3;
    const unsigned ks_b = ms_smem(ks);
    for (int tile = warp; tile < 10; tile += WARPS) {
      int rt = 0, ct = tile;
      while (ct > rt) {
        ct -= rt + 1;
        ++rt;
      }
      float acc[2][4] = {}, low[2][4] = {};
#pragma unroll
      for (int kt = 0; kt < DK / 16; ++kt) {
        unsigned a[3][4], b[2][3][2];
#pragma unroll
        for (int p = 0; p < 3; ++p)
          ms_ldm4(a[p], ks_b + 2 * ((p * CS_C + rt * 16 + (m & 1) * 8 + r) * KP + kt * 16 + (m >> 1) * 8));
        ms_load_b<3, false>(b, ks_b + 2 * ((ct * 16 + (m >> 1) * 8 + r) * KP + kt * 16 + (m & 1) * 8), 2 * CS_C * KP);
        ms_terms<2, 3, 3>(acc, low, a, b);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = rt * 16 + gg + (j >> 1) * 8, s = ct * 16 + i * 8 + 2 * c + (j & 1);
          L[t * CS_C + s] = s < t ? bt[t] * cs_gap(runs, t, s) * (acc[i][j] + low[i][j]) : 0.f;
        }
    }
  }
  // the thread's column of the right-hand sides
  const bool is_k = tid < DK;
  float x[CS_C];
  {
    const float* src = is_k ? kn + (size_t)base * Cq + hk * DK + tid : vc + (size_t)base * Cv + (size_t)h * DV + (tid - DK);
    const long stride = is_k ? Cq : Cv;
#pragma unroll
    for (int t = 0; t < CS_C; ++t) x[t] = t < n ? src[(size_t)t * stride] : 0.f;
  }
#pragma unroll
  for (int t = 0; t < CS_C; ++t) x[t] *= is_k ? bt[t] * pre[t] : bt[t];
  __syncthreads();
#pragma unroll
  for (int t = 1; t < CS_C; ++t) {
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int s = 0; s < t; s += 4) {
      const float4 l4 = *reinterpret_cast<const float4*>(L + t * CS_C + s);
      s0 = fmaf(l4.x, x[s], s0);
      if (s + 1 < t) s1 = fmaf(l4.y, x[s + 1], s1);
      if (s + 2 < t) s0 = fmaf(l4.z, x[s + 2], s0);
      if (s + 3 < t) s1 = fmaf(l4.w, x[s + 3], s1);
    }
    x[t] -= s0 + s1;
  }
  float* dst = is_k ? w + ((size_t)item * H + h) * CS_C * DK + tid : u + ((size_t)item * H + h) * CS_C * DV + (tid - DK);
  const int pitch = is_k ? DK : DV;
#pragma unroll
  for (int t = 0; t < CS_C; ++t) dst[t * pitch] = x[t];
}

// ---------------------------------------------------------------------------------------------------------------
// Delta rule, the walk: for the entry's chunks in order  s0 <- S,  u <- U - W S (in place),  S <- G(C, -) S + k^T (G(C, s) u).
// 16 value columns a CTA are the M side of both products; a warp holds an eighth of the key channels of S^T [16 x DK] in
// its accumulators, which are the first product's operand as they stand; the warps' parts of W S meet in shared memory.
// Two chains of 48 MMAs and three barriers a chunk; W and k of the next chunk are fetched a whole chunk ahead (float32, the
// terms are made on the way into the registers: as bfloat16 terms they are half as many bytes again, and the 8 CTAs of a head
// read them all).
// ---------------------------------------------------------------------------------------------------------------
template <int DK>
__global__ void __launch_bounds__(CS_THREADS)
delta_walk_kernel(float* __restrict__ u, const float* __restrict__ w, const float* __restrict__ kn,
                  const float* __restrict__ suf_in, const float* __restrict__ gam, float* __restrict__ s0,
                  float* __restrict__ state, long state_stride, int num_slots, const int* __restrict__ cu_q,
                  const int* __restrict__ req_slot, int H, int Hk, int dv) {
  constexpr int WARPS = CS_THREADS / 32, KW = DK / WARPS;      // key channels a warp: 16, or 8 of heads of 64
  constexpr int FP = DK + 4, UP = CS_C + 8, RP = CS_C + 4;
  constexpr int NT = KW / 8;
  extern __shared__ __align__(16) unsigned char cs_smem[];
  float* wf = reinterpret_cast<float*>(cs_smem);               // [2][64][FP]
  float* kf = wf + 2 * CS_C * FP;                              // [2][64][FP]
  float* red = kf + 2 * CS_C * FP;                             // [WARPS][16][RP]
  bf16* us = reinterpret_cast<bf16*>(red + WARPS * 16 * RP);   // [3][16][UP]: G(C, s) u, a row a value column
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c0 = blockIdx.x * 16, h = blockIdx.y, e = blockIdx.z, hk = h / (H / Hk);
  const int slot = req_slot[e];
  if (slot < 0 || slot >= num_slots) return;
  const int start = cu_q[e], last = cu_q[e + 1];
  const int first = cs_first_item(e, cu_q), chunks = (last - start + CS_C - 1) / CS_C;
  if (chunks == 0) return;
  const int m = lane >> 3, r = lane & 7, g = lane >> 2, c = lane & 3;
  const int kw = warp * KW;                             // the warp's first key channel
  const unsigned us_b = ms_smem(us);
  const long Cq = (long)Hk * DK;
  auto fetch = [&](int chunk) {
    const float* ws = w + ((size_t)(first + chunk) * H + h) * CS_C * DK;
    const float* ks = kn + (size_t)(start + chunk * CS_C) * Cq + hk * DK;
    const int n = min(CS_C, last - start - chunk * CS_C);
    float* wd = wf + (chunk & 1) * CS_C * FP;
    float* kd = kf + (chunk & 1) * CS_C * FP;
#pragma unroll
    for (int i = tid; i < CS_C * DK / 4; i += CS_THREADS) {
      const int t = i / (DK / 4), cc = (i % (DK / 4)) * 4;
      ms_copy16(ms_smem(wd + t * FP + cc), ws + (size_t)t * DK + cc);
      if (t < n) ms_copy16(ms_smem(kd + t * FP + cc), ks + (size_t)t * Cq + cc);
      else *reinterpret_cast<float4*>(kd + t * FP + cc) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    ms_commit();
  };
  fetch(0);
  float* rec = state + (size_t)slot * state_stride + ((size_t)h * dv + c0) * DK + kw;
  float S[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const float2 a = *reinterpret_cast<const float2*>(rec + (size_t)g * DK + nt * 8 + 2 * c);
    const float2 b = *reinterpret_cast<const float2*>(rec + (size_t)(g + 8) * DK + nt * 8 + 2 * c);
    S[nt][0] = a.x; S[nt][1] = a.y; S[nt][2] = b.x; S[nt][3] = b.y;
  }
  const int un = tid & 15, ut = (tid >> 4) * 4;         // the value column and the 4 tokens of u that a thread joins
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const size_t ih = (size_t)(first + chunk) * H + h;
    float* urow = u + (ih * CS_C + ut) * dv + c0 + un;
    float uv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) uv[i] = urow[(size_t)i * dv];
    const float4 f4 = *reinterpret_cast<const float4*>(suf_in + ih * CS_C + ut);
    const float gc = gam[ih];
    const float* wb = wf + (chunk & 1) * CS_C * FP;
    const float* kb = kf + (chunk & 1) * CS_C * FP;
    float* sdst = s0 + (ih * dv + c0) * DK + kw;
    unsigned a[3][4] = {};
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      *reinterpret_cast<float2*>(sdst + (size_t)g * DK + nt * 8 + 2 * c) = make_float2(S[nt][0], S[nt][1]);
      *reinterpret_cast<float2*>(sdst + (size_t)(g + 8) * DK + nt * 8 + 2 * c) = make_float2(S[nt][2], S[nt][3]);
      ms_split(S[nt][0], S[nt][1], a[0][2 * nt], a[1][2 * nt], a[2][2 * nt]);
      ms_split(S[nt][2], S[nt][3], a[0][2 * nt + 1], a[1][2 * nt + 1], a[2][2 * nt + 1]);
    }
    ms_wait<0>();
    __syncthreads();                                    // this chunk's W and k are here, the last one's have been read
    if (chunk + 1 < chunks) fetch(chunk + 1);
    // (W S)^T [16 x 64] over the warp's key channels (heads of 64: the upper half of the step of 16 is zeros)
#pragma unroll
    for (int nt = 0; nt < 8; nt += 4) {
      float part[4][4] = {}, low[4][4] = {};
      unsigned b[4][3][2] = {};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float* src = wb + ((nt + i) * 8 + g) * FP + kw + 2 * c;
#pragma unroll
        for (int q = 0; q < NT; ++q) {
          const float2 v = *reinterpret_cast<const float2*>(src + 8 * q);
          ms_split(v.x, v.y, b[i][0][q], b[i][1][q], b[i][2][q]);
        }
      }
      ms_terms<4, 3, 3>(part, low, a, b);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float* rd = red + (warp * 16 + g) * RP + (nt + i) * 8 + 2 * c;
        *reinterpret_cast<float2*>(rd) = make_float2(part[i][0] + low[i][0], part[i][1] + low[i][1]);
        *reinterpret_cast<float2*>(rd + 8 * RP) = make_float2(part[i][2] + low[i][2], part[i][3] + low[i][3]);
      }
    }
    __syncthreads();                                    // the parts are there
    {
      float4 t4 = *reinterpret_cast<const float4*>(red + un * RP + ut);
#pragma unroll
      for (int wp = 1; wp < WARPS; ++wp) {
        const float4 x4 = *reinterpret_cast<const float4*>(red + (wp * 16 + un) * RP + ut);
        t4.x += x4.x; t4.y += x4.y; t4.z += x4.z; t4.w += x4.w;
      }
      uv[0] -= t4.x; uv[1] -= t4.y; uv[2] -= t4.z; uv[3] -= t4.w;
#pragma unroll
      for (int i = 0; i < 4; ++i) urow[(size_t)i * dv] = uv[i];
      uint2 p0, p1, p2;
      ms_split(uv[0] * f4.x, uv[1] * f4.y, p0.x, p1.x, p2.x);
      ms_split(uv[2] * f4.z, uv[3] * f4.w, p0.y, p1.y, p2.y);
      *reinterpret_cast<uint2*>(us + un * UP + ut) = p0;
      *reinterpret_cast<uint2*>(us + (16 + un) * UP + ut) = p1;
      *reinterpret_cast<uint2*>(us + (32 + un) * UP + ut) = p2;
    }
    float low[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        S[nt][j] *= gc;
        low[nt][j] = 0.f;
      }
    __syncthreads();
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
      unsigned ua[3][4], b[NT][3][2];
#pragma unroll
      for (int p = 0; p < 3; ++p) ms_ldm4(ua[p], us_b + 2 * ((p * 16 + (m & 1) * 8 + r) * UP + kt * 16 + (m >> 1) * 8));
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float* src = kb + (kt * 16 + q * 8 + 2 * c) * FP + kw + nt * 8 + g;
          ms_split(src[0], src[FP], b[nt][0][q], b[nt][1][q], b[nt][2][q]);
        }
      ms_terms<NT, 3, 3>(S, low, ua, b);
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) S[nt][j] += low[nt][j];
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    *reinterpret_cast<float2*>(rec + (size_t)g * DK + nt * 8 + 2 * c) = make_float2(S[nt][0], S[nt][1]);
    *reinterpret_cast<float2*>(rec + (size_t)(g + 8) * DK + nt * 8 + 2 * c) = make_float2(S[nt][2], S[nt][3]);
  }
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

template <typename T, int DK>
static int cs_read(const CsRows<T>& in, const int* cu_q, const int* req_slot, int E, int num_slots, const float* s0,
                   float* o, int H, int dv, int items, cudaStream_t stream) {
  constexpr int NPL = sizeof(T) == 2 ? 1 : 3;
  constexpr int KROWS = NPL * (DK + 8) > 3 * 72 ? NPL * (DK + 8) : 3 * 72;
  const size_t smem = 2 * (size_t)CS_C * ((NPL + 3) * (DK + 8) + KROWS + NPL * 72);
  const cudaError_t rc = cs_room<chunk_read_kernel<T, DK>>(smem);
  if (rc != cudaSuccess) return (int)rc;
  ll_launch(chunk_read_kernel<T, DK>, dim3(items, H), dim3(CS_THREADS), smem, stream, in, cu_q, req_slot, E, num_slots, s0, o,
            H, dv);
  return LL_LAUNCH_RESULT();
}

template <typename T, int DK>
static int cs_decay(const CsRows<T>& in, float* state, long slot_stride, int num_slots, const int* cu_q,
                    const int* req_slot, float* o, int E, int H, int dv, int write_state, int* status, float* ds, float* gam,
                    int items, cudaStream_t stream) {
  constexpr int NPL = sizeof(T) == 2 ? 1 : 3;
  const size_t smem = 2 * (size_t)CS_C * (NPL * (DK + 8) + 3 * 72);
  const cudaError_t rc = cs_room<chunk_write_kernel<T, DK>>(smem);
  if (rc != cudaSuccess) return (int)rc;
  ll_launch(chunk_write_kernel<T, DK>, dim3(items, H, dv / 64), dim3(CS_THREADS), smem, stream, in, cu_q, req_slot, E,
            num_slots, ds, gam, H, dv);
  ll_launch(chunk_prefix_kernel, dim3((DK * dv + 4 * CS_PREFIX_THREADS - 1) / (4 * CS_PREFIX_THREADS), H, E),
            dim3(CS_PREFIX_THREADS), 0, stream, ds, (const float*)gam, state, slot_stride, num_slots, cu_q, req_slot, H,
            DK * dv, write_state, status);
  const int first = LL_LAUNCH_RESULT();
  if (first != 0) return first;
  return cs_read<T, DK>(in, cu_q, req_slot, E, num_slots, ds, o, H, dv, items, stream);
}

// The recurrence of ll_decay_scan (linear_attention.cu) by chunks: three launches.  `items`: at least the number of chunks
// of 64 tokens of the step's entries; ds: float32 [items][H][dv][dk], gam: float32 [items][H].
extern "C" int ll_chunk_decay_scan(int dtype, const void* proj, long stride, int q_off, int k_off, int v_off,
                                   const float* decay, float* state, long slot_stride, int num_slots, const int* cu_q,
                                   const int* req_slot, float* o, int num_entries, int H, int dk, int dv, int write_state,
                                   int* status, int hpg, const float* tok_decay, const float* tok_scale,
                                   const float* skip, float* ds, float* gam, int items, cudaStream_t stream) {
  if (num_entries <= 0 || items <= 0) return 0;
  if (H <= 0 || (dk != 64 && dk != 128) || dv <= 0 || dv % 64 != 0 || hpg <= 0 || H % hpg != 0 || H > 65535 ||
      num_entries > 65535 || (decay == nullptr && tok_decay == nullptr))
    return (int)cudaErrorInvalidValue;
  LL_DISPATCH_DTYPE(dtype, {
    CsRows<T> in{(const T*)proj, stride, q_off, k_off, v_off, decay, tok_decay, tok_scale, skip, nullptr, nullptr, hpg};
    if (dk == 128)
      return cs_decay<T, 128>(in, state, slot_stride, num_slots, cu_q, req_slot, o, num_entries, H, dv, write_state, status,
                              ds, gam, items, stream);
    return cs_decay<T, 64>(in, state, slot_stride, num_slots, cu_q, req_slot, o, num_entries, H, dv, write_state, status, ds,
                           gam, items, stream);
  });
  return 0;
}

template <int DK, int DV>
static int cs_delta(const float* qn, const float* kn, const float* vc, const float* beta, const float* g, float* state,
                    long state_stride, int num_slots, const int* cu_q, const int* req_slot, float* o, int E, int H, int Hk,
                    float* s0, float* u, float* w, float* suf, float* gam, int items, cudaStream_t stream) {
  const size_t solve = 2 * (size_t)3 * CS_C * (DK + 8) + 4 * CS_C * CS_C;
  const size_t walk = 4 * (size_t)(4 * CS_C * (DK + 4) + 8 * 16 * (CS_C + 4)) + 2 * 3 * 16 * (CS_C + 8);
  cudaError_t rc = cs_room<delta_solve_kernel<DK, DV>>(solve);
  if (rc != cudaSuccess) return (int)rc;
  rc = cs_room<delta_walk_kernel<DK>>(walk);
  if (rc != cudaSuccess) return (int)rc;
  ll_launch(delta_solve_kernel<DK, DV>, dim3(items, H), dim3(DK + DV), solve, stream, kn, vc, beta, g, cu_q, req_slot, E, u,
            w, suf, gam, H, Hk);
  ll_launch(delta_walk_kernel<DK>, dim3(DV / 16, H, E), dim3(CS_THREADS), walk, stream, u, (const float*)w, kn,
            (const float*)suf, (const float*)gam, s0, state, state_stride, num_slots, cu_q, req_slot, H, Hk, DV);
  const int first = LL_LAUNCH_RESULT();
  if (first != 0) return first;
  CsRows<float> in{qn, (long)Hk * DK, 0, 0, 0, nullptr, g, nullptr, nullptr, kn, u, H / Hk};
  return cs_read<float, DK>(in, cu_q, req_slot, E, num_slots, s0, o, H, DV, items, stream);
}

// The recurrence of ll_delta_recurrence (delta_rule.cu) with one decay a head, by chunks: three launches.  Scratch:
// s0 float32 [items][H][dv][dk], u float32 [items][H][64][dv], w float32 [items][H][64][dk], suf float32 [items][H][64],
// gam float32 [items][H].
extern "C" int ll_chunk_delta_scan(const float* qn, const float* kn, const float* vc, const float* beta, const float* g,
                                   float* state, long state_stride, int num_slots, const int* cu_q, const int* req_slot,
                                   float* o, int num_entries, int H, int Hk, int dk, int dv, float* s0, float* u,
                                   float* w, float* suf, float* gam, int items, cudaStream_t stream) {
  if (num_entries <= 0 || items <= 0) return 0;
  if (H <= 0 || Hk <= 0 || H % Hk || H > 65535 || num_entries > 65535) return (int)cudaErrorInvalidValue;
#define CS_DELTA(DK, DV)                                                                                              \
  return cs_delta<DK, DV>(qn, kn, vc, beta, g, state, state_stride, num_slots, cu_q, req_slot, o, num_entries, H, Hk, s0, u, \
                          w, suf, gam, items, stream)
  if (dk == 128 && dv == 128) CS_DELTA(128, 128);
  if (dk == 128 && dv == 64) CS_DELTA(128, 64);
  if (dk == 64 && dv == 128) CS_DELTA(64, 128);
  if (dk == 64 && dv == 64) CS_DELTA(64, 64);
#undef CS_DELTA
  return (int)cudaErrorInvalidValue;
}
