// Matrix-state recurrences of prompt portions, 64 tokens at a time.
//
// A linear recurrence S_t = a_t S_(t-1) + k_t v_t^T, o_t = S_t^T q_t (linear attention with decay, retention, a
// state-space layer) walked token by token is bound by its chain: 2,048 tokens took 320 us with 12 heads (790 us as a delta
// rule), at 2 % of the chip's arithmetic.  Cut into chunks of 64 tokens (C), with G(t, s) = a_(s+1) ... a_t,
//     o_t     = G(t, -) S0^T q_t + sum over s <= t of G(t, s) (q_t . k_s) v_s         S0: the state before the chunk
//     S_end   = G(C, -) S0 + sum over s of k_s (G(C, s) v_s)^T
// the work between two chunks' states is matrix products, and chunks meet only in S0:
//   chunk_write    per (chunk, head, 64 value columns): sum of k_s (G(C, s) v_s)^T
//   chunk_prefix   per (entry, head, part of the state): the states before every chunk, and the record's new state
//   chunk_read     per (chunk, head): the read-outs
// (The delta rule, whose written values depend on the state: delta_chunks.cu.)
//
// Everything is float32 as in the walk by tokens: decays are running products (a decay that underflows to 0 stays 0,
// nothing is divided), products of float32 numbers are made of bfloat16 terms that hold all 24 bits (mma_split.cuh), and
// operands that are stored as bfloat16 are taken as they are.  A chunk starts where the step's portion does, so the order
// of the sums depends on how a prompt was cut into portions, within rounding.  Infinities have no bfloat16 terms and a
// product with 0 makes NaN of them, so a number that is not finite would show in the chunk's tokens before it, too: a thread
// that finds a state or a read-out not finite makes that number again token by token (`cs_again`), as the walk does.
//
// Taken for longer portions, key heads of 64 or 128 channels and value heads of a multiple of 64: see `ops.chunked_scan`.
#include "chunk_scan.cuh"

// Where the rows of a chunk come from: q, k and v heads of a row a token.
template <typename T> struct CsRows {
  const T* proj;
  long stride;
  int q_off, k_off, v_off;
  const float* decay;        // one a head, or
  const float* tok_decay;    // one a (token, head) [tokens, H]
  const float* tok_scale;    // a factor on a token's v, or null
  const float* skip;         // one a head: its own v added to a token's read-out, or null
  int hpg;                   // heads that read the same q and k
};

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
  const T *vrow = prow + in.v_off + (size_t)h * dv, *krow = prow + in.k_off;
  const long vstride = in.stride;
  // (float32: an address of its own.  As an offset from the row's, the compiler moved loads forward into 255 registers and a spill:
  // 57.8 us for 2,048 tokens of 12 heads of 128, 56.0 this way with 179; heads of 64, 128 registers and two CTAs an SM, 34.6 / 30.4.)
  if (sizeof(T) == 4) asm("" : "+l"(vrow));
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
    CsRows<T> in{(const T*)proj, stride, q_off, k_off, v_off, decay, tok_decay, tok_scale, skip, hpg};
    if (dk == 128)
      return cs_decay<T, 128>(in, state, slot_stride, num_slots, cu_q, req_slot, o, num_entries, H, dv, write_state, status,
                              ds, gam, items, stream);
    return cs_decay<T, 64>(in, state, slot_stride, num_slots, cu_q, req_slot, o, num_entries, H, dv, write_state, status, ds,
                           gam, items, stream);
  });
  return 0;
}
