// Gated delta rule: a linear recurrence with a matrix state per head.
//
// Per request and head the state S [dk, dv] (float32) evolves token by token:
//     S <- diag(g) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// with q, k unit vectors (q also times dk^-1/2), beta in (0, 1) and a decay g in (0, 1] that is
// one number per head or one per head and key channel.  q, k and v come out of a short causal
// convolution over time (per channel, `taps` taps, the last one the current token's) and SiLU.
// A request's record in the state pool is float32 [heads][dv][dk] for S (a value column's key channels side by
// side, as the lanes of the scan hold them) followed by
// [(taps - 1), channels] for the last taps - 1 inputs of the convolutions (oldest first;
// channels = q | k | v), so that a request can go on in a later step from where it stopped.
//
// Four kernels (a long portion's recurrence goes by chunks instead: delta_chunks.cu; a step of single tokens
// takes one launch for all of them, delta_step, where its sizes allow it), all reading the step's device arrays only (so that
// a step of single tokens can be captured and replayed):
//   delta_prepare      per token: convolution + SiLU, unit vectors, beta, decay -> float32 buffers
//   delta_conv_update  per entry of several tokens: the new last taps - 1 inputs of the record
//   delta_recurrence   per (entry, head, 16 value columns): the scan over the entry's tokens
//   delta_out          per (token, head): o / rms(o) * weight * gate -> storage type
// Every value column of S evolves on its own (S^T k and S^T q are per column), so the scan is
// spread over value columns as well as over requests and heads; the order of every sum depends
// on the sizes only; in the scan by tokens never on how they were cut into steps or batched.
#include "common.cuh"

__device__ __forceinline__ float dr_sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float dr_silu(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float dr_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

struct DeltaShape {
  int H, Hk, dk, dv, taps;
  int per_channel;   // decay: 0 one per head, 1 one per head and key channel
};

// proj: the step's projections, row t at proj + t * proj_stride, with q at column q_off (Hk*dk wide), k at k_off
// (Hk*dk), v at v_off (H*dv), b at b_off (H).  a_in: the decay's input, [tokens, H] or [tokens, H*dk].
//
// A warp makes one unit of one token: a q or k head (convolution, SiLU, unit vector), a v head (convolution, SiLU), the decays
// (of a head with one a channel, else of all heads) or the betas; a block takes a unit of eight neighbouring tokens, whose
// convolutions read nearly the same rows.  VEC channels a lane and access; four taps, the usual number, unrolled.  Bound by
// the lanes' loads in flight: 2,047 tokens of 2,048 channels 25 us (41 with a loop over the taps).  (A block a token with its
// channels in shared memory took 41 us too, and 14.7 us for one token, which left 147 SMs idle; now 4 us.)
// An entry of one token moves its convolutions' last inputs up here: nobody else reads them.
#define DP_TOKENS 8
template <typename T, int VEC> struct DpVec;
template <typename T> struct DpVec<T, 1> {
  __device__ static void load(const T* p, float (&v)[1]) { v[0] = to_f32<T>(p[0]); }
};
template <> struct DpVec<float, 4> {
  __device__ static void load(const float* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  }
};
template <> struct DpVec<bf16, 4> {
  __device__ static void load(const bf16* p, float (&v)[4]) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
};
template <int VEC> __device__ __forceinline__ void dp_store(float* p, const float (&v)[VEC]) {
  if (VEC == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1 % VEC], v[2 % VEC], v[3 % VEC]);
  else p[0] = v[0];
}

// What one token's projections of a unit (a q, k or v head, the betas, or decays) come to, by one warp.
template <typename T, int VEC, int TAPS>
__device__ __forceinline__ void delta_prepare_token(
    int t, int unit, int lane, const T* __restrict__ proj, long proj_stride, int q_off, int k_off, int v_off, int b_off,
    const T* __restrict__ a_in, long a_stride, const float* __restrict__ conv_q, const float* __restrict__ conv_k,
    const float* __restrict__ conv_v, const float* __restrict__ A_log, const float* __restrict__ dt_bias, float* state,
    long state_stride, long tail_off, const int* __restrict__ token_req, const int* __restrict__ cu_q,
    const int* __restrict__ ctx_len, const int* __restrict__ req_slot, const int* __restrict__ positions, float* __restrict__ qn,
    float* __restrict__ kn, float* __restrict__ vc, float* __restrict__ beta, float* __restrict__ g, const DeltaShape& s) {
  constexpr int PIECES = 8 / VEC;                 // of a q or k head of up to 256 channels: kept between the sum and the output
  const int e = token_req[t];
  const int slot = e >= 0 ? req_slot[e] : -1;
  if (slot < 0) return;   // padding entry: the scan writes its (zero) output
  const int Cq = s.Hk * s.dk, Cv = s.H * s.dv, C = 2 * Cq + Cv, K = s.taps;
  const T* row = proj + (size_t)t * proj_stride;
  if (unit >= 2 * s.Hk + s.H) {
    if (unit == 2 * s.Hk + s.H) {                 // betas
      for (int h = lane; h < s.H; h += 32) beta[(size_t)t * s.H + h] = dr_sigmoid(to_f32<T>(row[b_off + h]));
    } else if (!s.per_channel) {                  // decays, one a head
      for (int h = lane; h < s.H; h += 32) {
        const float a = to_f32<T>(a_in[(size_t)t * a_stride + h]) + dt_bias[h];
        g[(size_t)t * s.H + h] = expf(-expf(A_log[h]) * dr_softplus(a));
      }
    } else {                                      // decays of a head's channels
      const int h = unit - (2 * s.Hk + s.H) - 1;
      const float rate = -expf(A_log[h]);
      const T* ar = a_in + (size_t)t * a_stride + (size_t)h * s.dk;
      const float* br = dt_bias + (size_t)h * s.dk;
      float* gr = g + ((size_t)t * s.H + h) * s.dk;
      for (int i = lane; i < s.dk; i += 32) gr[i] = expf(rate * dr_softplus(to_f32<T>(ar[i]) + br[i]));
    }
    return;
  }
  // a head's channels: where they lie in the projections, in the filters, among the record's inputs and in the output
  const int kind = unit < s.Hk ? 0 : unit < 2 * s.Hk ? 1 : 2, head = unit - (kind == 0 ? 0 : kind == 1 ? s.Hk : 2 * s.Hk);
  const int width = kind == 2 ? s.dv : s.dk, c0 = head * width;
  const float* filt = (kind == 0 ? conv_q : kind == 1 ? conv_k : conv_v) + (size_t)c0 * K;
  const T* col = row + (kind == 0 ? q_off : kind == 1 ? k_off : v_off) + c0;
  const int first = cu_q[e], ctx = ctx_len[e], p = positions[t];
  const bool alone = cu_q[e + 1] - first == 1;
  float* tail = state + (size_t)slot * state_stride + tail_off + (kind == 0 ? 0 : kind == 1 ? Cq : 2 * Cq) + c0;
  auto convolved = [&](int c, float (&acc)[VEC]) {
#pragma unroll
    for (int k = 0; k < VEC; ++k) acc[k] = 0.f;
    if (TAPS == 4) {
      float x[4][VEC];
      float4 f[VEC];
#pragma unroll
      for (int k = 0; k < VEC; ++k) f[k] = *reinterpret_cast<const float4*>(filt + (size_t)(c + k) * 4);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int k = 0; k < VEC; ++k) x[j][k] = 0.f;
        if (t - j >= first) {
          DpVec<T, VEC>::load(col - (size_t)j * proj_stride + c, x[j]);
        } else if (p - j >= 0) {         // an input of an earlier step
          const float* src = tail + (size_t)(p - j - ctx + 3) * C + c;
#pragma unroll
          for (int k = 0; k < VEC; ++k) x[j][k] = src[k];
        }
      }
      if (alone) {                       // place 2 - j of the record holds input j from now on
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
          for (int k = 0; k < VEC; ++k) tail[(size_t)(2 - j) * C + c + k] = x[j][k];
      }
#pragma unroll
      for (int k = 0; k < VEC; ++k) {    // oldest input first
        acc[k] = fmaf(f[k].x, x[3][k], acc[k]);
        acc[k] = fmaf(f[k].y, x[2][k], acc[k]);
        acc[k] = fmaf(f[k].z, x[1][k], acc[k]);
        acc[k] = dr_silu(fmaf(f[k].w, x[0][k], acc[k]));
      }
      return;
    }
    for (int j = K - 1; j >= 0; --j) {   // oldest input first
      float x[VEC];
#pragma unroll
      for (int k = 0; k < VEC; ++k) x[k] = 0.f;
      if (t - j >= first) {
        DpVec<T, VEC>::load(col - (size_t)j * proj_stride + c, x);
      } else if (p - j >= 0) {           // an input of an earlier step
        const float* src = tail + (size_t)(p - j - ctx + K - 1) * C + c;
#pragma unroll
        for (int k = 0; k < VEC; ++k) x[k] = src[k];
      }
      if (alone && j < K - 1) {          // place K - 2 - j of the record holds this input from now on
        float* dst = tail + (size_t)(K - 2 - j) * C + c;
#pragma unroll
        for (int k = 0; k < VEC; ++k) dst[k] = x[k];
      }
#pragma unroll
      for (int k = 0; k < VEC; ++k) acc[k] = fmaf(filt[(size_t)(c + k) * K + K - 1 - j], x[k], acc[k]);
    }
#pragma unroll
    for (int k = 0; k < VEC; ++k) acc[k] = dr_silu(acc[k]);
  };
  if (kind == 2) {
    for (int c = VEC * lane; c < width; c += 32 * VEC) {
      float y[VEC];
      convolved(c, y);
      dp_store<VEC>(vc + (size_t)t * Cv + c0 + c, y);
    }
    return;
  }
  float y[PIECES][VEC], ss = 0.f;        // unit vectors
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int c = (i * 32 + lane) * VEC;
    if (c < width) {
      convolved(c, y[i]);
#pragma unroll
      for (int k = 0; k < VEC; ++k) ss = fmaf(y[i][k], y[i][k], ss);
    }
  }
  ss = warp_sum(ss);
  float inv = 1.0f / sqrtf(ss + 1e-6f);
  if (kind == 0) inv *= 1.0f / sqrtf((float)s.dk);
  float* dst = (kind == 0 ? qn : kn) + (size_t)t * Cq + c0;
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int c = (i * 32 + lane) * VEC;
    if (c < width) {
#pragma unroll
      for (int k = 0; k < VEC; ++k) y[i][k] *= inv;
      dp_store<VEC>(dst + c, y[i]);
    }
  }
}

// TAPS 4: filters of four taps at 16-byte boundaries, all loads of a channel's convolution on their way at once; 0: any.
// RUN: neighbouring tokens a warp takes of a head.  With more than one (long portions, four taps) the filter's numbers, twice as many
// bytes as a token's inputs, are read once for them and the inputs once and not four times, all of them on their way
// together; tokens at an entry's start are served one by one.  2,047 tokens of two entries, 12 heads on 2 of 128: 25 us a token
// at a time, 18 with eight.
template <typename T, int VEC, int TAPS, int RUN>
__global__ void __launch_bounds__(32 * DP_TOKENS)
delta_prepare_kernel(const T* __restrict__ proj, long proj_stride, int q_off, int k_off, int v_off, int b_off,
                     const T* __restrict__ a_in, long a_stride, const float* __restrict__ conv_q,
                     const float* __restrict__ conv_k, const float* __restrict__ conv_v,
                     const float* __restrict__ A_log, const float* __restrict__ dt_bias, float* state, long state_stride,
                     long tail_off, const int* __restrict__ token_req, const int* __restrict__ cu_q,
                     const int* __restrict__ ctx_len, const int* __restrict__ req_slot, const int* __restrict__ positions,
                     float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ vc, float* __restrict__ beta,
                     float* __restrict__ g, int num_tokens, DeltaShape s) {
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int lane = threadIdx.x & 31, t_first = (blockIdx.x * DP_TOKENS + (threadIdx.x >> 5)) * RUN;
  const int Cq = s.Hk * s.dk, Cv = s.H * s.dv, C = 2 * Cq + Cv, K = s.taps;
  const int unit = blockIdx.y;
  if (RUN > 1 && unit < 2 * s.Hk + s.H && t_first + RUN <= num_tokens) {
    const int e = token_req[t_first], slot = e >= 0 ? req_slot[e] : -1;
    const int kind = unit < s.Hk ? 0 : unit < 2 * s.Hk ? 1 : 2, head = unit - (kind == 0 ? 0 : kind == 1 ? s.Hk : 2 * s.Hk);
    const int width = kind == 2 ? s.dv : s.dk, c0 = head * width;
    // all of one live entry, and so are the three inputs before them; heads of at most 32 accesses of a warp
    if (slot >= 0 && token_req[t_first + RUN - 1] == e && t_first - 3 >= cu_q[e] && width <= 32 * VEC) {
      const float* filt = (kind == 0 ? conv_q : kind == 1 ? conv_k : conv_v) + (size_t)c0 * 4;
      const int c = VEC * lane;
      const bool on = c < width;
      const T* col = proj + (size_t)(t_first - 3) * proj_stride + (kind == 0 ? q_off : kind == 1 ? k_off : v_off) + c0 + c;
      float x[RUN + 3][VEC], f[VEC][4];
#pragma unroll
      for (int j = 0; j < RUN + 3; ++j) {
#pragma unroll
        for (int k = 0; k < VEC; ++k) x[j][k] = 0.f;
        if (on) DpVec<T, VEC>::load(col + (size_t)j * proj_stride, x[j]);
      }
#pragma unroll
      for (int k = 0; k < VEC; ++k) {
        const float4 w = on ? *reinterpret_cast<const float4*>(filt + (size_t)(c + k) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        f[k][0] = w.x;
        f[k][1] = w.y;
        f[k][2] = w.z;
        f[k][3] = w.w;
      }
#pragma unroll
      for (int i = 0; i < RUN; ++i) {
        float y[VEC];
#pragma unroll
        for (int k = 0; k < VEC; ++k) {      // oldest input first
          y[k] = 0.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) y[k] = fmaf(f[k][j], x[i + j][k], y[k]);
        }
        ll_silu_all<VEC>(y);
        if (kind == 2) {
          if (on) dp_store<VEC>(vc + (size_t)(t_first + i) * Cv + c0 + c, y);
          continue;
        }
        float ss = 0.f;                      // unit vectors
#pragma unroll
        for (int k = 0; k < VEC; ++k) ss = fmaf(y[k], y[k], ss);
        ss = warp_sum(ss);
        float inv = 1.0f / sqrtf(ss + 1e-6f);
        if (kind == 0) inv *= 1.0f / sqrtf((float)s.dk);
#pragma unroll
        for (int k = 0; k < VEC; ++k) y[k] *= inv;
        if (on) dp_store<VEC>((kind == 0 ? qn : kn) + (size_t)(t_first + i) * Cq + c0 + c, y);
      }
      return;
    }
  }
#pragma unroll 1
  for (int t = t_first; t < min(t_first + RUN, num_tokens); ++t)
    delta_prepare_token<T, VEC, TAPS>(t, unit, lane, proj, proj_stride, q_off, k_off, v_off, b_off, a_in, a_stride, conv_q, conv_k,
                                      conv_v, A_log, dt_bias, state, state_stride, tail_off, token_req, cu_q, ctx_len, req_slot,
                                      positions, qn, kn, vc, beta, g, s);
}

// The record's last taps - 1 inputs after the step: inputs of this step where it brought enough tokens,
// else what the record held, moved up.  A thread owns a channel and goes from the oldest place to the
// newest, reading only places above the one it writes.
template <typename T>
__global__ void delta_conv_update_kernel(const T* __restrict__ proj, long proj_stride, int q_off, int k_off, int v_off,
                                         float* __restrict__ state, long state_stride, long tail_off,
                                         const int* __restrict__ cu_q, const int* __restrict__ ctx_len,
                                         const int* __restrict__ req_slot, DeltaShape s) {
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int e = blockIdx.x;
  const int slot = req_slot[e];
  if (slot < 0) return;
  const int Cq = s.Hk * s.dk, Cv = s.H * s.dv, C = 2 * Cq + Cv, K = s.taps;
  const int first = cu_q[e], L = cu_q[e + 1] - first, ctx = ctx_len[e];
  if (L == 1) return;          // (delta_prepare has done it)
  float* tail = state + (size_t)slot * state_stride + tail_off;
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x) {
    const int col = c < Cq ? q_off + c : c < 2 * Cq ? k_off + c - Cq : v_off + c - 2 * Cq;
    for (int i = 0; i < K - 1; ++i) {
      const int pos = ctx + L - (K - 1) + i;   // the position whose input place i holds afterwards
      float x = 0.f;
      if (pos >= ctx) x = to_f32<T>(proj[(size_t)(first + pos - ctx) * proj_stride + col]);
      else if (pos >= 0) x = tail[(size_t)(i + L) * C + c];
      tail[(size_t)i * C + c] = x;
    }
  }
}

// The scan.  What bounds it is the chain of dependent operations from one token to the next of a value column, so
// a column is spread over as many lanes as leave each lane DR_NR = 4 key channels (8 for heads of more than 128
// channels): two short multiply-add chains and log2(LANES) shuffle steps a sum, all columns of all heads resident
// at once, and enough warps a scheduler to fill the gaps that one warp's dependent instructions leave (a capture
// of the 8-channel version showed 0.27 instructions issued a cycle and scheduler with 1.3 warps each).  A block of 128 threads owns 128 / LANES value columns of one (entry, head); lane l holds
// channels l, l + LANES, ....  The tokens' q, k, decay, v and beta come through shared memory in chunks of DR_CH
// tokens, copied asynchronously (cp.async) a chunk ahead, so that the scan waits for memory once a chunk and meets
// no barrier between the tokens of a chunk; rows are padded with zeros to LANES * DR_NR channels so that the inner
// loops carry no bounds checks.  Sums run in two interleaved chains and then over the lanes, in a fixed order.
// The read-out is taken from the state before the token's write plus the write's own share (see the loop), which
// is the same number as reading the state after the write.
#define DR_THREADS 128
#define DR_CH 16
__device__ __forceinline__ void dr_copy4(float* dst_smem, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void dr_copy16(float* dst_smem, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
template <int DR_LANES, int DR_NR>
__global__ void __launch_bounds__(DR_THREADS)
delta_recurrence_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vc,
                        const float* __restrict__ beta, const float* __restrict__ g, float* __restrict__ state,
                        long state_stride, const int* __restrict__ cu_q, const int* __restrict__ req_slot,
                        float* __restrict__ o, DeltaShape s) {
  extern __shared__ float sm[];   // two buffers of [q | k | decay][DR_CH][dkp], v [DR_CH][DR_COLS], beta, head decay [DR_CH]
  constexpr int DR_COLS = DR_THREADS / DR_LANES;
  constexpr int dkp = DR_LANES * DR_NR;
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int e = blockIdx.x, h = blockIdx.y;
  const int tid = threadIdx.x, l = tid % DR_LANES, cl = tid / DR_LANES;
  const int col0 = blockIdx.z * DR_COLS, col = col0 + cl;
  const bool live_col = col < s.dv;
  const int first = cu_q[e], last = cu_q[e + 1];
  const int slot = req_slot[e];
  const int Cq = s.Hk * s.dk, Cv = s.H * s.dv, dk = s.dk;
  if (slot < 0) {
    if (live_col && l == 0)
      for (int t = first; t < last; ++t) o[(size_t)t * Cv + (size_t)h * s.dv + col] = 0.f;
    return;
  }
  const int hk = h / (s.H / s.Hk);
  const int ng = s.per_channel ? s.H * dk : s.H;
  const bool pc = s.per_channel != 0;
  constexpr int buf_floats = DR_CH * (3 * dkp + DR_COLS + 2);
  const bool wide = (dk % 4) == 0 && (Cq % 4) == 0 && (ng % 4 == 0 || !pc) &&
                    (((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)g) % 16) == 0;
  float* S_ptr = state + (size_t)slot * state_stride + (size_t)h * dk * s.dv;
  float S[DR_NR];
#pragma unroll
  for (int i = 0; i < DR_NR; ++i) {
    const int c = l + DR_LANES * i;
    S[i] = (live_col && c < dk) ? S_ptr[(size_t)col * dk + c] : 0.f;
  }
  // the padding channels dk .. dkp - 1 of every row: zeros, written once (the copies never touch them)
  for (int idx = tid; idx < 2 * 3 * DR_CH * (dkp - dk); idx += DR_THREADS) {
    const int row = idx / (dkp - dk), c = dk + idx % (dkp - dk);
    const int buf = row / (3 * DR_CH), rr = row % (3 * DR_CH);
    sm[(size_t)buf * buf_floats + rr * dkp + c] = 0.f;
  }
  auto load_chunk = [&](int t0, int buf) {
    float* b = sm + (size_t)buf * buf_floats;
    const int nt = min(DR_CH, last - t0);
    for (int i = 0; i < nt; ++i) {
      const float* qs = qn + (size_t)(t0 + i) * Cq + (size_t)hk * dk;
      const float* ks = kn + (size_t)(t0 + i) * Cq + (size_t)hk * dk;
      const float* gs = g + (size_t)(t0 + i) * ng + (size_t)h * dk;
      if (wide) {     // rows of a multiple of four channels at 16-byte addresses: four numbers a copy
        for (int c = tid * 4; c < dk; c += DR_THREADS * 4) {
          dr_copy16(b + i * dkp + c, qs + c);
          dr_copy16(b + (DR_CH + i) * dkp + c, ks + c);
          if (pc) dr_copy16(b + (2 * DR_CH + i) * dkp + c, gs + c);
        }
      } else {
        for (int c = tid; c < dk; c += DR_THREADS) {
          dr_copy4(b + i * dkp + c, qs + c);
          dr_copy4(b + (DR_CH + i) * dkp + c, ks + c);
          if (pc) dr_copy4(b + (2 * DR_CH + i) * dkp + c, gs + c);
        }
      }
    }
    float* bv = b + 3 * DR_CH * dkp;
    for (int idx = tid; idx < nt * DR_COLS; idx += DR_THREADS) {
      const int i = idx / DR_COLS, cc = idx % DR_COLS;
      if (col0 + cc < s.dv) dr_copy4(bv + idx, vc + (size_t)(t0 + i) * Cv + (size_t)h * s.dv + col0 + cc);
      else bv[idx] = 0.f;
    }
    if (tid < nt) {
      dr_copy4(bv + DR_CH * DR_COLS + tid, beta + (size_t)(t0 + tid) * s.H + h);
      if (!pc) dr_copy4(bv + DR_CH * DR_COLS + DR_CH + tid, g + (size_t)(t0 + tid) * ng + h);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (first < last) load_chunk(first, 0);
  for (int t0 = first; t0 < last; t0 += DR_CH) {
    const int buf = ((t0 - first) / DR_CH) & 1;
    const bool more = t0 + DR_CH < last;
    if (more) {
      load_chunk(t0 + DR_CH, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* b = sm + (size_t)buf * buf_floats;
    const float* bv = b + 3 * DR_CH * dkp;
    const int nt = min(DR_CH, last - t0);
    for (int i = 0; i < nt; ++i) {
      const float* sq = b + i * dkp + l;
      const float* sk = b + (DR_CH + i) * dkp + l;
      const float* sg = b + (2 * DR_CH + i) * dkp + l;
      const float v = bv[i * DR_COLS + cl];
      const float bt = bv[DR_CH * DR_COLS + i];
      const float gh = pc ? 1.f : bv[DR_CH * DR_COLS + DR_CH + i];
      // Both sums of a token read the state as the token before left it: with S' = diag(g) S + k u^T,
      //   S^T (g . k) is what u needs, and o = S'^T q = S^T (g . q) + u (k . q),
      // so the two reductions over the lanes (and the one of k . q, which does not touch the state) run side
      // by side, and the chain from token to token is one reduction, not two.
      float kr[DR_NR], dec[DR_NR];
      float d0 = 0.f, d1 = 0.f, o0 = 0.f, o1 = 0.f, kq = 0.f;
#pragma unroll
      for (int j = 0; j < DR_NR; ++j) {
        kr[j] = sk[DR_LANES * j];
        dec[j] = pc ? sg[DR_LANES * j] : gh;
        const float qv = sq[DR_LANES * j];
        const float gk = dec[j] * kr[j], gq = dec[j] * qv;
        kq = fmaf(kr[j], qv, kq);
        if (j & 1) {
          d1 = fmaf(S[j], gk, d1);
          o1 = fmaf(S[j], gq, o1);
        } else {
          d0 = fmaf(S[j], gk, d0);
          o0 = fmaf(S[j], gq, o0);
        }
      }
      float dot = d0 + d1, oq = o0 + o1;
#pragma unroll
      for (int x = 1; x < DR_LANES; x <<= 1) {
        dot += __shfl_xor_sync(0xffffffffu, dot, x);
        oq += __shfl_xor_sync(0xffffffffu, oq, x);
        kq += __shfl_xor_sync(0xffffffffu, kq, x);
      }
      const float u = bt * (v - dot);
      oq = fmaf(u, kq, oq);
#pragma unroll
      for (int j = 0; j < DR_NR; ++j) S[j] = fmaf(dec[j], S[j], kr[j] * u);
      if (live_col && l == 0) o[(size_t)(t0 + i) * Cv + (size_t)h * s.dv + col] = oq;
    }
    __syncthreads();   // everyone is done with this buffer before the chunk after the next is copied into it
  }
#pragma unroll
  for (int i = 0; i < DR_NR; ++i) {
    const int c = l + DR_LANES * i;
    if (live_col && c < dk) S_ptr[(size_t)col * dk + c] = S[i];
  }
}

// out[t, h*dv + j] = o / sqrt(mean_j(o^2) + eps) * w[j] * act(gate[t, h*dv + j]); act: 0 SiLU, 1 sigmoid.  A warp a (token,
// head), VEC numbers a lane and access; heads of up to 256 numbers stay in registers between the sum and the output.
template <typename T, int VEC>
__global__ void delta_out_kernel(T* __restrict__ out, const float* __restrict__ o, const float* __restrict__ w,
                                 const T* __restrict__ gate, long gate_stride, float eps, int num_pairs, int H, int dv,
                                 int gate_act) {
  constexpr int PIECES = 8 / VEC;
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int pair = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (pair >= num_pairs) return;
  const int lane = threadIdx.x & 31;
  const int t = pair / H, h = pair % H;
  const float* src = o + (size_t)pair * dv;
  const T* gt = gate + (size_t)t * gate_stride + (size_t)h * dv;
  T* dst = out + (size_t)pair * dv;
  float x[PIECES][VEC];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int c = (i * 32 + lane) * VEC;
    if (c < dv) {
      DpVec<float, VEC>::load(src + c, x[i]);
#pragma unroll
      for (int k = 0; k < VEC; ++k) ss = fmaf(x[i][k], x[i][k], ss);
    }
  }
  for (int c = 256 + lane; c < dv; c += 32) ss = fmaf(src[c], src[c], ss);
  ss = warp_sum(ss);
  const float inv = 1.0f / sqrtf(ss / (float)dv + eps);
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int c = (i * 32 + lane) * VEC;
    if (c < dv) {
      float z[VEC];
      T r[VEC];
      DpVec<T, VEC>::load(gt + c, z);
#pragma unroll
      for (int k = 0; k < VEC; ++k)
        r[k] = from_f32<T>(x[i][k] * inv * w[c + k] * (gate_act == 0 ? dr_silu(z[k]) : dr_sigmoid(z[k])));
      if (VEC == 4 && sizeof(T) == 2) *reinterpret_cast<uint2*>(dst + c) = *reinterpret_cast<const uint2*>(r);
      else if (VEC == 4) *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<const uint4*>(r);
      else dst[c] = r[0];
    }
  }
  for (int c = 256 + lane; c < dv; c += 32) {
    const float z = to_f32<T>(gt[c]);
    dst[c] = from_f32<T>(src[c] * inv * w[c] * (gate_act == 0 ? dr_silu(z) : dr_sigmoid(z)));
  }
}

extern "C" int ll_delta_prepare(int dtype, const void* proj, long proj_stride, int q_off, int k_off, int v_off,
                                int b_off, const void* a_in, long a_stride, const float* conv_q, const float* conv_k,
                                const float* conv_v, const float* A_log, const float* dt_bias, float* state,
                                long state_stride, long tail_off, const int* token_req, const int* cu_q,
                                const int* ctx_len, const int* req_slot, const int* positions, float* qn, float* kn,
                                float* vc, float* beta, float* g, int num_tokens, int num_entries, int H, int Hk, int dk,
                                int dv, int taps, int per_channel, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  if (H <= 0 || Hk <= 0 || H % Hk || dk <= 0 || dv <= 0 || taps < 1) return (int)cudaErrorInvalidValue;
  DeltaShape s{H, Hk, dk, dv, taps, per_channel};
  const int C = 2 * Hk * dk + H * dv;
  const int units = 2 * Hk + H + 1 + (per_channel ? H : 1);
  // four channels a lane and access: heads, columns and rows at multiples of four numbers
  const int esz = dtype == LL_DTYPE_F32 ? 4 : 2;
  const bool vec = dk % 4 == 0 && dv % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && v_off % 4 == 0 && proj_stride % 4 == 0 &&
                   (uintptr_t)proj % (4 * esz) == 0 && ((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)vc) % 16 == 0;
  const bool four = vec && taps == 4 && ((uintptr_t)conv_q | (uintptr_t)conv_k | (uintptr_t)conv_v) % 16 == 0;
  // eight tokens a warp where the portions are long enough for most warps to have a run and there are enough of them (2,047 tokens
  // of two entries 18 us and 25 one by one; a step of many single tokens would walk through eight of them in turn)
  const int run = four && num_tokens >= 512 && num_tokens >= 32 * (long)num_entries ? 8 : 1;
  const dim3 grid((num_tokens + DP_TOKENS * run - 1) / (DP_TOKENS * run), units), block(32 * DP_TOKENS);
#define DP_ARGS                                                                                                             \
  grid, block, 0, stream, (const T*)proj, proj_stride, q_off, k_off, v_off, b_off, (const T*)a_in, a_stride, conv_q, conv_k, \
      conv_v, A_log, dt_bias, state, state_stride, tail_off, token_req, cu_q, ctx_len, req_slot, positions, qn, kn, vc, beta, \
      g, num_tokens, s
  LL_DISPATCH_DTYPE(dtype, {
    if (run > 1) ll_launch(delta_prepare_kernel<T, 4, 4, 8>, DP_ARGS);
    else if (four) ll_launch(delta_prepare_kernel<T, 4, 4, 1>, DP_ARGS);
    else if (vec) ll_launch(delta_prepare_kernel<T, 4, 0, 1>, DP_ARGS);
    else ll_launch(delta_prepare_kernel<T, 1, 0, 1>, DP_ARGS);
    if (taps > 1 && num_tokens != num_entries) {      // (as many tokens as entries: one each)
      const int by = (C + 255) / 256;
      ll_launch(delta_conv_update_kernel<T>, dim3(num_entries, by < 8 ? by : 8), dim3(256), 0, stream, (const T*)proj,
                proj_stride, q_off, k_off, v_off, state, state_stride, tail_off, cu_q, ctx_len, req_slot, s);
    }
  });
#undef DP_ARGS
  return LL_LAUNCH_RESULT();
}

extern "C" int ll_delta_recurrence(const float* qn, const float* kn, const float* vc, const float* beta,
                                   const float* g, float* state, long state_stride, const int* cu_q,
                                   const int* req_slot, float* o, int num_entries, int H, int Hk, int dk, int dv,
                                   int per_channel, cudaStream_t stream) {
  if (num_entries <= 0) return 0;
  if (H <= 0 || Hk <= 0 || H % Hk || dk <= 0 || dk > 256 || dv <= 0) return (int)cudaErrorInvalidValue;
  DeltaShape s{H, Hk, dk, dv, 0, per_channel};
#define DR_LAUNCH(LANES, NR)                                                                                        \
  do {                                                                                                              \
    constexpr int cols = DR_THREADS / LANES;                                                                        \
    dim3 grid(num_entries, H, (dv + cols - 1) / cols), block(DR_THREADS);                                           \
    const size_t smem = sizeof(float) * 2 * DR_CH * (3 * (size_t)LANES * NR + cols + 2);                            \
    if (smem > 48 * 1024)                                                                                           \
      cudaFuncSetAttribute(delta_recurrence_kernel<LANES, NR>, cudaFuncAttributeMaxDynamicSharedMemorySize,         \
                           (int)smem);                                                                              \
    ll_launch(delta_recurrence_kernel<LANES, NR>, grid, block, smem, stream, qn, kn, vc, beta, g, state,            \
              state_stride, cu_q, req_slot, o, s);                                                                  \
  } while (0)
  if (dk <= 4) DR_LAUNCH(1, 4);
  else if (dk <= 8) DR_LAUNCH(2, 4);
  else if (dk <= 16) DR_LAUNCH(4, 4);
  else if (dk <= 32) DR_LAUNCH(8, 4);
  else if (dk <= 64) DR_LAUNCH(16, 4);
  else if (dk <= 128) DR_LAUNCH(32, 4);
  else DR_LAUNCH(32, 8);
#undef DR_LAUNCH
  return LL_LAUNCH_RESULT();
}

extern "C" int ll_delta_out(int dtype, void* out, const float* o, const float* w, const void* gate, long gate_stride,
                            float eps, int num_tokens, int H, int dv, int gate_act, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  const int pairs = num_tokens * H;
  const int esz = dtype == LL_DTYPE_F32 ? 4 : 2;
  const bool vec = dv % 4 == 0 && gate_stride % 4 == 0 && ((uintptr_t)gate | (uintptr_t)out) % (4 * esz) == 0 &&
                   (uintptr_t)o % 16 == 0;
  LL_DISPATCH_DTYPE(dtype, {
    if (vec)
      ll_launch(delta_out_kernel<T, 4>, dim3((pairs + 3) / 4), dim3(128), 0, stream, (T*)out, o, w, (const T*)gate, gate_stride,
                eps, pairs, H, dv, gate_act);
    else
      ll_launch(delta_out_kernel<T, 1>, dim3((pairs + 3) / 4), dim3(128), 0, stream, (T*)out, o, w, (const T*)gate, gate_stride,
                eps, pairs, H, dv, gate_act);
  });
  return LL_LAUNCH_RESULT();
}

// A step of single tokens in one launch, a CTA a (token, head): what delta_prepare, delta_recurrence and delta_out do, and the second
// products of decays and gates that come through a few numbers (decay_rank, gate_rank).  For one token those are five launches in a
// chain of 1.6 to 3 us each; for many the scan's loop over chunks of 16 tokens is made for more than one.  D: channels of a key and of
// a value head.  What does not depend on the step (filters, the ranks' matrices) is asked for before the wait; then a thread's part of
// the state is on its way, all at once, while
//   warp 0, 1, 2   make the head's q, k and v (four channels a lane, as delta_prepare_token),
//   the warps from the fifth on the decays of the key channels and (for heads of 128 the first four) the gates, a number a thread.
// A thread has 16 channels of four columns (heads of 64: of one), which share what it reads of q, k and decays: 1,024 threads with a
// column each read four times as much of shared memory, and took 9.1 us for a token and 14.4 for 16 (12 heads; this way 7.8 and 8.5).
// The heads that read the same q and k are a cluster: their inputs in the record move up when all of them have been read.  Every sum
// but the ranks' has the order that it has in the kernels one by one, so that a token's bits do not depend on what it shares a step
// with.  Whole layers of 12 heads, launches one by one / this way: 1 token 18.6 / 14.5 us, 16 tokens 35.1 / 18.7, 64 tokens 90 / 43.
template <typename T> struct DeltaStep {
  const T *proj, *a_in, *gate;           // a_in, gate: rows of their own numbers, or of the ranks' inputs
  const T *w_a, *w_g;                    // [H * D or H, a_rank], [H * D, g_rank], or null
  long stride, a_stride, gate_stride;
  int q_off, k_off, v_off, b_off, a_rank, g_rank;
  const float *conv_q, *conv_k, *conv_v, *A_log, *dt_bias, *norm;
  float* state;
  long state_stride, tail_off;
  const int *req_slot, *positions;
  T* y;
  float eps;
  int H, Hk, per_channel, gate_act;
};

// pieces of 16 bytes from one row of a rank's matrix to the next in shared memory: odd, so that neighbouring threads' rows lie in
// different banks
template <typename T> __host__ __device__ __forceinline__ int ds_pitch(int rank) { return (rank * (int)sizeof(T) / 16) | 1; }
template <typename T> __device__ __forceinline__ float ds_dot(const uint4* row, const float* x, int rank) {
  constexpr int N = 16 / (int)sizeof(T);
  float acc[4] = {};
#pragma unroll 4
  for (int p = 0; p < rank / N; ++p) {
    const uint4 w = row[p];
    const T* v = reinterpret_cast<const T*>(&w);
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      const float4 x4 = *reinterpret_cast<const float4*>(x + p * N + i);
      acc[0] = fmaf(to_f32<T>(v[i]), x4.x, acc[0]);
      acc[1] = fmaf(to_f32<T>(v[i + 1]), x4.y, acc[1]);
      acc[2] = fmaf(to_f32<T>(v[i + 2]), x4.z, acc[2]);
      acc[3] = fmaf(to_f32<T>(v[i + 3]), x4.w, acc[3]);
    }
  }
  return (acc[0] + acc[1]) + (acc[2] + acc[3]);
}

template <typename T, int D>
__global__ void __launch_bounds__(256, 2)
delta_step_kernel(DeltaStep<T> s) {
  // lanes of delta_recurrence that a thread stands for, threads that share a column, columns a thread and their distance
  constexpr int VL = 4, TPC = D / 16, THREADS = 256, NC = D * TPC / THREADS, STEP = D / NC;
  extern __shared__ __align__(16) uint4 mat_a[];               // the rows of w_a, then of w_g
  __shared__ __align__(16) float qs[D], ks[D], vs[D], gs[D], zs[D], os[D];
  __shared__ __align__(16) float ax[128], gx[128];
  __shared__ float beta;
  LL_PDL_TRIGGER();
  const int e = blockIdx.x, h = blockIdx.z, hk = h / (s.H / s.Hk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_decay = tid - 128, n_gate = D == 128 ? tid : tid - 192;      // the key channel or value column of a thread
  const bool is_decay = n_decay >= 0 && n_decay < D, is_gate = n_gate >= 0 && n_gate < D;
  const int drow = s.per_channel ? h * D + n_decay : h;
  // before the wait: filters and the head's rows of the ranks' matrices
  float4 f[4];
  constexpr int width = D / 4;                                 // lanes of warps 0 to 2 with channels
  const float* filt = warp == 0 ? s.conv_q + (size_t)hk * D * 4 : warp == 1 ? s.conv_k + (size_t)hk * D * 4 : s.conv_v + (size_t)h * D * 4;
  if (warp < 3 && lane < width) {
#pragma unroll
    for (int k = 0; k < 4; ++k) f[k] = reinterpret_cast<const float4*>(filt)[lane * 4 + k];
  }
  const int pitch_a = ds_pitch<T>(s.a_rank), pitch_g = ds_pitch<T>(s.g_rank), rows_a = s.per_channel ? D : 1;
  uint4* mat_g = mat_a + (s.a_rank > 0 ? rows_a * pitch_a : 0);
  auto fetch = [&](uint4* dst, int pitch, const T* src, int rank, int rows) {
    const int pieces = rank * (int)sizeof(T) / 16;
    for (int i = tid; i < rows * pieces; i += THREADS) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(dst + i / pieces * pitch + i % pieces);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(reinterpret_cast<const uint4*>(src) + i) : "memory");
    }
  };
  if (s.a_rank > 0) fetch(mat_a, pitch_a, s.w_a + (size_t)h * rows_a * s.a_rank, s.a_rank, rows_a);
  if (s.g_rank > 0) fetch(mat_g, pitch_g, s.w_g + (size_t)h * D * s.g_rank, s.g_rank, D);
  const int col = tid / TPC, l = tid % TPC;
  const float a_log = s.A_log[h], bias = is_decay ? s.dt_bias[drow] : 0.f, weight = s.norm[tid % D];
  LL_PDL_WAIT();
  const int slot = s.req_slot[e], t = e, p = s.positions[t];   // (an entry a token)
  T* yrow = s.y + (size_t)t * s.H * D + (size_t)h * D;
  if (slot < 0) {                                              // a padding entry (the cluster's CTAs have the same one)
    if (tid < D) yrow[tid] = from_f32<T>(0.f);
    return;
  }
  float* rec = s.state + (size_t)slot * s.state_stride;
  float* srow = rec + ((size_t)h * D + col) * D + l * VL;
  float S[NC][4][VL];                                          // columns col + n STEP, key channels j D / 4 + l VL + i
#pragma unroll
  for (int n = 0; n < NC; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"      // (in this place: they are the most bytes)
                   : "=f"(S[n][j][0]), "=f"(S[n][j][1]), "=f"(S[n][j][2]), "=f"(S[n][j][3])
                   : "l"(srow + (size_t)n * STEP * D + j * (D / 4)));
  const T* row = s.proj + (size_t)t * s.stride;
  for (int i = tid; i < s.a_rank; i += THREADS) ax[i] = to_f32<T>(s.a_in[(size_t)t * s.a_stride + i]);
  for (int i = tid; i < s.g_rank; i += THREADS) gx[i] = to_f32<T>(s.gate[(size_t)t * s.gate_stride + i]);
  const int Cq = s.Hk * D, C = 2 * Cq + s.H * D;
  const int c = 4 * lane, chan = warp == 0 ? hk * D + c : warp == 1 ? Cq + hk * D + c : 2 * Cq + h * D + c;      // among the record's inputs
  if (warp < 3 && lane < width) {
    const float* tail = rec + s.tail_off + chan;
    float x[4][4];
    DpVec<T, 4>::load(row + (warp == 0 ? s.q_off + hk * D : warp == 1 ? s.k_off + hk * D : s.v_off + h * D) + c, x[0]);
#pragma unroll
    for (int j = 1; j < 4; ++j) DpVec<float, 4>::load(tail + (size_t)(3 - j) * C, x[j]);      // inputs of earlier steps
#pragma unroll
    for (int j = 1; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) x[j][k] = p - j >= 0 ? x[j][k] : 0.f;
    float acc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {                              // oldest input first
      acc[k] = fmaf(f[k].x, x[3][k], 0.f);
      acc[k] = fmaf(f[k].y, x[2][k], acc[k]);
      acc[k] = fmaf(f[k].z, x[1][k], acc[k]);
      acc[k] = dr_silu(fmaf(f[k].w, x[0][k], acc[k]));
    }
    if (warp < 2) {                                            // unit vectors
      float ss = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) ss = fmaf(acc[k], acc[k], ss);
#pragma unroll
      for (int o = width / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(D == 128 ? 0xffffffffu : 0xffffu, ss, o);
      float inv = 1.0f / sqrtf(ss + 1e-6f);
      if (warp == 0) inv *= 1.0f / sqrtf((float)D);
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] *= inv;
    }
    float* dst = warp == 0 ? qs : warp == 1 ? ks : vs;
    *reinterpret_cast<float4*>(dst + c) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  } else if (tid == 96) {
    beta = dr_sigmoid(to_f32<T>(row[s.b_off + h]));
  }
  if (s.a_rank > 0 || s.g_rank > 0) {                          // the ranks' rows and inputs
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
  }
  if (is_decay) {
    const float a = s.a_rank > 0 ? round_to<T>(ds_dot<T>(mat_a + (s.per_channel ? n_decay * pitch_a : 0), ax, s.a_rank))
                                 : to_f32<T>(s.a_in[(size_t)t * s.a_stride + drow]);
    gs[n_decay] = expf(-expf(a_log) * dr_softplus(a + bias));
  }
  if (is_gate) {
    const float z = s.g_rank > 0 ? round_to<T>(ds_dot<T>(mat_g + n_gate * pitch_g, gx, s.g_rank))
                                 : to_f32<T>(s.gate[(size_t)t * s.gate_stride + (size_t)h * D + n_gate]);
    zs[n_gate] = s.gate_act == 0 ? dr_silu(z) : dr_sigmoid(z);
  }
  __syncthreads();
  asm volatile("barrier.cluster.arrive;" ::: "memory");        // this CTA has read the record's inputs of q and k
  // the token, as delta_recurrence has it and with its sums in its order: S^T (g . k) and S^T (g . q) side by side, then the write
  float dot[NC][VL] = {}, oq[NC][VL] = {}, d1[NC][VL] = {}, o1[NC][VL] = {}, kq[VL] = {};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int ch = j * (D / 4) + l * VL;
    const float4 k4 = *reinterpret_cast<const float4*>(ks + ch), q4 = *reinterpret_cast<const float4*>(qs + ch);
    const float4 g4 = *reinterpret_cast<const float4*>(gs + ch);
    const float kv[VL] = {k4.x, k4.y, k4.z, k4.w}, qv[VL] = {q4.x, q4.y, q4.z, q4.w}, gv[VL] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
    for (int i = 0; i < VL; ++i) {
      const float gk = gv[i] * kv[i], gq = gv[i] * qv[i];
      kq[i] = fmaf(kv[i], qv[i], kq[i]);
#pragma unroll
      for (int n = 0; n < NC; ++n) {
        if (j & 1) {
          d1[n][i] = fmaf(S[n][j][i], gk, d1[n][i]);
          o1[n][i] = fmaf(S[n][j][i], gq, o1[n][i]);
        } else {
          dot[n][i] = fmaf(S[n][j][i], gk, dot[n][i]);
          oq[n][i] = fmaf(S[n][j][i], gq, oq[n][i]);
        }
      }
    }
  }
  float k_q = (kq[0] + kq[1]) + (kq[2] + kq[3]), u[NC];
#pragma unroll
  for (int w = 1; w < TPC; w <<= 1) k_q += __shfl_xor_sync(0xffffffffu, k_q, w);
#pragma unroll
  for (int n = 0; n < NC; ++n) {
#pragma unroll
    for (int i = 0; i < VL; ++i) {
      dot[n][i] += d1[n][i];
      oq[n][i] += o1[n][i];
    }
    float d = (dot[n][0] + dot[n][1]) + (dot[n][2] + dot[n][3]), o = (oq[n][0] + oq[n][1]) + (oq[n][2] + oq[n][3]);
#pragma unroll
    for (int w = 1; w < TPC; w <<= 1) {
      d += __shfl_xor_sync(0xffffffffu, d, w);
      o += __shfl_xor_sync(0xffffffffu, o, w);
    }
    u[n] = beta * (vs[col + n * STEP] - d);
    if (l == 0) os[col + n * STEP] = fmaf(u[n], k_q, o);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int ch = j * (D / 4) + l * VL;
    const float4 k4 = *reinterpret_cast<const float4*>(ks + ch), g4 = *reinterpret_cast<const float4*>(gs + ch);
#pragma unroll
    for (int n = 0; n < NC; ++n)
      *reinterpret_cast<float4*>(srow + (size_t)n * STEP * D + j * (D / 4)) =
          make_float4(fmaf(g4.x, S[n][j][0], k4.x * u[n]), fmaf(g4.y, S[n][j][1], k4.y * u[n]), fmaf(g4.z, S[n][j][2], k4.z * u[n]),
                      fmaf(g4.w, S[n][j][3], k4.w * u[n]));
  }
  __syncthreads();
  if (tid < D) {      // norm and gate, as delta_out: every warp adds the squares up
    float ss = 0.f;
    if (lane < width) {
      const float4 v = *reinterpret_cast<const float4*>(os + 4 * lane);
      ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss);
    }
    ss = warp_sum(ss);
    yrow[tid] = from_f32<T>(os[tid] * (1.0f / sqrtf(ss / (float)D + s.eps)) * weight * zs[tid]);
  }
  asm volatile("barrier.cluster.wait;" ::: "memory");          // every head of the cluster has read them
  if (lane < width && (warp == 2 || (warp < 2 && h == hk * (s.H / s.Hk)))) {      // a place holds the input behind it from now on
    float* tail = rec + s.tail_off + chan;
    float own[4], old[4] = {};
    if (p >= 2) DpVec<float, 4>::load(tail + C, old);
    dp_store<4>(tail, old);
#pragma unroll
    for (int k = 0; k < 4; ++k) old[k] = 0.f;
    if (p >= 1) DpVec<float, 4>::load(tail + 2 * C, old);
    dp_store<4>(tail + C, old);
    DpVec<T, 4>::load(row + (warp == 0 ? s.q_off + hk * D : warp == 1 ? s.k_off + hk * D : s.v_off + h * D) + c, own);
    dp_store<4>(tail + 2 * C, own);
  }
}

// A step of one token an entry (which brings position ctx_len) with key and value heads of 64 or 128, four taps and at most eight
// heads that read the same q and k; a_in and gate: the ranks' inputs where w_a, w_g are not null.  Rows at multiples of four numbers,
// records, filters and ranks' rows at multiples of 16 bytes; the head's rows of w_a and w_g together at most DS_ROOM bytes.
#define DS_ROOM 40960
extern "C" int ll_delta_step(int dtype, const void* proj, long stride, int q_off, int k_off, int v_off, int b_off, const void* a_in,
                             long a_stride, const void* w_a, int a_rank, const void* gate, long gate_stride, const void* w_g,
                             int g_rank, const float* conv_q, const float* conv_k, const float* conv_v, const float* A_log,
                             const float* dt_bias, const float* norm, float* state, long state_stride, long tail_off,
                             const int* req_slot, const int* positions, void* y, float eps, int num_entries, int H,
                             int Hk, int d, int per_channel, int gate_act, cudaStream_t stream) {
  if (num_entries <= 0) return 0;
  const int esz = dtype == LL_DTYPE_F32 ? 4 : 2;
  if (H <= 0 || Hk <= 0 || H % Hk || H / Hk > 8 || H > 65535 || (d != 64 && d != 128) || a_rank < 0 || g_rank < 0 || a_rank > 128 ||
      g_rank > 128 || a_rank % 8 || g_rank % 8 || state_stride % 4 || tail_off % 4 || stride % 4 || (q_off | k_off | v_off) % 4 ||
      (uintptr_t)proj % (4 * esz) || ((uintptr_t)conv_q | (uintptr_t)conv_k | (uintptr_t)conv_v | (uintptr_t)state) % 16 ||
      ((uintptr_t)w_a | (uintptr_t)w_g) % 16)
    return (int)cudaErrorInvalidValue;
  LL_DISPATCH_DTYPE(dtype, {
    const size_t smem = 16 * ((a_rank > 0 ? (size_t)(per_channel ? d : 1) * ds_pitch<T>(a_rank) : 0) +
                              (g_rank > 0 ? (size_t)d * ds_pitch<T>(g_rank) : 0));
    if (smem > DS_ROOM) return (int)cudaErrorInvalidValue;
    const DeltaStep<T> s{(const T*)proj, (const T*)a_in, (const T*)gate, (const T*)w_a, (const T*)w_g, stride, a_stride, gate_stride,
                         q_off, k_off, v_off, b_off, a_rank, g_rank, conv_q, conv_k, conv_v, A_log, dt_bias, norm, state,
                         state_stride, tail_off, req_slot, positions, (T*)y, eps, H, Hk, per_channel, gate_act};
    if (d == 128) ll_launch_cluster(delta_step_kernel<T, 128>, dim3(num_entries, 1, H), dim3(256), smem, stream, H / Hk, s);
    else ll_launch_cluster(delta_step_kernel<T, 64>, dim3(num_entries, 1, H), dim3(256), smem, stream, H / Hk, s);
  });
  return LL_LAUNCH_RESULT();
}
