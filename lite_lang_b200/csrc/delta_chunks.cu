// The gated delta rule of prompt portions, 64 tokens at a time (what a chunk is: chunk_scan.cu), with one decay a head as written here or
// one a key channel (delta_solve_channels).
//
//     S <- a_t S;   u_t = beta_t (v_t - S^T k_t);   S <- S + k_t u_t^T;   o_t = S^T q_t
// With L(t, s) = beta_t G(t, s) (k_t . k_s), s < t, the values that a chunk writes are u = U - W S0 with
//     (1 + L) U = [beta_t v_t],   (1 + L) W = [beta_t G(t, -) k_t]
// and with M(t, s) = G(t, s) (q_t . k_s), s <= t, its read-outs are o_t = G(t, -) S0^T q_t + sum over s of M(t, s) u_s:
//   delta_solve    per (chunk, head): U, W and M; the system is solved in blocks of 16 tokens on tensor cores
//   delta_walk     per (entry, head, 16 value columns): the chunks in order, two products a chunk
//   delta_read     per (chunk, head): the read-outs
// All float32: products are made of bfloat16 terms that hold all 24 bits (mma_split.cuh), decays are running products of float64
// rounded once, nothing is divided.  A number that is not finite would show before its own token (0 times an infinity is NaN): a
// thread that finds such a U, W or read-out makes it again token by token, with multiply-adds.  (A state may have NaN where the
// walk by tokens has an infinity.)
#include "chunk_scan.cuh"
#include "tc05.cuh"

#define DC_BLOCK 16       // tokens of a block of the system
#define DC_LP (CS_C + 8)  // pitch of L's and M's terms
#define DC_TP (DC_BLOCK + 8)
#define DC_GP (CS_C + 4)

// A running product of decays: float64, rounded once, so that neither the steps' roundings nor products below 2^-100 lose bits.  (The sum
// of two float32 numbers, whose error term underflows there, is as fast in delta_solve and takes 1 us of 70 less in
// delta_solve_channels.)
struct DcProduct {
  double p = 1.0;
  __device__ __forceinline__ void times(double a) { p *= a; }
  __device__ __forceinline__ void times(const DcProduct& a) { p *= a.p; }
  __device__ __forceinline__ float value() const { return (float)p; }
};

// G(t, s) for s <= t of a chunk's tokens in gs [64][DC_GP], and pre[t] = a_0 ... a_t, by 256 threads: thread (s, quarter) makes 16
// tokens' products, from the products of s's own quarter and of whole quarters between.  av: the decays.
__device__ __forceinline__ void dc_gaps(const double* av, float* gs, float* pre, DcProduct* tail, DcProduct* whole) {
  const int s = threadIdx.x & 63, quarter = threadIdx.x >> 6, own = s >> 4;
  if (quarter == own) {
    DcProduct p;
    gs[s * DC_GP + s] = 1.f;
    for (int t = s + 1; t < 16 * own + 16; ++t) {
      p.times(av[t]);
      gs[t * DC_GP + s] = p.value();
    }
    tail[s] = p;
    if ((s & 15) == 0) {
      p.times(av[s]);
      whole[own] = p;
    }
  }
  __syncthreads();
  if (quarter > own) {
    DcProduct p = tail[s];
    for (int j = own + 1; j < quarter; ++j) p.times(whole[j]);
#pragma unroll 4
    for (int t = 16 * quarter; t < 16 * quarter + 16; ++t) {
      p.times(av[t]);
      gs[t * DC_GP + s] = p.value();
    }
  } else if (quarter == own) {                          // a_0 ... a_s
    DcProduct p;
    for (int j = 0; j < own; ++j) p.times(whole[j]);
    for (int t = 16 * own; t <= s; ++t) p.times(av[t]);
    pre[s] = p.value();
  }
}

__device__ __forceinline__ float dc_term_sum(const bf16* plane, int at) {      // the float32 number that three terms hold
  return to_f32<bf16>(plane[at]) + (to_f32<bf16>(plane[CS_C * DC_LP + at]) + to_f32<bf16>(plane[2 * CS_C * DC_LP + at]));
}

// Operands that are made once and read by many CTAs lie in memory as the MMA's second operand stands in a warp's registers: of a tile
// of 16 (the inner dimension) by 8 a lane has three terms of two pairs of neighbours along the inner dimension, the first two terms in
// 16 bytes, the third in 8 of a second array.  They come whole, by one bulk copy.
struct DcFrag {
  unsigned b[3][2];
};
template <int TILES> __device__ __forceinline__ void dc_frag_put(unsigned* base, int tile, int lane, const DcFrag& f) {
  reinterpret_cast<uint4*>(base)[tile * 32 + lane] = make_uint4(f.b[0][0], f.b[0][1], f.b[1][0], f.b[1][1]);
  reinterpret_cast<uint2*>(base + TILES * 128)[tile * 32 + lane] = make_uint2(f.b[2][0], f.b[2][1]);
}
template <int TILES> __device__ __forceinline__ void dc_frag_get(DcFrag& f, const unsigned* __restrict__ base, int tile, int lane) {
  const uint4 x = reinterpret_cast<const uint4*>(base)[tile * 32 + lane];
  const uint2 y = reinterpret_cast<const uint2*>(base + TILES * 128)[tile * 32 + lane];
  f.b[0][0] = x.x; f.b[0][1] = x.y; f.b[1][0] = x.z; f.b[1][1] = x.w; f.b[2][0] = y.x; f.b[2][1] = y.y;
}
// where term p of the number (inner, other) of a tile lies, in bfloat16 numbers
template <int TILES> __device__ __forceinline__ size_t dc_frag_at(int p, int tile, int inner, int other) {
  const int lane = (other & 7) * 4 + ((inner & 7) >> 1), q = (inner >> 3) & 1;
  return p < 2 ? (size_t)(tile * 32 + lane) * 8 + (p * 2 + q) * 2 + (inner & 1)
               : (size_t)TILES * 256 + (size_t)(tile * 32 + lane) * 4 + q * 2 + (inner & 1);
}
__device__ __forceinline__ unsigned dc_turned(unsigned x) {      // an 8 x 8 tile of bfloat16 numbers, its rows and columns exchanged
  unsigned y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

// One column of the system by forward substitution: x_t = b_t - sum over s < t of L(t, s) x_s, for columns with numbers that are not
// finite.  rhs: the column's number of the chunk's first row, stride `rs`; x by `put` and `get`.
template <typename G, typename P>
__device__ __forceinline__ void dc_again(const bf16* Lp, const float* rhs, long rs, int n, const float* bt, const float* pre, G get, P put) {
#pragma unroll 1
  for (int t = 0; t < CS_C; ++t) {
    float x = t < n ? rhs[(size_t)t * rs] * (pre != nullptr ? bt[t] * pre[t] : bt[t]) : 0.f;
#pragma unroll 1
    for (int s = 0; s < t; ++s) x = fmaf(-dc_term_sum(Lp, t * DC_LP + s), get(s), x);
    put(t, x);
  }
}
template <int DK> __device__ __noinline__ void dc_again_w(const bf16* Lp, const float* rhs, long rs, int n, const float* bt,
                                                          const float* pre, unsigned* wt, int ch) {
  constexpr int TILES = DK / 2;
  auto at = [&](int p, int t) { return dc_frag_at<TILES>(p, ch / 16 * 8 + t / 8, ch & 15, t & 7); };
  bf16* x = reinterpret_cast<bf16*>(wt);
  dc_again(Lp, rhs, rs, n, bt, pre, [&](int t) { return to_f32<bf16>(x[at(0, t)]) + (to_f32<bf16>(x[at(1, t)]) + to_f32<bf16>(x[at(2, t)])); },
           [&](int t, float v) {
             unsigned term[3];
             ms_split(v, 0.f, term[0], term[1], term[2]);
#pragma unroll 1
             for (int p = 0; p < 3; ++p) reinterpret_cast<unsigned short*>(wt)[at(p, t)] = (unsigned short)term[p];
           });
}
__device__ __noinline__ void dc_again_u(const bf16* Lp, const float* rhs, long rs, int n, const float* bt, float* u) {
  dc_again(Lp, rhs, rs, n, bt, nullptr, [&](int t) { return u[t]; }, [&](int t, float x) { u[t] = x; });
}

// The inverse of a block 1 + L_ii of the four in Ld, a column a thread (tid < 64): x_i = [i = j] - sum over m < i of L(i, m) x_m, its
// terms without the ones.
__device__ __forceinline__ void dc_invert(const float* Ld, bf16* Tp, int tid) {
  const int blk = tid >> 4, j = tid & 15;
  const float* l = Ld + blk * 16 * 20;
  float x[DC_BLOCK];
#pragma unroll
  for (int i = 0; i < DC_BLOCK; ++i) {
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int m = 0; m < i; m += 4) {
      const float4 l4 = *reinterpret_cast<const float4*>(l + i * 20 + m);
      s0 = fmaf(-l4.x, x[m], s0);
      if (m + 1 < i) s1 = fmaf(-l4.y, x[m + 1], s1);
      if (m + 2 < i) s0 = fmaf(-l4.z, x[m + 2], s0);
      if (m + 3 < i) s1 = fmaf(-l4.w, x[m + 3], s1);
    }
    x[i] = j < i ? s0 + s1 : j == i ? 1.f : 0.f;
  }
#pragma unroll
  for (int i = 0; i < DC_BLOCK; ++i) {
    unsigned p0, p1, p2;
    ms_split(i == j ? 0.f : x[i], 0.f, p0, p1, p2);
    unsigned short* d = reinterpret_cast<unsigned short*>(Tp + (blk * 16 + i) * DC_TP + j);
    d[0] = (unsigned short)p0;
    d[CS_C * DC_TP] = (unsigned short)p1;
    d[2 * CS_C * DC_TP] = (unsigned short)p2;
  }
}

// 16 columns (tile `tile`: W's, or U's behind them) of the system: X^T block by block, rhs(i, nt, j) the right-hand side's number of the
// lane, next(i) what is asked for behind the i-th.  W's terms go to wrow, U's numbers to urow.  Whether a number is not finite.
template <int TILES, typename R, typename N>
__device__ __forceinline__ bool dc_columns(unsigned Lp_b, unsigned Tp_b, bool is_k, int tile, unsigned* wrow, float* urow, R rhs, N next) {
  const int lane = threadIdx.x & 31, mt = lane >> 3, r = lane & 7, c = lane & 3;
  unsigned xa[3][3][4];                               // the terms of X^T's first three blocks
  bool odd = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float acc[2][4] = {}, low[2][4] = {};
#pragma unroll
    for (int m = 0; m < i; ++m) {
      unsigned b[2][3][2];
      ms_load_b<3, false>(b, Lp_b + 2 * ((i * 16 + (mt >> 1) * 8 + r) * DC_LP + m * 16 + (mt & 1) * 8), 2 * CS_C * DC_LP);
      ms_terms<2, 3, 3>(acc, low, xa[m], b);
    }
    unsigned ra[3][4];
    float y[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        y[nt][j] = rhs(i, nt, j) - (acc[nt][j] + low[nt][j]);
      }
      ms_split(y[nt][0], y[nt][1], ra[0][2 * nt], ra[1][2 * nt], ra[2][2 * nt]);
      ms_split(y[nt][2], y[nt][3], ra[0][2 * nt + 1], ra[1][2 * nt + 1], ra[2][2 * nt + 1]);
    }
    next(i);
    unsigned b[2][3][2];
    ms_load_b<3, false>(b, Tp_b + 2 * ((i * 16 + (mt >> 1) * 8 + r) * DC_TP + (mt & 1) * 8), 2 * CS_C * DC_TP);
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[nt][j] = low[nt][j] = 0.f;
    ms_terms<2, 3, 3>(acc, low, ra, b);
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[nt][j] = y[nt][j] + (acc[nt][j] + low[nt][j]);
        odd |= !(fabsf(acc[nt][j]) < INFINITY);
      }
      const int t = i * 16 + nt * 8 + 2 * c;
      unsigned lo[3], hi[3];                          // the terms of columns gr and gr + 8
      if (i < 3 || is_k) {
        ms_split(acc[nt][0], acc[nt][1], lo[0], lo[1], lo[2]);
        ms_split(acc[nt][2], acc[nt][3], hi[0], hi[1], hi[2]);
      }
      if (i < 3) {
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          xa[i][p][2 * nt] = lo[p];
          xa[i][p][2 * nt + 1] = hi[p];
        }
      }
      if (is_k) {
        DcFrag f;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          f.b[p][0] = dc_turned(lo[p]);
          f.b[p][1] = dc_turned(hi[p]);
        }
        dc_frag_put<TILES>(wrow, tile * 8 + 2 * i + nt, lane, f);
      } else {
        float* d = urow + t;
        *reinterpret_cast<float2*>(d) = make_float2(acc[nt][0], acc[nt][1]);
        *reinterpret_cast<float2*>(d + 8 * CS_C) = make_float2(acc[nt][2], acc[nt][3]);
      }
    }
  }
  return odd;
}

// ---------------------------------------------------------------------------------------------------------------
// ut [items][H][DV][64] = U^T; wt [items][H] = W's terms, tiles (16 key channels, 8 tokens), kp [items][Hk] = the terms of the chunk's
// k, tiles (16 tokens, 8 key channels), as DcFrag; m [items][H][64][64] = M; pre, suf [items][H][64] = G(t, -), G(C, s); gam [items][H] = G(C, -).
//
// The system by blocks of 16 tokens: the four blocks on L's diagonal are inverted by substitution (a column a thread, 120
// multiply-adds), everything else is products: X_i = (1 + L_ii)^-1 (B_i - sum over m < i of
// L_im X_m), made as X^T with 16 columns of the right-hand sides a warp on the M side, so that a block's result is the next
// products' operand as it stands in the registers.  Two CTAs an SM, chains of short products between barriers: tensor pipe 23 %
// active.  384 (chunk, head) pairs 43 us with M (a thread a column with all 2,016 multiply-adds took as long without M, which then
// took chunk_read 19 us more).
// ---------------------------------------------------------------------------------------------------------------
template <int DK, int DV>
__global__ void __launch_bounds__(CS_THREADS, 2)
delta_solve_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vc,
                   const float* __restrict__ beta, const float* __restrict__ g, const int* __restrict__ cu_q,
                   const int* __restrict__ req_slot, int E, int item0, float* __restrict__ ut, unsigned* __restrict__ wt,
                   unsigned* __restrict__ kp, float* __restrict__ mm, float* __restrict__ suf_out, float* __restrict__ pre_out,
                   float* __restrict__ gam, int H, int Hk) {
  constexpr int KP = DK + 8, TILES = DK / 2;                     // tiles of 16 by 8 of 64 tokens' k or W
  extern __shared__ __align__(16) unsigned char cs_smem[];
  bf16* ks = reinterpret_cast<bf16*>(cs_smem);                   // [3][64][KP]
  bf16* Lp = ks + 3 * CS_C * KP;                                 // [3][64][DC_LP]
  bf16* Tp = Lp + 3 * CS_C * DC_LP;                              // [3][64][DC_TP]: (1 + L_ii)^-1 - 1 of the blocks on the diagonal
  float* Ld = reinterpret_cast<float*>(Tp + 3 * CS_C * DC_TP);   // [64][20]: these blocks of L
  float* gs = Ld + CS_C * 20;                                    // [64][DC_GP]
  __shared__ float bt[CS_C], pre[CS_C];
  __shared__ double av[CS_C];
  __shared__ DcProduct tail[CS_C], whole[4];
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int item = blockIdx.x, h = blockIdx.y, group = H / Hk, hk = h / group;
  int e, chunk;
  if (!cs_item(item0 + item, cu_q, E, e, chunk)) return;
  if (req_slot[e] < 0) return;
  const int base = cu_q[e] + chunk * CS_C, n = min(CS_C, cu_q[e + 1] - base);
  const long Cq = (long)Hk * DK, Cv = (long)H * DV;
  const size_t ih = (size_t)item * H + h;
  const float* krow = kn + (size_t)base * Cq + hk * DK;
  const int mt = lane >> 3, r = lane & 7, gr = lane >> 2, c = lane & 3;
  const unsigned ks_b = ms_smem(ks);
  // M's rows warp / 2: what it needs of q, all of it on its way together with k
  const int rq = warp >> 1, tq = rq * 16 + gr;
  float2 qv[DK / 16][4];
  if ((warp & 1) <= rq) {
    const float* q0 = qn + (size_t)(base + tq) * Cq + hk * DK + 2 * c;
    const float2 z = make_float2(0.f, 0.f);
#pragma unroll
    for (int kt = 0; kt < DK / 16; ++kt) {
      qv[kt][0] = tq < n ? *reinterpret_cast<const float2*>(q0 + kt * 16) : z;
      qv[kt][1] = tq + 8 < n ? *reinterpret_cast<const float2*>(q0 + 8 * Cq + kt * 16) : z;
      qv[kt][2] = tq < n ? *reinterpret_cast<const float2*>(q0 + kt * 16 + 8) : z;
      qv[kt][3] = tq + 8 < n ? *reinterpret_cast<const float2*>(q0 + 8 * Cq + kt * 16 + 8) : z;
    }
  }
  {
    CsTile<float, DK, KP, CS_THREADS> kt_;
    kt_.ask(krow, Cq, n);
    if (tid < CS_C) {
      av[tid] = tid < n ? g[(size_t)(base + tid) * H + h] : 1.f;
      bt[tid] = tid < n ? beta[(size_t)(base + tid) * H + h] : 0.f;
    }
    kt_.put(ks);
  }
  __syncthreads();
  dc_gaps(av, gs, pre, tail, whole);
  __syncthreads();
  if (tid < CS_C) {
    suf_out[ih * CS_C + tid] = gs[(CS_C - 1) * DC_GP + tid];
    pre_out[ih * CS_C + tid] = pre[tid];
  }
  if (tid == CS_C) gam[ih] = pre[CS_C - 1];
  // M's tiles, every second one of the row's columns
  {
    const int half = warp & 1;
    float acc[2][2][4] = {}, low[2][2][4] = {};
    if (half <= rq) {
#pragma unroll
      for (int kt = 0; kt < DK / 16; ++kt) {
        unsigned a[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) ms_split(qv[kt][j].x, qv[kt][j].y, a[0][j], a[1][j], a[2][j]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int ct = half + 2 * j;
          if (ct <= rq) {
            unsigned b[2][3][2];
            ms_load_b<3, false>(b, ks_b + 2 * ((ct * 16 + (mt >> 1) * 8 + r) * KP + kt * 16 + (mt & 1) * 8), 2 * CS_C * KP);
            ms_terms<2, 3, 3>(acc[j], low[j], a, b);
          }
        }
      }
    }
    float* mrow = mm + ih * CS_C * CS_C;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int ct = half + 2 * j;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int t = tq + 8 * q, s = ct * 16 + i * 8 + 2 * c;
          float2 x = make_float2(0.f, 0.f);
          if (ct <= rq) {
            if (s <= t) x.x = gs[t * DC_GP + s] * (acc[j][i][2 * q] + low[j][i][2 * q]);
            if (s + 1 <= t) x.y = gs[t * DC_GP + s + 1] * (acc[j][i][2 * q + 1] + low[j][i][2 * q + 1]);
          }
          *reinterpret_cast<float2*>(mrow + t * CS_C + s) = x;
        }
    }
  }
  float bx[4][2][4];                                    // 16 columns of a right-hand side: asked for long before they are needed
  auto ask_b = [&](int tile, int i) {
    const bool is_k = tile < DK / 16;
    const int c0 = is_k ? tile * 16 : tile * 16 - DK;
    const float* rhs = is_k ? krow + c0 + gr : vc + (size_t)base * Cv + (size_t)h * DV + c0 + gr;
    const long rs = is_k ? Cq : Cv;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = i * 16 + nt * 8 + 2 * c + (j & 1);
        bx[i][nt][j] = t < n ? rhs[(size_t)t * rs + 8 * (j >> 1)] : 0.f;
      }
  };
#pragma unroll
  for (int i = 0; i < 4; ++i) ask_b(warp, i);
  // L's tiles of 16 by 16, the lower triangle: rows 3 - warp / 2, every second tile of columns
  {
    const int rt = 3 - (warp >> 1), half = warp & 1;
    float acc[2][2][4] = {}, low[2][2][4] = {};
    if (half <= rt) {
#pragma unroll 2
      for (int kt = 0; kt < DK / 16; ++kt) {
        unsigned a[3][4];
#pragma unroll
        for (int p = 0; p < 3; ++p)
          ms_ldm4(a[p], ks_b + 2 * ((p * CS_C + rt * 16 + (mt & 1) * 8 + r) * KP + kt * 16 + (mt >> 1) * 8));
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int ct = half + 2 * j;
          if (ct <= rt) {
            unsigned b[2][3][2];
            ms_load_b<3, false>(b, ks_b + 2 * ((ct * 16 + (mt >> 1) * 8 + r) * KP + kt * 16 + (mt & 1) * 8), 2 * CS_C * KP);
            ms_terms<2, 3, 3>(acc[j], low[j], a, b);
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int ct = half + 2 * j;
      if (ct > rt) continue;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int t = rt * 16 + gr + q * 8, s = ct * 16 + i * 8 + 2 * c;
          const float x = s < t ? bt[t] * gs[t * DC_GP + s] * (acc[j][i][2 * q] + low[j][i][2 * q]) : 0.f;
          const float y = s + 1 < t ? bt[t] * gs[t * DC_GP + s + 1] * (acc[j][i][2 * q + 1] + low[j][i][2 * q + 1]) : 0.f;
          unsigned p0, p1, p2;
          ms_split(x, y, p0, p1, p2);
          unsigned* d = reinterpret_cast<unsigned*>(Lp + t * DC_LP + s);
          d[0] = p0;
          d[CS_C * DC_LP / 2] = p1;
          d[CS_C * DC_LP] = p2;
          if (ct == rt) *reinterpret_cast<float2*>(Ld + t * 20 + i * 8 + 2 * c) = make_float2(x, y);
        }
    }
  }
  __syncthreads();
  if (tid < CS_C) dc_invert(Ld, Tp, tid);
  if (h == hk * group) {                                // k's terms, once for the heads that read it
    unsigned* dst = kp + ((size_t)item * Hk + hk) * TILES * 192;
    for (int tile = 2 * warp; tile < TILES; tile += CS_THREADS / 16) {
      DcFrag f[2];
      const int kt = tile / (DK / 8), cb = tile % (DK / 8);
      ms_load_b<3, true>(reinterpret_cast<unsigned(*)[3][2]>(f), ks_b + 2 * ((kt * 16 + (mt & 1) * 8 + r) * KP + (cb + (mt >> 1)) * 8),
                         2 * CS_C * KP);
      dc_frag_put<TILES>(dst, tile, lane, f[0]);
      dc_frag_put<TILES>(dst, tile + 1, lane, f[1]);
    }
  }
  // X^T, 16 columns of the right-hand sides at a time: W's first, then U's
  const unsigned Lp_b = ms_smem(Lp), Tp_b = ms_smem(Tp);
  __syncthreads();
#pragma unroll 1
  for (int tile = warp; tile < (DK + DV) / 16; tile += CS_THREADS / 32) {
    const bool is_k = tile < DK / 16;
    const int c0 = is_k ? tile * 16 : tile * 16 - DK;
    unsigned* wrow = wt + ih * TILES * 192;
    const bool odd = dc_columns<TILES>(
        Lp_b, Tp_b, is_k, tile, wrow, ut + (ih * DV + c0 + gr) * CS_C,
        [&](int i, int nt, int j) {
          const int t = i * 16 + nt * 8 + 2 * c + (j & 1);
          return bx[i][nt][j] * (is_k ? bt[t] * pre[t] : bt[t]);
        },
        [&](int i) {
          if (tile + CS_THREADS / 32 < (DK + DV) / 16) ask_b(tile + CS_THREADS / 32, i);
        });
    // columns gr and gr + 8 of the tile have a number that is not finite in some lane of the four: its first lane makes them again
    const unsigned bad = __ballot_sync(0xffffffffu, odd);
    __syncwarp();
    if (((bad >> (lane & 28)) & 15) != 0 && c == 0) {
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        const int col = c0 + gr + 8 * q;
        if (is_k) dc_again_w<DK>(Lp, krow + col, Cq, n, bt, pre, wrow, col);
        else dc_again_u(Lp, vc + (size_t)base * Cv + (size_t)h * DV + col, Cv, n, bt, ut + (ih * DV + col) * CS_C);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// The same with a decay a key channel: L(t, s) = beta_t sum over the channels of k_t G(t, s) k_s, and so on.  A quotient of running
// products would overflow, so G is made of factors that are at most one: within a block of 16 tokens (s, t of the same) a thread has
// 8 or 16 channels of k_s and multiplies decay by decay while it adds up the products with the tokens behind; between blocks
// G(t, s) = R(t) B Y(s), R from t's block's start, Y to s's block's end, B the blocks between, and k_t R(t), q_t R(t) and k_s Y(s) B are
// the operands of products on the tensor cores.  What the walk multiplies the state by is rounded once (DcProduct).
// qd [items][H][64][DK] = G(t, -) q_t, kp [items][H] = the terms of G(C, s) k_s, gam [items][H][DK] = G(C, -); the rest as above.
// One CTA an SM (191 KB of shared memory).  Two entries of together 2,047 tokens, 12 heads: the three kernels 154 us, the walk by tokens
// 857; its error against 64 bits is half the walk's.
// ---------------------------------------------------------------------------------------------------------------
#define DC_CH_THREADS 512
template <int DK, int DV>
__global__ void __launch_bounds__(DC_CH_THREADS, 1)
delta_solve_channels_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vc,
                            const float* __restrict__ beta, const float* __restrict__ g, const int* __restrict__ cu_q,
                            const int* __restrict__ req_slot, int E, int item0, float* __restrict__ ut, unsigned* __restrict__ wt,
                            unsigned* __restrict__ kp, float* __restrict__ mm, float* __restrict__ qd, float* __restrict__ gam, int H,
                            int Hk) {
  constexpr int FP = DK + 8, TILES = DK / 2, WARPS = DC_CH_THREADS / 32, PIECES = DK / 4;
  extern __shared__ __align__(16) unsigned char cs_smem[];
  float* kf = reinterpret_cast<float*>(cs_smem);                 // [64][FP] each: k, q
  float* qf = kf + CS_C * FP;
  float* rf = qf + CS_C * FP;                                    // decays, R, at last k G(t, -)
  float* yf = rf + CS_C * FP;                                    // Y, at last k G(C, s)
  bf16* Lp = reinterpret_cast<bf16*>(yf + CS_C * FP);            // [3][64][DC_LP]
  bf16* Tp = Lp + 3 * CS_C * DC_LP;                              // [3][64][DC_TP]
  float* Ld = reinterpret_cast<float*>(Tp + 3 * CS_C * DC_TP);   // [64][20]
  DcProduct* blk = reinterpret_cast<DcProduct*>(Ld + CS_C * 20);      // [4][DK]: whole blocks
  float* front = reinterpret_cast<float*>(blk + 4 * DK);         // [4][DK]: the blocks in front of a block
  float* behind = front + 4 * DK;                                // [4][DK]: behind it
  float* mid = behind + 4 * DK;                                  // [4][DK]: between blocks 0 and 2, 1 and 3, 0 and 3; ones
  __shared__ float bt[CS_C];
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int item = blockIdx.x, h = blockIdx.y, hk = h / (H / Hk);
  int e, chunk;
  if (!cs_item(item0 + item, cu_q, E, e, chunk)) return;
  if (req_slot[e] < 0) return;
  const int base = cu_q[e] + chunk * CS_C, n = min(CS_C, cu_q[e + 1] - base);
  const long Cq = (long)Hk * DK, Cv = (long)H * DV;
  const size_t ih = (size_t)item * H + h;
  const int gr = lane >> 2, c = lane & 3;
  {
    const float* krow = kn + (size_t)base * Cq + hk * DK;
    const float* qrow = qn + (size_t)base * Cq + hk * DK;
    const float* arow = g + ((size_t)base * H + h) * DK;
    constexpr int N = CS_C * PIECES / DC_CH_THREADS;
    float4 v[3][N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int i = j * DC_CH_THREADS + tid, t = i / PIECES, ch = i % PIECES * 4;
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      v[0][j] = t < n ? *reinterpret_cast<const float4*>(krow + (size_t)t * Cq + ch) : z;
      v[1][j] = t < n ? *reinterpret_cast<const float4*>(qrow + (size_t)t * Cq + ch) : z;
      v[2][j] = t < n ? *reinterpret_cast<const float4*>(arow + (size_t)t * H * DK + ch) : make_float4(1.f, 1.f, 1.f, 1.f);
    }
    if (tid < CS_C) bt[tid] = tid < n ? beta[(size_t)(base + tid) * H + h] : 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int i = j * DC_CH_THREADS + tid, at = i / PIECES * FP + i % PIECES * 4;
      *reinterpret_cast<float4*>(kf + at) = v[0][j];
      *reinterpret_cast<float4*>(qf + at) = v[1][j];
      *reinterpret_cast<float4*>(rf + at) = v[2][j];
    }
  }
  __syncthreads();
  float* mrow = mm + ih * CS_C * CS_C;
  auto put_l = [&](int t, int s, float x, float y) {             // L(t, s) and L(t, s + 1)
    unsigned p0, p1, p2;
    ms_split(x, y, p0, p1, p2);
    unsigned* d = reinterpret_cast<unsigned*>(Lp + t * DC_LP + s);
    d[0] = p0;
    d[CS_C * DC_LP / 2] = p1;
    d[CS_C * DC_LP] = p2;
  };
  // the blocks on the diagonal: eight threads a token s, channels 4 (tid % 8) + 32 j
  {
    const int s = tid >> 3, cg = tid & 7, b0 = s & ~15;
    float kg[DK / 8], v[32];
#pragma unroll
    for (int j = 0; j < DK / 32; ++j) *reinterpret_cast<float4*>(kg + 4 * j) = *reinterpret_cast<const float4*>(kf + s * FP + cg * 4 + 32 * j);
#pragma unroll
    for (int tt = 0; tt < 16; ++tt) {
      const int t = b0 + tt;
      float dk = 0.f, dq = 0.f;
#pragma unroll
      for (int j = 0; j < DK / 32; ++j) {
        const int at = t * FP + cg * 4 + 32 * j;
        const float4 a4 = *reinterpret_cast<const float4*>(rf + at), k4 = *reinterpret_cast<const float4*>(kf + at);
        const float4 q4 = *reinterpret_cast<const float4*>(qf + at);
        const float av[4] = {a4.x, a4.y, a4.z, a4.w}, kv[4] = {k4.x, k4.y, k4.z, k4.w}, qv[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (t > s) kg[4 * j + i] *= av[i];
          dk = fmaf(kv[i], kg[4 * j + i], dk);
          dq = fmaf(qv[i], kg[4 * j + i], dq);
        }
      }
      v[2 * tt] = dk;
      v[2 * tt + 1] = dq;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)                              // a lane keeps half of what it has at each step: two tokens t at last
#pragma unroll
      for (int i = 0; i < 4 * o; ++i) {
        const float other = __shfl_xor_sync(0xffffffffu, cg & o ? v[i] : v[i + 4 * o], o);
        v[i] = (cg & o ? v[i + 4 * o] : v[i]) + other;
      }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = b0 + 2 * cg + i;
      const float x = s < t ? bt[t] * v[2 * i] : 0.f;
      unsigned p0, p1, p2;
      ms_split(x, 0.f, p0, p1, p2);
      unsigned short* d = reinterpret_cast<unsigned short*>(Lp + t * DC_LP + s);
      d[0] = (unsigned short)p0;
      d[CS_C * DC_LP] = (unsigned short)p1;
      d[2 * CS_C * DC_LP] = (unsigned short)p2;
      Ld[t * 20 + (s & 15)] = x;
      mrow[t * CS_C + s] = s <= t ? v[2 * i + 1] : 0.f;
    }
  }
  __syncthreads();
  // R, Y and whole blocks: a thread a channel and block
  if (tid < 4 * DK) {
    const int ch = tid % DK, b = tid / DK;
    float* a = rf + b * 16 * FP + ch;
    float* y = yf + b * 16 * FP + ch;
    double av[16];
    DcProduct p;
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      av[t] = a[t * FP];
      p.times(av[t]);
      a[t * FP] = p.value();
    }
    blk[b * DK + ch] = p;
    p = DcProduct();
#pragma unroll
    for (int t = 15; t >= 0; --t) {
      y[t * FP] = p.value();
      p.times(av[t]);
    }
  }
  __syncthreads();
  if (tid < DK) {
    const DcProduct b0 = blk[tid], b1 = blk[DK + tid], b2 = blk[2 * DK + tid], b3 = blk[3 * DK + tid];
    DcProduct f = b0, w = b3;
    front[tid] = 1.f;
    front[DK + tid] = f.value();
    f.times(b1);
    front[2 * DK + tid] = f.value();
    f.times(b2);
    front[3 * DK + tid] = f.value();
    f.times(b3);
    gam[ih * DK + tid] = f.value();
    behind[3 * DK + tid] = 1.f;
    behind[2 * DK + tid] = w.value();
    w.times(b2);
    behind[DK + tid] = w.value();
    w.times(b1);
    behind[tid] = w.value();
    mid[tid] = b1.value();
    mid[DK + tid] = b2.value();
    DcProduct m = b1;
    m.times(b2);
    mid[2 * DK + tid] = m.value();
    mid[3 * DK + tid] = 1.f;
  }
  __syncthreads();
  // the blocks below the diagonal, L's and M's, a warp each; two more warps invert the ones on it
  if (warp < 12) {
    const int pair = warp >> 1, I = pair < 1 ? 1 : pair < 3 ? 2 : 3, J = pair - (I * (I - 1)) / 2;
    const float* row = (warp & 1 ? qf : kf) + (I * 16 + gr) * FP + 2 * c;
    const float* fac = rf + (I * 16 + gr) * FP + 2 * c;
    const float* col = kf + (J * 16 + gr) * FP + 2 * c;
    const float* yac = yf + (J * 16 + gr) * FP + 2 * c;
    const float* between = mid + (I - J == 1 ? 3 : I - J == 3 ? 2 : J) * DK + 2 * c;
    float acc[2][4] = {}, low[2][4] = {};
#pragma unroll 2
    for (int kt = 0; kt < DK / 16; ++kt) {
      unsigned a[3][4], b[2][3][2];
      auto two = [](const float* p, const float* q) {
        const float2 x = *reinterpret_cast<const float2*>(p), y = *reinterpret_cast<const float2*>(q);
        return make_float2(x.x * y.x, x.y * y.y);
      };
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int at = kt * 16 + (j & 1) * 8 * FP + (j >> 1) * 8;
        const float2 x = two(row + at, fac + at);
        ms_split(x.x, x.y, a[0][j], a[1][j], a[2][j]);
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int at = kt * 16 + nt * 8 * FP + q * 8;
          const float2 x = two(col + at, yac + at), y = *reinterpret_cast<const float2*>(between + kt * 16 + q * 8);
          ms_split(x.x * y.x, x.y * y.y, b[nt][0][q], b[nt][1][q], b[nt][2][q]);
        }
      ms_terms<2, 3, 3>(acc, low, a, b);
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int t = I * 16 + gr + 8 * q, s = J * 16 + nt * 8 + 2 * c;
        const float x = acc[nt][2 * q] + low[nt][2 * q], y = acc[nt][2 * q + 1] + low[nt][2 * q + 1];
        if (warp & 1) *reinterpret_cast<float2*>(mrow + t * CS_C + s) = make_float2(x, y);
        else put_l(t, s, bt[t] * x, bt[t] * y);
      }
  } else if (warp < 14) {
    dc_invert(Ld, Tp, tid - 12 * 32);
  }
  __syncthreads();
  // k from the chunk's start and to its end in the factors' places, q from its start for the read-outs
  for (int i = tid; i < CS_C * PIECES; i += DC_CH_THREADS) {
    const int t = i / PIECES, ch = i % PIECES * 4, at = t * FP + ch;
    const float4 k4 = *reinterpret_cast<const float4*>(kf + at), q4 = *reinterpret_cast<const float4*>(qf + at);
    const float4 f4 = *reinterpret_cast<const float4*>(front + (t >> 4) * DK + ch), b4 = *reinterpret_cast<const float4*>(behind + (t >> 4) * DK + ch);
    float4 r4 = *reinterpret_cast<const float4*>(rf + at), y4 = *reinterpret_cast<const float4*>(yf + at);
    r4 = make_float4(r4.x * f4.x, r4.y * f4.y, r4.z * f4.z, r4.w * f4.w);
    y4 = make_float4(y4.x * b4.x, y4.y * b4.y, y4.z * b4.z, y4.w * b4.w);
    *reinterpret_cast<float4*>(rf + at) = make_float4(k4.x * r4.x, k4.y * r4.y, k4.z * r4.z, k4.w * r4.w);
    *reinterpret_cast<float4*>(yf + at) = make_float4(k4.x * y4.x, k4.y * y4.y, k4.z * y4.z, k4.w * y4.w);
    *reinterpret_cast<float4*>(qd + (ih * CS_C + t) * DK + ch) = make_float4(q4.x * r4.x, q4.y * r4.y, q4.z * r4.z, q4.w * r4.w);
  }
  __syncthreads();
  unsigned* kdst = kp + ih * TILES * 192;
  for (int tile = warp; tile < TILES; tile += WARPS) {
    DcFrag f;
    const float* src = yf + (tile / (DK / 8) * 16 + 2 * c) * FP + tile % (DK / 8) * 8 + gr;
#pragma unroll
    for (int q = 0; q < 2; ++q) ms_split(src[8 * q * FP], src[(8 * q + 1) * FP], f.b[0][q], f.b[1][q], f.b[2][q]);
    dc_frag_put<TILES>(kdst, tile, lane, f);
  }
  const unsigned Lp_b = ms_smem(Lp), Tp_b = ms_smem(Tp);
#pragma unroll 1
  for (int tile = warp; tile < (DK + DV) / 16; tile += WARPS) {
    const bool is_k = tile < DK / 16;
    const int c0 = is_k ? tile * 16 : tile * 16 - DK;
    const float* vrow = vc + (size_t)base * Cv + (size_t)h * DV + c0 + gr;
    unsigned* wrow = wt + ih * TILES * 192;
    float bx[4][2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = i * 16 + nt * 8 + 2 * c + (j & 1);
          bx[i][nt][j] = is_k ? rf[t * FP + c0 + gr + 8 * (j >> 1)] : t < n ? vrow[(size_t)t * Cv + 8 * (j >> 1)] : 0.f;
        }
    const bool odd = dc_columns<TILES>(
        Lp_b, Tp_b, is_k, tile, wrow, ut + (ih * DV + c0 + gr) * CS_C,
        [&](int i, int nt, int j) { return bx[i][nt][j] * bt[i * 16 + nt * 8 + 2 * c + (j & 1)]; }, [](int) {});
    const unsigned bad = __ballot_sync(0xffffffffu, odd);
    __syncwarp();
    if (((bad >> (lane & 28)) & 15) != 0 && c == 0) {
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        const int col = c0 + gr + 8 * q;
        if (is_k) dc_again_w<DK>(Lp, rf + col, FP, n, bt, nullptr, wrow, col);
        else dc_again_u(Lp, vrow + 8 * q, Cv, n, bt, ut + (ih * DV + col) * CS_C);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// For the entry's chunks in order  s0 <- S,  u <- U - W S (in place),  S <- G(C, -) S + k^T (G(C, s) u).
//
// 16 value columns a CTA are the M side of both products, so the state's and u's terms are operands from shared memory that every
// warp reads.  First product: two teams of four warps take half of the key channels each, a warp 16 of the chunk's tokens, and the
// teams exchange half of their sums, so that each makes u for 8 tokens a warp; second product: a warp keeps the state of an eighth
// of the key channels.  W's and k's terms, made by delta_solve as the MMA's operand, come by one bulk copy each, a chunk ahead.
// Bound by shared memory and the tensor pipe in turn (96 MMAs and 768 clocks of shared memory a scheduler and product) and by the
// hand-overs.  (Two entries of together 2,047 tokens, 12 heads: 99 us with all parts of W S added up over eight warps; 70 with the
// terms made here from float32, 1,180 instructions a warp and chunk; 55 with four warps, or eight that all read all of the state's
// terms; 59 with W's and k's terms straight from L2 and two CTAs an SM.)  The longest entries' CTAs come first.
// ---------------------------------------------------------------------------------------------------------------
template <int DK, bool CH>
__global__ void __launch_bounds__(CS_THREADS)
delta_walk_kernel(float* __restrict__ ut, const unsigned* __restrict__ wt, const unsigned* __restrict__ kp,
                  const float* __restrict__ suf_in, const float* __restrict__ gam, float* __restrict__ s0,
                  float* __restrict__ state, long state_stride, int num_slots, const int* __restrict__ cu_q,
                  const int* __restrict__ req_slot, int E, int item0, int items, int H, int Hk, int dv, int* status) {
  constexpr int WARPS = CS_THREADS / 32, KW = DK / WARPS;      // key channels a warp: 16, or 8 of heads of 64
  constexpr int SP = DK + 8, UP = CS_C + 8;
  constexpr int NT = KW / 8, KH = DK / 32, TILES = DK / 2;     // KH: steps of 16 channels a team
  constexpr int WORDS = TILES * 192, BYTES = 4 * WORDS;
  extern __shared__ __align__(128) unsigned char dw_smem[];
  unsigned* wb = reinterpret_cast<unsigned*>(dw_smem);         // [2][WORDS]
  unsigned* kb = wb + 2 * WORDS;                               // [2][WORDS]
  bf16* ss = reinterpret_cast<bf16*>(kb + 2 * WORDS);          // [3][16][SP]: S, a row a value column
  bf16* us = ss + 3 * 16 * SP;                                 // [3][16][UP]: G(C, s) u, a row a value column
  float4* xb = reinterpret_cast<float4*>(us + 3 * 16 * UP);    // [WARPS][32]: sums for the other team
  __shared__ __align__(8) unsigned long long full[4];          // W's and k's two places
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) at_mbar_init(at_smem(full + i), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int c0 = blockIdx.x * 16, h = blockIdx.y, hk = h / (H / Hk);
  int e = blockIdx.z;
  if (E > 1 && E <= 32) {                                      // the entry that is blockIdx.z-th by length
    const int mine = lane < E ? cu_q[lane + 1] - cu_q[lane] : -1;
    int rank = 0;
    for (int j = 0; j < E; ++j) {
      const int other = __shfl_sync(0xffffffffu, mine, j);
      rank += other > mine || (other == mine && j < lane);
    }
    e = __ffs(__ballot_sync(0xffffffffu, lane < E && rank == (int)blockIdx.z)) - 1;
  }
  const int slot = req_slot[e];
  if (slot < 0 || slot >= num_slots) return;
  // of the entry's chunks those of the call: `first`, the place of their first one in the call's scratch, and their number
  const int at = cs_first_item(e, cu_q) - item0, first = max(at, 0);
  const int chunks = min(at + (cu_q[e + 1] - cu_q[e] + CS_C - 1) / CS_C, items) - first;
  if (chunks <= 0) return;
  const int m = lane >> 3, r = lane & 7, g = lane >> 2, c = lane & 3;
  const int team = warp >> 2, kw = warp * KW;           // the warp's first key channel in the second product
  const int tw = (warp & 3) * 16 + team * 8;            // the first of the eight tokens whose u it makes
  bool dead = false;
  auto copy = [&](const unsigned* dst, const unsigned* src, int place) {      // by one thread
    const unsigned bar = at_smem(full + place);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // what has been read from the place, then the copy
    at_mbar_expect_tx(bar, BYTES);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(ms_smem(dst)),
                 "l"(src), "r"(BYTES), "r"(bar)
                 : "memory");
  };
  auto fetch_w = [&](int chunk) {
    if (chunk < chunks && tid == 0) copy(wb + (chunk & 1) * WORDS, wt + ((size_t)(first + chunk) * H + h) * WORDS, chunk & 1);
  };
  auto fetch_k = [&](int chunk) {
    if (chunk < chunks && tid == 0) copy(kb + (chunk & 1) * WORDS, kp + ((size_t)(first + chunk) * (CH ? H : Hk) + (CH ? h : hk)) * WORDS, 2 + (chunk & 1));
  };
  fetch_w(0);
  fetch_k(0);
  fetch_w(1);
  fetch_k(1);
  float* rec = state + (size_t)slot * state_stride + ((size_t)h * dv + c0) * DK + kw;
  float S[NT][4];
  auto hand_over = [&]() {                              // the state's terms to all warps
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        unsigned p0, p1, p2;
        ms_split(S[nt][2 * q], S[nt][2 * q + 1], p0, p1, p2);
        unsigned* d = reinterpret_cast<unsigned*>(ss + (g + 8 * q) * SP + kw + nt * 8 + 2 * c);
        d[0] = p0;
        d[16 * SP / 2] = p1;
        d[16 * SP] = p2;
      }
  };
  auto put_state = [&](float* d) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      *reinterpret_cast<float2*>(d + (size_t)g * DK + nt * 8 + 2 * c) = make_float2(S[nt][0], S[nt][1]);
      *reinterpret_cast<float2*>(d + (size_t)(g + 8) * DK + nt * 8 + 2 * c) = make_float2(S[nt][2], S[nt][3]);
    }
  };
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const float2 a = *reinterpret_cast<const float2*>(rec + (size_t)g * DK + nt * 8 + 2 * c);
    const float2 b = *reinterpret_cast<const float2*>(rec + (size_t)(g + 8) * DK + nt * 8 + 2 * c);
    S[nt][0] = a.x; S[nt][1] = a.y; S[nt][2] = b.x; S[nt][3] = b.y;
  }
  hand_over();
  const int row = (m & 1) * 8 + r;                      // the lane's row of a 16 x 16 tile that ldmatrix reads
  const unsigned ss_at = ms_smem(ss) + 2 * (row * SP + team * KH * 16 + (m >> 1) * 8);
  const unsigned us_at = ms_smem(us) + 2 * (row * UP + (m >> 1) * 8);
  auto load_w = [&](DcFrag (&f)[2], int chunk, int i) {         // W's terms: 16 of the team's channels, 16 tokens
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
      dc_frag_get<TILES>(f[nt], wb + (chunk & 1) * WORDS, (team * KH + i) * 8 + (warp & 3) * 2 + nt, lane);
  };
  auto load_k = [&](DcFrag (&f)[NT], int chunk, int kt) {       // k's terms: 16 tokens, the warp's channels
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) dc_frag_get<TILES>(f[nt], kb + (chunk & 1) * WORDS, kt * (DK / 8) + warp * NT + nt, lane);
  };
  __syncthreads();                                      // the barriers are made; the state's terms
  DcFrag fw[2][2], fk[2][NT];
  at_mbar_wait(at_smem(full), 0, status, dead);
  load_w(fw[0], 0, 0);
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const size_t ih = (size_t)(first + chunk) * H + h;
    // (W S)^T [16 x 16]: the team's channels
    float lead[2][4] = {}, part[2][2][4] = {};
    unsigned a[2][3][4];
#pragma unroll
    for (int p = 0; p < 3; ++p) ms_ldm4(a[0][p], ss_at + 2 * p * 16 * SP);
    float* urow = ut + (ih * dv + c0 + g) * CS_C + tw + 2 * c;
    const float2 u0 = *reinterpret_cast<const float2*>(urow), u1 = *reinterpret_cast<const float2*>(urow + 8 * CS_C);
    float2 f2 = make_float2(1.f, 1.f), gc[NT];            // (CH: the decays to the chunk's end are in k's terms)
    if (!CH) f2 = *reinterpret_cast<const float2*>(suf_in + ih * CS_C + tw + 2 * c);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      if (CH) gc[nt] = *reinterpret_cast<const float2*>(gam + ih * DK + kw + nt * 8 + 2 * c);
      else gc[nt].x = gc[nt].y = gam[ih];
    }
    put_state(s0 + (ih * dv + c0) * DK + kw);
#pragma unroll
    for (int i = 0; i < KH; ++i) {
      const int now = i & 1, then = now ^ 1;
      if (i + 1 < KH) {
        load_w(fw[then], chunk, i + 1);
#pragma unroll
        for (int p = 0; p < 3; ++p) ms_ldm4(a[then][p], ss_at + 2 * (p * 16 * SP + (i + 1) * 16));
      }
      float t[2][4] = {};
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) ms_mma(t[nt], a[now][0], fw[now][nt].b[0][0], fw[now][nt].b[0][1]);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) ms_mma(part[nt][0], a[now][0], fw[now][nt].b[1][0], fw[now][nt].b[1][1]);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) ms_mma(part[nt][1], a[now][0], fw[now][nt].b[2][0], fw[now][nt].b[2][1]);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) ms_mma(part[nt][0], a[now][1], fw[now][nt].b[0][0], fw[now][nt].b[0][1]);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) ms_mma(part[nt][1], a[now][1], fw[now][nt].b[1][0], fw[now][nt].b[1][1]);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) ms_mma(part[nt][1], a[now][2], fw[now][nt].b[0][0], fw[now][nt].b[0][1]);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int j = 0; j < 4; ++j) lead[nt][j] += t[nt][j];
    }
    float mine[4];
    {
      float gone[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float x0 = lead[0][j] + (part[0][0][j] + part[0][1][j]), x1 = lead[1][j] + (part[1][0][j] + part[1][1][j]);
        mine[j] = team == 0 ? x0 : x1;
        gone[j] = team == 0 ? x1 : x0;
      }
      xb[warp * 32 + lane] = make_float4(gone[0], gone[1], gone[2], gone[3]);
    }
    at_mbar_wait(at_smem(full + 2 + (chunk & 1)), (chunk >> 1) & 1, status, dead);
    load_k(fk[0], chunk, 0);
    __syncthreads();                                    // the teams' sums; the state's terms and W have been read
    fetch_w(chunk + 2);
    const float4 other = xb[(warp ^ 4) * 32 + lane];
    const float x[4] = {u0.x - (mine[0] + other.x), u0.y - (mine[1] + other.y), u1.x - (mine[2] + other.z), u1.y - (mine[3] + other.w)};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      unsigned p0, p1, p2;
      ms_split(x[2 * q] * f2.x, x[2 * q + 1] * f2.y, p0, p1, p2);
      unsigned* d = reinterpret_cast<unsigned*>(us + (g + 8 * q) * UP + tw + 2 * c);
      d[0] = p0;
      d[16 * UP / 2] = p1;
      d[16 * UP] = p2;
    }
    __syncthreads();                                    // u's terms
#pragma unroll
    for (int p = 0; p < 3; ++p) ms_ldm4(a[0][p], us_at + 2 * p * 16 * UP);
    *reinterpret_cast<float2*>(urow) = make_float2(x[0], x[1]);
    *reinterpret_cast<float2*>(urow + 8 * CS_C) = make_float2(x[2], x[3]);
    float low[NT][2][4] = {};
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) S[nt][j] *= j & 1 ? gc[nt].y : gc[nt].x;
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
      const int now = kt & 1, then = now ^ 1;
      if (kt + 1 < 4) {
        load_k(fk[then], chunk, kt + 1);
#pragma unroll
        for (int p = 0; p < 3; ++p) ms_ldm4(a[then][p], us_at + 2 * (p * 16 * UP + (kt + 1) * 16));
      }
      float t[NT][4] = {};
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) ms_mma(t[nt], a[now][0], fk[now][nt].b[0][0], fk[now][nt].b[0][1]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) ms_mma(low[nt][0], a[now][0], fk[now][nt].b[1][0], fk[now][nt].b[1][1]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) ms_mma(low[nt][1], a[now][0], fk[now][nt].b[2][0], fk[now][nt].b[2][1]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) ms_mma(low[nt][0], a[now][1], fk[now][nt].b[0][0], fk[now][nt].b[0][1]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) ms_mma(low[nt][1], a[now][1], fk[now][nt].b[1][0], fk[now][nt].b[1][1]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) ms_mma(low[nt][1], a[now][2], fk[now][nt].b[0][0], fk[now][nt].b[0][1]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int j = 0; j < 4; ++j) S[nt][j] += t[nt][j];
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) S[nt][j] += low[nt][0][j] + low[nt][1][j];
    if (chunk + 1 == chunks) break;
    hand_over();
    at_mbar_wait(at_smem(full + ((chunk + 1) & 1)), ((chunk + 1) >> 1) & 1, status, dead);
    load_w(fw[0], chunk + 1, 0);
    __syncthreads();                                    // the state's terms; u's and k have been read
    fetch_k(chunk + 2);
  }
  put_state(rec);
}

// The read-out of one token and value column again, token by token from the state in front of the chunk
// (token j's decay of channel ch: decay[j * step + ch * per_channel])
template <int DK>
__device__ __noinline__ float dc_number(const float* q, const float* k, long stride, const float* u, const float* state, const float* decay,
                                        long step, int per_channel, int t) {
  float a = 0.f;
  for (int ch = 0; ch < DK && a == a; ++ch)
    a = fmaf(cs_again<float>(state + ch, k + ch, stride, u, 1, t, [&](int j) { return decay[j * step + ch * per_channel]; },
                             [](int) { return 1.f; }),
             q[(size_t)t * stride + ch], a);
  return a;
}

// ---------------------------------------------------------------------------------------------------------------
// o_t = G(t, -) S0^T q_t + sum over s <= t of M(t, s) u_s.
//
// A warp has
// 16 value columns of all 64 tokens, so that it alone reads its part of the state and of u: they, too, come straight into registers,
// where their terms are made, and no barrier stands between the first and the last product.  Tokens are the M side; q's and M's terms
// lie in shared memory.  Two CTAs an SM.  (Tokens shared out over the warps, with state and u through shared memory 64 columns at a
// time and one CTA an SM: 46 us for 384 (chunk, head) pairs; norm and gate behind the products here: 43 us instead of 27 and a kernel
// of 10.)
// ---------------------------------------------------------------------------------------------------------------
template <int DK, int DV, bool CH>
__global__ void __launch_bounds__(CS_THREADS, 2)
delta_read_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ g,
                  const int* __restrict__ cu_q, const int* __restrict__ req_slot, int E, int item0, int num_slots,
                  const float* __restrict__ s0, const float* __restrict__ ut, const float* __restrict__ mm,
                  const float* __restrict__ pre_in, float* __restrict__ o, int H, int Hk) {
  constexpr int KP = DK + 8;
  extern __shared__ __align__(16) unsigned char cs_smem[];
  bf16* qs = reinterpret_cast<bf16*>(cs_smem);                 // [3][64][KP]
  bf16* Mp = qs + 3 * CS_C * KP;                               // [3][64][DC_LP]
  __shared__ float av[CS_C], pre[CS_C];
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int item = blockIdx.x, h = blockIdx.y, hk = h / (H / Hk);
  int e, chunk;
  if (!cs_item(item0 + item, cu_q, E, e, chunk)) return;
  const int slot = req_slot[e];
  const int base = cu_q[e] + chunk * CS_C, n = min(CS_C, cu_q[e + 1] - base);
  const long Cq = (long)Hk * DK, Cv = (long)H * DV;
  float* orow = o + (size_t)base * Cv + (size_t)h * DV;
  if (slot < 0 || slot >= num_slots) {       // a padding entry: defined output, nothing read
    for (int i = tid; i < n * DV; i += CS_THREADS) orow[(size_t)(i / DV) * Cv + i % DV] = 0.f;
    return;
  }
  const size_t ih = (size_t)item * H + h;
  const float* qrow = qn + (size_t)base * Cq + hk * DK;
  const int mt = lane >> 3, r = lane & 7, gr = lane >> 2, c = lane & 3;
  {
    CsTile<float, DK, KP, CS_THREADS> qt;
    CsTile<float, CS_C, DC_LP, CS_THREADS> m_;
    if (CH) qt.ask(pre_in + ih * CS_C * DK, DK, n);
    else qt.ask(qrow, Cq, n);
    m_.ask(mm + ih * CS_C * CS_C, CS_C, CS_C);
    if (!CH && tid < CS_C) {
      av[tid] = tid < n ? g[(size_t)(base + tid) * H + h] : 1.f;
      pre[tid] = pre_in[ih * CS_C + tid];
    }
    qt.put(qs);
    m_.put(Mp);
  }
  __syncthreads();
  const unsigned qs_b = ms_smem(qs), mp_b = ms_smem(Mp);
  const int v0 = warp * 16;
  if (v0 >= DV) return;
  float acc[4][2][4] = {};
  const float* srow = s0 + (ih * DV + v0 + gr) * DK + 2 * c;
  const float* urow = ut + (ih * DV + v0 + gr) * CS_C + 2 * c;
  float2 raw[2][2];                                          // [8 columns][8 channels or tokens]
  auto ask = [&](const float* p, int pitch) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q) raw[i][q] = *reinterpret_cast<const float2*>(p + (size_t)(8 * i) * pitch + 8 * q);
  };
  auto terms = [&](unsigned (&b)[2][3][2]) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q) ms_split(raw[i][q].x, raw[i][q].y, b[i][0][q], b[i][1][q], b[i][2][q]);
  };
  float low[4][2][4] = {};
  ask(srow, DK);
#pragma unroll 1
  for (int kt = 0; kt < DK / 16; ++kt) {
    unsigned b[2][3][2];
    terms(b);
    if (kt + 1 < DK / 16) ask(srow + (kt + 1) * 16, DK);
    else ask(urow, CS_C);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      unsigned a[3][4];
#pragma unroll
      for (int p = 0; p < 3; ++p)
        ms_ldm4(a[p], qs_b + 2 * ((p * CS_C + i * 16 + (mt & 1) * 8 + r) * KP + kt * 16 + (mt >> 1) * 8));
      ms_terms<2, 3, 3>(acc[i], low[i], a, b);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float f0 = CH ? 1.f : pre[i * 16 + gr], f1 = CH ? 1.f : pre[i * 16 + gr + 8];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][nt][j] = (acc[i][nt][j] + low[i][nt][j]) * (j < 2 ? f0 : f1);
        low[i][nt][j] = 0.f;
      }
  }
#pragma unroll
  for (int kt = 0; kt < 4; ++kt) {
    unsigned b[2][3][2];
    terms(b);
    if (kt + 1 < 4) ask(urow + (kt + 1) * 16, CS_C);
#pragma unroll
    for (int i = kt; i < 4; ++i) {
      unsigned a[3][4];
#pragma unroll
      for (int p = 0; p < 3; ++p)
        ms_ldm4(a[p], mp_b + 2 * ((p * CS_C + i * 16 + (mt & 1) * 8 + r) * DC_LP + kt * 16 + (mt >> 1) * 8));
      ms_terms<2, 3, 3>(acc[i], low[i], a, b);
    }
  }
  bool odd = false;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][nt][j] += low[i][nt][j];
        odd |= !(fabsf(acc[i][nt][j]) < INFINITY);
      }
  if (odd) {
    const float* krow = kn + (size_t)base * Cq + hk * DK;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = i * 16 + gr + 8 * (j >> 1);
          const size_t v = ih * DV + v0 + nt * 8 + 2 * c + (j & 1);
          if (t < n && !(fabsf(acc[i][nt][j]) < INFINITY))
            acc[i][nt][j] = CH ? dc_number<DK>(qrow, krow, Cq, ut + v * CS_C, s0 + v * DK, g + ((size_t)base * H + h) * DK, (long)H * DK, 1, t)
                               : dc_number<DK>(qrow, krow, Cq, ut + v * CS_C, s0 + v * DK, av, 1, 0, t);
        }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int t = i * 16 + gr + 8 * q;
      if (t >= n) continue;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
        *reinterpret_cast<float2*>(orow + (size_t)t * Cv + v0 + nt * 8 + 2 * c) = make_float2(acc[i][nt][2 * q], acc[i][nt][2 * q + 1]);
    }
}

template <int DK, int DV, bool CH>
static int dc_scan(const float* qn, const float* kn, const float* vc, const float* beta, const float* g, float* state,
                   long state_stride, int num_slots, const int* cu_q, const int* req_slot, float* o, int E, int H, int Hk,
                   float* s0, float* ut, unsigned* wt, unsigned* kp, float* m, float* suf, float* pre, float* gam, int items, int most,
                   int* status, cudaStream_t stream) {
  const size_t solve = CH ? 4 * (size_t)CS_C * (4 * (DK + 8) + 20) + 2 * (size_t)3 * CS_C * (DC_LP + DC_TP) + 4 * (size_t)20 * DK
                          : 2 * (size_t)3 * CS_C * (DK + 8 + DC_LP + DC_TP) + 4 * (size_t)CS_C * (20 + DC_GP);
  const size_t walk = 2 * (size_t)4 * 3 * CS_C * DK + 2 * (size_t)3 * 16 * (DK + 8 + CS_C + 8) + 16 * (size_t)CS_THREADS;
  const size_t read = 2 * (size_t)3 * CS_C * (DK + 8 + DC_LP);
  cudaError_t rc;
  if constexpr (CH) rc = cs_room<delta_solve_channels_kernel<DK, DV>>(solve);
  else rc = cs_room<delta_solve_kernel<DK, DV>>(solve);
  if (rc != cudaSuccess) return (int)rc;
  rc = cs_room<delta_walk_kernel<DK, CH>>(walk);
  if (rc != cudaSuccess) return (int)rc;
  rc = cs_room<delta_read_kernel<DK, DV, CH>>(read);
  if (rc != cudaSuccess) return (int)rc;
  for (int item0 = 0; item0 < items; item0 += most) {
    const int part = items - item0 < most ? items - item0 : most;
    if constexpr (CH)
      ll_launch(delta_solve_channels_kernel<DK, DV>, dim3(part, H), dim3(DC_CH_THREADS), solve, stream, qn, kn, vc, beta, g, cu_q,
                req_slot, E, item0, ut, wt, kp, m, pre, gam, H, Hk);
    else
      ll_launch(delta_solve_kernel<DK, DV>, dim3(part, H), dim3(CS_THREADS), solve, stream, qn, kn, vc, beta, g, cu_q, req_slot, E,
                item0, ut, wt, kp, m, suf, pre, gam, H, Hk);
    ll_launch(delta_walk_kernel<DK, CH>, dim3(DV / 16, H, E), dim3(CS_THREADS), walk, stream, ut, (const unsigned*)wt, (const unsigned*)kp,
              (const float*)suf, (const float*)gam, s0, state, state_stride, num_slots, cu_q, req_slot, E, item0, part, H, Hk, DV, status);
    ll_launch(delta_read_kernel<DK, DV, CH>, dim3(part, H), dim3(CS_THREADS), read, stream, qn, kn, g, cu_q, req_slot, E, item0,
              num_slots, (const float*)s0, (const float*)ut, (const float*)m, (const float*)pre, o, H, Hk);
  }
  return LL_LAUNCH_RESULT();
}

// The recurrence of ll_delta_recurrence (delta_rule.cu) by chunks: three launches.  `chunks`: at least the number of chunks of 64 tokens
// of the step's entries.  More than `items` of them are done `items` at a time, the states go on in the records (the same bits).
// Scratch, 32 bits a number, at multiples of 16 bytes: s0 [items][H][dv][dk], ut [items][H][dv][64], wt
// [items][H][96 dk], m [items][H][64][64]; with one decay a head kp [items][Hk][96 dk], suf and pre [items][H][64], gam [items][H];
// with one a channel kp [items][H][96 dk], pre [items][H][64][dk], gam [items][H][dk] and no suf.
extern "C" int ll_chunk_delta_scan(const float* qn, const float* kn, const float* vc, const float* beta, const float* g,
                                   float* state, long state_stride, int num_slots, const int* cu_q, const int* req_slot,
                                   float* o, int num_entries, int H, int Hk, int dk, int dv, int per_channel, float* s0, float* ut,
                                   void* wt, void* kp, float* m, float* suf, float* pre, float* gam, int items, int chunks,
                                   int* status, cudaStream_t stream) {
  if (num_entries <= 0 || chunks <= 0) return 0;
  if (items <= 0) return (int)cudaErrorInvalidValue;
  if (H <= 0 || Hk <= 0 || H % Hk || H > 65535 || num_entries > 65535 || ((uintptr_t)wt | (uintptr_t)kp | (uintptr_t)ut) % 16 != 0)
    return (int)cudaErrorInvalidValue;
  if (per_channel && ((uintptr_t)g | (uintptr_t)pre | (uintptr_t)gam) % 16 != 0) return (int)cudaErrorInvalidValue;
#define DC_SCAN(DK, DV)                                                                                                              \
  if (dk == DK && dv == DV)                                                                                                          \
  return per_channel ? dc_scan<DK, DV, true>(qn, kn, vc, beta, g, state, state_stride, num_slots, cu_q, req_slot, o, num_entries, H, \
                                             Hk, s0, ut, (unsigned*)wt, (unsigned*)kp, m, suf, pre, gam, chunks, items, status, stream)      \
                     : dc_scan<DK, DV, false>(qn, kn, vc, beta, g, state, state_stride, num_slots, cu_q, req_slot, o, num_entries, H, \
                                              Hk, s0, ut, (unsigned*)wt, (unsigned*)kp, m, suf, pre, gam, chunks, items, status, stream)
  DC_SCAN(128, 128);
  DC_SCAN(128, 64);
  DC_SCAN(64, 128);
  DC_SCAN(64, 64);
#undef DC_SCAN
  return (int)cudaErrorInvalidValue;
}
