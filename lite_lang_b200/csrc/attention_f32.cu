// Paged attention in true float32 on tensor cores (head size 64 or 128, any page size and group): prompt portions, and single tokens
// (groups of up to 16 heads have a kernel of their own, attn_f32_few).
//
// The float32 path's general kernel (attention_generic.cu) gives a block a (token, kv head) pair and reads the keys once for
// its group of heads only: 337 us for two prompts of 262 and 439 tokens with 12 heads of 128 on 2 kv heads (50 us here).  Here a CTA
// takes 64 rows (a row = a (token, query head of the kv head's group) pair, token-major), so the keys are read once for 64 rows, and
// both products run on mma.sync with every float32 operand as three bfloat16 terms that hold its 24 bits (mma_split.cuh):
//   S [64 x 32]  = Q K^T     a warp 16 rows, 6 products a step of 16 channels
//   O [64 x HD] += P V       P from the accumulators' registers
// Two groups of four warps walk the tiles of 32 keys alternately, each with its own maximum, sum and O, and meet at the end in
// shared memory: two tiles are on their way at a time and one group's softmax lies beside the other's products.  A tile's rows
// come by cp.async as stored, a tile ahead of the group's use of them (the pages' numbers a tile ahead of that), and become
// terms in shared memory when their turn comes: asked for where they were needed, the trips to memory were 40 % of the time.
//
// Scores, softmax (expf) and sums are float32.  Keys that a row may not see get probability 0 by selection; the V of keys that
// no row of the CTA sees are zeros, whatever the page holds.  Tiles start at multiples of 32 positions and a group takes every
// other one of the context's, so the order of a row's sums depends on its position only.
//
// Infinities and numbers above 3.39e38 have no bfloat16 terms, and a probability of 0 makes NaN of an infinity in V that other
// rows of the CTA see: a row that comes out with NaN is made again by a warp in multiply-adds (`af_plain_row`), as
// attention_generic.cu would.
#include "mma_split.cuh"

#define AF_THREADS 256
#define AF_TK 32
#define AF_ROWS 64

struct AttnF32Params {
  float* out;
  long out_stride;
  const float* q;
  long q_stride;
  const float* k_cache;      // [pages, nkv, page_size, HD]
  const float* v_cache;
  const int* block_table;
  int bt_stride;
  const int* cu_q;
  const int* ctx_len;
  const int* req_slot;
  int n_entries, nkv, group, page_size, num_pages, window, row_blocks;
  float scale;
  int* status;
};

// one row by one warp: keys lo .. pos of the table `bt`, HD / 32 channels a lane
template <int HD>
__device__ __forceinline__ void af_plain_row(const AttnF32Params& p, const int* bt, int kvh, int lo, int pos, const float* q, float* out) {
  constexpr int N = HD / 32;
  const int lane = threadIdx.x & 31;
  float x[N], o[N] = {}, m = -INFINITY, l = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = q[lane + 32 * i];
  for (int j = lo; j <= pos && l == l; ++j) {        // (a sum that is NaN stays NaN)
    const int lp = j / p.page_size, page = lp < p.bt_stride ? bt[lp] : -1;
    if (page < 0 || page >= p.num_pages) continue;   // (has been reported)
    const size_t at = (((size_t)page * p.nkv + kvh) * p.page_size + j % p.page_size) * HD;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) s = fmaf(x[i], p.k_cache[at + lane + 32 * i], s);
    s = warp_sum(s) * p.scale;
    const float n = fmaxf(m, s), u = n == -INFINITY ? 0.f : n, f = expf(m - u), w = expf(s - u);
    m = n;
    l = fmaf(l, f, w);
#pragma unroll
    for (int i = 0; i < N; ++i) o[i] = fmaf(o[i], f, w * p.v_cache[at + lane + 32 * i]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) out[lane + 32 * i] = l != l ? l : l > 0.f ? o[i] / l : 0.f;
}

template <int HD>
__global__ void __launch_bounds__(AF_THREADS, 1)
attn_f32_kernel(const AttnF32Params p) {
  constexpr int P = HD + 8, NO = HD / 8, LOADS = AF_TK * HD / 4 / 128;      // 16-byte pieces of K (and of V) a thread brings
  constexpr int TERMS = 3 * P * (AF_ROWS + 4 * AF_TK);         // bfloat16 numbers before the rows as stored
  extern __shared__ __align__(16) unsigned char af_smem[];
  bf16* qs = reinterpret_cast<bf16*>(af_smem);                 // [3][64][P]
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = warp >> 2, gt = tid & 127;
  bf16* ks = qs + 3 * AF_ROWS * P + half * (6 * AF_TK * P);    // this group's tile: K [3][32][P], V [3][32][P]
  bf16* vs = ks + 3 * AF_TK * P;
  float* raw = reinterpret_cast<float*>(qs + TERMS) + half * (2 * AF_TK * HD);       // K [32][HD], V [32][HD] as stored
  const int kvh = blockIdx.y;
  int rb = p.row_blocks - 1 - blockIdx.x;                      // the later, heavier blocks of the step first
  int entry = -1, rows = 0;
  for (int e = 0; e < p.n_entries; ++e) {
    const int n = (p.cu_q[e + 1] - p.cu_q[e]) * p.group, nb = (n + AF_ROWS - 1) / AF_ROWS;
    if (rb < nb) {
      entry = e;
      rows = n;
      break;
    }
    rb -= nb;
  }
  if (entry < 0) return;
  const int slot = p.req_slot[entry], tok0 = p.cu_q[entry], ctx = p.ctx_len[entry];
  const int r0 = rb * AF_ROWS, rl = min(rows, r0 + AF_ROWS) - 1;       // rows r0 .. rl of the entry
  const int head0 = kvh * p.group;
  if (slot < 0) {
    for (int i = tid; i < (rl - r0 + 1) * HD; i += AF_THREADS) {
      const int r = r0 + i / HD;
      p.out[(size_t)(tok0 + r / p.group) * p.out_stride + (size_t)(head0 + r % p.group) * HD + i % HD] = 0.f;
    }
    return;
  }
  const int hi = ctx + rl / p.group, lo = p.window > 0 ? max(0, ctx + r0 / p.group - p.window + 1) : 0;
  const int tile0 = lo / AF_TK, tiles = hi / AF_TK - tile0 + 1;
  const int* bt = p.block_table + (size_t)slot * p.bt_stride;
  const int own = half ^ (tile0 & 1);                          // this group's first tile: the even or the odd ones of the context

  // lane l: where the row of key l of a tile starts in the planes (-1: not seen by any row of the CTA)
  auto place = [&](int tile) -> long {
    const int pos = (tile0 + tile) * AF_TK + lane;
    if (pos < lo || pos > hi) return -1;
    const int lp = pos / p.page_size, page = lp < p.bt_stride ? bt[lp] : -1;
    if (page < 0 || page >= p.num_pages) {
      set_status(p.status, LL_ERR_PAGE_RANGE);
      return -1;
    }
    return (((long)page * p.nkv + kvh) * p.page_size + pos % p.page_size) * HD;
  };
  const unsigned raw_b = ms_smem(raw);
  auto ask = [&](long base) {                                  // a tile's rows (keys that nobody sees: zeros)
#pragma unroll
    for (int j = 0; j < LOADS; ++j) {
      const int i = j * 128 + gt, kk = i / (HD / 4), c = (i % (HD / 4)) * 4;
      const long at = __shfl_sync(0xffffffffu, base, kk);
      const long from = (at < 0 ? 0 : at) + c;
      const int bytes = at < 0 ? 0 : 16;
      const unsigned dst = raw_b + 4 * (kk * HD + c);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(p.k_cache + from), "r"(bytes) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 4 * AF_TK * HD), "l"(p.v_cache + from), "r"(bytes)
                   : "memory");
    }
    ms_commit();
  };
  auto put4 = [](bf16* d, const float4& v, int plane) {
    uint2 t0, t1, t2;
    ms_split(v.x, v.y, t0.x, t1.x, t2.x);
    ms_split(v.z, v.w, t0.y, t1.y, t2.y);
    *reinterpret_cast<uint2*>(d) = t0;
    *reinterpret_cast<uint2*>(d + plane) = t1;
    *reinterpret_cast<uint2*>(d + 2 * plane) = t2;
  };
  auto put = [&](bf16* dst, const float* src) {
#pragma unroll
    for (int j = 0; j < LOADS; ++j) {
      const int i = j * 128 + gt, kk = i / (HD / 4), cc = (i % (HD / 4)) * 4;
      put4(dst + kk * P + cc, *reinterpret_cast<const float4*>(src + kk * HD + cc), AF_TK * P);
    }
  };
  long next = -1;
  if (own < tiles) ask(place(own));
  if (own + 2 < tiles) next = place(own + 2);
  for (int i = tid; i < AF_ROWS * (HD / 4); i += AF_THREADS) {
    const int rr = i / (HD / 4), c = (i % (HD / 4)) * 4, r = r0 + rr;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r <= rl) v = *reinterpret_cast<const float4*>(p.q + (size_t)(tok0 + r / p.group) * p.q_stride + (size_t)(head0 + r % p.group) * HD + c);
    put4(qs + rr * P + c, v, AF_ROWS * P);
  }
  __syncthreads();
  const int m8 = lane >> 3, r8 = lane & 7, g = lane >> 2, c = lane & 3;
  const int row = (warp & 3) * 16;
  const unsigned qs_b = ms_smem(qs), ks_b = ms_smem(ks), vs_b = ms_smem(vs);
  const int ra = r0 + row + g, rb8 = ra + 8;                   // the thread's two rows, their positions
  const int pa = ra <= rl ? ctx + ra / p.group : -1, pb = rb8 <= rl ? ctx + rb8 / p.group : -1;
  const int la = p.window > 0 ? pa - p.window + 1 : 0, lb = p.window > 0 ? pb - p.window + 1 : 0;
  float o[NO][4], m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
#pragma unroll
  for (int i = 0; i < NO; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  for (int tile = own; tile < tiles; tile += 2) {
    ms_wait<0>();
    asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");      // the rows are here, the tile before has been read
    put(ks, raw);
    put(vs, raw + AF_TK * HD);
    asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
    if (tile + 2 < tiles) ask(next);
    if (tile + 4 < tiles) next = place(tile + 4);
    float s[4][4], low[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = low[i][j] = 0.f;
#pragma unroll
    for (int kt = 0; kt < HD / 16; ++kt) {
      unsigned a[3][4], b[4][3][2];
#pragma unroll
      for (int q = 0; q < 3; ++q)
        ms_ldm4(a[q], qs_b + 2 * ((q * AF_ROWS + row + (m8 & 1) * 8 + r8) * P + kt * 16 + (m8 >> 1) * 8));
      const unsigned at = ks_b + 2 * (((m8 >> 1) * 8 + r8) * P + kt * 16 + (m8 & 1) * 8);
      ms_load_b<3, false>(b, at, 2 * AF_TK * P);
      ms_load_b<3, false>(b + 2, at + 2 * 16 * P, 2 * AF_TK * P);
      ms_terms<4, 3, 3>(s, low, a, b);
    }
    const int k0 = (tile0 + tile) * AF_TK;
    float x0 = -INFINITY, x1 = -INFINITY;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int pos = k0 + i * 8 + 2 * c + (j & 1);
        const bool seen = j < 2 ? (pos <= pa && pos >= la) : (pos <= pb && pos >= lb);
        s[i][j] = seen ? (s[i][j] + low[i][j]) * p.scale : -INFINITY;
        if (j < 2) x0 = fmaxf(x0, s[i][j]);
        else x1 = fmaxf(x1, s[i][j]);
      }
#pragma unroll
    for (int w = 1; w < 4; w <<= 1) {
      x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, w));
      x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, w));
    }
    const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
    const float u0 = n0 == -INFINITY ? 0.f : n0, u1 = n1 == -INFINITY ? 0.f : n1;
    const float f0 = expf(m0 - u0), f1 = expf(m1 - u1);          // (-inf: nothing so far, 0)
    m0 = n0;
    m1 = n1;
    float t0 = 0.f, t1 = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s[i][0] = expf(s[i][0] - u0);
      s[i][1] = expf(s[i][1] - u0);
      s[i][2] = expf(s[i][2] - u1);
      s[i][3] = expf(s[i][3] - u1);
      t0 += s[i][0] + s[i][1];
      t1 += s[i][2] + s[i][3];
    }
    l0 = l0 * f0 + t0;
    l1 = l1 * f1 + t1;
    unsigned a[2][3][4];
#pragma unroll
    for (int kt = 0; kt < 2; ++kt)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        ms_split(s[2 * kt + q][0], s[2 * kt + q][1], a[kt][0][2 * q], a[kt][1][2 * q], a[kt][2][2 * q]);
        ms_split(s[2 * kt + q][2], s[2 * kt + q][3], a[kt][0][2 * q + 1], a[kt][1][2 * q + 1], a[kt][2][2 * q + 1]);
      }
#pragma unroll
    for (int nt = 0; nt < NO; nt += 4) {
      float d[4][4], small[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) d[i][j] = small[i][j] = 0.f;
#pragma unroll
      for (int kt = 0; kt < 2; ++kt) {
        unsigned b[4][3][2];
        const unsigned at = vs_b + 2 * ((kt * 16 + (m8 & 1) * 8 + r8) * P + nt * 8 + (m8 >> 1) * 8);
        ms_load_b<3, true>(b, at, 2 * AF_TK * P);
        ms_load_b<3, true>(b + 2, at + 32, 2 * AF_TK * P);
        ms_terms<4, 3, 3>(d, small, a[kt], b);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[nt + i][j] = fmaf(o[nt + i][j], j < 2 ? f0 : f1, d[i][j] + small[i][j]);
    }
  }
  // sums over the four lanes of a row, then the second group's rows join the first's
#pragma unroll
  for (int w = 1; w < 4; w <<= 1) {
    l0 += __shfl_xor_sync(0xffffffffu, l0, w);
    l1 += __shfl_xor_sync(0xffffffffu, l1, w);
  }
  __syncthreads();                                             // nobody's tile or query is needed any more
  float* meet = reinterpret_cast<float*>(af_smem);             // [64][HD + 8]: O, then maximum and sum at HD, HD + 1
  if (half == 1) {
    float* d0 = meet + (row + g) * P;
    float* d1 = d0 + 8 * P;
#pragma unroll
    for (int i = 0; i < NO; ++i) {
      *reinterpret_cast<float2*>(d0 + i * 8 + 2 * c) = make_float2(o[i][0], o[i][1]);
      *reinterpret_cast<float2*>(d1 + i * 8 + 2 * c) = make_float2(o[i][2], o[i][3]);
    }
    if (c == 0) {
      d0[HD] = m0; d0[HD + 1] = l0;
      d1[HD] = m1; d1[HD + 1] = l1;
      d0[HD + 2] = d1[HD + 2] = 0.f;      // not zero: the row has NaN
    }
  }
  __syncthreads();
  if (half == 0) {
    float* s0 = meet + (row + g) * P;
    float* s1 = s0 + 8 * P;
    bool nan0 = false, nan1 = false;
    auto weights = [](float m, float l, float mq, float lq, float& w, float& wq) {
      const float top = fmaxf(m, mq), u = top == -INFINITY ? 0.f : top;
      w = expf(m - u);
      wq = expf(mq - u);
      const float sum = l * w + lq * wq, inv = sum > 0.f ? 1.0f / sum : 0.f;
      w *= inv;
      wq *= inv;
    };
    float w0, q0, w1, q1;
    weights(m0, l0, s0[HD], s0[HD + 1], w0, q0);
    weights(m1, l1, s1[HD], s1[HD + 1], w1, q1);
    float* oa = p.out + (size_t)(tok0 + ra / p.group) * p.out_stride + (size_t)(head0 + ra % p.group) * HD + 2 * c;
    float* ob = p.out + (size_t)(tok0 + rb8 / p.group) * p.out_stride + (size_t)(head0 + rb8 % p.group) * HD + 2 * c;
#pragma unroll
    for (int i = 0; i < NO; ++i) {
      const float2 x = *reinterpret_cast<const float2*>(s0 + i * 8 + 2 * c), y = *reinterpret_cast<const float2*>(s1 + i * 8 + 2 * c);
      const float2 a = make_float2(o[i][0] * w0 + x.x * q0, o[i][1] * w0 + x.y * q0);
      const float2 b = make_float2(o[i][2] * w1 + y.x * q1, o[i][3] * w1 + y.y * q1);
      nan0 |= a.x != a.x || a.y != a.y;
      nan1 |= b.x != b.x || b.y != b.y;
      if (ra <= rl) *reinterpret_cast<float2*>(oa + i * 8) = a;
      if (rb8 <= rl) *reinterpret_cast<float2*>(ob + i * 8) = b;
    }
    if (nan0) s0[HD + 2] = 1.f;
    if (nan1) s1[HD + 2] = 1.f;
  }
  __syncthreads();
  for (int rr = warp; rr <= rl - r0; rr += AF_THREADS / 32)
    if (meet[rr * P + HD + 2] != 0.f) {
      const int r = r0 + rr, pos = ctx + r / p.group;
      const size_t t = tok0 + r / p.group, h = (size_t)(head0 + r % p.group) * HD;
      af_plain_row<HD>(p, bt, kvh, p.window > 0 ? max(0, pos - p.window + 1) : 0, pos, p.q + t * p.q_stride + h, p.out + t * p.out_stride + h);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Steps of single tokens, groups of at most 16 heads: a warp has all rows (16, those behind the group's are zeros) and tiles of 16
// keys of its own, so that no row of the other kernel's 64 is multiplied for nothing (its four warps a tile had 16 rows each, and the
// tensor pipe of a step of single tokens was busy with zeros).  Keys and values come by cp.async as stored, two of a warp's three
// places on their way, and become terms in the registers of the one warp that needs them.  A cluster of CTAs takes the warps' tiles in
// turn (tile t to warp t mod 8 C), so that few tokens fill the SMs too; the order of a row's sums depends on C, that is on how many
// tokens decode together, within rounding.  12 heads on 2, contexts around 2,000 (heads of 128), the other kernel /
// this one, us: 1 token 194 / 15, 16 tokens 268 / 32, 64 tokens 278 / 96.
// ---------------------------------------------------------------------------------------------------------------
#define AF_FEW 16
__device__ __forceinline__ void af_cluster_sync() {
  asm volatile("barrier.cluster.arrive;" ::: "memory");
  asm volatile("barrier.cluster.wait;" ::: "memory");
}
__device__ __forceinline__ float af_peer(const float* x, int z) {      // CTA z's number of that place
  unsigned at;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(ms_smem(x)), "r"(z));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}

template <int HD>
__global__ void __launch_bounds__(AF_THREADS, 1)
attn_f32_few_kernel(const AttnF32Params p, int ctas) {
  constexpr int P = HD + 8, PF = HD + 8, NO = HD / 8, WARPS = AF_THREADS / 32, PLACES = 3, LOADS = AF_FEW * HD / 4 / 32;
  constexpr int PLACE = AF_FEW * PF;                           // numbers of a place: 16 keys or values
  extern __shared__ __align__(16) unsigned char af_smem[];
  __shared__ float top[WARPS][AF_FEW], sum[WARPS][AF_FEW], part[2][AF_FEW];
  __shared__ int bad[AF_FEW];
  bf16* qs = reinterpret_cast<bf16*>(af_smem);                 // [3][16][P]
  float* places = reinterpret_cast<float*>(qs + 3 * AF_FEW * P);
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int entry = blockIdx.x, kvh = blockIdx.y, rank = blockIdx.z;
  const int slot = p.req_slot[entry], t = p.cu_q[entry], pos = p.ctx_len[entry], head0 = kvh * p.group;
  float* out = p.out + (size_t)t * p.out_stride + (size_t)head0 * HD;
  if (slot < 0) {                                              // (the cluster's CTAs have the same entry)
    if (rank == 0)
      for (int i = tid; i < p.group * HD; i += AF_THREADS) out[i] = 0.f;
    return;
  }
  const float* qrow = p.q + (size_t)t * p.q_stride + (size_t)head0 * HD;
  const int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0, first = lo / AF_FEW, tiles = pos / AF_FEW - first + 1;
  const int* bt = p.block_table + (size_t)slot * p.bt_stride;
  const int step = WARPS * ctas;
  float* mine = places + warp * PLACES * PLACE;
  // lane l: where the row of key l % 16 of a tile starts in the planes; -1: not seen
  auto place = [&](int tile) -> long {
    const int at = (first + tile) * AF_FEW + (lane & 15);
    if (tile >= tiles || at < lo || at > pos) return -1;
    const int lp = at / p.page_size, page = lp < p.bt_stride ? bt[lp] : -1;
    if (page < 0 || page >= p.num_pages) {
      set_status(p.status, LL_ERR_PAGE_RANGE);
      return -1;
    }
    return (((long)page * p.nkv + kvh) * p.page_size + at % p.page_size) * HD;
  };
  auto ask = [&](const float* plane, long base, int where) {   // 16 rows (zeros for keys that are not seen)
    const unsigned dst = ms_smem(mine + where * PLACE);
#pragma unroll
    for (int j = 0; j < LOADS; ++j) {
      const int i = j * 32 + lane, kk = i / (HD / 4), c = (i % (HD / 4)) * 4;
      const long at = __shfl_sync(0xffffffffu, base, kk);
      const int bytes = at < 0 ? 0 : 16;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 4 * (kk * PF + c)), "l"(plane + (at < 0 ? 0 : at) + c), "r"(bytes)
                   : "memory");
    }
  };
  int tile = rank * WARPS + warp, asked = tile;                // the next tile to ask K of
  long kbase = place(asked), vbase = -1;
  int where = 0;                                               // the place that is asked for next
  auto next_k = [&]() {
    if (asked < tiles) ask(p.k_cache, kbase, where);
    ms_commit();
    vbase = kbase;
    asked += step;
    kbase = place(asked);
    where = where == PLACES - 1 ? 0 : where + 1;
  };
  auto next_v = [&]() {
    if (asked - step < tiles) ask(p.v_cache, vbase, where);
    ms_commit();
    where = where == PLACES - 1 ? 0 : where + 1;
  };
  next_k();
  next_v();
  next_k();
  for (int i = tid; i < AF_FEW * (HD / 4); i += AF_THREADS) {
    const int r = i / (HD / 4), c = (i % (HD / 4)) * 4;
    const float4 v = r < p.group ? *reinterpret_cast<const float4*>(qrow + (size_t)r * HD + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    uint2 t0, t1, t2;
    ms_split(v.x, v.y, t0.x, t1.x, t2.x);
    ms_split(v.z, v.w, t0.y, t1.y, t2.y);
    *reinterpret_cast<uint2*>(qs + r * P + c) = t0;
    *reinterpret_cast<uint2*>(qs + (AF_FEW + r) * P + c) = t1;
    *reinterpret_cast<uint2*>(qs + (2 * AF_FEW + r) * P + c) = t2;
  }
  if (tid < AF_FEW) bad[tid] = 0;
  __syncthreads();
  const int m8 = lane >> 3, r8 = lane & 7, g = lane >> 2, c = lane & 3;
  const unsigned qs_b = ms_smem(qs) + 2 * (((m8 & 1) * 8 + r8) * P + (m8 >> 1) * 8);
  float o[NO][4], m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
#pragma unroll
  for (int i = 0; i < NO; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  int have = 0;                                                // the place that is read next
  for (; tile < tiles; tile += step) {
    ms_wait<PLACES - 1>();
    __syncwarp();
    const float* kf = mine + have * PLACE + g * PF + 2 * c;
    float s[2][4] = {}, low[2][4] = {};
#pragma unroll
    for (int kt = 0; kt < HD / 16; ++kt) {
      unsigned a[3][4], b[2][3][2];
#pragma unroll
      for (int q = 0; q < 3; ++q) ms_ldm4(a[q], qs_b + 2 * (q * AF_FEW * P + kt * 16));
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 x = *reinterpret_cast<const float2*>(kf + nt * 8 * PF + kt * 16 + q * 8);
          ms_split(x.x, x.y, b[nt][0][q], b[nt][1][q], b[nt][2][q]);
        }
      ms_terms<2, 3, 3>(s, low, a, b);
    }
    __syncwarp();
    next_v();
    have = have == PLACES - 1 ? 0 : have + 1;
    const int k0 = (first + tile) * AF_FEW;
    float x0 = -INFINITY, x1 = -INFINITY;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int at = k0 + i * 8 + 2 * c + (j & 1);
        s[i][j] = at <= pos && at >= lo ? (s[i][j] + low[i][j]) * p.scale : -INFINITY;
        if (j < 2) x0 = fmaxf(x0, s[i][j]);
        else x1 = fmaxf(x1, s[i][j]);
      }
#pragma unroll
    for (int w = 1; w < 4; w <<= 1) {
      x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, w));
      x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, w));
    }
    const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
    const float u0 = n0 == -INFINITY ? 0.f : n0, u1 = n1 == -INFINITY ? 0.f : n1;
    const float f0 = expf(m0 - u0), f1 = expf(m1 - u1);          // (-inf: nothing so far, 0)
    m0 = n0;
    m1 = n1;
    float t0 = 0.f, t1 = 0.f;
    unsigned a[3][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      s[i][0] = expf(s[i][0] - u0);
      s[i][1] = expf(s[i][1] - u0);
      s[i][2] = expf(s[i][2] - u1);
      s[i][3] = expf(s[i][3] - u1);
      t0 += s[i][0] + s[i][1];
      t1 += s[i][2] + s[i][3];
      ms_split(s[i][0], s[i][1], a[0][2 * i], a[1][2 * i], a[2][2 * i]);
      ms_split(s[i][2], s[i][3], a[0][2 * i + 1], a[1][2 * i + 1], a[2][2 * i + 1]);
    }
    l0 = l0 * f0 + t0;
    l1 = l1 * f1 + t1;
    ms_wait<PLACES - 1>();
    __syncwarp();
    const float* vf = mine + have * PLACE + 2 * c * PF + g;
#pragma unroll
    for (int nt = 0; nt < NO; nt += 4) {
      float d[4][4], small[4][4];
      unsigned b[4][3][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) d[i][j] = small[i][j] = 0.f;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float* at = vf + 8 * q * PF + (nt + i) * 8;
          ms_split(at[0], at[PF], b[i][0][q], b[i][1][q], b[i][2][q]);
        }
      }
      ms_terms<4, 3, 3>(d, small, a, b);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[nt + i][j] = fmaf(o[nt + i][j], j < 2 ? f0 : f1, d[i][j] + small[i][j]);
    }
    __syncwarp();
    next_k();
    have = have == PLACES - 1 ? 0 : have + 1;
  }
  ms_wait<0>();
#pragma unroll
  for (int w = 1; w < 4; w <<= 1) {
    l0 += __shfl_xor_sync(0xffffffffu, l0, w);
    l1 += __shfl_xor_sync(0xffffffffu, l1, w);
  }
  __syncwarp();                                                // the warp's first place holds its rows from now on
  {
    float* d0 = mine + g * PF + 2 * c;
#pragma unroll
    for (int i = 0; i < NO; ++i) {
      *reinterpret_cast<float2*>(d0 + i * 8) = make_float2(o[i][0], o[i][1]);
      *reinterpret_cast<float2*>(d0 + 8 * PF + i * 8) = make_float2(o[i][2], o[i][3]);
    }
    if (c == 0) {
      top[warp][g] = m0; sum[warp][g] = l0;
      top[warp][g + 8] = m1; sum[warp][g + 8] = l1;
    }
  }
  __syncthreads();
  // the CTA's rows: against their largest score, not divided, in the second place of warp 0
  float* own = places + PLACE;
  for (int i = tid; i < p.group * HD; i += AF_THREADS) {
    const int r = i / HD, ch = i % HD;
    float m = -INFINITY, l = 0.f, x = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) m = fmaxf(m, top[w][r]);
    const float u = m == -INFINITY ? 0.f : m;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float f = expf(top[w][r] - u);
      l = fmaf(sum[w][r], f, l);
      x = fmaf(places[w * PLACES * PLACE + r * PF + ch], f, x);
    }
    if (ctas > 1) {
      own[r * PF + ch] = x;
      if (ch == 0) {
        part[0][r] = m;
        part[1][r] = l;
      }
    } else {
      const float y = l > 0.f ? x / l : l != l ? l : 0.f;
      out[i] = y;
      if (y != y) bad[r] = 1;
    }
  }
  if (ctas > 1) {
    af_cluster_sync();
    for (int i = tid; rank + i / HD * ctas < p.group; i += AF_THREADS) {      // every C-th row a CTA
      const int r = rank + i / HD * ctas, ch = i % HD;
      float mz[8], m = -INFINITY, l = 0.f, x = 0.f;
#pragma unroll
      for (int z = 0; z < 8; ++z) {
        mz[z] = z < ctas ? af_peer(&part[0][r], z) : -INFINITY;
        m = fmaxf(m, mz[z]);
      }
      const float u = m == -INFINITY ? 0.f : m;
#pragma unroll
      for (int z = 0; z < 8; ++z)
        if (z < ctas) {
          const float f = expf(mz[z] - u);
          l = fmaf(af_peer(&part[1][r], z), f, l);
          x = fmaf(af_peer(own + r * PF + ch, z), f, x);
        }
      const float y = l > 0.f ? x / l : l != l ? l : 0.f;
      out[r * HD + ch] = y;
      if (y != y) bad[r] = 1;
    }
    af_cluster_sync();                                         // the rows have been read
  }
  __syncthreads();
  for (int r = warp; r < p.group; r += WARPS)
    if (bad[r]) af_plain_row<HD>(p, bt, kvh, lo, pos, qrow + (size_t)r * HD, out + (size_t)r * HD);
}

// q: float32, head h of token t at q + t * q_stride + h * hd; out float32 [tokens, nh * hd].  cu_q, ctx_len, req_slot: the
// entries' arrays (cu_q[e] counts the step's tokens); row_blocks: sum over the entries of ceil(new tokens * group / 64).  ctas: 0, or
// for entries of one token each and groups of at most 16 heads 1, 2, 4 or 8 CTAs a token and kv head.
extern "C" int ll_attn_f32(float* out, long out_stride, const float* q, long q_stride, const float* k_cache,
                           const float* v_cache, const int* block_table, int bt_stride, const int* cu_q, const int* ctx_len,
                           const int* req_slot, int n_entries, int row_blocks, int nh, int nkv, int hd, int page_size,
                           int num_pages, int window, float scale, int ctas, int* status, cudaStream_t stream) {
  if (row_blocks <= 0 || n_entries <= 0) return 0;
  if ((hd != 64 && hd != 128) || nkv <= 0 || nh % nkv != 0 || nkv > 65535 || page_size <= 0 || (q_stride % 4) != 0 ||
      (out_stride % 2) != 0 || (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache) % 16) != 0 || ((uintptr_t)out % 8) != 0)
    return (int)cudaErrorInvalidValue;
  AttnF32Params p{out, out_stride, q, q_stride, k_cache, v_cache, block_table, bt_stride, cu_q, ctx_len, req_slot, n_entries,
                  nkv, nh / nkv, page_size, num_pages, window, row_blocks, scale, status};
  if (ctas != 0) {
    if ((ctas != 1 && ctas != 2 && ctas != 4 && ctas != 8) || p.group > AF_FEW || row_blocks != n_entries) return (int)cudaErrorInvalidValue;
    const size_t few = 2 * (size_t)3 * AF_FEW * (hd + 8) + 4 * (size_t)(AF_THREADS / 32) * 3 * AF_FEW * (hd + 8);
    const dim3 grid(n_entries, nkv, ctas);
    if (hd == 128) {
      const cudaError_t rc = cudaFuncSetAttribute(attn_f32_few_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)few);
      if (rc != cudaSuccess) return (int)rc;
      ll_launch_cluster(attn_f32_few_kernel<128>, grid, dim3(AF_THREADS), few, stream, ctas, p, ctas);
    } else {
      const cudaError_t rc = cudaFuncSetAttribute(attn_f32_few_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)few);
      if (rc != cudaSuccess) return (int)rc;
      ll_launch_cluster(attn_f32_few_kernel<64>, grid, dim3(AF_THREADS), few, stream, ctas, p, ctas);
    }
    return LL_LAUNCH_RESULT();
  }
  const size_t smem = 2 * (size_t)(hd + 8) * 3 * (AF_ROWS + 4 * AF_TK) + 4 * (size_t)hd * 4 * AF_TK;
  if (hd == 128) {
    const cudaError_t rc = cudaFuncSetAttribute(attn_f32_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (rc != cudaSuccess) return (int)rc;
    ll_launch(attn_f32_kernel<128>, dim3(row_blocks, nkv), dim3(AF_THREADS), smem, stream, p);
  } else {
    const cudaError_t rc = cudaFuncSetAttribute(attn_f32_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (rc != cudaSuccess) return (int)rc;
    ll_launch(attn_f32_kernel<64>, dim3(row_blocks, nkv), dim3(AF_THREADS), smem, stream, p);
  }
  return LL_LAUNCH_RESULT();
}
