// Routed feed-forward (mixture of experts): the router and the activation between the two products.
//
// Router, per token, all in float32: logits z = Wr x over the experts, scores by softmax (or sigmoid) over
// all experts, the `top` experts with the largest choice scores (ties: the lower index; the choice scores are the
// scores, or the scores plus a number an expert that the weights do not see), their weights the scores
// themselves or the scores divided by their sum, times a constant.  The choice may be kept to the best groups of
// neighbouring experts.  Outputs of the router beyond the experts stand for the token's row itself (identities).  The result is a dense row of weights per token, zero for
// experts that were not chosen, plus the chosen indices and weights.
//
// The experts' first products run as one product over all experts' rows (an always-on expert's rows first);
// `moe_act` then applies the activation and multiplies every hidden unit by the weight of its expert for that
// token (1 for the always-on rows, 0 for experts not chosen), so that one second product over all hidden units
// gives the weighted sum of the chosen experts' outputs plus the always-on expert's.
#include "mma_split.cuh"
#include "moe_act.cuh"

#define MOE_MAX_E 256

// Wr: float32 [E, hidden]; x: T [tokens, hidden]; gates: float32 [tokens, E]; top_idx int32 / top_w float32
// [tokens, top].  score_fn: 0 softmax over all experts, 1 sigmoid, 2 the `top` largest logits are chosen and
// their weights are a softmax taken over just those logits.  `bias` (float32 [E], optional) is added to the
// logits.  With `shared_w` (float32 [tokens]) the router matrix has one more row, the gate of an expert that
// every token uses: shared_w[t] = sigmoid(Wr[E] . x).  E counts all outputs of the router; `gates` has `real` columns,
// and outputs real .. E - 1 are identities, whose weights add up to identity_w[t].  choice_bias (float32 [E], optional)
// is added to the scores for the choice.  With `keep` < `count`, only outputs of the `keep` groups (E / count neighbours
// each) with the largest best choice score can be chosen.  A place that finds nothing left gets top_idx -1 and weight 0.
//
// Two kernels.  `moe_router_tc_kernel`: portions of bfloat16 rows and at most 32 outputs (experts and the shared one's gate), 16 tokens a
// block on tensor cores.  `moe_router_kernel`: a block takes TOK tokens: one, with a warp an output for at most 24 of them (AWARP),
// which has asked for the first pieces of its row before the token's was there (more outputs keep their warps' loads in flight
// anyway, and were 8 % slower with it: 64 outputs of 2,048 9.2 and 10.0 us, 32 6.4 and 7.0); or eight in long portions, four a warp: the router's
// matrix is then read once for four tokens.  Its warps share out the outputs, and then the tokens, whose scores a warp each makes and picks from.  Bound by
// the loads' latency and the warps in flight.  A lane sums its pieces of four numbers of a row, then the lanes are added up: an
// order that depends on the sizes only.  In `moe_pick` a lane has one of at most 32 outputs, and a pick is one maximum over the
// warp and a ballot.
// Fewest tokens that go to tensor cores.  The other kernel has a token a block, of a warp an output for at most 24 outputs (as many
// blocks an SM as 32 warps hold) and of 32 warps for more: it is the faster one while that is one round of blocks over the 148
// SMs, with 32 warps two.  With at most 8 outputs a tile of the MMA is half empty.  Measured on a B200 (a token a block / tensor
// cores, us): 17 outputs of 1,536, 256 tokens 10.5 / 9.1, 384 14.8 / 9.2; 16 of 2,048, 256 6.3 / 10.0, 320 11.2 / 10.1; 9 of
// 3,584, 384 7.5 / 12.5; 32 of 2,048, 256 11.4 / 12.5, 320 16.8 / 12.5; 32 of 4,096, 256 14.7 / 19.6, 320 21.0 / 19.6; eight
// tokens a block: 9 of 3,584, 512 16.1 / 12.5; 32 of 7,168, 512 39.8 / 29.8; 4 of 1,024, 2,048 6.1 / 8.1, 4,096 12.1 / 8.5.
static int moe_tc_least(int rows) {
  if (rows <= 8) return 4096;
  if (rows > 24) return 2 * 148 + 1;
  const int round = 148 * (32 / rows);
  return round + 1 > 256 ? round + 1 : 256;
}
__device__ __forceinline__ float4 moe_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 moe_load4(const bf16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
// a float32 number as an unsigned one of the same order; NaN below all, the zeros equal
__device__ __forceinline__ unsigned moe_order(float v) {
  const unsigned u = __float_as_uint(v + 0.0f);
  return v != v ? 0u : (u & 0x80000000u) ? ~u : u | 0x80000000u;
}
// What a token's logits z [E + 1] (by one warp, in shared memory, the choice scores and the groups' best behind them) come to:
// its scores, its choice and the weights.
__device__ __forceinline__ void moe_pick(float* z, int t, float* __restrict__ gates, int* __restrict__ top_idx, float* __restrict__ top_w,
                                         float* __restrict__ shared_w, int E, int top, int score_fn, int renormalize,
                                         const float* __restrict__ choice_bias, int count, int keep, float weight_scale,
                                         float* __restrict__ identity_w, int real) {
  const int lane = threadIdx.x & 31;
  float* cs = z + E + 1;                                 // choice scores
  float* gb = cs + E;                                    // the groups' best
  if (shared_w && lane == 0) shared_w[t] = 1.0f / (1.0f + expf(-z[E]));
  if (score_fn == 2) {
    // the logits themselves are compared; the weights are made from the chosen ones below
  } else if (score_fn == 0) {
    float m = -INFINITY;
    for (int e = lane; e < E; e += 32) m = fmaxf(m, z[e]);
    m = warp_max(m);
    float sum = 0.f;
    for (int e = lane; e < E; e += 32) sum += expf(z[e] - m);
    sum = warp_sum(sum);
    for (int e = lane; e < E; e += 32) z[e] = expf(z[e] - m) / sum;
  } else {
    for (int e = lane; e < E; e += 32) z[e] = 1.0f / (1.0f + expf(-z[e]));
  }
  __syncwarp();
  float* gr = gates + (size_t)t * real;
  for (int e = lane; e < real; e += 32) gr[e] = 0.f;
  for (int e = lane; e < E; e += 32) cs[e] = z[e] + (choice_bias ? choice_bias[e] : 0.f);
  __syncwarp();
  if (keep < count) {
    const int size = E / count;
    for (int g = lane; g < count; g += 32) {
      float best = -INFINITY;
      for (int e = g * size; e < (g + 1) * size; ++e) best = fmaxf(best, cs[e]);
      gb[g] = best;
    }
    __syncwarp();
    // a group is out if at least `keep` groups are better (among equals the lower index is)
    for (int g = lane; g < count; g += 32) {
      int better = 0;
      for (int o = 0; o < count; ++o) better += (gb[o] > gb[g] || (gb[o] == gb[g] && o < g)) ? 1 : 0;
      if (better >= keep)
        for (int e = g * size; e < (g + 1) * size; ++e) cs[e] = -INFINITY;
    }
    __syncwarp();
  }
  float total = 0.f, ident = 0.f;
  for (int k = 0; k < top; ++k) {
    int arg = E;
    if (E <= 32) {
      const unsigned mine = lane < E ? moe_order(cs[lane]) : 0u, most = __reduce_max_sync(0xffffffffu, mine);
      if (most > 0x007fffffu) arg = __ffs(__ballot_sync(0xffffffffu, mine == most)) - 1;      // (above minus infinity: something is left)
    } else {
      float best = -INFINITY;
      for (int e = lane; e < E; e += 32) {
        const float v = cs[e];
        if (v > best) {   // (a lane walks upwards, so it keeps its lowest index among equals)
          best = v;
          arg = e;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
        if (ob > best || (ob == best && oa < arg)) {
          best = ob;
          arg = oa;
        }
      }
    }
    if (arg >= E) {       // nothing left to choose
      if (lane == 0) {
        top_idx[(size_t)t * top + k] = -1;
        top_w[(size_t)t * top + k] = 0.f;
      }
      continue;
    }
    const float w = z[arg] * weight_scale;
    if (lane == 0) {
      top_idx[(size_t)t * top + k] = arg;
      top_w[(size_t)t * top + k] = w;
      if (arg < real) gr[arg] = w;
      cs[arg] = -INFINITY;
    }
    if (arg >= real) ident += w;
    total += z[arg];
    __syncwarp();
  }
  if (identity_w && lane == 0) identity_w[t] = (renormalize && total > 0.f) ? ident / total : ident;
  if (score_fn == 2) {
    // softmax over the chosen logits (the first chosen is the largest), summed in the order they were chosen
    __syncwarp();
    const float m = top_w[(size_t)t * top];
    float sum = 0.f;
    for (int k = 0; k < top; ++k) sum += expf(top_w[(size_t)t * top + k] - m);
    __syncwarp();
    for (int k = lane; k < top; k += 32) {
      const float w = expf(top_w[(size_t)t * top + k] - m) / sum;
      top_w[(size_t)t * top + k] = w;
      gr[top_idx[(size_t)t * top + k]] = w;
    }
    return;
  }
  if (renormalize && total > 0.f) {
    __syncwarp();
    for (int e = lane; e < real; e += 32) gr[e] = gr[e] / total;
    for (int k = lane; k < top; k += 32) top_w[(size_t)t * top + k] /= total;
  }
}

template <typename T, int TOK, bool AWARP>
__global__ void __launch_bounds__(TOK == 1 ? 1024 : 512)
moe_router_kernel(const T* __restrict__ x, long x_stride, const float* __restrict__ Wr, const float* __restrict__ bias,
                  float* __restrict__ gates, int* __restrict__ top_idx, float* __restrict__ top_w,
                  float* __restrict__ shared_w, int num_tokens, int hidden, int E, int top, int score_fn,
                  int renormalize, const float* __restrict__ choice_bias, int count, int keep, float weight_scale,
                  float* __restrict__ identity_w, int real, int pitch) {
  extern __shared__ __align__(16) float moe_smem[];      // [TOK]: logits / scores [E + 1], choice scores [E], groups' best
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tok0 = blockIdx.x * TOK, nt = min(TOK, num_tokens - tok0);
  const int zs = 2 * E + 1 + count;
  T* xrow = reinterpret_cast<T*>(moe_smem + (TOK * zs + 3) / 4 * 4);     // the tokens' rows, `pitch` apart
  const int n_rows = E + (shared_w ? 1 : 0), threads = AWARP ? (int)blockDim.x : TOK == 1 ? 1024 : 512, warps = threads / 32;
  const bool vec = (hidden & 3) == 0;
  constexpr int AHEAD = AWARP ? 8 : 0;                    // pieces of the warp's row that are asked for now
  float4 head[AHEAD > 0 ? AHEAD : 1];
  if (AHEAD > 0 && vec && warp < n_rows) {
#pragma unroll
    for (int j = 0; j < AHEAD; ++j)
      if (4 * lane + 128 * j < hidden) head[j] = *reinterpret_cast<const float4*>(Wr + (size_t)warp * hidden + 4 * lane + 128 * j);
  }
  constexpr int VEC = 16 / (int)sizeof(T);
  if ((hidden % VEC) == 0 && (x_stride % VEC) == 0 && ((uintptr_t)x % 16) == 0) {
    const int per = hidden / VEC;
    for (int i = threadIdx.x; i < nt * per; i += threads) {
      const int k = i / per, c = (i - k * per) * VEC;
      *reinterpret_cast<uint4*>(xrow + (size_t)k * pitch + c) =
          *reinterpret_cast<const uint4*>(x + (size_t)(tok0 + k) * x_stride + c);
    }
  } else {
    for (int k = 0; k < nt; ++k)
      for (int i = threadIdx.x; i < hidden; i += threads) xrow[(size_t)k * pitch + i] = x[(size_t)(tok0 + k) * x_stride + i];
  }
  __syncthreads();
  constexpr int PER = TOK < 4 ? TOK : 4;                  // tokens of a warp at a time
  const int units = n_rows * (TOK / PER);
  for (int n = warp; n < units; n += warps) {
    // (blocks start at different outputs: at the same ones they would all ask the same few lines of L2 at a time)
    const int un = TOK == 1 ? n : (n + blockIdx.x * 5) % units, e = un / (TOK / PER), k0 = un % (TOK / PER) * PER;
    const T* xs = xrow + (size_t)k0 * pitch;
    float a[PER][4];
#pragma unroll
    for (int k = 0; k < PER; ++k) a[k][0] = a[k][1] = a[k][2] = a[k][3] = 0.f;
    const float* wrow = Wr + (size_t)e * hidden;
    auto add = [&](int i, const float4& w4) {
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const float4 x4 = moe_load4(xs + (size_t)k * pitch + i);
        a[k][0] = fmaf(w4.x, x4.x, a[k][0]);
        a[k][1] = fmaf(w4.y, x4.y, a[k][1]);
        a[k][2] = fmaf(w4.z, x4.z, a[k][2]);
        a[k][3] = fmaf(w4.w, x4.w, a[k][3]);
      }
    };
    if (vec) {
      int i = 4 * lane;
      if (AHEAD > 0 && n == warp) {
#pragma unroll
        for (int j = 0; j < AHEAD; ++j, i += 128)
          if (i < hidden) add(i, head[j]);
      }
#pragma unroll(TOK == 1 ? 8 : 4)
      for (; i < hidden; i += 128) add(i, *reinterpret_cast<const float4*>(wrow + i));
    } else {
      for (int i = lane; i < hidden; i += 32)
#pragma unroll
        for (int k = 0; k < PER; ++k) a[k][0] = fmaf(wrow[i], to_f32<T>(xs[(size_t)k * pitch + i]), a[k][0]);
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const float v = warp_sum((a[k][0] + a[k][1]) + (a[k][2] + a[k][3]));
      if (lane == 0 && k0 + k < nt) moe_smem[(k0 + k) * zs + e] = v + ((bias && e < E) ? bias[e] : 0.f);
    }
  }
  __syncthreads();
  if (warp >= nt) return;                                // (from here on a warp a token)
  moe_pick(moe_smem + warp * zs, tok0 + warp, gates, top_idx, top_w, shared_w, E, top, score_fn, renormalize, choice_bias, count, keep,
           weight_scale, identity_w, real);
}

// Long portions, bfloat16 rows and at most 32 outputs: 16 tokens a block, on tensor cores.  A row is bfloat16 as it is and the
// router's numbers are three bfloat16 terms that hold all 24 bits, so a product is three of mma.sync, with the leading
// one's steps added with rounded additions (mma_split.cuh); the block's sixteen warps share out k and meet in shared memory.  (The
// multiply-adds of 16 tokens and 17 outputs are 29,000 warp instructions with their conversions, these 11,000.)
#define MOE_TC_TOKENS 16
#define MOE_TC_WARPS 16
#define MOE_TC_STEPS 3              // steps of 16 whose numbers are on their way together
template <int NT>
__global__ void __launch_bounds__(32 * MOE_TC_WARPS)
moe_router_tc_kernel(const bf16* __restrict__ x, long x_stride, const float* __restrict__ Wr, const float* __restrict__ bias,
                     float* __restrict__ gates, int* __restrict__ top_idx, float* __restrict__ top_w, float* __restrict__ shared_w,
                     int num_tokens, int hidden, int E, int top, int score_fn, int renormalize,
                     const float* __restrict__ choice_bias, int count, int keep, float weight_scale, float* __restrict__ identity_w,
                     int real) {
  extern __shared__ __align__(16) float moe_smem[];      // [16]: logits [E + 1], choice scores [E], groups' best; then the warps' sums
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int tok0 = blockIdx.x * MOE_TC_TOKENS, nt = min(MOE_TC_TOKENS, num_tokens - tok0);
  const int zs = 2 * E + 1 + count, n_rows = E + (shared_w ? 1 : 0);
  float* sums = moe_smem + (MOE_TC_TOKENS * zs + 3) / 4 * 4;      // [warps][16][8 NT + 1]
  const int steps = hidden / 16, each = (steps + MOE_TC_WARPS - 1) / MOE_TC_WARPS;
  float acc[NT][4], low[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = low[i][j] = 0.f;
  const bool r0 = g < nt, r1 = g + 8 < nt;
  const bf16* x0 = x + (size_t)(tok0 + (r0 ? g : 0)) * x_stride + 2 * c;
  const bf16* x1 = x + (size_t)(tok0 + (r1 ? g + 8 : 0)) * x_stride + 2 * c;
  const int s1 = min(steps, (warp + 1) * each);
  for (int s0 = warp * each; s0 < s1; s0 += MOE_TC_STEPS) {
    unsigned a[MOE_TC_STEPS][1][4];
    float2 w[MOE_TC_STEPS][NT][2];
#pragma unroll
    for (int j = 0; j < MOE_TC_STEPS; ++j) {
      const int s = s0 + j;
      const bool on = s < s1;
      a[j][0][0] = on && r0 ? *reinterpret_cast<const unsigned*>(x0 + 16 * s) : 0u;
      a[j][0][1] = on && r1 ? *reinterpret_cast<const unsigned*>(x1 + 16 * s) : 0u;
      a[j][0][2] = on && r0 ? *reinterpret_cast<const unsigned*>(x0 + 16 * s + 8) : 0u;
      a[j][0][3] = on && r1 ? *reinterpret_cast<const unsigned*>(x1 + 16 * s + 8) : 0u;
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const float* wr = Wr + (size_t)(8 * i + g) * hidden + 16 * s + 2 * c;
        w[j][i][0] = w[j][i][1] = make_float2(0.f, 0.f);
        if (on && 8 * i + g < n_rows) {
          w[j][i][0] = *reinterpret_cast<const float2*>(wr);
          w[j][i][1] = *reinterpret_cast<const float2*>(wr + 8);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < MOE_TC_STEPS; ++j) {
      unsigned b[NT][3][2];
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) ms_split(w[j][i][h].x, w[j][i][h].y, b[i][0][h], b[i][1][h], b[i][2][h]);
      ms_terms<NT, 1, 3>(acc, low, a[j], b);
    }
  }
  constexpr int SP = 8 * NT + 1;
  float* mine = sums + warp * MOE_TC_TOKENS * SP;
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) mine[(g + 8 * (j >> 1)) * SP + 8 * i + 2 * c + (j & 1)] = acc[i][j] + low[i][j];
  __syncthreads();
  for (int i = threadIdx.x; i < MOE_TC_TOKENS * n_rows; i += 32 * MOE_TC_WARPS) {
    const int k = i / n_rows, e = i - k * n_rows;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < MOE_TC_WARPS; ++w) v += sums[(w * MOE_TC_TOKENS + k) * SP + e];
    if (!(fabsf(v) < INFINITY) && k < nt) {      // (an infinity has no terms: the sum again by multiply-adds)
      v = 0.f;
      for (int j = 0; j < hidden; ++j) v = fmaf(Wr[(size_t)e * hidden + j], __bfloat162float(x[(size_t)(tok0 + k) * x_stride + j]), v);
    }
    moe_smem[k * zs + e] = v + ((bias && e < E) ? bias[e] : 0.f);
  }
  __syncthreads();
  for (int k = warp; k < nt; k += MOE_TC_WARPS)
    moe_pick(moe_smem + k * zs, tok0 + k, gates, top_idx, top_w, shared_w, E, top, score_fn, renormalize, choice_bias, count, keep,
             weight_scale, identity_w, real);
}

// h: T [tokens, shared_ff + E * ff] in place: h = act(h) * weight, weight 1 for the first shared_ff columns,
// gates[t, (col - shared_ff) / ff] for the rest.  A thread takes VEC neighbouring columns of a row (one 16-byte
// access where the row's width allows it).
template <typename T, int VEC>
__global__ void moe_act_kernel(T* __restrict__ h, const float* __restrict__ gates, int num_tokens, int width,
                               int shared_ff, int ff, int E, int act) {
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int per_row = (width + VEC - 1) / VEC;
  const long total = (long)num_tokens * per_row;
  const long step = (long)gridDim.x * blockDim.x;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += step) {
    const int t = (int)(idx / per_row);
    const int c0 = (int)(idx - (long)t * per_row) * VEC;
    T* p = h + (size_t)t * width + c0;
    T v[VEC];
    if (VEC > 1) {
      // the piece lies inside one expert (the launcher checked the widths): if that expert was not chosen for
      // the token, zeros are written and nothing is read
      if (c0 >= shared_ff && gates[(size_t)t * E + (c0 - shared_ff) / ff] == 0.f) {
        *reinterpret_cast<uint4*>(p) = make_uint4(0, 0, 0, 0);
        continue;
      }
      *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(p);
    } else {
      v[0] = p[0];
    }
#pragma unroll
    for (int u = 0; u < VEC; ++u) {
      const int c = c0 + u;
      const float w = c < shared_ff ? 1.f : gates[(size_t)t * E + (c - shared_ff) / ff];
      // an expert that was not chosen contributes an exact zero whatever its first product gave
      v[u] = from_f32<T>(w == 0.f ? 0.f : moe_weighted_activation(to_f32<T>(v[u]), w, act));
    }
    if (VEC > 1) {
      *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(v);
    } else {
      p[0] = v[0];
    }
  }
}

extern "C" int ll_moe_router(int dtype, const void* x, long x_stride, const float* Wr, const float* bias, float* gates,
                             int* top_idx, float* top_w, float* shared_w, int num_tokens, int hidden, int E, int top,
                             int score_fn, int renormalize, const float* choice_bias, int count, int keep,
                             float weight_scale, float* identity_w, int real, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  if (real <= 0 || real > E || (real < E && identity_w == nullptr) || count < 1 || E % count != 0 || keep < 1 || keep > count)
    return (int)cudaErrorInvalidValue;
  if (E <= 0 || E > MOE_MAX_E || top <= 0 || top > E || hidden <= 0) return (int)cudaErrorInvalidValue;
  const int zs = 2 * E + 1 + count, pitch = (hidden + 7) / 8 * 8;
  const int rows = E + (shared_w != nullptr ? 1 : 0);
#define MOE_ROUTER_LAUNCH(TOK, AWARP)                                                                                    \
  do {                                                                                                                   \
    const size_t smem = sizeof(float) * (size_t)((TOK * zs + 3) / 4 * 4) + sizeof(T) * (size_t)TOK * pitch;              \
    if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;                                                            \
    if (smem > 48 * 1024)                                                                                                \
      cudaFuncSetAttribute(moe_router_kernel<T, TOK, AWARP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);    \
    const int warps = TOK > 1 ? 16 : !AWARP ? 32 : rows > 8 ? rows : 8;                                                  \
    ll_launch(moe_router_kernel<T, TOK, AWARP>, dim3((num_tokens + TOK - 1) / TOK), dim3(32 * warps), smem, stream, (const T*)x, x_stride, \
              Wr, bias, gates, top_idx, top_w, shared_w, num_tokens, hidden, E, top, score_fn, renormalize, choice_bias, count, \
              keep, weight_scale, identity_w, real, pitch);                                                              \
  } while (0)
  if (dtype == LL_DTYPE_BF16 && num_tokens >= moe_tc_least(rows) && rows <= 32 && hidden % 16 == 0 && x_stride % 2 == 0 && ((uintptr_t)x % 4) == 0 &&
      ((uintptr_t)Wr % 8) == 0) {
    const int tiles = (rows + 7) / 8;
    const size_t smem = sizeof(float) * ((size_t)(MOE_TC_TOKENS * zs + 3) / 4 * 4 + (size_t)MOE_TC_WARPS * MOE_TC_TOKENS * (8 * tiles + 1));
    const dim3 grid((num_tokens + MOE_TC_TOKENS - 1) / MOE_TC_TOKENS);
#define MOE_ROUTER_TC(NT)                                                                                                       \
  case NT:                                                                                                                      \
    ll_launch(moe_router_tc_kernel<NT>, grid, dim3(32 * MOE_TC_WARPS), smem, stream, (const bf16*)x, x_stride, Wr, bias, gates, top_idx, \
              top_w, shared_w, num_tokens, hidden, E, top, score_fn, renormalize, choice_bias, count, keep, weight_scale, identity_w, \
              real);                                                                                                            \
    break
    switch (tiles) {
      MOE_ROUTER_TC(1);
      MOE_ROUTER_TC(2);
      MOE_ROUTER_TC(3);
      MOE_ROUTER_TC(4);
    }
#undef MOE_ROUTER_TC
    return LL_LAUNCH_RESULT();
  }
  LL_DISPATCH_DTYPE(dtype, {
    if (num_tokens >= 512 && sizeof(float) * 8 * (size_t)zs + sizeof(T) * 8 * (size_t)pitch <= 100 * 1024)
      MOE_ROUTER_LAUNCH(8, false);
    else if (rows <= 24)
      MOE_ROUTER_LAUNCH(1, true);
    else
      MOE_ROUTER_LAUNCH(1, false);
  });
#undef MOE_ROUTER_LAUNCH
  return LL_LAUNCH_RESULT();
}

extern "C" int ll_moe_act(int dtype, void* h, const float* gates, int num_tokens, int shared_ff, int ff, int E, int act,
                          int sms, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  const int width = shared_ff + E * ff;
  if (width <= 0 || (E > 0 && ff <= 0)) return (int)cudaErrorInvalidValue;
  const long most = (long)(sms > 0 ? sms : 148) * 16;
  LL_DISPATCH_DTYPE(dtype, {
    constexpr int VEC = 16 / (int)sizeof(T);
    const bool wide = (width % VEC) == 0 && (shared_ff % VEC) == 0 && (ff % VEC) == 0 && ((uintptr_t)h % 16) == 0;
    const long total = (long)num_tokens * (wide ? width / VEC : width);
    const long want = (total + 255) / 256;
    const int blocks = (int)(want < most ? want : most);
    if (wide)
      ll_launch(moe_act_kernel<T, VEC>, dim3(blocks), dim3(256), 0, stream, (T*)h, gates, num_tokens, width, shared_ff,
                ff, E, act);
    else
      ll_launch(moe_act_kernel<T, 1>, dim3(blocks), dim3(256), 0, stream, (T*)h, gates, num_tokens, width, shared_ff,
                ff, E, act);
  });
  return LL_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------------------------------
// Grouped path (many tokens): the (token, chosen expert) pairs are put in the order of the experts, the rows
// of the chosen tokens are gathered, and two grouped products (one group an expert, the groups' ends known on
// the device only) run over them; only the chosen experts' arithmetic is done.
// ---------------------------------------------------------------------------------------------------------

// One block.  ends [E]: the end of every expert's run of rows; row_token, row_w [pairs + E]: token and routing
// weight of every row; pair_row [pairs]: the row of pair (t, k).  Every expert's run starts with one row that no
// pair points at (token 0, weight 0), so that no run is empty: a grouped product does not have to cope with an
// expert that nobody chose.  Which row inside an expert's run a pair gets is decided by atomics; a row's result
// does not depend on its place.
__global__ void __launch_bounds__(1024)
moe_sort_kernel(const int* __restrict__ top_idx, const float* __restrict__ top_w, int pairs, int top, int E,
                int* __restrict__ ends, int* __restrict__ row_token, float* __restrict__ row_w,
                int* __restrict__ pair_row) {
  __shared__ int count[MOE_MAX_E];
  __shared__ int start[MOE_MAX_E];
  __shared__ int used;
  LL_PDL_WAIT();      // (no early release: what runs next may be a library kernel that does not wait itself)
  for (int e = threadIdx.x; e < E; e += blockDim.x) count[e] = 1;
  __syncthreads();
#pragma unroll 8
  for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
    const int e = top_idx[p];
    if (e >= 0 && e < E) atomicAdd(&count[e], 1);
  }
  __syncthreads();
  if (threadIdx.x < 32) {      // a warp adds the counts up, 32 experts at a time
    int at = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + threadIdx.x, n = e < E ? count[e] : 0;
      int sum = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (threadIdx.x >= o) sum += v;
      }
      if (e < E) {
        const int first = at + sum - n;
        row_token[first] = 0;
        row_w[first] = 0.f;
        start[e] = first + 1;
        ends[e] = at + sum;
      }
      at += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (threadIdx.x == 0) used = at;
  }
  __syncthreads();
  // rows behind the last run (pairs that no expert has: identities): a token that exists, weight 0
  for (int row = used + threadIdx.x; row < pairs + E; row += blockDim.x) {
    row_token[row] = 0;
    row_w[row] = 0.f;
  }
#pragma unroll 8
  for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
    const int e = top_idx[p];
    if (e >= 0 && e < E) {
      const int row = atomicAdd(&start[e], 1);
      row_token[row] = p / top;
      row_w[row] = top_w[p];
      pair_row[p] = row;
    } else {
      pair_row[p] = -1;
    }
  }
}

// dst[row, :] = x[row_token[row], :]
template <typename T>
__global__ void moe_gather_rows_kernel(T* __restrict__ dst, const T* __restrict__ x, long x_stride,
                                       const int* __restrict__ row_token, int hidden) {
  LL_PDL_WAIT();      // (no early release: a library product may run next, which does not wait itself; see grouped_product)
  const int row = blockIdx.x;
  const T* src = x + (size_t)row_token[row] * x_stride;
  T* d = dst + (size_t)row * hidden;
  constexpr int VEC = 16 / (int)sizeof(T);
  if ((hidden % VEC) == 0 && ((uintptr_t)src % 16) == 0 && ((uintptr_t)d % 16) == 0) {
    for (int i = threadIdx.x; i < hidden / VEC; i += blockDim.x)
      reinterpret_cast<uint4*>(d)[i] = reinterpret_cast<const uint4*>(src)[i];
  } else {
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) d[i] = src[i];
  }
}

// VEC neighbouring numbers, one access
template <typename T, int VEC> struct MoePiece {
  alignas(sizeof(T) * VEC) T v[VEC];
  __device__ __forceinline__ void load(const T* p) {
    if constexpr (VEC > 1) *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(p);
    else v[0] = p[0];
  }
  __device__ __forceinline__ void store(T* p) const {
    if constexpr (VEC > 1) *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(v);
    else p[0] = v[0];
  }
};

// h[row, :] = act(h[row, :]) * row_w[row], in place; VEC neighbouring numbers of a row a thread
template <typename T, int VEC>
__global__ void moe_row_act_kernel(T* __restrict__ h, const float* __restrict__ row_w, long total_vec, int ff, int act) {
  LL_PDL_WAIT();      // (no early release: what runs next may be a library kernel that does not wait itself)
  const long step = (long)gridDim.x * blockDim.x;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total_vec; idx += step) {
    const float w = row_w[(idx * VEC) / ff];
    T v[VEC];
    if (VEC > 1) *reinterpret_cast<uint4*>(v) = reinterpret_cast<const uint4*>(h)[idx];
    else v[0] = h[idx];
#pragma unroll
    for (int u = 0; u < VEC; ++u) v[u] = from_f32<T>(moe_weighted_activation(to_f32<T>(v[u]), w, act));
    if (VEC > 1) reinterpret_cast<uint4*>(h)[idx] = *reinterpret_cast<const uint4*>(v);
    else h[idx] = v[0];
  }
}

// out[t, :] = base[t, :] + sum over k (in the order of k) of y[pair_row[t, k], :]; float32 sums, one rounding.
// A thread takes VEC neighbouring columns of one token (16-byte accesses where the width allows it), four rows' loads on
// their way at once: bound by memory.
template <typename T, int VEC>
__global__ void moe_combine_kernel(T* __restrict__ out, const T* __restrict__ base, const T* __restrict__ y,
                                   const int* __restrict__ pair_row, int top, int hidden) {
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int t = blockIdx.x;
  const int* rows = pair_row + (size_t)t * top;
  for (int c = threadIdx.x * VEC; c < hidden; c += blockDim.x * VEC) {
    float a[VEC];
#pragma unroll
    for (int u = 0; u < VEC; ++u) a[u] = 0.f;
    for (int k0 = 0; k0 < top; k0 += 4) {
      MoePiece<T, VEC> v[4];
      bool on[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = k0 + i < top ? rows[k0 + i] : -1;
        on[i] = row >= 0;
        if (on[i]) v[i].load(y + (size_t)row * hidden + c);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (on[i]) {
#pragma unroll
          for (int u = 0; u < VEC; ++u) a[u] += to_f32<T>(v[i].v[u]);
        }
    }
    MoePiece<T, VEC> o;
    if (base) {
      o.load(base + (size_t)t * hidden + c);
#pragma unroll
      for (int u = 0; u < VEC; ++u) a[u] += to_f32<T>(o.v[u]);
    }
#pragma unroll
    for (int u = 0; u < VEC; ++u) o.v[u] = from_f32<T>(a[u]);
    o.store(out + (size_t)t * hidden + c);
  }
}

extern "C" int ll_moe_sort(const int* top_idx, const float* top_w, int num_tokens, int top, int E, int* ends,
                           int* row_token, float* row_w, int* pair_row, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  if (E <= 0 || E > MOE_MAX_E || top <= 0) return (int)cudaErrorInvalidValue;
  ll_launch(moe_sort_kernel, dim3(1), dim3(1024), 0, stream, top_idx, top_w, num_tokens * top, top, E, ends, row_token,
            row_w, pair_row);
  return LL_LAUNCH_RESULT();
}

extern "C" int ll_moe_gather_rows(int dtype, void* dst, const void* x, long x_stride, const int* row_token, int rows,
                                  int hidden, cudaStream_t stream) {
  if (rows <= 0) return 0;
  LL_DISPATCH_DTYPE(dtype, ll_launch(moe_gather_rows_kernel<T>, dim3(rows), dim3(128), 0, stream, (T*)dst, (const T*)x,
                                     x_stride, row_token, hidden));
  return LL_LAUNCH_RESULT();
}

extern "C" int ll_moe_row_act(int dtype, void* h, const float* row_w, int rows, int ff, int act, int sms,
                              cudaStream_t stream) {
  if (rows <= 0) return 0;
  const long most = (long)(sms > 0 ? sms : 148) * 16;
  LL_DISPATCH_DTYPE(dtype, {
    constexpr int VEC = 16 / (int)sizeof(T);
    const bool wide = (ff % VEC) == 0 && ((uintptr_t)h % 16) == 0;
    const long total = (long)rows * ff / (wide ? VEC : 1);
    const long want = (total + 255) / 256;
    const int blocks = (int)(want < most ? want : most);
    if (wide) ll_launch(moe_row_act_kernel<T, VEC>, dim3(blocks), dim3(256), 0, stream, (T*)h, row_w, total, ff, act);
    else ll_launch(moe_row_act_kernel<T, 1>, dim3(blocks), dim3(256), 0, stream, (T*)h, row_w, total, ff, act);
  });
  return LL_LAUNCH_RESULT();
}

extern "C" int ll_moe_combine(int dtype, void* out, const void* base, const void* y, const int* pair_row,
                              int num_tokens, int top, int hidden, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  LL_DISPATCH_DTYPE(dtype, {
    constexpr int VEC = 16 / (int)sizeof(T);
    const bool wide = (hidden % VEC) == 0 && ((uintptr_t)out % 16) == 0 && ((uintptr_t)base % 16) == 0 && ((uintptr_t)y % 16) == 0;
    const int threads = wide && hidden < 256 * VEC ? (hidden / VEC + 31) / 32 * 32 : 256;
    if (wide)
      ll_launch(moe_combine_kernel<T, VEC>, dim3(num_tokens), dim3(threads), 0, stream, (T*)out, (const T*)base, (const T*)y,
                pair_row, top, hidden);
    else
      ll_launch(moe_combine_kernel<T, 1>, dim3(num_tokens), dim3(256), 0, stream, (T*)out, (const T*)base, (const T*)y,
                pair_row, top, hidden);
  });
  return LL_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------------------------------
// Experts with a gate: an expert is down(a * sigmoid(alpha a) * (c + 1)) with a = min(gate x, limit) and
// c = clamp(up x, -limit, limit), or (a limit of 0) down(silu(gate x) * (up x)).  The first product's rows are, expert by expert, the gate rows then the up
// rows (an always-on expert's first).
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float moe_gate(float g, float u, float limit, float alpha) {
  return limit > 0.f ? ll_clamped_swish(g, u, limit, alpha) : g / (1.0f + expf(-g)) * u;
}

// in: T [tokens, 2 * (shared_ff + E * ff)]; out: T [tokens, shared_ff + E * ff] = activation times the
// expert's weight for the token: gates[t, e] for expert e (zero: not chosen, zeros are written and nothing is
// read), shared_w[t] (null: 1) for the always-on expert, which has a limit of its own.
// A thread takes VEC neighbouring units (one 16-byte access where the widths allow it: they lie inside one expert then).
template <typename T, int VEC>
__global__ void moe_gated_act_kernel(T* __restrict__ out, const T* __restrict__ in, const float* __restrict__ gates,
                                     const float* __restrict__ shared_w, int num_tokens, int shared_ff, int ff, int E,
                                     float limit, float shared_limit, float alpha) {
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int width = shared_ff + E * ff;
  const int per_row = width / VEC;
  const long total = (long)num_tokens * per_row;
  const long step = (long)gridDim.x * blockDim.x;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += step) {
    const int t = (int)(idx / per_row);
    const int c = (int)(idx - (long)t * per_row) * VEC;
    const T* row = in + (size_t)t * 2 * width;
    T* dst = out + (size_t)t * width + c;
    float w, lim;
    const T *gp, *up;
    T g[VEC], u[VEC], y[VEC];
    if (c < shared_ff) {
      w = shared_w ? shared_w[t] : 1.f;
      gp = row + c;
      up = gp + shared_ff;
      lim = shared_limit;
    } else {
      const int e = (c - shared_ff) / ff;
      w = gates[(size_t)t * E + e];
      gp = row + 2 * shared_ff + (size_t)e * 2 * ff + (c - shared_ff - e * ff);
      up = gp + ff;
      lim = limit;
      if (w == 0.f) {      // an expert that was not chosen contributes an exact zero whatever its first product gave
        if (VEC > 1) *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
        else dst[0] = from_f32<T>(0.f);
        continue;
      }
    }
    if (VEC > 1) {
      *reinterpret_cast<uint4*>(g) = *reinterpret_cast<const uint4*>(gp);
      *reinterpret_cast<uint4*>(u) = *reinterpret_cast<const uint4*>(up);
    } else {
      g[0] = gp[0];
      u[0] = up[0];
    }
#pragma unroll
    for (int k = 0; k < VEC; ++k) y[k] = from_f32<T>(moe_gate(to_f32<T>(g[k]), to_f32<T>(u[k]), lim, alpha) * w);
    if (VEC > 1) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(y);
    else dst[0] = y[0];
  }
}

// in: T [rows, 2 * ff] (gate columns, then up columns); out: T [rows, ff] = activation times row_w[row].
// A thread takes VEC neighbouring units of a row (16-byte accesses where the width allows it).
template <typename T, int VEC>
__global__ void moe_row_gated_act_kernel(T* __restrict__ out, const T* __restrict__ in, const float* __restrict__ row_w,
                                         long total_vec, int ff, float limit, float alpha) {
  LL_PDL_WAIT();      // (no early release: what runs next may be a library kernel that does not wait itself)
  const long step = (long)gridDim.x * blockDim.x;
  const int per_row = ff / VEC;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total_vec; idx += step) {
    // (a 64-bit division is a subroutine)
    const long r = total_vec <= 0xffffffffl ? (long)((unsigned)idx / (unsigned)per_row) : idx / per_row;
    const int j = (int)(idx - r * per_row) * VEC;
    const float w = row_w ? row_w[r] : 1.f;
    const T* p = in + (size_t)r * 2 * ff + j;
    T g[VEC], u[VEC], y[VEC];
    if (VEC > 1) {
      *reinterpret_cast<uint4*>(g) = *reinterpret_cast<const uint4*>(p);
      *reinterpret_cast<uint4*>(u) = *reinterpret_cast<const uint4*>(p + ff);
    } else {
      g[0] = p[0];
      u[0] = p[ff];
    }
#pragma unroll
    for (int k = 0; k < VEC; ++k)
      y[k] = from_f32<T>(moe_gate(to_f32<T>(g[k]), to_f32<T>(u[k]), limit, alpha) * w);
    if (VEC > 1) *reinterpret_cast<uint4*>(out + (size_t)r * ff + j) = *reinterpret_cast<const uint4*>(y);
    else out[(size_t)r * ff + j] = y[0];
  }
}

extern "C" int ll_moe_gated_act(int dtype, void* out, const void* in, const float* gates, const float* shared_w,
                                int num_tokens, int shared_ff, int ff, int E, float limit, float shared_limit,
                                float alpha, int sms, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  const long width = shared_ff + (long)E * ff;
  if (width <= 0 || (E > 0 && ff <= 0)) return (int)cudaErrorInvalidValue;
  const long most = (long)(sms > 0 ? sms : 148) * 16;
  LL_DISPATCH_DTYPE(dtype, {
    constexpr int VEC = 16 / (int)sizeof(T);
    const bool wide = shared_ff % VEC == 0 && ff % VEC == 0 && ((uintptr_t)in % 16) == 0 && ((uintptr_t)out % 16) == 0;
    const long want = (num_tokens * width / (wide ? VEC : 1) + 255) / 256;
    const dim3 grid((int)(want < most ? want : most));
    if (wide)
      ll_launch(moe_gated_act_kernel<T, VEC>, grid, dim3(256), 0, stream, (T*)out, (const T*)in, gates, shared_w,
                num_tokens, shared_ff, ff, E, limit, shared_limit, alpha);
    else
      ll_launch(moe_gated_act_kernel<T, 1>, grid, dim3(256), 0, stream, (T*)out, (const T*)in, gates, shared_w,
                num_tokens, shared_ff, ff, E, limit, shared_limit, alpha);
  });
  return LL_LAUNCH_RESULT();
}

extern "C" int ll_moe_row_gated_act(int dtype, void* out, const void* in, const float* row_w, int rows, int ff,
                                    float limit, float alpha, int sms, cudaStream_t stream) {
  if (rows <= 0) return 0;
  const long most = (long)(sms > 0 ? sms : 148) * 16;
  LL_DISPATCH_DTYPE(dtype, {
    constexpr int VEC = 16 / (int)sizeof(T);
    const bool wide = (ff % VEC) == 0 && ((uintptr_t)in % 16) == 0 && ((uintptr_t)out % 16) == 0;
    const long total = (long)rows * ff / (wide ? VEC : 1);
    const long want = (total + 255) / 256;
    const int blocks = (int)(want < most ? want : most);
    if (wide)
      ll_launch(moe_row_gated_act_kernel<T, VEC>, dim3(blocks), dim3(256), 0, stream, (T*)out, (const T*)in, row_w,
                total, ff, limit, alpha);
    else
      ll_launch(moe_row_gated_act_kernel<T, 1>, dim3(blocks), dim3(256), 0, stream, (T*)out, (const T*)in, row_w, total,
                ff, limit, alpha);
  });
  return LL_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------------------------------------
// Experts of one or two tokens: only the matrices of experts that one of the tokens has chosen (and the one for every token) are
// read.  The products over all experts' stacked matrices read every one of them: for a token of four out of sixteen experts 3.4 times
// the bytes.  A warp makes a hidden unit (moe_few_up: a row of the first matrix, or a gate row and an up row), or a part of an output
// (moe_few_down: a row of the second matrix at the chosen experts' columns), 16 bytes a lane and load, float32 sums.  Which experts:
// every CTA looks through the gates.  Hidden units of experts that were not chosen are neither made nor read; those of
// a token for an expert that only another one has chosen are zeros, and the second product leaves them out.  Bound by the weights and,
// from two tokens on, by the multiply-adds on the CUDA cores.  Whole parts, all experts' products / this way, us: one token 1.5B sizes
// 59 / 32, 3B 88 / 40, 7B 191 / 85, gated 60 / 31, 86 / 38, 196 / 82; two tokens gated 60 / 50, 87 / 63, 196 / 132.  (With the pieces of
// all chosen experts in one row, shared out by their place in it: 34, 41, 88, 32, 39, 85; 54, 67, 142; a token's order of sums then
// depended on the other one's experts.)  That way two tokens without a gate took 59 / 65, 89 / 81, 191 / 175, which stay with the
// other kernels, as do three (60 / 80).  Loads for the second product that are asked for on a condition, one after the other: 38, 48, 113.
// ---------------------------------------------------------------------------------------------------------------
#define MOE_FEW_THREADS 256
#define MOE_FEW_EXPERTS 256
struct MoeFew {
  const float* gates;        // [M][E]
  const float* shared_w;     // [M] or null: 1
  int shared_ff, ff, E;
};
// the chosen experts in order, by all threads; behind it all of them may read `list`, and (several tokens) `takers`: who chose it, a bit
// a token
template <int M>
__device__ __forceinline__ int moe_few_list(const MoeFew& p, unsigned char* list, unsigned char* takers, int* count) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    int n = 0;
    for (int e0 = 0; e0 < p.E; e0 += 32) {
      unsigned who = 0;
      if (e0 + lane < p.E) {
#pragma unroll
        for (int t = 0; t < M; ++t) who |= (p.gates[(size_t)t * p.E + e0 + lane] != 0.f ? 1u : 0u) << t;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, who != 0);
      if (who != 0) {
        const int at = n + __popc(hit & ((1u << lane) - 1));
        list[at] = (unsigned char)(e0 + lane);
        if (M > 1) takers[at] = (unsigned char)who;
      }
      n += __popc(hit);
    }
    if (lane == 0) *count = n;
  }
  __syncthreads();
  return *count;
}
__device__ __forceinline__ void moe_few_eight(const uint4& v, float (&x)[8]) {
  const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[2 * i] = __uint_as_float(w[i] << 16);
    x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

template <int M, bool GATED>
__global__ void __launch_bounds__(MOE_FEW_THREADS)
moe_few_up_kernel(bf16* __restrict__ out, const bf16* __restrict__ x, long x_stride, const bf16* __restrict__ w, int K, MoeFew p, int act,
                  float limit, float shared_limit, float alpha) {
  constexpr int R = GATED ? 2 : 1, DEPTH = 4;
  extern __shared__ __align__(16) unsigned char mf_smem[];
  uint4* xs = reinterpret_cast<uint4*>(mf_smem);                 // [M][K / 8]
  __shared__ unsigned char list[MOE_FEW_EXPERTS], takers[M > 1 ? MOE_FEW_EXPERTS : 1];
  __shared__ int count;
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int lane = threadIdx.x & 31, pieces = K / 8, width = p.shared_ff + p.E * p.ff;
  for (int i = threadIdx.x; i < M * pieces; i += MOE_FEW_THREADS)
    xs[i] = reinterpret_cast<const uint4*>(x + (size_t)(i / pieces) * x_stride)[i % pieces];
  const int units = p.shared_ff + moe_few_list<M>(p, list, takers, &count) * p.ff;
  for (int r = blockIdx.x * (MOE_FEW_THREADS / 32) + (threadIdx.x >> 5); r < units; r += gridDim.x * (MOE_FEW_THREADS / 32)) {
    const bool own = r >= p.shared_ff;
    const int slot = own ? (r - p.shared_ff) / p.ff : 0, f = own ? r - p.shared_ff - slot * p.ff : r, e = own ? list[slot] : 0;
    const int col = own ? p.shared_ff + e * p.ff + f : f, apart = own ? p.ff : p.shared_ff;
    const size_t first = GATED ? (own ? 2 * (size_t)p.shared_ff + (size_t)e * 2 * p.ff + f : f) : col;
    const uint4* row = reinterpret_cast<const uint4*>(w + first * K);
    const uint4* row2 = row + (size_t)(GATED ? apart : 0) * pieces;
    float acc[R][M] = {};
    for (int c0 = lane; c0 < pieces; c0 += 32 * DEPTH) {
      uint4 v[R][DEPTH];
#pragma unroll
      for (int d = 0; d < DEPTH; ++d) {
        const int c = c0 + 32 * d;
        v[0][d] = c < pieces ? __ldcs(row + c) : make_uint4(0, 0, 0, 0);
        if (GATED) v[R - 1][d] = c < pieces ? __ldcs(row2 + c) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int d = 0; d < DEPTH; ++d) {
        const int c = min(c0 + 32 * d, pieces - 1);
        float a[R][8];
#pragma unroll
        for (int q = 0; q < R; ++q) moe_few_eight(v[q][d], a[q]);
#pragma unroll
        for (int t = 0; t < M; ++t) {
          float b[8];
          moe_few_eight(xs[t * pieces + c], b);
          if (c0 + 32 * d >= pieces) continue;
#pragma unroll
          for (int q = 0; q < R; ++q)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[q][t] = fmaf(a[q][i], b[i], acc[q][t]);
        }
      }
    }
#pragma unroll
    for (int t = 0; t < M; ++t) {
#pragma unroll
        for (int q = 0; q < R; ++q) acc[q][t] = warp_sum(acc[q][t]);
      if (lane == t) {
        const float weight = own ? p.gates[(size_t)t * p.E + e] : p.shared_w != nullptr ? p.shared_w[t] : 1.f;
        const float z = to_f32<bf16>(from_f32<bf16>(acc[0][t]));
        float y;
        if (GATED) y = moe_gate(z, to_f32<bf16>(from_f32<bf16>(acc[R - 1][t])), own ? limit : shared_limit, alpha) * weight;
        else y = moe_weighted_activation(z, weight, act);
        out[(size_t)t * width + col] = from_f32<bf16>(own && weight == 0.f ? 0.f : y);
      }
    }
  }
}

// out [M][N] float32; w [N][shared_ff + E ff]; a row of w by four warps: block b of 32 pieces of expert e's columns goes to warp
// (b + e + 1) mod 4 (the columns for every token: b mod 4), whose lanes add up in the order of the experts.  So the order of a token's sum
// depends on its own experts alone, not on what the other token has chosen.
template <int M>
__global__ void __launch_bounds__(MOE_FEW_THREADS)
moe_few_down_kernel(float* __restrict__ out, const bf16* __restrict__ h, const bf16* __restrict__ w, int N, MoeFew p) {
  constexpr int PARTS = 4, DEPTH = M == 1 ? 4 : 3, ROWS = MOE_FEW_THREADS / 32 / PARTS;
  __shared__ unsigned char list[MOE_FEW_EXPERTS], takers[M > 1 ? MOE_FEW_EXPERTS : 1];
  __shared__ int count;
  __shared__ float sums[MOE_FEW_THREADS / 32][M];
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = warp % PARTS;
  const int width = p.shared_ff + p.E * p.ff, f8 = p.ff / 8, s8 = p.shared_ff / 8;
  const int live = moe_few_list<M>(p, list, takers, &count);
  for (int n0 = blockIdx.x * ROWS; n0 < N; n0 += gridDim.x * ROWS) {
    const int n = n0 + warp / PARTS;
    float acc[M] = {};
    if (n < N) {
      const uint4* row = reinterpret_cast<const uint4*>(w + (size_t)n * width);
      const uint4* rows = reinterpret_cast<const uint4*>(h);
      int run = -1, c = 32 * part + lane, len = s8, first = 0;      // the columns for every token, then the chosen experts'
      int next = list[0];
      unsigned who = (1u << M) - 1;
      while (run < live) {
        uint4 v[DEPTH], b[DEPTH][M];
        unsigned take[DEPTH];
#pragma unroll
        for (int d = 0; d < DEPTH; ++d) {
          if (c - lane >= len) {                                    // (the same for all lanes; an expert may have no block for the warp)
            ++run;
            c = 32 * ((part - next - 1) & (PARTS - 1)) + lane;
            len = f8;
            first = s8 + next * f8;
            if (M > 1) who = takers[run & (MOE_FEW_EXPERTS - 1)];
            next = list[(run + 1) & (MOE_FEW_EXPERTS - 1)];
          }
          const bool there = run < live && c < len;
          const int at = there ? first + c : 0;                     // (behind the end: some piece that is not used)
          take[d] = there ? who : 0;
          v[d] = __ldcs(row + at);
#pragma unroll
          for (int t = 0; t < M; ++t) b[d][t] = rows[(size_t)t * (width / 8) + at];
          c += 32 * PARTS;
        }
#pragma unroll
        for (int d = 0; d < DEPTH; ++d) {
          float a[8];
          moe_few_eight(v[d], a);
#pragma unroll
          for (int t = 0; t < M; ++t) {
            if (((take[d] >> t) & 1) == 0) continue;
            float z[8];
            moe_few_eight(b[d][t], z);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[t] = fmaf(a[i], z[i], acc[t]);
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < M; ++t) {
      acc[t] = warp_sum(acc[t]);
      if (lane == 0) sums[warp][t] = acc[t];
    }
    __syncthreads();
    if (threadIdx.x < ROWS * M) {
      const int q = threadIdx.x / M, t = threadIdx.x % M;
      if (n0 + q < N) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < PARTS; ++i) s += sums[q * PARTS + i][t];
        out[(size_t)t * N + n0 + q] = s;
      }
    }
    __syncthreads();
  }
}

// out float32 [M][N] = the experts' outputs for one row of x, or two with gated experts, bfloat16; hidden: bfloat16 [M][shared_ff + E ff], scratch.
// gated: limits and alpha as in ll_moe_gated_act, else act as in ll_gemm_stream_experts.  K, ff, shared_ff: multiples of 8; rows of x
// and matrices at multiples of 16 bytes; E at most 256.
extern "C" int ll_moe_few(float* out, void* hidden, const void* x, long x_stride, const void* w_up, const void* w_down, int M, int K, int N,
                          const float* gates, const float* shared_w, int shared_ff, int ff, int E, int gated, int act, float limit,
                          float shared_limit, float alpha, int sms, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (M > (gated ? 2 : 1) || K <= 0 || K % 8 || ff <= 0 || ff % 8 || shared_ff < 0 || shared_ff % 8 || E <= 0 || E > MOE_FEW_EXPERTS || x_stride % 8 ||
      (long)M * K * 2 > 49152 || ((uintptr_t)x | (uintptr_t)w_up | (uintptr_t)w_down | (uintptr_t)hidden) % 16)
    return (int)cudaErrorInvalidValue;
  const MoeFew p{gates, shared_w, shared_ff, ff, E};
  const size_t smem = (size_t)M * K * 2;
  const dim3 grid(4 * sms);
  const size_t own = 48 * 1024 - 1024;      // (the kernel has up to 528 bytes beside the rows: more than 48 KB together has to be asked for)
#define MOE_FEW(MM, GATED)                                                                                                         \
  if (M == MM && (gated != 0) == GATED) {                                                                                          \
    const cudaError_t rc = smem <= own ? cudaSuccess : cudaFuncSetAttribute(moe_few_up_kernel<MM, GATED>,                          \
                                                                            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (rc != cudaSuccess) return (int)rc;                                                                                         \
    ll_launch(moe_few_up_kernel<MM, GATED>, grid, dim3(MOE_FEW_THREADS), smem, stream, (bf16*)hidden, (const bf16*)x, x_stride,      \
              (const bf16*)w_up, K, p, act, limit, shared_limit, alpha);                                                            \
    ll_launch(moe_few_down_kernel<MM>, grid, dim3(MOE_FEW_THREADS), 0, stream, out, (const bf16*)hidden, (const bf16*)w_down, N, p); \
  }
  MOE_FEW(1, false)
  MOE_FEW(1, true)
  MOE_FEW(2, true)
#undef MOE_FEW
  return LL_LAUNCH_RESULT();
}
