// Products of routed experts over many tokens on the fifth-generation tensor cores, two SMs a tile: every group of rows (the
// rows that chose an expert, ends on the device only; and, first, all tokens for an expert that everybody uses) times its
// own weights, with the experts' activation and the rows' weights in the epilogue.
//
//   up    hidden[row] = act(gate, up)(x W_e^T) * weight[row]      gated: gate and up rows of the expert, the products never leave
//         or act(x W_e^T) * weight[row]                            the chip (the library's product wrote 59 MB for a second kernel)
//   down  y[row] = hidden[row] W_e^T
//
// The weights' rows are the M side here (256 a pair of CTAs, cta_group::2), a group's rows the N side: N is any multiple of
// 32, so a group of 550 rows costs three tiles of 192 rows and not three of 256 (a token row as a lane of tensor memory
// would make the last tile of every group full width: 25 % more arithmetic for 16 experts and 8,192 rows).  A group's
// rows are cut into equal tiles of at most 256.  Gated: each CTA's 128 lanes are 64 gate features and the 64 up features
// beside them.
//
// Roles, barriers, ring and bounded waits as in gemm_pair.cu: warp 0 brings two boxes a stage (TMA, no multicast: 128 rows of
// weights, 128 or 64 token rows, x 64 k; a TMA instruction takes its thread about 130 clocks, so four boxes a stage were
// slower than the MMAs), warp 1 of the even CTA issues the MMAs into one of two accumulators of 256 columns,
// eight warps read the other.  A lane is a feature, rows are written as features side by side, so the accumulator is turned in
// shared memory: 128 rows at a time as bfloat16 [row][lane] (the product rounded as the unfused path stored it), from where
// consecutive threads take 16 bytes of gate and of up, and store 16 bytes.  The activations are those of the kernels that follow a
// product alone (moe_gate, moe_weighted_activation), to the bit: 2 % of a whole part of 2,048 tokens (204 and 208 us) against the
// exponential and reciprocal instructions alone, whose exponent is off by 2^-20 at gates of 20.
//
// Every CTA counts the groups' tiles itself and the pairs take them round-robin, a group's rows fastest (its weights are
// read once from memory, its rows stay in L2).
// Measured on a B200, 2,048 tokens, 4 of 16 experts of 1,536 -> 1,792 and one for all, gated: up with its activation 91 us (1.24
// PFLOP/s of what is asked for; library products and two activation kernels 126), down 49 (58).  Bound by the loads: with 64
// rows a group a stage still takes 620 clocks (5 stages of 32 KB, weights from memory), with 512 rows 578, its MMAs 512.
// Needs K % 8 == 0 and features % 8 == 0, 16-byte aligned rows.
#include "moe_act.cuh"
#include "tc05_pair.cuh"

#define GG_THREADS 320
#define GG_STAGES 5
#define GG_BOX (64 * 128)                   // 64 rows x 64 k
#define GG_STAGE_BYTES (4 * GG_BOX)         // two boxes of weights, two of rows
#define GG_STG_BYTES (128 * 256)
#define GG_MAX_GROUPS 257
#define GG_SMEM (1024 + GG_STAGES * GG_STAGE_BYTES + GG_STG_BYTES + (2 * GG_STAGES + 4) * 8 + 16 + (2 * GG_MAX_GROUPS + 2) * 4)

struct GgGroup {          // what differs between the expert that everybody uses and the routed ones
  bf16* out;              // [rows, N]
  int N, K;               // features (gated: units, W has N gate and N up rows), inner size
  const float* row_w;     // a weight a row, or null
  float limit;            // gated: the activation's
};
struct GgParams {
  GgGroup s, r;           // everybody's (n_shared rows; none: no such group) and the routed ones
  int n_shared, E;
  GateAct gate;           // gated: the activation, but for its limit
  const int* ends;        // int32 [E]: where every expert's run of rows ends
  int act;                // without a gate: -1 none, else an activation of moe_act.cuh
  int* status;
};

// 128 rows of the weights [group][sub: gate, up][row][k]: 64 of gate and 64 of up, or 128
__device__ __forceinline__ void gg_load_w(unsigned dst, const CUtensorMap* map, int k, int row, int group, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
      "l"(map), "r"(k), "r"(row), "r"(0), "r"(group), "r"(bar)
      : "memory");
}

// A tile: `n` rows (N of the MMA: `nw`) from `row` on, the `ft`-th tile of features of group `grp` (-1: everybody's)
struct GgTile {
  int grp, row, n, nw, ft;
};
struct GgTiles {
  const int *cum, *first;      // tiles before a group, rows before a routed group [groups + 1]
  int shared, n_shared, g;
  // the t-th tile (called with growing t)
  __device__ __forceinline__ GgTile at(int t) {
    while (t >= cum[g + 1]) ++g;
    const int r0 = g < shared ? 0 : first[g], rows = g < shared ? n_shared : first[g + 1] - r0;
    const int T = (rows + 255) / 256, width = ((rows + T - 1) / T + 31) / 32 * 32;
    const int local = t - cum[g];
    GgTile o;
    o.ft = local / T;
    const int m = local - o.ft * T;
    o.row = r0 + m * width;
    o.n = min(width, rows - m * width);
    o.nw = (o.n + 31) / 32 * 32;
    o.grp = g - shared;
    return o;
  }
};

template <bool GATED>
__global__ void __launch_bounds__(GG_THREADS)
gemm_group_kernel(const GgParams p, const __grid_constant__ CUtensorMap w_shared, const __grid_constant__ CUtensorMap x_shared,
                  const __grid_constant__ CUtensorMap w_routed, const __grid_constant__ CUtensorMap x_routed,
                  const __grid_constant__ CUtensorMap x_routed64) {
  constexpr int FT = GATED ? 128 : 256;      // features a tile
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* stg = smem + GG_STAGES * GG_STAGE_BYTES;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(stg + GG_STG_BYTES);
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 2 * GG_STAGES + 4);
  int* cum = reinterpret_cast<int*>(tmem_slot + 2);
  int* first = cum + GG_MAX_GROUPS + 1;
  const unsigned stage0 = gp_smem(smem);
  const unsigned full0 = gp_smem(bars), empty0 = gp_smem(bars + GG_STAGES);
  const unsigned acc_full0 = gp_smem(bars + 2 * GG_STAGES), acc_empty0 = gp_smem(bars + 2 * GG_STAGES + 2);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const unsigned rank = gp_cluster_rank();   // 0: issues the MMAs and owns the `full` and `acc_empty` barriers
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  if (tid == 32) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&w_routed) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&x_routed) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&x_routed64) : "memory");
    if (p.n_shared > 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&w_shared) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&x_shared) : "memory");
    }
  }
  if (tid == 0) {
    for (int s = 0; s < GG_STAGES; ++s) {
      gp_mbar_init(full0 + 8 * s, 1);    // the even CTA's producer announces both CTAs' bytes
      gp_mbar_init(empty0 + 8 * s, 1);   // one commit
    }
    for (int b = 0; b < 2; ++b) {
      gp_mbar_init(acc_full0 + 8 * b, 1);    // one commit
      gp_mbar_init(acc_empty0 + 8 * b, 16);  // the eight epilogue warps of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // all of this SM's tensor memory: two accumulators of 256 columns; both CTAs take part
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gp_smem(tmem_slot)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  gp_cluster_sync();   // both CTAs' barriers are initialised and both allocations are known
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_slot;
  const bool paired = gp_ld_cluster(gp_mapa(gp_smem(tmem_slot), rank ^ 1u)) == tmem;
  if (!paired && tid == 0) set_status(p.status, LL_ERR_TMEM_PAIR);
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();

  // ---- the groups' tiles, counted by one warp ----
  const int shared = p.n_shared > 0 ? 1 : 0, groups = shared + p.E;
  if (warp == 0) {
    int before = 0;
    if (lane == 0) cum[0] = 0;
    for (int g0 = 0; g0 < groups; g0 += 32) {
      const int g = g0 + lane, e = g - shared;
      int r0 = 0, r1 = 0;
      if (g < groups && e >= 0) {
        r0 = e > 0 ? p.ends[e - 1] : 0;
        r1 = p.ends[e];
      } else if (g < groups) {
        r1 = p.n_shared;
      }
      const int N = e >= 0 ? p.r.N : p.s.N;
      const int n = r1 > r0 ? (r1 - r0 + 255) / 256 * ((N + FT - 1) / FT) : 0;
      int sum = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      if (g < groups) {
        cum[g + 1] = before + sum;
        if (e >= 0) first[g] = r0;
        if (g == groups - 1) first[groups] = r1;
      }
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
  }
  __syncthreads();
  const int tiles = cum[groups];
  GgTiles walk = {cum, first, shared, p.n_shared, 0};

  bool dead = false;
  if (paired) {
    if (warp == 0) {
      // ------------------------------ producer ------------------------------
      {
        int s = 0;
        const unsigned lead_full = gp_mapa(full0, 0);
        unsigned ph = 1;      // (a fresh barrier counts as passed in this phase)
        for (int t = pair; t < tiles; t += pairs) {
          const GgTile o = walk.at(t);
          const CUtensorMap* wm = o.grp < 0 ? &w_shared : &w_routed;
          const int more = o.nw > 128 ? 1 : 0;      // (a box has 64 or 128 of the CTA's half of the rows)
          const CUtensorMap* xm = o.grp < 0 ? &x_shared : more ? &x_routed : &x_routed64;
          const int grp = o.grp < 0 ? 0 : o.grp, half = o.nw / 2;
          const int kboxes = ((o.grp < 0 ? p.s.K : p.r.K) + 63) / 64;
          const int x_row = o.row + (int)rank * half;
          const int w_row = o.ft * FT + (int)rank * (FT / 2);
          const unsigned bytes = 2u * (3 + (more | (o.grp < 0 ? 1 : 0))) * GG_BOX;
          for (int k = 0; k < 64 * kboxes; k += 64) {
            gp_mbar_wait(empty0 + 8 * s, ph, p.status, dead);
            if (gp_elect()) {
              if (rank == 0) gp_mbar_expect_tx(full0 + 8 * s, bytes);
              const unsigned bar = lead_full + 8 * s, at = stage0 + s * GG_STAGE_BYTES;
              gg_load_w(at, wm, k, w_row, grp, bar);
              gp_tma_load(at + 2 * GG_BOX, xm, k, x_row, bar);
            }
            __syncwarp();
            if (++s == GG_STAGES) {
              s = 0;
              ph ^= 1;
            }
          }
        }
      }
    } else if (warp == 1) {
      // ------------------------------ MMA issue (even CTA) ------------------------------
      if (rank == 0) {
        const unsigned long long desc0 = gp_desc(stage0);
        int tl = 0, s = 0;
        unsigned ph = 0;
        for (int t = pair; t < tiles; t += pairs, ++tl) {
          const GgTile o = walk.at(t);
          // instruction descriptor: float32 accumulate, bfloat16 A and B, both K-major, M = 256 (the pair's)
          const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(o.nw >> 3) << 17) | ((256u >> 4) << 24);
          const int b = tl & 1, kboxes = ((o.grp < 0 ? p.s.K : p.r.K) + 63) / 64;
          // both CTAs' epilogues of the tile before last must have read this accumulator
          gp_mbar_wait(acc_empty0 + 8 * b, (unsigned)(((tl >> 1) & 1) ^ 1), p.status, dead);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned acc = tmem + (unsigned)(b * 256);
          for (int kc = 0; kc < kboxes; ++kc) {
            gp_mbar_wait(full0 + 8 * s, ph, p.status, dead);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned long long a_desc = desc0 + (unsigned)(s * (GG_STAGE_BYTES >> 4)), b_desc = a_desc + (2 * GG_BOX >> 4);
            if (gp_elect()) {
#pragma unroll
              for (int k16 = 0; k16 < 4; ++k16)      // (16 of k are 32 bytes further)
                gp_mma(acc, a_desc + 2 * k16, b_desc + 2 * k16, idesc, (kc > 0 || k16 > 0) ? 1u : 0u);
              gp_commit_pair(empty0 + 8 * s);   // the stage is free in both CTAs once these MMAs have read it
            }
            __syncwarp();
            if (++s == GG_STAGES) {
              s = 0;
              ph ^= 1;
            }
          }
          if (gp_elect()) gp_commit_pair(acc_full0 + 8 * b);  // the tile's accumulator is complete once all its MMAs are done
        }
      }
    } else {
      // ------------------------------ epilogue (warps 2..9) ------------------------------
      const int ew = warp & 3;          // the 32 tensor-memory lanes this warp may read: 32 ew .. 32 ew + 31
      const int eh = (warp - 2) >> 2;   // which half of every 128 columns it takes
      const int e = tid - 64;
      const unsigned acc_empty_lead = gp_mapa(acc_empty0, 0);
      int tl = 0;
      for (int t = pair; t < tiles; t += pairs, ++tl) {
        const GgTile o = walk.at(t);
        const bool all = o.grp < 0;
        bf16* g_out = all ? p.s.out : p.r.out;
        const float* g_w = all ? p.s.row_w : p.r.row_w;
        const int g_N = all ? p.s.N : p.r.N;
        const GateAct gate = {p.gate.act, all ? p.s.limit : p.r.limit, p.gate.alpha};
        const int b = tl & 1;
        constexpr int PIECES = GATED ? 8 : 16, STEP = 256 / PIECES, MINE = 128 / STEP;      // 16 bytes of features; a thread's rows
        const int piece = e & (PIECES - 1), j0 = e / PIECES, f = o.ft * FT + (int)rank * (FT / 2) + 8 * piece;
        const bool weigh = GATED || p.act >= 0;
        // the weight of the thread's r-th row of the tile, asked for a row ahead (the first one while the MMAs run)
        auto ask = [&](int r) {
          const int j = r / MINE * 128 + j0 + (r % MINE) * STEP;
          return weigh && g_w != nullptr && j < o.n ? g_w[o.row + j] : 1.f;
        };
        float w_next = ask(0);
        gp_mbar_wait(acc_full0 + 8 * b, (unsigned)((tl >> 1) & 1), p.status, dead);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned taddr = tmem + ((unsigned)(32 * ew) << 16) + (unsigned)(b * 256);
#pragma unroll 1
        for (int c0 = 0; c0 < o.nw; c0 += 128) {
          {
            unsigned v0[32], v1[32];
            const int c = c0 + 64 * eh;
            if (c < o.nw) gp_ld32_issue(taddr + c, v0);
            if (c + 32 < o.nw) gp_ld32_issue(taddr + c + 32, v1);
            gp_ld_wait2(v0, v1);
            bf16* d = reinterpret_cast<bf16*>(stg) + (size_t)(64 * eh) * 128 + 32 * ew + lane;
            if (c < o.nw) {
#pragma unroll
              for (int i = 0; i < 32; ++i) d[128 * i] = __float2bfloat16_rn(__uint_as_float(v0[i]));
            }
            if (c + 32 < o.nw) {
#pragma unroll
              for (int i = 0; i < 32; ++i) d[128 * (32 + i)] = __float2bfloat16_rn(__uint_as_float(v1[i]));
            }
          }
          if (c0 + 128 >= o.nw) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) gp_mbar_arrive_cluster(acc_empty_lead + 8 * b);
          }
          asm volatile("bar.sync 1, 256;" ::: "memory");   // 128 rows are staged
          if (f < g_N && !weigh) {
#pragma unroll
            for (int i = 0; i < MINE; ++i) {
              const int j = j0 + i * STEP;
              if (c0 + j < o.n)
                *reinterpret_cast<uint4*>(g_out + (size_t)(o.row + c0 + j) * g_N + f) =
                    *reinterpret_cast<const uint4*>(stg + j * 256 + 16 * piece);
            }
          } else if (f < g_N) {
#pragma unroll 1
            for (int i = 0; i < MINE; ++i) {      // (eight or sixteen copies of the activations' code left the instruction cache)
              const int j = j0 + i * STEP;
              const float w = w_next;
              w_next = ask(c0 / 128 * MINE + i + 1);
              if (c0 + j >= o.n) break;
              const unsigned char* src = stg + j * 256 + 16 * piece;
              float z[8];
              gp_unpack8(*reinterpret_cast<const uint4*>(src), z);
              if (GATED) {
                float u[8];
                gp_unpack8(*reinterpret_cast<const uint4*>(src + 128), u);
                if (gate.act == 2) ll_gated_divided<2, 8>(z, u, gate);
                else ll_gated_divided<0, 8>(z, u, gate);
#pragma unroll
                for (int k = 0; k < 8; ++k) z[k] *= w;
              } else {
                const float ws[8] = {w, w, w, w, w, w, w, w};
                moe_weighted_act_any<8>(z, ws, p.act);
              }
              *reinterpret_cast<uint4*>(g_out + (size_t)(o.row + c0 + j) * g_N + f) = gp_pack8(z);
            }
          }
          asm volatile("bar.sync 1, 256;" ::: "memory");   // they may be overwritten
        }
      }
    }
  }
  // ---- everyone is done, in both CTAs (nobody's shared or tensor memory is still in use): free ----
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  gp_cluster_sync();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// Weights of `groups` groups, [subs][rows][K] each: strides in elements; boxes of 128 rows x 64 k (64 of each of two subs).
static int gg_weights_map(CUtensorMap* map, const void* base, int K, int rows, int subs, int groups, long row_stride,
                          long sub_stride, long group_stride) {
  gp_encode_fn enc = gp_encoder();
  if (enc == nullptr) return (int)cudaErrorNotSupported;
  const cuuint64_t dims[4] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)subs, (cuuint64_t)groups};
  const cuuint64_t strides[3] = {(cuuint64_t)row_stride * 2, (cuuint64_t)sub_stride * 2, (cuuint64_t)group_stride * 2};
  const cuuint32_t box[4] = {64, (cuuint32_t)(128 / subs), (cuuint32_t)subs, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}
static int gg_rows_map(CUtensorMap* map, const void* base, long rows, int K, long stride, int box_rows) {
  gp_encode_fn enc = gp_encoder();
  if (enc == nullptr) return (int)cudaErrorNotSupported;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)stride * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

template <bool GATED>
static int gg_launch(const GgParams& p, const CUtensorMap& ws, const CUtensorMap& xs, const CUtensorMap& wr, const CUtensorMap& xr,
                     const CUtensorMap& xr64, int pairs, cudaStream_t stream) {
  cudaFuncSetAttribute(gemm_group_kernel<GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GG_SMEM);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(GG_THREADS);
  cfg.dynamicSmemBytes = GG_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = ll_pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaLaunchKernelEx(&cfg, gemm_group_kernel<GATED>, p, ws, xs, wr, xr, xr64);
  return LL_LAUNCH_RESULT();
}

// Routed rows x [rows, K_e] (contiguous) with `ends`, weights w of E groups: gated [E][2][N_e][K_e] contiguous, else rows N_e of
// row stride w_row, group stride w_group.  n_shared > 0: also all rows of xs [n_shared, K_s] (row stride xs_stride) times ws
// (gated: gate rows, then up rows, contiguous; else row stride ws_row).  gated: 0 no, 1 SiLU, 3 clamped swish (limits, alpha);
// act: -1 none, or an activation of moe_act.cuh (+ 16: the weight goes inside).  out / out_s: bfloat16 [rows, N] contiguous.
extern "C" int ll_gemm_group(void* out, const void* x, const void* w, int rows, int N_e, int K_e, long w_row, long w_group, int E,
                             const int* ends, const float* row_w, void* out_s, const void* xs, long xs_stride, const void* ws,
                             int n_shared, int N_s, int K_s, long ws_row, const float* row_w_s, int gated, float limit,
                             float limit_s, float alpha, int act, int sm_count, int* status, cudaStream_t stream) {
  if (rows <= 0 || E <= 0 || E >= GG_MAX_GROUPS || N_e <= 0 || K_e <= 0 || (N_e % 8) != 0 || (K_e % 8) != 0 || sm_count < 2 ||
      (w_row % 8) != 0 || (w_group % 8) != 0 || (uintptr_t)out % 16 != 0 || (uintptr_t)x % 16 != 0 || (uintptr_t)w % 16 != 0 ||
      ends == nullptr || (gated != 0 && gated != 1 && gated != 3))
    return (int)cudaErrorInvalidValue;
  if (n_shared > 0 && (N_s <= 0 || K_s <= 0 || (N_s % 8) != 0 || (K_s % 8) != 0 || (ws_row % 8) != 0 || (xs_stride % 8) != 0 ||
                       (uintptr_t)out_s % 16 != 0 || (uintptr_t)xs % 16 != 0 || (uintptr_t)ws % 16 != 0))
    return (int)cudaErrorInvalidValue;
  GgParams p;
  p.r = {reinterpret_cast<bf16*>(out), N_e, K_e, row_w, limit};
  p.s = {reinterpret_cast<bf16*>(out_s), N_s, K_s, row_w_s, limit_s};
  p.gate = {gated > 0 ? gated - 1 : 0, 0.f, alpha};
  p.n_shared = n_shared > 0 ? n_shared : 0;
  p.E = E;
  p.ends = ends;
  p.act = gated ? -1 : act;
  p.status = status;
  CUtensorMap wmap, xmap, xmap64, wmap_s = {}, xmap_s = {};
  int rc = gg_weights_map(&wmap, w, K_e, N_e, gated ? 2 : 1, E, w_row, gated ? (long)N_e * K_e : w_row, w_group);
  if (rc == 0) rc = gg_rows_map(&xmap, x, rows, K_e, K_e, 128);
  if (rc == 0) rc = gg_rows_map(&xmap64, x, rows, K_e, K_e, 64);
  if (rc == 0 && n_shared > 0) rc = gg_weights_map(&wmap_s, ws, K_s, N_s, gated ? 2 : 1, 1, ws_row, gated ? (long)N_s * K_s : ws_row, ws_row);
  if (rc == 0 && n_shared > 0) rc = gg_rows_map(&xmap_s, xs, n_shared, K_s, xs_stride, 128);
  if (rc != 0) return rc;
  const int ft = gated ? 128 : 256;
  const long most_tiles = ((rows + 255l) / 256 + E) * ((N_e + ft - 1) / ft) + (n_shared > 0 ? (n_shared + 255l) / 256 * ((N_s + ft - 1) / ft) : 0);
  const int pairs = most_tiles < sm_count / 2 ? (int)most_tiles : sm_count / 2;
  return gated ? gg_launch<true>(p, wmap_s, xmap_s, wmap, xmap, xmap64, pairs, stream)
               : gg_launch<false>(p, wmap_s, xmap_s, wmap, xmap, xmap64, pairs, stream);
}
