// Latent attention of single tokens and short portions on tensor cores (bfloat16, mma.sync m16n8k16).
//
// The same work as `latent_attention_kernel` (latent_attention.cu): per (token, group of heads, part of the keys) an
// online softmax over the request's cached rows [R latent | r rotated] with the latent-space queries, returning
// sum_j p_j c_j a head.  All heads read the same rows, so the heads are the M side of the products: a CTA takes up to 16
// heads and tiles of 64 keys,
//   S [16 heads x 64 keys]  = Q [16 x KD] K^T     a warp has 8 keys; the queries stay in its registers
//   O [16 heads x R]       += P [16 x 64] C        a warp has R / 8 columns, P from shared memory
// with KD = R + r.  What bounds a tile is the chain of a CTA's own instructions (96 mma.sync a warp at 8 clocks each, two warps a
// scheduler, are 1,500 clocks), so everything else is taken off the eight warps: others bring the rows through a ring of
// stages, the exponentials are made once, by the warp whose keys they belong to, and a tile costs two barriers of all and one
// of a pair of warps.  Rows come as TMA boxes, a page's rows a box of [KD / BW][rows][BW] (BW: 64 columns, or 32 or 16 where KD is
// no multiple), swizzled so that the 8 x 16-byte ldmatrix reads meet different banks; a row a bulk copy comes at 16.6 bytes
// a clock and SM, cp.async at 37, boxes of 16 KB at 88 (measured alone).  Pages that are no multiple of 8 rows come by cp.async
// into the same places.  Rows of positions that are not visible are zeroed (a tile's garbage times a weight of 0 may be NaN).
// The softmax weights enter the second product as two bfloat16 terms (hi + lo, sixteen bits of mantissa), accumulated in
// float32.  Tiles start at multiples of 64 positions.
//
// A token's keys are shared out over a thread-block cluster: its own number of tiles, over as many CTAs as the host says
// (steps are captured for a class of contexts, so the host does not know the lengths), each an equal run of them.  The CTAs
// meet in distributed shared memory: each adds up its share of the columns in the order of the parts.  (Through memory
// and a second kernel: 16 parts of 16 tokens and 12 heads are 6 MB out and in again.)
// Measured on a B200 (12 heads, a latent of 512; before, with tiles of 32 keys by cp.async, P in shared memory and parts through
// memory / now, us): 16 tokens behind 2,048 25.4 / 17.0, 64 tokens 65.9 / 37.1 (134 MB: 3.6 TB/s), one token 21.0 / 13.6, 16
// tokens of 28 heads behind 4,096 65 / 34.7, one token behind 8,000 48 / 19.7.  A tile of 64 keys is 3,100 clocks: S 950, the
// maxima and P 500, the second product 1,250; to the first tile 3,000, the parts' meeting 5,000 (6 CTAs).
// Taken for: bfloat16, KD a multiple of 16 and at most 1,024, R a multiple of 32 and at most 512.
#include <atomic>

#include "tc05.cuh"

#define LM_TK 64
#define LM_WARPS 8                // that compute
#define LM_LOADERS 4              // warps that bring the rows (TMA: the first of them)
#define LM_THREADS (32 * (LM_WARPS + LM_LOADERS))
#define LM_HEADS 16
#define LM_UNITS 4                // units of 16 columns a warp, at most (UPW: 1 to 4; the eight warps have 128 UPW columns, at least R)
#define LM_PPITCH (2 * LM_TK + 16)      // bytes from one head's row of P to the next
#define LM_MAX_STAGES 3
#define LM_MAX_SMEM (218 * 1024)  // dynamic shared memory of any launch
#define LM_LOG2E 1.4426950408889634f

__device__ __forceinline__ void lm_mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                       unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void lm_ldmatrix_x4(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3, unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void lm_ldmatrix_x4_trans(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3, unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ unsigned lm_pack(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<unsigned*>(&v);
}

__device__ __forceinline__ void lm_cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of this CTA's shared-memory location `addr` in CTA `rank` of the cluster, a store and a load there
__device__ __forceinline__ unsigned lm_mapa(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void lm_st_cluster2(unsigned addr, float x, float y) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1,%2};" ::"r"(addr), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ float2 lm_ld_cluster2(unsigned addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void lm_cp_async16(unsigned dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}

// q: [tokens, H, KD]; cache: one plane [pages, 1, page_size, KD]; out: [tokens, H, R].  `first`: the launch's first
// token.  gridDim = (tokens, ceil(H / 16), parts), a cluster the parts of a (token, group of heads).  STEPS: steps of 16 of KD
// a warp takes, half of KD's, whose queries are kept in registers (0: any number, queries from shared memory).  bw: columns a
// block of a tile; box_rows: rows a box (64 without TMA); `map`: the plane as [KD / bw][rows][bw].  FULL: 128 UPW = R, so that
// every warp has UPW units, without a look at R.
template <int STEPS, int UPW, bool FULL, bool TMA>
__global__ void __launch_bounds__(LM_THREADS, 1)
latent_attention_mma_kernel(bf16* __restrict__ out, const bf16* __restrict__ q, const bf16* __restrict__ cache,
                            const int* __restrict__ block_table, int bt_stride, const int* __restrict__ token_req,
                            const int* __restrict__ req_slot, const int* __restrict__ positions, int first, int H, int R,
                            int r, int page_size, int num_pages, int window, float scale_log2, int* status, int stages,
                            int bw, int box_rows, const float* __restrict__ sink, const __grid_constant__ CUtensorMap map) {
  extern __shared__ unsigned char lm_raw[];
  unsigned char* lm_smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(lm_raw) + 1023) & ~uintptr_t(1023));
  __shared__ unsigned long long bars[2 * LM_MAX_STAGES];
  __shared__ float4 xchg[LM_WARPS * 32];             // halves of scores, between the two warps of 16 keys
  __shared__ __align__(16) float wmax[LM_HEADS * LM_WARPS];      // [16 rows][8 warps]
  __shared__ __align__(8) float2 ml[16 * LM_HEADS];  // the rows' maxima and sums in every part
  __shared__ float wts[16 * LM_HEADS];               // what a part's sums are multiplied by, 1 / the sum of all folded in
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned full0 = at_smem(bars), empty0 = at_smem(bars + LM_MAX_STAGES);
  if (tid == 0) {
    for (int s = 0; s < stages; ++s) {
      at_mbar_init(full0 + 8 * s, TMA ? 1 : 32 * LM_LOADERS);
      at_mbar_init(empty0 + 8 * s, LM_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  LL_PDL_TRIGGER();
  // (the step's index arrays were there before the step's first kernel)
  const int t = first + blockIdx.x;
  const int entry = token_req[t];
  const int p = positions[t];
  const int slot = entry >= 0 ? req_slot[entry] : -1;
  const int h0 = blockIdx.y * LM_HEADS;
  const int hc = min(LM_HEADS, H - h0);
  const int g = lane >> 2, c = lane & 3;
  const int KD = R + r;
  const int pitch = 2 * KD + 16;                    // bytes from one row of the queries to the next
  const int tile_bytes = 2 * LM_TK * KD, blk = 2 * box_rows * bw, box = 2 * box_rows * KD;
  unsigned char* qs = lm_smem + (size_t)stages * tile_bytes;
  const unsigned k_base = at_smem(lm_smem), q_base = at_smem(qs);
  const unsigned ph_base = q_base + LM_HEADS * pitch, pl_base = ph_base + LM_HEADS * LM_PPITCH;      // P hi, P lo

  const int nsplit = gridDim.z, split = blockIdx.z;
  const int lo = (window > 0) ? max(0, p - window + 1) : 0;
  // this CTA's tiles: an equal run of the token's
  int tile_begin = lo / LM_TK, tiles = p / LM_TK - tile_begin + 1;
  {
    const int each = (tiles + nsplit - 1) / nsplit;
    tile_begin += split * each;
    tiles = max(0, min(each, tiles - split * each));
  }
  const int* bt = block_table + (size_t)(slot < 0 ? 0 : slot) * bt_stride;
  const int boxes = LM_TK / box_rows;
  int page = -2;              // TMA: a lane's page in the tile that comes next (-2: nothing to bring)
  auto look_box = [&](int tile) {
    const int pos = tile * LM_TK + lane * box_rows;
    page = (lane < boxes && pos + box_rows > lo && pos <= p) ? bt[pos / page_size] : -2;
    if (page != -2 && (page < 0 || page >= num_pages)) {
      set_status(status, LL_ERR_PAGE_RANGE);
      page = -2;
    }
  };
  if (TMA && warp == LM_WARPS) {
    if (lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(&map) : "memory");
    if (slot >= 0 && p >= 0 && tiles > 0) look_box(tile_begin);
  }
  __syncthreads();
  LL_PDL_WAIT();
  bf16* orow = out + ((size_t)t * H + h0) * R;
  if (slot < 0 || p < 0) {     // a padding entry (the whole cluster's): defined output, nothing read
    for (int i = split * LM_THREADS + tid; i < hc * R; i += nsplit * LM_THREADS) orow[i] = __float2bfloat16_rn(0.f);
    return;
  }
  // The parts' meeting below writes into the other CTAs' shared memory, which needs them to have started: everyone says so
  // here and waits for it there, behind the tiles (a CTA whose share is no tile at all gets there at once).
  if (nsplit > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  bool dead = false;
  const int units = R / 16, u0 = warp * UPW;      // (fewer than UPW units for the last warps unless FULL)
  float o_acc[2 * UPW][4];
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};   // rows g and g + 8 (l: this thread's share)

  // where a row of a tile begins, and what its 16-byte pieces' numbers within a block are XORed with
  auto row_at = [&](int row) { return (unsigned)((row / box_rows) * box + (row % box_rows) * 2 * bw); };
  auto row_x = [&](int row) { return bw == 64 ? row & 7 : bw == 32 ? (row >> 1) & 3 : (row >> 2) & 1; };
  if (warp >= LM_WARPS) {
    if (TMA) {
      // ---- a lane a box: boxes without a visible row are left out; a lane looks its page up a tile ahead ----
      if (warp == LM_WARPS) {
        for (int n = 0; n < tiles; ++n) {
          const int s = n % stages, pos = (tile_begin + n) * LM_TK + lane * box_rows;
          const int y = page == -2 ? -1 : page * page_size + pos % page_size;
          if (n + 1 < tiles) look_box(tile_begin + n + 1);
          if (n >= stages) {
            at_mbar_wait(empty0 + 8 * s, (unsigned)((n / stages - 1) & 1), status, dead);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the consumers' loads, then the copies
          }
          const unsigned live = __ballot_sync(0xffffffffu, y >= 0);
          if (lane == 0) at_mbar_expect_tx(full0 + 8 * s, __popc(live) * box);
          __syncwarp();
          if (y >= 0) at_tma_3d(k_base + s * tile_bytes + lane * box, &map, 0, y, 0, full0 + 8 * s);
        }
      }
    } else {
      // ---- a warp has every fourth row, 32 pieces a copy; lane l looks up the page of the warp's l-th row ----
      const int w = warp - LM_WARPS, vpr = KD / 8, cpb = bw / 8;
      long row = -1;                     // number of the row in the plane; -1: not visible
      auto look = [&](int tile) {
        const int pos = tile * LM_TK + w + LM_LOADERS * lane;
        row = -1;
        if (lane < LM_TK / LM_LOADERS && pos >= lo && pos <= p) {
          const int page = bt[pos / page_size];
          if (page < 0 || page >= num_pages) set_status(status, LL_ERR_PAGE_RANGE);
          else row = (long)page * page_size + pos % page_size;
        }
      };
      if (tiles > 0) look(tile_begin);
      for (int n = 0; n < tiles; ++n) {
        const int s = n % stages;
        const long mine = row;
        if (n + 1 < tiles) look(tile_begin + n + 1);
        if (n >= stages) at_mbar_wait(empty0 + 8 * s, (unsigned)((n / stages - 1) & 1), status, dead);
        __syncwarp();
        for (int j = 0; j < LM_TK / LM_LOADERS; ++j) {
          const int at = w + LM_LOADERS * j;
          const long from = __shfl_sync(0xffffffffu, mine, j);
          const unsigned dst = k_base + s * tile_bytes + row_at(at);
          for (int piece = lane; piece < vpr; piece += 32)
            lm_cp_async16(dst + (piece / cpb) * blk + (((piece % cpb) ^ row_x(at)) << 4), cache + (from < 0 ? 0 : from * KD + 8 * piece),
                          from < 0 ? 0 : 16);
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full0 + 8 * s) : "memory");
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else {
    // ---- the queries of the CTA's heads, as the first product's A operand (rows of heads that do not exist are zeros) ----
    for (int i = tid; i < LM_HEADS * (KD / 8); i += 32 * LM_WARPS) {
      const int row = i / (KD / 8), piece = i - row * (KD / 8);
      uint4 v = make_uint4(0, 0, 0, 0);
      if (row < hc) v = *reinterpret_cast<const uint4*>(q + ((size_t)t * H + h0 + row) * KD + 8 * piece);
      *reinterpret_cast<uint4*>(qs + (size_t)row * pitch + 16 * piece) = v;
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    // (lane l names row l % 8 of matrix l / 8: heads + 8 for the odd ones, channels + 8 for the last two)
    // (the pair's warps take the steps in turn: step 2 s + kh of KD's is step s of warp kh)
    const int kg = warp >> 1, kh = warp & 1;
    const unsigned qa = q_base + ((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + (lane >> 4) * 16 + 32 * kh;
    unsigned qf[STEPS > 0 ? STEPS : 1][4];
    if (STEPS > 0) {
#pragma unroll
      for (int s = 0; s < STEPS; ++s) lm_ldmatrix_x4(qf[s][0], qf[s][1], qf[s][2], qf[s][3], qa + 64 * s);
    }
#pragma unroll
    for (int i = 0; i < 2 * UPW; ++i) o_acc[i][0] = o_acc[i][1] = o_acc[i][2] = o_acc[i][3] = 0.f;

    const int srow = 16 * kg + (lane & 7) + (lane >> 4) * 8, shalf = (lane >> 3) & 1, sx = row_x(srow);
    const unsigned srow_at = row_at(srow);
    constexpr bool WIDE = STEPS % 2 == 0;              // blocks of 64 columns (four steps), else of 32
    const unsigned off0 = ((2 * kh + shalf) ^ sx) << 4, off1 = ((4 + 2 * kh + shalf) ^ sx) << 4;
    unsigned voff[UPW], vrow_at[LM_TK / 16];
#pragma unroll
    for (int u = 0; u < UPW; ++u) {
      const int piece = 2 * (u0 + u);
      voff[u] = (piece / (bw / 8)) * blk + (((piece % (bw / 8) + (lane >> 4)) ^ row_x(lane & 15)) << 4);
    }
#pragma unroll
    for (int ks = 0; ks < LM_TK / 16; ++ks) vrow_at[ks] = row_at(16 * ks + (lane & 15));

    for (int n = 0; n < tiles; ++n) {
      const int s_at = n % stages, tile0 = (tile_begin + n) * LM_TK;
      at_mbar_wait(full0 + 8 * s_at, (unsigned)((n / stages) & 1), status, dead);
      __syncwarp();
      const unsigned kt = k_base + s_at * tile_bytes;
      // ---- S of 16 keys over half of the channels; the pair of warps then has 8 of the keys each ----
      float sc[2][2][4];      // [8 keys][chain]
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) sc[i >> 1][i & 1][x] = 0.f;
      if (STEPS > 0) {
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
          unsigned b[4];
          lm_ldmatrix_x4(b[0], b[1], b[2], b[3], kt + srow_at + (WIDE ? (s >> 1) * blk + ((s & 1) ? off1 : off0) : s * blk + off0));
          lm_mma(sc[0][s & 1], qf[s][0], qf[s][1], qf[s][2], qf[s][3], b[0], b[1]);
          lm_mma(sc[1][s & 1], qf[s][0], qf[s][1], qf[s][2], qf[s][3], b[2], b[3]);
        }
      } else {
        for (int s = kh; s < KD / 16; s += 2) {
          unsigned a[4], b[4];
          lm_ldmatrix_x4(a[0], a[1], a[2], a[3], qa + 32 * (s - kh));
          lm_ldmatrix_x4(b[0], b[1], b[2], b[3], kt + srow_at + (2 * s / (bw / 8)) * blk + (((2 * s % (bw / 8) + shalf) ^ sx) << 4));
          lm_mma(sc[0][0], a[0], a[1], a[2], a[3], b[0], b[1]);
          lm_mma(sc[1][0], a[0], a[1], a[2], a[3], b[2], b[3]);
        }
      }
      if (TMA && (tile0 < lo || tile0 + LM_TK - 1 > p)) {      // a tile at an end: rows that are not visible become zeros
        for (int i = 0; i < 8; ++i) {
          const int row = 8 * warp + i, pos = tile0 + row;
          if (pos < lo || pos > p)
            for (int b = lane; b < KD / 8; b += 32)
              *reinterpret_cast<uint4*>(lm_smem + (size_t)s_at * tile_bytes + row_at(row) + (b / (bw / 8)) * blk + 16 * (b % (bw / 8))) =
                  make_uint4(0, 0, 0, 0);
        }
        // (read by the other warps behind the barriers below; the next box into this place comes after these writes)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      float v[4];
      {
        float lo8[4], hi8[4];      // scores of keys 0 .. 7 and 8 .. 15 over this warp's channels; the odd warp keeps the latter
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          lo8[x] = sc[0][0][x] + sc[0][1][x];
          hi8[x] = sc[1][0][x] + sc[1][1][x];
        }
        xchg[warp * 32 + lane] = kh ? make_float4(lo8[0], lo8[1], lo8[2], lo8[3]) : make_float4(hi8[0], hi8[1], hi8[2], hi8[3]);
        asm volatile("bar.sync %0, 64;" ::"r"(2 + kg) : "memory");
        const float4 other = xchg[(warp ^ 1) * 32 + lane];
        v[0] = (kh ? hi8[0] : lo8[0]) + other.x;
        v[1] = (kh ? hi8[1] : lo8[1]) + other.y;
        v[2] = (kh ? hi8[2] : lo8[2]) + other.z;
        v[3] = (kh ? hi8[3] : lo8[3]) + other.w;
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int pos = tile0 + 8 * warp + 2 * c + (x & 1);
        v[x] = (pos >= lo && pos <= p) ? v[x] * scale_log2 : -INFINITY;
      }
      // ---- the rows' maxima over the tile: a quad holds a row's 8 keys of this warp; the warps meet in shared memory
      float mx[2] = {fmaxf(v[0], v[1]), fmaxf(v[2], v[3])};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
      }
      if (c == 0) {
        wmax[g * LM_WARPS + warp] = mx[0];
        wmax[(g + 8) * LM_WARPS + warp] = mx[1];
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");      // (every warp has left the tile before: P may be overwritten)
      float alpha[2], msafe[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(wmax + (g + 8 * i) * LM_WARPS);
        const float4 b = *reinterpret_cast<const float4*>(wmax + (g + 8 * i) * LM_WARPS + 4);
        const float mt = at_max3(fmaxf(a.x, a.y), fmaxf(a.z, a.w), at_max3(fmaxf(b.x, b.y), b.z, b.w));
        const float m_new = fmaxf(m_run[i], mt);
        msafe[i] = (m_new == -INFINITY) ? 0.f : m_new;
        alpha[i] = at_ex2(m_run[i] - msafe[i]);
        m_run[i] = m_new;
      }
      // P into shared memory in two bfloat16 terms: hi, and what hi lost
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float a = at_ex2(v[2 * i] - msafe[i]), b = at_ex2(v[2 * i + 1] - msafe[i]);
        l_run[i] = l_run[i] * alpha[i] + (a + b);
        const __nv_bfloat162 hi = __floats2bfloat162_rn(a, b);
        unsigned char* dst = qs + LM_HEADS * (size_t)pitch + (g + 8 * i) * LM_PPITCH + 2 * (8 * warp + 2 * c);
        *reinterpret_cast<unsigned*>(dst) = *reinterpret_cast<const unsigned*>(&hi);
        *reinterpret_cast<unsigned*>(dst + LM_HEADS * LM_PPITCH) = lm_pack(a - __low2float(hi), b - __high2float(hi));
      }
      if (alpha[0] != 1.f || alpha[1] != 1.f) {
#pragma unroll
        for (int i = 0; i < 2 * UPW; ++i) {
          o_acc[i][0] *= alpha[0];
          o_acc[i][1] *= alpha[0];
          o_acc[i][2] *= alpha[1];
          o_acc[i][3] *= alpha[1];
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
      // ---- O = O alpha + P C over the warp's columns ----
      unsigned held = 0;
#pragma unroll
      for (int ks = 0; ks < LM_TK / 16; ++ks) {
        const unsigned pa0 = ((lane & 7) + ((lane >> 3) & 1) * 8) * LM_PPITCH + (lane >> 4) * 16 + 32 * ks;
        unsigned hi[4], lw[4];
        lm_ldmatrix_x4(hi[0], hi[1], hi[2], hi[3], ph_base + pa0);
        lm_ldmatrix_x4(lw[0], lw[1], lw[2], lw[3], pl_base + pa0);
        const unsigned vrow = kt + vrow_at[ks];
#pragma unroll
        for (int u = 0; u < UPW; ++u) {
          if (FULL || u0 + u < units) {
            unsigned b0, b1, b2, b3;
            lm_ldmatrix_x4_trans(b0, b1, b2, b3, vrow + voff[u]);
            if (ks == LM_TK / 16 - 1) held = b0;
            lm_mma(o_acc[2 * u], hi[0], hi[1], hi[2], hi[3], b0, b1);
            lm_mma(o_acc[2 * u + 1], hi[0], hi[1], hi[2], hi[3], b2, b3);
            lm_mma(o_acc[2 * u], lw[0], lw[1], lw[2], lw[3], b0, b1);
            lm_mma(o_acc[2 * u + 1], lw[0], lw[1], lw[2], lw[3], b2, b3);
          }
        }
      }
      // The place goes back when its values are here (an arrival behind loads may overtake them, and so may the next copy): the
      // producer's proxy fence stands between the arrivals and its next copy, and the arrival's address takes (no) part of the last
      // load, behind which a warp's earlier ones have come (seen, not promised; of every load: 43.2 -> 48.0 us for a decode step of 16)
      __syncwarp();
      if (lane == 0) at_mbar_arrive(empty0 + 8 * s_at + (held & (unsigned)(num_pages >> 31)));
    }
    // ---- the rows' sums: over the quad, then over the warps (wmax holds them now) ----
    asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 1);
      l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 2);
      if (c == 0) wmax[(g + 8 * i) * LM_WARPS + warp] = l_run[i];
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float4 a = *reinterpret_cast<const float4*>(wmax + (g + 8 * i) * LM_WARPS);
      const float4 b = *reinterpret_cast<const float4*>(wmax + (g + 8 * i) * LM_WARPS + 4);
      l_run[i] = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
    }
    if (nsplit == 1) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int row = g + 8 * i;
        if (row < hc) {
          // the key without a value: one more term of the sum
          const float l = sink ? l_run[i] + at_ex2(sink[h0 + row] * LM_LOG2E - m_run[i]) : l_run[i];
          const float inv = l > 0.f ? 1.0f / l : 0.f;
#pragma unroll
          for (int u = 0; u < 2 * UPW; ++u)
            if (u0 + u / 2 < units)
              *reinterpret_cast<__nv_bfloat162*>(orow + (size_t)row * R + 16 * u0 + 8 * u + 2 * c) =
                  __floats2bfloat162_rn(o_acc[u][2 * i] * inv, o_acc[u][2 * i + 1] * inv);
        }
      }
    }
  }
  if (nsplit == 1) return;
  // ---- the parts meet: the sums as they are into this CTA's shared memory (over the tiles, which everyone has left),
  // [16][R + 8]; the maxima and sums of the rows into every CTA's; then each CTA fetches and adds up its share of the columns.
  // (Sums handed over by remote stores instead, in pieces of the products' 8 bytes: 7,400 clocks against 5,000.) ----
  const int opitch = R + 8;
  float* osum = reinterpret_cast<float*>(lm_smem);
  __syncwarp();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");      // (the arrive is above the tiles)
  if (warp < LM_WARPS) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = g + 8 * i;
#pragma unroll
      for (int u = 0; u < 2 * UPW; ++u)
        if (u0 + u / 2 < units)
          *reinterpret_cast<float2*>(osum + (size_t)row * opitch + 16 * u0 + 8 * u + 2 * c) =
              make_float2(o_acc[u][2 * i], o_acc[u][2 * i + 1]);
      if (c == 0)
        for (int k = warp; k < nsplit; k += LM_WARPS)
          lm_st_cluster2(lm_mapa(at_smem(ml + split * LM_HEADS + row), k), m_run[i], l_run[i]);
    }
  }
  lm_cluster_sync();
  const int pairs = hc * R / 2, share = (pairs + nsplit - 1) / nsplit;
  const int at0 = split * share, at1 = min(pairs, at0 + share);
  float2 x[16];
  auto fetch = [&](int i) {      // number i of the rows' pairs of columns, from every part
    const int row = i / (R / 2), col = 2 * (i - row * (R / 2));
    const unsigned at = at_smem(osum + (size_t)row * opitch + col);
#pragma unroll
    for (int s = 0; s < 16; ++s)
      if (s < nsplit) x[s] = lm_ld_cluster2(lm_mapa(at, s));
  };
  if (at0 + tid < at1) fetch(at0 + tid);
  // (while they come) 16 threads a row: thread k has part k's maximum and sum
  if (tid < 16 * LM_HEADS) {
    const int row = tid >> 4, k = tid & 15;
    const float2 mine = k < nsplit ? ml[k * LM_HEADS + row] : make_float2(-INFINITY, 0.f);
    const float sk = (sink && row < hc) ? sink[h0 + row] * LM_LOG2E : -INFINITY;
    float M = mine.x;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    M = fmaxf(M, sk);
    const float w = mine.x == -INFINITY ? 0.f : exp2f(mine.x - M);
    float L = w * mine.y;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
    if (sk != -INFINITY) L += exp2f(sk - M);      // the key without a value
    wts[k * LM_HEADS + row] = L > 0.f ? w / L : 0.f;
  }
  __syncthreads();
  for (int i = at0 + tid; i < at1; i += LM_THREADS) {
    const int row = i / (R / 2), col = 2 * (i - row * (R / 2));
    if (i != at0 + tid) fetch(i);
    float2 a = make_float2(0.f, 0.f);
#pragma unroll
    for (int s = 0; s < 16; ++s)
      if (s < nsplit) {
        const float w = wts[s * LM_HEADS + row];
        a.x = fmaf(w, x[s].x, a.x);
        a.y = fmaf(w, x[s].y, a.y);
      }
    *reinterpret_cast<unsigned*>(orow + (size_t)row * R + col) = lm_pack(a.x, a.y);
  }
  lm_cluster_sync();      // nobody's sums are still being read
}

// Whether the tensor-core kernel takes these sizes (bfloat16 only; the launcher checks the dtype and alignment).
extern "C" int ll_latent_attention_mma_ok(int R, int r) {
  const int KD = R + r;
  return (KD % 16) == 0 && (R % 32) == 0 && R > 0 && R <= 128 * LM_UNITS && r >= 0 && KD <= 1024;
}

typedef CUresult (*lm_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static lm_encode_fn lm_encoder() {
  static lm_encode_fn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &r) == cudaSuccess &&
        r == cudaDriverEntryPointSuccess)
      fn = (lm_encode_fn)ptr;
  }
  return fn;
}
// The plane's rows as blocks of bw columns, [KD / bw][rows][bw]: boxes of all blocks of `box_rows` rows.
static int lm_make_map(CUtensorMap* map, const void* cache, long rows, int KD, int bw, int box_rows) {
  lm_encode_fn enc = lm_encoder();
  if (enc == nullptr) return (int)cudaErrorNotSupported;
  const cuuint64_t dims[3] = {(cuuint64_t)bw, (cuuint64_t)rows, (cuuint64_t)(KD / bw)};
  const cuuint64_t strides[2] = {(cuuint64_t)KD * 2, (cuuint64_t)bw * 2};
  const cuuint32_t box[3] = {(cuuint32_t)bw, (cuuint32_t)box_rows, (cuuint32_t)(KD / bw)};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(cache), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE,
                         bw == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : bw == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

struct LmArgs {
  dim3 grid;
  size_t smem;
  cudaStream_t stream;
  bf16* out;
  const bf16 *q, *cache;
  const int* block_table;
  int bt_stride;
  const int *token_req, *req_slot, *positions;
  int first, H, R, r, page_size, num_pages, window;
  float scale_log2;
  int *status, stages, bw, box_rows;
  const float* sink;
};
// What a variant needs to be launched with any size: the same for every call, since threads that launch or plan share it.
template <int STEPS, int UPW, bool FULL, bool TMA>
static void lm_allow() {
  auto kernel = latent_attention_mma_kernel<STEPS, UPW, FULL, TMA>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LM_MAX_SMEM);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}
template <int STEPS, int UPW, bool FULL, bool TMA>
static int lm_launch(const LmArgs& a, const CUtensorMap& map) {
  static_assert(UPW >= 1 && UPW <= LM_UNITS, "units a warp");
  if (a.R > 16 * LM_WARPS * UPW || (FULL && a.R != 16 * LM_WARPS * UPW)) return (int)cudaErrorInvalidValue;
  auto kernel = latent_attention_mma_kernel<STEPS, UPW, FULL, TMA>;
  lm_allow<STEPS, UPW, FULL, TMA>();
  ll_launch_cluster(kernel, a.grid, dim3(LM_THREADS), a.smem, a.stream, (int)a.grid.z, a.out, a.q, a.cache, a.block_table,
                    a.bt_stride, a.token_req, a.req_slot, a.positions, a.first, a.H, a.R, a.r, a.page_size, a.num_pages, a.window,
                    a.scale_log2, a.status, a.stages, a.bw, a.box_rows, a.sink, map);
  return LL_LAUNCH_RESULT();
}
template <int STEPS, int UPW, bool FULL>
static int lm_launch(const LmArgs& a, const CUtensorMap& map, bool tma) {
  return tma ? lm_launch<STEPS, UPW, FULL, true>(a, map) : lm_launch<STEPS, UPW, FULL, false>(a, map);
}
// Which variant serves a latent of R numbers and r rotated ones: units a warp, whether all warps have as many (R = 512), and the
// latents that models have (512, alone or with 32 or 64 rotated numbers, and 256 with them), whose steps are straight code.
struct LmVariant {
  int steps, upw;
  bool full;
};
static LmVariant lm_variant(int R, int r) {
  const int steps = (R + r) % 32 == 0 ? (R + r) / 32 : 0;
  if (R == 512) return {steps >= 16 && steps <= 18 ? steps : 0, 4, true};
  if (R == 256) return {steps >= 8 && steps <= 10 ? steps : 0, 2, false};
  return {0, (R + 16 * LM_WARPS - 1) / (16 * LM_WARPS), false};
}
// Columns of the result that the variant for these sizes makes (at least R), 0 where there is none
extern "C" int ll_latent_attention_mma_columns(int R, int r) {
  return ll_latent_attention_mma_ok(R, r) ? 16 * LM_WARPS * lm_variant(R, r).upw : 0;
}

// Clusters of `size` CTAs that are resident at once on the current device, a CTA an SM (an SM's shared memory holds one):
// measured on a B200 33 of 4, 26 of 5, 22 of 6, 15 of 7 to 9, 7 of 12 to 16.
static int lm_resident(int size) {
  static std::atomic<int> known[64][17];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = known[dev][size].load(std::memory_order_relaxed);
  if (n == 0) {
    auto kernel = latent_attention_mma_kernel<16, 4, true, true>;
    lm_allow<16, 4, true, true>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, size);
    cfg.blockDim = dim3(LM_THREADS);
    cfg.dynamicSmemBytes = LM_MAX_SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = size;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    if (n <= 0) n = -1;      // (none)
    known[dev][size].store(n, std::memory_order_relaxed);
  }
  return n;
}
// CTAs that share a (token, group of heads)'s keys: as many as let all `pairs` of them run at once, up to a tile each.
extern "C" int ll_latent_attention_mma_splits(int pairs, int tiles) {
  for (int size = tiles < 16 ? tiles : 16; size > 1; --size)
    if (lm_resident(size) >= pairs) return size;
  return 1;
}

// `nsplit`: CTAs that share a (token, group of heads)'s keys (1 to 16: a cluster)
extern "C" int ll_latent_attention_mma(void* out, const void* q, const void* cache, const int* block_table, int bt_stride,
                                       const int* token_req, const int* req_slot, const int* positions, int first,
                                       int num_tokens, int H, int R, int r, int page_size, int num_pages, int window,
                                       float scale, int* status, int nsplit, const float* sink, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  if (!ll_latent_attention_mma_ok(R, r) || H <= 0 || page_size <= 0 || nsplit < 1) return (int)cudaErrorInvalidValue;
  const int KD = R + r;
  LmArgs a;
  a.bw = KD % 64 == 0 ? 64 : KD % 32 == 0 ? 32 : 16;
  a.box_rows = 1;
  while (a.box_rows < LM_TK && page_size % (2 * a.box_rows) == 0) a.box_rows *= 2;
  const bool tma = a.box_rows >= 8 && KD / a.bw <= 256 && (long)num_pages * page_size < (1l << 31);
  if (!tma) a.box_rows = LM_TK;
  CUtensorMap map = {};
  if (tma) {
    const int rc = lm_make_map(&map, cache, (long)num_pages * page_size, KD, a.bw, a.box_rows);
    if (rc != 0) return rc;
  }
  const size_t beside = 1024 + (size_t)LM_HEADS * (2 * KD + 16) + 2 * LM_HEADS * LM_PPITCH, tile = (size_t)LM_TK * 2 * KD;
  a.stages = LM_MAX_STAGES;
  while (a.stages > 1 && beside + a.stages * tile > LM_MAX_SMEM) --a.stages;      // (a tile of KD = 1,024 fits once)
  a.smem = beside + a.stages * tile;
  a.grid = dim3(num_tokens, (H + LM_HEADS - 1) / LM_HEADS, nsplit < 16 ? nsplit : 16);
  a.stream = stream;
  a.out = (bf16*)out;
  a.q = (const bf16*)q;
  a.cache = (const bf16*)cache;
  a.block_table = block_table;
  a.bt_stride = bt_stride;
  a.token_req = token_req;
  a.req_slot = req_slot;
  a.positions = positions;
  a.first = first;
  a.H = H;
  a.R = R;
  a.r = r;
  a.page_size = page_size;
  a.num_pages = num_pages;
  a.window = window;
  a.scale_log2 = scale * LM_LOG2E;
  a.status = status;
  a.sink = sink;
  const LmVariant v = lm_variant(R, r);
  if (v.steps == 16) return lm_launch<16, 4, true>(a, map, tma);
  if (v.steps == 17) return lm_launch<17, 4, true>(a, map, tma);
  if (v.steps == 18) return lm_launch<18, 4, true>(a, map, tma);
  if (v.steps == 8) return lm_launch<8, 2, false>(a, map, tma);
  if (v.steps == 9) return lm_launch<9, 2, false>(a, map, tma);
  if (v.steps == 10) return lm_launch<10, 2, false>(a, map, tma);
  if (v.full) return lm_launch<0, 4, true>(a, map, tma);
  if (v.upw == 1) return lm_launch<0, 1, false>(a, map, tma);
  if (v.upw == 2) return lm_launch<0, 2, false>(a, map, tma);
  if (v.upw == 3) return lm_launch<0, 3, false>(a, map, tma);
  return lm_launch<0, 4, false>(a, map, tma);
}
