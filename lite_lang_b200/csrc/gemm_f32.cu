// True float32 products of many rows on the fifth-generation tensor cores: y[M, N] = x[M, K] * W[N, K]^T.
//
// The library's float32 product runs on the multiply-add units (54 TFLOP/s of 701 x 17,920 x 1,536).  Here every number is
// the sum of three bfloat16 numbers that hold all its 24 bits (mma_split.cuh), and a product the sum of the six products of
// terms down to 2^-16 of the largest, made by tcgen05.mma on pairs of CTAs (a tile of 256 rows x 256 columns, as in
// gemm_pair.cu): a sixth of the bfloat16 rate is five times the multiply-add units'.
//
// Accuracy.  The tensor cores cut their running sum off instead of rounding it, which over a long chain costs far more than
// the terms' last bits.  So a chain is 64 numbers of k long: the five small products first, while the sum is small, then
// the leading product's four steps; then the eight epilogue warps of each CTA take the sum out of tensor memory and add it to
// their registers with rounded additions (128 a thread), while the next chain runs in the other half of tensor memory.
// Measured against float64 the result is nearer than the library's (see the tests).
//
// Infinities and numbers above 3.39e38 have no such terms (the first one rounds to infinity, the second is NaN), so every
// sum that one of them is in comes out as NaN.  A thread that finds NaN among its sums makes the outputs again by
// multiply-adds of the numbers as stored (`gf_plain`): an infinity stays one, as in a float32 product.  (Numbers below
// 2^-109 lose their last bits: a bfloat16 number ends at 2^-133.)
//
// x comes as its three terms (`f32_terms_kernel`, [3][M][K]: x is small and read by every column tile).  W stays float32 in
// memory: its rows come by TMA into two buffers of 128 x 32, and four warps write their terms into the stage in the layout
// that the MMAs read (the MMAs of 64 numbers of k take 3,072 clocks at the tensor cores' full rate, and shared memory, which the
// MMAs read 196 KB of meanwhile, nine tenths of that).
//
// Roles in a CTA (512 threads, registers shared out between the warpgroups): warp 0 loads x's terms, warp 2 W; warp 1 of the even
// CTA issues the MMAs; warps 4-11 add a step's sum to theirs; warps 12-15 make W's terms.  A stage is 64 numbers of k: three terms of
// 128 rows of x and three of 128 rows of W, 96 KB; two stages.
// Measured on a B200, 701 x 17,920 x 1,536 gated (two thirds of a wave's last round are work): 241 us with the loads and MMAs issued by
// one lane, W's terms made by two warps and, between their sums, by the adding ones, and IEEE divisions in the epilogue (a step
// of 64 numbers 5,600 clocks; a tile's end 26,000); 170 us now (3,790 and 8,500).  What is left above the MMAs' 3,072 is the way
// from a stage that is free to its terms: 3,000 clocks, a third of them the fence before the MMAs may read.
//
// Where the tiles do not fill the chip, k is cut into `splits` parts of a work item each, whose results are
// [splits][M][N] and added up in the order of the parts (`f32_join_kernel`, or the norm that reads them).
// Gated: the even CTA's rows of W are gate rows and the odd one's the up rows of the same features (act(gate) * up
// leaves; one part).
//
// Every mbarrier wait is bounded and records LL_ERR_WAIT_TIMEOUT in the status word that the call was given (a model's step
// gives its own); the kernel then runs to its end with a wrong output and frees its memory.
#include <cuda.h>

#include "mma_split.cuh"

#define LL_ERR_WAIT_TIMEOUT 5
#define LL_ERR_TMEM_PAIR 7
#define GF_THREADS 512
// registers a thread of the warpgroups {loads and MMAs, sums, sums, terms}: together the 4 x 128 of the launch
#define GF_REGS_ISSUE 56
#define GF_REGS_SUMS 176
#define GF_REGS_TERMS 104
#define GF_TERM_BYTES (128 * 128)                 // one term of 128 rows x 64
#define GF_STAGE_BYTES (6 * GF_TERM_BYTES)
#define GF_RAW_BYTES (128 * 32 * 4)               // W as stored: 128 rows x 32, two of them
#define GF_SMEM (1024 + 2 * GF_STAGE_BYTES + 2 * GF_RAW_BYTES + 256)

__device__ __forceinline__ void gf_mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void gf_mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gf_mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void gf_mbar_arrive_cluster(unsigned bar_cluster) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster) : "memory");
}
__device__ __forceinline__ bool gf_mbar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void gf_mbar_wait(unsigned bar, unsigned parity, int* status, bool& dead) {
  if (dead || gf_mbar_try(bar, parity)) return;
  const long long t0 = clock64();
  while (!gf_mbar_try(bar, parity)) {
    if (clock64() - t0 > 4000000000ll) {
      set_status(status, LL_ERR_WAIT_TIMEOUT);
      dead = true;
      return;
    }
  }
}
// One lane of a converged warp, always the same (whole warps run the loops that issue copies and MMAs, so that their operands
// stay in uniform registers; in a branch of one lane an MMA took 145 clocks to issue).
__device__ __forceinline__ bool gf_elect() {
  unsigned p;
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ unsigned gf_cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void gf_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned gf_mapa(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ unsigned gf_ld_cluster(unsigned addr_cluster) {
  unsigned v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr_cluster) : "memory");
  return v;
}
// TMA box into this CTA's shared memory; its bytes complete on a barrier of the pair's even CTA (or this one's)
__device__ __forceinline__ void gf_tma_load(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar_cluster)
      : "memory");
}
// K-major operand tile, rows of 128 bytes with the 128-byte swizzle: groups of 8 rows are 1024 bytes apart
__device__ __forceinline__ unsigned long long gf_desc(unsigned smem_addr) {
  return (unsigned long long)((smem_addr >> 4) & 0x3FFF) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void gf_mma(unsigned tmem_d, unsigned long long desc_a, unsigned long long desc_b, unsigned idesc,
                                       unsigned accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void gf_commit_pair(unsigned bar) {
  const unsigned short mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(mask)
               : "memory");
}
// 16 columns of the thread's lane of tensor memory: asked for, and there (the registers are tied to the wait)
__device__ __forceinline__ void gf_ld16_issue(unsigned taddr, unsigned (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void gf_ld16_wait(unsigned (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

// terms[p][i] of x[M][K] (row stride x_stride): four numbers a thread
__global__ void __launch_bounds__(256)
f32_terms_kernel(bf16* __restrict__ terms, const float* __restrict__ x, long x_stride, long rows, int K) {
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int per = K / 4;
  const long total = rows * per, plane = rows * (long)K;
  for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long)gridDim.x * 256) {
    const long t = i / per;
    const int c = (int)(i - t * per) * 4;
    const float4 v = *reinterpret_cast<const float4*>(x + t * x_stride + c);
    uint2 p0, p1, p2;
    ms_split(v.x, v.y, p0.x, p1.x, p2.x);
    ms_split(v.z, v.w, p0.y, p1.y, p2.y);
    bf16* d = terms + t * K + c;
    *reinterpret_cast<uint2*>(d) = p0;
    *reinterpret_cast<uint2*>(d + plane) = p1;
    *reinterpret_cast<uint2*>(d + 2 * plane) = p2;
  }
}

// out (+)= the parts, added in their order
__global__ void __launch_bounds__(256)
f32_join_kernel(float* __restrict__ out, long out_stride, const float* __restrict__ parts, int splits, long rows, int N,
                int accumulate) {
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();
  const int per = N / 4;
  const long total = rows * per, plane = rows * (long)N;
  for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long)gridDim.x * 256) {
    const long t = i / per;
    const int c = (int)(i - t * per) * 4;
    float4 s = *reinterpret_cast<const float4*>(parts + t * N + c);
    for (int p = 1; p < splits; ++p) {
      const float4 v = *reinterpret_cast<const float4*>(parts + p * plane + t * N + c);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    float4* d = reinterpret_cast<float4*>(out + t * out_stride + c);
    if (accumulate) {
      const float4 v = *d;
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    *d = s;
  }
}

struct GfParams {
  const float* x;                    // the operands as stored (and their row strides), for sums that are NaN
  const float* w;
  long x_stride, w_stride;
  float* out;
  long out_stride, part_stride;      // numbers from a row, and from a part, to the next
  int M, N, K;                       // rows, output features (gated: W has 2 N rows), inner size
  int m_tiles, tiles, splits;        // tiles of 256 rows, all tiles, parts of k
  GateAct gate;
  int* status;
};

// a sum over numbers k0 .. k1 - 1 of k in float32
__device__ __noinline__ float gf_plain(const float* x, const float* w, int k0, int k1) {
  float s = 0.f;
  for (int k = k0; k < k1 && s == s; k += 4) {       // (K is a multiple of 8; NaN stays NaN)
    const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
    s = fmaf(a.x, b.x, s);
    s = fmaf(a.y, b.y, s);
    s = fmaf(a.z, b.z, s);
    s = fmaf(a.w, b.w, s);
  }
  return s;
}

// The activation of 64 pairs (gate numbers, then up numbers) to dst[0 .. left - 1].  (The divisions of ll_gated, with a branch
// each, made a tile's end 26,000 clocks, eight of its 24 steps.)  Returns whether some pair has to be made again by the division.
template <int ACT>
__device__ __forceinline__ bool gf_gate_row(float* dst, const float (&v)[128], int left, const GateAct& k) {
  DivideMet met;
#pragma unroll
  for (int i = 0; i < 64; i += 4) {
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = ll_gated_divide<ACT>(v[i + j], v[64 + i + j], k, met);
    if (i < left) *reinterpret_cast<float4*>(dst + i) = make_float4(o[0], o[1], o[2], o[3]);      // (N is a multiple of 4)
  }
  return met.far();
}

template <bool GATED>
__global__ void __launch_bounds__(GF_THREADS, 1)
gemm_f32_kernel(const GfParams p, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap) {
  constexpr int COLS = GATED ? 128 : 256;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* raw = smem + 2 * GF_STAGE_BYTES;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(raw + 2 * GF_RAW_BYTES);
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 14);
  const unsigned stage0 = ms_smem(smem);
  const unsigned a_full0 = ms_smem(bars), b_full0 = a_full0 + 16;          // even CTA: x's terms, W's terms of a stage are there
  const unsigned free0 = a_full0 + 32;                                     // both: the MMAs have read the stage
  const unsigned acc_full0 = a_full0 + 48, acc_empty0 = a_full0 + 64;      // both; even CTA
  const unsigned raw_full0 = a_full0 + 80, raw_empty0 = a_full0 + 96;      // this CTA's buffers of W as stored

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const unsigned rank = gf_cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      gf_mbar_init(a_full0 + 8 * s, 1);        // the even CTA announces both CTAs' bytes
      gf_mbar_init(b_full0 + 8 * s, 8);        // the four warps that make terms, of both CTAs
      gf_mbar_init(free0 + 8 * s, 1);
      gf_mbar_init(acc_full0 + 8 * s, 1);
      gf_mbar_init(acc_empty0 + 8 * s, 16);
      gf_mbar_init(raw_full0 + 8 * s, 1);
      gf_mbar_init(raw_empty0 + 8 * s, 4);     // the warps that make terms
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ms_smem(tmem_slot)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  gf_cluster_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_slot;
  const bool paired = gf_ld_cluster(gf_mapa(ms_smem(tmem_slot), rank ^ 1u)) == tmem;
  if (!paired && tid == 0) set_status(p.status, LL_ERR_TMEM_PAIR);
  LL_PDL_TRIGGER();
  LL_PDL_WAIT();

  bool dead = false;
  const int kboxes = (p.K + 63) / 64, per = (kboxes + p.splits - 1) / p.splits;
  const int items = p.tiles * p.splits;
  // item: a tile and a part of k, rows fastest; k boxes k0 .. k1 - 1 (never empty: the launcher chose the parts so)
  auto work = [&](int item, int& mt, int& nt, int& part, int& k0, int& k1) {
    part = item / p.tiles;
    const int t = item - part * p.tiles;
    mt = t % p.m_tiles;
    nt = t / p.m_tiles;
    k0 = part * per;
    k1 = min(kboxes, k0 + per);
  };
  if (paired) {
    if (warp < 4) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(GF_REGS_ISSUE));
      if (warp == 0) {
        // ------------------------------ loads of x's terms ------------------------------
        const unsigned lead_a_full = gf_mapa(a_full0, 0);
        int s = 0;
        unsigned ph = 1;      // (a fresh barrier counts as passed in this phase)
        for (int item = pair; item < items; item += pairs) {
          int mt, nt, part, k0, k1;
          work(item, mt, nt, part, k0, k1);
          const int x_row = mt * 256 + (int)rank * 128;
          for (int kc = k0; kc < k1; ++kc) {
            gf_mbar_wait(free0 + 8 * s, ph, p.status, dead);
            if (gf_elect()) {
              if (rank == 0) gf_mbar_expect_tx(a_full0 + 8 * s, 2 * 3 * GF_TERM_BYTES);
#pragma unroll
              for (int q = 0; q < 3; ++q)
                gf_tma_load(stage0 + s * GF_STAGE_BYTES + q * GF_TERM_BYTES, &xmap, kc * 64, q * p.M + x_row, lead_a_full + 8 * s);
            }
            __syncwarp();
            s ^= 1;
            if (s == 0) ph ^= 1;
          }
        }
      } else if (warp == 2) {
        // ------------------------------ loads of W as stored ------------------------------
        const unsigned own_full = gf_mapa(raw_full0, rank);
        unsigned ph = 1;
        for (int item = pair; item < items; item += pairs) {
          int mt, nt, part, k0, k1;
          work(item, mt, nt, part, k0, k1);
          const int w_row = GATED ? (int)rank * p.N + nt * 128 : nt * 256 + (int)rank * 128;
          for (int kc = k0; kc < k1; ++kc, ph ^= 1) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              gf_mbar_wait(raw_empty0 + 8 * q, ph, p.status, dead);
              if (gf_elect()) {
                gf_mbar_expect_tx(raw_full0 + 8 * q, GF_RAW_BYTES);
                gf_tma_load(ms_smem(raw) + q * GF_RAW_BYTES, &wmap, kc * 64 + q * 32, w_row, own_full + 8 * q);
              }
              __syncwarp();
            }
          }
        }
      } else if (warp == 1 && rank == 0) {
        // ------------------------------ MMA issue (even CTA) ------------------------------
        constexpr unsigned IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((256u >> 4) << 24);
        const unsigned long long desc0 = gf_desc(stage0);
        int s = 0;
        unsigned ph = 0;
        for (int item = pair; item < items; item += pairs) {
          int mt, nt, part, k0, k1;
          work(item, mt, nt, part, k0, k1);
          for (int kc = k0; kc < k1; ++kc) {
            gf_mbar_wait(acc_empty0 + 8 * s, ph ^ 1, p.status, dead);
            gf_mbar_wait(a_full0 + 8 * s, ph, p.status, dead);
            gf_mbar_wait(b_full0 + 8 * s, ph, p.status, dead);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned acc = tmem + (unsigned)(s * 256);
            const unsigned long long a = desc0 + (unsigned)(s * (GF_STAGE_BYTES >> 4)), b = a + (3 * GF_TERM_BYTES >> 4);
            // (term of x, term of W): the small products first, the leading one last; 16 of k are 32 bytes further
            constexpr int TA[6] = {2, 1, 0, 1, 0, 0}, TB[6] = {0, 1, 2, 0, 1, 0};
            if (gf_elect()) {
#pragma unroll
              for (int q = 0; q < 6; ++q)
#pragma unroll
                for (int k16 = 0; k16 < 4; ++k16)
                  gf_mma(acc, a + TA[q] * (GF_TERM_BYTES >> 4) + 2 * k16, b + TB[q] * (GF_TERM_BYTES >> 4) + 2 * k16, IDESC,
                         (q > 0 || k16 > 0) ? 1u : 0u);
              gf_commit_pair(free0 + 8 * s);
              gf_commit_pair(acc_full0 + 8 * s);
            }
            __syncwarp();
            s ^= 1;
            if (s == 0) ph ^= 1;
          }
        }
      }
    } else if (warp >= 12) {
      // ------------------------------ W's terms ------------------------------
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(GF_REGS_TERMS));
      const unsigned b_full_lead = gf_mapa(b_full0, 0);
      // thread e has numbers 8 c .. 8 c + 7 of a buffer in rows r, r + 32, ... r + 96: 32 bytes as stored, 16 a term.  Of eight
      // threads half have rows 4 further, and read the halves of their 32 bytes in the other order: all meet different banks
      const int e = tid - 384, c = e & 3, t = e >> 2, odd = t & 1, r = odd * 4 + ((t >> 1) & 3) + (t & 24);
      const unsigned char* src = raw + r * 128 + c * 32;
      int s = 0;
      unsigned ph = 1, rph = 0;
      for (int item = pair; item < items; item += pairs) {
        int mt, nt, part, k0, k1;
        work(item, mt, nt, part, k0, k1);
        for (int kc = k0; kc < k1; ++kc, rph ^= 1) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float4 v[4][2];
            gf_mbar_wait(raw_full0 + 8 * q, rph, p.status, dead);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              v[j][0] = *reinterpret_cast<const float4*>(src + q * GF_RAW_BYTES + 4096 * j + 16 * odd);
              v[j][1] = *reinterpret_cast<const float4*>(src + q * GF_RAW_BYTES + 4096 * j + 16 - 16 * odd);
            }
            if (q == 0) gf_mbar_wait(free0 + 8 * s, ph, p.status, dead);
            unsigned char* dst = smem + s * GF_STAGE_BYTES + 3 * GF_TERM_BYTES + r * 128 + (((q * 4 + c) ^ (r & 7)) << 4);
#pragma unroll
            for (int j = 0; j < 4; ++j) {      // (32 rows further: 4,096 bytes, the same swizzle)
              const float4 lo = odd ? v[j][1] : v[j][0], hi = odd ? v[j][0] : v[j][1];
              uint4 t0, t1, t2;
              ms_split(lo.x, lo.y, t0.x, t1.x, t2.x);
              ms_split(lo.z, lo.w, t0.y, t1.y, t2.y);
              ms_split(hi.x, hi.y, t0.z, t1.z, t2.z);
              ms_split(hi.z, hi.w, t0.w, t1.w, t2.w);
              *reinterpret_cast<uint4*>(dst + 4096 * j) = t0;
              *reinterpret_cast<uint4*>(dst + 4096 * j + GF_TERM_BYTES) = t1;
              *reinterpret_cast<uint4*>(dst + 4096 * j + 2 * GF_TERM_BYTES) = t2;
            }
            // (the buffer is given back behind the last use of what was read from it: an arrival right behind the loads
            // overtook them, and the next copy was in their place)
            __syncwarp();
            if (lane == 0) gf_mbar_arrive(raw_empty0 + 8 * q);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) gf_mbar_arrive_cluster(b_full_lead + 8 * s);
          s ^= 1;
          if (s == 0) ph ^= 1;
        }
      }
    } else {
      // ------------------------------ sums (warps 4..11) ------------------------------
      asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(GF_REGS_SUMS));
      const int ew = warp & 3;              // the 32 tensor-memory lanes this warp may read
      const int eh = (warp - 4) >> 2;       // its columns: 64 eh .. + 63 and 128 + 64 eh .. + 63
      const unsigned acc_empty_lead = gf_mapa(acc_empty0, 0);
      float sum[128];
      int s = 0;
      unsigned ph = 0;
      for (int item = pair; item < items; item += pairs) {
        int mt, nt, part, k0, k1;
        work(item, mt, nt, part, k0, k1);
#pragma unroll
        for (int i = 0; i < 128; ++i) sum[i] = 0.f;
        for (int kc = k0; kc < k1; ++kc) {
          gf_mbar_wait(acc_full0 + 8 * s, ph, p.status, dead);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned taddr = tmem + ((unsigned)(32 * ew) << 16) + (unsigned)(s * 256 + 64 * eh);
          unsigned v[2][16];      // (the next 16 columns are on their way while these are added)
          gf_ld16_issue(taddr, v[0]);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            gf_ld16_wait(v[c & 1]);
            if (c < 7) gf_ld16_issue(taddr + ((c + 1) >> 2) * 128 + ((c + 1) & 3) * 16, v[(c + 1) & 1]);
#pragma unroll
            for (int i = 0; i < 16; ++i) sum[16 * c + i] += __uint_as_float(v[c & 1][i]);
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) gf_mbar_arrive_cluster(acc_empty_lead + 8 * s);
          s ^= 1;
          if (s == 0) ph ^= 1;
        }
        const int row = mt * 256 + (int)rank * 128 + 32 * ew + lane;
        if (row < p.M) {
          float* dst = p.out + part * p.part_stride + (size_t)row * p.out_stride;
          bool nan = false;
#pragma unroll
          for (int i = 0; i < 128; ++i) nan |= sum[i] != sum[i];
          if (GATED) {
            const int f0 = nt * 128 + 64 * eh, left = p.N - f0;
            bool odd = false;
            if (p.gate.act == 0) odd = gf_gate_row<0>(dst + f0, sum, left, p.gate);
            else if (p.gate.act == 2) odd = gf_gate_row<2>(dst + f0, sum, left, p.gate);
            else if (p.gate.act == 3) odd = gf_gate_row<3>(dst + f0, sum, left, p.gate);
            else gf_gate_row<1>(dst + f0, sum, left, p.gate);
            if (odd) {
#pragma unroll
              for (int i = 0; i < 64; ++i)
                if (i < left) dst[f0 + i] = ll_gated(sum[i], sum[64 + i], p.gate);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 128; i += 4) {
              const int f = nt * COLS + (i >> 6) * 128 + 64 * eh + (i & 63);
              if (f < p.N) *reinterpret_cast<float4*>(dst + f) = make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
            }
          }
          if (nan) {
            const float* xr = p.x + (size_t)row * p.x_stride;
            const int last = min(p.K, k1 * 64);
#pragma unroll 1
            for (int i = 0; i < (GATED ? 64 : 128); ++i) {
              const int f = nt * COLS + 64 * eh + (GATED ? i : (i >> 6) * 128 + (i & 63));
              if (f >= p.N) continue;
              if (GATED) {      // (an activation may have made a number of NaN)
                const float g = gf_plain(xr, p.w + (size_t)f * p.w_stride, k0 * 64, last);
                dst[f] = ll_gated(g, gf_plain(xr, p.w + (size_t)(p.N + f) * p.w_stride, k0 * 64, last), p.gate);
              } else if (dst[f] != dst[f]) {
                dst[f] = gf_plain(xr, p.w + (size_t)f * p.w_stride, k0 * 64, last);
              }
            }
          }
        }
        __syncwarp();
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  gf_cluster_sync();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

typedef CUresult (*gf_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static gf_encode_fn gf_encoder() {
  static gf_encode_fn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (gf_encode_fn)ptr;
  }
  return fn;
}

static int gf_make_map(CUtensorMap* map, const void* base, long rows, long K, long stride, bool terms) {
  gf_encode_fn enc = gf_encoder();
  if (enc == nullptr) return (int)cudaErrorNotSupported;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)stride * (terms ? 2 : 4)};
  const cuuint32_t box[2] = {terms ? 64u : 32u, 128};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, terms ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         terms ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

template <bool GATED>
static int gf_launch(GfParams& p, const void* terms, int sm_count, cudaStream_t stream) {
  CUtensorMap xmap, wmap;
  int rc = gf_make_map(&xmap, terms, 3l * p.M, p.K, p.K, true);
  if (rc == 0) rc = gf_make_map(&wmap, p.w, GATED ? 2l * p.N : (long)p.N, p.K, p.w_stride, false);
  if (rc != 0) return rc;
  const cudaError_t ac = cudaFuncSetAttribute(gemm_f32_kernel<GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GF_SMEM);
  if (ac != cudaSuccess) return (int)ac;
  const int items = p.tiles * p.splits, most = sm_count / 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (items < most ? items : most), 1, 1);
  cfg.blockDim = dim3(GF_THREADS);
  cfg.dynamicSmemBytes = GF_SMEM;
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
  cudaLaunchKernelEx(&cfg, gemm_f32_kernel<GATED>, p, xmap, wmap);
  return LL_LAUNCH_RESULT();
}

// x: float32 [M, K] (row stride a multiple of 4); w: float32 [N, K] (gated: [2 N, K], gate rows first), row stride w_stride, a
// multiple of 4; out: float32 [M, N]; K a multiple of 8, N of 4; terms: bfloat16 scratch [3][M][K].  splits > 1 (not gated):
// parts: float32 scratch [splits][M][N], joined into out (`accumulate`: added to it) unless out is null.  Launches two or
// three kernels.
extern "C" int ll_gemm_f32(float* out, long out_stride, const float* x, long x_stride, const float* w, long w_stride, int M,
                           int N, int K, void* terms, float* parts, int splits, int accumulate, int gated, float limit,
                           float alpha, int sm_count, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (K % 8) != 0 || (N % 4) != 0 || (x_stride % 4) != 0 || (w_stride % 4) != 0 || sm_count < 2 || gated < 0 ||
      gated > 4 || splits < 1 || (gated && splits != 1) || ((splits > 1 || accumulate) && parts == nullptr) ||
      (out == nullptr && parts == nullptr) || (out_stride % 4) != 0 ||
      (((uintptr_t)out | (uintptr_t)x | (uintptr_t)w | (uintptr_t)terms | (uintptr_t)parts) % 16) != 0)
    return (int)cudaErrorInvalidValue;
  const int kboxes = (K + 63) / 64, per = (kboxes + splits - 1) / splits;
  if ((long)per * (splits - 1) >= kboxes) return (int)cudaErrorInvalidValue;        // a part without work
  const bool join = splits > 1 || accumulate || out == nullptr;
  const long pieces = (long)M * (K / 4), most = 16l * sm_count;
  ll_launch(f32_terms_kernel, dim3((unsigned)((pieces + 255) / 256 < most ? (pieces + 255) / 256 : most)), dim3(256), 0, stream,
            (bf16*)terms, x, x_stride, (long)M, K);
  GfParams p;
  p.x = x;
  p.w = w;
  p.x_stride = x_stride;
  p.w_stride = w_stride;
  p.out = join ? parts : out;
  p.out_stride = join ? N : out_stride;
  p.part_stride = (long)M * N;
  p.M = M;
  p.N = N;
  p.K = K;
  p.m_tiles = (M + 255) / 256;
  p.tiles = p.m_tiles * ((N + (gated ? 127 : 255)) / (gated ? 128 : 256));
  p.splits = splits;
  p.gate = {gated > 0 ? gated - 1 : 0, limit, alpha};
  p.status = status;
  const int rc = gated ? gf_launch<true>(p, terms, sm_count, stream)
                       : gf_launch<false>(p, terms, sm_count, stream);
  if (rc != 0 || !join || out == nullptr) return rc;
  const long out_pieces = (long)M * (N / 4);
  ll_launch(f32_join_kernel, dim3((unsigned)((out_pieces + 255) / 256 < most ? (out_pieces + 255) / 256 : most)), dim3(256), 0,
            stream, out, out_stride, (const float*)parts, splits, (long)M, N, accumulate);
  return LL_LAUNCH_RESULT();
}
