// gemm_tc.cuh — prefill linear layers on the 5th-generation tensor cores (tcgen05 / UMMA), sm_100a.
//
//   C[M,N] = epilogue( A[M,K] · W[N,K]^T )      A, W, C in D (bf16 | f16), fp32 accumulation in TMEM
//
// Replaces, for seq > 1, the reference's `linear_forward` (backends/mod.rs:206-241 -> candle matmul -> cuBLAS
// gemm) for the four projections of a block (attention.rs:162-164,354; mlp.rs:22,30) with the epilogues the
// reference runs as separate tensor ops fused in: +bias (->D), +residual (transformer.rs:123,131),
// silu(gate)*up on the row-interleaved Wgu (mlp.rs:22-28).  Rounding points as everywhere: the fp32
// accumulator is rounded to D before any epilogue op.
//
// Structure (one persistent CTA per SM, 384 threads, warp-specialised):
//   warp 0   TMA producer: cp.async.bulk.tensor.2d of a 128x64 A tile and a W tile (128 or 256 rows, or this CTA's half of 256 as
//            one of a pair) per k-block into a 4- or 6-stage shared-memory ring, 128-byte swizzle, completion on full[] mbarriers
//   warp 1   MMA issuer: one thread issues tcgen05.mma.kind::f16 (M = 128 with cta_group::1, 256 over a pair of SMs with
//            cta_group::2; N = 128 or 256; K = 16) x4 per k-block from shared-memory descriptors into one of two TMEM
//            accumulators (128 lanes x BN fp32 columns each); tcgen05.commit releases the smem stage / publishes the accumulator
//   warp 2   TMEM allocator (2 x BN columns)
//   warps 4-11  epilogue: tcgen05.ld 32x32b.x32 (thread = accumulator row, every other warp of the same rows the other half of the
//            columns), fused epilogue, 16-byte global stores; overlaps with the MMAs of the next tile through the second accumulator.
//            Two warps per scheduler, because one alone issued an instruction every six cycles: 65,000 cycles for a gated tile of
//            128 x 256, twice its products' time (64 experts of 2816 x 2048 for 1000 tokens: 230 -> 180 us; four warps per scheduler 176, since
//            by then the scheduler is busy with the exponentials and divisions themselves).
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace cake {

// Tile: 128 x BN with BN in {128, 256}.  A 128x128 tile needs 32 KB of operands per 2.1 MFLOP k-block = 64 flop/B, i.e.
// ~240 GB/s per SM at the tensor peak — more than one SM pulls out of L2, which capped the kernel at ~55 % tensor-pipe
// activity.  128x256 (all 512 TMEM columns: two 128x256 fp32 accumulators) moves 48 KB per 4.2 MFLOP = 87 flop/B.
constexpr int TC_BM = 128, TC_BK = 64, TC_EPI_WARPS = 8, TC_THREADS = 128 + 32 * TC_EPI_WARPS;
constexpr int TC_BN = 128;                     // granularity the host checks N against (BN = 256 when N % 256 == 0)
template <int BN, bool PAIR = false> struct TcCfg {
  static constexpr int STAGES = (BN == 256 && !PAIR) ? 4 : 6;
  static constexpr int STAGE_BYTES = (TC_BM + (PAIR ? BN / 2 : BN)) * TC_BK * 2;  // 32 KB | 48 KB | 32 KB
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
};
// TCE_RESIDUAL_F32: C (fp32) = residual (fp32) + accumulator, nothing rounded to D — the output projection of a block whose
// residual stream is fp32 (f32_stream.cuh)
// TCE_SOFTCAP_F32: C (fp32) = cap * tanh(accumulator / cap) (cap == 0: the accumulator itself) — fp32 logits of such a model
// TCE_ACT: C (D) = act(accumulator), a feed-forward without a gate
enum { TCE_PLAIN = 0, TCE_RESIDUAL = 1, TCE_SWIGLU = 2, TCE_RESIDUAL_F32 = 3, TCE_SOFTCAP_F32 = 4, TCE_ACT = 5 };

struct TcParams {
  const void *bias;      // [N] D or nullptr (TCE_PLAIN)
  const void *residual;  // [M,N] D (TCE_RESIDUAL)
  void *C;               // [M,N] D  ([M,N/2] for TCE_SWIGLU)
  int M, N, K;
  int act;  // TCE_ACT: as plain_act; TCE_SWIGLU: 0 silu, 1 gelu_tanh, 2 the clamped form of gated_pair (its limit travels in cap)
  int ldc;  // TCE_SWIGLU / TCE_PLAIN: row stride of C in elements when it is a column range of a wider buffer (0 = N/2 resp. N;
            // a multiple of 8, like the column offset folded into C)
  float cap; // TCE_SOFTCAP_F32; TCE_SWIGLU with act 2: the limit
  // grouped product (a routed feed-forward): the rows of A are sorted by group in blocks of TC_BM rows, tile_group[m0 / TC_BM]
  // names the group of a row block (< 0: the block is empty and skipped), and group g multiplies by rows g * N .. g * N + N - 1
  // of W (map_b covers all groups).  nullptr: one group.
  const int *tile_group = nullptr;
  const int *tile_rows = nullptr;  // grouped: rows of a block that are there (nullptr: all TC_BM); the others are neither read nor written
  // TCE_RESIDUAL_F32: optional [M] fp32, C = residual + row_scale[m] * accumulator (a per-row gate on the product)
  const float *row_scale = nullptr;
  // k-block coordinate of W wraps at this many elements (0 = never): A = [P_hi | P_lo] against one copy of W
  int b_kwrap = 0;
  int w_early = 0;  // W is a weight: its first stages are requested before the wait for the kernel in front
  // `batch` products in one launch (the heads of a latent-attention layer: 16 launches of 8 CTAs were 158 us for 1000 rows): product h reads
  // A's columns from h * a_step, W's rows from h * N and writes C's columns from h * c_step (TCE_PLAIN / TCE_RESIDUAL / TCE_ACT rows of ldc)
  int batch = 1, a_step = 0, c_step = 0;
  int *err = nullptr;
};

// Tile rasterisation: groups of TC_GM m-tiles (16 x 128 rows = 16 MB of A at K=4096) are walked n-major, so the A
// group stays in the 126 MB L2 while each W tile streams once per group.  With plain m-fastest order a 1 GB A
// (bs=32 x 4k) is re-read for every W tile column: measured 815 TFLOP/s, HBM-bound.
constexpr int TC_GM = 16;
__device__ __forceinline__ void tc_tile(int t, int tiles_m, int tiles_n, int bn, int &m0, int &n0) {
  const int per_group = TC_GM * tiles_n;
  const int mg = t / per_group, r = t % per_group;
  const int gm = min(TC_GM, tiles_m - mg * TC_GM);
  m0 = (mg * TC_GM + r % gm) * TC_BM;
  n0 = (r / gm) * bn;
}

// ---- PTX wrappers ------------------------------------------------------------------------------------
// yes == 0: nothing (a predicate, not a branch)
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int c0, int c1, uint64_t *bar, uint32_t yes = 1u) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t"
      "@p cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(yes)
      : "memory");
}
// the same load with its completion counted on a barrier of the pair's first CTA (a shared::cluster address)
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *map, int c0, int c1, uint32_t bar, uint32_t yes) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t"
      "@p cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(yes)
      : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint64_t *bar, uint32_t yes = 1u) {  // arrive on the barrier at this offset in both CTAs of the pair
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t"
               "@p tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3), "r"(yes)
               : "memory");
}
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t tmem_c, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_c),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t *bar, uint32_t yes = 1u) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t"
               "@p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)), "r"(yes)
               : "memory");
}
__device__ __forceinline__ void tc_mma_f16(uint32_t tmem_c, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_c),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// shared-memory matrix descriptor, K-major operand, 128-byte swizzle, tile rows of 64 D elements (128 B):
// start address >> 4 | LBO = 1 (unused for swizzled K-major) | SBO = 1024 B (8 rows x 128 B) >> 4 |
// version 1 (sm_100) | layout type 2 (SWIZZLE_128B)
__device__ __forceinline__ uint64_t tc_smem_desc(const void *tile) {
  const uint64_t addr = (uint64_t)(smem_u32(tile) & 0x3ffff) >> 4;
  return addr | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor, kind::f16: D = f32, A/B = bf16 (1) or f16 (0), both K-major, N >> 3, M >> 4
template <typename T> __device__ __forceinline__ uint32_t tc_idesc(int bn);
template <> __device__ __forceinline__ uint32_t tc_idesc<__nv_bfloat16>(int bn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}
template <> __device__ __forceinline__ uint32_t tc_idesc<__half>(int bn) {
  return (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}

// PAIR (BN == 256 only, launched as clusters of 2 CTAs): one 256 x 256 tile on two SMs, tcgen05.mma.cta_group::2.  Each CTA loads its own 128
// rows of A and one 128-row half of the W tile and keeps its 128 rows of the accumulator; the first CTA's MMA thread multiplies both.  A
// stage is 32 KB for the work that took 48 KB, so six are in flight instead of four: a product of one round over the chip is bound by the
// ring's round trip (0.42 us per k-block with four stages, the tensor cores need 0.27).
template <typename T, int EPI, int BN, bool PAIR = false>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const TcParams p) {
  static_assert(!PAIR || BN == 256, "the pair is built for 256 columns");
  typedef TcCfg<BN, PAIR> Cfg;
  extern __shared__ unsigned char smem_raw_tc[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw_tc) + 1023) & ~(uintptr_t)1023);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t *empty = full + Cfg::STAGES;
  uint64_t *acc_full = empty + Cfg::STAGES;   // [2]
  uint64_t *acc_empty = acc_full + 2;       // [2]
  uint64_t *drained = acc_empty + 2;
  uint32_t *tmem_ptr = reinterpret_cast<uint32_t *>(drained + 1);
  int *gave_up = reinterpret_cast<int *>(tmem_ptr + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int tiles_m = (p.M + TC_BM - 1) / TC_BM;
  const int tiles_n = p.N / BN;
  const int kblocks = p.K / TC_BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; a++) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], (PAIR ? 2 : 1) * TC_EPI_WARPS); }  // (a warp of the epilogue arrives once)
    mbar_init(drained, 1);
    *gave_up = 0;
    mbar_fence_init();
  }
  if (warp == 2) {  // TMEM: 2 x BN columns = two 128 x BN fp32 accumulators
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)), "n"(2 * BN) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)), "n"(2 * BN) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (PAIR) cluster_sync_all();  // the peer's barriers exist before anything arrives on them
  pdl_launch_dependents();
  if (!p.w_early || warp != 0) pdl_wait();
  const uint32_t tmem_base = *tmem_ptr;
  // Row blocks behind the last one in use don't count: the tiles are dealt out over the chip without them (83 of 111 blocks in use, 1000 tokens: dealt out
  // with the empty ones some SMs had 7.8 tiles of 6.2; three layers 1981 -> 1922 us).
  if (p.tile_group) {
    int used = 0;
    for (int i = lane; i < tiles_m; i += 32)
      if (p.tile_group[i] >= 0) used = i + 1;
    tiles_m = __reduce_max_sync(0xffffffffu, used);
  }
  // work distribution: one tile per CTA and round; PAIR: one (256-row, 256-column) unit per cluster and round
  const uint32_t crank = PAIR ? cluster_rank() : 0u;
  const int first = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, stride = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int units_m = PAIR ? (tiles_m + 1) / 2 : tiles_m, per_product = units_m * tiles_n, n_units = per_product * p.batch;
  auto unit_tile = [&](int u, int &m0, int &n0) -> int {  // returns the product
    const int h = p.batch > 1 ? u / per_product : 0;
    u -= h * per_product;
    tc_tile(u, units_m, tiles_n, BN, m0, n0);   // m0 in units of TC_BM rows of the unit grid
    if (PAIR) m0 = m0 * 2 + (int)crank * TC_BM;
    return h;
  };

  int issued = 0;              // warp 0: stages requested
  int left = MBAR_TRIES;  // of this thread's waits
  if (warp == 0) {
    // ===================== TMA producer ==================================================================
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
      int s = 0, early = 0;
      uint32_t ph = 0;
      int a_boxes = 2;  // a grouped product's A comes in boxes of 64 rows: experts of 1000 tokens have 50 rows for the most part
      auto expect = [&](int st) {  // PAIR: the first CTA's barrier counts both CTAs' bytes
        if (!PAIR) mbar_arrive_expect_tx_if(left, &full[st], Cfg::STAGE_BYTES - (2 - a_boxes) * (TC_BM / 2 * TC_BK * 2));
        else if (crank == 0) mbar_arrive_expect_tx_if(left, &full[st], 2 * Cfg::STAGE_BYTES);
      };
      auto load_a = [&](int st, int col, int m0) {
        unsigned char *d = smem + (size_t)st * Cfg::STAGE_BYTES;
        if (PAIR) tma_load_2d_pair(d, &map_a, col, m0, cluster_map(smem_u32(&full[st]), 0u), left);
        else {
          tma_load_2d(d, &map_a, col, m0, &full[st], left);
          if (p.tile_group && a_boxes > 1) tma_load_2d(d + TC_BM / 2 * TC_BK * 2, &map_a, col, m0 + TC_BM / 2, &full[st], left);
        }
      };
      auto load_w = [&](int st, int kb, int wrow) {
        unsigned char *d = smem + (size_t)st * Cfg::STAGE_BYTES + TC_BM * TC_BK * 2;
        if (PAIR) tma_load_2d_pair(d, &map_b, kb * TC_BK, wrow + (int)crank * 128, cluster_map(smem_u32(&full[st]), 0u), left);  // a 128-row box: our half of the W tile
        else tma_load_2d(d, &map_b, p.b_kwrap ? (kb * TC_BK) % p.b_kwrap : kb * TC_BK, wrow, &full[st], left);
      };
      if (p.w_early) {  // (not a grouped product: the groups are another kernel's output)
        if (first < n_units) {
          int m0, n0;
          const int h = unit_tile(first, m0, n0);
          for (; early < Cfg::STAGES && early < kblocks; early++) { expect(early); load_w(early, early, h * p.N + n0); }
        }
        pdl_wait();
      }
      for (int t = first; t < n_units; t += stride) {
        int m0, n0;
        const int h = unit_tile(t, m0, n0);
        int wrow = h * p.N + n0;
        if (p.tile_group) {
          const int g = p.tile_group[m0 / TC_BM];
          if (g < 0) continue;
          wrow += g * p.N;
          a_boxes = p.tile_rows && p.tile_rows[m0 / TC_BM] <= TC_BM / 2 ? 1 : 2;
        }
        for (int kb = 0; kb < kblocks; kb++) {
          if (early > 0) early--;
          else {
            mbar_wait_lim(&empty[s], ph ^ 1u, p.err, left);
            expect(s);
            load_w(s, kb, wrow);
          }
          load_a(s, h * p.a_step + kb * TC_BK, m0);
          issued += left ? 1 : 0;
          if (++s == Cfg::STAGES) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (one thread; the warp runs the loop with it) ========================
    if (crank == 0) {
      const uint32_t one = elect_one();
      const uint64_t da0 = tc_smem_desc(smem), db0 = tc_smem_desc(smem + TC_BM * TC_BK * 2);
      const uint32_t idesc = PAIR ? tc_idesc<T>(BN) + ((uint32_t)(TC_BM >> 4) << 24) : tc_idesc<T>(BN);  // PAIR: M = 256
      int s = 0;
      uint32_t ph = 0;
      int it = 0;
      for (int t = first; t < n_units; t += stride) {
        if (p.tile_group) {
          int m0, n0;
          unit_tile(t, m0, n0);
          if (p.tile_group[m0 / TC_BM] < 0) continue;
        }
        const int a = it & 1;
        const uint32_t aph = (uint32_t)(it >> 1) & 1u;
        it++;
        mbar_wait_lim(&acc_empty[a], aph ^ 1u, p.err, left);  // the epilogue has drained this accumulator
        tc_fence_after();
        const uint32_t tmem_c = tmem_base + (uint32_t)(a * BN);
        for (int kb = 0; kb < kblocks; kb++) {
          mbar_wait_lim(&full[s], ph, p.err, left);
          __syncwarp();  // every lane has seen this phase before one of them begins what completes the next
          tc_fence_after();
          const uint64_t da = da0 + (uint64_t)(s * (Cfg::STAGE_BYTES >> 4)), db = db0 + (uint64_t)(s * (Cfg::STAGE_BYTES >> 4));
          if (one) {
#pragma unroll
            for (int k = 0; k < TC_BK / 16; k++)  // +32 bytes (2 x 16 B units) per K=16 slab inside the swizzle atom
              if (PAIR) tc_mma_f16_pair(tmem_c, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb | k) ? 1u : 0u);
              else tc_mma_f16(tmem_c, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb | k) ? 1u : 0u);
            if (PAIR) tc_commit_pair(&empty[s], left);  // arrives (in both CTAs) when the MMAs above have read the stage
            else tc_commit(&empty[s], left);
          }
          __syncwarp();
          if (++s == Cfg::STAGES) { s = 0; ph ^= 1u; }
        }
        if (one) {
          if (PAIR) tc_commit_pair(&acc_full[a], left);  // accumulator complete
          else tc_commit(&acc_full[a], left);
        }
        __syncwarp();
      }
    }
  } else if (warp >= 4) {
    // ===================== epilogue warps (TMEM lanes 32*(warp%4) .. +32, every fourth warp the same lanes and another range of columns) ====
    constexpr int CW = BN / (TC_EPI_WARPS / 4);  // columns of a warp
    const int wq = warp & 3, cw0 = ((warp - 4) >> 2) * CW;
    const T *bias = reinterpret_cast<const T *>(p.bias);
    const T *res = reinterpret_cast<const T *>(p.residual);
    T *C = reinterpret_cast<T *>(p.C);
    const int ld = p.ldc ? p.ldc : EPI == TCE_SWIGLU ? p.N / 2 : p.N;
    int it = 0;
    for (int t = first; t < n_units; t += stride) {
      int m0, n0;
      const int h = unit_tile(t, m0, n0);
      if (p.tile_group && p.tile_group[m0 / TC_BM] < 0) continue;
      const int a = it & 1;
      const uint32_t aph = (uint32_t)(it >> 1) & 1u;
      it++;
      const int row = m0 + wq * 32 + lane, m_end = p.tile_rows ? min(p.M, m0 + p.tile_rows[m0 / TC_BM]) : p.M;
      // the residual of a chunk of 32 columns: the first one is on its way while the products run, the next one while a chunk is finished
      constexpr int RW = EPI == TCE_RESIDUAL ? 4 : EPI == TCE_RESIDUAL_F32 ? 8 : 1;
      uint4 rr[RW];
      auto load_res = [&](int col) {
        if ((EPI != TCE_RESIDUAL && EPI != TCE_RESIDUAL_F32) || row >= m_end) return;
        const uint4 *r4 = EPI == TCE_RESIDUAL ? reinterpret_cast<const uint4 *>(res + (size_t)row * ld + h * p.c_step + col)
                                              : reinterpret_cast<const uint4 *>(reinterpret_cast<const float *>(p.residual) + (size_t)row * p.N + col);
#pragma unroll
        for (int j = 0; j < RW; j++) rr[j] = r4[j];
      };
      load_res(n0 + cw0);
      mbar_wait_lim(&acc_full[a], aph, p.err, left);
      if (!__all_sync(0xffffffffu, left != 0)) break;
      tc_fence_after();
#pragma unroll 1
      for (int c0 = cw0; c0 < cw0 + CW && m0 + wq * 32 < m_end; c0 += 32) {
        uint32_t r[32];
        tc_ld32(tmem_base + ((uint32_t)(wq * 32) << 16) + (uint32_t)(a * BN + c0), r);
        if (row < m_end) {
          if (EPI == TCE_SWIGLU) {
            uint32_t o[8];
            auto pairs = [&](int act) {
#pragma unroll
              for (int j = 0; j < 8; j++)
                o[j] = pack2x<T>(gated_pair<T>(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), act, p.cap),
                                 gated_pair<T>(__uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]), act, p.cap));
            };
            if (p.act == 0) pairs(0);  // the common one without a branch per pair
            else pairs(p.act);
            uint4 *dst = reinterpret_cast<uint4 *>(C + (size_t)row * ld + (n0 + c0) / 2);
            dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
            dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
          } else if (EPI == TCE_SOFTCAP_F32) {
            float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(p.C) + (size_t)row * p.N + n0 + c0);
#pragma unroll
            for (int j = 0; j < 8; j++) {
              float v[4];
#pragma unroll
              for (int e = 0; e < 4; e++) {
                const float a = __uint_as_float(r[4 * j + e]);
                v[e] = p.cap > 0.f ? p.cap * tanhf(a / p.cap) : a;
              }
              dst[j] = make_float4(v[0], v[1], v[2], v[3]);
            }
          } else if (EPI == TCE_RESIDUAL_F32) {
            float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(p.C) + (size_t)row * p.N + n0 + c0);
            const float rs = p.row_scale ? p.row_scale[row] : 1.0f;
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const uint4 q = rr[j % RW];
              r[4 * j] = __float_as_uint(fmaf(rs, __uint_as_float(r[4 * j]), __uint_as_float(q.x)));
              r[4 * j + 1] = __float_as_uint(fmaf(rs, __uint_as_float(r[4 * j + 1]), __uint_as_float(q.y)));
              r[4 * j + 2] = __float_as_uint(fmaf(rs, __uint_as_float(r[4 * j + 2]), __uint_as_float(q.z)));
              r[4 * j + 3] = __float_as_uint(fmaf(rs, __uint_as_float(r[4 * j + 3]), __uint_as_float(q.w)));
            }
            if (c0 + 32 < cw0 + CW) load_res(n0 + c0 + 32);
#pragma unroll
            for (int j = 0; j < 8; j++) reinterpret_cast<uint4 *>(dst)[j] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          } else {
            uint32_t o[16];
            const size_t off = (size_t)row * ld + h * p.c_step + n0 + c0;  // TCE_PLAIN may write a column range of a wider buffer
#pragma unroll
            for (int j = 0; j < 16; j++) {
              float v0, v1;
              if (EPI == TCE_ACT) {
                v0 = plain_act<T>(__uint_as_float(r[2 * j]), p.act);
                v1 = plain_act<T>(__uint_as_float(r[2 * j + 1]), p.act);
              } else {
                v0 = rnd<T>(__uint_as_float(r[2 * j]));
                v1 = rnd<T>(__uint_as_float(r[2 * j + 1]));
              }
              if (EPI == TCE_PLAIN && bias) {
                v0 = rnd<T>(v0 + DT<T>::to_f(bias[n0 + c0 + 2 * j]));
                v1 = rnd<T>(v1 + DT<T>::to_f(bias[n0 + c0 + 2 * j + 1]));
              }
              if (EPI == TCE_RESIDUAL) {
                const uint4 q = rr[(j / 4) % RW];
                const float2 rv = DT<T>::unpack2((j & 3) == 0 ? q.x : (j & 3) == 1 ? q.y : (j & 3) == 2 ? q.z : q.w);
                v0 += rv.x;
                v1 += rv.y;
              }
              o[j] = pack2x<T>(v0, v1);
            }
            if (c0 + 32 < cw0 + CW) load_res(n0 + c0 + 32);
            uint4 *dst = reinterpret_cast<uint4 *>(C + off);
#pragma unroll
            for (int j = 0; j < 4; j++) dst[j] = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(cluster_map(smem_u32(&acc_empty[a]), 0u));
        else mbar_arrive(&acc_empty[a]);
      }
    }
  }
  if (!left) *gave_up = 1;
  tc_fence_before();
  __syncthreads();
  if (*gave_up) {  // (PAIR: the first CTA's barriers count both CTAs' copies and products)
    if (warp == 0 && lane == 0 && crank == 0)
      for (int i = max(0, issued - Cfg::STAGES); i < issued; i++) mbar_drain(&full[i % Cfg::STAGES], (uint32_t)(i / Cfg::STAGES) & 1u);
    if (warp == 1 && crank == 0 && elect_one()) {
      if (PAIR) tc_commit_pair(drained);
      else tc_commit(drained);
      mbar_drain(drained, 0);
    }
    __syncthreads();
  }
  if (PAIR) cluster_sync_all();  // nobody leaves while the peer may still signal our barriers or read our operands
  if (warp == 2) {
    tc_fence_after();
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(2 * BN) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(2 * BN) : "memory");
  }
}

}  // namespace cake
