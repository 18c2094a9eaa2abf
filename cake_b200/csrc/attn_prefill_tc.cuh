// attn_prefill_tc.cuh — causal GQA flash attention for prefill (seq > 1, head_dim 128) on the 5th-generation tensor
// cores (tcgen05 / UMMA + TMEM), sm_100a.
//
// Same operator and the same rounding points as attn_prefill_mma_kernel (attn_prefill.cuh), which restates
// cake-core/src/models/common/attention.rs:299-349 (scores = q k^T * 1/sqrt(hd) in fp32, causal mask, fp32 softmax,
// probabilities x V, one rounding to D at the end): S in fp32 from D operands, P kept to ~16 mantissa bits as
// P_hi + P_lo (two D operands), O accumulated in fp32, rounded once.  What changes is who multiplies: mma.sync tops out
// near 465 TFLOP/s on this part (ncu: HMMA pipe 50 % active at 231 TFLOP/s), a quarter of what tcgen05 delivers.
//
// One CTA = one tile of 128 query rows (the G query heads of one key head x 128 / G tokens) and a range of keys; two CTAs per SM
// (2 x 256 TMEM columns, 2 x 97 KB shared memory), so one CTA's softmax overlaps the other's MMAs.  192 threads:
//   warps 0-3  softmax: thread = query row (TMEM lane).  tcgen05.ld of the 128 x 64 S tile, scale + mask + running max /
//              sum entirely in-thread (no shuffles), P_hi / P_lo packed to D and stored with tcgen05.st over the S tile they
//              came from (the MMA takes its A operand from TMEM), lazy rescale of O in TMEM (only when the row max grew by
//              more than tau, P stays <= e^tau; the final O / l is the same quotient), epilogue O / l -> D -> global
//   warp 4     TMA producer: Q tile once, then 64-key K and V tiles through two-stage rings (3-D maps: keys past the
//              visible length and query rows past S are zero-filled by the TMA unit, nothing uninitialised reaches an MMA)
//   warp 5     TMEM allocator + MMA issuer (one thread): S = Q K^T (8 x M128 N64 K16, operands from shared memory) into one
//              of two S buffers — S of tile j+1 is issued BEFORE P V of tile j, so the softmax of j+1 runs under it —
//              and O += P_hi V + P_lo V (8 x M128 N128 K16, P from TMEM, V consumed straight from its [key][hd] cache
//              layout as an MN-major B operand)
#pragma once
#include "gemm_tc.cuh"

namespace cake {

constexpr int FT_BM = 128, FT_BN = 64, FT_HD = 128, FT_THREADS = 192;
constexpr int FT_Q_BYTES = FT_BM * FT_HD * 2;   // 32 KB: two 128-row x 64-dim boxes
constexpr int FT_KV_BYTES = FT_BN * FT_HD * 2;  // 16 KB: two 64-key x 64-dim boxes
constexpr int FT_SMEM_BYTES = FT_Q_BYTES + 4 * FT_KV_BYTES + 1024 /*align*/ + 128 /*barriers*/;  // Q + 2 K stages + 2 V stages
constexpr int FT_TMEM_COLS = 256;               // S/P buffers: columns 0..63 and 64..127 (P_hi | P_lo packed over S), O: 128..255

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int c0, int c1, int c2, uint64_t *bar, uint32_t yes = 1u) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %6, 0;\n\t"
      "@p cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(yes)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
      "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[tmem] (+)= A[tmem] x B[smem]: the A operand (M = lane, K packed two D values per 32-bit column) comes from tensor memory
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t tmem_c, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_c),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ float ft_ex2(float x) {  // MUFU.EX2: 2^x, 2^-inf = 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// MN-major B operand (V: rows = keys = K dimension, 64 contiguous head dims = one 128-byte swizzle row):
// LBO = distance between the two 64-dim halves, SBO = 1024 B between groups of 8 keys
__device__ __forceinline__ uint64_t ft_desc_mn(const void *tile, uint32_t lbo_bytes) {
  const uint64_t addr = (uint64_t)(smem_u32(tile) & 0x3ffff) >> 4;
  return addr | ((uint64_t)(lbo_bytes >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// barriers: Q, two stages of K, K consumed, V, V consumed, S, then P (128 arrivals), O, and the products of a CTA that gave up a wait
constexpr int FT_BARS = 14;
// a CTA that gave up: its copies and products in flight end before it leaves
__device__ __forceinline__ void ft_drain(uint64_t *bars, int warp, int lane, int k_loads, int v_loads) {
  if (warp == 4 && lane == 0) {
    if (k_loads > 0) mbar_drain(&bars[0], 0);
    for (int i = max(0, k_loads - 2); i < k_loads; i++) mbar_drain(&bars[1 + (i & 1)], (uint32_t)(i >> 1) & 1u);
    for (int i = max(0, v_loads - 2); i < v_loads; i++) mbar_drain(&bars[5 + (i & 1)], (uint32_t)(i >> 1) & 1u);
  }
  if (warp == 5 && elect_one()) {
    tc_commit(&bars[FT_BARS - 1]);
    mbar_drain(&bars[FT_BARS - 1], 0);
  }
  __syncthreads();
}

// Query rows of a tile: the G query heads of one key head side by side, row = token * G + head, so that one pass over K and V serves
// all of them (a step of one token has G rows, not one) and a tile of a causal prompt spans 128 / G tokens: less of its last key
// tiles is masked.  `splits` CTAs of a cluster cut the tile's keys between them where tiles alone don't fill the chip (few rows on a
// long context); each finishes 128 / splits of the columns, with the partial sums and the running maxima exchanged over the cluster.
struct FtParams {
  void *y;
  int S, n_heads, n_kv, pos0;
  int G, tpt, splits_log2;  // query heads per key head, tokens per tile
  float scale_log2, tau_log2;
  int *err;
};

// SPLIT: clusters that cut the keys; without it every CTA sees its rows' first key in its first tile.
template <typename T, bool SPLIT>
__global__ void __launch_bounds__(FT_THREADS, 2)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const FtParams p) {
  extern __shared__ unsigned char ft_smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(ft_smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char *q_s = smem;
  unsigned char *k_s = q_s + FT_Q_BYTES;       // [2] stages
  unsigned char *v_s = k_s + 2 * FT_KV_BYTES;  // [2] stages
  uint64_t *bars = reinterpret_cast<uint64_t *>(v_s + 2 * FT_KV_BYTES);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 3, *v_full = bars + 5, *v_empty = bars + 7, *s_full = bars + 9,
           *p_full = bars + 11, *o_full = bars + 12;
  uint32_t *tmem_ptr = reinterpret_cast<uint32_t *>(bars + FT_BARS);
  int *gave_up = reinterpret_cast<int *>(tmem_ptr + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.S, pos0 = p.pos0, G = p.G, tpt = p.tpt, lg = SPLIT ? p.splits_log2 : 0, splits = 1 << lg;
  const int rank = (int)blockIdx.x & (splits - 1);                        // the cluster's CTAs are neighbours along x
  const int mt = (int)(gridDim.x >> lg) - 1 - (int)(blockIdx.x >> lg);  // heavy (late) query tiles first
  const int kvh = blockIdx.y, b = blockIdx.z, t0 = mt * tpt;
  const int kv_end = pos0 + min(S, t0 + tpt);  // keys visible to the last query of this tile
  const int all_tiles = (kv_end + FT_BN - 1) / FT_BN;
  const int j0 = (all_tiles * rank) >> lg, n_tiles = ((all_tiles * (rank + 1)) >> lg) - j0;  // 0: fewer tiles than CTAs
  const int rows = G * min(tpt, S - t0);  // of 128
  const int row = (warp & 3) * 32 + lane, tok = row / G;  // softmax warps: this thread's query row and its token

  if (threadIdx.x == 0) {
    for (int i = 0; i < FT_BARS; i++) mbar_init(&bars[i], i == 11 ? 128u : 1u);
    *gave_up = 0;
    mbar_fence_init();
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)), "n"(FT_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t tmem_base = *tmem_ptr;
  const uint32_t tmem_o = tmem_base + 128u;  // S/P buffer i at columns 64 i

  const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
  const bool busy = warp < 4 && warp * 32 < rows;  // a warp without rows keeps the barriers' counts and computes nothing
  float m_run = -INFINITY, l_run = 0.f;            // m_run: reference max of the raw scores (unscaled)

  int left = MBAR_TRIES;    // of this thread's waits
  int k_loads = 0, v_loads = 0;  // warp 4: tiles requested
  if (warp == 4) {
    // ===================== TMA producer ====================================================================
    if (lane == 0 && n_tiles > 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
      mbar_arrive_expect_tx(q_full, (uint32_t)(2 * G * tpt * 128));
      tma_load_4d(q_s, &map_q, 0, kvh * G, t0, b, q_full);
      tma_load_4d(q_s + FT_Q_BYTES / 2, &map_q, 64, kvh * G, t0, b, q_full);
      const int slab = b * p.n_kv + kvh;
      for (int j = 0; j < n_tiles; j++) {
        const int st = j & 1;
        const uint32_t eph = (uint32_t)((j >> 1) - 1) & 1u;  // the stage's previous use (tile j-2) has been consumed
        unsigned char *kd = k_s + st * FT_KV_BYTES, *vd = v_s + st * FT_KV_BYTES;
        if (j >= 2) mbar_wait_lim(&k_empty[st], eph, p.err, left);
        mbar_arrive_expect_tx_if(left, &k_full[st], FT_KV_BYTES);
        tma_load_3d(kd, &map_k, 0, (j0 + j) * FT_BN, slab, &k_full[st], left);
        tma_load_3d(kd + FT_KV_BYTES / 2, &map_k, 64, (j0 + j) * FT_BN, slab, &k_full[st], left);
        k_loads += left ? 1 : 0;
        if (j >= 2) mbar_wait_lim(&v_empty[st], eph, p.err, left);
        mbar_arrive_expect_tx_if(left, &v_full[st], FT_KV_BYTES);
        tma_load_3d(vd, &map_v, 0, (j0 + j) * FT_BN, slab, &v_full[st], left);
        tma_load_3d(vd + FT_KV_BYTES / 2, &map_v, 64, (j0 + j) * FT_BN, slab, &v_full[st], left);
        v_loads += left ? 1 : 0;
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    // ===================== MMA issuer (one thread; the warp runs the loop with it) ==========================
    if (n_tiles > 0) {
      const uint32_t one = elect_one();
      const uint32_t idesc_s = tc_idesc<T>(FT_BN);                   // M128 N64, A and B K-major
      const uint32_t idesc_o = tc_idesc<T>(FT_HD) | (1u << 16);      // M128 N128, A from TMEM, B (V) MN-major
      auto issue_s = [&](int j) {  // S_j = Q K_j^T into S buffer j&1
        const int st = j & 1;
        mbar_wait_lim(&k_full[st], (uint32_t)(j >> 1) & 1u, p.err, left);
        __syncwarp();  // every lane has seen this phase before one of them begins what completes the next
        tc_fence_after();
        const uint64_t q0 = tc_smem_desc(q_s), kt = tc_smem_desc(k_s) + (uint64_t)(st * (FT_KV_BYTES >> 4));
        if (one) {
#pragma unroll
          for (int k = 0; k < FT_HD / 16; k++) {  // head dims 16k..16k+15: box k/4, 32-byte slab k%4 inside the swizzle row
            const uint64_t da = q0 + (uint64_t)((k >> 2) * (FT_Q_BYTES / 2 >> 4) + (k & 3) * 2);
            const uint64_t db = kt + (uint64_t)((k >> 2) * (FT_KV_BYTES / 2 >> 4) + (k & 3) * 2);
            tc_mma_f16(tmem_base + (uint32_t)(st * 64), da, db, idesc_s, k ? 1u : 0u);
          }
          tc_commit(&k_empty[st], left);
          tc_commit(&s_full[st], left);
        }
        __syncwarp();
      };
      mbar_wait_lim(q_full, 0, p.err, left);
      issue_s(0);
      for (int j = 0; j < n_tiles; j++) {
        const int st = j & 1;
        // S of the next tile first: its buffer held P of tile j-1, whose P V is already queued ahead of it in the pipe
        if (j + 1 < n_tiles) issue_s(j + 1);
        mbar_wait_lim(p_full, (uint32_t)j & 1u, p.err, left);  // P_j in TMEM (over S_j), O rescaled
        mbar_wait_lim(&v_full[st], (uint32_t)(j >> 1) & 1u, p.err, left);
        __syncwarp();
        tc_fence_after();
        const uint64_t vt = ft_desc_mn(v_s, FT_KV_BYTES / 2) + (uint64_t)(st * (FT_KV_BYTES >> 4));
        if (one) {
#pragma unroll
          for (int half = 0; half < 2; half++)
#pragma unroll
            for (int ks = 0; ks < FT_BN / 16; ks++) {  // keys 16ks..16ks+15 = 8 packed columns of P_hi (0..31) or P_lo (32..63)
              const uint32_t ta = tmem_base + (uint32_t)(st * 64 + half * 32 + ks * 8);
              tc_mma_f16_ts(tmem_o, ta, vt + (uint64_t)(ks * (2048 >> 4)), idesc_o, (j | half | ks) ? 1u : 0u);
            }
          tc_commit(&v_empty[st], left);
          tc_commit(o_full, left);
        }
        __syncwarp();
      }
    }
    __syncwarp();
  } else if (!busy) {
    for (int j = 0; j < n_tiles; j++) {  // (P V of tile j-1 first: an arrival for tile j must not join the barrier's previous phase)
      if (j > 0) mbar_wait_lim(o_full, (uint32_t)(j - 1) & 1u, p.err, left);
      mbar_arrive(p_full);
    }
    if (n_tiles > 0) mbar_wait_lim(o_full, (uint32_t)(n_tiles - 1) & 1u, p.err, left);
  } else if (n_tiles > 0) {
    // ===================== softmax / correction (thread = query row) ========================================
    const int qp = pos0 + t0 + tok;  // absolute position of this row's query
    for (int j = 0; j < n_tiles; j++) {
      const uint32_t tmem_sp = tmem_base + lane_addr + (uint32_t)((j & 1) * 64);
      mbar_wait_lim(&s_full[j & 1], (uint32_t)(j >> 1) & 1u, p.err, left);
      tc_fence_after();
      float sv[FT_BN];
      {
        uint32_t r[32];
        tc_ld32(tmem_sp, r);
#pragma unroll
        for (int i = 0; i < 32; i++) sv[i] = __uint_as_float(r[i]);
        tc_ld32(tmem_sp + 32u, r);
#pragma unroll
        for (int i = 0; i < 32; i++) sv[32 + i] = __uint_as_float(r[i]);
      }
      // causal mask (attention.rs:314-341) — only tiles reaching past the first row's position need the compare
      float mx = -INFINITY;
      const int k0 = (j0 + j) * FT_BN;
      if (k0 + FT_BN - 1 > pos0 + t0) {
#pragma unroll
        for (int i = 0; i < FT_BN; i++) {
          if (k0 + i > qp) sv[i] = -INFINITY;
          mx = fmaxf(mx, sv[i]);
        }
      } else {
#pragma unroll
        for (int i = 0; i < FT_BN; i++) mx = fmaxf(mx, sv[i]);
      }
      // running max with lazy update: keep the old reference while the new max exceeds it by at most tau
      float fac = 1.f;
      bool resc = false;
      if (j == 0) {
        m_run = mx;
      } else if ((mx - m_run) * p.scale_log2 > p.tau_log2) {
        fac = ft_ex2((m_run - mx) * p.scale_log2);
        m_run = mx;
        resc = true;
      }
      // p = exp((s - m) / sqrt(hd)) = 2^(s c - m c), c = log2(e) / sqrt(hd): one FFMA + one MUFU.EX2 per score; 2^-inf = 0 masks
      // (a row that has seen no key of this CTA's range yet keeps m = -inf: its scores count from 0)
      const float mc = SPLIT && m_run == -INFINITY ? 0.f : m_run * p.scale_log2;
      float rs = 0.f;
#pragma unroll
      for (int i = 0; i < FT_BN; i++) {
        const float e = ft_ex2(fmaf(sv[i], p.scale_log2, -mc));
        sv[i] = e;
        rs += e;
      }
      l_run = l_run * fac + rs;
      if (j > 0) {
        mbar_wait_lim(o_full, (uint32_t)(j - 1) & 1u, p.err, left);  // P V of the previous tile is complete: O stable
        tc_fence_after();
        if (__any_sync(0xffffffffu, resc)) {
#pragma unroll 1
          for (int c0 = 0; c0 < FT_HD; c0 += 32) {
            uint32_t r[32];
            tc_ld32(tmem_o + lane_addr + (uint32_t)c0, r);
#pragma unroll
            for (int i = 0; i < 32; i++) r[i] = __float_as_uint(__uint_as_float(r[i]) * fac);
            tc_st32(tmem_o + lane_addr + (uint32_t)c0, r);
          }
        }
      }
      // P = P_hi + P_lo, both in D, packed two keys per column over the S tile: columns 0..31 P_hi, 32..63 P_lo
      {
        uint32_t hi[32], lo[32];
#pragma unroll
        for (int i = 0; i < 32; i++) {
          const float p0 = sv[2 * i], p1 = sv[2 * i + 1];
          hi[i] = pack2x<T>(p0, p1);
          const float2 hf = DT<T>::unpack2(hi[i]);
          lo[i] = pack2x<T>(p0 - hf.x, p1 - hf.y);
        }
        tc_st32(tmem_sp, hi);
        tc_st32(tmem_sp + 32u, lo);
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(p_full);
    }
    mbar_wait_lim(o_full, (uint32_t)(n_tiles - 1) & 1u, p.err, left);  // every MMA of this CTA has completed
    tc_fence_after();
  }
  // ---- epilogue: O / l, one rounding to D (attention.rs:346), store (b, s, h, hd) ---------------------------
  T *dst = reinterpret_cast<T *>(p.y) + ((size_t)(b * S + t0 + tok) * p.n_heads + kvh * G + row - tok * G) * FT_HD;
  if (!SPLIT) {
    if (busy) {
      const float inv = 1.0f / l_run;
#pragma unroll 1
      for (int c0 = 0; c0 < FT_HD; c0 += 32) {
        uint32_t r[32];
        tc_ld32(tmem_o + lane_addr + (uint32_t)c0, r);
        if (row < rows) {
          uint32_t o[16];
#pragma unroll
          for (int i = 0; i < 16; i++) o[i] = pack2x<T>(__uint_as_float(r[2 * i]) * inv, __uint_as_float(r[2 * i + 1]) * inv);
          uint4 *d4 = reinterpret_cast<uint4 *>(dst + c0);
#pragma unroll
          for (int i = 0; i < 4; i++) d4[i] = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
        }
      }
    }
  } else {
    // merge over the cluster.  Q's place: (m, l) of every CTA, [source][row]; K's and V's: partial sums, [source][column of my share][row]
    const int sp = splits, share = FT_HD >> lg;
    float2 *ml = reinterpret_cast<float2 *>(q_s);
    float *part = reinterpret_cast<float *>(k_s);
    __syncwarp();
    cluster_arrive();  // every CTA's operands are consumed
    cluster_wait();
    if (busy) {
      const uint32_t a = smem_u32(ml + rank * FT_BM + row);
      for (int q = 0; q < sp; q++) {
        const uint32_t to = cluster_map(a, (uint32_t)q);
        st_cluster_f32(to, m_run);
        st_cluster_f32(to + 4, l_run);
      }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    float inv = 0.f;
    if (busy) {
      float M = -INFINITY, L = 0.f;
      for (int q = 0; q < sp; q++) M = fmaxf(M, ml[q * FT_BM + row].x);
      for (int q = 0; q < sp; q++) {
        const float2 v = ml[q * FT_BM + row];
        L += v.x == -INFINITY ? 0.f : v.y * ft_ex2((v.x - M) * p.scale_log2);
      }
      inv = 1.0f / L;
      const float w = m_run == -INFINITY ? 0.f : ft_ex2((m_run - M) * p.scale_log2);
      const uint32_t a = smem_u32(part + (size_t)rank * share * FT_BM + row);
#pragma unroll 1
      for (int c0 = 0; c0 < FT_HD; c0 += 16) {
        uint32_t r[16];
        if (n_tiles > 0) tc_ld16(tmem_o + lane_addr + (uint32_t)c0, r);
        const uint32_t to = cluster_map(a, (uint32_t)(c0 / share)) + (uint32_t)((c0 % share) * FT_BM * 4);  // share is a multiple of 16
#pragma unroll
        for (int i = 0; i < 16; i++) st_cluster_f32(to + (uint32_t)(i * FT_BM * 4), n_tiles > 0 ? __uint_as_float(r[i]) * w : 0.f);
      }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (busy && row < rows) {
      const float *mine = part + row;
      uint4 *d4 = reinterpret_cast<uint4 *>(dst + rank * share);
      for (int c0 = 0; c0 < share; c0 += 8) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = 0.f;
        for (int q = 0; q < sp; q++)
#pragma unroll
          for (int i = 0; i < 8; i++) v[i] += mine[(size_t)(q * share + c0 + i) * FT_BM];
        d4[c0 / 8] = make_uint4(pack2x<T>(v[0] * inv, v[1] * inv), pack2x<T>(v[2] * inv, v[3] * inv), pack2x<T>(v[4] * inv, v[5] * inv),
                                pack2x<T>(v[6] * inv, v[7] * inv));
      }
    }
  }
  if (!left) *gave_up = 1;
  tc_fence_before();
  __syncthreads();
  if (*gave_up) ft_drain(bars, warp, lane, k_loads, v_loads);
  if (warp == 5) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(FT_TMEM_COLS) : "memory");
  }
}

}  // namespace cake
