// gemm_skinny.cuh — linear layers of a few rows (single tokens, batched steps, short prompts) on tcgen05, sm_100a.
//
//   C[M,N] = epilogue( A[M,K] · W[N,K]^T )      same operator, epilogues and rounding points as gemm_tc.cuh
//
// Bound: the stream of W out of HBM (2 N K bytes; A and C are a few hundred KB).  gemm_tc_kernel gives a product of at most 128
// rows N / 128 CTAs, each with one 128 x 64 slice of W in flight per k-block: 32 CTAs for a 4096-wide output pull 1.7 TB/s.
// Here
//   * W is the MMA's 128-row operand and the rows of A are its columns (16 .. 256 of them, as many as there are, rounded up to 16),
//     so that a stage carries 16 KB of W and little else, and a product of up to 256 rows reads W once;
//   * a 128-row slice of W is cut along K between the S CTAs of a cluster, which brings the grid up to the chip; the S fp32 partial
//     sums meet in shared memory over the cluster (every CTA finishes nt / S of the rows, sums in rank order: deterministic).  A CTA lays its
//     sums down in its own shared memory and sends each other CTA's rows there as one bulk copy, counted on a barrier of the receiver:
//     with a store per sum between two cluster barriers the exchange was 2.1 us of a kernel's 5.1 (37 rows of 1024 x 1024, eight CTAs);
//   * the first ring of W is requested before griddepcontrol.wait: weights don't depend on the kernel in front.
// One CTA = one slice, 192 threads: warp 0 TMA producer, warp 1 MMA issuer and TMEM owner, warps 2-5 epilogue (thread = row of W).
#pragma once
#include "gemm_tc.cuh"

namespace cake {

constexpr int SK_BM = 128, SK_THREADS = 192, SK_MAX_SPLIT = 8, SK_MAX_STAGES = 8;
constexpr int SK_MAX_ROWS = 256, SK_SMEM_MAX = 220 * 1024;
constexpr int SK_W_BYTES = SK_BM * TC_BK * 2;  // 16 KB of W per stage
__host__ __device__ inline int sk_stage_bytes(int nt) { return SK_W_BYTES + nt * TC_BK * 2; }
// Shared memory: the ring; over it, when it has been read, a CTA's own sums [nt][128]; and the sums it receives, [split - 1][nt / split][128], behind
// the ring (SK_APART: peers may send as soon as they like) or over it, behind the own sums (SK_OVER).  SK_LEAN, 256 rows cut in four: the share that
// a CTA keeps stays in tensor memory until the last pass fetches it 16 rows at a time, as an uncut slice's rows.
enum { SK_OVER = 0, SK_APART = 1, SK_LEAN = 2 };
__host__ __device__ inline int sk_sums_floats(int nt, int split, int how) { return (how == SK_LEAN ? nt / split * (split - 1) : nt) * SK_BM; }
__host__ __device__ inline int sk_recv_at(int nt, int stages, int split, int how) {  // in floats
  const int ring = stages * sk_stage_bytes(nt) / 4, sums = sk_sums_floats(nt, split, how);
  return how == SK_APART && ring > sums ? ring : sums;
}
__host__ inline size_t sk_smem_bytes(int nt, int stages, int split, int how) {
  size_t bytes = (size_t)stages * sk_stage_bytes(nt);
  if (split > 1) {
    const size_t end = ((size_t)sk_recv_at(nt, stages, split, how) + (size_t)nt / split * (split - 1) * SK_BM + (how == SK_LEAN ? 16 * SK_BM : 0)) * 4;
    if (bytes < end) bytes = end;
  }
  return bytes + 1024 /*align*/ + 256;
}

struct SkParams {
  const void *bias, *residual;
  void *C;
  int M, N, K, act, ldc;
  float cap;
  const int *tile_group;     // as TcParams: rows sorted by group in blocks of TC_BM; a block's first `rows` rows are all it uses
  const float *row_scale;
  int nt, rows;              // rows of A per tile: as columns of the MMA (a multiple of 16), and those of them that are there
  int a_shared;              // every row block multiplies the same rows of A, the first ones
  int m_tiles;               // row tiles, TC_BM rows apart
  int split, stages;
  int how;                   // SK_OVER, SK_APART or SK_LEAN
  int *err;                  // host-mapped: a wait that ran out
  int tries;                 // 0, or (a test's) what a thread's waits may spend instead of MBAR_TRIES; those of a cluster's first CTA nothing
};

// What an epilogue reads beside the sums, four columns of row m of A from column n on (nothing where the row is not `in`)
template <typename T, int EPI, bool VEC> struct SkRes {
  static constexpr int WORDS = EPI == TCE_RESIDUAL_F32 ? 4 : EPI == TCE_RESIDUAL ? 2 : 1;
  uint32_t w[WORDS];
  __device__ __forceinline__ void load(const SkParams &p, bool in, int m, int n) {
    if (!in) return;
    if (EPI == TCE_RESIDUAL) {
      const uint16_t *src = reinterpret_cast<const uint16_t *>(p.residual) + (size_t)m * (p.ldc ? p.ldc : p.N) + n;
      const uint2 v = VEC ? *reinterpret_cast<const uint2 *>(src) : make_uint2(src[0] | (uint32_t)src[1] << 16, src[2] | (uint32_t)src[3] << 16);
      w[0] = v.x; w[WORDS > 1 ? 1 : 0] = v.y;
    } else if (EPI == TCE_RESIDUAL_F32) {
      const uint32_t *src = reinterpret_cast<const uint32_t *>(p.residual) + (size_t)m * p.N + n;
      const uint4 v = VEC ? *reinterpret_cast<const uint4 *>(src) : make_uint4(src[0], src[1], src[2], src[3]);
      w[0] = v.x; w[WORDS > 1 ? 1 : 0] = v.y; w[WORDS > 2 ? 2 : 0] = v.z; w[WORDS > 3 ? 3 : 0] = v.w;
    }
  }
};
// the sums of row m, columns n .. n + 3 -> C
template <typename T, int EPI, bool VEC>
__device__ __forceinline__ void sk_store(const SkParams &p, int m, int n, const float (&v)[4], const float (&bias)[4], const SkRes<T, EPI, VEC> &res) {
  if (EPI == TCE_SOFTCAP_F32 || EPI == TCE_RESIDUAL_F32) {
    float *dst = reinterpret_cast<float *>(p.C) + (size_t)m * p.N + n;
    const float rs = EPI == TCE_RESIDUAL_F32 && p.row_scale ? p.row_scale[m] : 1.0f;
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (EPI == TCE_RESIDUAL_F32) o[j] = fmaf(rs, v[j], __uint_as_float(res.w[j % SkRes<T, EPI, VEC>::WORDS]));
      else o[j] = p.cap > 0.f ? p.cap * tanhf(v[j] / p.cap) : v[j];
    }
    if (VEC) *reinterpret_cast<float4 *>(dst) = make_float4(o[0], o[1], o[2], o[3]);
    else { dst[0] = o[0]; dst[1] = o[1]; dst[2] = o[2]; dst[3] = o[3]; }
  } else if (EPI == TCE_SWIGLU) {  // columns 2i and 2i + 1 are gate and up
    T *dst = reinterpret_cast<T *>(p.C) + (size_t)m * (p.ldc ? p.ldc : p.N / 2) + n / 2;
    const uint32_t u = pack2x<T>(gated_pair<T>(v[0], v[1], p.act, p.cap), gated_pair<T>(v[2], v[3], p.act, p.cap));
    if (VEC) *reinterpret_cast<uint32_t *>(dst) = u;
    else { reinterpret_cast<uint16_t *>(dst)[0] = (uint16_t)u; reinterpret_cast<uint16_t *>(dst)[1] = (uint16_t)(u >> 16); }
  } else {
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      o[j] = EPI == TCE_ACT ? plain_act<T>(v[j], p.act) : rnd<T>(v[j]);
      if (EPI == TCE_PLAIN && p.bias) o[j] = rnd<T>(o[j] + bias[j]);
      if (EPI == TCE_RESIDUAL) {
        const float2 r2 = DT<T>::unpack2(res.w[(j / 2) % SkRes<T, EPI, VEC>::WORDS]);
        o[j] += j & 1 ? r2.y : r2.x;
      }
    }
    T *dst = reinterpret_cast<T *>(p.C) + (size_t)m * (p.ldc ? p.ldc : p.N) + n;
    const uint2 u = make_uint2(pack2x<T>(o[0], o[1]), pack2x<T>(o[2], o[3]));
    if (VEC) *reinterpret_cast<uint2 *>(dst) = u;
    else {
      uint16_t *d16 = reinterpret_cast<uint16_t *>(dst);
      d16[0] = (uint16_t)u.x; d16[1] = (uint16_t)(u.x >> 16); d16[2] = (uint16_t)u.y; d16[3] = (uint16_t)(u.y >> 16);
    }
  }
}

// VEC: C and the residual take accesses of four columns (their addresses and row strides); an instance of its own for what does not, since a kernel of
// a few microseconds pays for instructions on its way that it does not run
template <typename T, int EPI, bool VEC>
__device__ __forceinline__ void sk_product(const CUtensorMap &map_w, const CUtensorMap &map_a, const SkParams &p, const int block) {
  extern __shared__ unsigned char smem_raw_sk[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw_sk) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[SK_MAX_STAGES], empty[SK_MAX_STAGES], acc_full, drained, got;
  __shared__ uint32_t tmem_ptr;
  __shared__ int gave_up;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.split, nt = p.nt, stage_bytes = sk_stage_bytes(nt);
  const int unit = block / S, rank = block % S;  // the cluster's CTAs are neighbours along x
  const int mt = unit % p.m_tiles, n0 = (unit / p.m_tiles) * SK_BM;
  const int m0 = mt * TC_BM, m_end = min(p.M, m0 + p.rows), a0 = p.a_shared ? 0 : m0;
  const int kblocks = p.K / TC_BK, kb0 = (int)((long)kblocks * rank / S), kb1 = (int)((long)kblocks * (rank + 1) / S), nkb = kb1 - kb0;
  uint32_t cols = 32;
  while ((int)cols < nt) cols <<= 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(&acc_full, 1);
    mbar_init(&drained, 1);
    mbar_init(&got, 1);
    gave_up = 0;
    mbar_fence_init();
    if (S > 1) mbar_arrive_expect_tx(&got, (uint32_t)(nt / S * (S - 1) * SK_BM * 4));
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_ptr)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();
  if (S > 1 && p.how == SK_APART) cluster_arrive_relaxed();  // this CTA's barrier exists (mbar_fence_init) and its place for sums is free
  const uint32_t tmem = tmem_ptr;

  int group = 0;
  if (p.tile_group) {  // written by an earlier kernel: nothing can be requested before it has ended
    pdl_wait();
    group = p.tile_group[mt];
  }
  const bool live = group >= 0;  // cluster-uniform
  int issued = 0;                // warp 0: stages requested
  int left = !p.tries ? MBAR_TRIES : rank ? p.tries : 0;  // of this thread's waits

  if (warp == 0) {
    if (lane == 0 && live) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
      const int wrow = n0 + group * p.N;
      const int pre = min(nkb, p.stages);
      for (int i = 0; i < pre; i++) {
        mbar_arrive_expect_tx(&full[i], (uint32_t)stage_bytes);
        tma_load_2d(smem + (size_t)i * stage_bytes, &map_w, (kb0 + i) * TC_BK, wrow, &full[i]);
      }
      if (!p.tile_group) pdl_wait();
      for (int i = 0; i < pre; i++) tma_load_2d(smem + (size_t)i * stage_bytes + SK_W_BYTES, &map_a, (kb0 + i) * TC_BK, a0, &full[i]);
      int s = 0;
      uint32_t ph = 0;
      issued = pre;
#pragma unroll 1  // a CTA comes round here a few times: straight-line code only waits for its own instructions (prompt of 37 tokens 430 -> 424 us)
      for (int i = pre; i < nkb; i++) {
        mbar_wait_lim(&empty[s], ph, p.err, left);
        unsigned char *st = smem + (size_t)s * stage_bytes;
        mbar_arrive_expect_tx_if(left, &full[s], (uint32_t)stage_bytes);
        tma_load_2d(st, &map_w, (kb0 + i) * TC_BK, wrow, &full[s], left);
        tma_load_2d(st + SK_W_BYTES, &map_a, (kb0 + i) * TC_BK, a0, &full[s], left);
        issued += left ? 1 : 0;
        if (++s == p.stages) { s = 0; ph ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (!p.tile_group) pdl_wait();  // (also keeps the bounded waits from counting the kernel in front)
    if (live) {
      const uint32_t idesc = tc_idesc<T>(nt), one = elect_one();
      const uint64_t dw0 = tc_smem_desc(smem), da0 = tc_smem_desc(smem + SK_W_BYTES);
      int s = 0;
      uint32_t ph = 0;
#pragma unroll 1
      for (int i = 0; i < nkb; i++) {
        mbar_wait_lim(&full[s], ph, p.err, left);
        __syncwarp();  // every lane has seen this phase before one of them begins what completes the next
        tc_fence_after();
        const uint64_t dw = dw0 + (uint64_t)(s * (stage_bytes >> 4)), da = da0 + (uint64_t)(s * (stage_bytes >> 4));
        if (one) {
#pragma unroll
          for (int k = 0; k < TC_BK / 16; k++) tc_mma_f16(tmem, dw + (uint64_t)(k * 2), da + (uint64_t)(k * 2), idesc, (i | k) ? 1u : 0u);
          tc_commit(&empty[s], left);
        }
        __syncwarp();
        if (++s == p.stages) { s = 0; ph ^= 1u; }
      }
      if (one) tc_commit(&acc_full, left);
    }
    __syncwarp();
  }
  if (!p.tile_group && warp > 1) pdl_wait();  // the residual, and C's previous readers, belong to the kernels in front
  const int wq = warp & 3;
  const uint32_t trow = tmem + ((uint32_t)(wq * 32) << 16);
  const int share = nt / S, f0 = m0 + rank * share;  // rows this CTA finishes: all of the tile, or its share of them
  float *sums = reinterpret_cast<float *>(smem);     // this CTA's sums, over its drained ring: [row of A][128 columns]
  const int recv = sk_recv_at(nt, p.stages, S, p.how);  // the others', from here on: [rank but this][row within the share][128 columns]
  bool go = warp >= 2 && live;                       // warps that finish rows
  // A warp finishes its 32 columns four rows at a time, a lane four columns of one row: loads and stores of 8 bytes (16 of fp32), and the
  // residual of four passes is on its way.  (A thread per column took a pair of rows at a time, each behind its residual's way from L2: 0.1
  // us a row, 35.9 us for N = K = 4096, 200 rows.  Eight columns a lane: the gated form's code is twice as long, and a step of one row,
  // which runs it once, waits for it: 187 -> 189 us for four Nigenex layers.)
  const int fr = lane >> 3, fc = wq * 32 + (lane & 7) * 4, fn = n0 + fc;
  float bias[4] = {0.f, 0.f, 0.f, 0.f};
  SkRes<T, EPI, VEC> res[4];
  if (go) {
    if (EPI == TCE_PLAIN && p.bias) {
#pragma unroll
      for (int j = 0; j < 4; j++) bias[j] = DT<T>::to_f(reinterpret_cast<const T *>(p.bias)[fn + j]);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) res[i].load(p, fr + 4 * i < share && f0 + fr + 4 * i < m_end, f0 + fr + 4 * i, fn);
    mbar_wait_lim(&acc_full, 0, p.err, left);
    go = __all_sync(0xffffffffu, left != 0);
    tc_fence_after();
  }
  if (S > 1) {
    __syncwarp();
    if (p.how != SK_APART) cluster_arrive();  // this CTA's ring is drained: its MMAs have read all that was loaded
    if (warp >= 2) {
      if (go) {
#pragma unroll 1
        for (int c0 = 0; c0 < nt; c0 += 32) {  // (the accumulator has a power of two of columns, 32 at least)
          uint32_t r[32];
          float *dst = sums + (size_t)c0 * SK_BM + wq * 32 + lane;
          if (p.how == SK_LEAN) {
            if (c0 / share == rank) continue;
            if (c0 / share > rank) dst -= share * SK_BM;
          }
          tc_ld32(trow + (uint32_t)c0, r);
#pragma unroll
          for (int j = 0; j < 16; j++) dst[j * SK_BM] = __uint_as_float(r[j]);
          if (c0 + 16 < nt)
#pragma unroll
            for (int j = 16; j < 32; j++) dst[j * SK_BM] = __uint_as_float(r[j]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      } else if (live) gave_up = 1;
      __syncwarp();
      cluster_wait();
      named_bar_sync(1, SK_THREADS - 64);
      if (warp == 2 && lane < S - 1 && live && !*(volatile int *)&gave_up) {  // a lane per receiver, every CTA beginning with another one
        const int to = (rank + 1 + lane) & (S - 1);
        const uint32_t bytes = (uint32_t)(share * SK_BM * 4), slot = (uint32_t)(rank - (rank > to)) * bytes;
        bulk_s2s(cluster_map(smem_u32(sums + recv) + slot, (uint32_t)to), smem_u32(sums) + (uint32_t)(to - (p.how == SK_LEAN && to > rank)) * bytes, bytes, cluster_map(smem_u32(&got), (uint32_t)to));
      }
      __syncwarp();
      if (go) {
        mbar_wait_lim(&got, 0, p.err, left);
        go = __all_sync(0xffffffffu, left != 0);
      }
      if (!go && live) mbar_drain(&got, 0);  // gave up: what peers have sent all the same lands before anybody leaves
      cluster_arrive_relaxed();  // (waited for at the end: nobody leaves while sums are on their way)
    } else {
      cluster_wait();
      cluster_arrive_relaxed();
    }
  }
  // The last pass is a loop, not straight-line code: a kernel of a few microseconds runs its epilogue once, and unrolled over 16 rows it
  // waited for its own instructions (233 -> 315 us for four Nigenex layers).  A row's residual is read by the lane that stores it, before
  // it does: C may be the residual's own buffer.
  if (go) {
    const bool kept = S == 1 || p.how == SK_LEAN;  // own rows are still in tensor memory
    const int own16 = S == 1 ? 0 : recv + (S - 1) * share * SK_BM;
#pragma unroll 1
    for (int c0 = 0; c0 < share && f0 + c0 < m_end; c0 += 4) {
      if (kept && !(c0 & 12)) {  // through shared memory too: the warp's own columns, 16 rows at a time
        uint32_t r[16];
        tc_ld16(trow + (uint32_t)(rank * share + c0), r);
        float *mine = sums + own16 + wq * 32 + lane;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 16; j++) mine[j * SK_BM] = __uint_as_float(r[j]);
        __syncwarp();
      }
      const int m = f0 + c0 + fr;
      SkRes<T, EPI, VEC> ahead;
      ahead.load(p, c0 + fr + 16 < share && m + 16 < m_end, m + 16, fn);
      if (c0 + fr < share && m < m_end) {
        const int at = (c0 + fr) * SK_BM + fc, stride = share * SK_BM, own = kept ? own16 + ((c0 & 12) + fr) * SK_BM + fc : at + rank * stride;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
        for (int q = 0; q < S; q++) {  // in rank order
          const int off = q == rank ? own : recv + at + (q - (q > rank)) * stride;
          const float4 x = *reinterpret_cast<const float4 *>(sums + off);
          v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
        }
        sk_store<T, EPI, VEC>(p, m, fn, v, bias, res[0]);
      }
      res[0] = res[1]; res[1] = res[2]; res[2] = res[3];
      res[3] = ahead;
    }
  }
  if (!left) gave_up = 1;
  tc_fence_before();
  __syncthreads();
  if (gave_up) {
    if (threadIdx.x == 0)
      for (int i = max(0, issued - p.stages); i < issued; i++) mbar_drain(&full[i % p.stages], (uint32_t)(i / p.stages) & 1u);
    if (warp == 1 && elect_one()) {
      tc_commit(&drained);
      mbar_drain(&drained, 0);
    }
    __syncthreads();
  }
  if (S > 1) cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
  }
}

template <typename T, int EPI, bool VEC>
__global__ void __launch_bounds__(SK_THREADS, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const SkParams p) {
  sk_product<T, EPI, VEC>(map_w, map_a, p, (int)blockIdx.x);
}
// Two products side by side, the clusters from first_ctas on work on the second: a routed feed-forward's experts and its shared expert, or a block's
// attention projections and the input half of its feed-forward, which alone are too short to come up to speed.  Both are cut into clusters of the same size.
template <typename T, int EPI, int EPI2>
__global__ void __launch_bounds__(SK_THREADS, 2)
gemm_skinny_two_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w2,
                       const __grid_constant__ CUtensorMap map_a2, const SkParams p, const SkParams p2, const int first_ctas) {
  const bool second = (int)blockIdx.x >= first_ctas;
  if (EPI == EPI2) {
    const SkParams q = second ? p2 : p;
    sk_product<T, EPI, true>(second ? map_w2 : map_w, second ? map_a2 : map_a, q, (int)blockIdx.x - (second ? first_ctas : 0));
  } else if (second) {
    sk_product<T, EPI2, true>(map_w2, map_a2, p2, (int)blockIdx.x - first_ctas);
  } else {
    sk_product<T, EPI, true>(map_w, map_a, p, (int)blockIdx.x);
  }
}

}  // namespace cake
