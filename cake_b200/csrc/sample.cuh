// sample.cuh — device-side token samplers: the tail of TextModelBase::next_token
// (text_model.rs:102-118 create_logits_processor, :429-460 the sampling step) without shipping the logits to the
// host: one cluster of SAMPLE_CTAS CTAs reads the (vocab,) logits of the last position from L2/HBM and writes 4 bytes.
//
// The arithmetic behind `LogitsProcessor::sample` lives in candle-transformers 0.9.2 (generation/mod.rs) and
// candle-nn 0.9.2 (sampling.rs), crates that are not vendored with the reference; restated from their published
// algorithm (oracle/sampling.py holds the CPU restatement the tests compare with):
//   all kinds        logits -> f32
//   GumbelSoftmax    argmax(logits + T * g),  g = -log(-log(u)),  u ~ U(1e-7, 0.999)      (candle_nn::sampling)
//   All / TopK / TopP / TopKThenTopP:
//                    prs = softmax(logits * (1/T))  (max-subtracted, f32), then
//     All            multinomial(prs)                         (rand WeightedIndex: first i with cumsum_i > x*total)
//     TopK{k}        the k most probable tokens, multinomial over them
//     TopP{p}        sort descending, keep tokens while the running sum before them is < p, multinomial over the
//                    kept probabilities in VOCABULARY order (the others zeroed)       (p <= 0 or >= 1: All)
//     TopKThenTopP   top-k, then the nucleus rule inside those k
// What cannot be pinned: (1) the random stream — candle draws from rand::StdRng / the device RNG, here a counter-based
// Philox4x32-10 keyed by (seed, step); tests supply the uniforms instead (`noise`); (2) candle's TopK builds its
// candidate list with select_nth_unstable, whose ORDER is unspecified, so which token a given uniform selects is
// implementation-defined there; here the candidates are ordered by probability (descending, ties by lower id).
// Everything is deterministic: reductions and scans use fixed trees, never floating-point atomics.
#pragma once
#include "common.cuh"

namespace cake {

enum SampleKind { SAMPLE_ARGMAX = 0, SAMPLE_ALL = 1, SAMPLE_TOPK = 2, SAMPLE_TOPP = 3, SAMPLE_TOPK_TOPP = 4, SAMPLE_GUMBEL = 5 };
constexpr int SAMPLE_THREADS = 1024, SAMPLE_CTAS = 8;
constexpr int SAMPLE_SMEM_MAX = 208 * 1024;  // logits and probabilities of a CTA's part of the vocabulary; those of a larger part stay in global memory
__host__ __device__ inline int sample_per_thread(int V) { return ((V + SAMPLE_CTAS * SAMPLE_THREADS - 1) / (SAMPLE_CTAS * SAMPLE_THREADS)) | 1; }
__host__ inline size_t sample_smem(int V) { return (size_t)sample_per_thread(V) * SAMPLE_THREADS * 6; }  // odd: a thread's run of entries has no bank conflicts
constexpr int SAMPLE_MAX_K = 1024;   // candidates sorted in shared memory (top-k requests above this are refused by the host)

struct SampleArgs {
  int kind, top_k;
  float temperature, top_p;
  unsigned long long seed;
};

// ---- Philox4x32-10 (counter-based; Salmon et al. 2011) ------------------------------------------------------------
__device__ __forceinline__ uint4 philox4x32(uint4 ctr, uint2 key) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
    const unsigned long long p0 = (unsigned long long)0xD2511F53u * ctr.x, p1 = (unsigned long long)0xCD9E8D57u * ctr.z;
    ctr = make_uint4((uint32_t)(p1 >> 32) ^ ctr.y ^ key.x, (uint32_t)p1, (uint32_t)(p0 >> 32) ^ ctr.w ^ key.y, (uint32_t)p0);
    key.x += 0x9E3779B9u;
    key.y += 0xBB67AE85u;
  }
  return ctr;
}
__device__ __forceinline__ float u01(uint32_t r) { return (float)(r >> 8) * (1.0f / 16777216.0f); }  // [0, 1)
// uniform for vocabulary entry v (Gumbel) / the single draw of a step (v = 0xffffffff)
__device__ __forceinline__ float sample_uniform(const SampleArgs &s, unsigned step, unsigned v) {
  const uint4 r = philox4x32(make_uint4(v >> 2, step, 0x5a4d504cu, 0u), make_uint2((uint32_t)s.seed, (uint32_t)(s.seed >> 32)));
  const uint32_t w = (v & 3) == 0 ? r.x : (v & 3) == 1 ? r.y : (v & 3) == 2 ? r.z : r.w;
  return u01(w);
}

// Bound: latency, not bytes (300 KB of logits): one CTA took 31 bisection passes of 125 dependent loads each over the vocabulary, 380 us for
// 128256 entries.  The vocabulary is cut between the CTAs of a cluster, which keep their probabilities in shared memory; a pass looks
// at seven thresholds at once and its sums meet over the cluster; the thresholds are logits, whose 16 bits take six passes (a
// probability's 30 bits took ten: 97 us).  A nucleus is searched between the largest logit and where it can end (see sample_threshold), entries below a
// pass's lowest threshold are passed over, and the logits are read 16 bytes at a time: the call 95 -> 77 us at 128256 bf16 entries, three passes.
// Every reduction has a fixed order (threads, warps, ranks): a draw is a function of (logits, seed, step).
struct SampleShared {
  float warp[SAMPLE_THREADS / 32][9];    // a warp's sums (rows of nine: no bank conflicts down a column)
  float slot[2][SAMPLE_CTAS][8];         // the CTAs' sums, written by the peers; two sets in turn
  float scan[2][SAMPLE_THREADS / 32 + 1];
  float c_p[SAMPLE_MAX_K];
  int c_i[SAMPLE_MAX_K];
};

struct SampleCluster {
  SampleShared &sh;
  int rank, set = 0;
  // v[0..N) of every thread of the cluster, combined with `op` in a fixed order
  template <int N, typename Op> __device__ __forceinline__ void reduce(float (&v)[N], float neutral, Op op) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int t = 0; t < N; t++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[t] = op(v[t], __shfl_xor_sync(0xffffffffu, v[t], o));
      if (lane == 0) sh.warp[warp][t] = v[t];
    }
    __syncthreads();
    if (warp < N) {  // one warp per sum
      float x = sh.warp[lane][warp];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x = op(x, __shfl_xor_sync(0xffffffffu, x, o));
      if (lane < SAMPLE_CTAS) st_cluster_f32(cluster_map(smem_u32(&sh.slot[set][rank][warp]), (uint32_t)lane), x);
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
#pragma unroll
    for (int t = 0; t < N; t++) {
      v[t] = neutral;
#pragma unroll
      for (int r = 0; r < SAMPLE_CTAS; r++) v[t] = op(v[t], sh.slot[set][r][t]);
    }
    set ^= 1;
  }
  template <int N> __device__ __forceinline__ void sum(float (&v)[N]) {
    reduce<N>(v, 0.f, [](float a, float b) { return a + b; });
  }
  __device__ __forceinline__ float max1(float x) {
    float v[1] = {x};
    reduce<1>(v, -INFINITY, [](float a, float b) { return fmaxf(a, b); });
    return v[0];
  }
  __device__ __forceinline__ float sum1(float x) {
    float v[1] = {x};
    sum<1>(v);
    return v[0];
  }
  __device__ __forceinline__ int min_i(int x) {  // (vocabulary indices and 0x7fffffff compare as floats' bit patterns do)
    float v[1] = {__int_as_float(x)};
    reduce<1>(v, __int_as_float(0x7fffffff), [](float a, float b) { return __int_as_float(min(__float_as_int(a), __float_as_int(b))); });
    return __float_as_int(v[0]);
  }
  // exclusive prefix over the cluster's threads in vocabulary order, and the total
  __device__ __forceinline__ float scan(float x, float &total) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    float *ws = sh.scan[set];
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    if (tid < 32) {
      const float wt = ws[tid];
      float winc = wt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, winc, o);
        if (tid >= o) winc += t;
      }
      ws[tid] = winc - wt;
      if (tid == 31) ws[32] = winc;
    }
    __syncthreads();
    const float mine = ws[warp] + (inc - x);
    if (tid < SAMPLE_CTAS) st_cluster_f32(cluster_map(smem_u32(&sh.slot[set][rank][0]), (uint32_t)tid), ws[32]);
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    float before = 0.f;
    total = 0.f;
#pragma unroll
    for (int r = 0; r < SAMPLE_CTAS; r++) {
      if (r == rank) before = total;
      total += sh.slot[set][r][0];
    }
    set ^= 1;
    return before + mine;
  }
};

// 16-bit floats in rising order as 0 .. 65535, and back
template <typename T> __device__ __forceinline__ uint32_t sample_key(float x) {
  const T d = DT<T>::from_f(x);
  const uint32_t h = *reinterpret_cast<const uint16_t *>(&d);
  return h & 0x8000u ? ~h & 0xffffu : h | 0x8000u;
}
template <typename T> __device__ __forceinline__ float sample_unkey(uint32_t k) {
  const uint16_t h = (uint16_t)(k & 0x8000u ? k & 0x7fffu : ~k);
  return DT<T>::to_f(*reinterpret_cast<const T *>(&h));
}
// The largest logit at which the entries that are at least as large still reach `want`, in number (COUNT) or in probability: with tau its
// probability, reach(P >= tau) >= want > reach(P > tau), as probabilities rise with logits.  Seven thresholds a pass, log8 of the patterns from `from` to
// `to`, between which it lies, passes.  All 65536 are six.  From the largest logit to where a nucleus can end, both above zero, there are a few hundred in
// bf16 (128 an octave: three passes) and a few thousand in f16 (1024 an octave: four); where the end lies below zero, the range holds every small
// exponent, some 33000 patterns: five passes, or six.
template <typename T, bool COUNT>
__device__ __forceinline__ float sample_threshold(SampleCluster &cl, const T *L, const float *P, int i0, int i1, float want, float from, float to) {
  uint32_t lo = sample_key<T>(from), hi = sample_key<T>(to) + 1u;
  while (hi - lo > 1u) {
    const uint32_t step = max(1u, (hi - lo) / 8u);
    float m[7], th[7];
#pragma unroll
    for (int t = 0; t < 7; t++) {
      m[t] = 0.f;
      th[t] = sample_unkey<T>(min(hi - 1u, lo + (uint32_t)(t + 1) * step));
    }
    for (int i = i0; i < i1; i++) {
      const float x = DT<T>::to_f(L[i]);
      if (!(x >= th[0])) continue;   // (most entries are below the lowest threshold)
      const float v = COUNT ? 1.f : P[i];
#pragma unroll
      for (int t = 0; t < 7; t++) m[t] += x >= th[t] ? v : 0.f;
    }
    cl.sum<7>(m);
    int best = 0;
#pragma unroll
    for (int t = 0; t < 7; t++)
      if (lo + (uint32_t)(t + 1) * step < hi && m[t] >= want && best == t) best = t + 1;  // reach() falls as the threshold rises
    const uint32_t next = lo + (uint32_t)(best + 1) * step;
    lo += (uint32_t)best * step;
    if (best < 7 && next < hi) hi = next;
  }
  return sample_unkey<T>(lo);
}

// `noise`: nullable; tests pass the uniforms explicitly — vocab floats in [0,1) for Gumbel, one float otherwise.
// P: scratch of V floats, used when a CTA's part of the vocabulary is larger than its shared memory (in_smem == 0).
template <typename T>
__global__ void __cluster_dims__(SAMPLE_CTAS, 1, 1) __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const T *__restrict__ logits, int V, SampleArgs s, float *P_global, int in_smem, const float *__restrict__ noise, const int *d_step,
              int step_bias, uint32_t *token_out, uint32_t *ring, int ring_cap) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ float sample_smem_p[];
  __shared__ SampleShared sh;
  const int tid = threadIdx.x, per = sample_per_thread(V);
  SampleCluster cl{sh, (int)cluster_rank()};
  const int base = (int)min((long)V, (long)cl.rank * per * SAMPLE_THREADS);
  const int n = (int)min((long)V - base, (long)per * SAMPLE_THREADS);  // this CTA's entries: [base, base + n)
  const T *lg = logits + base;
  const unsigned step = (unsigned)((d_step ? *d_step : 0) + step_bias);
  auto finish = [&](int tok) {
    if (cl.rank == 0 && tid == 0) {
      *token_out = (uint32_t)tok;
      if (ring) ring[step % (unsigned)ring_cap] = (uint32_t)tok;
    }
  };
  cluster_arrive();  // every CTA runs before the first store to a peer
  cluster_wait();

  if (s.kind == SAMPLE_ARGMAX || s.temperature <= 0.f || s.kind == SAMPLE_GUMBEL) {  // first maximum wins
    // candle_nn::sampling::gumbel_softmax: minus_g = log(-log(u)), u in [1e-7, 0.999); T == 1: logits - minus_g, else
    // logits + minus_g * (-T); argmax
    const bool gumbel = s.kind == SAMPLE_GUMBEL && s.temperature > 0.f;
    float best = -INFINITY;
    int idx = 0x7fffffff;
    for (int i = tid; i < n; i += SAMPLE_THREADS) {
      float v = DT<T>::to_f(lg[i]);
      if (gumbel) {
        const float r = noise ? noise[base + i] : sample_uniform(s, step, (unsigned)(base + i));
        const float u = 1e-7f + r * (0.999f - 1e-7f);
        const float minus_g = logf(-logf(u));
        v = (s.temperature == 1.0f) ? v - minus_g : v + minus_g * (-s.temperature);
      }
      if (v > best) { best = v; idx = base + i; }
    }
    const float bm = cl.max1(best);
    finish(cl.min_i(best == bm ? idx : 0x7fffffff));
    return;
  }

  // ---- prs = softmax(logits * (1/T)) in f32 ------------------------------------------------------------------
  float *P = in_smem ? sample_smem_p : P_global + base;
  const T *L = lg;
  const float inv_t = (float)(1.0 / (double)s.temperature);
  float top = -INFINITY;   // the largest logit (times 1/T rises with it)
  T *keep = reinterpret_cast<T *>(sample_smem_p + (size_t)per * SAMPLE_THREADS);
  if (in_smem && ((uintptr_t)lg & 15) == 0) {   // 16 bytes a load: one or two round trips to L2 for a thread's entries
#pragma unroll 3
    for (int i = tid * 8; i + 8 <= n; i += SAMPLE_THREADS * 8) {
      const uint4 v = *reinterpret_cast<const uint4 *>(lg + i);
      *reinterpret_cast<uint4 *>(keep + i) = v;
      float f[8];
      unpack8<T>(v, f);
#pragma unroll
      for (int e = 0; e < 8; e++) top = fmaxf(top, f[e]);
    }
    for (int e = (n & ~7) + tid; e < n; e += SAMPLE_THREADS) {
      keep[e] = lg[e];
      top = fmaxf(top, DT<T>::to_f(lg[e]));
    }
  } else {
#pragma unroll 4
    for (int i = tid; i < n; i += SAMPLE_THREADS) {
      const T x = lg[i];
      if (in_smem) keep[i] = x;
      top = fmaxf(top, DT<T>::to_f(x));
    }
  }
  if (in_smem) L = keep;
  top = cl.max1(top);   // (its barriers order the copies, of other entries than a thread reads below)
  const float mx = __fmul_rn(top, inv_t);
  auto weight = [&](T x) { return expf(__fsub_rn(__fmul_rn(DT<T>::to_f(x), inv_t), mx)); };  // (no contraction: a threshold's own has the same bits)
  float sum = 0.f;
  for (int i = tid; i < n; i += SAMPLE_THREADS) {
    const float e = weight(L[i]);
    P[i] = e;
    sum += e;
  }
  sum = cl.sum1(sum);
  for (int i = tid; i < n; i += SAMPLE_THREADS) P[i] = P[i] / sum;
  __syncthreads();
  const float u = noise ? noise[0] : sample_uniform(s, step, 0xffffffffu);
  const int i0 = min(n, tid * per), i1 = min(n, i0 + per);  // this thread's run of entries

  const bool want_k = (s.kind == SAMPLE_TOPK || s.kind == SAMPLE_TOPK_TOPP) && s.top_k < V;
  const bool want_p = (s.kind == SAMPLE_TOPP || s.kind == SAMPLE_TOPK_TOPP) && s.top_p > 0.f && s.top_p < 1.f;
  if (!want_k) {
    // All (also TopK with k >= vocab, TopP with p outside (0,1)): every entry.  TopP: those above the probability tau at which the running
    // sum in falling order crosses p, and the first ties at tau until the sum before one reaches p.  Drawn in vocabulary order.
    uint32_t tau = 0u;
    float eq_before = 0.f;
    int need = 0x7fffffff;
    if (want_p) {
      // Entries more than d below the largest one have less than V e^(-d / T) / sum of the probability together, which is at most half of 1 - p (sum >= 1):
      // the nucleus ends above them.  A p within 1e-3 of 1, where the roundings of the sums come near 1 - p, and logits that are not finite search all.
      const float d = logf(2.f * (float)V / (1.f - s.top_p)) * s.temperature;
      const bool near = s.top_p < 0.999f && top - d > -INFINITY && top < INFINITY;
      tau = __float_as_uint(weight(DT<T>::from_f(sample_threshold<T, false>(cl, L, P, i0, i1, s.top_p, near ? top - d : -INFINITY, near ? top : INFINITY))) / sum);
      float m[1] = {0.f}, eq = 0.f, n_eq;
      for (int i = i0; i < i1; i++) {
        const uint32_t b = __float_as_uint(P[i]);
        m[0] += b > tau ? P[i] : 0.f;
        eq += b == tau ? 1.f : 0.f;
      }
      cl.sum<1>(m);
      eq_before = cl.scan(eq, n_eq);
      need = 0;
      for (float cum = m[0]; cum < s.top_p && (float)need < n_eq; need++) cum += __uint_as_float(tau);
    }
    auto kept = [&](uint32_t b, int &rank) { return b > tau || (b == tau && rank++ < need); };
    int rank = (int)eq_before;
    float loc = 0.f, total;
    for (int i = i0; i < i1; i++) loc += kept(__float_as_uint(P[i]), rank) ? P[i] : 0.f;
    float run = cl.scan(loc, total);
    const float target = u * total;  // rand::distributions::WeightedIndex: the first entry whose inclusive prefix sum exceeds it
    int found = 0x7fffffff, last = -1;
    rank = (int)eq_before;
    for (int i = i0; i < i1; i++) {
      if (!kept(__float_as_uint(P[i]), rank)) continue;
      run += P[i];
      if (P[i] > 0.f) last = base + i;
      if (run > target && found == 0x7fffffff) found = base + i;
    }
    int r = cl.min_i(found);
    if (r == 0x7fffffff) {  // u * total rounded up to the total itself: the last kept entry (WeightedIndex can return len-1)
      r = 0x7ffffffe - cl.min_i(last < 0 ? 0x7fffffff : 0x7ffffffe - last);
      if (r < 0) r = 0;
    }
    finish(r);
    return;
  }

  // ---- the K most probable entries, ties at the K-th in vocabulary order, to the first CTA ---------------------
  const int K = s.top_k;
  const uint32_t lo = __float_as_uint(weight(DT<T>::from_f(sample_threshold<T, true>(cl, L, P, i0, i1, (float)K, -INFINITY, INFINITY))) / sum);
  float gt = 0.f, eq = 0.f, n_gt, n_eq;
  for (int i = i0; i < i1; i++) {
    const uint32_t b = __float_as_uint(P[i]);
    gt += b > lo ? 1.f : 0.f;
    eq += b == lo ? 1.f : 0.f;
  }
  int at_gt = (int)cl.scan(gt, n_gt);
  int at_eq = (int)cl.scan(eq, n_eq) + (int)n_gt;
  for (int i = i0; i < i1; i++) {
    const uint32_t b = __float_as_uint(P[i]);
    if (b < lo) continue;
    const int at = b > lo ? at_gt++ : at_eq++;
    if (at >= K) continue;
    st_cluster_f32(cluster_map(smem_u32(&sh.c_p[at]), 0u), P[i]);
    st_cluster_f32(cluster_map(smem_u32(&sh.c_i[at]), 0u), __int_as_float(base + i));
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (cl.rank != 0) return;
  // ---- sort the K candidates: probability descending, ties by lower id (bitonic, shared memory) ---------------
  float *c_p = sh.c_p;
  int *c_i = sh.c_i;
  int np = 1;
  while (np < K) np <<= 1;
  for (int i = K + tid; i < np; i += SAMPLE_THREADS) { c_p[i] = -1.f; c_i[i] = 0x7fffffff; }
  __syncthreads();
  for (int k2 = 2; k2 <= np; k2 <<= 1)
    for (int j = k2 >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < np; i += SAMPLE_THREADS) {
        const int l = i ^ j;
        if (l > i) {
          const bool up = ((i & k2) == 0);
          const bool a_first = (c_p[i] > c_p[l]) || (c_p[i] == c_p[l] && c_i[i] < c_i[l]);  // i should precede l
          if (a_first != up) {
            const float tp = c_p[i]; c_p[i] = c_p[l]; c_p[l] = tp;
            const int ti = c_i[i]; c_i[i] = c_i[l]; c_i[l] = ti;
          }
        }
      }
      __syncthreads();
    }
  // TopK / TopKThenTopP: draw over the sorted candidates (our defined order: probability descending), a short sequential walk
  if (tid == 0) {
    int m = K;
    if (want_p) {  // nucleus rule inside the k candidates (sample_topk_topp: sort, clip, multinomial)
      float cum = 0.f;
      for (m = 0; m < K; m++) {
        if (cum >= s.top_p) break;
        cum += c_p[m];
      }
    }
    float total = 0.f;
    for (int j = 0; j < m; j++) total += c_p[j];
    const float target = u * total;
    float run = 0.f;
    int pick = m - 1;
    for (int j = 0; j < m; j++) {
      run += c_p[j];
      if (run > target) { pick = j; break; }
    }
    finish(c_i[pick < 0 ? 0 : pick]);
  }
}

}  // namespace cake
