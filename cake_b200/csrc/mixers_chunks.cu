// mixers_chunks.cu — the gated linear recurrence of mixers.cuh over many tokens, in chunks of 64.  sm_100a only.
//
//   S_t = a_t S_{t-1} + b_t k_t v_t^T,  o_t = S_t^T q_t + skip v_t      (state [dk, dv] per head, everything fp32)
//
// Walking the tokens one by one takes 0.2 us each whatever the chip could do beside it: 64 or 128 CTAs, a chain of 1000 steps (16 heads of 128 x 128:
// 223 us, here 74; 64 heads of 128 x 64: 181 us, here 126, of which the outputs are 80, bound by the FMA pipe and the way to shared memory).  A chunk's part of the recurrence needs the state in front of it only linearly, so
//   1. every chunk's own contribution U = sum_j (prod_{t > j} a_t) b_j k_j v_j^T and decay prod a_t are formed side by side,
//   2. one pass over the chunks turns U into the state in front of each chunk (S <- decay S + U) and leaves the last one behind,
//   3. every chunk's outputs are formed side by side: o_i = sum_{j <= i} (prod_{j < t <= i} a_t) b_j (q_i . k_j) v_j + (prod_{t <= i} a_t) S^T q_i.
// The same sums in another order, and in fp32 on the FMA pipe as before: rotated q and k, decays and states are fp32 values, and a split
// into 16-bit parts for the tensor cores would take nine products of each.  Products of decays are formed by running multiplication,
// not as quotients or exponentials of sums, so that strong decays (down to 0) keep their relative precision, and in fp64: 64 roundings of a
// constant decay all fall to one side (retention, 1000 tokens, error against 64 bits 3.6e-7 with fp32 products, 2.1e-7 with fp64, 2.5e-7 token by token).
#include "mixers.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include <algorithm>

#include "common.cuh"

namespace cake {
namespace mx {

constexpr int CH_T = 64, CH_N = 64, CH_THREADS = 256;  // tokens of a chunk, state columns of a CTA
constexpr size_t CH_STATE_BYTES = (size_t)64 << 20;    // states in front of chunks that are held at once: they stay in L2 between the passes

struct Chunks {
  Recurrence r;
  int t0, n;        // first token and number of chunks of this pass over the recurrence
  int init;         // the state buffer holds the state in front of t0
  float *u, *decay; // [B, heads, n, dk, dv], [B, heads, n]
};

// Four values of D as they lie in memory.  Everything staged is read-only for the kernel and asked for with non-coherent loads, all of a
// thread's before its first store to shared memory: loop by loop a CTA spent 8 us on its way to the first product.
template <typename T> struct Raw4 { uint2 u; };
template <> struct Raw4<float> { float4 u; };
template <typename T> __device__ __forceinline__ void ch_get(Raw4<T> &r, const T *s) { r.u = __ldg(reinterpret_cast<const uint2 *>(s)); }
__device__ __forceinline__ void ch_get(Raw4<float> &r, const float *s) { r.u = __ldg(reinterpret_cast<const float4 *>(s)); }
template <typename T> __device__ __forceinline__ float4 ch_float4(const Raw4<T> &r) {
  const float2 a = DT<T>::unpack2(r.u.x), b = DT<T>::unpack2(r.u.y);
  return make_float4(a.x, a.y, b.x, b.y);
}
template <> __device__ __forceinline__ float4 ch_float4<float>(const Raw4<float> &r) { return r.u; }
__device__ __forceinline__ void ch_rotate(float4 &a, float4 &b, const float4 &c, const float4 &s) {
  const float4 x = a, y = b;
  a.x = fmaf(y.x, -s.x, x.x * c.x); a.y = fmaf(y.y, -s.y, x.y * c.y); a.z = fmaf(y.z, -s.z, x.z * c.z); a.w = fmaf(y.w, -s.w, x.w * c.w);
  b.x = fmaf(x.x, s.x, y.x * c.x); b.y = fmaf(x.y, s.y, y.y * c.y); b.z = fmaf(x.z, s.z, y.z * c.z); b.w = fmaf(x.w, s.w, y.w * c.w);
}
// The chunk's rows of q (N = 2 only) and k, rotated, and its values, as fp32; rows past the last token are zeros.
template <typename T, int DK, bool ROPE, int N>
__device__ __forceinline__ void ch_stage(const Recurrence &p, int col, size_t m0, int pos, int nt, float *qs, float *ks, int pitch, int vcol, float *vs) {
  constexpr int G = DK / 8, IT = CH_T * G / CH_THREADS, VT = CH_T * CH_N / 4 / CH_THREADS;
  Raw4<T> a[N][IT], b[N][IT], rv[VT];
  float4 c[IT], s[IT];
#pragma unroll
  for (int e = 0; e < IT; e++) {
    const int idx = threadIdx.x + CH_THREADS * e, tt = min(idx / G, nt - 1), i = (idx % G) * 4;
#pragma unroll
    for (int w = 0; w < N; w++) {
      const T *row = reinterpret_cast<const T *>(w ? p.q : p.k) + (m0 + tt) * (w ? p.ldq : p.ldk) + col + i;
      ch_get(a[w][e], row);
      ch_get(b[w][e], row + DK / 2);
    }
    if (ROPE) {
      c[e] = __ldg(reinterpret_cast<const float4 *>(p.cos_t + (size_t)(pos + tt) * (DK / 2) + i));
      s[e] = __ldg(reinterpret_cast<const float4 *>(p.sin_t + (size_t)(pos + tt) * (DK / 2) + i));
    }
  }
#pragma unroll
  for (int e = 0; e < VT; e++) {
    const int idx = threadIdx.x + CH_THREADS * e, tt = min(idx / (CH_N / 4), nt - 1), n = (idx % (CH_N / 4)) * 4;
    ch_get(rv[e], reinterpret_cast<const T *>(p.v) + (m0 + tt) * p.ldv + vcol + n);
  }
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int e = 0; e < IT; e++) {
    const int idx = threadIdx.x + CH_THREADS * e, tt = idx / G, i = (idx % G) * 4;
#pragma unroll
    for (int w = 0; w < N; w++) {
      float4 x = ch_float4<T>(a[w][e]), y = ch_float4<T>(b[w][e]);
      if (ROPE) ch_rotate(x, y, c[e], s[e]);
      float *dst = (w ? qs : ks) + tt * pitch + i;
      *reinterpret_cast<float4 *>(dst) = tt < nt ? x : zero;
      *reinterpret_cast<float4 *>(dst + DK / 2) = tt < nt ? y : zero;
    }
  }
#pragma unroll
  for (int e = 0; e < VT; e++) {
    const int idx = threadIdx.x + CH_THREADS * e, tt = idx / (CH_N / 4);
    reinterpret_cast<float4 *>(vs)[idx] = tt < nt ? ch_float4<T>(rv[e]) : zero;
  }
}
// a_t and b_t of a chunk (1 and 0 past the last token)
template <typename T> __device__ __forceinline__ void ch_factors(const Recurrence &p, int h, size_t m0, int nt, float *as, float *bs) {
  const int t = threadIdx.x;
  if (t >= CH_T) return;
  float a = 1.f, b = 0.f;
  if (t < nt) {
    a = p.decay ? p.decay[h] : 1.f;
    b = p.kscale;
    if (p.dt) {
      const float z = DT<T>::to_f(reinterpret_cast<const T *>(p.dt)[(m0 + t) * p.lddt + h]) + DT<T>::to_f(reinterpret_cast<const T *>(p.dt_bias)[h]);
      const float d = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));
      a = expf(-expf(DT<T>::to_f(reinterpret_cast<const T *>(p.a_log)[h])) * d);
      b = d;
    }
  }
  as[t] = a;
  bs[t] = b;
}

// Pass 1.  One CTA: 64 columns of a chunk's U; a thread DK / 16 rows x 4 columns.
template <int DK> constexpr int ch_state_smem() { return (CH_T * DK + CH_T * CH_N + 3 * CH_T) * (int)sizeof(float); }
template <typename T, int DK, bool ROPE>
__global__ void __launch_bounds__(CH_THREADS, 3) chunk_state_kernel(const Chunks c) {
  extern __shared__ __align__(16) float ch_sm[];
  const Recurrence &p = c.r;
  float *ks = ch_sm, *vs = ks + CH_T * DK, *as = vs + CH_T * CH_N, *bs = as + CH_T, *ws = bs + CH_T;
  const int ncb = p.dv / CH_N, h = blockIdx.x / ncb, cb = blockIdx.x % ncb, ci = blockIdx.y, b = blockIdx.z;
  const int t0 = c.t0 + ci * CH_T, nt = min(CH_T, p.S - t0);
  const size_t m0 = (size_t)b * p.S + t0;
  ch_factors<T>(p, h, m0, nt, as, bs);
  ch_stage<T, DK, ROPE, 1>(p, (h / p.group_div) * DK, m0, p.pos0 + t0, nt, nullptr, ks, DK, h * p.dv + cb * CH_N, vs);
  __syncthreads();
  if (threadIdx.x < CH_T) {  // w_j = b_j prod_{t > j} a_t
    double w = bs[threadIdx.x];
#pragma unroll 8
    for (int t = 0; t < CH_T; t++) w *= t > (int)threadIdx.x ? as[t] : 1.f;
    ws[threadIdx.x] = (float)w;
  } else if (threadIdx.x == CH_T && cb == 0) {
    double w = 1.0;
#pragma unroll 8
    for (int t = 0; t < CH_T; t++) w *= as[t];
    c.decay[((size_t)b * p.heads + h) * c.n + ci] = (float)w;
  }
  __syncthreads();
  constexpr int DT_ = DK / 16;  // rows of a thread (8 or 4)
  const int d0 = (threadIdx.x / 16) * DT_, n0 = (threadIdx.x % 16) * 4;
  float acc[DT_][4] = {};
#pragma unroll 4
  for (int j = 0; j < CH_T; j++) {
    const float w = ws[j];
    float4 v = *reinterpret_cast<const float4 *>(vs + j * CH_N + n0);
    v.x *= w; v.y *= w; v.z *= w; v.w *= w;
    float k[DT_];
#pragma unroll
    for (int i = 0; i < DT_; i += 4) {
      const float4 k4 = *reinterpret_cast<const float4 *>(ks + j * DK + d0 + i);
      k[i] = k4.x; k[i + 1] = k4.y; k[i + 2] = k4.z; k[i + 3] = k4.w;
    }
#pragma unroll
    for (int i = 0; i < DT_; i++) {
      acc[i][0] = fmaf(k[i], v.x, acc[i][0]);
      acc[i][1] = fmaf(k[i], v.y, acc[i][1]);
      acc[i][2] = fmaf(k[i], v.z, acc[i][2]);
      acc[i][3] = fmaf(k[i], v.w, acc[i][3]);
    }
  }
  float *u = c.u + ((((size_t)b * p.heads + h) * c.n + ci) * DK + d0) * p.dv + cb * CH_N + n0;
#pragma unroll
  for (int i = 0; i < DT_; i++) *reinterpret_cast<float4 *>(u + (size_t)i * p.dv) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}

// Pass 2.  A thread: four entries of a head's state, through the chunks in order; eight chunks' U are on their way.
__global__ void __launch_bounds__(CH_THREADS) chunk_scan_kernel(const Chunks c) {
  const Recurrence &p = c.r;
  const size_t per = (size_t)p.dk * p.dv / 4, idx = (size_t)blockIdx.x * CH_THREADS + threadIdx.x;
  const size_t bh = blockIdx.y;
  if (idx >= per) return;
  float4 *state = reinterpret_cast<float4 *>(p.state) + bh * per + idx;
  float4 *u = reinterpret_cast<float4 *>(c.u) + bh * c.n * per + idx;
  const float *decay = c.decay + bh * c.n;
  float4 s = c.init ? *state : make_float4(0.f, 0.f, 0.f, 0.f);
  constexpr int AHEAD = 8;
  float4 w[AHEAD];
  float a[AHEAD];
  for (int i0 = 0; i0 < c.n; i0 += AHEAD) {
#pragma unroll
    for (int e = 0; e < AHEAD; e++)
      if (i0 + e < c.n) { w[e] = u[(size_t)(i0 + e) * per]; a[e] = decay[i0 + e]; }
#pragma unroll
    for (int e = 0; e < AHEAD; e++)
      if (i0 + e < c.n) {
        u[(size_t)(i0 + e) * per] = s;
        s.x = fmaf(a[e], s.x, w[e].x); s.y = fmaf(a[e], s.y, w[e].y); s.z = fmaf(a[e], s.z, w[e].z); s.w = fmaf(a[e], s.w, w[e].w);
      }
  }
  *state = s;
}

// Pass 3.  One CTA: 64 columns of a chunk's outputs.  Thread (ti, tn) of 16 x 16 forms P for rows 4 ti .. + 3 and keys tn + 16 r, then the outputs
// of the same rows and columns 4 tn .. + 3: a warp holds eight rows, so keys behind them cost it nothing.  Two CTAs per SM: the state in front
// of the chunk waits in registers and takes the keys' place.
template <int DK> constexpr int ch_out_smem() { return (2 * CH_T * (DK + 4) + CH_T * CH_N + CH_T * (CH_T + 4) + 3 * CH_T) * (int)sizeof(float); }
template <typename T, int DK, bool ROPE>
__global__ void __launch_bounds__(CH_THREADS, 2) chunk_out_kernel(const Chunks c) {
  extern __shared__ __align__(16) float ch_sm[];
  const Recurrence &p = c.r;
  constexpr int QP = DK + 4, PP = CH_T + 4, SR = DK * CH_N / 4 / CH_THREADS;
  static_assert(DK * CH_N <= CH_T * QP, "the state fits in the keys' place");
  float *qs = ch_sm, *ks = qs + CH_T * QP, *vs = ks + CH_T * QP, *ps = vs + CH_T * CH_N, *as = ps + CH_T * PP, *bs = as + CH_T, *cum = bs + CH_T;
  const int ncb = p.dv / CH_N, h = blockIdx.x / ncb, cb = blockIdx.x % ncb, ci = blockIdx.y, b = blockIdx.z;
  const int t0 = c.t0 + ci * CH_T, nt = min(CH_T, p.S - t0), warp = threadIdx.x >> 5;
  const size_t m0 = (size_t)b * p.S + t0;
  ch_factors<T>(p, h, m0, nt, as, bs);
  ch_stage<T, DK, ROPE, 2>(p, (h / p.group_div) * DK, m0, p.pos0 + t0, nt, qs, ks, QP, h * p.dv + cb * CH_N, vs);
  __syncthreads();
  if (threadIdx.x < CH_T) {  // P[i][j] starts as b_j prod_{j < t <= i} a_t
    const int j = threadIdx.x;
    double w = bs[j];
#pragma unroll 8
    for (int i = 0; i < CH_T; i++) {
      w *= i > j ? as[i] : 1.f;
      ps[i * PP + j] = (float)w;
    }
  } else if (threadIdx.x == CH_T) {
    double w = 1.0;
#pragma unroll 8
    for (int i = 0; i < CH_T; i++) { w *= as[i]; cum[i] = (float)w; }
  }
  float4 st[SR];
  const float *u = c.u + (((size_t)b * p.heads + h) * c.n + ci) * DK * p.dv + cb * CH_N;
#pragma unroll
  for (int e = 0; e < SR; e++) {
    const int idx = threadIdx.x + CH_THREADS * e, d = idx / (CH_N / 4), n = (idx % (CH_N / 4)) * 4;
    st[e] = __ldg(reinterpret_cast<const float4 *>(u + (size_t)d * p.dv + n));
  }
  const int ti = threadIdx.x / 16, tn = threadIdx.x % 16;
  float s[4][4] = {};
  const int groups = warp / 2 + 1;  // of 16 keys that the warp's rows see
  // (sums of 32 products each, then added up: rounding errors like those of eight warps' partial sums)
#pragma unroll 1
  for (int d0 = 0; d0 < DK; d0 += 32) {
    float z[4][4] = {};
#pragma unroll 2
    for (int d = d0; d < d0 + 32; d += 4) {
      float4 q[4];
#pragma unroll
      for (int r = 0; r < 4; r++) q[r] = *reinterpret_cast<const float4 *>(qs + (4 * ti + r) * QP + d);
#pragma unroll
      for (int g = 0; g < 4; g++)
        if (g < groups) {
          const float4 k = *reinterpret_cast<const float4 *>(ks + (tn + 16 * g) * QP + d);
#pragma unroll
          for (int r = 0; r < 4; r++) {
            z[r][g] = fmaf(q[r].x, k.x, z[r][g]);
            z[r][g] = fmaf(q[r].y, k.y, z[r][g]);
            z[r][g] = fmaf(q[r].z, k.z, z[r][g]);
            z[r][g] = fmaf(q[r].w, k.w, z[r][g]);
          }
        }
    }
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int g = 0; g < 4; g++) s[r][g] += z[r][g];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int g = 0; g < 4; g++)
      if (g < groups) {
        const int i = 4 * ti + r, j = tn + 16 * g;
        ps[i * PP + j] = j <= i ? ps[i * PP + j] * s[r][g] : 0.f;
      }
#pragma unroll
  for (int e = 0; e < SR; e++) reinterpret_cast<float4 *>(ks)[threadIdx.x + CH_THREADS * e] = st[e];
  __syncthreads();
  float o[4][4] = {};
  auto rows4 = [&](float (&o)[4][4], const float *x, int pitch, int at, const float *y) {  // o[r] += sum of four x[row r][at ..] y[at ..][columns]
    float4 w[4];
#pragma unroll
    for (int r = 0; r < 4; r++) w[r] = *reinterpret_cast<const float4 *>(x + (4 * ti + r) * pitch + at);
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float4 v = *reinterpret_cast<const float4 *>(y + (at + e) * CH_N + 4 * tn);
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float f = e == 0 ? w[r].x : e == 1 ? w[r].y : e == 2 ? w[r].z : w[r].w;
        o[r][0] = fmaf(f, v.x, o[r][0]);
        o[r][1] = fmaf(f, v.y, o[r][1]);
        o[r][2] = fmaf(f, v.z, o[r][2]);
        o[r][3] = fmaf(f, v.w, o[r][3]);
      }
    }
  };
#pragma unroll 1
  for (int d0 = 0; d0 < DK; d0 += 32) {
    float z[4][4] = {};
#pragma unroll 2
    for (int d = d0; d < d0 + 32; d += 4) rows4(z, qs, QP, d, ks);
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int e = 0; e < 4; e++) o[r][e] += z[r][e];
  }
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int e = 0; e < 4; e++) o[r][e] *= cum[4 * ti + r];
#pragma unroll 2
  for (int j = 0; j < 8 * warp; j += 4) rows4(o, ps, PP, j, vs);
  // the warp's own eight tokens: a value behind a row is left out, not multiplied by 0 (it may be an infinity)
  for (int j = 8 * warp; j < 8 * warp + 8; j++) {
    const float4 v = *reinterpret_cast<const float4 *>(vs + j * CH_N + 4 * tn);
#pragma unroll
    for (int r = 0; r < 4; r++)
      if (j <= 4 * ti + r) {
        const float f = ps[(4 * ti + r) * PP + j];
        o[r][0] = fmaf(f, v.x, o[r][0]);
        o[r][1] = fmaf(f, v.y, o[r][1]);
        o[r][2] = fmaf(f, v.z, o[r][2]);
        o[r][3] = fmaf(f, v.w, o[r][3]);
      }
  }
  const float skip = p.skip ? DT<T>::to_f(reinterpret_cast<const T *>(p.skip)[h]) : 0.f;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int i = 4 * ti + r;
    if (i >= nt) break;
    const float4 v = *reinterpret_cast<const float4 *>(vs + i * CH_N + 4 * tn);
    *reinterpret_cast<float4 *>(p.o + (m0 + i) * ((size_t)p.heads * p.dv) + (size_t)h * p.dv + cb * CH_N + 4 * tn) =
        make_float4(fmaf(skip, v.x, o[r][0]), fmaf(skip, v.y, o[r][1]), fmaf(skip, v.z, o[r][2]), fmaf(skip, v.w, o[r][3]));
  }
}

// Chunks whose states are held at once; 0: the recurrence walks token by token.
static int chunks_at_once(int B, int S, int heads, int dk, int dv) {
  if ((dk != 64 && dk != 128) || dv % CH_N || dv < 1 || S < CHUNK_MIN_TOKENS) return 0;
  const size_t state = (size_t)B * heads * dk * dv * sizeof(float);
  const size_t fit = CH_STATE_BYTES / state;
  if (fit < 4) return 0;
  return (int)std::min<size_t>((size_t)(S + CH_T - 1) / CH_T, fit);
}
size_t recurrence_scratch(int B, int S, int heads, int dk, int dv) {
  const int n = chunks_at_once(B, S, heads, dk, dv);
  return (size_t)B * heads * n * ((size_t)dk * dv + 1) * sizeof(float);
}
template <typename T, int DK, bool ROPE> static cudaError_t launch_chunks(cudaStream_t st, const Recurrence &p, int at_once, int *n_launches) {
  static int attr_dev = -1;  // per instantiation: the device the attributes were last set on (the values never change)
  int dev = 0;
  cudaGetDevice(&dev);
  if (attr_dev != dev) {
    cudaError_t e = cudaFuncSetAttribute(chunk_state_kernel<T, DK, ROPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, ch_state_smem<DK>());
    if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_out_kernel<T, DK, ROPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, ch_out_smem<DK>());
    if (e != cudaSuccess) return e;
    attr_dev = dev;
  }
  Chunks c{p, 0, 0, p.pos0 > 0, p.scratch, nullptr};
  for (; c.t0 < p.S; c.t0 += c.n * CH_T, c.init = 1) {
    c.n = std::min(at_once, (p.S - c.t0 + CH_T - 1) / CH_T);
    c.decay = c.u + (size_t)p.B * p.heads * c.n * DK * p.dv;
    const dim3 grid(p.heads * (p.dv / CH_N), c.n, p.B);
    chunk_state_kernel<T, DK, ROPE><<<grid, CH_THREADS, ch_state_smem<DK>(), st>>>(c);
    chunk_scan_kernel<<<dim3((unsigned)((size_t)DK * p.dv / 4 + CH_THREADS - 1) / CH_THREADS, p.B * p.heads), CH_THREADS, 0, st>>>(c);
    chunk_out_kernel<T, DK, ROPE><<<grid, CH_THREADS, ch_out_smem<DK>(), st>>>(c);
    *n_launches += 3;
  }
  return cudaGetLastError();
}
int recurrence_chunks(cudaStream_t st, int dtype, const Recurrence &p, int *n_launches) {
  const int at_once = p.scratch && !p.a_chan && !p.a_tok && p.qscale == 1.f ? chunks_at_once(p.B, p.S, p.heads, p.dk, p.dv) : 0;
  const bool rope = p.cos_t && p.rope_dims > 0;
  const uintptr_t in_align = dtype == 2 ? 15 : 7;
  if (!at_once || (rope && p.rope_dims != p.dk) || p.ldq % 4 || p.ldk % 4 || p.ldv % 4 || (((uintptr_t)p.q | (uintptr_t)p.k | (uintptr_t)p.v) & in_align) ||
      (((uintptr_t)p.state | (uintptr_t)p.o | (uintptr_t)p.scratch | (rope ? (uintptr_t)p.cos_t | (uintptr_t)p.sin_t : 0)) & 15))
    return (int)cudaErrorNotSupported;
  auto run = [&](auto tag) {
    typedef decltype(tag) T;
    if (p.dk == 128) return rope ? launch_chunks<T, 128, true>(st, p, at_once, n_launches) : launch_chunks<T, 128, false>(st, p, at_once, n_launches);
    return rope ? launch_chunks<T, 64, true>(st, p, at_once, n_launches) : launch_chunks<T, 64, false>(st, p, at_once, n_launches);
  };
  return (int)(dtype == 2 ? run(float()) : dtype == 1 ? run(__half()) : run(__nv_bfloat16()));
}

}  // namespace mx
}  // namespace cake
