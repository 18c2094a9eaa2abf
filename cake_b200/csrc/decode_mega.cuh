// decode_mega.cuh — the decode hot loop as ONE persistent kernel per shard-step.
//
// Why: with one kernel per op (5 per layer) every dependency between ops is a kernel boundary that
// costs ~3 us of HBM idle time even with programmatic dependent launch (profiles/gemv_sweep_r01.txt:
// o_proj 7.2 us streamed vs 5.1 us ideal) — 130 boundaries per token = ~0.4 ms of a 2.3 ms budget.
// Here the whole walk  [rms_1+qkv -> rope/append/attention -> o_proj+res -> rms_2+gate_up+silu*mul ->
// down+res] x layers (+ ln_f/lm_head/argmax on the master)  runs inside one grid of one CTA per SM:
//   * one warp is the PRODUCER: it walks the same static phase list and issues TMA bulk copies of the
//     next weight rows (32 KB stages, evict_first) and of this CTA's K/V cache tile into a 5-6 stage
//     shared-memory ring.  It waits for no other CTA, so HBM keeps streaming while the
//     consumers exchange a vector — the ring (~160 KB/SM, ~24 MB chip-wide) absorbs the bubbles;
//   * the other warps are CONSUMERS: per phase they gather the previous phase's output vector (RMS-normalised
//     in-kernel), multiply-accumulate the staged rows in fp32 and run the fused epilogue;
//   * a vector travels from phase to phase as PACKETS of 32 bits in global memory (L2): the 16-bit value and a 16-bit tag
//     that changes with every layer.  A CTA stores the packets of its rows and goes on; whoever needs the vector reads the packets
//     themselves until their tags are right.  One store and one load lie between two phases where a grid barrier
//     has the release of the CTA's stores, its arrival, the poll and only then the load of the vector.
// Bound by HBM where a layer's weights are large (8B: 436 MB a layer) and by the chain of five exchanges per layer where they are not
// (0.6B: 31 MB, 5 us of stream).  With grid barriers and fp32 conversions in 16 warps: 32 us a layer at 0.6B, 24 tokens 25.1 ms, 8B two layers 187 us; now
// 15 us, 14.1 ms and 184 to 186 us.  From a CTA's last row of a phase to the next phase's complete input 0.9 to 1.4 us pass at 0.6B and 3.3 to 4.2 at 8B, where CTAs
// end further apart (9.5 behind the down product, whose groups are one row of 28 KB); a product of 12 MB takes 2.1 us behind it.
// Arithmetic and rounding points are identical to the per-op kernels (gemv.cuh / attn_decode.cuh), correctly rounded divisions and square roots
// included (a Newton step on the fast instructions in their place saved 0.3 ms over 24 tokens and was an ulp off in places); only the
// fp32 summation order within a dot product differs (tests/test_gpu_parity.py::test_megakernel_equals_per_op_kernels).
//
// A packet buffer is written again one layer later; no reader may still be in front of it.  A CTA that has not gathered the input of
// phase p has published nothing from phase p on, and whoever writes that input again (phase p - 1 of the next layer) has gathered, directly or
// through others, ALL outputs of phases p .. p - 2 (four of the five phases; a vector is complete only when every owner of a row has published).  So
// it is enough that every CTA owns rows of at least two phases whatever the tickets say (mk_every_cta); where a model is too small for that,
// all CTAs meet at one grid barrier per layer, between the gathering of the last phase's input and its output (`meet`).
#pragma once
#include "common.cuh"
#include "gemv.cuh"
#include "attn_decode.cuh"

namespace cake {

constexpr int MK_CW = 8;                        // consumer warps: few, so that a thread has 168 registers (what spills lands in L2 beside 220 KB of shared memory)
constexpr int MK_CT = MK_CW * 32;               // consumer threads
constexpr int MK_THREADS = (MK_CW + 1) * 32;    // + producer warp
constexpr int MK_STAGE_BYTES = 32768;
constexpr int MK_BATCH = 512;                   // row segments whose sums are kept until an epilogue takes them
constexpr int MK_MAX_STAGES = 6;
constexpr int MK_MAX_LAYERS = 96;
constexpr int MK_HEAD_TICKET = 4 * MK_MAX_LAYERS;

struct MkLayer {
  const void *wqkv, *wo, *wgu, *wd, *ln1, *ln2, *bqkv, *qn, *kn;
  void *kc, *vc;
};
struct MkGeom {  // one decode GEMV type; a stage holds 2^RSL row segments of KC columns (planned by the host: no divisions in the kernel)
  int N, K, KC, RSL, nchunk;   // nchunk = K / KC; above 1 a stage holds one segment
  int n_groups, batch;         // groups of 2^RSL rows; groups between two epilogues
  int unit, cnt, rem;          // static groups: CTA c has unit * (cnt + (c < rem)) of them
  int pool;                    // first group of the pool (n_groups: none)
};
// the vectors that travel as packets (uint32_t: value | tag << 16)
struct MkPackets {
  uint32_t *xa, *qkv, *y, *xb, *mm;   // layer output, projections, attention, behind the o product, act(gate) * up
  uint64_t *acc, *ml;                 // attention of several splits: fp32 values | 32-bit tag << 32; ml holds (max, sum) pairs
};
struct MkArgs {
  const MkLayer *layers;
  int n_layers;
  MkGeom g[5];               // qkv, o, gate_up, down, head
  int hidden, inter, n_heads, n_kv, hd, rot, cap, nsplit, max_k;
  float eps, scale;
  const void *x_in;          // input hidden state (nullptr on the master: embed row of *d_token)
  const void *embed;
  const uint32_t *d_token;
  void *x_out;               // output hidden state of this shard
  MkPackets pk;
  const void *cos_t, *sin_t;
  int *d_pos, *d_step;
  unsigned long long *gbar;      // [0] monotonic barrier arrival counter, [1] its value at launch start, [2] layers run so far (the tags)
  int has_head, advance, n_stages, vocab;
  int meet;                      // one grid barrier per layer: some CTA may own no row of a layer (see the top)
  int keep_x;                    // the residual stream stays in shared memory between the phase that reads it and the one that adds it
  const void *ln_f, *lm_head;
  void *logits;
  float *part_val;
  int *part_idx;
  unsigned *argmax_counter;
  uint32_t *token_out, *token_ring;
  int ring_cap;
  // shard-to-shard hand-off over NVLink peer memory (fused into this kernel; no NCCL kernel in the step):
  //   inbox_ctr != nullptr: wait until the previous shard has delivered step *ring_seq into our inbox (x_in)
  //   peer_ctr  != nullptr: x_out is the next shard's inbox; signal it when every CTA has written its rows
  const unsigned long long *inbox_ctr;
  unsigned long long *peer_ctr;
  unsigned long long *ring_seq;   // hand-offs received so far (device-resident, never reset)
  unsigned *tickets;          // [phase] work-claim counters: a layer's zeroed before every launch that has a layer's phase with a pool,
                              // the head's (MK_HEAD_TICKET) by the last CTA of the launch in front
  int off_x, off_res, off_part, off_loc, off_rows;  // shared memory (mk_layout)
  unsigned long long *trace;  // optional: %globaltimer stamps of CTA 0 at phase boundaries (profiling aid)
  // always on (3 stores per launch): %globaltimer of CTA 0 at kernel entry / input acquired / exit, ring of
  // MK_STEP_RING steps x 2 launches (tag 0: the layer launch, tag 1: rank 0's head-only launch when sharded) x 4 u64
  unsigned long long *step_trace;
  int trace_tag;
  int act;     // mlp.rs:25-26: 0 silu, 1 gelu_tanh
  int window;  // cache.rs:173-205 sliding window (0 = full context): attention covers the last `window` positions
  int *err;    // host-mapped: set by a wait for packets that ran out
  int polls, inbox_polls;   // what a thread's waits may spend (MK_POLLS, MK_INBOX_POLLS; less in a test)
};
constexpr int MK_STEP_RING = 2048;
__device__ __forceinline__ unsigned long long mk_gtime() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// what the consumers look up per layer, copied to shared memory at the start
struct MkRow {
  const void *ln1, *ln2, *bqkv, *qn, *kn;
  void *kc, *vc;
};
__host__ __device__ inline size_t mk_xs_bytes(int max_k, int es) {
  size_t b = (size_t)max_k * es;
  const size_t attn = (size_t)(ATTN_MAX_G * 256 * 4) + (size_t)ATTN_MAX_G * ATTN_TILE * 4 + (size_t)2 * 256 * 4;
  return b > attn ? b : attn;  // the attention phase overlays its scratch on the x buffer
}
// Shared memory: barriers, stage rows and scratch at fixed places, the ring, then what the model's sizes decide.
// A thread that is done with a phase begins the next one at once, so an area is reused only where a barrier of the consumers lies between its
// last reader and its next writer:
//   x (off_x)        written by a gather.  Its readers in front: a product's loop, which ends with a barrier before the epilogue; attention's queries,
//                    scores and new rows, all read before the barrier behind the last tile's sums.  The merge of split attention reads on while
//                    other threads of the CTA gather already, so its parts lie in the partial sums' area and not here.
//                    Attention writes over x behind the qkv product's barrier.
//   partial sums     written by a product's loop, behind the barrier of its gather, and by the merge of attention, behind attention's first barriers: all
//                    epilogues (and the merge) are over when the CTA's threads have met there.  Batches of one product: the barrier behind an epilogue.
//   loc (off_loc)    as the partial sums.
//   residual copy    written by the gathers of qkv and gate_up without a barrier in front: an epilogue reads row r before it publishes r, and a gather writes
//                    over r only when it has seen that packet.
//   scratch          a warp's sum of squares: written in front of a gather's barrier, read behind it, and the next one is written after at least
//                    one product's barriers; the head's winners: behind the last product's barrier.
constexpr int MK_OFF_EMPTY = 8 * MK_MAX_STAGES, MK_OFF_STAGE_ROW = 16 * MK_MAX_STAGES, MK_OFF_SCRATCH = 256, MK_OFF_RING = 1024;
inline size_t mk_layout(MkArgs &a, int es) {
  size_t off = MK_OFF_RING + (size_t)a.n_stages * MK_STAGE_BYTES;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = (off + bytes + 15) & ~(size_t)15;
    return (int)at;
  };
  a.off_x = take(mk_xs_bytes(a.max_k, es));
  a.off_res = take(a.keep_x ? (size_t)a.hidden * es : 0);
  a.off_part = take(MK_BATCH * MK_CW * 4);  // partial sums [row][warp of the row]; the parts that the merge of split attention gathers
  a.off_loc = take(MK_BATCH * 4);           // first row of each group of a batch
  a.off_rows = take((size_t)a.n_layers * sizeof(MkRow));
  return off;
}

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

struct MkRing {
  unsigned char *sm;
  int n_stages;
  int s;
  uint32_t ph;
  __device__ __forceinline__ uint64_t *full() const { return reinterpret_cast<uint64_t *>(sm) + s; }
  __device__ __forceinline__ uint64_t *empty() const { return reinterpret_cast<uint64_t *>(sm + MK_OFF_EMPTY) + s; }
  // first weight row held by a stage, or -1 = end-of-phase marker (phases with a pool)
  __device__ __forceinline__ int &row() const { return reinterpret_cast<int *>(sm + MK_OFF_STAGE_ROW)[s]; }
  __device__ __forceinline__ unsigned char *data() const { return sm + MK_OFF_RING + (size_t)s * MK_STAGE_BYTES; }
  __device__ __forceinline__ void advance() {
    if (++s == n_stages) { s = 0; ph ^= 1u; }
  }
};

// The row groups of a GEMV are split into a static part and a pool claimed one group at a time through an atomic ticket.  Per-SM HBM
// bandwidth is not uniform (measured: the slowest CTA of the 8B gate_up phase finished 5.5 us after the fastest with static
// rows), so fast SMs take more pool groups and all CTAs end together: 75 % static (CTA c owns groups [c*cnt, (c+1)*cnt)).  A phase of at most
// MK_SHORT groups per CTA sits in the ring before its input is there, and the CTA that claims one group more than the others is late:
// all of it is static, dealt out evenly; so are rows that take several stages (K of more than a stage), and gate and up rows where a stage holds one row.  A row's dot product
// is computed by one CTA with a fixed lane/warp mapping whichever CTA it is -> results stay bit-deterministic.
constexpr int MK_SHORT = 4;
inline void mk_plan_split(MkGeom &g, int gran, int grid) {  // gran: rows that stay together (gate and up of a pair)
  g.n_groups = (g.N + (1 << g.RSL) - 1) >> g.RSL;
  g.batch = (MK_BATCH >> g.RSL) / g.nchunk;
  if (g.nchunk > 1 || gran > 1 << g.RSL || g.n_groups <= MK_SHORT * grid) {
    g.unit = gran > 1 << g.RSL ? gran : 1;
    g.cnt = g.n_groups / g.unit / grid;
    g.rem = g.n_groups / g.unit % grid;
    g.pool = g.n_groups;
  } else {
    g.unit = 1;
    g.cnt = (int)(((long)g.n_groups * 3 / 4) / grid);
    g.rem = 0;
    g.pool = g.cnt * grid;
  }
}
// every CTA owns at least one row of this phase, whatever the tickets say
inline bool mk_every_cta(const MkGeom &g) { return g.cnt > 0; }
__device__ __forceinline__ int mk_first(const MkGeom &g) { return g.unit * ((int)blockIdx.x * g.cnt + min((int)blockIdx.x, g.rem)); }
__device__ __forceinline__ int mk_count(const MkGeom &g) { return g.unit * (g.cnt + ((int)blockIdx.x < g.rem ? 1 : 0)); }

template <typename T>
__device__ __forceinline__ void mk_produce_gemv(MkRing &rg, const MkGeom &g, const void *W, unsigned *ticket, uint64_t pol) {
  constexpr int es = sizeof(T);
  const size_t rowb = (size_t)g.K * es;
  const unsigned char *Wb = reinterpret_cast<const unsigned char *>(W);
  auto issue = [&](int grp) {
    const int row = grp << g.RSL, nr = min(1 << g.RSL, g.N - row);
    const uint32_t bytes = (uint32_t)nr * g.KC * es;   // (several rows only where a row is one segment)
    for (int k = 0; k < g.K; k += g.KC) {
      mbar_wait(rg.empty(), rg.ph ^ 1u);
      rg.row() = row;
      mbar_arrive_expect_tx(rg.full(), bytes);
      bulk_g2s(rg.data(), Wb + (size_t)row * rowb + (size_t)k * es, bytes, rg.full(), pol);
      rg.advance();
    }
  };
  const int first = mk_first(g), n = mk_count(g);
#pragma unroll 1
  for (int i = 0; i < n; i++) issue(first + i);
  if (g.pool == g.n_groups) return;
  pdl_wait();   // (a head launched early: its counter is zeroed by a launch in front; else at once)
  unsigned next = atomicAdd(ticket, 1u);
#pragma unroll 1
  while (g.pool + (int)next < g.n_groups) {
    const int cur = g.pool + (int)next;
    next = atomicAdd(ticket, 1u);  // claim ahead: the round trip overlaps the wait for a free stage
    issue(cur);
  }
  mbar_wait(rg.empty(), rg.ph ^ 1u);  // end-of-phase marker: the consumers do not know how many groups were claimed
  rg.row() = -1;
  mbar_arrive(rg.full());
  rg.advance();
}

struct MkAttnItem {
  int active, kvh, split, n_split, s0, s1, tile;
};
// The visible positions are cut over as many CTAs as have MK_SPLIT_MIN of them each; up to MK_SPLIT_ONE one CTA per key head takes them all:
// what further CTAs would save of its tile (0.4 us) is less than the exchange of their parts (1.5 us).
constexpr int MK_SPLIT_MIN = 64, MK_SPLIT_ONE = 128;
__device__ __forceinline__ MkAttnItem mk_attn_item(const MkArgs &a, int pos, int es) {
  MkAttnItem it;
  it.kvh = blockIdx.x / a.nsplit;
  it.split = blockIdx.x % a.nsplit;
  const int Tn = pos + 1;
  int per = (Tn + a.nsplit - 1) / a.nsplit;
  per = max((per + 7) & ~7, Tn <= MK_SPLIT_ONE ? MK_SPLIT_ONE : MK_SPLIT_MIN);
  it.n_split = (Tn + per - 1) / per;
  it.active = (int)blockIdx.x < a.n_kv * a.nsplit && it.split < it.n_split;
  it.s0 = min(Tn, it.split * per);
  it.s1 = min(Tn, it.s0 + per);
  const int rows = MK_STAGE_BYTES / (a.hd * es);
  it.tile = rows < ATTN_TILE ? rows : ATTN_TILE;
  if (!it.active) it.s0 = it.s1 = 0;
  return it;
}

template <typename T>
__device__ __forceinline__ void mk_produce_attn(MkRing &rg, const MkArgs &a, const MkLayer &L, int pos, uint64_t pol) {
  // sliding window: the visible rows start at ws = pos + 1 - window; everything below works on row indices relative to ws
  const int ws = (a.window > 0 && pos + 1 > a.window) ? pos + 1 - a.window : 0;
  pos -= ws;
  const MkAttnItem it = mk_attn_item(a, pos, (int)sizeof(T));
  if (!it.active) return;
  const int HD = a.hd;
  const T *kc = reinterpret_cast<const T *>(L.kc) + ((size_t)it.kvh * a.cap + ws) * HD;
  const T *vc = reinterpret_cast<const T *>(L.vc) + ((size_t)it.kvh * a.cap + ws) * HD;
  for (int t0 = it.s0; t0 < it.s1; t0 += it.tile) {
    const int t1 = min(it.s1, t0 + it.tile);
    const int nold = min(t1, pos) - t0;  // rows already in the cache (the appended row is handled by the consumers)
    for (int kv = 0; kv < 2; kv++) {
      mbar_wait(rg.empty(), rg.ph ^ 1u);
      if (nold > 0) {
        const uint32_t bytes = (uint32_t)nold * HD * sizeof(T);
        mbar_arrive_expect_tx(rg.full(), bytes);
        bulk_g2s(rg.data(), (kv ? vc : kc) + (size_t)t0 * HD, bytes, rg.full(), pol);
      } else {
        mbar_arrive(rg.full());
      }
      rg.advance();
    }
  }
}

// ---------------------------------------------------------------------------------------- packets
// A thread's waits for other CTAs share one budget: when it is spent the error word is set, and every later wait of the thread returns at once.
// A poll is a round trip to L2 (0.2 us in an idle chip, 0.6 us beside the weights), so a thread gives up after half a second or more (the 80 layers of
// a 70B model are 22 ms), and a launch whose waits all give up still ends.
constexpr int MK_POLLS = 1 << 21;
// The wait for the previous shard has a budget of its own, about a minute, as that rank may still read its prompt: MK_INBOX_FAST polls, then one every 8 us.
constexpr int MK_INBOX_FAST = 1 << 20, MK_INBOX_POLLS = MK_INBOX_FAST + (1 << 23);
struct MkWait {
  int left;
  int *err;
  __device__ __forceinline__ bool again() {
    if (left <= 0) return false;
    if (--left == 0) *reinterpret_cast<volatile int *>(err) = 1;
    return true;
  }
};
__device__ __forceinline__ uint4 pk_load4(const uint32_t *p) {
  uint4 u;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "l"(p));
  return u;
}
__device__ __forceinline__ uint32_t pk_load(const uint32_t *p) {
  uint32_t u;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(u) : "l"(p));
  return u;
}
__device__ __forceinline__ uint64_t pk_load64(const uint64_t *p) {
  uint64_t u;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(u) : "l"(p));
  return u;
}
// tag: in the upper 16 bits
__device__ __forceinline__ bool pk_stale4(const uint4 &u, uint32_t tag) {
  return (((u.x ^ tag) | (u.y ^ tag) | (u.z ^ tag) | (u.w ^ tag)) & 0xffff0000u) != 0;
}
__device__ __forceinline__ uint2 pk_values4(const uint4 &u) { return make_uint2(__byte_perm(u.x, u.y, 0x5410), __byte_perm(u.z, u.w, 0x5410)); }
template <typename T> __device__ __forceinline__ void pk_store(uint32_t *p, T v, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(tag | (uint32_t)*reinterpret_cast<const uint16_t *>(&v)) : "memory");
}
__device__ __forceinline__ void pk_store64(uint64_t *p, float v, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((uint64_t)__float_as_uint(v) | (uint64_t)tag << 32) : "memory");
}
__device__ __forceinline__ float pk_poll64(const uint64_t *p, uint32_t tag, MkWait &w) {
  uint64_t u = pk_load64(p);
  while ((uint32_t)(u >> 32) != tag && w.again()) u = pk_load64(p);
  return __uint_as_float((uint32_t)u);
}
template <typename T> __device__ __forceinline__ T pk_value(uint32_t u) {
  const uint16_t h = (uint16_t)u;
  T r;
  *reinterpret_cast<uint16_t *>(&r) = h;
  return r;
}
template <typename T> __device__ __forceinline__ float4 pk_floats4(const uint4 &u) {
  const uint2 v = pk_values4(u);
  const float2 a = DT<T>::unpack2(v.x), b = DT<T>::unpack2(v.y);
  return make_float4(a.x, a.y, b.x, b.y);
}

// ---------------------------------------------------------------------------------------- consumers
// `meet`: all CTAs of the grid, once per layer (release: bar.sync + red.release; acquire: poll)
__device__ __forceinline__ void mk_grid_sync(unsigned long long *ctr, unsigned long long target, int ct, MkWait &w) {
  named_bar_sync(1, MK_CT);  // every consumer thread of this CTA has issued its global writes
  if (ct == 0) {
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(ctr), "l"(1ULL) : "memory");
    while (ld_acquire_u64(ctr) < target && w.again()) {
    }
  }
  named_bar_sync(1, MK_CT);
}

// ring hand-off: the previous shard pushes our input over NVLink and bumps the counter once per CTA
__device__ __forceinline__ void mk_inbox_wait(const unsigned long long *ctr, unsigned long long want, MkWait &w) {
  const int fast = w.left - MK_INBOX_FAST;
  while (true) {
    unsigned long long v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(ctr) : "memory");
    if (v >= want || !w.again()) return;
    if (w.left < fast) __nanosleep(8000);
  }
}

// x -> shared (D) and, where the phase keeps the residual stream, a second copy; returns this thread's share of the sum of squares.
// A thread's packets are MK_CT quads apart.  The first four are polled (16 KB per CTA); the others are asked for when those are there, six at a time:
// polling every packet of a long vector (57 KB per CTA for the 8B down product) would take the L2 bandwidth that the weights need.
template <typename T>
__device__ __forceinline__ float mk_gather(T *xs, T *keep, const uint32_t *pk, int K, uint32_t tag, int ct, MkWait &w) {
  const int nq = K >> 2;
  float ss = 0.f;
  auto put = [&](int q, const uint4 &u) {
    const uint2 v = pk_values4(u);
    *reinterpret_cast<uint2 *>(xs + 4 * q) = v;
    if (keep) *reinterpret_cast<uint2 *>(keep + 4 * q) = v;
    const float2 f0 = DT<T>::unpack2(v.x), f1 = DT<T>::unpack2(v.y);
    ss += f0.x * f0.x + f0.y * f0.y + f1.x * f1.x + f1.y * f1.y;
  };
  uint4 u[6];
  const int n4 = min(4, (nq - ct + MK_CT - 1) / MK_CT);  // (0 or less: this thread has none)
  if (n4 > 0) {
    bool stale;
    do {
      stale = false;
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (i < n4) u[i] = pk_load4(pk + 4 * (ct + i * MK_CT));
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (i < n4) stale = stale || pk_stale4(u[i], tag);
    } while (stale && w.again());
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (i < n4) put(ct + i * MK_CT, u[i]);
  }
#pragma unroll 1
  for (int q = ct + 4 * MK_CT; q < nq; q += 6 * MK_CT) {
    bool stale;
    do {
      stale = false;
#pragma unroll
      for (int i = 0; i < 6; i++)
        if (q + i * MK_CT < nq) u[i] = pk_load4(pk + 4 * (q + i * MK_CT));
#pragma unroll
      for (int i = 0; i < 6; i++)
        if (q + i * MK_CT < nq) stale = stale || pk_stale4(u[i], tag);
    } while (stale && w.again());
#pragma unroll
    for (int i = 0; i < 6; i++)
      if (q + i * MK_CT < nq) put(q + i * MK_CT, u[i]);
  }
  return ss;
}
// the same from a plain vector (the step's input: complete before the launch, or acquired from the inbox)
template <typename T>
__device__ __forceinline__ float mk_copy_x(T *xs, T *keep, const T *x, int K, int ct) {
  float ss = 0.f;
  for (int q = ct; q < K / 4; q += MK_CT) {
    const uint2 v = __ldcg(reinterpret_cast<const uint2 *>(x) + q);
    reinterpret_cast<uint2 *>(xs)[q] = v;
    if (keep) reinterpret_cast<uint2 *>(keep)[q] = v;
    const float2 f0 = DT<T>::unpack2(v.x), f1 = DT<T>::unpack2(v.y);
    ss += f0.x * f0.x + f0.y * f0.y + f1.x * f1.x + f1.y * f1.y;
  }
  return ss;
}

// the largest value of a warp and its index; the smaller index where values are equal
__device__ __forceinline__ void mk_warp_best(float &best, int &idx) {
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
  }
}

// acc += w[0] x[0] and w[1] x[1] of two packed 16-bit pairs: the fused multiply-add that takes 16-bit factors and a 32-bit sum (the product is exact, the
// sum is rounded once, as with both factors converted to fp32).  It issues at the rate of the 32-bit one (1.13 cycles against 1.10, eight chains),
// so the conversions are gone: 64 instructions for a stage's 8 vectors of a lane where there were 128 to 192.
template <typename T> __device__ __forceinline__ void mk_fma2(float &lo, float &hi, uint32_t w, uint32_t x);
template <> __device__ __forceinline__ void mk_fma2<__nv_bfloat16>(float &lo, float &hi, uint32_t w, uint32_t x) {
  asm("{\n\t.reg .b16 a, b, c, d;\n\tmov.b32 {a, b}, %2;\n\tmov.b32 {c, d}, %3;\n\tfma.rn.f32.bf16 %0, a, c, %0;\n\tfma.rn.f32.bf16 %1, b, d, %1;\n\t}"
      : "+f"(lo), "+f"(hi) : "r"(w), "r"(x));
}
template <> __device__ __forceinline__ void mk_fma2<__half>(float &lo, float &hi, uint32_t w, uint32_t x) {
  asm("{\n\t.reg .b16 a, b, c, d;\n\tmov.b32 {a, b}, %2;\n\tmov.b32 {c, d}, %3;\n\tfma.rn.f32.f16 %0, a, c, %0;\n\tfma.rn.f32.f16 %1, b, d, %1;\n\t}"
      : "+f"(lo), "+f"(hi) : "r"(w), "r"(x));
}
// 8 weights times x, into four running sums
template <typename T> __device__ __forceinline__ void mk_dot8(float (&acc)[4], const uint4 &w, const uint4 &x) {
  mk_fma2<T>(acc[0], acc[1], w.x, x.x);
  mk_fma2<T>(acc[2], acc[3], w.y, x.y);
  mk_fma2<T>(acc[0], acc[1], w.z, x.z);
  mk_fma2<T>(acc[2], acc[3], w.w, x.w);
}
__device__ __forceinline__ bool mk_ready(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return __all_sync(0xffffffffu, ok);
}

// bookkeeping that a launch keeps in the scratch area, as 64-bit words behind the 32 + 32 words of the reductions
constexpr int MK_START = 32;
// stamps of CTA 0 in the optional trace: 1 + 10 per layer: input gathered, output published of qkv, attention (begin, end), o, gate_up, down
__device__ __forceinline__ void mk_stamp(const MkArgs &a, int l, int ph, int end) {
  if (a.trace && blockIdx.x == 0 && threadIdx.x == 0) a.trace[1 + 10 * l + 2 * ph + (ph ? 2 : 0) + end] = mk_gtime();
}
template <typename T> __device__ __forceinline__ const T *mk_x_in(const MkArgs &a) {
  if (a.x_in) return reinterpret_cast<const T *>(a.x_in);
  uint32_t tok = *a.d_token;  // master: the block input is the embedding row of the current token (text_model.rs:271)
  if (tok >= (uint32_t)a.vocab) tok = 0;  // memory safety only: host entry points reject out-of-range ids (EINVAL); in-kernel argmax ids are < vocab
  return reinterpret_cast<const T *>(a.embed) + (size_t)tok * a.hidden;
}
// 4 values normed: (x * inv) * w, rounded to D
template <typename T> __device__ __forceinline__ uint2 mk_normed(const uint2 &x, const uint2 &w, float inv) {
  const float2 a = DT<T>::unpack2(x.x), b = DT<T>::unpack2(x.y), wa = DT<T>::unpack2(w.x), wb = DT<T>::unpack2(w.y);
  return make_uint2(pack2x<T>(a.x * inv * wa.x, a.y * inv * wa.y), pack2x<T>(b.x * inv * wb.x, b.y * inv * wb.y));
}

// end-of-step bookkeeping by one thread
__device__ __forceinline__ void mk_end_of_step(const MkArgs &a, const float *scratch) {
  if (a.advance) { *a.d_pos += 1; *a.d_step += 1; }
  if (a.inbox_ctr) *a.ring_seq += 1ULL;
  a.gbar[1] = reinterpret_cast<const unsigned long long *>(scratch)[MK_START] + (a.meet ? (unsigned long long)a.n_layers * gridDim.x : 0ULL);
  a.gbar[2] += (unsigned long long)a.n_layers;
}

// the greedy token, by the CTA that is last
__device__ __forceinline__ void mk_head_end(const MkArgs &a, float *scratch, float best, int bidx) {
  const int ct = threadIdx.x, warp = ct >> 5, lane = ct & 31;
  mk_warp_best(best, bidx);
  int *scratch_i = reinterpret_cast<int *>(scratch + 32);
  if (lane == 0) { scratch[warp] = best; scratch_i[warp] = bidx; }
  named_bar_sync(1, MK_CT);
  if (warp != 0) return;
  // a lane per warp's best, then (the CTA that arrives last) the CTAs' bests, 32 at a time: for one thread both are chains of round trips
  best = lane < MK_CW ? scratch[lane] : -INFINITY;
  bidx = lane < MK_CW ? scratch_i[lane] : 0x7fffffff;
  mk_warp_best(best, bidx);
  unsigned ticket = 0;
  if (lane == 0) {
    a.part_val[blockIdx.x] = best;
    a.part_idx[blockIdx.x] = bidx;
    __threadfence();
    ticket = atomicAdd(a.argmax_counter, 1u);
  }
  ticket = __shfl_sync(0xffffffffu, ticket, 0);
  if (ticket != gridDim.x - 1) return;
  __threadfence();
  best = -INFINITY;
  bidx = 0x7fffffff;
#pragma unroll 1
  for (unsigned c = lane; c < gridDim.x; c += 32) {
    const float v = __ldcg(a.part_val + c);
    const int i = __ldcg(a.part_idx + c);
    if (v > best || (v == best && i < bidx)) { best = v; bidx = i; }
  }
  mk_warp_best(best, bidx);
  if (lane == 0) {
    *a.token_out = (uint32_t)bidx;
    if (a.token_ring) a.token_ring[*a.d_step % a.ring_cap] = (uint32_t)bidx;
    *a.argmax_counter = 0;
    a.tickets[MK_HEAD_TICKET] = 0;   // every CTA's producer has seen the end of the pool.  (A memset node in front of the kernel took 2.5 us of a 50 us head.)
    mk_end_of_step(a, scratch);  // this is the last CTA of the grid to finish
  }
}

// one product of the step: input gathered, staged rows, fused epilogue, packets out.  What only one end of it needs is worked out there: values that
// live across the loop over the stages cost registers that the loop needs.
template <typename T>
__device__ __forceinline__ void mk_gemv_phase(MkRing &rg, const MkArgs &a, unsigned char *sm, int l, int ph, uint32_t tag, int &left) {
  const int ct = threadIdx.x, warp = ct >> 5, lane = ct & 31;
  const bool head = l == a.n_layers;
  const MkGeom &g = a.g[head ? 4 : ph];
  T *xs = reinterpret_cast<T *>(sm + a.off_x), *res_s = reinterpret_cast<T *>(sm + a.off_res);
  float *partial = reinterpret_cast<float *>(sm + a.off_part), *scratch = reinterpret_cast<float *>(sm + MK_OFF_SCRATCH);
  int *loc_row = reinterpret_cast<int *>(sm + a.off_loc);
  const MkRow &L = reinterpret_cast<const MkRow *>(sm + a.off_rows)[head ? 0 : l];  // (not read for the head)
  const int RSL = g.RSL, nchunk = g.nchunk;
  const bool norm = head || ph == 0 || ph == 2;
  // ---- input
  const T *norm_w = reinterpret_cast<const T *>(head ? a.ln_f : !norm ? nullptr : ph == 0 ? L.ln1 : L.ln2);
  uint2 nw[4];  // this thread's norm weights, asked for before the input is waited for
  if (norm) {
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (ct + i * MK_CT < g.K / 4) nw[i] = reinterpret_cast<const uint2 *>(norm_w)[ct + i * MK_CT];
  }
  {
    T *keep = a.keep_x && norm && !head ? res_s : nullptr;
    MkWait w{left, a.err};
    float ss;
    if (l == 0 && ph == 0) {
      ss = mk_copy_x<T>(xs, keep, mk_x_in<T>(a), g.K, ct);
    } else {
      const uint32_t *in = ph == 0 ? a.pk.xa : ph == 1 ? a.pk.y : ph == 2 ? a.pk.xb : a.pk.mm;
      ss = mk_gather<T>(xs, keep, in, g.K, ph == 0 ? tag - 0x10000u : tag, ct, w);
    }
    if (norm) {
      ss = warp_sum(ss);
      if (lane == 0) scratch[warp] = ss;
    }
    named_bar_sync(1, MK_CT);
    if (a.meet && ph == 3) mk_grid_sync(a.gbar, reinterpret_cast<unsigned long long *>(scratch)[MK_START] + (unsigned long long)(l + 1) * gridDim.x, ct, w);
    left = w.left;
  }
  if (norm) {  // each thread the values it gathered
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < MK_CW / 4; i++) {
      const float4 f = reinterpret_cast<const float4 *>(scratch)[i];
      tot += (f.x + f.y) + (f.z + f.w);
    }
    const float inv = 1.0f / sqrtf(tot / (float)g.K + a.eps);
    uint2 *xq = reinterpret_cast<uint2 *>(xs);
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (ct + i * MK_CT < g.K / 4) xq[ct + i * MK_CT] = mk_normed<T>(xq[ct + i * MK_CT], nw[i], inv);
#pragma unroll 1
    for (int q = ct + 4 * MK_CT; q < g.K / 4; q += MK_CT) xq[q] = mk_normed<T>(xq[q], reinterpret_cast<const uint2 *>(norm_w)[q], inv);
    named_bar_sync(1, MK_CT);
  }
  mk_stamp(a, l, ph, 0);
  // ---- staged rows.  A warp takes two rows of 16, one of 8, or one and the other 8 / RS - 1 warps of its row a part of the columns each: at most
  // 8 vectors of 16 bytes a lane, 32 lanes side by side.  A lane's columns are the same for every stage: its x stays in registers.
  const bool pool = g.pool < g.n_groups, two = RSL == 4;
  const int wl = max(3 - RSL, 0), ks = warp & ((1 << wl) - 1), slot = warp >> wl;
  const int segv = g.KC / 8, nv = segv >> wl;
  const int cnt = (nv - lane + 31) >> 5;                  // this lane's vectors of a row
  const uint4 *xsv = reinterpret_cast<const uint4 *>(xs) + ks * nv + lane;
  const int at = slot * segv + ks * nv + lane, at4 = two ? at + 8 * segv : at + 128;   // the first four vectors, the other four (of a second row, if two)
  const uint4 z = make_uint4(0u, 0u, 0u, 0u);
  float best = -INFINITY;  // (head)
  int bidx = 0x7fffffff;
  const int kind = (pool ? 1 : 0) | (nchunk > 1 ? 2 : 0) | (two ? 4 : 0);
  int base = mk_first(g), left_groups = mk_count(g);
  bool more = true;
#pragma unroll 1
  while (more) {
    int n_groups = pool ? g.batch : min(g.batch, left_groups);
    left_groups -= n_groups;
    more = pool || left_groups > 0;
    const int n_stages = n_groups * nchunk;
    uint4 x[8], w[8];
    auto load_x = [&](const uint4 *xv) {
#pragma unroll
      for (int i = 0; i < 8; i++) x[i] = i < cnt ? xv[32 * i] : z;   // (two rows: at most four vectors)
    };
    // A stage is read half by half, the halves of the next stage (if it is there) as soon as the registers are free, so that the reads,
    // the products and the sums over the lanes of neighbouring stages overlap.
    auto load_a = [&](const uint4 *st) {
#pragma unroll
      for (int i = 0; i < 4; i++) w[i] = i < cnt ? st[at + 32 * i] : z;
    };
    auto load_b = [&](const uint4 *st) {
#pragma unroll
      for (int i = 0; i < 4; i++) w[4 + i] = (two ? i : i + 4) < cnt ? st[at4 + 32 * i] : z;
    };
    load_x(xsv);
    int k = 0;
    bool ready = false;   // the halves of stage i are already requested
#pragma unroll 1
    for (int i = 0; i < n_stages; i++) {
      int what = kind;  // (opaque: the compiler else writes the loop out once per kind, and the phases no longer fit the instruction cache)
      asm volatile("" : "+r"(what));
      if (!ready) {
        mbar_wait(rg.full(), rg.ph);
        const uint4 *st = reinterpret_cast<const uint4 *>(rg.data());
        load_a(st);
        load_b(st);
      }
      if (what & 1) {
        const int row = rg.row();
        if (row < 0) {
          __syncwarp();
          if (lane == 0) mbar_arrive(rg.empty());
          rg.advance();
          n_groups = i;
          more = false;
          break;
        }
        if (ct == 0) loc_row[i] = row;
      }
      if (what & 2) {  // the columns change from stage to stage
        load_x(xsv + k * segv);
        if (++k == nchunk) k = 0;
      }
      uint64_t *const done = rg.empty();
      rg.advance();
      ready = i + 1 < n_stages && mk_ready(rg.full(), rg.ph);
      const uint4 *st = reinterpret_cast<const uint4 *>(rg.data());
      float a0[4] = {0.f, 0.f, 0.f, 0.f}, a1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 4; c++) mk_dot8<T>(a0, w[c], x[c]);
      if (ready) load_a(st);
      if (what & 4) {
#pragma unroll
        for (int c = 0; c < 4; c++) mk_dot8<T>(a1, w[4 + c], x[c]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; c++) mk_dot8<T>(a1, w[4 + c], x[4 + c]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(done);
      if (ready) load_b(st);
      float s0 = (a0[0] + a0[1]) + (a0[2] + a0[3]);
      const float s1 = (a1[0] + a1[1]) + (a1[2] + a1[3]);
      float *pt = partial + (((i << RSL) + slot) << wl) + ks;
      if (what & 4) {  // two rows: half of the lanes for each
        const bool up = lane & 16;
        s0 = (up ? s1 : s0) + __shfl_xor_sync(0xffffffffu, up ? s0 : s1, 16);
      } else {
        s0 += s1;
        s0 += __shfl_xor_sync(0xffffffffu, s0, 16);
      }
#pragma unroll
      for (int o = 8; o; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      if ((lane & 15) == 0 && (lane == 0 || (what & 4))) pt[lane ? 8 : 0] = s0;  // (rows past N: never read)
    }
    named_bar_sync(1, MK_CT);
    const int n_local = n_groups << RSL;
    auto row_sum = [&](int li) {
      const float *p = partial + (li * nchunk << wl);
      float sum = p[0];
      if (wl > 0) {
        sum += p[1];
        if (wl > 1) {
          sum += p[2] + p[3];
          if (wl > 2) sum += (p[4] + p[5]) + (p[6] + p[7]);
        }
      }
#pragma unroll 1
      for (int i = 1 << wl; i < nchunk << wl; i++) sum += p[i];
      return rnd<T>(sum);
    };
#pragma unroll 1
    for (int li = ct << (ph == 2); li < n_local; li += MK_CT << (ph == 2)) {  // a row, or a gate and an up row
      const int row = pool ? loc_row[li >> RSL] + (li & ((1 << RSL) - 1)) : (base << RSL) + li;
      if (row >= g.N) continue;
      int what = head ? 4 : ph;
      asm volatile("" : "+r"(what));
      float v = row_sum(li);
      if (what == 4) {
        if (a.logits) reinterpret_cast<T *>(a.logits)[row] = DT<T>::from_f(v);
        if (v > best || (v == best && row < bidx)) { best = v; bidx = row; }  // first maximum wins
      } else if (what == 0) {
        if (L.bqkv) v = rnd<T>(v + DT<T>::to_f(reinterpret_cast<const T *>(L.bqkv)[row]));
        pk_store<T>(a.pk.qkv + row, DT<T>::from_f(v), tag);
      } else if (what == 2) {
        const float up = row_sum(li + 1);
        pk_store<T>(a.pk.mm + row / 2, DT<T>::from_f(gate_act<T>(v, a.act) * up), tag);
      } else {  // + residual
        T q;
        if (a.keep_x) q = res_s[row];
        else if (what == 1 && l == 0) q = ldcg_T<T>(mk_x_in<T>(a) + row);
        else q = pk_value<T>(pk_load((what == 1 ? a.pk.xa : a.pk.xb) + row));  // (gathered by this CTA before)
        const T o = DT<T>::from_f(v + DT<T>::to_f(q));
        pk_store<T>((what == 1 ? a.pk.xb : a.pk.xa) + row, o, tag);
        if (what == 3 && l == a.n_layers - 1 && a.x_out) reinterpret_cast<T *>(a.x_out)[row] = o;
      }
    }
    base += n_groups;
    if (more) named_bar_sync(1, MK_CT);  // the batch has been taken
  }
  if (head) mk_head_end(a, scratch, best, bidx);
  mk_stamp(a, l, ph, 1);
}

// Sum G per-lane values over the 16 lanes of a half-warp with a halving butterfly: after log2(G) exchange
// steps every lane owns ONE head's partial, then the remaining xor steps finish it.  G + log2(16/G) - 1
// shuffles instead of 4*G.  Returns the sum for head `g_out` (valid on every lane of the half-warp).
template <int G>
__device__ __forceinline__ float reduce16_heads(float (&s)[G], int lane, int &g_out) {
  int g = 0;
  int bit = 8;
#pragma unroll
  for (int n = G; n > 1; n >>= 1) {
    const bool upper = (lane & bit) != 0;
#pragma unroll
    for (int i = 0; i < n / 2; i++) {
      const float keep = upper ? s[i + n / 2] : s[i];
      const float send = upper ? s[i] : s[i + n / 2];
      s[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
    if (upper) g += n / 2;
    bit >>= 1;
  }
  float v = s[0];
#pragma unroll
  for (int b2 = 8; b2 >= 1; b2 >>= 1)
    if (b2 <= bit) v += __shfl_xor_sync(0xffffffffu, v, b2);
  g_out = g;
  return v;
}

// norm_rope_inplace with the position's cos/sin row already staged in shared memory as fp32 (D values); a lane holds its norm weights
template <typename T, int HD>
__device__ __forceinline__ void mk_norm_rope(float *buf, bool norm, const float (&w)[(HD + 31) / 32], float eps, const float *cs, const float *sn, int rot, int lane) {
  if (norm) {
    float ss = 0.f;
    for (int d = lane; d < HD; d += 32) ss += buf[d] * buf[d];
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)HD + eps);
#pragma unroll
    for (int i = 0; i < (HD + 31) / 32; i++)
      if (lane + 32 * i < HD) buf[lane + 32 * i] = rnd<T>(buf[lane + 32 * i] * inv * w[i]);
    __syncwarp();
  }
  const int half = rot / 2;
  for (int i = lane; i < half; i += 32) {
    const float c = cs[i], s = sn[i];
    const float x1 = buf[i], x2 = buf[i + half];
    buf[i] = rnd<T>(rnd<T>(x1 * c) - rnd<T>(x2 * s));
    buf[i + half] = rnd<T>(rnd<T>(x2 * c) + rnd<T>(x1 * s));
  }
  __syncwarp();
}

// Attention phase for this CTA's (kv head, split) item.  Same math as attn_decode_kernel (f32 scores,
// softmax and PV, one rounding of the result); K/V tiles come from the ring, prefetched by the producer while
// the qkv GEMV was still running.  G = n_heads / n_kv_heads is a template parameter so that all per-head
// state lives in registers.  The heads' packets are polled by the warps that norm and rotate them.  One split: its result is the output.
// Several: each publishes its columns, maximum and sum as packets, and each merges its share of the columns of all of them, in split order.
template <typename T, int HD, int G>
__device__ __forceinline__ void mk_consume_attn(MkRing &rg, const MkArgs &a, const MkRow &L, int pos, unsigned char *scr, float *parts,
                                                const float *rope_cs, uint32_t tag32, int &left, unsigned long long *tr) {
  const int ct = threadIdx.x, warp = ct >> 5, lane = ct & 31;
  const uint32_t tag = tag32 << 16;
  MkWait wt{left, a.err};
  auto stamp = [&](int i) {
    if (tr && ct == 0) tr[i] = mk_gtime();
  };
  stamp(0);
  constexpr int LPR = HD / 8;            // lanes per cached row (16 B each); HD in {16,64,128} -> 2, 8, 16
  constexpr int RPWI = 32 / LPR;         // rows per warp per iteration
  constexpr int NW = MK_CW;
  static_assert(HD == 16 || HD == 64 || HD == 128, "head_dim");
  // sliding window (cache.rs:173-205): rows below ws = pos + 1 - window are invisible; indices below are relative to ws
  const int ws = (a.window > 0 && pos + 1 > a.window) ? pos + 1 - a.window : 0;
  pos -= ws;
  const MkAttnItem it = mk_attn_item(a, pos, (int)sizeof(T));
  float *q_s = reinterpret_cast<float *>(scr);             // [G][HD]
  float *sc = q_s + ATTN_MAX_G * 256;                      // [ATTN_TILE][G]  (position-major: one vector per position)
  float *knew = sc + ATTN_MAX_G * ATTN_TILE;               // [2][HD] appended k / v row
  __shared__ float m_run[ATTN_MAX_G], l_run[ATTN_MAX_G], fac[ATTN_MAX_G];
  __shared__ float wgt[ATTN_MAX_G][ATTN_MAX_SPLIT];
  if (!it.active) return;  // CTA-uniform; inactive CTAs issue no stages either

  const float *cosr = rope_cs, *sinr = rope_cs + 128;  // this step's cos/sin row, staged once per launch
  T *kc = reinterpret_cast<T *>(L.kc) + ((size_t)it.kvh * a.cap + ws) * HD;
  T *vc = reinterpret_cast<T *>(L.vc) + ((size_t)it.kvh * a.cap + ws) * HD;
  const int kvh = it.kvh, split = it.split, s0 = it.s0, s1 = it.s1, TILE = it.tile;
  const bool owner = (pos >= s0 && pos < s1);

  // q of the G heads of this kv head, a warp each; in the split that holds the position the new key and value too
#pragma unroll 1
  for (int h = warp; h < (owner ? G + 2 : G); h += NW) {
    const bool is_q = h < G, is_k = h == G;
    float nw[(HD + 31) / 32];
    const T *norm_w = reinterpret_cast<const T *>(is_q ? L.qn : is_k ? L.kn : nullptr);
#pragma unroll
    for (int i = 0; i < (HD + 31) / 32; i++) nw[i] = norm_w && lane + 32 * i < HD ? DT<T>::to_f(norm_w[lane + 32 * i]) : 0.f;
    const int head = is_q ? kvh * G + h : is_k ? a.n_heads + kvh : a.n_heads + a.n_kv + kvh;
    float *dst = is_q ? q_s + h * HD : is_k ? knew : knew + HD;
    if (lane < HD / 4) {
      const uint32_t *src = a.pk.qkv + (size_t)head * HD + lane * 4;
      uint4 u = pk_load4(src);
      while (pk_stale4(u, tag) && wt.again()) u = pk_load4(src);
      *reinterpret_cast<float4 *>(dst + lane * 4) = pk_floats4<T>(u);
    }
    __syncwarp();
    if (is_q || is_k) mk_norm_rope<T, HD>(dst, norm_w != nullptr, nw, a.eps, cosr, sinr, a.rot, lane);
    if (!is_q) {
      T *row = is_k ? kc : vc;
      for (int d = lane; d < HD; d += 32) row[(size_t)pos * HD + d] = DT<T>::from_f(dst[d]);
    }
  }
  if (ct < ATTN_MAX_G) { m_run[ct] = -INFINITY; l_run[ct] = 0.f; }
  named_bar_sync(1, MK_CT);
  stamp(1);

  const int grp = lane / LPR, gl = lane % LPR;  // row group within the warp / lane within the row
  uint4 qreg[G];  // (D values: exact)
#pragma unroll
  for (int g = 0; g < G; g++) {
    const float *q = q_s + g * HD + gl * 8;
    qreg[g] = make_uint4(pack2x<T>(q[0], q[1]), pack2x<T>(q[2], q[3]), pack2x<T>(q[4], q[5]), pack2x<T>(q[6], q[7]));
  }
  float acc[G][8];  // PV accumulator: dims gl*8..+8 of every head, over this half-warp's positions
#pragma unroll
  for (int g = 0; g < G; g++)
#pragma unroll
    for (int i = 0; i < 8; i++) acc[g][i] = 0.f;

  T *Ks = nullptr, *Vs = nullptr;
  uint64_t *ek = nullptr, *ev = nullptr;
  for (int t0 = s0; t0 < s1; t0 += TILE) {
    const int tn = min(TILE, s1 - t0);
    if (t0 > s0) {  // release the previous tile's stages (the last tile's are kept for the final reduction)
      __syncwarp();
      if (lane == 0) { mbar_arrive(ek); mbar_arrive(ev); }
    }
    ek = rg.empty();
    Ks = reinterpret_cast<T *>(rg.data());
    mbar_wait(rg.full(), rg.ph);
    rg.advance();
    ev = rg.empty();
    Vs = reinterpret_cast<T *>(rg.data());
    mbar_wait(rg.full(), rg.ph);
    rg.advance();
    stamp(2);
    if (owner && pos >= t0 && pos < t0 + tn) {  // drop the appended row into its slot of the staged tiles
      const int slot = pos - t0;
      for (int d = ct; d < HD; d += MK_CT) {
        Ks[(size_t)slot * HD + d] = DT<T>::from_f(knew[d]);
        Vs[(size_t)slot * HD + d] = DT<T>::from_f(knew[HD + d]);
      }
    }
    named_bar_sync(1, MK_CT);
    // ---- scores: s[p][g] = (q_g . k_p) * scale, f32 ----------------------------------------------
    for (int pb = warp * RPWI; pb < tn; pb += NW * RPWI) {  // warp-uniform trip count (shuffles below)
      const int p = pb + grp;
      const bool valid = p < tn;
      uint4 kraw = make_uint4(0u, 0u, 0u, 0u);
      if (valid) kraw = *reinterpret_cast<const uint4 *>(Ks + (size_t)p * HD + gl * 8);
      float sg[G];
#pragma unroll
      for (int g = 0; g < G; g++) {
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
        mk_dot8<T>(s4, kraw, qreg[g]);
        sg[g] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
      }
      if (LPR == 16) {
        int gh;
        const float v = reduce16_heads<G>(sg, lane, gh);
        constexpr int FIN = (G >= 8) ? 1 : (G == 4 ? 3 : (G == 2 ? 7 : 15));  // lanes that hold a finished head
        if (valid && (gl & FIN) == 0) sc[p * G + gh] = v * a.scale;
      } else {
#pragma unroll
        for (int g = 0; g < G; g++) {
          float v = sg[g];
#pragma unroll
          for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (gl == 0 && valid) sc[p * G + g] = v * a.scale;
        }
      }
    }
    named_bar_sync(1, MK_CT);
    stamp(3);
    // ---- online softmax bookkeeping, one warp per head ---------------------------------------------
    for (int g = warp; g < G; g += NW) {
      float mx = -INFINITY;
      for (int p = lane; p < tn; p += 32) mx = fmaxf(mx, sc[p * G + g]);
      mx = warp_max(mx);
      const float m_new = fmaxf(m_run[g], mx);
      float sum = 0.f;
      for (int p = lane; p < tn; p += 32) {
        const float ev = expf(sc[p * G + g] - m_new);
        sc[p * G + g] = ev;
        sum += ev;
      }
      sum = warp_sum(sum);
      if (lane == 0) {
        const float f = (m_run[g] == -INFINITY) ? 0.f : expf(m_run[g] - m_new);
        fac[g] = f;
        l_run[g] = l_run[g] * f + sum;
        m_run[g] = m_new;
      }
    }
    named_bar_sync(1, MK_CT);
    stamp(4);
    // ---- PV: a lane owns dims gl*8..+8 of every head; one 16-byte V load feeds 8*G FMAs ------------
#pragma unroll
    for (int g = 0; g < G; g++) {
      const float f = fac[g];
#pragma unroll
      for (int i = 0; i < 8; i++) acc[g][i] *= f;
    }
    for (int p = warp * RPWI + grp; p < tn; p += NW * RPWI) {
      float vf[8];
      unpack8<T>(*reinterpret_cast<const uint4 *>(Vs + (size_t)p * HD + gl * 8), vf);
#pragma unroll
      for (int g = 0; g < G; g++) {
        const float ev = sc[p * G + g];
#pragma unroll
        for (int i = 0; i < 8; i++) acc[g][i] = fmaf(ev, vf[i], acc[g][i]);
      }
    }
    named_bar_sync(1, MK_CT);  // every warp is done with this tile's K, V and probabilities
    stamp(5);
  }

  // ---- combine the row groups: lanes of a warp first (shuffles), then the warps through the (dead)
  //      K stage of the last tile (an active split has at least one position, so there is one) -------------------------------
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1)
#pragma unroll
    for (int g = 0; g < G; g++)
#pragma unroll
      for (int i = 0; i < 8; i++) acc[g][i] += __shfl_xor_sync(0xffffffffu, acc[g][i], o);
  float *red = reinterpret_cast<float *>(Ks);  // [warp][G][HD] <= 32 KB
  static_assert(NW * ATTN_MAX_G * 128 * 4 <= MK_STAGE_BYTES, "the warps' sums");
  if (lane < LPR) {
    float *dst = red + (size_t)warp * G * HD;
#pragma unroll
    for (int g = 0; g < G; g++)
#pragma unroll
      for (int i = 0; i < 8; i++) dst[g * HD + lane * 8 + i] = acc[g][i];
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // what was written into the stages (these sums, the appended row) comes before the next copy into them
  named_bar_sync(1, MK_CT);
  const int ns = it.n_split;
  uint64_t *pacc = a.pk.acc + (size_t)kvh * G * HD * a.nsplit, *pml = a.pk.ml + (size_t)kvh * G * a.nsplit * 2;  // [column][split], [head][split][2]
  for (int i = ct; i < G * HD; i += MK_CT) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < NW; w++) sum += red[(size_t)w * G * HD + i];
    if (ns == 1) pk_store<T>(a.pk.y + (size_t)kvh * G * HD + i, DT<T>::from_f(sum * (1.0f / l_run[i / HD])), tag);
    else pk_store64(pacc + (size_t)i * ns + split, sum, tag32);
  }
  if (ns > 1 && ct < G) {
    pk_store64(pml + ((size_t)ct * ns + split) * 2, m_run[ct], tag32);
    pk_store64(pml + ((size_t)ct * ns + split) * 2 + 1, l_run[ct], tag32);
  }
  __syncwarp();
  named_bar_sync(1, MK_CT);
  if (lane == 0) { mbar_arrive(ek); mbar_arrive(ev); }
  stamp(6);
  if (ns > 1) {
    // ---- merge: this split's share of the columns; (column, split) pairs are contiguous, a thread polls one or a few of them.  The first warps have all
    // columns: the others gather the o product's input (over scr) while these still read `parts` and `wgt`.
    static_assert(G * HD + ATTN_MAX_SPLIT <= MK_BATCH * MK_CW, "the parts of a merge");
    const int c0 = G * HD * split / ns, nc = G * HD * (split + 1) / ns - c0, np = nc * ns;
    for (int i = ct; i < np; i += MK_CT) parts[i] = pk_poll64(pacc + (size_t)c0 * ns + i, tag32, wt);
    for (int g = warp; g < G; g += NW) {
      float m = -INFINITY, l = 0.f;
      if (lane < ns) {
        m = pk_poll64(pml + ((size_t)g * ns + lane) * 2, tag32, wt);
        l = pk_poll64(pml + ((size_t)g * ns + lane) * 2 + 1, tag32, wt);
      }
      const float M = warp_max(m);
      const float w = (m == -INFINITY) ? 0.f : expf(m - M);
      const float Lsum = warp_sum(w * l);
      wgt[g][lane] = w / Lsum;
    }
    named_bar_sync(1, MK_CT);
    for (int i = ct; i < nc; i += MK_CT) {
      const int g = (c0 + i) / HD;
      float o = 0.f;
      for (int s2 = 0; s2 < ns; s2++) o = fmaf(wgt[g][s2], parts[i * ns + s2], o);
      pk_store<T>(a.pk.y + (size_t)kvh * G * HD + c0 + i, DT<T>::from_f(o), tag);
    }
  }
  left = wt.left;
  stamp(7);
}

// ---------------------------------------------------------------------------------------- the kernel
template <typename T, int HD, int G>
__global__ void __launch_bounds__(MK_THREADS, 1) decode_mega_kernel(const __grid_constant__ MkArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr int es = sizeof(T);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.n_stages; s++) {
      mbar_init(reinterpret_cast<uint64_t *>(smem_raw) + s, 1);
      mbar_init(reinterpret_cast<uint64_t *>(smem_raw + MK_OFF_EMPTY) + s, MK_CW);
    }
    mbar_fence_init();
  }
  __syncthreads();
  const int pos = a.n_layers ? *a.d_pos : 0;
  MkRing rg{smem_raw, a.n_stages, 0, 0u};

  if (warp == MK_CW) {
    // ================= producer: stream weights and K/V tiles through the whole phase list ==========
    if (lane == 0) {
      const uint64_t pol_w = policy_evict_first(), pol_kv = policy_evict_last();
#pragma unroll 1
      for (int l = 0; l <= a.n_layers; l++) {
        if (l == a.n_layers && !a.has_head) break;
        const MkLayer &L = a.layers[l];  // (not read for the head)
        if (l < a.n_layers) {  // norm weights: one cache line each, into L2 before a consumer asks
          const int b = blockIdx.x * 128;
          if (b < a.hidden * es) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(L.ln1) + b));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(L.ln2) + b));
          }
          if (L.qn && b < HD * es) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(L.qn) + b));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(L.kn) + b));
          }
        }
#pragma unroll 1
        for (int ph = 0; ph < 4; ph++) {
          const bool head = l == a.n_layers;
          const MkGeom &g = a.g[head ? 4 : ph];
          const void *W = head ? a.lm_head : ph == 0 ? L.wqkv : ph == 1 ? L.wo : ph == 2 ? L.wgu : L.wd;
          mk_produce_gemv<T>(rg, g, W, a.tickets + (head ? MK_HEAD_TICKET : 4 * l + ph), pol_w);
          if (head) break;
          if (ph == 0) mk_produce_attn<T>(rg, a, L, pos, pol_kv);
        }
      }
    }
    return;
  }

  // ================= consumers ========================================================================
  // A launch without layers is placed while the kernel in front ends (launch_mega), and its producer streams the static rows meanwhile.
  pdl_wait();
  const int ct = threadIdx.x;
  __shared__ float rope_cs[256];  // cos (first 128) and sin (last 128) row of this step's position, as fp32
  {
    const int half = a.n_layers ? a.rot / 2 : 0;
    const T *cr = reinterpret_cast<const T *>(a.cos_t) + (size_t)pos * half, *sr = reinterpret_cast<const T *>(a.sin_t) + (size_t)pos * half;
    if (ct < half) rope_cs[ct] = DT<T>::to_f(cr[ct]);
    else if (ct >= 128 && ct - 128 < half) rope_cs[ct] = DT<T>::to_f(sr[ct - 128]);
    MkRow *rows = reinterpret_cast<MkRow *>(smem_raw + a.off_rows);
    for (int l = ct; l < a.n_layers; l += MK_CT) {
      const MkLayer &L = a.layers[l];
      rows[l] = MkRow{L.ln1, L.ln2, L.bqkv, L.qn, L.kn, L.kc, L.vc};
    }
    // gbar[0] is a monotonic arrival counter; gbar[1] holds its value at the start of this launch (written
    // by the previous launch's last thread), so barrier k of this launch completes at start + k*grid.
    if (ct == 0) reinterpret_cast<unsigned long long *>(smem_raw + MK_OFF_SCRATCH)[MK_START] = *reinterpret_cast<volatile unsigned long long *>(a.gbar + 1);
    named_bar_sync(1, MK_CT);
  }
  // the tag of layer l's packets is first + l; a buffer is written in every layer, so what is stale in it carries the tag in front
  const uint32_t first = (uint32_t)*reinterpret_cast<volatile unsigned long long *>(a.gbar + 2) + 1u;
  int left = a.polls;
  if (a.trace && blockIdx.x == 0 && ct == 0) a.trace[0] = mk_gtime();
  unsigned long long *const st_rec = (a.step_trace && blockIdx.x == 0 && ct == 0)
      ? a.step_trace + ((size_t)((unsigned)*a.d_step % MK_STEP_RING) * 2 + a.trace_tag) * 4 : nullptr;
  if (st_rec) st_rec[0] = mk_gtime();
  if (a.inbox_ctr) {
    if (ct == 0) {
      MkWait w{a.inbox_polls, a.err};
      mk_inbox_wait(a.inbox_ctr, (*reinterpret_cast<volatile unsigned long long *>(a.ring_seq) + 1ULL) * gridDim.x, w);
    }
    named_bar_sync(1, MK_CT);
  }
  if (st_rec) st_rec[1] = mk_gtime();
  // One loop over the phases and one body for the products: as straight-line code of five products the layer's instructions were fetched anew in
  // every phase.
#pragma unroll 1
  for (int l = 0; l <= a.n_layers; l++) {
    if (l == a.n_layers && !a.has_head) break;
    const uint32_t tag32 = first + (uint32_t)l;
#pragma unroll 1
    for (int ph = 0; ph < 4; ph++) {
      mk_gemv_phase<T>(rg, a, smem_raw, l, ph, tag32 << 16, left);
      if (l == a.n_layers) break;
      if (ph == 0) {  // qk-norm, RoPE, KV append, attention
        mk_stamp(a, l, 0, 2);
        mk_consume_attn<T, HD, G>(rg, a, reinterpret_cast<const MkRow *>(smem_raw + a.off_rows)[l], pos, smem_raw + a.off_x,
                                  reinterpret_cast<float *>(smem_raw + a.off_part), rope_cs, tag32, left,
                                  a.trace && blockIdx.x == 0 && l == 1 ? a.trace + 2048 : nullptr);
        mk_stamp(a, l, 0, 3);
      }
    }
  }
  if (a.peer_ctr && !a.has_head) {  // our rows of x_out are in the next shard's inbox: release them, one arrival per CTA
    named_bar_sync(1, MK_CT);
    if (ct == 0) {
      __threadfence_system();
      asm volatile("red.release.sys.global.add.u64 [%0], %1;" ::"l"(a.peer_ctr), "l"(1ULL) : "memory");
    }
  }
  if (st_rec) st_rec[2] = mk_gtime();
  // bookkeeping without a head: CTA 0 has gathered the last product's input, so every CTA has published something in this launch (mk_every_cta,
  // or all have met), and every CTA read *d_pos, *ring_seq, the barrier start value and the tag before it did.
  if (!a.has_head && blockIdx.x == 0 && ct == 0) mk_end_of_step(a, reinterpret_cast<const float *>(smem_raw + MK_OFF_SCRATCH));
}

// The decode kernel for a data type, head size and number of query heads per key head; nullptr: no instance (decode_mega.cu)
const void *mk_kernel(int dtype, int head_dim, int group);
// test aid: each kind of wait of the decode kernel on words of its own, twice by the same threads; fresh: what it waits for is there.
// out[i]: whether wait i ended by that, out[2 + i]: its kcycles (thread 0)
cudaError_t mk_wait_probe(cudaStream_t, int what, int fresh, int polls, int *err, int *out);

}  // namespace cake
