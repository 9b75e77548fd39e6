// Whole HMC iterations, leapfrog trajectories and single evaluations of a window whose rows fit on the chip, as
// ONE launch: rows, weights, momenta and gradients stay in shared memory, tensor memory and registers from the
// first step to the last.
//
// Why.  With one launch per leapfrog step the step of a single 58368-row window takes 12.0 us (TF32) although its
// arithmetic needs about 1 us: what counts are the launches, the re-reading and re-staging of the rows, the partial
// vectors' trip through a second launch and the accept launch.  Here a step is one pass over rows that are already
// where the tensor core reads them, plus an exchange of sums and weights between the CTAs of the window.
//
// Work split.  A window's rows are dealt in units of 32 (a warp's) to K clusters of C CTAs, at most 16 units per
// CTA (four warpgroups of four warps), so that nothing is loaded after the first step.
//
// Exchange.  Parameters travel in words of three, 322 of them for 961 parameters; word i belongs to rank
// i / wpm of every cluster, where C lanes work on it:
//   1. every CTA sends its sums for a word to the owner in its cluster (st.async into the owner's shared memory,
//      counted by the owner's mbarrier); lane l of the word reads rank l's, a shuffle tree adds them;
//   2. K > 1: the owner stores the cluster's sums through L2 in a 16-byte word {3 sums, sequence number}, and the
//      rank's threads read the words of all clusters, consecutive threads consecutive words (with every lane reading
//      the words it adds, 15 clusters needed 2,970 cycles for this hop instead of 1,870: what counts is the number
//      of L2 requests while everybody polls).  A word is written and read by single 16-byte accesses, which the memory model
//      keeps whole, so there is no flag, no fence and no grid-wide barrier.  Words alternate between two buffers:
//      a cluster sends step s + 2 only after it has read every word of step s + 1, which the others send after
//      they have read every word of step s;
//   3. every lane does the leapfrog update of its word's parameters (the same numbers in the same order in every
//      lane and every cluster) and lane l sends the new weights to rank l of the cluster.
// So a step costs two trips through the cluster's shared memory and, for windows of more than one cluster, one
// through L2.  The step is a chain of short latencies, and a taken branch costs some 50 - 100 of them (a two-turn loop
// over shared memory took 380 cycles where the straight code takes 60): its code is kept straight, with selects for
// the threads that differ.  No buffer of the two cluster trips needs a second copy: weights of step s + 1 leave their
// owners only after every rank's sums of step s have been read, sums of step s + 1 leave a rank only after it has
// every weight of step s + 1.
// (A first version without clusters exchanged everything through L2, owners spread over all CTAs: two
// trips, each 2,500 - 5,500 cycles with 148 CTAs polling the same lines: 9.4 us per step.)  The accept decision is
// taken by every warp that owns parameters, from the same shares in the same order.  No atomics.
//
// Waits that run out.  Every wait is bounded.  The words of another cluster (603) are the only ones that may really
// stay out: the CTAs of a cluster start together, what they send one another arrives, copies and MMAs end.  When they
// do, the CTA goes on with the step's exchange, whose sums then mean nothing, and says so in the fourth element of every
// weight it sends (at the end of a trajectory: in its shares of the log-prior).  So all ranks of the cluster learn of
// it at the same point, where everything sent has been received; they leave between two barriers of the next step with
// nothing in flight, and neither samples nor state are stored.  The other clusters' words then stay out too.
// For waits inside the cluster to run out something must be broken; a CTA then leaves by itself, does not arm its
// barriers again, waits once more for its copies and MMAs, and for 100 us after the cluster has stopped sending.
// Launches that start while the status word is set do nothing: the host takes the report, clears the words and
// the counter, and only then do sequence numbers start anew (old words could otherwise pass for new ones).
// Limits: `wait_ticks` for words of another cluster, 64 times that for the first ones of a launch (until then some of
// its CTAs may be waiting for SMs that another stream's kernel holds), four times as long inside a cluster.
//
// It replaces, for such windows, the reference's persistent kernel with an unbounded grid barrier
// (mcmc_step_tc.h:597-677) and its per-iteration host work (main.h:204-283).
#pragma once
#include "chain.cuh"
#include "common.cuh"
#include "philox.h"
#include "refstream.cuh"
#include "tc05.cuh"

namespace mcmc_b200 {

constexpr int RES_NWG = 4;                     // warpgroups = resident tiles per CTA
constexpr int RES_THREADS = RES_NWG * 128;
constexpr int RES_BAR_E = 1, RES_BAR_T = 5, RES_BAR_X = 9;  // named barriers: + warpgroup, + warpgroup, the exchange
constexpr uint32_t RES_DEAD_LO = 0x4c4f5354u, RES_DEAD_HI = 0x7ff8dead;  // a log-prior share that no sum makes

// ---- words through L2: single 16-byte accesses ----------------------------------------------
__device__ __forceinline__ void st_word16(uint4* p, uint32_t a, uint32_t b, uint32_t c, uint32_t seq) {
  asm volatile(
      "{\n\t.reg .b64 lo, hi;\n\t.reg .b128 v;\n\t"
      "mov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\tmov.b128 v, {lo, hi};\n\t"
      "st.relaxed.gpu.global.b128 [%0], v;\n\t}" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(seq)
      : "memory");
}
__device__ __forceinline__ uint4 ld_word16(const uint4* p) {
  uint4 r;
  asm volatile(
      "{\n\t.reg .b64 lo, hi;\n\t.reg .b128 v;\n\t"
      "ld.relaxed.gpu.global.b128 v, [%4];\n\tmov.b128 {lo, hi}, v;\n\t"
      "mov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
      : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
      : "l"(p)
      : "memory");
  return r;
}

// ---- words through the cluster's shared memory ----------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// 16 bytes into another CTA's shared memory, counted by that CTA's mbarrier
__device__ __forceinline__ void st_async16(uint32_t dst, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];" ::"r"(dst),
               "r"(bar), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

static __device__ __noinline__ void res_timeout(const ResidentParams& g, int code) {
  if (g.status) atomicExch(g.status, code);
  if (g.status_host) *reinterpret_cast<volatile int*>(g.status_host) = code;
}
__device__ __forceinline__ uint32_t res_ticks() { return (uint32_t)(clock64() >> 16); }  // of 33 us at 1.965 GHz
// mbarrier wait of the resident kernel: a bounded spin in line (each try_wait sleeps in hardware for a moment).  What ran out is noted
// and reported at the kernel's end: calls in line would lengthen a step's code, which should stay in the instruction cache (32 KB: straight
// code of 48 KB takes 2.7 cycles an instruction, of 32 KB 1.2).  The loop out of line is no way: the call costs registers, 0.3 to 0.6 us a step
static __shared__ int res_code;
__device__ __forceinline__ void res_wait(uint64_t* bar, uint32_t parity, const ResidentParams&, uint32_t limit, int code,
                                         bool& ok) {
  if (mbar_try_wait(bar, parity)) return;
  const uint32_t t0 = res_ticks();
  while (ok && !mbar_try_wait(bar, parity))
    if (res_ticks() - t0 > limit) {
      ok = false;
      res_code = code;
    }
}
// for a copy or MMAs that a wait has run out on already, before their memory is given back
__device__ __forceinline__ void res_drain(uint64_t* bar, uint32_t parity, const ResidentParams& g) {
  const uint32_t t0 = res_ticks();
  while (!mbar_try_wait(bar, parity) && res_ticks() - t0 <= g.wait_ticks) {}
}

// One momentum draw: N(0,1) of (window, iteration, parameter), or the reference's stream
__device__ __forceinline__ float res_momentum(const AcceptParams& a, uint32_t gwin, int iter, int p) {
  return a.ref_streams ? refstream_normal(a.seed + REF_DRAWS_PER_ITER * (unsigned long long)iter + p)
                       : philox_normal(a.seed, gwin, (uint32_t)iter, STREAM_MOMENTUM, (uint32_t)p);
}
__device__ __forceinline__ double u2d(uint32_t lo, uint32_t hi) {
  return __longlong_as_double((long long)(((unsigned long long)hi << 32) | lo));
}
__device__ __forceinline__ uint2 d2u(double d) {
  const unsigned long long l = (unsigned long long)__double_as_longlong(d);
  return make_uint2((uint32_t)l, (uint32_t)(l >> 32));
}
// sums over the LPW lanes of a word; every lane gets them
template <int LPW>
__device__ __forceinline__ void word_sum(float v[3]) {
#pragma unroll
  for (int o = LPW >> 1; o > 0; o >>= 1) {
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
  }
}
template <int LPW>
__device__ __forceinline__ double word_sum(double v) {
#pragma unroll
  for (int o = LPW >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Tile = the precision's arithmetic for the CTA's rows (resident_tf32.cu, resident_fp32.cu):
//   Tile::H, Tile::SMEM               hidden units, bytes of dynamic shared memory
//   Tile(smem, g, win, u0, u1)       per-thread constants; rows 32 u0 .. 32 u1 of the window are this CTA's
//   setup(tmap, g, win)              loads the rows; false when they did not arrive
//   stage(v)                         word `threadIdx.x` of the weights (the first ResWords::N threads)
//   step(g, row_loss, last, ok)      forward, loss, backward of this warpgroup's tile
//   collects()                       the word whose sum this thread makes, or -1
//   collect(last, v)                 after the CTA barrier that follows step: the CTA's sums for that word
//   teardown(g, dead)                gives memory back; dead: after one more wait for MMAs
//   X_PLACE, x_at(u)                 whether it has room for the words of all clusters, once the CTA's sums are sent; word u
// The parameters of a word, in an order of their own: words 0 .. 306 are W0 and b0 (the last one two of them), the next
// fourteen W1 and b1, the last word is the log-likelihood.
template <int H>
struct ResWords {
  static constexpr int P = 22 * H + 2 * H + 1;
  static constexpr int W0 = (23 * H + 2) / 3;           // words of W0 and b0
  static constexpr int N = W0 + (H + 1 + 2) / 3 + 1;    // all words
  static constexpr int PAD = 3 * W0 - 23 * H;           // empty places of word W0 - 1
  static constexpr int PER_RANK8 = (N + 7) / 8;         // words of a rank of eight
  __device__ static int param(int t, int q) { return t < W0 ? 3 * t + q : 3 * t + q - PAD; }
  __device__ static bool valid(int t, int q) { return t < W0 ? 3 * t + q < 23 * H : 3 * t + q - PAD < P; }
};

__device__ __forceinline__ float res_w0(const ResidentParams& g, int p) { return __ldcg(g.w0 + p); }
__device__ __forceinline__ float res_w0(const ResidentEvalParams& g, int p) { return g.w_val[p]; }

// MULTI: windows of several clusters, which are clusters of eight.  (Windows of one do without the exchange through L2, its code and its
// registers: 1000 rows TF32 2.94 -> 2.75 us a step)
template <class Tile, int C, bool MULTI, class Params>
__global__ void __launch_bounds__(RES_THREADS, 1)
resident_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ Params g) {
  using Words = ResWords<Tile::H>;
  constexpr int P = Words::P, NWORDS = Words::N;
  constexpr int WPM = (NWORDS + C - 1) / C;            // words per rank
  constexpr int XWARPS = (WPM * C + 31) / 32;          // warps that own words
  static_assert(WPM * C <= RES_THREADS && NWORDS <= RES_THREADS, "one thread per lane of a word");
  constexpr int XT = XWARPS * 32;
  constexpr int STR = (WPM + 7) / 8 * 8;               // a cluster's words start on a line
  constexpr int NR = MULTI ? (WPM * RES_MAX_CLUSTERS + XT - 1) / XT : 1;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = smem_align1024(smem_raw);
  __shared__ __align__(16) uint4 part_in[C][WPM];           // sums of every rank for the words owned here
  __shared__ __align__(16) uint4 w_in[NWORDS];              // weights
  __shared__ __align__(16) uint4 h_in[2][C * XWARPS + 1];   // {kinetic, log-prior} shares; log-likelihood
  __shared__ __align__(16) uint4 x_in_[MULTI && !Tile::X_PLACE ? RES_MAX_CLUSTERS * WPM : 1];  // words of all clusters
  __shared__ __align__(8) uint64_t bar_part, bar_w, bar_h;
  // A word's parameters: where they stand at the start of a trajectory (position, gradient, momentum) and now (position, momentum).
  // A step needs their 15 registers for other things, and what it spills comes back from L2, next to all of L1 being shared memory.
  // With these, the chain's state below and a kernel of its own for windows of one cluster, us a step (10-step trajectories): TF32 1000
  // rows 2.88 -> 2.75, 4096 3.97 -> 3.86, 58368 5.76 -> 5.41; FP32 4.76 -> 4.50, 8.17 -> 8.07, 9.87 -> 9.56
  __shared__ float kept[15][XT];
  __shared__ struct { double ll, lp; int iter, n_acc; uint32_t gwin; } at_[XWARPS];  // the chain, as every warp that owns parameters follows it
  __shared__ int dead_;  // a wait has run out, here or in another CTA of the cluster
  volatile int& dead = dead_;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = C == 1 ? 0 : (int)cluster_rank();
  const int K = MULTI ? g.clusters : 1;
  const int cl = (int)blockIdx.x / C;
  const int win = cl / K, k = cl - win * K;
  const int cta = k * C + rank, n_cta = K * C;
  const int units = (g.n_rows + 31) / 32;
  Tile c(base, g, win, (int)((long long)cta * units / n_cta), (int)((long long)(cta + 1) * units / n_cta));
  auto x_in = [&](int u) -> uint4& {
    if constexpr (Tile::X_PLACE) return c.x_at(u);
    else return x_in_[u];
  };
  if (tid == 0) {
    mbar_init(&bar_part, 1);
    mbar_init(&bar_w, 1);
    mbar_init(&bar_h, 1);
    mbar_fence_init();
    dead = 0;
    res_code = 0;
  }
  // ---- what this thread owns ----
  const int wl = tid / C, l = tid % C;       // word of this rank, lane of the word
  const int word = rank * WPM + wl;
  const bool mine = wl < WPM && word < NWORDS;
  const bool ll_word = word == NWORDS - 1;
  const bool chain = g.mode == RES_CHAIN;
  const AcceptParams& a = g.a;
  uint32_t seq = __ldcg(g.seq + win);
  // ---- state of the word's parameters, the same in each of its lanes: read first, so that it arrives beside the rows ----
  const size_t so = (size_t)win * g.Pp;
  float eps = chain ? __ldcg(a.eps + win) : g.eps_scalar;
  auto& at = at_[min(warp, XWARPS - 1)];
  if (warp < XWARPS) {  // (all lanes the same)
    at.ll = chain ? a.ll_cur[win] : 0.0;
    at.lp = chain ? a.lp_cur[win] : 0.0;
    at.iter = chain ? a.iter[win] : 0;
    at.n_acc = 0;
    at.gwin = chain ? (uint32_t)a.gwin[win] : 0u;
  }
  bool has[3];
  float* const kp = &kept[0][min(tid, XT - 1)];
  auto w_s = [&](int q) -> float& { return kp[q * XT]; };
  auto g_s = [&](int q) -> float& { return kp[(3 + q) * XT]; };
  auto m_s = [&](int q) -> float& { return kp[(6 + q) * XT]; };
  auto w_at = [&](int q) -> float& { return kp[(9 + q) * XT]; };
  auto m_at = [&](int q) -> float& { return kp[(12 + q) * XT]; };
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int p = Words::param(word, q);
    has[q] = mine && Words::valid(word, q);
    float w0 = 0.f, g0 = 0.f, m0 = 0.f;
    if (has[q]) {
      w0 = chain ? __ldcg(a.w_cur + so + p) : res_w0(g, p);
      if (g.mode != RES_EVAL) {
        g0 = __ldcg((chain ? a.g_cur + so : g.g0) + p);
        m0 = __ldcg((chain ? a.m_start + so : g.m0) + p);
      }
    }
    if (tid < XT) {
      w_s(q) = w0;
      g_s(q) = g0;
      m_s(q) = m0;
      // half kick, drift (mcmc_step_ffma.h:106-120)
      const bool drift = has[q] && g.mode != RES_EVAL;
      const float m1 = drift ? fmaf(eps * 0.5f, g0, m0) : 0.f;
      m_at(q) = m1;
      w_at(q) = drift ? fmaf(eps, m1, w0) : w0;
    }
  }
  // (a status that is set already: see above)
  const int pending = __ldcg(g.status);
  if (pending != 0 && g.status_host && blockIdx.x == 0 && tid == 0)
    *reinterpret_cast<volatile int*>(g.status_host) = pending;
  const bool loaded = c.setup(&tmap, g, win);  // (holds a CTA barrier)
  if (!loaded || pending != 0) dead = 1;
  bool ok = true;     // no wait of this thread inside the cluster has run out
  bool lost = false;  // the launch has given up
  const int my_words = min(WPM, NWORDS - rank * WPM);
  const uint32_t part_bytes = (uint32_t)(my_words * C * 16), w_bytes = NWORDS * 16, h_bytes = (C * XWARPS + 1) * 16;
  if (tid == 0) {
    mbar_expect_tx(&bar_part, part_bytes);
    mbar_expect_tx(&bar_w, w_bytes);
    mbar_expect_tx(&bar_h, h_bytes);
  }
  if (C > 1) cluster_sync_all();  // every rank's barriers exist before anyone sends
  else __syncthreads();

  // ---- where this thread sends ----
  const int out = max(c.collects(), 0);      // the word of which this thread sends the CTA's sums
  const uint32_t part_dst = mapa(smem_u32(&part_in[rank][out % WPM]), out / WPM);
  const uint32_t part_bar = mapa(smem_u32(&bar_part), out / WPM);
  const uint32_t w_dst = mapa(smem_u32(&w_in[mine ? word : 0]), l), w_bar = mapa(smem_u32(&bar_w), l);
  constexpr uint32_t H_BUF = (C * XWARPS + 1) * 16;
  // words through L2: [2 buffers][windows][ranks][clusters][STR]
  const size_t msg_buf = (size_t)g.windows * C * K * STR;
  uint4* const msg = g.msg + ((size_t)win * C + rank) * K * STR;
  uint32_t x_src[NR];
  bool x_has[NR];
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int u = tid + i * XT;
    x_has[i] = MULTI && tid < XT && u < my_words * K;
    x_src[i] = (uint32_t)(u / my_words * STR + u % my_words);
  }
  // limits of the waits that may last until the last CTA of the launch has started, and of the others
  auto limit = [&](uint32_t n) { return g.wait_ticks << (n < 2 ? 8 : 2); };

  auto send_weights = [&](const float (&w)[3], bool bad) {
    if (mine) st_async16(w_dst, w_bar, __float_as_uint(w[0]), __float_as_uint(w[1]), __float_as_uint(w[2]), bad);
  };
  uint32_t n = 0;        // steps done in this launch: the mbarrier phases follow it
  uint32_t n_traj = 0;
  {
    const float w[3] = {w_at(0), w_at(1), w_at(2)};
    send_weights(w, dead != 0);
  }

  const int L = g.n_steps;
  for (int it = 0; it < g.n_iter; ++it) {
    for (int s = 0; s < L; ++s, ++n) {
      const uint32_t ph = n & 1;
      const bool last = s == L - 1;
      ++seq;
      // ---- weights of this step ----
      res_wait(&bar_w, ph, g, limit(n), 601, ok);
      if (tid == 0 && ok) mbar_expect_tx(&bar_w, w_bytes);
      {
        const uint4 v = w_in[min(tid, NWORDS - 1)];
        if (!ok || v.w != 0u) dead = 1;
        c.stage(v);  // (ends in a CTA barrier)
      }
      // ---- this warpgroup's tile ----
      c.step(g, last ? g.row_loss : nullptr, last, ok);
      const bool leave = dead != 0;  // the same in every thread: nobody writes it between the step's two barriers
      __syncthreads();
      if (leave) {
        lost = true;
        it = g.n_iter;
        break;
      }
      // ---- the CTA's sums to their owners ----
      {
        uint4 v;
        if (c.collect(last, v)) {
          st_async16(part_dst, part_bar, v.x, v.y, v.z, 0u);
        }
      }
      if (warp >= XWARPS) continue;
      float w[3], m[3], m_nx[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        w[q] = w_at(q);
        m[q] = m_at(q);
      }
      if (last && chain) {
#pragma unroll
        for (int q = 0; q < 3; ++q) m_nx[q] = has[q] ? res_momentum(a, at.gwin, at.iter + 1, Words::param(word, q)) : 0.f;
      }
      // ---- owners: the cluster's sum, then the window's ----
      // (the log-likelihood is wanted at the end of a trajectory only)
      const bool ll_warp = last && rank == C - 1 && warp == (NWORDS - 1 - (C - 1) * WPM) * C / 32;
      res_wait(&bar_part, ph, g, limit(n), 602, ok);
      if (tid == 0 && ok) mbar_expect_tx(&bar_part, part_bytes);
      const uint4 x = part_in[l][min(wl, WPM - 1)];
      float v[3] = {__uint_as_float(x.x), __uint_as_float(x.y), __uint_as_float(x.z)};
      word_sum<C>(v);
      double ll = 0.0;
      bool bad = !ok;
      if (ll_warp) ll = word_sum<C>(ll_word ? u2d(x.x, x.y) : 0.0);
      if (MULTI) {
        uint4* const mb = msg + (seq & 1) * msg_buf;
        if (mine && l == 0) {
          const uint2 d = d2u(ll);
          st_word16(mb + k * STR + wl, ll_word ? d.x : __float_as_uint(v[0]), ll_word ? d.y : __float_as_uint(v[1]),
                    __float_as_uint(v[2]), seq);
        }
        uint4 y[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) y[i] = x_has[i] ? ld_word16(mb + x_src[i]) : make_uint4(0u, 0u, 0u, seq);
        auto missing = [&]() {
          bool r = false;
#pragma unroll
          for (int i = 0; i < NR; ++i) r |= y[i].w != seq;
          return r;
        };
        // (one loop over all words, not one a word: steps of 16384 rows and more 2 to 5 % shorter)
        const uint32_t t0 = res_ticks();
#pragma unroll 1
        while (missing()) {
#pragma unroll
          for (int i = 0; i < NR; ++i)  // (a word that has arrived is read once more: its value stays)
            if (x_has[i]) y[i] = ld_word16(mb + x_src[i]);
          if (__builtin_expect(res_ticks() - t0 > g.wait_ticks << (n == 0 ? 6 : 0), 0)) {
            dead = 1;
            res_code = 603;
            break;
          }
        }
#pragma unroll
        for (int i = 0; i < NR; ++i)
          if (x_has[i]) x_in(tid + i * XT) = y[i];
        if (!ok) dead = 1;
        named_sync(RES_BAR_X, XT);
        bad = dead != 0;
        // lane l adds clusters l and l + 8
        const int wi = min(wl, my_words - 1);
        const uint4 y0 = x_in(min(l, K - 1) * my_words + wi), y1 = x_in(min(l + C, K - 1) * my_words + wi);
        const bool one = l < K, two = l + C < K;
        v[0] = (one ? __uint_as_float(y0.x) : 0.f) + (two ? __uint_as_float(y1.x) : 0.f);
        v[1] = (one ? __uint_as_float(y0.y) : 0.f) + (two ? __uint_as_float(y1.y) : 0.f);
        v[2] = (one ? __uint_as_float(y0.z) : 0.f) + (two ? __uint_as_float(y1.z) : 0.f);
        word_sum<C>(v);
        if (ll_warp)
          ll = word_sum<C>(ll_word ? (one ? u2d(y0.x, y0.y) : 0.0) + (two ? u2d(y1.x, y1.y) : 0.0) : 0.0);
      }
      float gf[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) gf[q] = fmaf(w[q], g.prior.neg_inv_s2, v[q]);
      if (!last) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          m[q] = fmaf(eps, gf[q], m[q]);
          w[q] = fmaf(eps, m[q], w[q]);
        }
        send_weights(w, bad);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          w_at(q) = w[q];
          m_at(q) = m[q];
        }
        continue;
      }
      // ---- end of the trajectory: this warp's share of the log-prior and of the kinetic difference ----
      double lp = 0.0, dk = 0.0;
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (has[q] && l == 0) {
          const float u = w[q] * g.prior.inv_s;
          const float pl = fmaf(-0.5f * u, u, -g.prior.norm);
          lp += (double)pl;
          if (chain) {  // closing half kick (kernel_helpers.h:163-175)
            const float mf = fmaf(eps * 0.5f, gf[q], m[q]);
            dk += 0.5 * ((double)m_s(q) * (double)m_s(q) - (double)mf * (double)mf);
          } else if (k == 0 && !bad) {
            const int p = Words::param(word, q);
            g.g_out[p] = gf[q];
            if (g.w_out) g.w_out[p] = w[q];
            if (g.m_out) g.m_out[p] = m[q];
            if (g.zero_out) g.zero_out[p] = 0.f;
            if (g.prior_loss) g.prior_loss[p] = pl;
          }
        }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lp += __shfl_xor_sync(0xffffffffu, lp, o);
        dk += __shfl_xor_sync(0xffffffffu, dk, o);
      }
      const uint32_t hb = n_traj & 1;
      bad = __any_sync(0xffffffffu, bad);
      if (lane < C) {
        const uint2 x1 = d2u(dk), x2 = bad ? make_uint2(RES_DEAD_LO, RES_DEAD_HI) : d2u(lp);
        st_async16(mapa(smem_u32(&h_in[0][rank * XWARPS + warp]), lane) + hb * H_BUF, mapa(smem_u32(&bar_h), lane), x1.x,
                   x1.y, x2.x, x2.y);
      }
      if (ll_warp && mine && ll_word) {
        const uint2 x1 = d2u(ll);
        st_async16(mapa(smem_u32(&h_in[0][C * XWARPS]), l) + hb * H_BUF, mapa(smem_u32(&bar_h), l), x1.x, x1.y, 0u, 0u);
      }
      res_wait(&bar_h, hb, g, limit(n), 604, ok);
      if (tid == 0 && ok) mbar_expect_tx(&bar_h, h_bytes);
      ++n_traj;
      dk = lp = 0.0;
      bad = !ok;
      for (int i = lane; i < C * XWARPS; i += 32) {
        const uint4 x1 = h_in[hb][i];
        dk += u2d(x1.x, x1.y);
        lp += u2d(x1.z, x1.w);
        bad |= x1.z == RES_DEAD_LO && x1.w == RES_DEAD_HI;
      }
      lost = __any_sync(0xffffffffu, bad);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lp += __shfl_xor_sync(0xffffffffu, lp, o);
        dk += __shfl_xor_sync(0xffffffffu, dk, o);
      }
      const double ll_new = u2d(h_in[hb][C * XWARPS].x, h_in[hb][C * XWARPS].y);
      if (lost) {
        if (it + 1 < g.n_iter) send_weights(w, true);
        continue;
      }
      if (!chain) {
        if (k == 0 && rank == 0 && tid == 0) {
          g.scalars[0] = ll_new;
          g.scalars[1] = lp;
        }
        continue;
      }
      const int iter = at.iter;
      const double la = (ll_new - at.ll) + (lp - at.lp) + dk;
      const float la_f = (float)la;
      const float log_u = a.ref_streams ? a.ref_log_u[iter % a.ref_cap]
                                        : logf(philox_accept_uniform(a.seed, at.gwin, (uint32_t)iter));
      const bool acc = log_u < la_f;  // main.h:242; a NaN ratio rejects
      float eps_next = eps;
      if (iter < a.adapt_steps) {  // main.h:266-276
        const float lmr = fminf(la_f, 0.f);
        eps_next = eps + eps * (lmr < a.log_target ? a.dec_adj : a.inc_adj);
      }
      if (k == 0 && rank == 0 && tid == 0 && iter < a.trace_iters) {
        const size_t ti = (size_t)win * a.trace_iters + iter;
        a.tr_log_u[ti] = log_u;
        a.tr_log_acpt[ti] = la;
        a.tr_accept[ti] = acc;
        a.tr_eps[ti] = eps;
      }
      __syncwarp();  // (every lane has read what follows)
      if (acc) {
        at.ll = ll_new;
        at.lp = lp;
      }
      const int n_acc = at.n_acc;
      __syncwarp();
      at.n_acc = n_acc + (acc ? 1 : 0);
      at.iter = iter + 1;
      __syncwarp();
      eps = eps_next;
      const int store = iter - a.burn_in;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        if (acc) {
          w_s(q) = w[q];
          g_s(q) = gf[q];
        }
        m_s(q) = m_nx[q];
        // start of the next trajectory (main.h:207-218)
        m[q] = fmaf(eps * 0.5f, g_s(q), m_nx[q]);
        w[q] = fmaf(eps, m[q], w_s(q));
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        w_at(q) = w[q];
        m_at(q) = m[q];
      }
      if (it + 1 < g.n_iter) send_weights(w, false);
      if (k == 0 && l == 0) {
#pragma unroll
        for (int q = 0; q < 3; ++q)
          if (has[q]) {
            const int p = Words::param(word, q);
            if (store >= 0 && store < a.sample_capacity)
              a.samples[((size_t)win * a.sample_capacity + store) * P + p] = w_s(q);
            if (iter + 1 < a.trace_iters) a.tr_mom[((size_t)win * a.trace_iters + iter + 1) * P + p] = m_s(q);
          }
      }
    }
  }
  // ---- the state the next launch (of either kind) starts from; of a launch that gave up: the one it started from ----
  if (chain && !lost && k == 0 && l == 0) {
#pragma unroll
    for (int q = 0; q < 3; ++q)
      if (has[q]) {
        const size_t p = so + Words::param(word, q);
        a.w_cur[p] = w_s(q);
        a.g_cur[p] = g_s(q);
        a.w_start[p] = w_s(q);
        a.m_start[p] = m_s(q);
        a.m0[p] = m_s(q);
      }
  }
  if (k == 0 && rank == 0 && tid == 0) {
    if (chain && !lost) {
      a.ll_cur[win] = at.ll;
      a.lp_cur[win] = at.lp;
      a.eps[win] = eps;
      a.iter[win] = at.iter;
      a.n_accept[win] += at.n_acc;
    }
    // (every cluster of the window has read the counter: this one has used words that carry later values)
    g.seq[win] = seq;
  }
  if (!ok) dead = 1;
  c.teardown(g, dead);  // (begins with a CTA barrier)
  if (tid == 0 && *reinterpret_cast<volatile int*>(&res_code) != 0) res_timeout(g, res_code);
  if (C > 1) cluster_sync_all();  // no rank leaves while another may still write to it
  if (dead) __nanosleep(100000);
}

// ---- host side ----------------------------------------------------------------------------
// CTAs that wait for one another's words have to be resident together.  The hardware sees to that within a cluster; for
// windows of several clusters the launch is cooperative.
template <typename K, typename Params>
static cudaError_t resident_launch(K kernel, int cluster, size_t smem, const void* tmap, const Params& g,
                                   cudaStream_t st, int* max_clusters) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(max_clusters ? cluster : (g.windows * g.clusters - g.missing) * cluster);
  cfg.blockDim = dim3(RES_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g.clusters > 1 ? 2 : 1;
  if (max_clusters) {
    cfg.numAttrs = 1;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return e != cudaSuccess ? e : cudaOccupancyMaxActiveClusters(max_clusters, kernel, &cfg);
  }
  return cudaLaunchKernelEx(&cfg, kernel, *reinterpret_cast<const CUtensorMap*>(tmap), g);
}

template <class Tile, int C>
static cudaError_t resident_launch_c(const void* tmap, const ResidentParams& g, cudaStream_t st, int* max_clusters) {
  if (C == 8 && (max_clusters || g.clusters > 1)) {
    cudaError_t e = resident_launch(resident_kernel<Tile, C, C == 8, ResidentParams>, C, Tile::SMEM, tmap, g, st, max_clusters);
    if (e != cudaSuccess || !max_clusters) return e;
    int single = 0;  // (the kernel for windows of one cluster each takes no more of anything; its attribute is set here)
    e = resident_launch(resident_kernel<Tile, C, false, ResidentParams>, C, Tile::SMEM, tmap, g, st, &single);
    if (e == cudaSuccess && single < *max_clusters) *max_clusters = single;
    return e;
  }
  return resident_launch(resident_kernel<Tile, C, false, ResidentParams>, C, Tile::SMEM, tmap, g, st, max_clusters);
}
template <class Tile>
static cudaError_t resident_launch_any(int cluster, const void* tmap, const ResidentParams& g, cudaStream_t st, int* max_clusters) {
  switch (cluster) {
    case 1: return resident_launch_c<Tile, 1>(tmap, g, st, max_clusters);
    case 2: return resident_launch_c<Tile, 2>(tmap, g, st, max_clusters);
    case 4: return resident_launch_c<Tile, 4>(tmap, g, st, max_clusters);
    case 8: return resident_launch_c<Tile, 8>(tmap, g, st, max_clusters);
  }
  return cudaErrorInvalidValue;
}

template <class Tile, bool MULTI, class Params>
static cudaError_t resident_launch_single_m(const void* tmap, const Params& g, cudaStream_t st) {
  static bool attr_done[64] = {};
  auto kernel = resident_kernel<Tile, 8, MULTI, Params>;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Tile::SMEM);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_done[dev] = true;
  }
  return resident_launch(kernel, 8, Tile::SMEM, tmap, g, st, nullptr);
}
// ... of explicit calls, in clusters of eight: nobody has asked how many there can be
template <class Tile, class Params>
static cudaError_t resident_launch_single(const void* tmap, const Params& g, cudaStream_t st) {
  return g.clusters > 1 ? resident_launch_single_m<Tile, true>(tmap, g, st) : resident_launch_single_m<Tile, false>(tmap, g, st);
}

}  // namespace mcmc_b200
