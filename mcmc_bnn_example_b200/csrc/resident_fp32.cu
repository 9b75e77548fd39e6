// Tile arithmetic of the resident kernel in FP32 mode (resident.cuh has the launch structure, split_mma.cuh the forward product on
// the tensor core, fp32_split.cuh what a warp does with its 32 rows behind it, int_mma.cuh the sums over rows on the integer tensor core): every
// warp owns one 32-row unit for the whole launch, its rows in three parts in tensor memory and once more, as integers, in shared memory.
// A CTA's sums come out of one accumulator, where the backward pass by FFMA left every warp 960 products of 32 rows (2,250 cycles)
// and sixteen partial sums.  us a step, one B200, by FFMA and now (trajectories of ten steps; on one cluster 4096 rows, eight windows): 8 x 4096 rows 8.4 and 7.0, 16384 7.5 and
// 6.55, 58368 10.1 and 8.5, 70 windows of 800 rows 8.1 and 6.1.  CTAs of one tile stay with FFMA (resident_fp32_ffma.cu).
// What bounds a step (clock reads, 58368 rows, 16,500 cycles): weights arrive and are cut up 0 - 350, first z 1,300, tanh and dL/dz of a
// scheduler's four warps one after the other, 1,030 cycles each (MUFU 640), until 7,000; the last tile's sums 7,850, read out and
// sent 9,500; then the exchange (resident.cuh), 7,000.
// What cost more than it gave: conversions of float to integer (the tanh's pipe: 440 cycles a warp), polls by warps that have
// nothing to do, a scale from the step itself, sums issued by every tile's last warp, one accumulator pair for the product (tiles wait for
// one another, 9.1 us), everything that made a step spill more than L1 holds (up to 2 us).
#include <cuda.h>
#include "fp32_split.cuh"
#include "resident.cuh"

namespace mcmc_b200 {

struct ResFp32 {
  static constexpr int H = SPLIT_H, D = SPLIT_D;
  using Words = ResWords<H>;
  using Warp = SplitWarp;
  static constexpr int NWARPS = RES_NWG * 4;
  static_assert(Warp::ROWS == 32 && NWARPS == RES_UNITS, "a warp owns one 32-row unit");
  // the sums of dW0 and db0 of a warp whose values no integers hold, after the shuffle over its two row subsets a lane's 6 features x 5
  // units; they take the place of its dL/dz
  static constexpr int GROUP = 6 * H, GSTR = GROUP + 8;
  static_assert(4 * GSTR <= Warp::ES, "sums fit where dL/dz was");
  static_assert(Warp::ES * 4 == INT_E_WARP && RES_UNITS * 32 * KP <= NWARPS * Warp::ES, "rows land where dL/dz will be");
  static constexpr int RS = H + 4;   // dW1 and db1 of a warp's rows
  // float offsets.  XI: features as integers; OWN: a thread's constants (target, factor of its line of sums, where its word's weights go),
  // registers that the step needs for other things; XS: the features' scales.  The sums over rows take the weights' place once the product is done; words of other
  // clusters take that of dL/dz.  (Up to 195 KB in all leave 60 KB of L1, for what a step spills; beyond that it is 28 KB, and half of it
  // comes back from L2: 1000 rows 4.5 us a step, and 5.7)
  static constexpr int WB = 0, S = WB, XI = WB + SPLIT_B_BYTES / 4, ES = XI + RES_UNITS * INT_X_WARP / 4, OWN = ES + NWARPS * Warp::ES,
                       XS = OWN + 4 * RES_THREADS, W1 = XS + KP, RW1 = W1 + RS, RLL = RW1 + NWARPS * RS, MISC = RLL + NWARPS * 2,
                       BAR = MISC + NWARPS + 4;
  static_assert(INT_S_FLOATS * 4 <= SPLIT_B_BYTES && 4 * GSTR + 4 * 64 <= Warp::ES && RES_MAX_CLUSTERS * Words::PER_RANK8 <= NWARPS * 64,
                "shared places");
  // barriers: rows landed; per tile, forward done, accumulators read, dL/dz written; sums over rows done; the scale is known
  static constexpr int NBARS = 3 + 3 * RES_NWG;
  static constexpr size_t SMEM = 1024 + (BAR + 2 * NBARS) * 4;
  static_assert(XI % 64 == 0 && ES % 4 == 0 && XS % 4 == 0 && W1 % 4 == 0 && RW1 % 4 == 0 && RLL % 2 == 0 && BAR % 2 == 0, "alignment");
  // Tensor memory: two accumulator pairs for the product, which the tiles take in turn and whose place, when all have been read, becomes
  // the sums over rows; and the rows' parts for the whole launch
  static constexpr int A_COL0 = 2 * SPLIT_Z_COLS, TMEM_COLS = 512;
  static_assert(INT_ACC_COLS <= A_COL0 && A_COL0 + RES_NWG * SPLIT_A_COLS <= TMEM_COLS, "tensor memory budget");

  // named barriers: a warp's turn is over (those of the last four are not needed)
  static constexpr int BAR_LO = 1, BAR_HI = 10;
  static_assert(BAR_LO + 8 <= RES_BAR_X && BAR_HI > RES_BAR_X && BAR_HI + 4 <= 16, "barrier numbers");
  __device__ __forceinline__ static int bar_turn(int w) { return w < 8 ? BAR_LO + w : BAR_HI + w - 8; }

  Warp lanes;
  float* base;
  int warp, wg, n_units, nt;
  int row0;          // this warp's first row in the window
  bool active, plain_x, plain, fresh;   // fresh: a trajectory begins
  int rows_are;
  uint32_t tmem, par, first_par;
  // What is in XI of this warp's rows.  FLOATS: a feature is beyond its range in one of them; FLOATS_NOW: a dL/dpred was, earlier in this
  // trajectory
  enum { INTS, FLOATS, FLOATS_NOW };
  __device__ __forceinline__ float& own(int i) const { return base[OWN + i * RES_THREADS + threadIdx.x]; }

  __device__ __forceinline__ uint64_t* bar_rows() const { return reinterpret_cast<uint64_t*>(base + BAR); }
  __device__ __forceinline__ uint64_t* bar_fwd(int w) const { return bar_rows() + 1 + w; }
  __device__ __forceinline__ uint64_t* bar_read(int w) const { return bar_rows() + 1 + RES_NWG + w; }
  __device__ __forceinline__ uint64_t* bar_e(int w) const { return bar_rows() + 1 + 2 * RES_NWG + w; }
  __device__ __forceinline__ uint64_t* bar_sum() const { return bar_rows() + 1 + 3 * RES_NWG; }
  __device__ __forceinline__ uint64_t* bar_scale() const { return bar_rows() + 2 + 3 * RES_NWG; }
  // statistics of dL/dpred per parity of the step; the sums' factor; whether a warp has taken FFMA
  __device__ __forceinline__ uint32_t* stat(int ph) const { return reinterpret_cast<uint32_t*>(base + MISC) + ph; }
  __device__ __forceinline__ float& sum_f() const { return base[MISC + 2]; }
  __device__ __forceinline__ volatile uint32_t* far() const { return reinterpret_cast<volatile uint32_t*>(base + MISC + 4); }
  __device__ __forceinline__ uint32_t far_warps() const {
    return __ballot_sync(0xffffffffu, lanes.lane < NWARPS && far()[lanes.lane & (NWARPS - 1)] != 0u);
  }
  // words of clusters: 64 behind each warp's sums
  static constexpr bool X_PLACE = true;
  __device__ __forceinline__ uint4& x_at(int u) const {
    return reinterpret_cast<uint4*>(base + ES + 4 * GSTR)[(u >> 6) * (Warp::ES / 4) + (u & 63)];
  }
  static __device__ __forceinline__ uint32_t a_col(int w) { return A_COL0 + w * SPLIT_A_COLS; }
  static __device__ __forceinline__ uint32_t z_col(int w) { return (w & 1) * SPLIT_Z_COLS; }

  __device__ __forceinline__ ResFp32(unsigned char* b, const ResidentParams& g, int win, int u0, int u1)
      : base(reinterpret_cast<float*>(b)) {
    warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    wg = warp >> 2;
    n_units = u1 - u0;
    nt = (n_units + 3) / 4;
    active = warp < n_units;
    row0 = (u0 + warp) * 32;
    par = first_par = 0;
    plain_x = plain = false;
    rows_are = INTS;
    fresh = true;
    const int t = threadIdx.x;
    uint32_t off[3];
    for (int q = 0; q < 3; ++q) {
      const int p = Words::param(t, q);
      // (threads and places of a word without a parameter write where feature 28 of unit 0 would be: nobody reads there)
      uint32_t dst = smem_u32(b) + split_b_off(0, 28);
      if (t < Words::N - 1 && Words::valid(t, q)) {
        if (p < D * H + H) dst = smem_u32(b) + split_b_off(p % H, p / H & ~3) + (p / H & 3) * 4;
        else dst = smem_u32(base + W1 + p - (D * H + H));
      }
      // (feature 23 is no weight, but the product reads it: sums have been there.  Threads behind the last word bring its zeros)
      if (t >= Words::N && t < Words::N + H) dst = smem_u32(b) + q * SPLIT_B_PART + split_b_off(t - Words::N, 20) + 12;
      off[q] = (dst - smem_u32(b)) >> 2;
    }
    own(0) = own(1) = 0.f;
    own(2) = __uint_as_float(off[0] | off[1] << 16);
    own(3) = __uint_as_float(off[2]);
  }

  __device__ __forceinline__ bool setup(const CUtensorMap*, const ResidentParams& g, int win) {
    __shared__ uint32_t tmem_slot, x_stat[KP], x_max[KP];
    float* const x_scale = base + XS;
    bool ok = true;
    const int tid = threadIdx.x;
    if (tid == 0) {
      auto warps_of = [&](int w) { return min(max(n_units - 4 * w, 1), 4); };
      mbar_init(bar_rows(), 1);
      for (int w = 0; w < RES_NWG; ++w) {
        mbar_init(bar_fwd(w), 1);
        mbar_init(bar_read(w), warps_of(w));
        mbar_init(bar_e(w), warps_of(w));
      }
      mbar_init(bar_sum(), 1);
      mbar_init(bar_scale(), warps_of(0));
      mbar_fence_init();
      // (the rows come beside all that follows; nothing else is written where they land)
      if (n_units > 0) {
        const uint32_t bytes = (uint32_t)n_units * 32 * KP * 4;
        mbar_expect_tx(bar_rows(), bytes);
        bulk_g2s(base + ES, g.xaug + ((size_t)(g.data_window0 + win) * g.rows_pad + row0) * KP, bytes, bar_rows());
      }
    }
    __syncwarp();
    if (warp == 0) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                   "r"((uint32_t)TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid < KP) x_stat[tid] = x_max[tid] = 0u;
    if (tid < BAR - MISC) base[MISC + tid] = 0.f;
    // what an MMA may read before it is written
    for (int i = tid; i < (ES - WB) / 4; i += RES_THREADS)
      reinterpret_cast<float4*>(base + WB)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    // sums that nothing writes stay zero
    for (int i = tid; i < MISC - RW1; i += RES_THREADS) base[RW1 + i] = 0.f;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = tmem_slot;
    bool wide = false;
    if (n_units > 0) {
      res_wait(bar_rows(), 0, g, g.wait_ticks << 2, 611, ok);
      if (!ok) res_drain(bar_rows(), 0, g);
      if (g.test_code == 611) res_wait(bar_rows(), 1, g, g.wait_ticks << 2, 611, ok);  // (nothing ends this phase)
      // (four values a load, and the columns' statistics a lane each: a float at a time, with reductions over the warp and every thread working
      // out all scales, an evaluation took 6 us longer)
      float v[KP];
#pragma unroll
      for (int ch = 0; ch < KP / 4; ++ch) {
        const float4 x = active ? reinterpret_cast<const float4*>(base + ES + tid * KP)[ch] : make_float4(0.f, 0.f, 0.f, 0.f);
        v[4 * ch] = x.x;
        v[4 * ch + 1] = x.y;
        v[4 * ch + 2] = x.z;
        v[4 * ch + 3] = x.w;
      }
      if (active) {
        own(0) = base[ES + (warp * 32 + lanes.own()) * KP + COL_Y];
        if (lanes.lane <= D) {
          const float* x = base + ES + warp * 32 * KP + lanes.lane;
          uint32_t st = 0u, mx = 0u;
#pragma unroll 16
          for (int r = 0; r < 32; ++r) {
            const float f = x[r * KP];
            st += int_stat(f);
            mx = max(mx, __float_as_uint(f) & 0x7fffffffu);
          }
          atomicAdd(&x_stat[lanes.lane], st);
          atomicMax(&x_max[lanes.lane], mx);
        }
      }
      if (4 * wg < n_units) {  // the tile's rows to tensor memory, zeros for warps without rows
        const uint32_t a_t = tmem + a_col(wg) + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float r[8] = {v[8 * j], v[8 * j + 1], v[8 * j + 2], v[8 * j + 3], v[8 * j + 4], v[8 * j + 5], v[8 * j + 6], j == 2 ? 0.f : v[8 * j + 7]};
#pragma unroll
          for (int k = 0; k < 8; ++k) wide |= split_wide(r[k]);
          split_store_row(a_t, j, r);
        }
        tc_wait_st();
        tc_fence_before();
      }
      __syncthreads();
      // features as integers: a scale each, from the CTA's rows
      auto x_exp = [&](int k) { return int_range_exp(min(int_scale_exp(x_stat[k], INT_ROOM_X), int_max_exp(x_max[k]))); };
      if (tid < KP) x_scale[tid] = tid > D ? 0.f : int_scale(x_exp(tid));  // (the target has none)
      __syncthreads();
      bool in = true;
#pragma unroll
      for (int ch = 0; ch < KP / 4; ++ch) {
        const float4 f = reinterpret_cast<const float4*>(x_scale)[ch];
        in &= fabsf(v[4 * ch]) * f.x < INT_TOP && fabsf(v[4 * ch + 1]) * f.y < INT_TOP && fabsf(v[4 * ch + 2]) * f.z < INT_TOP &&
              (ch == KP / 4 - 1 || fabsf(v[4 * ch + 3]) * f.w < INT_TOP);
      }
      if (!__all_sync(0xffffffffu, in)) rows_are = FLOATS;
      float4* const xi = reinterpret_cast<float4*>(base + XI + warp * 32 * KP);
#pragma unroll
      for (int ch = 0; ch < KP / 4; ++ch) {
        const float4 x = make_float4(v[4 * ch], v[4 * ch + 1], v[4 * ch + 2], v[4 * ch + 3]);
        if (rows_are != INTS) xi[lanes.lane * (KP / 4) + ch] = x;
        else int_store_x4(smem_u32(xi) + int_x_off(lanes.lane, ch), x, reinterpret_cast<const float4*>(x_scale)[ch]);
      }
      const int k = (warp & 3) * 8 + (lanes.lane >> 2);  // the line whose sums this lane reads
      own(1) = k <= D ? int_unscale(x_exp(k) + 8 * (lanes.lane & 3) + INT_READ_SHIFT) : 0.f;
      fence_proxy_async_smem();
    }
    plain_x = __syncthreads_or(wide) != 0;
    return ok;
  }

  // word `threadIdx.x` of the weights
  __device__ __forceinline__ void stage(const uint4& v) {
    const bool word = (int)threadIdx.x < Words::N - 1;
    const uint32_t x[3] = {word ? v.x : 0u, word ? v.y : 0u, word ? v.z : 0u};
    const uint32_t off = __float_as_uint(own(2)), b = smem_u32(base);
    const uint32_t s_dst[3] = {b + (off & 0xffffu) * 4, b + (off >> 16) * 4, b + __float_as_uint(own(3)) * 4};
    bool wide = plain_x;
    if ((int)threadIdx.x < Words::W0) {
#pragma unroll
      for (int q = 0; q < 3; ++q) wide |= split_store_weight(s_dst[q], __uint_as_float(x[q]));
    } else {
#pragma unroll
      for (int q = 0; q < 3; ++q) asm volatile("st.shared.b32 [%0], %1;" ::"r"(s_dst[q]), "r"(x[q]) : "memory");
    }
    fence_proxy_async_smem();
    plain = __syncthreads_or(wide) != 0;
  }

  // The backward pass of a warp with a value beyond the range, which no integer holds, by FFMA.  A dL/dpred that is likely stays there, so
  // the warp's rows remain floats until the trajectory's end.  (Functions of their own, so that the step does without the registers; a
  // list of such rows instead, added to the sums one by one, cost every step 0.4 us)
  static __device__ __noinline__ void ints_to_floats(float* xi, uint32_t a_t) {
    float4* const row = reinterpret_cast<float4*>(xi) + (threadIdx.x & 31) * (KP / 4);
#pragma unroll 1
    for (int j = 0; j < 3; ++j) {
      float hi[8], r[8];
      tc_ld8(a_t + 8 * j, hi);
      tc_ld8(a_t + SPLIT_K + 8 * j, r);   // (a row's middle part is all that is left of it)
      tc_wait_ld();
      row[2 * j] = make_float4(hi[0] + r[0], hi[1] + r[1], hi[2] + r[2], hi[3] + r[3]);
      row[2 * j + 1] = make_float4(hi[4] + r[4], hi[5] + r[5], hi[6] + r[6], hi[7] + r[7]);
    }
    __syncwarp();
  }
  static __device__ __noinline__ void far_backward(const float* xi, float* es) {
    const Warp lanes;
    uint64_t acc[Warp::KPT / 2][Warp::UPT] = {};
    lanes.backward<2>(xi, es, acc);
    __syncwarp();  // dL/dz has been read by every lane
    lanes.store_dw0(acc, es + (2 * lanes.kh + lanes.rsub) * GSTR);
  }
  static __device__ __noinline__ void floats_to_ints(float* xi, const float* x_scale) {
    const int lane = threadIdx.x & 31;
    float4 x[KP / 4];
#pragma unroll
    for (int ch = 0; ch < KP / 4; ++ch) x[ch] = reinterpret_cast<const float4*>(xi)[lane * (KP / 4) + ch];
    __syncwarp();
#pragma unroll
    for (int ch = 0; ch < KP / 4; ++ch)
      int_store_x4(smem_u32(xi) + int_x_off(lane, ch), x[ch], reinterpret_cast<const float4*>(x_scale)[ch]);
    fence_proxy_async_smem();
  }

  __device__ __forceinline__ void rows_to_floats() {
    if (rows_are != INTS) return;
    ints_to_floats(base + XI + warp * 32 * KP, tmem + a_col(wg) + ((uint32_t)((warp & 3) * 32) << 16));
    rows_are = FLOATS_NOW;
  }

  __device__ __forceinline__ void step(const ResidentParams& g, float* row_loss, bool last, bool& ok) {
    const uint32_t ph = par;
    par ^= 1;
    if (n_units == 0) return;
    const bool first = fresh;
    fresh = last;
    const uint32_t fph = first_par;
    first_par ^= first ? 1u : 0u;
    const uint32_t limit = g.wait_ticks << 2;
    if (warp == NWARPS - 1) {
      // the product's MMAs of all tiles, by the warp whose own rows come last; accumulators' next tile when they have been read
      const uint32_t on = elect_one(), tm = __shfl_sync(0xffffffffu, tmem, 0), wb = smem_u32(base + WB);
      for (int w = 0; w < nt; ++w) {
        if (w >= 2) res_wait(bar_read(w - 2), ph, g, limit, 613, ok);
        tc_fence_after();
        split_issue(tm + z_col(w), tm + a_col(w), wb, on);
        tc_commit_if(bar_fwd(w), on);
      }
    }
    float* es = base + ES + warp * Warp::ES;
    uint64_t dw1[5] = {};
    float dy = 0.f, pred = 0.f;
    bool near = true;
    const bool valid = lanes.own() < g.n_rows - row0;
    auto give_scale = [&]() {
      const uint32_t st = __reduce_add_sync(0xffffffffu, int_stat(dy));
      if (lanes.lane == 0 && st) atomicMax(stat(ph), int_stat_word(int_scale_exp(st, INT_ROOM_E)));
    };
    if (active) {
      uint64_t h[4][5];
      res_wait(bar_fwd(wg), ph, g, limit, 612, ok);
      tc_fence_after();
      if (__builtin_expect(plain, 0)) {
        rows_to_floats();
        Warp::plain<2>(base + XI + warp * 32 * KP, reinterpret_cast<const unsigned char*>(base + WB), es);
        lanes.load_plain(es, h);
      } else {
        lanes.load(tmem + z_col(wg) + ((uint32_t)((warp & 3) * 32) << 16), h);
      }
      tc_fence_before();
      // (another tile or the sums take the accumulators' place)
      __syncwarp();
      if (lanes.lane == 0) mbar_arrive(bar_read(wg));
      float d[4];
      // The four warps of a scheduler take turns at the tanh, which MUFU bounds: side by side they would all end it late, and only
      // then go on.  4096 rows 8.63 us a step without turns, 7.8 with them; 58368 rows 10.2 and 9.45
      if (warp >= 4) named_sync(bar_turn(warp - 4), 64);
      lanes.front(h, base + W1, g.lik, own(0), valid, d, dy, pred, [&](int i) {
        if (i == 3 && warp + 4 < n_units) named_arrive(bar_turn(warp), 64);
      });
      // The first tile's rows give the scale, to all of them, in a trajectory's first step, and to the next step: a step that had to
      // wait for its own would be 0.2 us longer.  It is the smallest that one of the tile's warps asks for, since an outlier may well
      // move the mean of 32 exponents, but nothing outside its warp should depend on it
      if (__builtin_expect(first, 0)) {
        if (rows_are == FLOATS_NOW) {
          floats_to_ints(base + XI + warp * 32 * KP, base + XS);
          rows_are = INTS;
        }
        if (wg == 0) {
          give_scale();
          __syncwarp();
          if (lanes.lane == 0) mbar_arrive(bar_scale());
        }
        res_wait(bar_scale(), fph, g, limit, 614, ok);
      }
      const int se = int_stat_exp(*reinterpret_cast<volatile uint32_t*>(stat(first ? ph : ph ^ 1)));
      const float scale = int_scale(se);
      // (A few rows whose dL/dpred is much smaller than the first tile's are no accident: FFMA has all their bits)
      const float m = fabsf(dy) * scale;
      const uint32_t out = __ballot_sync(0xffffffffu, m != 0.f && !(m >= INT_LOW && m < INT_TOP));
      near = rows_are == INTS && (out == 0u || (__popc(out) < INT_FEW && __all_sync(0xffffffffu, m < INT_TOP)));
      if (__builtin_expect(near, 1)) {
        lanes.store_ei(h, d, scale, es, dw1);
        fence_proxy_async_smem();
      } else {
        lanes.store_es(h, d, es, dw1);
      }
      if (threadIdx.x == 0) sum_f() = int_unscale(se);
      if (lanes.lane == 0) far()[warp] = near ? 0u : 1u;
      __syncwarp();
      if (lanes.lane == 0) mbar_arrive(bar_e(wg));
      if (__builtin_expect(!near, 0)) {
        rows_to_floats();
        far_backward(base + XI + warp * 32 * KP, es);
      }
      if (wg == 0 && !first) give_scale();
      if (__builtin_expect(last, 0)) {
        if (g.test_code == 612) res_wait(bar_fwd(wg), ph ^ 1, g, limit, 612, ok);  // (nothing ends this phase)
        // (nor this one before the next trajectory.  In every step, behind the wait for sums, the question took 0.1 us)
        if (g.test_code == 614) res_wait(bar_scale(), first_par, g, limit, 614, ok);
        const float loss = valid ? lik_loss(g.lik, own(0), pred) : 0.f;
        store_row_loss(row_loss, row0 + lanes.own(), loss, valid);
        double ld = (double)loss;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, o);
        if (lanes.lane == 0) reinterpret_cast<double*>(base + RLL)[warp] = ld;
      }
      float* rw1 = base + RW1 + warp * RS;
      lanes.store_dw1(dw1, rw1);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dy += __shfl_xor_sync(0xffffffffu, dy, o);
      if (lanes.lane == 0) rw1[H] = dy;
    }
    // Sums over rows, by a warp that has no rows, or is done with them first
    if (warp == (n_units < RES_UNITS ? NWARPS - 1 : 0)) {
      const uint32_t on = elect_one(), tm = __shfl_sync(0xffffffffu, tmem, 0);
      if (nt > 2) res_wait(bar_read(nt - 2), ph, g, limit, 614, ok);  // (their place must have been read)
      if (nt > 1) res_wait(bar_read(nt - 1), ph, g, limit, 614, ok);
      uint32_t more = 0u;
#pragma unroll 1
      for (int w = 0; w < nt; ++w) {
        res_wait(bar_e(w), ph, g, limit, 614, ok);
        tc_fence_after();
        const uint32_t far = far_warps() >> 4 * w;
        const uint64_t xd = int_x_desc(smem_u32(base + XI) + w * 4 * INT_X_WARP);
        const uint64_t ed = int_e_desc(smem_u32(base + ES) + w * 4 * INT_E_WARP);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (4 * w + i < n_units && !(far >> i & 1)) {
            int_mma_if(tm, umma_desc_advance(xd, i * (INT_X_WARP >> 4)), umma_desc_advance(ed, i * (INT_E_WARP >> 4)), more, on);
            more = 1u;
          }
      }
      tc_commit_if(bar_sum(), on);
      res_wait(bar_sum(), ph, g, limit, 614, ok);
    }
    // the CTA's sums, ten units a warp
    __syncthreads();
    tc_fence_after();
    if ((warp & 3) < INT_LINES / 32) {
      float v[10];
      int_read_out<10>(tmem + wg * 40 + ((uint32_t)((warp & 3) * 32) << 16), own(1), v);
      const bool none = __popc(far_warps()) == n_units;  // (no MMA has been issued)
#pragma unroll
      for (int j = 0; j < 10; ++j) base[S + (wg * 10 + j) * INT_S_STR + (warp & 3) * 32 + lanes.lane] = none ? 0.f : v[j];
    }
    tc_fence_before();
    if (g.test_code == 613 && warp == NWARPS - 1)  // (nothing ends this phase)
      res_wait(bar_read(0), ph ^ 1, g, limit, 613, ok);
  }

  // Words of W0 and b0 go to the threads of the same number; those of W1 and b1 and the log-likelihood to the last warp
  static constexpr int LAST = NWARPS - 1, NW1 = Words::N - 1 - Words::W0;
  static_assert(NW1 < 32 && Words::W0 <= LAST * 32, "word assignment");
  __device__ __forceinline__ int collects() const {
    if (warp == LAST) return lanes.lane <= NW1 ? Words::W0 + lanes.lane : -1;
    return (int)threadIdx.x < Words::W0 ? (int)threadIdx.x : -1;
  }
  __device__ __forceinline__ bool collect(bool last, uint4& v) const {
    float s[3] = {};
    if (warp == LAST) {
      const float* r = base + RW1 + 3 * min(lanes.lane, NW1 - 1);
#pragma unroll 2
      for (int w = 0; w < NWARPS; ++w)
#pragma unroll
        for (int q = 0; q < 3; ++q) s[q] += r[w * RS + q];
      v = make_uint4(__float_as_uint(s[0]), __float_as_uint(s[1]), __float_as_uint(s[2]), 0u);
      if (last && lanes.lane == NW1) {
        const double* d = reinterpret_cast<const double*>(base + RLL);
        double t[2] = {};
#pragma unroll 2
        for (int w = 0; w < NWARPS; ++w) t[w & 1] += d[w];
        const uint2 u = d2u(t[0] + t[1]);
        v.x = u.x;
        v.y = u.y;
      }
      return lanes.lane <= NW1;
    }
    if (threadIdx.x == 0) *stat(par) = 0u;  // the step's, whose scale has been read
    const int t = min((int)threadIdx.x, Words::W0 - 1);
    const float inv = sum_f();
    // parameter 3 t + q: feature k, unit j
    const int k0 = 3 * t / H, j0 = 3 * t - k0 * H;
    float w1[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const bool next = j0 + q >= H;
      const int j = next ? j0 + q - H : j0 + q;
      s[q] = n_units > 0 ? int_sum4(base + S, next ? k0 + 1 : k0, j) * inv : 0.f;
      w1[q] = base[W1 + j];
    }
    const uint32_t fb = far_warps();
    if (__builtin_expect(fb != 0u, 0)) {  // what went by FFMA
      const float* gp = base + ES + 3 * t + 8 * (3 * t / GROUP);
#pragma unroll 1
      for (int w0 = 0; w0 < n_units; w0 += 4, gp += 4 * Warp::ES)
#pragma unroll
        for (int w = 0; w < 4; ++w)
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const float v = gp[w * Warp::ES + q];
            s[q] += fb >> (w0 + w) & 1 ? v : 0.f;
          }
    }
    float o[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) o[q] = w1[q] * s[q];
    // (a place without a parameter would get the sum of target x dL/dz, and its value a vote on the path in `stage`)
    if (t == Words::W0 - 1 && Words::PAD == 1) o[2] = 0.f;
    v = make_uint4(__float_as_uint(o[0]), __float_as_uint(o[1]), __float_as_uint(o[2]), 0u);
    return (int)threadIdx.x < Words::W0;
  }
  __device__ __forceinline__ void teardown(const ResidentParams& g, const volatile int& dead) {
    tc_fence_before();
    __syncthreads();
    if (warp == 0 && dead)
      for (int w = 0; w <= nt; ++w) res_drain(w < nt ? bar_fwd(w) : bar_sum(), par ^ 1, g);
    if (warp == 0)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS)
                   : "memory");
  }
};

// Windows whose CTAs have one tile at most take the tile arithmetic without integers (resident_fp32_ffma.cu): as fast there, and an outlier
// costs it nothing.  us a step, integers and FFMA (ten a trajectory): 148 windows of 128 rows 4.88, 4.15; 1000 rows 5.00, 4.52; 4097 6.10, 5.76; with
// targets that are outliers 1000 rows 6.2, 4.51.  More tiles: 8 x 4096 rows 7.0, 8.4; 16384 6.55, 7.5; 58368 8.5, 10.1; with outliers, a hundred a trajectory, 9.6, 9.65.
// So do evaluations on host pointers and calls of one step, for which making integers of the rows and a scale, 1 to 2 us together, does not pay.
// us a call alone, integers and FFMA: evaluations of 2048, 20000 and 58368 rows 37.0, 39.5, 42.4 and 35.3, 37.3, 41.0; us a call among others: one step
// of 1500, 2048, 4096, 20000 and 58368 rows 17.1, 18.1, 20.9, 19.8, 23.0 and 15.8, 16.1, 18.9, 16.9, 20.9 (with FFMA for all calls of several tiles 16.8, 16.8,
// 20.3, 18.8, 22.5).  Two steps of 2048, 20000 and 58368 rows, alone: 33.4, 36.9, 41.7 and 37.6, 44.2, 49.8.
bool resident_one_tile(int rows, int clusters, int cluster) {
  const int units = (rows + 31) / 32, ctas = clusters * cluster;
  return (units + ctas - 1) / ctas <= 4;
}
cudaError_t launch_resident_fp32(int cluster, const void* tmap, const ResidentParams& g, cudaStream_t st,
                                 int* max_clusters) {
  if (!max_clusters && cluster == 8 && g.mode == RES_STEPS && g.n_steps == 1 && !resident_one_tile(g.n_rows, g.clusters, cluster))
    return launch_resident_step_fp32(tmap, g, st);
  if (!max_clusters)
    return resident_one_tile(g.n_rows, g.clusters, cluster) ? launch_resident_fp32_ffma(cluster, tmap, g, st, nullptr)
                                                   : resident_launch_any<ResFp32>(cluster, tmap, g, st, nullptr);
  int n = 0;
  cudaError_t e = resident_launch_any<ResFp32>(cluster, tmap, g, st, max_clusters);
  if (e == cudaSuccess) e = launch_resident_fp32_ffma(cluster, tmap, g, st, &n);
  if (e == cudaSuccess && n < *max_clusters) *max_clusters = n;
  return e;
}

}  // namespace mcmc_b200
