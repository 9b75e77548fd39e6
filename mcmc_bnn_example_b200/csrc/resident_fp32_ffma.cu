// Tile arithmetic of the resident kernel in FP32 mode for CTAs of one tile (128 rows) at most, for evaluations on host
// pointers and for calls of one step: the forward product on the tensor core (split_mma.cuh), the backward pass by FFMA, every warp for itself (fp32_split.cuh).
// resident_fp32.cu has the rest, and the line between the two.  The rows' three parts stay in tensor memory for the launch, the rows
// themselves in shared memory.
// us a step on one B200 (ten a trajectory): 1000 rows (one cluster of eight) 4.5, 148 windows of 128 rows 4.15, 4097 rows (five clusters) 5.8.  A chain of
// latencies: weights cut up, 24 MMAs, 40 tanh a row, 960 products of 32 rows a warp (2,250 cycles), exchange (resident.cuh).
#include <cuda.h>
#include "fp32_split.cuh"
#include "resident.cuh"

namespace mcmc_b200 {

template <int TILES>
struct ResFp32Ffma {
  static constexpr int H = SPLIT_H, D = SPLIT_D;
  using Words = ResWords<H>;
  using Warp = SplitWarp;
  static constexpr int NWARPS = RES_NWG * 4, ROW_WARPS = 4 * TILES;   // those with rows, a 32-row unit each
  // a warp's sums of dW0 and db0, after the shuffle over its two row subsets a lane's 6 features x 5 units: eight
  // floats between the feature groups make the stores free of bank conflicts.  They take the place of its dL/dz.
  static constexpr int GROUP = 6 * H, GSTR = GROUP + 8;
  static_assert(4 * GSTR <= Warp::ES, "sums fit where dL/dz was");
  static constexpr int RS = H + 4;   // dW1 and db1 of a warp's rows
  // float offsets
  static constexpr int WB = 0, XB = WB + SPLIT_B_BYTES / 4, ES = XB + ROW_WARPS * 32 * KP, W1 = ES + ROW_WARPS * Warp::ES,
                       RW1 = W1 + RS, RLL = RW1 + ROW_WARPS * RS, BAR = RLL + ROW_WARPS * 2;
  static constexpr bool TURNS = TILES > 1;
  // barriers: rows landed; per tile, forward done; per accumulator buffer that tiles share, read
  static constexpr int NZ = TURNS ? 2 : 1, NBARS = 1 + TILES + (TURNS ? NZ : 0);
  static constexpr size_t SMEM = 1024 + (BAR + 2 * NBARS) * 4;
  static_assert(XB % 4 == 0 && W1 % 4 == 0 && RW1 % 4 == 0 && RLL % 2 == 0 && BAR % 2 == 0, "vector alignment");
  // accumulators, which the tiles take in turn; the rows' parts for the whole launch
  static constexpr int A_COL0 = NZ * SPLIT_Z_COLS, TMEM_COLS = TURNS ? 512 : 256;
  static_assert(A_COL0 + TILES * SPLIT_A_COLS <= TMEM_COLS, "tensor memory budget");
  static __device__ __forceinline__ uint32_t a_col(int w) { return A_COL0 + w * SPLIT_A_COLS; }
  static __device__ __forceinline__ uint32_t z_col(int w) { return w % NZ * SPLIT_Z_COLS; }
  // named barriers: a warp's turn is over (those of the last four are not needed)
  static constexpr int BAR_LO = 1, BAR_HI = 10;
  static_assert(BAR_LO + 8 <= RES_BAR_X && BAR_HI > RES_BAR_X && BAR_HI + 4 <= 16, "barrier numbers");
  __device__ __forceinline__ static int bar_turn(int w) { return w < 8 ? BAR_LO + w : BAR_HI + w - 8; }
  static constexpr bool X_PLACE = false;
  Warp lanes;
  float* base;
  int warp, wg, n_units;
  int row0;          // this warp's first row in the window
  bool active, plain_x, plain;
  uint32_t s_dst[3], tmem, par;

  __device__ __forceinline__ uint64_t* bar_rows() const { return reinterpret_cast<uint64_t*>(base + BAR); }
  __device__ __forceinline__ uint64_t* bar_fwd(int w) const { return bar_rows() + 1 + w; }
  __device__ __forceinline__ uint64_t* bar_read(int b) const { return bar_rows() + 1 + TILES + b; }

  __device__ __forceinline__ ResFp32Ffma(unsigned char* b, const ResidentParams& g, int, int u0, int u1)
      : base(reinterpret_cast<float*>(b)) {
    warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    wg = TURNS ? warp >> 2 : 0;
    n_units = u1 - u0;
    active = warp < n_units;
    row0 = (u0 + warp) * 32;
    par = 0;
    plain_x = plain = false;
    const int t = threadIdx.x;
    for (int q = 0; q < 3; ++q) {
      const int p = Words::param(t, q);
      // (threads and places of a word without a parameter write where feature 28 of unit 0 would be: nobody reads there)
      s_dst[q] = smem_u32(b) + split_b_off(0, 28);
      if (t >= Words::N - 1 || !Words::valid(t, q)) continue;
      if (p < D * H + H) s_dst[q] = smem_u32(b) + split_b_off(p % H, p / H & ~3) + (p / H & 3) * 4;
      else s_dst[q] = smem_u32(base + W1 + p - (D * H + H));
    }
  }

  __device__ __forceinline__ bool setup(const CUtensorMap*, const ResidentParams& g, int win) {
    __shared__ uint32_t tmem_slot;
    bool ok = true;
    const int tid = threadIdx.x;
    if (warp == 0) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                   "r"((uint32_t)TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
      mbar_init(bar_rows(), 1);
      for (int w = 0; w < TILES; ++w) mbar_init(bar_fwd(w), 1);
      for (int b = 0; TURNS && b < NZ; ++b) mbar_init(bar_read(b), 4);
      mbar_fence_init();
    }
    // sums that nothing writes stay zero: those of warps without rows; and what the last MMAs read behind the weights
    for (int i = tid; i < (W1 - ES) / 4; i += RES_THREADS)
      reinterpret_cast<float4*>(base + ES)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = tid; i < (XB - WB) / 4; i += RES_THREADS)
      reinterpret_cast<float4*>(base + WB)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = tid; i < BAR - RW1; i += RES_THREADS) base[RW1 + i] = 0.f;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = tmem_slot;
    bool wide = false;
    if (n_units > 0) {
      const uint32_t bytes = (uint32_t)n_units * 32 * KP * 4;
      if (tid == 0) {
        mbar_expect_tx(bar_rows(), bytes);
        bulk_g2s(base + XB, g.xaug + ((size_t)(g.data_window0 + win) * g.rows_pad + row0) * KP, bytes, bar_rows());
      }
      res_wait(bar_rows(), 0, g, g.wait_ticks << 2, 611, ok);
      if (!ok) res_drain(bar_rows(), 0, g);
      if (g.test_code == 611) res_wait(bar_rows(), 1, g, g.wait_ticks << 2, 611, ok);  // (nothing ends this phase)
      if (TURNS ? 4 * wg < n_units : warp < ROW_WARPS) {  // the tile's rows to tensor memory, zeros for warps without rows
        const float* x = base + XB + tid * KP;
        const uint32_t a_t = tmem + a_col(wg) + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          float v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            v[k] = active && 8 * j + k <= D ? x[8 * j + k] : 0.f;
            wide |= split_wide(v[k]);
          }
          split_store_row(a_t, j, v);
        }
        tc_wait_st();
        tc_fence_before();
      }
    }
    plain_x = __syncthreads_or(wide) != 0;
    return ok;
  }

  // word `threadIdx.x` of the weights
  __device__ __forceinline__ void stage(const uint4& v) {
    const uint32_t x[3] = {v.x, v.y, v.z};
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

  __device__ __forceinline__ void step(const ResidentParams& g, float* row_loss, bool last, bool& ok) {
    if (n_units == 0) return;
    const uint32_t ph = par;
    par ^= 1;
    const int nt = TURNS ? (n_units + 3) / 4 : 1;
    if (warp == NWARPS - 1) {  // (rows of its own, if any, come last)
      const uint32_t on = elect_one(), tm = __shfl_sync(0xffffffffu, tmem, 0);
      for (int w = 0; w < nt; ++w) {
        if (w >= NZ) res_wait(bar_read(w % NZ), ph, g, g.wait_ticks << 2, 613, ok);  // a buffer's second tile when its first has been read
        tc_fence_after();
        split_issue(tm + z_col(w), tm + a_col(w), smem_u32(base + WB), on);
        tc_commit_if(bar_fwd(w), on);
      }
      if (g.test_code == 613)  // (nothing ends the second phase)
        for (uint32_t p = 0; p < 2; ++p) res_wait(bar_fwd(0), ph ^ p, g, g.wait_ticks << 2, 613, ok);
    }
    if (!active) return;
    const float* xb = base + XB + warp * 32 * KP;
    float* es = base + ES + warp * Warp::ES;
    const int left = g.n_rows - row0;
    uint64_t h[4][5];
    res_wait(bar_fwd(wg), ph, g, g.wait_ticks << 2, 612, ok);
    tc_fence_after();
    lanes.load(tmem + z_col(wg) + ((uint32_t)((warp & 3) * 32) << 16), h);
    tc_fence_before();
    if (TURNS && wg + NZ < nt) {  // another tile takes the buffer (so this one is full: all its warps come here)
      __syncwarp();
      if (lanes.lane == 0) mbar_arrive(bar_read(wg % NZ));
    }
    if (plain) {
      Warp::plain<2>(xb, reinterpret_cast<const unsigned char*>(base + WB), es);
      lanes.load_plain(es, h);
    }
    uint64_t dw1[5] = {};
    float dy, pred;
    const int own = lanes.own();
    const bool valid = own < left;
    const float y = xb[own * KP + COL_Y];
    // (a scheduler's four warps take turns at the tanh: resident_fp32.cu)
    if (TURNS && warp >= 4) named_sync(bar_turn(warp - 4), 64);
    lanes.block(h, base + W1, g.lik, y, valid, es, dw1, dy, pred, [&](int i) {
      if (TURNS && i == 3 && warp + 4 < n_units) named_arrive(bar_turn(warp), 64);
    });
    if (last) {
      if (g.test_code == 612) res_wait(bar_fwd(wg), ph ^ 1, g, g.wait_ticks << 2, 612, ok);  // (nothing ends this phase)
      const float loss = valid ? lik_loss(g.lik, y, pred) : 0.f;
      store_row_loss(row_loss, row0 + own, loss, valid);
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
    uint64_t acc[Warp::KPT / 2][Warp::UPT] = {};
    lanes.backward<2>(xb, es, acc);
    // dW0: lanes 16 apart have the two row subsets; the lower one keeps features 0 - 5 of the twelve, the upper 6 - 11
    __syncwarp();  // dL/dz has been read by every lane
    lanes.store_dw0(acc, es + (2 * lanes.kh + lanes.rsub) * GSTR);
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
#pragma unroll 4
      for (int w = 0; w < ROW_WARPS; ++w)
#pragma unroll
        for (int q = 0; q < 3; ++q) s[q] += r[w * RS + q];
      v = make_uint4(__float_as_uint(s[0]), __float_as_uint(s[1]), __float_as_uint(s[2]), 0u);
      if (last && lanes.lane == NW1) {
        const double* d = reinterpret_cast<const double*>(base + RLL);
        double t[2] = {};
#pragma unroll
        for (int w = 0; w < ROW_WARPS; ++w) t[w & 1] += d[w];
        const uint2 u = d2u(t[0] + t[1]);
        v.x = u.x;
        v.y = u.y;
      }
      return lanes.lane <= NW1;
    }
    const int t = min((int)threadIdx.x, Words::W0 - 1);
    const float* gp = base + ES + 3 * t + 8 * (3 * t / GROUP);
    // (four warps to a turn: straight code for sixteen took 1,100 of a step's cycles to fetch)
#pragma unroll 1
    for (int w0 = 0; w0 < (TURNS ? n_units : 1); w0 += 4, gp += 4 * Warp::ES)
#pragma unroll
      for (int w = 0; w < 4; ++w)
#pragma unroll
        for (int q = 0; q < 3; ++q) s[q] += gp[w * Warp::ES + q];
    float o[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) o[q] = base[W1 + (3 * t + q) % H] * s[q];
    // (a place without a parameter would get the sum of target x dL/dz, and its value a vote on the path in `stage`)
    if (t == Words::W0 - 1 && Words::PAD == 1) o[2] = 0.f;
    v = make_uint4(__float_as_uint(o[0]), __float_as_uint(o[1]), __float_as_uint(o[2]), 0u);
    return (int)threadIdx.x < Words::W0;
  }
  __device__ __forceinline__ void teardown(const ResidentParams& g, const volatile int& dead) {
    tc_fence_before();
    __syncthreads();
    if (warp == 0 && dead)
      for (int w = 0; 4 * w < n_units; ++w) res_drain(bar_fwd(w), par ^ 1, g);
    if (warp == 0)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS)
                   : "memory");
  }
};

cudaError_t launch_resident_fp32_ffma(int cluster, const void* tmap, const ResidentParams& g, cudaStream_t st,
                                      int* max_clusters) {
  return resident_launch_any<ResFp32Ffma<1>>(cluster, tmap, g, st, max_clusters);
}

cudaError_t launch_resident_eval_fp32(const void* tmap, const ResidentEvalParams& g, cudaStream_t st) {
  return (g.n_rows + 31) / 32 <= 4 * 8 * g.clusters ? resident_launch_single<ResFp32Ffma<1>>(tmap, g, st)
                                                    : resident_launch_single<ResFp32Ffma<RES_NWG>>(tmap, g, st);
}
cudaError_t launch_resident_step_fp32(const void* tmap, const ResidentParams& g, cudaStream_t st) {
  return resident_launch_single<ResFp32Ffma<RES_NWG>>(tmap, g, st);
}

}  // namespace mcmc_b200
