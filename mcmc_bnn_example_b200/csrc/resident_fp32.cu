// Tile arithmetic of the resident kernel in FP32 mode (resident.cuh has the launch structure, fp32_tile.cuh what a warp
// does with its 32 rows): every warp owns one 32-row unit for the whole launch.
// One launch per step took 29.5 us a step for a 58368-row window, this takes 12.5 (2000 steps, one B200); a log density
// and gradient of 1000 rows from host pointers takes 30 us instead of 64.
// What bounds a step: no pipe (at 512 rows a CTA the one that serves shared memory is 71 % busy, issue slots 58 %, FMA 52 %).
// A block takes a scheduler 3,600 cycles, of which its multiplications keep the FMA pipe busy for 2,240: they, the tanh and the
// multiplications after it overlap as far as the warps of a scheduler are in different phases.  Then the exchange.
#include <cuda.h>
#include "fp32_tile.cuh"
#include "resident.cuh"

namespace mcmc_b200 {

struct ResFp32 {
  static constexpr int H = 40, D = 22;
  using Words = ResWords<H>;
  using Warp = Fp32Warp<H>;
  static constexpr int NWARPS = RES_NWG * 4;
  static_assert(Warp::ROWS == 32 && NWARPS == RES_UNITS, "a warp owns one 32-row unit");
  // a warp's sums of dW0 and db0, after the shuffle over its two row subsets a lane's 6 features x 5 units: eight
  // floats between the feature groups make the stores free of bank conflicts.  They take the place of its dL/dz.
  static constexpr int GROUP = 6 * H, GSTR = GROUP + 8;
  static_assert(4 * GSTR <= Warp::ES, "sums fit where dL/dz was");
  static constexpr int RS = H + 4;   // dW1 and db1 of a warp's rows
  // float offsets
  static constexpr int XB = 0, ES = XB + RES_UNITS * 32 * KP, WP = ES + NWARPS * Warp::ES, B0 = WP + Warp::WP,
                       W1 = B0 + H, RW1 = W1 + RS, DYS = RW1 + NWARPS * RS, RLL = DYS + NWARPS * 32,
                       DUMMY = RLL + NWARPS * 2, BAR = DUMMY + 4;
  static constexpr size_t SMEM = 1024 + (BAR + 4) * 4;
  static_assert(WP % 4 == 0 && DYS % 4 == 0 && RLL % 2 == 0 && BAR % 2 == 0, "vector alignment");

  // The four warps of a scheduler get the weights at the same moment.  In step with one another they would all multiply,
  // then all wait for their tanh (646 cycles of the MUFU pipe each), and so on; so each starts this many cycles after the
  // one before it, about the multiplications of half a block.  58368 rows, us a step: 12.91 (0), 12.61 (300), 12.46 (500
  // to 700), 12.57 (1000), 12.69 (1300).  Two to four units to a scheduler, 0 and 600: 1100 rows 7.10, 6.98; 2048 rows 7.61,
  // 7.43; 3000 rows 9.60, 9.22; 4096 rows 11.75, 11.14; single evaluations 0 to 0.6 less.  A scheduler's first unit never
  // waits.
  static constexpr uint32_t TURN = 600;

  Warp lanes;
  float* base;
  int warp, n_units;
  int row0;          // this warp's first row in the window
  bool active;
  uint32_t s_dst[3];

  __device__ __forceinline__ ResFp32(unsigned char* b, const ResidentParams& g, int, int u0, int u1)
      : base(reinterpret_cast<float*>(b)) {
    warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    n_units = u1 - u0;
    active = warp < n_units;
    row0 = (u0 + warp) * 32;
    const int t = threadIdx.x;
    for (int q = 0; q < 3; ++q) {
      const int p = Words::param(t, q);
      float* dst = base + DUMMY;
      if (t < Words::N - 1 && Words::valid(t, q))
        dst = base + (p < D * H ? WP + Warp::w_off(p / H, p % H) : p < D * H + H ? B0 + p - D * H : W1 + p - (D * H + H));
      s_dst[q] = smem_u32(dst);
    }
  }

  __device__ __forceinline__ bool setup(const CUtensorMap*, const ResidentParams& g, int win) {
    bool ok = true;
    const int tid = threadIdx.x;
    uint64_t* bar = reinterpret_cast<uint64_t*>(base + BAR);
    if (tid == 0) {
      mbar_init(bar, 1);
      mbar_fence_init();
    }
    // sums that nothing writes stay zero: those of warps without rows
    for (int i = tid; i < (WP - ES) / 4; i += RES_THREADS)
      reinterpret_cast<float4*>(base + ES)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = tid; i < DUMMY - RW1; i += RES_THREADS) base[RW1 + i] = 0.f;
    __syncthreads();
    if (n_units > 0) {
      const uint32_t bytes = (uint32_t)n_units * 32 * KP * 4;
      if (tid == 0) {
        mbar_expect_tx(bar, bytes);
        bulk_g2s(base + XB, g.xaug + ((size_t)(g.data_window0 + win) * g.rows_pad + row0) * KP, bytes, bar);
      }
      res_wait(bar, 0, g, g.wait_ticks << 2, 611, ok);
      if (!ok) res_drain(bar, 0, g);
      if (g.test_code == 611) res_wait(bar, 1, g, g.wait_ticks << 2, 611, ok);  // (nothing ends this phase)
    }
    __syncthreads();
    return ok;
  }

  // word `threadIdx.x` of the weights
  __device__ __forceinline__ void stage(const uint4& v) {
    const uint32_t x[3] = {v.x, v.y, v.z};
#pragma unroll
    for (int q = 0; q < 3; ++q) asm volatile("st.shared.b32 [%0], %1;" ::"r"(s_dst[q]), "r"(x[q]) : "memory");
    __syncthreads();
  }

  __device__ __forceinline__ void step(const ResidentParams& g, float* row_loss, bool last, bool&) {
    if (!active) return;
    if (warp >= 4) {  // (a scheduler's first warp waits for nothing: looking at the clock cost it 0.02 to 0.04 us a step)
      const uint32_t t0 = (uint32_t)clock64();
      while ((uint32_t)clock64() - t0 < (uint32_t)(warp >> 2) * TURN) {}
    }
    const float* xb = base + XB + warp * 32 * KP;
    float* es = base + ES + warp * Warp::ES;
    uint64_t dw1[Warp::HPL] = {};
    float dy = 0.f, loss;
    const int left = g.n_rows - row0;
    if (last) {
      lanes.block<true>(xb, base + WP, base + B0, base + W1, base[W1 + H], g.lik, left, base + DYS + warp * 32, es, dw1,
                        dy, loss);
      const int r = lanes.loss_row();
      if (row_loss && r < left) row_loss[row0 + r] = loss;
      double ld = (double)loss;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, o);
      if (lanes.lane == 0) reinterpret_cast<double*>(base + RLL)[warp] = ld;
    } else {
      lanes.block<false>(xb, base + WP, base + B0, base + W1, base[W1 + H], g.lik, left, base + DYS + warp * 32, es, dw1,
                         dy, loss);
    }
    uint64_t acc[Warp::KPT / 2][Warp::HPL];
#pragma unroll
    for (int k = 0; k < Warp::KPT / 2; ++k)
#pragma unroll
      for (int j = 0; j < Warp::HPL; ++j) acc[k][j] = 0ull;
    lanes.backward<2>(xb, es, acc);
    // dW1 over the four row groups (lane bits 0 and 2), db1 over the rows
    float* rw1 = base + RW1 + warp * RS;
#pragma unroll
    for (int j = 0; j < Warp::HPL; ++j) {
      float a, b;
      unpack2(dw1[j], a, b);
      a += b;
      a += __shfl_xor_sync(0xffffffffu, a, 1);
      a += __shfl_xor_sync(0xffffffffu, a, 4);
      if (lanes.rg == 0) rw1[lanes.cg * Warp::HPL + j] = a;
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) dy += __shfl_xor_sync(0xffffffffu, dy, o);
    if (lanes.lane == 0) rw1[H] = dy;
    // dW0: lanes 16 apart have the two row subsets; the lower one keeps features 0 - 5 of the twelve, the upper 6 - 11
    __syncwarp();  // dL/dz has been read by every lane
    float* gp = es + (2 * lanes.kh + lanes.rsub) * GSTR + lanes.bcg * Warp::HPL;
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int j = 0; j < Warp::HPL; ++j) {
        float s0, s1, k0, k1;
        unpack2(lanes.rsub ? acc[k][j] : acc[k + 3][j], s0, s1);
        unpack2(lanes.rsub ? acc[k + 3][j] : acc[k][j], k0, k1);
        gp[2 * k * H + j] = k0 + __shfl_xor_sync(0xffffffffu, s0, 16);
        gp[(2 * k + 1) * H + j] = k1 + __shfl_xor_sync(0xffffffffu, s1, 16);
      }
  }

  // Words of W0 and b0 go to the threads of the same number; those of W1 and b1 and the log-likelihood to the last warp
  static constexpr int LAST = NWARPS - 1, NW1 = Words::N - 1 - Words::W0;
  static_assert(NW1 < 32 && Words::W0 <= LAST * 32, "word assignment");
  __device__ __forceinline__ int collects() const {
    if (warp == LAST) return lanes.lane <= NW1 ? Words::W0 + lanes.lane : -1;
    return (int)threadIdx.x < Words::W0 ? (int)threadIdx.x : -1;
  }
  __device__ __forceinline__ bool collect(bool last, uint4& v) const {
    float s[3][2] = {};
    if (warp == LAST) {
      const float* r = base + RW1 + 3 * min(lanes.lane, NW1 - 1);
#pragma unroll
      for (int w = 0; w < NWARPS; ++w)
#pragma unroll
        for (int q = 0; q < 3; ++q) s[q][w & 1] += r[w * RS + q];
      v = make_uint4(__float_as_uint(s[0][0] + s[0][1]), __float_as_uint(s[1][0] + s[1][1]),
                     __float_as_uint(s[2][0] + s[2][1]), 0u);
      if (last && lanes.lane == NW1) {
        const double* d = reinterpret_cast<const double*>(base + RLL);
        double t[2] = {};
#pragma unroll
        for (int w = 0; w < NWARPS; ++w) t[w & 1] += d[w];
        const uint2 u = d2u(t[0] + t[1]);
        v.x = u.x;
        v.y = u.y;
      }
      return lanes.lane <= NW1;
    }
    const int t = min((int)threadIdx.x, Words::W0 - 1);
    const float* gp = base + ES + 3 * t + 8 * (3 * t / GROUP);
#pragma unroll
    for (int w = 0; w < NWARPS; ++w)
#pragma unroll
      for (int q = 0; q < 3; ++q) s[q][w & 1] += gp[w * Warp::ES + q];
    float o[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) o[q] = base[W1 + (3 * t + q) % H] * (s[q][0] + s[q][1]);
    v = make_uint4(__float_as_uint(o[0]), __float_as_uint(o[1]), __float_as_uint(o[2]), 0u);
    return (int)threadIdx.x < Words::W0;
  }
  __device__ __forceinline__ void teardown(const ResidentParams&, const volatile int&) {}
};

cudaError_t launch_resident_fp32(int cluster, const void* tmap, const ResidentParams& g, cudaStream_t st,
                                 int* max_clusters) {
  switch (cluster) {
    case 1: return resident_launch(resident_kernel<ResFp32, 1, ResidentParams>, 1, ResFp32::SMEM, tmap, g, st, max_clusters);
    case 2: return resident_launch(resident_kernel<ResFp32, 2, ResidentParams>, 2, ResFp32::SMEM, tmap, g, st, max_clusters);
    case 4: return resident_launch(resident_kernel<ResFp32, 4, ResidentParams>, 4, ResFp32::SMEM, tmap, g, st, max_clusters);
    case 8: return resident_launch(resident_kernel<ResFp32, 8, ResidentParams>, 8, ResFp32::SMEM, tmap, g, st, max_clusters);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_resident_eval_fp32(const void* tmap, const ResidentEvalParams& g, cudaStream_t st) {
  return resident_launch_eval<ResFp32>(tmap, g, st);
}

}  // namespace mcmc_b200
