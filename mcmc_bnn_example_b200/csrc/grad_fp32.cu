// FP32 (FFMA) fused leapfrog-update + forward + backward kernel.
//
// Stands in for leapfrog_step_kernel of the reference
// (include/mcmc/mcmc_step_ffma.h:154-379): same math, different mapping.
//   * grid = (slices, windows): many independent windows per launch, each
//     window's rows split over `slices` CTAs;
//   * every warp works through its own row blocks (fp32_tile.cuh), which arrive through the bulk-copy engine double
//     buffered: nothing in the row loop waits for another warp;
//   * dW0 stays in the lanes' registers for the whole range (the reference keeps it in shared memory and adds to it
//     with atomics, mcmc_step_ffma.h:346-367);
//   * no atomics: the warps' sums -> shared memory -> one partial vector per CTA; the next launch (or the accept
//     kernel) sums the partials of a window in a fixed order, so results are bit-reproducible.
#include "fp32_tile.cuh"

namespace mcmc_b200 {

constexpr int FP32_TILE = 128;

template <int H>
struct Fp32Geom {
  using Warp = Fp32Warp<H>;
  static constexpr int NW = FP32_TILE / Warp::ROWS, NT = NW * 32;
  static constexpr int PP = (Warp::P + 3) / 4 * 4;
  static constexpr int XS = Warp::ROWS * KP;          // floats of a block's rows
  static constexpr int WARP = 2 * XS + Warp::ES + Warp::ROWS;   // two stages of rows, dL/dz, dL/dpred
  static constexpr int SUBS = NW * Warp::RSUB;        // row subsets whose dW0 is added up at the end
  static constexpr int BIG = NW * WARP > SUBS * PP ? NW * WARP : SUBS * PP;   // the sums take the place of the blocks
  static constexpr size_t SMEM = sizeof(float) * (BIG + Warp::WP + 2 * H + 4);
};

template <int H, int MINB>
__global__ void __launch_bounds__(Fp32Geom<H>::NT, MINB) grad_fp32_kernel(const GradParams g) {
  using G = Fp32Geom<H>;
  using Warp = Fp32Warp<H>;
  constexpr int D = Warp::D, HPL = Warp::HPL, KPT = Warp::KPT, NT = G::NT, NW = G::NW, PP = G::PP;
  constexpr uint32_t BLOCK_BYTES = G::XS * sizeof(float);

  extern __shared__ __align__(128) float smem[];
  float* const wp = smem + G::BIG;      // W0 in pairs of features
  float* const b0 = wp + Warp::WP;
  float* const w1 = b0 + H;             // W1, b1
  __shared__ __align__(8) uint64_t bars[NW][2];
  __shared__ float red_w1[NW][H];
  __shared__ float red_db1[NW];
  __shared__ double red_ll[NW];

  const Warp lanes;
  const int tid = threadIdx.x, lane = lanes.lane;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int win = blockIdx.y;
  const int slice = blockIdx.x;
  const int S = gridDim.x;
  const int t0 = (int)((long long)slice * g.n_tiles / S);
  const int t1 = (int)((long long)(slice + 1) * g.n_tiles / S);
  float* const xs = smem + warp * G::WARP;
  float* const es = xs + 2 * G::XS;
  float* const dys = es + Warp::ES;
  const float* const src = g.xaug + (long long)(g.data_window0 + win) * g.window_stride + warp * G::XS;
  auto fetch = [&](int t) {
    const int st = (t - t0) & 1;
    mbar_expect_tx(&bars[warp][st], BLOCK_BYTES);
    bulk_g2s(xs + st * G::XS, src + (size_t)t * FP32_TILE * KP, BLOCK_BYTES, &bars[warp][st]);
  };

  if (lane == 0) {
    mbar_init(&bars[warp][0], 1);
    mbar_init(&bars[warp][1], 1);
    mbar_fence_init();
  }
  __syncwarp();
  // The first rows may be fetched ahead of the dependency wait only when no kernel directly before
  // this one in the stream wrote the dataset (inside a chain none does; right after a repack one did).
  const bool early_rows = g.data_fresh == 0;
  if (lane == 0 && t0 < t1 && early_rows) fetch(t0);
  pdl_trigger();
  pdl_wait();
  if (lane == 0 && t0 < t1 && !early_rows) fetch(t0);
  // fused leapfrog update; parameters land in the layout the lanes read
  {
    float w[(Warp::P + NT - 1) / NT];
    leapfrog_params(g, win, tid, NT, Warp::P, slice == 0, w);
#pragma unroll
    for (int i = 0; i < (Warp::P + NT - 1) / NT; ++i) {
      const int p = tid + i * NT;
      if (p < Warp::P) wp[p < D * H ? Warp::w_off(p / H, p % H) : p + (Warp::WP - D * H)] = w[i];
    }
  }
  __syncthreads();

  uint64_t acc[KPT / 2][HPL], dw1[HPL];
#pragma unroll
  for (int j = 0; j < HPL; ++j) {
    dw1[j] = 0ull;
#pragma unroll
    for (int k = 0; k < KPT / 2; ++k) acc[k][j] = 0ull;
  }
  float db1 = 0.f;
  double llacc = 0.0;
  bool ok = true;

#pragma unroll 1
  for (int t = t0; t < t1 && ok; ++t) {
    const int it = t - t0;
    if (lane == 0 && t + 1 < t1) fetch(t + 1);
    ok = __all_sync(0xffffffffu, mbar_wait(&bars[warp][it & 1], (it >> 1) & 1, g.status, 101));
    const float* xb = xs + (it & 1) * G::XS;
    const int r0 = t * FP32_TILE + warp * Warp::ROWS;
    float loss;
    lanes.template block<true>(xb, wp, b0, w1, w1[H], g.lik, g.n_rows - r0, dys, es, dw1, db1, loss);
    if (lanes.loss_first()) {
      llacc += (double)loss;
      const int row = r0 + lanes.loss_row();
      if (g.row_loss && row < g.n_rows) g.row_loss[(long long)win * g.row_loss_stride + row] = loss;
    }
    lanes.template backward<8>(xb, es, acc);
    __syncwarp();  // rows and dL/dz have been read: the next copy and the next block may overwrite them
  }

  // ---- reduce: row subsets / row groups -> CTA partial ----
  // dW1: the lanes that share a unit group; db1: a row is in lanes 16 (128 units: 8 and 16) apart
  float v1[HPL];
#pragma unroll
  for (int j = 0; j < HPL; ++j) {
    float a, b;
    unpack2(dw1[j], a, b);
    a += b;
    a += __shfl_xor_sync(0xffffffffu, a, 1);
    v1[j] = H == 40 ? a + __shfl_xor_sync(0xffffffffu, a, 4) : a;
  }
  if (lanes.rg == 0) {
#pragma unroll
    for (int j = 0; j < HPL; ++j) red_w1[warp][lanes.cg * HPL + j] = v1[j];
  }
#pragma unroll
  for (int o = H == 40 ? 8 : 4; o > 0; o >>= 1) db1 += __shfl_xor_sync(0xffffffffu, db1, o);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) llacc += __shfl_xor_sync(0xffffffffu, llacc, o);
  if (lane == 0) {
    red_db1[warp] = db1;
    red_ll[warp] = llacc;
  }
  __syncthreads();  // every warp is done with its rows
  {
    float* r = smem + (warp * Warp::RSUB + lanes.rsub) * PP;
#pragma unroll
    for (int k = 0; k < KPT; ++k) {
      const int kk = lanes.kh * KPT + k;
      if (kk <= D) {  // feature 23 is y: not a gradient row
#pragma unroll
        for (int j = 0; j < HPL; ++j) {
          float lo, hi;
          unpack2(acc[k / 2][j], lo, hi);
          r[kk * H + lanes.bcg * HPL + j] = (k & 1) ? hi : lo;
        }
      }
    }
  }
  __syncthreads();
  float* po = g.partial_out + ((size_t)win * S + slice) * g.Pp;
  for (int p = tid; p < Warp::P; p += NT) {
    float s;
    if (p < D * H + H) {
      s = smem[p];
#pragma unroll
      for (int r = 1; r < G::SUBS; ++r) s += smem[r * PP + p];
      s *= w1[p % H];   // dL/dz was left without it
    } else if (p < D * H + 2 * H) {
      const int h = p - (D * H + H);
      s = red_w1[0][h];
#pragma unroll
      for (int w = 1; w < NW; ++w) s += red_w1[w][h];
    } else {
      s = red_db1[0];
#pragma unroll
      for (int w = 1; w < NW; ++w) s += red_db1[w];
    }
    po[p] = s;
  }
  if (tid == 0) {
    double s = red_ll[0];
#pragma unroll
    for (int w = 1; w < NW; ++w) s += red_ll[w];
    g.ll_out[(size_t)win * S + slice] = s;
  }
}

// ---- host side -----------------------------------------------------------
template <int H, int MINB>
static cudaError_t fp32_attr() {
  return cudaFuncSetAttribute(grad_fp32_kernel<H, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)Fp32Geom<H>::SMEM);
}
template <int H, int MINB>
static cudaError_t launch_fp32_t(const GradParams& g, int slices, int windows, cudaStream_t st) {
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && !attr_done[dev]) {
    cudaError_t e = fp32_attr<H, MINB>();
    if (e != cudaSuccess) return e;
    attr_done[dev] = true;
  }
  return launch_chain_kernel(grad_fp32_kernel<H, MINB>, dim3(slices, windows), dim3(Fp32Geom<H>::NT),
                             Fp32Geom<H>::SMEM, st, g);
}

int fp32_tile_rows(int H) { (void)H; return FP32_TILE; }

cudaError_t launch_grad_fp32(int H, const GradParams& g, int slices, int windows, cudaStream_t st) {
  if (H == 40) return launch_fp32_t<40, 3>(g, slices, windows, st);
  if (H == 128) return launch_fp32_t<128, 1>(g, slices, windows, st);
  return cudaErrorInvalidValue;
}

template <int H, int MINB>
static int fp32_ctas_per_sm() {
  int n = 0;
  fp32_attr<H, MINB>();
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, grad_fp32_kernel<H, MINB>, Fp32Geom<H>::NT, Fp32Geom<H>::SMEM);
  return n;
}
int fp32_max_ctas_per_sm(int H) { return H == 40 ? fp32_ctas_per_sm<40, 3>() : H == 128 ? fp32_ctas_per_sm<128, 1>() : 0; }

}  // namespace mcmc_b200
