// FP32 fused leapfrog-update + forward + backward kernels.
//
// They stand in for leapfrog_step_kernel of the reference
// (include/mcmc/mcmc_step_ffma.h:154-379): same math, different mapping.  grad_fp32_split_kernel (below) has the forward product of
// 40 units on the tensor core; grad_fp32_kernel does everything by FFMA, for 128 units and for batches of small windows:
//   * grid = (slices, windows): many independent windows per launch, each
//     window's rows split over `slices` CTAs;
//   * every warp works through its own row blocks (fp32_tile.cuh), which arrive through the bulk-copy engine double
//     buffered: nothing in the row loop waits for another warp;
//   * dW0 stays in the lanes' registers for the whole range (the reference keeps it in shared memory and adds to it
//     with atomics, mcmc_step_ffma.h:346-367);
//   * no atomics: the warps' sums -> shared memory -> one partial vector per CTA; the next launch (or the accept
//     kernel) sums the partials of a window in a fixed order, so results are bit-reproducible.
#include "fp32_split.cuh"
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

// LOSS: the rows' log-likelihood is wanted (the last step of a trajectory, evaluations)
template <int H, int MINB, bool LOSS>
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
    lanes.template block<LOSS>(xb, wp, b0, w1, w1[H], g.lik, g.n_rows - r0, dys, es, dw1, db1, loss);
    if (LOSS && lanes.loss_first()) {
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

// ---- 40 units: the forward product on the tensor core (split_mma.cuh, fp32_split.cuh) --------------
// Persistent, one CTA per SM (a kernel with tensor memory gets no more), over the segments of the host's work table as in
// grad_tf32.cu; without a table a CTA has one slice of the one window.  Three compute warpgroups, each with tiles of 128 rows of its own
// (a row per thread where rows are cut into parts, 32 rows per warp everywhere else), and a control warp for each that
// issues its MMAs.  A warpgroup takes z of a tile into registers, puts the next tile's rows in their place in tensor memory and goes
// on: the next tile's MMAs run during the epilogue and the backward pass of this one.  Only there the four warps of a
// warpgroup wait for one another.
// A tile takes 2,640 cycles (FFMA: 3,700) and 1,445 instructions a warp, of them 540 packed FMAs; issue slots are 55 %, the FMA pipe
// 52 % busy, three warps a scheduler.  16 windows of 40013 rows: 73.7 us a step before, 65 (first version), 58.6 (shared memory
// through its own address space, packed tanh, five operations for three parts), 57.8 (backward unrolled 16 times; 2: 68.3, 4:
// 62.0, 8: 59.8), 58.2 with all products of parts (24 MMAs instead of 18); without the losses 0 to 2 % less.  25 windows of 58368
// rows 156 and 118, two 25.5 and 18.8.  Single FMAs in the backward pass: 61.2.
constexpr int FSP_NWG = 3, FSP_THREADS = FSP_NWG * 128 + 128;
// registers: 512 threads start with 128 each (3 * 128 * 160 + 128 * 32 = 65,536)
constexpr int FSP_COMPUTE_REGS = 160, FSP_CTRL_REGS = 32;
struct FspGeom {
  using Warp = SplitWarp;
  static constexpr int NW = FSP_NWG * 4;
  static constexpr int XS = Warp::ROWS * KP;           // floats of a warp's rows
  static constexpr int WARP = 2 * XS + Warp::ES;       // two stages of rows, dL/dz
  static_assert(Warp::ES >= KP * SPLIT_H, "a warp's sums take the place of its dL/dz");
  static constexpr int WB = 0, ROWS0 = WB + SPLIT_B_BYTES / 4, W1 = ROWS0 + NW * WARP;   // float offsets
  static constexpr size_t SMEM = 1024 + (W1 + SPLIT_H + 4) * 4;
  static constexpr int Z_COL0 = FSP_NWG * SPLIT_A_COLS, TMEM_COLS = 512;
  static_assert(Z_COL0 + FSP_NWG * SPLIT_Z_COLS <= TMEM_COLS, "tensor memory budget");
};

template <bool LOSS>
__global__ void __launch_bounds__(FSP_THREADS, 1) grad_fp32_split_kernel(const GradParams g) {
  using G = FspGeom;
  using Warp = SplitWarp;
  constexpr int D = SPLIT_D, H = SPLIT_H, P = Warp::P, NWG = FSP_NWG, NW = G::NW, NCOMPUTE = NWG * 128;
  constexpr uint32_t WARP_BYTES = G::XS * sizeof(float);

  extern __shared__ unsigned char smem_raw[];
  unsigned char* const wb = smem_align1024(smem_raw);
  float* const base = reinterpret_cast<float*>(wb);
  float* const w1 = base + G::W1;       // W1, b1
  __shared__ __align__(8) uint64_t bar_rows[NW][2], bar_fwd[NWG];
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(8) float red_w1[NW][H];
  __shared__ float red_db1[NW];
  __shared__ double red_ll[NW];

  const Warp lanes;
  const int tid = threadIdx.x, lane = lanes.lane;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const bool is_ctrl = warp >= NW;
  const int wg = is_ctrl ? warp - NW : warp >> 2;
  const int seg0 = g.segs ? g.seg_ptr[blockIdx.x] : 0, seg1 = g.segs ? g.seg_ptr[blockIdx.x + 1] : 1;
  auto segment = [&](int sg) {  // window, first tile, end tile, slot
    if (g.segs) return g.segs[sg];
    const int S = gridDim.x, s = blockIdx.x;
    return make_int4(0, (int)((long long)s * g.n_tiles / S), (int)((long long)(s + 1) * g.n_tiles / S), s);
  };
  // tiles t0 + wg, t0 + wg + NWG, ... of a segment are this warpgroup's
  auto tiles = [&](const int4& seg) { return wg < NWG ? (seg.z - seg.y - wg + NWG - 1) / NWG : 0; };
  float* const xs = base + G::ROWS0 + warp * G::WARP;
  uint32_t n_done = 0;  // tiles of this warpgroup in earlier segments; tile n of all uses row stage n % 2
  auto fetch = [&](const int4& seg, int i) {  // rows of this warp in tile i of a segment
    const uint32_t st = (n_done + i) & 1;
    const float* src = g.xaug + (long long)(g.data_window0 + seg.x) * g.window_stride +
                       ((size_t)(seg.y + wg + i * NWG) * FP32_TILE + (warp & 3) * Warp::ROWS) * KP;
    mbar_expect_tx(&bar_rows[warp][st], WARP_BYTES);
    bulk_g2s(xs + st * G::XS, src, WARP_BYTES, &bar_rows[warp][st]);
  };
  auto fetch_first = [&](const int4& seg) {
    if (!is_ctrl && lane == 0) {
      const int n = tiles(seg);
      for (int i = 0; i < 2 && i < n; ++i) fetch(seg, i);
    }
  };

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"((uint32_t)G::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (!is_ctrl && lane == 0) {
    mbar_init(&bar_rows[warp][0], 1);
    mbar_init(&bar_rows[warp][1], 1);
    if ((warp & 3) == 0) mbar_init(&bar_fwd[wg], 1);
    mbar_fence_init();
  }
  __syncwarp();
  // The first rows may be fetched ahead of the dependency wait only when no kernel directly before
  // this one in the stream wrote the dataset (inside a chain none does; right after a repack one did).
  const bool early_rows = g.data_fresh == 0;
  if (early_rows && seg0 < seg1) fetch_first(segment(seg0));
  // what the MMAs read besides weights: feature 23, and the lines behind the last part
  for (int i = tid; i < SPLIT_B_BYTES / 16; i += FSP_THREADS)
    reinterpret_cast<float4*>(wb)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_trigger();
  pdl_wait();
  if (!early_rows && seg0 < seg1) fetch_first(segment(seg0));

  // Every segment has three CTA-wide barriers, executed by both roles:
  //   S1 parameters staged   S2 all tiles of the segment done   S3 read-out done
  if (is_ctrl) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FSP_CTRL_REGS));
    const uint32_t on = elect_one(), tm = __shfl_sync(0xffffffffu, tmem, 0);
    for (int sg = seg0; sg < seg1; ++sg) {
      const int n = tiles(segment(sg));
      __syncthreads_or(0);  // S1
      for (int i = 0; i < n; ++i) {
        named_sync(BAR_ROWS0 + wg, 160);
        tc_fence_after();
        split_issue(tm + G::Z_COL0 + wg * SPLIT_Z_COLS, tm + wg * SPLIT_A_COLS, smem_u32(wb), on);
        tc_commit_if(&bar_fwd[wg], on);
      }
      __syncthreads();  // S2
      __syncthreads();  // S3
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FSP_COMPUTE_REGS));
    bool ok = true;
    const uint32_t sub = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t a_t = tmem + wg * SPLIT_A_COLS + sub, z_t = tmem + G::Z_COL0 + wg * SPLIT_Z_COLS + sub;
    float* const es = xs + 2 * G::XS;
    const int own = lanes.own();
    for (int sg = seg0; sg < seg1; ++sg) {
      const int4 seg = segment(sg);
      const int win = seg.x, my_nt = tiles(seg);
      bool wide = false;
      {
        // fused leapfrog update; parameters land where the MMAs read them.  (Loading the next segment's during this one's
        // read-out took registers from the tile loop: 16 windows of 40013 rows 58.6 us a step, 59.8 with it)
        constexpr int N = (P + NCOMPUTE - 1) / NCOMPUTE;
        float w[N];
        leapfrog_params(g, win, tid, NCOMPUTE, P, seg.w == 0, w);
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int p = tid + i * NCOMPUTE;
          if (p < D * H + H) {
            const int k = p / H, n = p - k * H;
            wide |= split_store_weight(smem_u32(wb) + split_b_off(n, k & ~3) + (k & 3) * 4, w[i]);
          } else if (p < P) {
            w1[p - (D * H + H)] = w[i];
          }
        }
        fence_proxy_async_smem();
      }
      const bool plain_w = __syncthreads_or(wide) != 0;  // S1

      // a tile's rows, once they have landed, to tensor memory; whether one of the warp's takes the plain path
      auto stage_rows = [&](int i) {
        const uint32_t n = n_done + i;
        mbar_wait_q(&bar_rows[warp][n & 1], (n >> 1) & 1, g.status, 101, ok);
        const float* x = xs + (n & 1) * G::XS + lane * KP;
        float far = 0.f;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float4 lo = *reinterpret_cast<const float4*>(x + 8 * j), hi = *reinterpret_cast<const float4*>(x + 8 * j + 4);
          const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, j == 2 ? 0.f : hi.w};
#pragma unroll
          for (int k = 0; k < 8; k += 2) far = split_max(far, v[k], v[k + 1]);
          split_store_row(a_t, j, v);
        }
        tc_wait_st();
        tc_fence_before();
        named_arrive(BAR_ROWS0 + wg, 160);
        return __any_sync(0xffffffffu, split_wide(far)) != 0;
      };
      uint64_t acc[Warp::KPT / 2][Warp::UPT] = {};
      uint64_t dw1[5] = {};
      float db1 = 0.f;
      double llacc = 0.0;
      bool plain = my_nt > 0 ? stage_rows(0) : false;

#pragma unroll 1
      for (int i = 0; i < my_nt; ++i) {
        const uint32_t n = n_done + i;
        const float* xb = xs + (n & 1) * G::XS;
        mbar_wait_q(&bar_fwd[wg], n & 1, g.status, 102, ok);
        tc_fence_after();
        uint64_t h[4][5];
        lanes.load(z_t, h);
        tc_fence_before();
        if (plain || plain_w) {
          Warp::plain<1>(xb, wb, es);
          lanes.load_plain(es, h);
        }
        if (i + 1 < my_nt) plain = stage_rows(i + 1);
        const int row = (seg.y + wg + i * NWG) * FP32_TILE + (warp & 3) * Warp::ROWS + own;
        const bool valid = row < g.n_rows;
        const float y = xb[own * KP + COL_Y];
        float dy, pred;
        lanes.block(h, w1, g.lik, y, valid, es, dw1, dy, pred, [](int) {});
        if (LOSS) {
          const float loss = valid ? lik_loss(g.lik, y, pred) : 0.f;
          llacc += (double)loss;
          store_row_loss(g.row_loss, (long long)win * g.row_loss_stride + row, loss, valid);
        }
        db1 += dy;
        lanes.backward<16>(xb, es, acc);
        __syncwarp();  // rows and dL/dz have been read: the next copy and the next tile may overwrite them
        if (lane == 0 && i + 2 < my_nt) fetch(seg, i + 2);
      }
      n_done += my_nt;
      if (sg + 1 < seg1) fetch_first(segment(sg + 1));

      // ---- lanes -> warp ----
      lanes.store_dw1(dw1, red_w1[warp]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        db1 += __shfl_xor_sync(0xffffffffu, db1, o);
        llacc += __shfl_xor_sync(0xffffffffu, llacc, o);
      }
      if (lane == 0) {
        red_db1[warp] = db1;
        red_ll[warp] = llacc;
      }
      lanes.store_dw0(acc, es + (lanes.kh * Warp::KPT + lanes.rsub * 6) * H);
      __syncthreads();  // S2
      // ---- warps -> one partial vector for (window, slot) ----
      const size_t slot = (size_t)win * g.slices_out + seg.w;
      float* po = g.partial_out + slot * g.Pp;
      for (int p = tid; p < P; p += NCOMPUTE) {
        float s;
        if (p < D * H + H) {
          const float* r = base + G::ROWS0 + 2 * G::XS + p;
          s = r[0];
#pragma unroll
          for (int w = 1; w < NW; ++w) s += r[w * G::WARP];
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
        g.ll_out[slot] = s;
      }
      __syncthreads();  // S3: the next segment's parameters may take the place of this one's
    }
    if (g.test_code == 102) mbar_wait_q(&bar_fwd[wg], n_done & 1, g.status, 102, ok);  // (nothing ends this phase)
    if (!ok) {  // copies and MMAs that did not arrive in time
      for (uint32_t i = 1; i <= 2 && i <= n_done; ++i) {
        const uint32_t n = n_done - i;
        mbar_drain(&bar_rows[warp][n & 1], (n >> 1) & 1);
        if (i == 1) mbar_drain(&bar_fwd[wg], n & 1);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)G::TMEM_COLS)
                 : "memory");
}

// ---- host side -----------------------------------------------------------
template <int H, int MINB, bool LOSS>
static cudaError_t fp32_attr() {
  return cudaFuncSetAttribute(grad_fp32_kernel<H, MINB, LOSS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)Fp32Geom<H>::SMEM);
}
template <int H, int MINB, bool LOSS>
static cudaError_t launch_fp32_t(const GradParams& g, int slices, int windows, cudaStream_t st) {
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && !attr_done[dev]) {
    cudaError_t e = fp32_attr<H, MINB, LOSS>();
    if (e != cudaSuccess) return e;
    attr_done[dev] = true;
  }
  return launch_chain_kernel(grad_fp32_kernel<H, MINB, LOSS>, dim3(slices, windows), dim3(Fp32Geom<H>::NT),
                             Fp32Geom<H>::SMEM, st, g);
}

int fp32_tile_rows(int H) { (void)H; return FP32_TILE; }

cudaError_t launch_grad_fp32(int H, const GradParams& g, int slices, int windows, cudaStream_t st) {
  if (H == 40) return g.no_loss ? launch_fp32_t<40, 3, false>(g, slices, windows, st) : launch_fp32_t<40, 3, true>(g, slices, windows, st);
  // (128 units with the losses always: without them 8 windows of 40013 rows took 108 us a step instead of 106.5)
  if (H == 128) return launch_fp32_t<128, 1, true>(g, slices, windows, st);
  return cudaErrorInvalidValue;
}

template <bool LOSS>
static cudaError_t launch_split_t(const GradParams& g, int ctas, cudaStream_t st) {
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !attr_done[dev]) {
    cudaError_t e =
        cudaFuncSetAttribute(grad_fp32_split_kernel<LOSS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FspGeom::SMEM);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_done[dev] = true;
  }
  return launch_chain_kernel(grad_fp32_split_kernel<LOSS>, dim3(ctas), dim3(FSP_THREADS), FspGeom::SMEM, st, g);
}
cudaError_t launch_grad_fp32_split(const GradParams& g, int ctas, cudaStream_t st) {
  return g.no_loss ? launch_split_t<false>(g, ctas, st) : launch_split_t<true>(g, ctas, st);
}

template <int H, int MINB>
static int fp32_ctas_per_sm() {
  int n = 0;
  fp32_attr<H, MINB, true>();
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, grad_fp32_kernel<H, MINB, true>, Fp32Geom<H>::NT, Fp32Geom<H>::SMEM);
  return n;
}
int fp32_max_ctas_per_sm(int H) { return H == 40 ? fp32_ctas_per_sm<40, 3>() : H == 128 ? fp32_ctas_per_sm<128, 1>() : 0; }

}  // namespace mcmc_b200
