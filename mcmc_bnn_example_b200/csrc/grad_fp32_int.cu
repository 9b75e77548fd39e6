// FP32 gradients of 40 units, rows streamed: forward product and sums over rows both on the tensor core (split_mma.cuh, int_mma.cuh,
// fp32_split.cuh).  grad_fp32.cu has the kernel whose backward pass goes by FFMA, which stays for segments of few tiles (plan_ints in
// api.cu draws the line).
//
// Persistent, one CTA per SM (a kernel with tensor memory gets no more), over the segments of the host's work table as in
// grad_tf32.cu.  Four compute warpgroups take tiles of 128 rows in turn (a row per thread where rows are cut into parts and made
// integers, 32 rows per warp everywhere else); one control warp issues the product's MMAs, another those of the sums.  Tensor memory: the
// sums, 160 columns for the whole CTA (integers: their order is of no consequence), and two places for a tile's rows and accumulators,
// which the tiles take in turn: z is in a warpgroup's registers soon after it is there.
// The integers are those of x dL/dpred, feature by feature, and of 1 - h^2, which needs no range: its step is 2^-30, where h alone leaves an error of 2^-24.
// A feature's range is 2^12 over the mean exponent of its x dL/dpred, 2^7 over the largest at most, in the first tiles' rows; those are 32 of every
// sixteenth of the segment (row_at), 16 of which are looked at.  So a feature's error is measured against its own terms: its step is 2^-19 of
// a mean that they have in those rows, and smaller terms elsewhere cost no more than in a chain of FFMAs that has begun with them.  (x and
// dL/dpred as two integers, the latter with one range for all: a feature that is only there where dL/dpred is a hundredth of what it was in
// the segment's first tile was 8e-6 off, 1e-4 with a thousandth; FFMA 5e-7, here 1.4e-7 and 2e-7.)  A warp whose 32 rows have a product beyond its range
// adds them up by FFMA on the spot, from the products and the integers of 1 - h^2 (unit_far: 1.3 us; left for the segment's end, with their forward
// product once more, they took 9 us, side by side on 16 warps); rows of infinities, NaN and values from 2^60 on, whose z the tensor core does not
// know, are left for the segment's end.  A feature that is zero in all the rows looked at has no range; should it be there later, the warp sees whether it
// is what 1 would be (unit_again).
// Gradients' error against 64 bits, here / by FFMA, segments of 24, 64, 118 and 938 tiles: N(0,1) features 0.81, 0.59, 0.65, 0.58, the worst feature of 23
// 0.93, 0.88, 0.96, 0.93; 16 other distributions and orders of rows 0.71 and 0.80 in the mean, none above 1.01 and 1.07 but for a late indicator's 1.27 over
// 24 tiles (FFMA adds up to 1,600 rows in a chain; the room takes most of what bits are to spare for short ones; 2^13: 1.14 over 24 tiles).
// A tile takes 2,140 cycles of an SM (FFMA 2,640) and 1,320 instructions a warp, issue slots 62 % busy, MUFU 30 %, tensor pipe 42 %.  What an
// instruction less gave was little; what a spill less gave was much, for shared memory leaves 28 KB of L1: hence functions of few registers for all that is
// rare (FFMA's code in line: 57 us a step for 16 windows of 40013 rows; the first tiles' statistics in line, with 28 bytes spilled: 50.3).
// The next tile's rows go to tensor memory before this one's products are made integers: its forward product goes on beside them (the same windows:
// 52.7 us without).
// us a step, FFMA and here: 16 x 40013 rows 57.9, 46.8; 25 x 58368 118, 96; 100 x 10000 87.1, 72.5; 6 x 58368 35.7, 31.1; 200 x 4000 75.4, 67.0; with 17 features of
// zeros (16 x 40013 and 6 x 58368) 57.9, 51.1 and 35.7, 33.2; an indicator that begins late 58.0, 46.7 and 35.7, 33.0; one in a thousand rows 57.9, 56.6 and 35.7, 37.7; 22
// lognormal features (sigma 1.5) 57.9, 51.8 and 35.7, 36.0; Cauchy ones 57.9, 88 and 35.7, 57.5; 0.2 % targets with outliers of 300 sigma 58.0, 66.4 and 35.7, 41.9.
#include "fp32_split.cuh"

namespace mcmc_b200 {

constexpr int FIN_TILE = 128;

constexpr int FIN_NWG = 4, FIN_THREADS = FIN_NWG * 128 + 128;
// registers: 640 threads start with 96 each (4 * 128 * 112 + 128 * 32 = 61,440)
constexpr int FIN_COMPUTE_REGS = 112, FIN_CTRL_REGS = 32;
constexpr int FIN_SUB = 1000;                      // tiles of a segment between two read-outs: 128,000 rows' products of bytes fit 31 bits
constexpr int FIN_ROOM = 12, FIN_ROOM_MAX = 7;      // above the mean exponent of a feature x dL/dpred, above their largest
constexpr float FIN_ONE = 1073741824.f;            // 1 - h^2 = 1 as an integer
// a feature that is zero in all rows that ranges come from: as if it were 1, and its largest value among 32 rows has 22 bits at least
constexpr int FIN_ROOM_NEW = 5;
constexpr float FIN_LOW_NEW = 4194304.f;
constexpr int FIN_MOST = 97;                       // ranges up to 2^97 and from 2^-77 on: sums and their factors are floats
struct FinGeom {
  using Warp = SplitWarp;
  static constexpr int NW = FIN_NWG * 4;
  static constexpr int XS = Warp::ROWS * KP;           // floats of a warp's rows, and words of their integers
  static constexpr int WARP = 2 * XS + Warp::ES;       // two stages of rows, dL/dz
  static_assert(XS * 4 == INT_X_WARP && Warp::ES * 4 == INT_E_WARP && Warp::ES >= KP * SPLIT_H, "shared places");
  static constexpr int WB = 0, ROWS0 = WB + SPLIT_B_BYTES / 4, S = ROWS0 + NW * WARP, W1 = S + INT_S_FLOATS, SCALE = W1 + SPLIT_H + 4, UNIT = SCALE + KP, NEW = UNIT + KP;
  static constexpr size_t SMEM = 1024 + (NEW + KP) * 4;
  static_assert(S % 4 == 0 && W1 % 4 == 0 && SCALE % 4 == 0 && KP % 4 == 0, "vector alignment");
  static constexpr int PLACE = SPLIT_A_COLS + SPLIT_Z_COLS, PLACE0 = INT_ACC_COLS, TMEM_COLS = 512;
  static_assert(PLACE0 + 2 * PLACE <= TMEM_COLS, "tensor memory budget");
};

// A warp's first 32 rows (floats at xb), times `dy` (of row `lane`) in their place; their features' statistics, a lane a feature, if z was `known`
static __device__ __noinline__ void unit_statistics(float* xb, float dy, bool known, uint32_t* x_stat, uint32_t* x_max) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int ch = 0; ch < KP / 4; ++ch) {
    float4* const x = reinterpret_cast<float4*>(xb + lane * KP + 4 * ch);
    *x = make_float4(x->x * dy, x->y * dy, x->z * dy, ch == KP / 4 - 1 ? 0.f : x->w * dy);
  }
  __syncwarp();
  if (lane <= SPLIT_D && known) {
    uint32_t st = 0u, mx = 0u;
#pragma unroll 16
    for (int r = 0; r < SplitWarp::ROWS; r += 2) {
      const float p = xb[r * KP + lane];
      st += int_stat(p);
      mx = max(mx, __float_as_uint(p) & 0x7fffffffu);
    }
    atomicAdd(&x_stat[lane], st);
    atomicMax(&x_max[lane], mx);
  }
  __syncwarp();
}
// ... of all warps: the ranges (every warp writes the same): three arrays of KP, scale, unit and new (FinGeom)
static __device__ __noinline__ void unit_ranges(const volatile uint32_t* st, const volatile uint32_t* mx, float* scale) {
  constexpr int D = SPLIT_D;
  const int lane = threadIdx.x & 31;
  if (lane < KP) {
    const bool is_new = lane < D && st[lane] == 0u;
    const int e = is_new ? int_scale_exp(st[D], FIN_ROOM_NEW) : min(int_scale_exp(st[lane], FIN_ROOM), int_max_exp(mx[lane]) + FIN_ROOM_MAX);
    const float u = int_scale(int_range_exp<FIN_MOST>(e));
    scale[lane] = lane > D || is_new ? 0.f : u;
    scale[KP + lane] = lane > D ? 0.f : u;
    scale[2 * KP + lane] = is_new ? int_scale(INT_NONE) : 0.f;
  }
  __syncwarp();
}

// A warp's 32 rows of which a product is beyond the range: floats at xb, times `dy` (of row `lane`).  Where all that is wrong is a feature whose range was not
// known (scale and unit differ), they become integers all the same, if it is as large as they were taken to be or zero.  Returns whether.
static __device__ __noinline__ bool unit_again(float* xb, float dy, const float* scale, const float* unit) {
  const int lane = threadIdx.x & 31;
  float v[KP];
#pragma unroll
  for (int ch = 0; ch < KP / 4; ++ch) {
    float4 x = *reinterpret_cast<const float4*>(xb + lane * KP + 4 * ch);
    if (ch == KP / 4 - 1) x.w = 0.f;
    v[4 * ch] = x.x * dy;
    v[4 * ch + 1] = x.y * dy;
    v[4 * ch + 2] = x.z * dy;
    v[4 * ch + 3] = x.w * dy;
  }
  __syncwarp();
#pragma unroll
  for (int ch = 0; ch < KP / 4; ++ch)
    *reinterpret_cast<float4*>(xb + lane * KP + 4 * ch) = make_float4(v[4 * ch], v[4 * ch + 1], v[4 * ch + 2], v[4 * ch + 3]);
  __syncwarp();
  bool in = true;
  if (lane < KP) {
    float top = 0.f;
#pragma unroll 8
    for (int r = 0; r < SplitWarp::ROWS; r += 2) top = split_max(top, xb[r * KP + lane], xb[(r + 1) * KP + lane]);
    const float t = top * unit[lane];
    in = t < INT_TOP && (scale[lane] == unit[lane] || top == 0.f || t >= FIN_LOW_NEW);
  }
  if (!__all_sync(0xffffffffu, in)) return false;
#pragma unroll
  for (int ch = 0; ch < KP / 4; ++ch)
    int_store_x4(smem_u32(xb) + int_x_off(lane, ch), make_float4(v[4 * ch], v[4 * ch + 1], v[4 * ch + 2], v[4 * ch + 3]),
                 reinterpret_cast<const float4*>(unit)[ch]);
  return true;
}

// The sums of such rows by FFMA, added to acc: their products with dL/dpred are floats at xb (unit_again), 1 - h^2 integers at es, which become floats.  Where
// a product is no float, the rows are read once more, and dL/dpred (`dy` of row `lane`) goes to 1 - h^2, which may well be zero
static __device__ __noinline__ void unit_far(float* xb, float* es, uint64_t* acc, const float* rows, float dy) {
  const SplitWarp lanes;
  float top = 0.f;
#pragma unroll
  for (int ch = 0; ch < KP / 4; ++ch) {
    const float4 p = *reinterpret_cast<const float4*>(xb + lanes.lane * KP + 4 * ch);
    top = split_max(split_max(top, p.x, p.y), p.z, p.w);
  }
  const bool floats = __all_sync(0xffffffffu, top < __int_as_float(0x7f800000)) != 0;
  if (!floats)
    for (int i = lanes.lane; i < SplitWarp::ROWS * KP / 4; i += 32)
      reinterpret_cast<float4*>(xb)[i] = reinterpret_cast<const float4*>(rows)[i];
  const uint32_t* const src = reinterpret_cast<const uint32_t*>(es) + (lanes.c >> 1) * 32 + lanes.q * 4 + (lanes.c & 1) * 2;  // (store_ei)
  uint2 e[4][5];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int n = 0; n < 5; ++n) e[i][n] = *reinterpret_cast<const uint2*>(src + i * (2 * INT_E_ROW) + n * 64);
  __syncwarp();
  auto value = [](uint32_t w) { return (float)(int)((w ^ 0x808080u) - 0x808080u) * (1.f / FIN_ONE); };  // (int_digits2)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float f = __shfl_sync(0xffffffffu, floats ? 1.f : dy, lanes.q + 8 * i);
#pragma unroll
    for (int n = 0; n < 5; ++n)
      *reinterpret_cast<float2*>(es + (lanes.q + 8 * i) * SPLIT_H + 2 * lanes.c + 8 * n) = make_float2(f * value(e[i][n].x), f * value(e[i][n].y));
  }
  __syncwarp();
  SplitWarp::backward_lean<2>(xb, es, acc);
}

template <bool LOSS>
__global__ void __launch_bounds__(FIN_THREADS, 1) grad_fp32_int_kernel(const GradParams g) {
  using G = FinGeom;
  using Warp = SplitWarp;
  constexpr int D = SPLIT_D, H = SPLIT_H, P = Warp::P, NWG = FIN_NWG, NW = G::NW, NCOMPUTE = NWG * 128;
  constexpr uint32_t WARP_BYTES = G::XS * sizeof(float);

  extern __shared__ unsigned char smem_raw[];
  unsigned char* const wb = smem_align1024(smem_raw);
  float* const base = reinterpret_cast<float*>(wb);
  float* const w1 = base + G::W1;       // W1, b1
  float* const x_scale = base + G::SCALE;
  // Features that are zero in the segment's first rows have no scale, and their values, should there be any, another unit; 2^126 in
  // x_new, in which others have 0
  float* const x_unit = base + G::UNIT;
  float* const x_new = base + G::NEW;
  // rows of a warp landed; per place, product done and read; per warpgroup, rows in tensor memory, integers written, sums done; the scale is known.
  // (No named barriers between the roles: they have no limit, and a warp that goes on behind a wait that ran out would arrive at one for its next
  // tile before the control warp has come for this one; their counts lose step then, and somebody waits for good.  All waits here end.)
  __shared__ __align__(8) uint64_t bar_rows[NW][2], bar_fwd[2], bar_read[2], bar_in[NWG], bar_e[NWG], bar_sum[NWG], bar_scale;
  __shared__ uint32_t tmem_slot, x_stat[KP], x_max[KP], none;
  __shared__ int late;                          // code of a wait that ran out
  __shared__ uint32_t far[NW];                  // the warp's rows of its tile are not among the integers
  constexpr int FAR_WORDS = (FIN_SUB / NWG + 31) / 32;
  __shared__ uint32_t far_tiles[NW][FAR_WORDS], far_any[NW];   // ... earlier: which tiles of the part
  __shared__ __align__(8) float red_w1[NW][H];
  __shared__ float red_db1[NW];
  __shared__ double red_ll[NW];

  const Warp lanes;
  const int tid = threadIdx.x, lane = lanes.lane;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const bool is_ctrl = warp >= NW;
  const int wg = warp >> 2;
  const int seg0 = g.segs ? g.seg_ptr[blockIdx.x] : 0, seg1 = g.segs ? g.seg_ptr[blockIdx.x + 1] : 1;
  auto segment = [&](int sg) {  // window, first tile, end tile, slot
    if (g.segs) return g.segs[sg];
    const int S = gridDim.x, s = blockIdx.x;
    return make_int4(0, (int)((long long)s * g.n_tiles / S), (int)((long long)(s + 1) * g.n_tiles / S), s);
  };
  // Tiles are numbered through a CTA's segments: tile n is warpgroup n % 4's, takes place n % 2 and the warp's stage n / 4 % 2.  Which rows
  // those are: a warp's tiles are a stretch of the segment, one after the other, so that the first tiles' rows, from which ranges
  // come, are of all its parts
  float* const xs = base + G::ROWS0 + warp * G::WARP;
  float* const es = xs + 2 * G::XS;
  auto row_at = [&](const int4& seg, int i) {  // the first row of this warp in tile i of a segment
    const int len = (seg.z - seg.y) >> 2, more = (seg.z - seg.y) & 3, j = i & 3;
    return seg.y * FIN_TILE + (4 * (j * len + min(j, more)) + (warp & 3) * (len + (j < more ? 1 : 0)) + (i >> 2)) * Warp::ROWS;
  };
  auto rows_at = [&](const int4& seg, int i) {
    return g.xaug + (long long)(g.data_window0 + seg.x) * g.window_stride + (size_t)row_at(seg, i) * KP;
  };
  auto fetch = [&](int n, int sg, int n0) {  // tile n, in segment sg, whose first one is n0, or a later one
    int4 seg = segment(sg);
    while (n - n0 >= seg.z - seg.y) {
      n0 += seg.z - seg.y;
      if (++sg == seg1) return;
      seg = segment(sg);
    }
    uint64_t* const bar = &bar_rows[warp][n >> 2 & 1];
    mbar_expect_tx(bar, WARP_BYTES);
    bulk_g2s(xs + (n >> 2 & 1) * G::XS, rows_at(seg, n - n0), WARP_BYTES, bar);
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
    if ((warp & 3) == 0) {
      mbar_init(&bar_in[wg], 4);
      mbar_init(&bar_e[wg], 4);
      mbar_init(&bar_sum[wg], 1);
    }
    if (warp < 2) {
      mbar_init(&bar_fwd[warp], 1);
      mbar_init(&bar_read[warp], 4);
    }
    if (warp == 0) mbar_init(&bar_scale, NW);
    mbar_fence_init();
  }
  __syncwarp();
  // The first rows may be fetched ahead of the dependency wait only when no kernel directly before
  // this one in the stream wrote the dataset (inside a chain none does; right after a repack one did).
  const bool early_rows = g.data_fresh == 0, fetches = !is_ctrl && lane == 0 && seg0 < seg1;
  if (early_rows && fetches) fetch(wg, seg0, 0);
  // what the MMAs read besides weights: feature 23, and the lines behind the last part
  for (int i = tid; i < SPLIT_B_BYTES / 16; i += FIN_THREADS)
    reinterpret_cast<float4*>(wb)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (tid < KP) x_stat[tid] = x_max[tid] = 0u;
  if (tid < NW * FAR_WORDS) far_tiles[tid / FAR_WORDS][tid % FAR_WORDS] = 0u;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_trigger();
  pdl_wait();
  if (!early_rows && fetches) fetch(wg, seg0, 0);

  bool ok = true;
  auto wait = [&](uint64_t* bar, uint32_t parity, int c) {  // (in line: a call would cost the tile loop registers)
    if (mbar_try_wait(bar, parity)) return;
    for (uint32_t i = 0; ok && !mbar_try_wait_hint(bar, parity, 20000u); ++i)
      if (i >= MBAR_WAIT_SLICES) {
        ok = false;
        late = c;
      }
  };
  // ... of the control warps: tries without a time to sleep (with one, as above, they woke up late behind a segment's start: 200 windows of 4000 rows 71.1
  // us a step, 66.8 so), for 1.3 s at 1.965 GHz
  auto wait_c = [&](uint64_t* bar, uint32_t parity, int c) {
    if (mbar_try_wait(bar, parity)) return;
    const uint32_t t0 = (uint32_t)(clock64() >> 16);
    while (ok && !mbar_try_wait(bar, parity))
      if ((uint32_t)(clock64() >> 16) - t0 > 40000u) {
        ok = false;
        late = c;
      }
  };
  auto hand_over = [&](uint64_t* bar) {  // to a control warp
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };
  auto place = [&](int n) { return G::PLACE0 + (n & 1) * G::PLACE; };

  // Every segment begins with a CTA-wide barrier and has three for each of its parts (of FIN_SUB tiles), executed by both roles:
  //   S1 parameters staged   S2 all tiles of the part done   S3 sums read out   S4 and stored
  int n0 = 0;  // number of the segment's first tile
  if (is_ctrl) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FIN_CTRL_REGS));
    const uint32_t on = elect_one(), tm = __shfl_sync(0xffffffffu, tmem, 0);
    for (int sg = seg0; sg < seg1; ++sg) {
      const int4 seg = segment(sg);
      const int end = n0 + seg.z - seg.y;
      __syncthreads_or(0);  // S1
      int p0 = n0, n = n0, rows = n0;  // tiles whose product has been issued, whose rows have come
      do {
        const int p1 = min(p0 + FIN_SUB, end);
        if (warp == NW) {
          // A warpgroup brings the next part's first tile before this part's end, the third and fourth behind the products of the first two
          for (; n < min(p1 + 2, end); ++n) {
            if (n == rows) {
              wait_c(&bar_in[n & 3], n >> 2 & 1, 106);
              ++rows;
            }
            if (n >= 2) wait_c(&bar_read[n & 1], (n - 2) >> 1 & 1, 103);
            if (g.test_code == 103 && n == n0 + 2) wait_c(&bar_read[n & 1], n >> 1 & 1, 103);  // (nothing ends this phase before what follows)
            tc_fence_after();
            split_issue(tm + place(n) + SPLIT_A_COLS, tm + place(n), smem_u32(wb), on);
            tc_commit_if(&bar_fwd[n & 1], on);
          }
          for (; rows < min(p1 + NWG, end); ++rows) wait_c(&bar_in[rows & 3], rows >> 2 & 1, 106);
        } else if (warp == NW + 1) {
          uint32_t more = 0u;
          for (int n = p0; n < p1; ++n) {
            wait_c(&bar_e[n & 3], n >> 2 & 1, 107);
            tc_fence_after();
            const uint32_t skip = __ballot_sync(0xffffffffu, lane < 4 && reinterpret_cast<volatile uint32_t*>(far)[(n & 3) * 4 + (lane & 3)] != 0u);
            const uint32_t w0 = smem_u32(base + G::ROWS0 + (n & 3) * 4 * G::WARP);
            const uint64_t xd = int_x_desc(w0 + (n >> 2 & 1) * WARP_BYTES), ed = int_e_desc(w0 + 2 * WARP_BYTES);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (!(skip >> i & 1)) {
                int_mma_if(tm, umma_desc_advance(xd, i * (G::WARP * 4 >> 4)), umma_desc_advance(ed, i * (G::WARP * 4 >> 4)), more, on);
                more = 1u;
              }
            if (g.test_code == 104 && n == n0 + 1) wait_c(&bar_sum[n & 3], n >> 2 & 1, 104);  // (as above)
            tc_commit_if(&bar_sum[n & 3], on);
          }
          if (p1 > p0) wait_c(&bar_sum[(p1 - 1) & 3], (p1 - 1) >> 2 & 1, 104);
          if (lane == 0) none = more ^ 1u;
        }
        __syncthreads();  // S2
        __syncthreads();  // S3
        __syncthreads();  // S4
        p0 += FIN_SUB;
      } while (p0 < end);
      n0 = end;
    }
    if (!ok) {
      atomicExch(g.status, late);
      if (warp == NW + 1)  // (in line: no room for a call in so few registers)
        for (uint32_t i = 0; i < MBAR_WAIT_SLICES && !mbar_try_wait_hint(&bar_sum[(n0 - 1) & 3], (n0 - 1) >> 2 & 1, 20000u); ++i) {}
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FIN_COMPUTE_REGS));
    const uint32_t sub = (uint32_t)((warp & 3) * 32) << 16;
    const int own = lanes.own();
    for (int sg = seg0; sg < seg1; ++sg) {
      const int4 seg = segment(sg);
      const int win = seg.x, end = n0 + seg.z - seg.y;
      const int first = n0 + ((wg - n0) & 3);  // this warpgroup's first tile
      const int row0 = row_at(seg, first - n0) + own;
      bool wide = false;
      {
        // fused leapfrog update; parameters land where the MMAs read them
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

      bool plain = false, some_new = false;   // of the tile that comes next: rows for plain FFMA; of the segment: features without a scale
      float y = 0.f;
      // a tile's rows to tensor memory, once they have landed
      auto stage_rows = [&](int n) {
        float* const xb = xs + (n >> 2 & 1) * G::XS;
        wait(&bar_rows[warp][n >> 2 & 1], n >> 3 & 1, 101);
        if (n >= 2) wait(&bar_fwd[n & 1], (n - 2) >> 1 & 1, 102);
        tc_fence_after();
        y = xb[own * KP + COL_Y];
        float v[KP];
#pragma unroll
        for (int ch = 0; ch < KP / 4; ++ch) {
          const float4 v4 = *reinterpret_cast<const float4*>(xb + lane * KP + 4 * ch);
          v[4 * ch] = v4.x;
          v[4 * ch + 1] = v4.y;
          v[4 * ch + 2] = v4.z;
          v[4 * ch + 3] = ch == KP / 4 - 1 ? 0.f : v4.w;
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float p[8] = {v[8 * j], v[8 * j + 1], v[8 * j + 2], v[8 * j + 3], v[8 * j + 4], v[8 * j + 5], v[8 * j + 6], v[8 * j + 7]};
          split_store_row(tmem + place(n) + sub, j, p);
        }
        tc_wait_st();
        tc_fence_before();
        hand_over(&bar_in[wg]);
        float top = 0.f;
#pragma unroll
        for (int k = 0; k < KP; k += 2) top = split_max(top, v[k], v[k + 1]);
        plain = __any_sync(0xffffffffu, split_wide(top)) != 0;
      };
      // Integers of the tile's rows times dL/dpred (of row `lane`) in the rows' place; false: one is beyond its range
      auto products = [&](float* xb, float dy) __attribute__((always_inline)) {
        uint64_t t[KP / 2];
        const uint64_t dy2 = pack2(dy, dy);
#pragma unroll
        for (int ch = 0; ch < KP / 4; ++ch) {
          const float4 v = *reinterpret_cast<const float4*>(xb + lane * KP + 4 * ch);
          t[2 * ch] = mul2(pack2(v.x, v.y), dy2);
          t[2 * ch + 1] = mul2(pack2(v.z, ch == KP / 4 - 1 ? 0.f : v.w), dy2);
        }
        __syncwarp();  // every lane has read its row
        float top = 0.f;
#pragma unroll
        for (int ch = 0; ch < KP / 4; ++ch) {
          const float4 s = *reinterpret_cast<const float4*>(x_scale + 4 * ch);
          float t0, t1;
          t[2 * ch] = mul2(t[2 * ch], pack2(s.x, s.y));
          unpack2(t[2 * ch], t0, t1);
          top = split_max(top, t0, t1);
          t[2 * ch + 1] = mul2(t[2 * ch + 1], pack2(s.z, s.w));
          unpack2(t[2 * ch + 1], t0, t1);
          top = split_max(top, t0, t1);
        }
        if (some_new) {
          float x = 0.f;
#pragma unroll
          for (int ch = 0; ch < KP / 4; ++ch) {
            const float4 v = *reinterpret_cast<const float4*>(xb + lane * KP + 4 * ch), f = *reinterpret_cast<const float4*>(x_new + 4 * ch);
            x = split_max(x, v.x * f.x, v.y * f.y);
            x = split_max(x, v.z * f.z, v.w * f.w);
          }
          if (!(x < 1.f)) top = INT_TOP;
          __syncwarp();
        }
        if (__builtin_expect(!__all_sync(0xffffffffu, top < INT_TOP), 0)) return unit_again(xb, dy, x_scale, x_unit);
#pragma unroll
        for (int ch = 0; ch < KP / 4; ++ch) {
          const uint2 a = int_digits2(t[2 * ch]), b = int_digits2(t[2 * ch + 1]);
          *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(xb) + int_x_off(lane, ch)) = make_uint4(a.x, a.y, b.x, b.y);
        }
        return true;
      };
      uint64_t dw1[5] = {};
      float db1 = 0.f;
      double llacc = 0.0;
      if (first < end) stage_rows(first);
      else if (lane == 0) mbar_arrive(&bar_scale);

      int p0 = n0;
      do {
        const int p1 = min(p0 + FIN_SUB, end), pf = p0 + ((wg - p0) & 3);
        bool any_far = false;
        uint64_t acc[Warp::LEAN];  // sums by FFMA, once there are any
#pragma unroll 1
        for (int n = pf; n < p1; n += NWG) {
          wait(&bar_fwd[n & 1], n >> 1 & 1, 102);
          tc_fence_after();
          uint64_t h[4][5];
          lanes.load(tmem + place(n) + SPLIT_A_COLS + sub, h);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar_read[n & 1]);
          if (n >= NWG) wait(&bar_sum[wg], (n - NWG) >> 2 & 1, 104);  // the last tile's integers have been read
          if (lane == 0) {
            if (n + NWG < end) {
              uint64_t* const bar = &bar_rows[warp][(n + NWG) >> 2 & 1];
              mbar_expect_tx(bar, WARP_BYTES);
              bulk_g2s(xs + ((n + NWG) >> 2 & 1) * G::XS, rows_at(seg, n + NWG - n0), WARP_BYTES, bar);
            } else {
              fetch(n + NWG, sg, n0);
            }
          }
          const int row = row0 + (n - first) * (Warp::ROWS / NWG);
          const bool valid = row < g.n_rows;
          float d[4], dy, pred;
          lanes.front(h, w1, g.lik, y, valid, d, dy, pred, [](int) {});
          const bool known = !plain && !plain_w;  // what the tensor core made of these rows is their z
          if (__builtin_expect(known, 1)) {
            lanes.template store_ei<false>(h, d, FIN_ONE, es, dw1);
            if (LOSS) {
              const float loss = valid ? lik_loss(g.lik, y, pred) : 0.f;
              llacc += (double)loss;
              store_row_loss(g.row_loss, (long long)win * g.row_loss_stride + row, loss, valid);
            }
            db1 += dy;
          }
          if (n + NWG < end) stage_rows(n + NWG);  // (its product goes on beside what follows)
          const float dy_row = __shfl_sync(0xffffffffu, dy, lanes.owner());
          float dx = dy_row;
          if (__builtin_expect(n == first, 0)) {  // ranges: from every second of all warps' first 32 rows, 256 in all (all 512: 0.4 us more)
            unit_statistics(xs + (n >> 2 & 1) * G::XS, dx, known, x_stat, x_max);
            dx = 1.f;
            if (lane == 0) mbar_arrive(&bar_scale);
            wait(&bar_scale, (sg - seg0) & 1, 105);
            if (g.test_code == 105 && warp == 5) wait(&bar_scale, (sg - seg0 + 1) & 1, 105);  // (the next segment's)
            unit_ranges(x_stat, x_max, x_scale);
            some_new = __any_sync(0xffffffffu, lane < D && x_new[lane] > 0.f) != 0;
          }
          const bool near = products(xs + (n >> 2 & 1) * G::XS, dx) && known;
          if (__builtin_expect(!near, 0)) {
            if (!any_far)
              for (int i = 0; i < Warp::LEAN; ++i) acc[i] = 0ull;
            any_far = true;
            const int b = (n - pf) >> 2;
            if (known) unit_far(xs + (n >> 2 & 1) * G::XS, es, acc, rows_at(seg, n - n0), dy_row);
            else if (lane == 0) far_tiles[warp][b >> 5] |= 1u << (b & 31);
          }
          fence_proxy_async_smem();  // (also without an MMA: the next copy goes to where the rows' integers are)
          if (lane == 0) far[warp] = near ? 0u : 1u;
          hand_over(&bar_e[wg]);
        }
        // ---- rows whose z the tensor core does not know: all of them by FFMA; the sums of what has gone that way to where dL/dz was ----
        if (__builtin_expect(any_far, 0)) {
          const int last = pf + (p1 - 1 - pf) / NWG * NWG;
          wait(&bar_sum[wg], last >> 2 & 1, 104);
          float* const xb = xs + (last >> 2 & 1) * G::XS;
#pragma unroll 1
          for (int n = pf; n < p1; n += NWG) {
            const int b = (n - pf) >> 2;
            if (!(reinterpret_cast<volatile uint32_t*>(far_tiles[warp])[b >> 5] >> (b & 31) & 1u)) continue;
            const float4* src = reinterpret_cast<const float4*>(rows_at(seg, n - n0));
            __syncwarp();
            for (int i = lane; i < G::XS / 4; i += 32) reinterpret_cast<float4*>(xb)[i] = src[i];
            __syncwarp();
            uint64_t h[4][5];
            float d[4], dy, pred;
            Warp::plain<2>(xb, wb, es);
            lanes.load_plain(es, h);
            __syncwarp();
            const int row = row_at(seg, n - n0) + own;
            const bool valid = row < g.n_rows;
            const float yf = xb[own * KP + COL_Y];
            lanes.front(h, w1, g.lik, yf, valid, d, dy, pred, [](int) {});
            lanes.store_es(h, d, es, dw1);
            if (LOSS) {
              const float loss = valid ? lik_loss(g.lik, yf, pred) : 0.f;
              llacc += (double)loss;
              store_row_loss(g.row_loss, (long long)win * g.row_loss_stride + row, loss, valid);
            }
            db1 += dy;
            Warp::backward_lean<2>(xb, es, acc);
          }
          Warp::store_dw0_lean(acc, es + (lanes.kh * Warp::KPT + lanes.rsub * 6) * H);
          for (int i = lane; i < FAR_WORDS; i += 32) far_tiles[warp][i] = 0u;
          fence_proxy_async_smem();
        }
        if (lane == 0) far_any[warp] = any_far ? 1u : 0u;
        // ---- lanes -> warp ----
        if (p1 == end) {
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
        }
        __syncthreads();  // S2
        tc_fence_after();
        if ((warp & 3) < INT_LINES / 32) {
          const float unit = x_unit[(warp & 3) * 8 + (lane >> 2)];
          float v[10];
          int_read_out_long<10>(tmem + wg * 40 + sub, v);
          const float f = (float)(1 << 8 * (lane & 3)) / FIN_ONE, inv = unit > 0.f ? 1.f / unit : 0.f;
#pragma unroll
          for (int j = 0; j < 10; ++j)
            base[G::S + (wg * 10 + j) * INT_S_STR + (warp & 3) * 32 + lane] = none ? 0.f : v[j] * f * inv;
        }
        tc_fence_before();
        __syncthreads();  // S3
        // ---- one partial vector for (window, slot) ----
        const size_t slot = (size_t)win * g.slices_out + seg.w;
        float* po = g.partial_out + slot * g.Pp;
        // warps in the order of the segment's tiles, whichever warpgroup took its first one: bits depend on the segment alone
        auto nth = [&](int i) __attribute__((always_inline)) { return ((n0 + (i >> 2)) & 3) << 2 | (i & 3); };
        const uint32_t far_w = __ballot_sync(0xffffffffu, lane < NW && far_any[nth(lane & (NW - 1))] != 0u);
        for (int p = tid; p < P; p += NCOMPUTE) {
          float s;
          if (p < D * H + H) {
            s = int_sum4(base + G::S, p / H, p % H);
            for (uint32_t r = far_w; r; r &= r - 1) s += base[G::ROWS0 + nth(__ffs(r) - 1) * G::WARP + 2 * G::XS + p];
            s *= w1[p % H];   // dL/dz was left without it
            if (p0 > n0) s += po[p];
          } else if (p1 < end) {
            continue;
          } else if (p < D * H + 2 * H) {
            const int u = p - (D * H + H);
            s = red_w1[nth(0)][u];
#pragma unroll
            for (int w = 1; w < NW; ++w) s += red_w1[nth(w)][u];
          } else {
            s = red_db1[nth(0)];
#pragma unroll
            for (int w = 1; w < NW; ++w) s += red_db1[nth(w)];
          }
          po[p] = s;
        }
        if (tid == 0 && p1 == end) {
          double s = red_ll[nth(0)];
#pragma unroll
          for (int w = 1; w < NW; ++w) s += red_ll[nth(w)];
          g.ll_out[slot] = s;
        }
        if (p1 == end) {
          if (tid < KP) x_stat[tid] = x_max[tid] = 0u;
        }
        __syncthreads();  // S4: the next segment's parameters may take the place of this one's
        p0 += FIN_SUB;
      } while (p0 < end);
      n0 = end;
    }
    if (g.test_code == 102) wait(&bar_fwd[0], (n0 + 1) >> 1 & 1, 102);  // (nothing ends this phase)
    if (!ok) {  // copies and MMAs that did not arrive in time
      atomicExch(g.status, late);
      for (int n = max(n0 - 2 * NWG, 0); n < n0; ++n) {
        if ((n & 3) != wg) continue;
        mbar_drain(&bar_rows[warp][n >> 2 & 1], n >> 3 & 1);
        if (n >= n0 - 2) mbar_drain(&bar_fwd[n & 1], n >> 1 & 1);
        if (n >= n0 - NWG) mbar_drain(&bar_sum[wg], n >> 2 & 1);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)G::TMEM_COLS)
                 : "memory");
}

template <bool LOSS>
static cudaError_t launch_int_t(const GradParams& g, int ctas, cudaStream_t st) {
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !attr_done[dev]) {
    cudaError_t e =
        cudaFuncSetAttribute(grad_fp32_int_kernel<LOSS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FinGeom::SMEM);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_done[dev] = true;
  }
  return launch_chain_kernel(grad_fp32_int_kernel<LOSS>, dim3(ctas), dim3(FIN_THREADS), FinGeom::SMEM, st, g);
}
cudaError_t launch_grad_fp32_int(const GradParams& g, int ctas, cudaStream_t st) {
  return g.no_loss ? launch_int_t<false>(g, ctas, st) : launch_int_t<true>(g, ctas, st);
}

}  // namespace mcmc_b200
