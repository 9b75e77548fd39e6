// Forward-only pass over (stored samples x rows): posterior-mean prediction and the mean losses over the
// stored samples.  The reference evaluates its stored samples one at a time through the full
// forward+backward kernel with eps = 0 (output_final_loss, include/mcmc/main.h:78-115, followed by two CUB
// reductions per sample, kernel_helpers.h:190-216); here one launch covers all samples and all rows and
// computes no gradient.
//
//   * FP32 with the reference's tanh (kernel_helpers.h:32-44): the result is the FP32 forward pass
//     whatever precision the chain was sampled in;
//   * 40 units: forward_split_kernel, the product on the tensor core;
//   * 128 units: forward_samples_kernel, FFMA.  A CTA owns 512 rows (4 per thread, held in registers for the whole launch) and
//     walks through its chunk of the samples; a sample's 3073 parameters are staged in shared memory once per CTA, the next
//     one's while this one is worked on, and read as 16-byte broadcasts: 16 multiplications per load.  Two units to a
//     packed FMA, the row's feature as one value for both: that issues every 2.3 cycles of a scheduler where one with three
//     different pairs takes 2.8 and two single ones 2.1 to 2.3 and twice the issue slots, which the tanh needs (58368 rows x
//     800 samples: 6.42 ms a call instead of 7.15);
//   * PREDICT: per-row sums over the chunk's samples -> partial[chunk][row]; LOSS: per-sample sums over the
//     CTA's rows -> partial[tile][sample].  A second small launch adds the partials in a fixed order (and, for
//     LOSS, the log-prior of every sample).  Doubles, no atomics: bit-reproducible.
#include <algorithm>
#include "chain.cuh"
#include "common.cuh"
#include "split_mma.cuh"

namespace mcmc_b200 {

constexpr int FWD_THREADS = 128, FWD_RPT = 4, FWD_ROWS = FWD_THREADS * FWD_RPT;
constexpr int FWD_CTAS_PER_SM = 3;  // (registers: the rows)

template <int H, bool LOSS>
__global__ void __launch_bounds__(FWD_THREADS, FWD_CTAS_PER_SM) forward_samples_kernel(const ForwardParams a) {
  constexpr int D = 22, P = D * H + 2 * H + 1;
  constexpr int SW = (P + 3) / 4 * 4;
  // one sample: W0[k][j], b0, W1, b1
  extern __shared__ __align__(16) float sw_raw[];
  __shared__ double red[FWD_THREADS / 32];
  const int tid = threadIdx.x;
  const long long row0 = (long long)blockIdx.x * FWD_ROWS;
  const int s0 = (int)((long long)blockIdx.y * a.count / gridDim.y);
  const int s1 = (int)((long long)(blockIdx.y + 1) * a.count / gridDim.y);
  auto stage = [&](int s) {
    float* dst = sw_raw + (s & 1) * SW;
    for (int p = tid; p < P; p += FWD_THREADS) {
      const uint32_t d = smem_u32(dst + p);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(a.samples + (size_t)s * P + p) : "memory");
    }
  };
  if (s0 < s1) stage(s0);
  // rows tid, tid + 128, ...: consecutive threads read consecutive rows
  float x[FWD_RPT][D];
  float y[FWD_RPT];
  bool valid[FWD_RPT];
#pragma unroll
  for (int r = 0; r < FWD_RPT; ++r) {
    const long long row = row0 + r * FWD_THREADS + tid;
    valid[r] = row < a.n;
    const float* xr = a.x + row * a.x_stride;
#pragma unroll
    for (int k = 0; k < D; ++k) x[r][k] = valid[r] ? xr[k] : 0.f;
    y[r] = (LOSS && valid[r]) ? a.y[row * a.y_stride] : 0.f;
  }
  double acc[FWD_RPT];
#pragma unroll
  for (int r = 0; r < FWD_RPT; ++r) acc[r] = 0.0;

  for (int s = s0; s < s1; ++s) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // the sample has arrived, and nobody reads the other buffer any more
    if (s + 1 < s1) stage(s + 1);
    const float* sw = sw_raw + (s & 1) * SW;
    float pred[FWD_RPT];
#pragma unroll
    for (int r = 0; r < FWD_RPT; ++r) pred[r] = sw[D * H + 2 * H];
#pragma unroll 1
    for (int j0 = 0; j0 < H; j0 += 4) {
      uint64_t zp[FWD_RPT][2];
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(sw + D * H + j0);
#pragma unroll
      for (int r = 0; r < FWD_RPT; ++r) {
        zp[r][0] = b.x;
        zp[r][1] = b.y;
      }
#pragma unroll
      for (int k = 0; k < D; ++k) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(sw + k * H + j0);
#pragma unroll
        for (int r = 0; r < FWD_RPT; ++r) {
          zp[r][0] = fma2(w.x, pack2(x[r][k], x[r][k]), zp[r][0]);
          zp[r][1] = fma2(w.y, pack2(x[r][k], x[r][k]), zp[r][1]);
        }
      }
      float z[FWD_RPT][4];
#pragma unroll
      for (int r = 0; r < FWD_RPT; ++r) {
        unpack2(zp[r][0], z[r][0], z[r][1]);
        unpack2(zp[r][1], z[r][2], z[r][3]);
      }
      const float4 w1 = *reinterpret_cast<const float4*>(sw + D * H + H + j0);
#pragma unroll
      for (int r = 0; r < FWD_RPT; ++r) {
        pred[r] = fmaf(w1.x, tanh_ref(z[r][0]), pred[r]);
        pred[r] = fmaf(w1.y, tanh_ref(z[r][1]), pred[r]);
        pred[r] = fmaf(w1.z, tanh_ref(z[r][2]), pred[r]);
        pred[r] = fmaf(w1.w, tanh_ref(z[r][3]), pred[r]);
      }
    }
    if (LOSS) {
      double l = 0.0;
#pragma unroll
      for (int r = 0; r < FWD_RPT; ++r) {
        float loss, dy;
        lik_terms(a.lik, y[r], pred[r], loss, dy);
        if (valid[r]) l += (double)loss;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
      if ((tid & 31) == 0) red[tid >> 5] = l;
      __syncthreads();
      if (tid == 0) {
        double t = red[0];
#pragma unroll
        for (int w = 1; w < FWD_THREADS / 32; ++w) t += red[w];
        a.partial[(size_t)blockIdx.x * a.count + s] = t;
      }
    } else {
#pragma unroll
      for (int r = 0; r < FWD_RPT; ++r) acc[r] += (double)pred[r];
    }
  }
  if (!LOSS) {
#pragma unroll
    for (int r = 0; r < FWD_RPT; ++r) {
      const long long row = row0 + r * FWD_THREADS + tid;
      if (valid[r]) a.partial[(size_t)blockIdx.y * a.n + row] = acc[r];
    }
  }
}

// PREDICT: out[row] = sum over chunks / count.  LOSS: per sample the sum over row tiles -> out_ll[s], the
// log-prior of the sample -> out_lp[s] (one CTA per sample).
__global__ void forward_finish_predict(const double* partial, int chunks, long long n, int count, float* out) {
  const long long row = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (row >= n) return;
  double t = 0.0;
  for (int c = 0; c < chunks; ++c) t += partial[(size_t)c * n + row];
  out[row] = (float)(t / (double)count);
}
__global__ void __launch_bounds__(128) forward_finish_loss(const double* partial, int tiles, int count,
                                                           const float* samples, int P, PriorParams prior,
                                                           double* out_ll, double* out_lp) {
  __shared__ double dsc[32];
  const int s = blockIdx.x;
  double t = 0.0;
  for (int k = threadIdx.x; k < tiles; k += blockDim.x) t += partial[(size_t)k * count + s];
  const double ll = block_sum_f64(t, dsc);
  double lp = 0.0;
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const float w = samples[(size_t)s * P + p];
    const float q = w * prior.inv_s;
    lp += (double)fmaf(-0.5f * q, q, -prior.norm);
  }
  lp = block_sum_f64(lp, dsc);
  if (threadIdx.x == 0) {
    out_ll[s] = ll;
    out_lp[s] = lp;
  }
}

// ---- 40 units: the product on the tensor core (split_mma.cuh) ----------------------------------
// What bounds it: MUFU.  A tanh of ex2 and rcp takes a scheduler 16 cycles a warp, 40 of them 640 cycles for the four warps
// of a 128-row tile; the tile's 18 MMAs take the tensor pipe 430, everything else 280 issue slots.
//   * four compute warpgroups, a row per thread, the rows' parts in tensor memory as long as the CTA works on them.  Beside them is
//     room for two pairs of accumulators, which the warpgroups use in turn: one takes z into registers and hands its pair on, so
//     that MMAs run during everybody's tanh passes;
//   * two warps stage the samples' parts, up to FWS_NB samples ahead, and one for each pair of accumulators issues the MMAs;
//   * persistent, one CTA per SM (a kernel with tensor memory gets no more).  (row tile, sample) pairs, tile by tile, are cut
//     into one equal range per CTA: no last round that is nearly empty.  A tile's sums from several CTAs are added by
//     forward_split_finish in the order of the CTAs.
// A sample of 58368 rows takes 1.29 us (MUFU alone: 1.03; the FFMA kernel 2.3).  Three warpgroups with a pair each 1.48, four with
// two pairs and one issuing warp 1.44: its MMAs came 52 cycles apart, most of it waiting.  58368 rows x 800 samples, a call: 2.28 ms
// (FFMA), 1.81 (first version), 1.37; of that 0.35 are copies from and to pageable memory.
constexpr int FWS_NWG = FWS_ROWS / 128, FWS_THREADS = FWS_NWG * 128 + 128, FWS_NB = 3;
constexpr int FWS_Z_COL0 = FWS_NWG * SPLIT_A_COLS, FWS_NZ = 2;   // accumulator pairs
constexpr int FWS_TMEM_COLS = 512;
constexpr int FWS_W1 = SPLIT_H + 4;                       // W1, b1
constexpr int FWS_STAGERS = 2;                            // warps that stage samples
constexpr int FWS_QUADS = SPLIT_K / 4 * SPLIT_H;          // four features of a unit
constexpr int FWS_QPT = (FWS_QUADS + FWS_STAGERS * 32 - 1) / (FWS_STAGERS * 32);
static_assert(FWS_STAGERS + FWS_NZ == 4 && FWS_NWG % FWS_NZ == 0 && FWS_Z_COL0 + FWS_NZ * SPLIT_Z_COLS <= FWS_TMEM_COLS, "tensor memory budget");
constexpr size_t FWS_SMEM = 1024 + FWS_NB * SPLIT_B_BYTES;

// first CTA of `ctas` whose range of `units` reaches past unit u
__host__ __device__ inline long long fws_first_cta(long long u, long long units, int ctas) {
  return ((u + 1) * ctas - 1) / units;
}

// z of this thread's row by FFMA into its accumulators, for rows or samples that split_wide finds: even and odd features apart,
// added at the end
__device__ __noinline__ void fws_plain(const float* xr, bool valid, const float* smp, uint32_t z_t) {
#pragma unroll 1
  for (int j0 = 0; j0 < SPLIT_H; j0 += 8) {
    float z[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float even = __ldg(smp + SPLIT_D * SPLIT_H + j0 + j), odd = 0.f;
#pragma unroll 1
      for (int k = 0; k < SPLIT_D; k += 2) {
        even = fmaf(valid ? xr[k] : 0.f, __ldg(smp + k * SPLIT_H + j0 + j), even);
        odd = fmaf(valid ? xr[k + 1] : 0.f, __ldg(smp + (k + 1) * SPLIT_H + j0 + j), odd);
      }
      z[j] = even + odd;
    }
    __syncwarp();
    tc_st8(z_t + SPLIT_S0 + j0, make_float4(z[0], z[1], z[2], z[3]), make_float4(z[4], z[5], z[6], z[7]));
    tc_st8(z_t + j0, make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f));
  }
  tc_wait_st();
}

template <bool LOSS>
__global__ void __launch_bounds__(FWS_THREADS, 1) forward_split_kernel(const ForwardParams a) {
  constexpr int H = SPLIT_H, D = SPLIT_D, P = D * H + 2 * H + 1, NB = FWS_NB, NWG = FWS_NWG;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* const bs = smem_align1024(smem_raw);
  __shared__ __align__(16) float w1s[NB][FWS_W1];
  __shared__ double red[NB][NWG * 4];
  __shared__ int wide_w[NB][FWS_STAGERS];
  __shared__ __align__(8) uint64_t bar_b[NB], bar_done[NB], bar_z[NWG], bar_free[FWS_NZ], bar_a[NWG];
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  // samples [i0, i0 + n) of the flattened (tile, sample) list are this CTA's
  const long long cells = a.whole ? forward_split_tiles(a.n) : forward_split_tiles(a.n) * a.count;
  const long long c0 = cells * blockIdx.x / gridDim.x, c1 = cells * (blockIdx.x + 1) / gridDim.x;
  const long long u0 = a.whole ? c0 * a.count : c0, u1 = a.whole ? c1 * a.count : c1;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"((uint32_t)FWS_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int b = 0; b < NB; ++b) {
      mbar_init(&bar_b[b], FWS_STAGERS);
      mbar_init(&bar_done[b], NWG * 4);
    }
    for (int w = 0; w < NWG; ++w) {
      mbar_init(&bar_z[w], 1);
      mbar_init(&bar_a[w], 4);
    }
    for (int z = 0; z < FWS_NZ; ++z) mbar_init(&bar_free[z], 4);
    mbar_fence_init();
  }
  for (int i = tid; i < NB * SPLIT_B_BYTES / 16; i += FWS_THREADS)
    reinterpret_cast<float4*>(bs)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  bool ok = true;
  const long long n = u1 - u0;

  if (warp < NWG * 4) {
    // =====================  compute warpgroups: a row per thread  =====================
    const int wg = warp >> 2;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t a_t = tmem + wg * SPLIT_A_COLS + lanes, z_t = tmem + FWS_Z_COL0 + wg % FWS_NZ * SPLIT_Z_COLS + lanes;
    long long i = 0;
    uint32_t b = 0, use = 0;  // sample i is staged in buffer i % NB, for the i / NB-th time
    while (i < n) {
      // ---- a row tile (all of it, or the samples of it that this CTA has) ----
      const long long t = (u0 + i) / a.count;
      const long long end = min(n, (t + 1) * a.count - u0);
      const long long row = t * FWS_ROWS + tid;
      const bool valid = row < a.n;
      const float* const xr = a.x + row * a.x_stride;
      bool wide = false;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int f = 8 * j + k;
          v[k] = f < D ? (valid ? xr[f] : 0.f) : f == D ? 1.f : 0.f;
          wide |= split_wide(v[k]);
        }
        split_store_row(a_t, j, v);
      }
      wide = __any_sync(0xffffffffu, wide);
      const float y = (LOSS && valid) ? a.y[row * a.y_stride] : 0.f;
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_a[wg]);
      double acc = 0.0;
      for (; i < end; ++i) {
        mbar_wait_q(&bar_b[b], use & 1, a.status, 401, ok);
        mbar_wait_q(&bar_z[wg], (uint32_t)i & 1, a.status, 402, ok);
        tc_fence_after();
        if (wide || (wide_w[b][0] | wide_w[b][1])) fws_plain(xr, valid, a.samples + ((u0 + i) % a.count) * P, z_t);
        uint64_t z[H / 2];
#pragma unroll
        for (int c0 = 0; c0 < H; c0 += 16) {  // (in pieces: registers)
          float s1[16], s0[16];
#pragma unroll
          for (int c = 0; c < 16 && c0 + c < H; c += 8) {
            tc_ld8(z_t + c0 + c, s1 + c);
            tc_ld8(z_t + SPLIT_S0 + c0 + c, s0 + c);
          }
          tc_wait_ld();
#pragma unroll
          for (int c = 0; c < 16 && c0 + c < H; c += 2) z[(c0 + c) / 2] = add2(pack2(s0[c], s0[c + 1]), pack2(s1[c], s1[c + 1]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_free[wg % FWS_NZ]);
        uint64_t pred2 = pack2(w1s[b][H], 0.f);
#pragma unroll
        for (int j = 0; j < H; j += 4) {
          const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&w1s[b][j]);
          pred2 = fma2(w.x, tanh_ref2(z[j / 2]), pred2);
          pred2 = fma2(w.y, tanh_ref2(z[j / 2 + 1]), pred2);
        }
        float pred, pred1;
        unpack2(pred2, pred, pred1);
        pred += pred1;
        if (LOSS) {
          float loss, dy;
          lik_terms(a.lik, y, pred, loss, dy);
          double l = valid ? (double)loss : 0.0;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
          if (lane == 0) red[b][warp] = l;
        } else {
          acc += (double)pred;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_done[b]);
        if (++b == NB) b = 0, ++use;
      }
      if (!LOSS && valid) {
        const long long first = a.whole ? blockIdx.x : fws_first_cta(t * a.count, cells, gridDim.x);
        a.partial[(blockIdx.x - first) * a.n + row] = acc;
      }
    }
  } else if (warp < NWG * 4 + FWS_STAGERS) {
    // =====================  staging warps: a sample's weights in parts  =====================
    const int st = tid - NWG * 128, sw = warp - NWG * 4;
    float v[FWS_QPT][4], v1 = 0.f;
    int smp = n > 0 ? (int)(u0 % a.count) : 0;
    auto load = [&]() {  // the next sample
      const float* s = a.samples + (size_t)smp * P;
      if (++smp == a.count) smp = 0;
#pragma unroll
      for (int q = 0; q < FWS_QPT; ++q) {
        const int task = st + q * FWS_STAGERS * 32, k0 = task / H * 4, un = task % H;
#pragma unroll
        for (int k = 0; k < 4; ++k) v[q][k] = k0 + k <= D && task < FWS_QUADS ? __ldg(s + (k0 + k) * H + un) : 0.f;
      }
      if (st <= H) v1 = __ldg(s + (D + 1) * H + st);
    };
    // LOSS: the rows' sum of sample i, once every warp has delivered its own (one thread)
    auto finish = [&](long long i, uint32_t b) {
      if (LOSS && st == 0) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < NWG * 4; ++w) s += red[b][w];
        a.partial[u0 + i] = s;
      }
    };
    if (n > 0) load();
    uint32_t b = 0, use = 0;
    for (long long i = 0; i < n; ++i) {
      if (i >= NB) {
        mbar_wait_q(&bar_done[b], (use - 1) & 1, a.status, 403, ok);
        finish(i - NB, b);
        __syncwarp();
      }
      unsigned char* const base = bs + b * SPLIT_B_BYTES;
      bool wide = false;
#pragma unroll
      for (int q = 0; q < FWS_QPT; ++q) {
        const int task = st + q * FWS_STAGERS * 32, k0 = task / H * 4, un = task % H;
        float p[3][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          split_parts<SPLIT_W_BITS, true>(v[q][k], p[0][k], p[1][k], p[2][k]);
          wide |= split_wide(v[q][k]);
        }
        if (task < FWS_QUADS) {
          float* d = reinterpret_cast<float*>(base + split_b_off(un, k0));
#pragma unroll
          for (int r = 0; r < 3; ++r)
            *reinterpret_cast<float4*>(d + r * (SPLIT_B_PART / 4)) = make_float4(p[r][0], p[r][1], p[r][2], p[r][3]);
        }
      }
      if (st <= H) w1s[b][st] = v1;
      wide = __any_sync(0xffffffffu, wide);
      if (lane == 0) wide_w[b][sw] = wide;
      if (i + 1 < n) load();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_b[b]);
      if (++b == NB) b = 0, ++use;
    }
    if (LOSS)  // the last ones: buffer b is the next one to be used, so its sample is the oldest
      for (long long i = n - NB; i < n; ++i) {
        if (i >= 0) {
          mbar_wait_q(&bar_done[b], (use - 1) & 1, a.status, 404, ok);
          finish(i, b);
        }
        if (++b == NB) b = 0, ++use;
      }
  } else {
    // =====================  issuing warps: one for each pair of accumulators  =====================
    const int z = warp - NWG * 4 - FWS_STAGERS;
    const uint32_t on = elect_one();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0), b_smem = smem_u32(bs);
    long long next = 0;  // first sample of the next row tile
    uint32_t seg = 0, b = 0, use = 0, turn = 0;
    for (long long i = 0; i < n; ++i) {
      const bool tile = i == next;
      mbar_wait_q(&bar_b[b], use & 1, a.status, 405, ok);
      for (int w = z; w < NWG; w += FWS_NZ, ++turn) {
        if (turn > 0) mbar_wait_q(&bar_free[z], (turn - 1) & 1, a.status, 406, ok);
        if (tile) mbar_wait_q(&bar_a[w], seg & 1, a.status, 407, ok);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        if (ok) {
          split_issue(tm + FWS_Z_COL0 + z * SPLIT_Z_COLS, tm + w * SPLIT_A_COLS, b_smem + b * SPLIT_B_BYTES, on);
          tc_commit_if(&bar_z[w], on);
        }
      }
      if (tile) {
        ++seg;
        next = ((u0 + i) / a.count + 1) * a.count - u0;
      }
      if (++b == NB) b = 0, ++use;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)FWS_TMEM_COLS)
                 : "memory");
}

// PREDICT, 40 units: as forward_finish_predict, over the CTAs that had samples of the row's tile
__global__ void forward_split_finish(const ForwardParams a, int ctas, float* out) {
  const long long row = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (row >= a.n) return;
  int slots = 1;
  if (!a.whole) {
    const long long t = row / FWS_ROWS, cells = forward_split_tiles(a.n) * a.count;
    slots = (int)(fws_first_cta((t + 1) * a.count - 1, cells, ctas) - fws_first_cta(t * a.count, cells, ctas)) + 1;
  }
  double s = 0.0;
  for (int c = 0; c < slots; ++c) s += a.partial[c * a.n + row];
  out[row] = (float)(s / (double)a.count);
}

int forward_row_tiles(int H, long long n) {
  return H == SPLIT_H ? (int)forward_split_tiles(n) : (int)((n + FWD_ROWS - 1) / FWD_ROWS);
}

// Sample chunks per row tile, at most `most` and one per sample.  All CTAs take the same time, so what counts is how many
// rounds of the GPU they make and how many samples the longest one has; a CTA's start (its rows, its first sample)
// costs about two samples.  58368 rows x 800 samples: 8 chunks would be 2.07 rounds, paid as three.
int forward_chunks(int num_sms, long long n, int count, int most) {
  const long long tiles = (n + FWD_ROWS - 1) / FWD_ROWS, slots = (long long)num_sms * FWD_CTAS_PER_SM;
  long long best = 0;
  int ch = 1;
  for (int k = 1; k <= std::min(count, most); ++k) {
    const long long cost = (tiles * k + slots - 1) / slots * ((count + k - 1) / k + 2);
    if (k == 1 || cost < best) {
      best = cost;
      ch = k;
    }
  }
  return ch;
}

// CTAs of forward_split_kernel for this many rows and samples, and the most of them that share a row tile
int forward_split_ctas(int num_sms, const ForwardParams& a) {
  const long long cells = a.whole ? forward_split_tiles(a.n) : forward_split_tiles(a.n) * a.count;
  return (int)std::min<long long>(num_sms, cells);
}
int forward_split_slots(int num_sms, const ForwardParams& a) {
  if (a.whole) return 1;
  const long long ctas = forward_split_ctas(num_sms, a), least = forward_split_tiles(a.n) * a.count / ctas;
  return (int)std::min<long long>(ctas, a.count / least + 2);
}

template <bool LOSS>
static cudaError_t launch_forward_split_t(const ForwardParams& a, int ctas, cudaStream_t st) {
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(forward_split_kernel<LOSS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FWS_SMEM);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_done[dev] = true;
  }
  forward_split_kernel<LOSS><<<ctas, FWS_THREADS, FWS_SMEM, st>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_forward_split(const ForwardParams& a, int num_sms, bool loss, cudaStream_t st) {
  const int ctas = forward_split_ctas(num_sms, a);
  return loss ? launch_forward_split_t<true>(a, ctas, st) : launch_forward_split_t<false>(a, ctas, st);
}
cudaError_t launch_forward_split_finish(const ForwardParams& a, int num_sms, float* out, cudaStream_t st) {
  forward_split_finish<<<(unsigned)((a.n + 255) / 256), 256, 0, st>>>(a, forward_split_ctas(num_sms, a), out);
  return cudaGetLastError();
}

// (128 units; 40 go through forward_split_kernel)
cudaError_t launch_forward_samples(int H, const ForwardParams& a, int chunks, bool loss, cudaStream_t st) {
  constexpr int W = 128, P = 22 * W + 2 * W + 1;
  if (H != W) return cudaErrorInvalidValue;
  const size_t smem = 2 * sizeof(float) * ((P + 3) / 4 * 4);
  const dim3 grid((unsigned)((a.n + FWD_ROWS - 1) / FWD_ROWS), chunks);
  if (loss) forward_samples_kernel<W, true><<<grid, FWD_THREADS, smem, st>>>(a);
  else forward_samples_kernel<W, false><<<grid, FWD_THREADS, smem, st>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_forward_finish_predict(const double* partial, int chunks, long long n, int count, float* out,
                                          cudaStream_t st) {
  forward_finish_predict<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(partial, chunks, n, count, out);
  return cudaGetLastError();
}
cudaError_t launch_forward_finish_loss(const double* partial, int tiles, int count, const float* samples, int P,
                                       const PriorParams& prior, double* out_ll, double* out_lp, cudaStream_t st) {
  forward_finish_loss<<<count, 128, 0, st>>>(partial, tiles, count, samples, P, prior, out_ll, out_lp);
  return cudaGetLastError();
}

}  // namespace mcmc_b200
