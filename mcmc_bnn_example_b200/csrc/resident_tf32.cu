// Tile arithmetic of the resident kernel in TF32 mode (resident.cuh has the launch structure): the same tcgen05
// formulation as grad_tf32.cu — forward with the rows as A operand in tensor memory, E = (1 - h^2) dL/dpred through
// shared memory, backward with two 32-row groups per MMA — for ONE tile per warpgroup that never moves:
//   * the row tile stays in shared memory (backward operand) and in tensor memory (forward operand) for the whole
//     launch, y in a register;
//   * the tiles' backward MMAs accumulate, in a fixed order, into ONE accumulator that is read out once per step.
//     Issuing holds a warp up (about 70 cycles per MMA): the forward MMAs are issued by the warp whose turn comes
//     last, the backward MMAs by one of the first warpgroup, which is done first (or by a warp without rows);
//   * the warpgroups take turns at the tanh pass (MUFU bound, about 330 cycles for a warpgroup alone): in step with one
//     another all of them would finish it at the end of its 1,300 cycles, and the E stores and backward MMAs of the
//     first ones, 640 and 1,150 cycles for four tiles, would start only then.  A turn is handed over half way, where the
//     CTA has four tiles at its end (us a step, half way and at the end: 4096 rows 3.84 and 3.77, 58368 5.69 and 5.64; always
//     at the three-quarter mark, fewer tiles: 2000 rows 2.95 and 3.02, 30011 4.79 and 4.85);
//   * Z is read in the 16-lane quad shape: a thread holds 10 hidden units of 4 rows.  A row's output sum then takes
//     two shuffle levels inside the quad, but dW1 is 10 sums of 4 rows in registers instead of 40 sums of one: 10
//     shuffles instead of 45 per step (the shuffles were 1,800 of the step's cycles, the longest single item).
// What bounds a step: latencies in a row — 3 MMAs, 40 tanh per row, E through shared memory, 8 MMAs, read-out —
// and the exchange.
#include <cuda.h>
#include <utility>
#include "resident.cuh"

namespace mcmc_b200 {

struct ResTf32 {
  static constexpr int H = 40, D = 22, NF = 48, GM = 64, GN = 2 * H;
  static constexpr int TILE_BYTES = TF32_TILE * 128, GROUP_BYTES = 32 * 128;
  static constexpr int ES_ATOM_BYTES = H * 128, ES_WG_BYTES = 4 * ES_ATOM_BYTES;
  using Words = ResWords<H>;
  static constexpr int GPART = (3 * Words::W0 + 3) / 4 * 4;  // one row group's sums, in parameter order (padded)
  static constexpr int RS = 44;                             // row of a warp's sums: dW1, db1
  static constexpr int XB = 0, ES = XB + RES_NWG * TILE_BYTES, W0S = ES + RES_NWG * ES_WG_BYTES;
  static constexpr int GP = W0S + NF * 128;                 // [2 row groups][23 x H]
  static constexpr int RW1 = GP + (2 * GPART * 4 + 15) / 16 * 16;  // [warps][RS] dW1 and db1 of each warp's rows
  static constexpr int RLL = RW1 + RES_NWG * 4 * RS * 4;    // [warps] log-likelihood (double)
  static constexpr int W1S = RLL + RES_NWG * 4 * 8;         // [2H + 4]: W1, b1, (pad,) -W1, -W1[0], -W1[1]
  static constexpr int BARS = W1S + (2 * H + 8) * 4;        // per warpgroup: tile landed, forward done; backward done
  static constexpr int END = BARS + (RES_NWG * 2 + 1) * 8 + 8;
  static constexpr size_t SMEM = 1024 + END;
  static constexpr int A_COL0 = 0, A_STRIDE = 24, Z_COL0 = RES_NWG * A_STRIDE, Z_STRIDE = NF,
                       G_COL0 = Z_COL0 + RES_NWG * Z_STRIDE;
  static constexpr int TMEM_COLS = 512;
  static_assert(G_COL0 + GN <= TMEM_COLS, "tensor memory budget");

  static constexpr bool X_PLACE = false;
  unsigned char* base;
  int wg, wtid, warp, lane, row, n_units;
  bool tile_active, warp_active, next_active, valid;
  uint32_t tmem, par;
  float y;
  uint32_t e_off, s_dst[3], s_neg[3];
  int row0;

  __device__ __forceinline__ uint64_t* bar(int w, int k) const {
    return reinterpret_cast<uint64_t*>(base + BARS) + w * 2 + k;
  }
  __device__ __forceinline__ uint64_t* bar_bwd() const { return bar(RES_NWG, 0); }
  __device__ __forceinline__ float* w1s() const { return reinterpret_cast<float*>(base + W1S); }
  static constexpr int NEG = H + 4;   // w1s()[NEG + j] = -W1[j % H], j < H + 2

  __device__ __forceinline__ ResTf32(unsigned char* b, const ResidentParams& g, int win, int u0, int u1) : base(b) {
    const int tid = threadIdx.x;
    warp = tid >> 5;
    lane = tid & 31;
    wg = __shfl_sync(0xffffffffu, tid >> 7, 0);
    wtid = tid & 127;
    const int u = u0 + 4 * wg;                      // first 32-row unit of the tile
    tile_active = u < u1;
    warp_active = u + (warp & 3) < u1;
    next_active = u + 4 < u1;
    n_units = u1 - u0;
    row0 = (g.data_window0 + win) * g.rows_pad + u * 32;
    // the row whose loss this thread computes: quad q = lane / 4 holds rows q, q + 8, q + 16, q + 24 of the warp
    row = (u + (warp & 3)) * 32 + (lane >> 2) + 8 * (lane & 3);
    valid = warp_active && row < g.n_rows;
    par = 0;
    // E element (hidden j, row r): atom r / 32 (this warp), line j, 16-byte chunk (r % 32) / 4 ^ (j % 8).  This thread
    // stores rows q + 8 i and units 8 n + 2 c + e: chunk (q / 4 + 2 i) ^ (2 c + e), all 32 banks once per store
    const int q = lane >> 2, cc = lane & 3;
    // = (q / 4 ^ 2 c + e) ^ 2 i.  (One register instead of four: without it shared memory in its own address space made steps of 5000
    // to 30011 rows 1 % slower than through generic addresses; 7219 rows x 3 4.10 us generic, 4.16, 4.08 now)
    e_off = smem_u32(base + ES + wg * ES_WG_BYTES + (warp & 3) * ES_ATOM_BYTES) + 2 * cc * 128 + (((q >> 2) ^ (2 * cc)) << 4) +
            ((q & 3) << 2);
    stage_setup();
  }

  __device__ __forceinline__ bool setup(const CUtensorMap* tmap, const ResidentParams& g, int) {
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x;
    if (warp == 0) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                   "r"((uint32_t)TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
      for (int w = 0; w < RES_NWG; ++w)
        for (int k = 0; k < 2; ++k) mbar_init(bar(w, k), 1);
      mbar_init(bar_bwd(), 1);
      mbar_fence_init();
    }
    // operands and sums that nothing writes stay zero: padding rows of the weights, warps and warpgroups without rows
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = tid; i < (W0S + NF * 128 - ES) / 16; i += RES_THREADS) reinterpret_cast<float4*>(base + ES)[i] = zero;
    for (int i = tid; i < (W1S - GP) / 16; i += RES_THREADS) reinterpret_cast<float4*>(base + GP)[i] = zero;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = tmem_slot;
    y = 0.f;
    bool ok = true;
    if (tile_active) {
      unsigned char* xt = base + XB + wg * TILE_BYTES;
      if (wtid == 0) {
        mbar_expect_tx(bar(wg, 0), TILE_BYTES);
        tma_load_2d(xt, tmap, 0, row0, bar(wg, 0));
      }
      res_wait(bar(wg, 0), 0, g, g.wait_ticks << 2, 611, ok);
      if (!ok) res_drain(bar(wg, 0), 0, g);
      if (g.test_code == 611) res_wait(bar(wg, 0), 1, g, g.wait_ticks << 2, 611, ok);  // (nothing ends this phase)
      // this thread's row: 32-byte chunk j of row r sits at position j ^ (r % 4); once per launch, so bank
      // conflicts do not matter here.  Rows of other CTAs or windows in the tile are zeroed.
      const uint32_t xr = smem_u32(xt) + wtid * 128;
      const uint32_t a_t = tmem + A_COL0 + wg * A_STRIDE + ((uint32_t)((warp & 3) * 32) << 16);
      for (int j = 0; j < 3; ++j) {
        const uint32_t p = xr + ((j ^ (wtid & 3)) << 5);
        const float4 lo = warp_active ? lds128(p) : zero, hi = warp_active ? lds128(p + 16) : zero;
        tc_st8(a_t + j * 8, lo, hi);
        if (j == 2) reinterpret_cast<float*>(base + GP)[tid] = hi.w;  // y, on its way to the thread of its row
      }
      if (!warp_active)
        for (int j = 0; j < 8; ++j) reinterpret_cast<float4*>(xt + wtid * 128)[j] = zero;
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      y = reinterpret_cast<float*>(base + GP)[warp * 32 + (lane >> 2) + 8 * (lane & 3)];
    }
    __syncthreads();
    if (tid < RES_THREADS / 4) reinterpret_cast<float4*>(base + GP)[tid] = zero;
    fence_proxy_async_smem();
    return ok;
  }

  // word `threadIdx.x` of the weights: where its three values go (addresses found once, words of W1 twice, the second
  // copy negated; threads without a word write to a dummy place)
  __device__ __forceinline__ void stage_setup() {
    const int t = threadIdx.x;
    const uint32_t dummy = smem_u32(w1s() + 2 * H + 7);
    for (int q = 0; q < 3; ++q) {
      const int p = Words::param(t, q);
      s_dst[q] = s_neg[q] = dummy;
      if (t >= Words::N - 1 || !Words::valid(t, q)) continue;
      if (p < D * H + H) {
        // element (n = hidden unit, k) of the K-major B operand at n*128 + ((k/4) ^ (n%8))*16 + (k%4)*4
        const int k = p / H, n = p - k * H;
        s_dst[q] = smem_u32(base + W0S + n * 128 + (((k >> 2) ^ (n & 7)) << 4) + ((k & 3) << 2));
      } else {
        const int j = p - (D * H + H);
        s_dst[q] = smem_u32(w1s() + j);
        if (j < H) s_neg[q] = smem_u32(w1s() + NEG + j);
      }
    }
  }
  __device__ __forceinline__ void stage(const uint4& v) {
    st_shared(s_dst[0], v.x);
    st_shared(s_dst[1], v.y);
    st_shared(s_dst[2], v.z);
    if (warp == Words::W0 / 32 || warp == (Words::N - 1) / 32) {  // the warps with words of W1
      st_shared(s_neg[0], v.x ^ 0x80000000u);
      st_shared(s_neg[1], v.y ^ 0x80000000u);
      st_shared(s_neg[2], v.z ^ 0x80000000u);
      if (threadIdx.x == Words::W0) {  // -W1[0], -W1[1] once more after -W1[H - 1]
        w1s()[NEG + H] = -__uint_as_float(v.x);
        w1s()[NEG + H + 1] = -__uint_as_float(v.y);
      }
    }
    fence_proxy_async_smem();
    __syncthreads();
  }
  static __device__ __forceinline__ void st_shared(uint32_t a, uint32_t v) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
  }

  __device__ __forceinline__ void step(const ResidentParams& g, float* row_loss, bool last, bool& ok) {
    const int nt = (n_units + 3) / 4;
    if (warp == RES_NWG * 4 - 1) {
      issue_forward(nt);
      if (nt < RES_NWG)
        for (int w = 0; w < nt; ++w) issue_backward(w, nt, 160);
    }
    if (!tile_active) return;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t z_t = tmem + Z_COL0 + wg * Z_STRIDE + lanes;
    const float* w1 = w1s();
    uint64_t w1p[5];
#pragma unroll
    for (int n = 0; n < 5; ++n) w1p[n] = *reinterpret_cast<const uint64_t*>(w1 + 8 * n + 2 * (lane & 3));
    res_wait(bar(wg, 1), par, g, g.wait_ticks << 2, 612, ok);
    tc_fence_after();
    float dy_row = 0.f, loss = 0.f;
    if (wg > 0) named_sync(RES_BAR_T + wg, 256);  // the warpgroup before this one has had its turn
    if (warp_active) {
      uint64_t hp[4][5];
      float pr[4];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        // units 8n + 2c, 8n + 2c + 1 of rows q + 16 hf and q + 16 hf + 8
        float z[20];
        tc_ld_quad32(z_t + ((uint32_t)(hf * 16) << 16), z);
        tc_ld_quad8(z_t + ((uint32_t)(hf * 16) << 16) + 32, z + 16);
        tc_wait_ld();
#pragma unroll
        for (int i = 2 * hf; i < 2 * hf + 2; ++i) {
          uint64_t acc = 0ull;
#pragma unroll
          for (int n = 0; n < 5; ++n) {
            const float* p = z + 4 * n + 2 * (i & 1);
            hp[i][n] = pack2(tanh_fast(p[0]), tanh_fast(p[1]));
            acc = fma2(w1p[n], hp[i][n], acc);
          }
          float lo, hi;
          unpack2(acc, lo, hi);
          pr[i] = lo + hi;
        }
        if (next_active && hf == (nt == RES_NWG ? 1 : 0)) named_arrive(RES_BAR_T + wg + 1, 256);
      }
      // the quad's four lanes add up; lane c keeps row q + 8c
      const bool b1 = (lane & 2) != 0, b0 = (lane & 1) != 0;
      {
        const float s0 = b1 ? pr[0] : pr[2], s1 = b1 ? pr[1] : pr[3];
        float k0 = b1 ? pr[2] : pr[0], k1 = b1 ? pr[3] : pr[1];
        k0 += __shfl_xor_sync(0xffffffffu, s0, 2);
        k1 += __shfl_xor_sync(0xffffffffu, s1, 2);
        const float s = b0 ? k0 : k1;
        pr[0] = (b0 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, s, 1);
      }
      const float pred = pr[0] + w1[H];
      dy_row = lik_grad(g.lik, y, pred);
      dy_row = valid ? dy_row : 0.f;
      if (last) {
        loss = valid ? lik_loss(g.lik, y, pred) : 0.f;
        store_row_loss(row_loss, row, loss, valid);
      }
      // every lane of the quad needs the four dL/dpred
      float dy[4];
      {
        const float o1 = __shfl_xor_sync(0xffffffffu, dy_row, 1);
        const float a0 = b0 ? o1 : dy_row, a1 = b0 ? dy_row : o1;   // rows 8 (2 b1) and 8 (2 b1 + 1)
        const float c0 = __shfl_xor_sync(0xffffffffu, a0, 2), c1 = __shfl_xor_sync(0xffffffffu, a1, 2);
        dy[0] = b1 ? c0 : a0;
        dy[1] = b1 ? c1 : a1;
        dy[2] = b1 ? a0 : c0;
        dy[3] = b1 ? a1 : c1;
      }
      // t = dy h: the rows' share of dW1; -E = t h - dy to shared memory (grad_tf32.cu)
      uint64_t dw[5] = {0ull, 0ull, 0ull, 0ull, 0ull};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint64_t dy2 = pack2(dy[i], dy[i]), ndy2 = pack2(-dy[i], -dy[i]);
        const uint32_t off = e_off ^ (i << 5);
        store_e<0>(off, hp[i], dy2, ndy2, dw);
        store_e<1>(off, hp[i], dy2, ndy2, dw);
        store_e<2>(off, hp[i], dy2, ndy2, dw);
        store_e<3>(off, hp[i], dy2, ndy2, dw);
        store_e<4>(off, hp[i], dy2, ndy2, dw);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      if (nt == RES_NWG && wg == 0) {
        if (warp == 0) issue_backward(0, nt, 128);
        else named_arrive(RES_BAR_E, 128);
      } else {
        named_arrive(RES_BAR_E + wg, 160);
      }
      // dW1 of the warp's 32 rows (over the eight quads) while the MMAs run: units 8n + 2c + e
      float v[10];
#pragma unroll
      for (int n = 0; n < 5; ++n) unpack2(dw[n], v[2 * n], v[2 * n + 1]);
      const bool q2 = (lane & 16) != 0, q1 = (lane & 8) != 0;
#pragma unroll
      for (int n = 0; n < 5; ++n) {  // lanes with bit 4 keep e = 1, the others e = 0
        const float send = q2 ? v[2 * n] : v[2 * n + 1];
        v[n] = (q2 ? v[2 * n + 1] : v[2 * n]) + __shfl_xor_sync(0xffffffffu, send, 16);
      }
      {  // bit 3: n = 3, 4 or n = 0, 1, 2
        const float s0 = q1 ? v[0] : v[3], s1 = q1 ? v[1] : v[4], s2 = v[2];
        const float r0 = __shfl_xor_sync(0xffffffffu, s0, 8), r1 = __shfl_xor_sync(0xffffffffu, s1, 8);
        const float r2 = __shfl_xor_sync(0xffffffffu, s2, 8);
        v[0] = (q1 ? v[3] : v[0]) + r0;
        v[1] = (q1 ? v[4] : v[1]) + r1;
        v[2] = v[2] + r2;
      }
#pragma unroll
      for (int n = 0; n < 3; ++n) v[n] += __shfl_xor_sync(0xffffffffu, v[n], 4);
      float* rw1 = reinterpret_cast<float*>(base + RW1) + warp * RS + 2 * (lane & 3) + (q2 ? 1 : 0);
      if ((lane & 4) == 0) {
        rw1[q1 ? 24 : 0] = v[0];
        rw1[q1 ? 32 : 8] = v[1];
        if (!q1) rw1[16] = v[2];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dy_row += __shfl_xor_sync(0xffffffffu, dy_row, o);
      if (lane == 0) reinterpret_cast<float*>(base + RW1)[warp * RS + H] = dy_row;
      if (last) {
        double ld = (double)loss;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, o);
        if (lane == 0) reinterpret_cast<double*>(base + RLL)[warp] = ld;
      }
    } else {
      if (next_active) named_arrive(RES_BAR_T + wg + 1, 256);
      tc_fence_before();
      named_arrive(RES_BAR_E + wg, 160);
    }
    const uint32_t ph = par;
    par ^= 1;
    if (wg != 0) return;
    if (nt == RES_NWG && warp == 0)
      for (int w = 1; w < nt; ++w) issue_backward(w, nt, 160);
    // ---- the first warpgroup reads the accumulator out ----
    res_wait(bar_bwd(), ph, g, g.wait_ticks << 2, 613, ok);
    tc_fence_after();
    // accumulator row i = 32 * group + feature lives in lane 32 * (i / 16) + i % 16 (M = 64)
    {
      const int w = warp & 3, grp = w >> 1, k = (w & 1) * 16 + lane;
      float acc[H];
      tc_ld32(tmem + G_COL0 + lanes + grp * H, acc);
      tc_ld8(tmem + G_COL0 + lanes + grp * H + 32, acc + 32);
      tc_wait_ld();
      tc_fence_before();
      if (lane < 16 && k <= COL_ONE) {
        float* dst = reinterpret_cast<float*>(base + GP) + grp * GPART + k * H;
#pragma unroll
        for (int c = 0; c < H; c += 4)
          *reinterpret_cast<float4*>(dst + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
      }
    }
  }

  __device__ __forceinline__ void issue_forward(int nt) {
    constexpr uint32_t IDESC_FWD = umma_idesc_tf32(128, NF, 0, 0);
    const uint32_t on = elect_one();
    tc_fence_after();
    const uint64_t wdesc = umma_desc_k128(smem_u32(base + W0S));
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
#pragma unroll
    for (int w = 0; w < RES_NWG; ++w) {
      const uint32_t go = w < nt ? on : 0u;
#pragma unroll
      for (int kb = 0; kb < 3; ++kb)
        tc_mma_tf32_ts_if(tm + Z_COL0 + w * Z_STRIDE, tm + A_COL0 + w * A_STRIDE + kb * 8,
                          umma_desc_advance(wdesc, kb * 2), IDESC_FWD, kb > 0, go);
      tc_commit_if(bar(w, 1), go);
    }
  }
  // backward of tile w once its E is in shared memory (`count`: threads at the barrier, this warp included)
  __device__ __forceinline__ void issue_backward(int w, int nt, int count) {
    constexpr uint32_t IDESC_BWD = umma_idesc_tf32(GM, GN, 1, 0);
    named_sync(RES_BAR_E + w, count);
    tc_fence_after();
    const uint32_t on = elect_one();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t edesc = umma_desc_k128(smem_u32(base + ES + w * ES_WG_BYTES));
    const uint64_t xdesc = umma_desc_mn32(smem_u32(base + XB + w * TILE_BYTES), GROUP_BYTES);
    const uint32_t on2 = n_units - 4 * w > 2 ? on : 0u;  // a tile's second 64 rows only if there are any
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int p = q >> 2, kb = q & 3;
      tc_mma_tf32_ss_if(tm + G_COL0, umma_desc_advance(xdesc, p * (2 * GROUP_BYTES >> 4) + kb * 64),
                        umma_desc_advance(edesc, p * (2 * ES_ATOM_BYTES >> 4) + kb * 2), IDESC_BWD,
                        (w > 0 || q > 0) ? 1u : 0u, p ? on2 : on);
    }
    tc_commit_if(bar_bwd(), w == nt - 1 ? on : 0u);
  }
  // units 8N + 2c and 8N + 2c + 1 of one row
  template <int N>
  __device__ __forceinline__ void store_e(uint32_t off, const uint64_t* hp, uint64_t dy2, uint64_t ndy2, uint64_t* dw) {
    const uint64_t t2 = mul2(dy2, hp[N]);
    dw[N] = fma2(dy2, hp[N], dw[N]);
    float e0, e1;
    unpack2(fma2(t2, hp[N], ndy2), e0, e1);
    // the odd unit: next line, chunk ^ 1
    asm volatile("st.shared.f32 [%0+%2], %1;" ::"r"(off), "f"(e0), "n"(8 * N * 128) : "memory");
    asm volatile("st.shared.f32 [%0+%2], %1;" ::"r"(off ^ 16u), "f"(e1), "n"((8 * N + 1) * 128) : "memory");
  }

  // Words of W0 and b0 go to the threads of the same number; those of W1 and b1, which add over warps instead of row
  // groups, and the log-likelihood to the last warp
  static constexpr int LAST = RES_NWG * 4 - 1, NW1 = Words::N - 1 - Words::W0;  // 14 words of W1 and b1
  static_assert(NW1 < 32 && Words::W0 <= LAST * 32, "word assignment");
  __device__ __forceinline__ int collects() const {
    if (warp == LAST) return lane <= NW1 ? Words::W0 + lane : -1;
    return (int)threadIdx.x < Words::W0 ? (int)threadIdx.x : -1;
  }
  // this CTA's sums for its word (after the CTA barrier that follows step)
  __device__ __forceinline__ bool collect(bool last, uint4& v) const {
    if (warp == LAST) {
      const float* r = reinterpret_cast<const float*>(base + RW1) + 3 * min(lane, NW1 - 1);
      float s[3][2] = {};
#pragma unroll
      for (int w = 0; w < RES_NWG * 4; ++w)
#pragma unroll
        for (int q = 0; q < 3; ++q) s[q][w & 1] += r[w * RS + q];
      v = make_uint4(__float_as_uint(s[0][0] + s[0][1]), __float_as_uint(s[1][0] + s[1][1]),
                     __float_as_uint(s[2][0] + s[2][1]), 0u);
      if (last && lane == NW1) {
        const double* d = reinterpret_cast<const double*>(base + RLL);
        double t[2] = {};
#pragma unroll
        for (int w = 0; w < RES_NWG * 4; ++w) t[w & 1] += d[w];
        const uint2 u = d2u(t[0] + t[1]);
        v.x = u.x;
        v.y = u.y;
      }
      return lane <= NW1;
    }
    const int t = threadIdx.x;
    const float* gp = reinterpret_cast<const float*>(base + GP) + 3 * min(t, Words::W0 - 1);
    const float* nw = w1s() + NEG + (3 * min(t, Words::W0 - 1)) % H;  // E was stored negated and without its W1 factor
    v = make_uint4(__float_as_uint(nw[0] * (gp[0] + gp[GPART])), __float_as_uint(nw[1] * (gp[1] + gp[GPART + 1])),
                   __float_as_uint(nw[2] * (gp[2] + gp[GPART + 2])), 0u);
    return t < Words::W0;
  }

  __device__ __forceinline__ void teardown(const ResidentParams& g, const volatile int& dead) {
    tc_fence_before();
    __syncthreads();
    if (warp == 0 && dead) {
      for (int w = 0; 4 * w < n_units; ++w) res_drain(bar(w, 1), par ^ 1, g);
      if (n_units > 0) res_drain(bar_bwd(), par ^ 1, g);
    }
    if (warp == 0)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS)
                   : "memory");
  }
};

cudaError_t launch_resident_tf32(int cluster, const void* tmap, const ResidentParams& g, cudaStream_t st,
                                 int* max_clusters) {
  return resident_launch_any<ResTf32>(cluster, tmap, g, st, max_clusters);
}

cudaError_t launch_resident_eval_tf32(const void* tmap, const ResidentEvalParams& g, cudaStream_t st) {
  return resident_launch_single<ResTf32>(tmap, g, st);
}

}  // namespace mcmc_b200
