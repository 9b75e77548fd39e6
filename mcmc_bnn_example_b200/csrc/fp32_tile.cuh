// FP32 (FFMA) arithmetic of a block of rows, by one warp on its own: forward, output layer, loss, dL/dz through the
// warp's own shared memory, backward.  A warp never waits for another: the warps of a scheduler drift apart, and one's tanh pass
// (MUFU) runs beside another's multiplications.  For 128 units, and for 40 in large batches of small windows (grad_fp32.cu).
//
// Layouts.  What bounds the multiplications is feeding them: a 16-byte load of a whole warp takes four passes over
// shared memory, but two when lanes i and i ^ 1 (or i and i ^ 2) read the same address, measured; the same address in
// lanes 8 apart does not help.  So lane bits 0 and 1 go to different operands in both products:
//   * forward: a lane owns HALF rows x HPL hidden units at a time.  Features go in pairs, one packed FMA for two of them
//     (sums over the even and the odd features, added at the end): rows are read as they lie, weights are staged in
//     pairs.  Packed FMAs with three different operands issue every third cycle, so they save issue slots and not FMA
//     time; single ones took the same time for 40 units and 10 % more for 128.
//     Row group = lane bits 0, 2 (bit 0 for 128 units), unit group = the other bits.
//   * backward: a lane owns 12 features x HPL units of every second row (every row for 128 units): feature half =
//     bit 0, unit group = the next bits.  W1's factor of dL/dz is left to whoever reads the sums out.
// Forward and dL/dz take half of a block's rows at a time: a lane then holds 4 x HPL packed sums, not 8 x HPL.
#pragma once
#include "common.cuh"

namespace mcmc_b200 {

__device__ __forceinline__ void lds2x64(const float* p, uint64_t& a, uint64_t& b) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  a = v.x;
  b = v.y;
}

template <int H>
struct Fp32Warp {
  static constexpr int D = 22, P = D * H + 2 * H + 1;
  static constexpr int HPL = H == 40 ? 5 : 8;
  static constexpr int CG = H / HPL;            // unit groups
  static constexpr int RG = 32 / CG;            // forward: row groups
  static constexpr int HALF = 4;                // forward: rows per lane at a time
  static constexpr int HROWS = RG * HALF;       // ... and of the warp
  static constexpr int ROWS = 2 * HROWS;        // rows of a block
  static constexpr int RSUB = RG / 2;           // backward: row subsets
  static constexpr int KPT = 12;                // backward: features per lane
  static constexpr int ES = ROWS * H;           // floats of dL/dz
  static constexpr int WP = D / 2 * 2 * H;      // floats of the staged feature pairs
  static_assert(H == 40 || H == 128, "unit groups of 5 or 8");

  // staged weight of feature k and unit j: [pair of features][vectors of two units][group][unit][feature]
  __host__ __device__ static constexpr int w_off(int k, int j) {
    const int cg = j / HPL, u = j % HPL;
    return (k / 2) * (2 * H) + (u < HPL / 2 * 2 ? (u / 2) * (CG * 4) + cg * 4 + (u & 1) * 2
                                                : (HPL / 2) * (CG * 4) + cg * 2) + (k & 1);
  }

  static constexpr int M1 = H == 40 ? 8 : 4;    // lane bit of the second unit-group bit (the first is 2)

  int lane, cg, rg;        // forward
  int bcg, kh, rsub;       // backward
  int own;                 // the row of a half whose dL/dpred this lane computes (lanes 16 apart the same one)
  __device__ __forceinline__ Fp32Warp() {
    lane = threadIdx.x & 31;
    if (H == 40) {
      rg = (lane & 1) | ((lane >> 1) & 2);
      cg = ((lane >> 1) & 1) | ((lane >> 2) & 6);
    } else {
      rg = lane & 1;
      cg = lane >> 1;
    }
    own = ((lane & 2) | (lane & M1 ? 1 : 0)) * RG + rg;
    kh = lane & 1;
    bcg = (lane >> 1) & (CG - 1);
    rsub = RSUB == 1 ? 0 : lane >> 4;
  }

  // tanh(x W0 + b0) of this lane's rows of half hf, two rows to a pair; xb: the block's rows
  __device__ __forceinline__ void hidden(const float* xb, const float* wp, const float* b0, int hf,
                                         uint64_t (*hp)[HPL]) const {
    uint64_t z[HALF][HPL];
#pragma unroll
    for (int j = 0; j < HPL; ++j) {
      const uint64_t b = pack2(b0[cg * HPL + j], 0.f);
#pragma unroll
      for (int i = 0; i < HALF; ++i) z[i][j] = b;
    }
#pragma unroll
    for (int k4 = 0; k4 < (D + 3) / 4; ++k4) {
      uint64_t x[HALF][2];
#pragma unroll
      for (int i = 0; i < HALF; ++i) lds2x64(xb + (hf * HROWS + i * RG + rg) * KP + 4 * k4, x[i][0], x[i][1]);
#pragma unroll
      for (int k2 = 0; k2 < 2; ++k2) {
        if (4 * k4 + 2 * k2 >= D) continue;
        uint64_t w[HPL];
        const float* p = wp + (2 * k4 + k2) * (2 * H);
#pragma unroll
        for (int q = 0; q < HPL / 2; ++q) lds2x64(p + q * (CG * 4) + cg * 4, w[2 * q], w[2 * q + 1]);
        if (HPL & 1) w[HPL - 1] = *reinterpret_cast<const uint64_t*>(p + (HPL / 2) * (CG * 4) + cg * 2);
#pragma unroll
        for (int i = 0; i < HALF; ++i)
#pragma unroll
          for (int j = 0; j < HPL; ++j) z[i][j] = fma2(x[i][k2], w[j], z[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < HALF; i += 2)
#pragma unroll
      for (int j = 0; j < HPL; ++j) {
        float a, b, c, d;
        unpack2(z[i][j], a, b);
        unpack2(z[i + 1][j], c, d);
        hp[i / 2][j] = pack2(tanh_ref(a + b), tanh_ref(c + d));
      }
  }

  // Adds up the unit groups' shares of a half's predictions: a lane gets the one of its own row
  __device__ __forceinline__ float predict(const uint64_t (*hp)[HPL], const float* w1) const {
    float pr[HALF];
    uint64_t acc[2] = {};
#pragma unroll
    for (int j = 0; j < HPL; ++j) {
      const float w = w1[cg * HPL + j];
      const uint64_t w2 = pack2(w, w);
      acc[0] = fma2(w2, hp[0][j], acc[0]);
      acc[1] = fma2(w2, hp[1][j], acc[1]);
    }
    unpack2(acc[0], pr[0], pr[1]);
    unpack2(acc[1], pr[2], pr[3]);
    const bool up = (lane & 2) != 0, odd = (lane & M1) != 0;
    const float s0 = up ? pr[0] : pr[2], s1 = up ? pr[1] : pr[3];
    const float k0 = (up ? pr[2] : pr[0]) + __shfl_xor_sync(0xffffffffu, s0, 2);
    const float k1 = (up ? pr[3] : pr[1]) + __shfl_xor_sync(0xffffffffu, s1, 2);
    const float s = odd ? k0 : k1;
    float p = (odd ? k1 : k0) + __shfl_xor_sync(0xffffffffu, s, M1);
    if (CG == 16) p += __shfl_xor_sync(0xffffffffu, p, 8);
    return p + __shfl_xor_sync(0xffffffffu, p, 16);
  }

  // dL/dz of half hf without W1's factor to `es`; adds the lane's rows to dW1.  dys: ROWS floats of the warp's own
  __device__ __forceinline__ void elementwise(const uint64_t (*hp)[HPL], float dy_row, int hf, float* dys, float* es,
                                              uint64_t* dw1) const {
    dys += hf * HROWS;
    dys[(own % RG) * HALF + own / RG] = dy_row;   // (lanes with the same row write the same)
    __syncwarp();
    uint64_t dy[2];
    lds2x64(dys + rg * HALF, dy[0], dy[1]);
    const uint64_t minus1 = pack2(-1.f, -1.f), sign = 0x8000000080000000ull;
    const uint64_t ndy[2] = {dy[0] ^ sign, dy[1] ^ sign};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float e[2][HPL];
#pragma unroll
      for (int j = 0; j < HPL; ++j) {
        dw1[j] = fma2(dy[i], hp[i][j], dw1[j]);
        const uint64_t d = mul2(fma2(hp[i][j], hp[i][j], minus1), ndy[i]);  // tanh_t::bwd
        unpack2(d, e[0][j], e[1][j]);
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float* p = es + (hf * HROWS + (2 * i + r) * RG + rg) * H;
#pragma unroll
        for (int q = 0; q < HPL / 4; ++q)
          *reinterpret_cast<float4*>(p + q * (CG * 4) + cg * 4) =
              make_float4(e[r][4 * q], e[r][4 * q + 1], e[r][4 * q + 2], e[r][4 * q + 3]);
        if (HPL % 4) p[HPL / 4 * (CG * 4) + cg] = e[r][HPL - 1];
      }
    }
  }

  // Everything of a block up to dL/dz.  The lane's own row of half hf is block row hf HROWS + own; its loss is computed
  // in the lanes whose bit 4 is hf.  Returns the sum of the lane's two dL/dpred (each is in lanes 16 apart as well).
  template <bool LOSS>
  __device__ __forceinline__ void block(const float* xb, const float* wp, const float* b0, const float* w1, float b1,
                                        const LikParams& lik, int rows_left, float* dys, float* es, uint64_t* dw1,
                                        float& dy_sum, float& loss) const {
    float y_own = 0.f, pred_own = 0.f;
#pragma unroll(H == 40 ? 2 : 1)
    for (int hf = 0; hf < 2; ++hf) {
      uint64_t hp[2][HPL];
      hidden(xb, wp, b0, hf, hp);
      const float pred = predict(hp, w1) + b1;
      const float y = xb[(hf * HROWS + own) * KP + COL_Y];
      const float dy = hf * HROWS + own < rows_left ? lik_grad(lik, y, pred) : 0.f;
      if (LOSS && (lane >> 4) == hf) {
        y_own = y;
        pred_own = pred;
      }
      dy_sum += dy;
      elementwise(hp, dy, hf, dys, es, dw1);
    }
    __syncwarp();
    if (LOSS) loss = loss_row() < rows_left ? lik_loss(lik, y_own, pred_own) : 0.f;
  }
  // the block row of `loss`; for 128 units lanes 8 apart have the same one
  __device__ __forceinline__ int loss_row() const { return (lane >> 4) * HROWS + own; }
  __device__ __forceinline__ bool loss_first() const { return H == 40 || (lane & 8) == 0; }

  // acc[k][j] += features 12 kh + 2 k, + 1 of the rows x dL/dz (feature 22 is the constant 1: db0; 23 is y, unused)
  template <int UNROLL>
  __device__ __forceinline__ void backward(const float* xb, const float* es, uint64_t (*acc)[HPL]) const {
#pragma unroll UNROLL
    for (int s = 0; s < ROWS / RSUB; ++s) {
      const int row = s * RSUB + rsub;
      const float* xr = xb + row * KP + kh * KPT;
      uint64_t x[KPT / 2];
#pragma unroll
      for (int q = 0; q < KPT / 4; ++q) lds2x64(xr + 4 * q, x[2 * q], x[2 * q + 1]);
      const float* p = es + row * H;
      float e[HPL];
#pragma unroll
      for (int q = 0; q < HPL / 4; ++q) {
        const float4 t = *reinterpret_cast<const float4*>(p + q * (CG * 4) + bcg * 4);
        e[4 * q] = t.x;
        e[4 * q + 1] = t.y;
        e[4 * q + 2] = t.z;
        e[4 * q + 3] = t.w;
      }
      if (HPL % 4) e[HPL - 1] = p[HPL / 4 * (CG * 4) + bcg];
#pragma unroll
      for (int j = 0; j < HPL; ++j) {
        const uint64_t e2 = pack2(e[j], e[j]);
#pragma unroll
        for (int k = 0; k < KPT / 2; ++k) acc[k][j] = fma2(x[k], e2, acc[k][j]);
      }
    }
  }
};

}  // namespace mcmc_b200
