// FP32 arithmetic of a warp's 32 rows for 40 hidden units, behind the forward product on the tensor core (split_mma.cuh):
// z out of tensor memory, output layer, loss, dL/dz; and the backward pass by FFMA, or integers for it (int_mma.cuh).  No warp waits
// for another inside it.
//
// Layouts.  z is read in the 16-lane quad shape: quad q = lane / 4 holds rows q, q + 8, q + 16, q + 24, its lane c units
// 8 n + 2 c and the next one (n < 5).  A row's output is then a sum over four lanes, dW1 ten sums per lane.  dL/dz goes to
// es[row][unit], eight bytes a store, free of bank conflicts (rows are 40 floats apart: 8 q + 2 c).
// Backward: a lane owns 12 features x 5 units of every second row.  What bounds it is feeding the multiplications: a 16-byte load
// of a whole warp takes four passes over shared memory, but two when neighbouring lanes read the same address; so the
// feature half is lane bit 0, and the unit group the next three bits: units 4 b .. 4 b + 3 and 32 + b.  Features go in pairs through
// packed FMAs (their common factor, dL/dz, is one value for both: 2.3 cycles a packed FMA instead of 2.8).
// W1's factor of dL/dz is left to whoever reads the sums out.
#pragma once
#include "int_mma.cuh"

namespace mcmc_b200 {

struct SplitWarp {
  static constexpr int H = SPLIT_H, D = SPLIT_D, P = D * H + 2 * H + 1;
  static constexpr int ROWS = 32, ES = ROWS * H;
  static constexpr int KPT = 12, UPT = 5;   // backward: features and units per lane

  int lane, q, c;          // forward
  int bcg, kh, rsub;       // backward
  __device__ __forceinline__ SplitWarp() {
    lane = threadIdx.x & 31;
    q = lane >> 2;
    c = lane & 3;
    kh = lane & 1;
    bcg = (lane >> 1) & 7;
    rsub = lane >> 4;
  }
  __device__ __forceinline__ int own() const { return q + 8 * c; }  // the row whose dL/dpred this lane computes
  __device__ __forceinline__ int owner() const { return 4 * (lane & 7) + (lane >> 3); }  // the lane that has row `lane`'s

  static __device__ __forceinline__ uint64_t lds64(const float* p) { return *reinterpret_cast<const uint64_t*>(p); }

  // z of rows and units as the quads hold them, from tensor memory (z_t with the warp's lanes)
  __device__ __forceinline__ void load(uint32_t z_t, uint64_t (&z)[4][5]) const {
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const uint32_t t = z_t + ((uint32_t)(hf * 16) << 16);
      float s1[16], s0[16];
      tc_ld_quad32(t, s1);
      tc_ld_quad32(t + SPLIT_S0, s0);
      tc_wait_ld();
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          z[2 * hf + i][n] = add2(pack2(s0[4 * n + 2 * i], s0[4 * n + 2 * i + 1]), pack2(s1[4 * n + 2 * i], s1[4 * n + 2 * i + 1]));
    }
    float s1[2][4], s0[2][4];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const uint32_t t = z_t + ((uint32_t)(hf * 16) << 16) + 32;
      tc_ld_quad8(t, s1[hf]);
      tc_ld_quad8(t + SPLIT_S0, s0[hf]);
    }
    tc_wait_ld();
#pragma unroll
    for (int hf = 0; hf < 2; ++hf)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        z[2 * hf + i][4] = add2(pack2(s0[hf][2 * i], s0[hf][2 * i + 1]), pack2(s1[hf][2 * i], s1[hf][2 * i + 1]));
  }
  // the same by FFMA, for values that split_wide finds: the lane's row, through es.  A weight is the sum of its parts
  // (split_store_weight).  Even and odd features apart, added at the end.  UNITS side by side, four features' weights a load (58368 rows on the
  // chip, Cauchy features: 31.5 us a step, 151 with a weight at a time); what registers more would need, a caller's loop loses
  template <int UNITS>
  static __device__ __noinline__ void plain(const float* xb, const unsigned char* b, float* es) {
    static_assert(D == 22 && KP == 24, "the bias is the third of the last four");
    const int lane = threadIdx.x & 31;
    const float4* x = reinterpret_cast<const float4*>(xb + lane * KP);
    auto weights = [&](int j, int c) {
      const float4* p = reinterpret_cast<const float4*>(b + split_b_off(j, 4 * c));
      const float4 hi = p[0], mid = p[SPLIT_B_PART / 16], lo = p[2 * (SPLIT_B_PART / 16)];
      return make_float4(hi.x + (mid.x + lo.x), hi.y + (mid.y + lo.y), hi.z + (mid.z + lo.z), hi.w + (mid.w + lo.w));
    };
#pragma unroll 1
    for (int j = 0; j < H; j += UNITS) {
      float even[UNITS], odd[UNITS];
#pragma unroll
      for (int u = 0; u < UNITS; ++u) {
        even[u] = weights(j + u, KP / 4 - 1).z;  // the bias first
        odd[u] = 0.f;
      }
#pragma unroll
      for (int c = 0; c < KP / 4; ++c) {
        const float4 v = x[c];
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
          const float4 w = weights(j + u, c);
          even[u] = fmaf(v.x, w.x, even[u]);
          odd[u] = fmaf(v.y, w.y, odd[u]);
          if (c < KP / 4 - 1) {
            even[u] = fmaf(v.z, w.z, even[u]);
            odd[u] = fmaf(v.w, w.w, odd[u]);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < UNITS; ++u) es[lane * H + j + u] = even[u] + odd[u];
    }
    __syncwarp();
  }

  __device__ __forceinline__ void load_plain(const float* es, uint64_t (&z)[4][5]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int n = 0; n < 5; ++n) z[i][n] = lds64(es + (q + 8 * i) * H + 8 * n + 2 * c);
  }

  // Output layer and loss: h in place of z, d[i] = dL/dpred of row q + 8 i.  `valid`, y, dy and pred are those of the lane's own row.
  // turn(i): called when the tanh of the i-th of a quad's four rows are under way
  template <class Turn>
  __device__ __forceinline__ void front(uint64_t (&h)[4][5], const float* w1, const LikParams& lik, float y, bool valid,
                                        float (&d)[4], float& dy, float& pred, Turn turn) const {
    float pr[4];
    {
      uint64_t w1p[5];
#pragma unroll
      for (int n = 0; n < 5; ++n) w1p[n] = lds64(w1 + 8 * n + 2 * c);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint64_t acc = 0ull;
#pragma unroll
        for (int n = 0; n < 5; ++n) {
          h[i][n] = tanh_ref2(h[i][n]);
          acc = fma2(w1p[n], h[i][n], acc);
        }
        float a, b;
        unpack2(acc, a, b);
        pr[i] = a + b;
        turn(i);
      }
    }
    // the quad's four lanes add up; lane c keeps row q + 8 c
    const bool b1 = (lane & 2) != 0, b0 = (lane & 1) != 0;
    const float s0 = b1 ? pr[0] : pr[2], s1 = b1 ? pr[1] : pr[3];
    const float k0 = (b1 ? pr[2] : pr[0]) + __shfl_xor_sync(0xffffffffu, s0, 2);
    const float k1 = (b1 ? pr[3] : pr[1]) + __shfl_xor_sync(0xffffffffu, s1, 2);
    const float s = b0 ? k0 : k1;
    pred = (b0 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, s, 1) + w1[H];
    dy = valid ? lik_grad(lik, y, pred) : 0.f;
    // every lane of the quad needs the four dL/dpred
    {
      const float o1 = __shfl_xor_sync(0xffffffffu, dy, 1);
      const float a0 = b0 ? o1 : dy, a1 = b0 ? dy : o1;
      const float c0 = __shfl_xor_sync(0xffffffffu, a0, 2), c1 = __shfl_xor_sync(0xffffffffu, a1, 2);
      d[0] = b1 ? c0 : a0;
      d[1] = b1 ? c1 : a1;
      d[2] = b1 ? a0 : c0;
      d[3] = b1 ? a1 : c1;
    }
  }
  // dL/dz without W1's factor to es, the lane's rows added to dw (units 8 n + 2 c, + 1)
  __device__ __forceinline__ void store_es(const uint64_t (&h)[4][5], const float (&d)[4], float* es, uint64_t (&dw)[5]) const {
    const uint64_t minus1 = pack2(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint64_t d2 = pack2(d[i], d[i]), nd2 = pack2(-d[i], -d[i]);
      float* p = es + (q + 8 * i) * H + 2 * c;
#pragma unroll
      for (int n = 0; n < 5; ++n) {
        dw[n] = fma2(d2, h[i][n], dw[n]);
        *reinterpret_cast<uint64_t*>(p + 8 * n) = mul2(fma2(h[i][n], h[i][n], minus1), nd2);  // tanh_t::bwd
      }
    }
    __syncwarp();
  }
  // the same as integers, d times `scale`, to the warp's INT_E_WARP bytes (int_mma.cuh).  WITH_D false: without d's factor
  template <bool WITH_D = true>
  __device__ __forceinline__ void store_ei(const uint64_t (&h)[4][5], const float (&d)[4], float scale, float* ei,
                                           uint64_t (&dw)[5]) const {
    const uint64_t minus1 = pack2(-1.f, -1.f);
    uint32_t* const dst = reinterpret_cast<uint32_t*>(ei) + (c >> 1) * 32 + q * 4 + (c & 1) * 2;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float nd = WITH_D ? -d[i] * scale : -scale;
      const uint64_t d2 = pack2(d[i], d[i]), nd2 = pack2(nd, nd);
#pragma unroll
      for (int n = 0; n < 5; ++n) {
        dw[n] = fma2(d2, h[i][n], dw[n]);
        *reinterpret_cast<uint2*>(dst + i * (2 * INT_E_ROW) + n * 64) = int_digits2(fma2(h[i][n], h[i][n], minus1), nd2);
      }
    }
  }
  template <class Turn>
  __device__ __forceinline__ void block(uint64_t (&h)[4][5], const float* w1, const LikParams& lik, float y, bool valid,
                                        float* es, uint64_t (&dw)[5], float& dy, float& pred, Turn turn) const {
    float d[4];
    front(h, w1, lik, y, valid, d, dy, pred, turn);
    store_es(h, d, es, dw);
  }

  // Sums of dw over the eight quads to out[unit], on an 8-byte boundary.  (All lanes make all sums: halving what a lane keeps takes fewer shuffles, but
  // three times the code)
  __device__ __forceinline__ void store_dw1(uint64_t (&dw)[5], float* out) const {
#pragma unroll
    for (int o = 16; o > 2; o >>= 1)
#pragma unroll
      for (int n = 0; n < 5; ++n) dw[n] = add2(dw[n], __shfl_xor_sync(0xffffffffu, dw[n], o));
    if (q == 0)
#pragma unroll
      for (int n = 0; n < 5; ++n) *reinterpret_cast<uint64_t*>(out + 8 * n + 2 * c) = dw[n];
  }

  // Sums of acc over the two row subsets, lanes 16 apart: the lower lane keeps features 0 - 5 of its twelve, the upper one 6 - 11.
  // out: where feature 12 kh + 6 rsub of unit 0 goes, features H apart
  __device__ __forceinline__ void store_dw0(const uint64_t (*acc)[UPT], float* out) const {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float o[2][UPT];
#pragma unroll
      for (int j = 0; j < UPT; ++j) {
        const uint64_t send = rsub ? acc[k][j] : acc[k + 3][j], keep = rsub ? acc[k + 3][j] : acc[k][j];
        unpack2(add2(keep, __shfl_xor_sync(0xffffffffu, send, 16)), o[0][j], o[1][j]);
      }
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        float* p = out + (2 * k + f) * H;
        *reinterpret_cast<float4*>(p + 4 * bcg) = make_float4(o[f][0], o[f][1], o[f][2], o[f][3]);
        p[32 + bcg] = o[f][4];
      }
    }
  }

  // acc[k][u] += features 12 kh + 2 k, + 1 of the rows x dL/dz (feature 22 is the constant 1: db0; 23 is y, unused)
  template <int UNROLL>
  __device__ __forceinline__ void backward(const float* xb, const float* es, uint64_t (*acc)[UPT]) const {
#pragma unroll UNROLL
    for (int s = 0; s < ROWS / 2; ++s) {
      const int row = 2 * s + rsub;
      const float* xr = xb + row * KP + kh * KPT;
      uint64_t x[KPT / 2];
#pragma unroll
      for (int k = 0; k < KPT / 4; ++k) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(xr + 4 * k);
        x[2 * k] = v.x;
        x[2 * k + 1] = v.y;
      }
      const float4 e4 = *reinterpret_cast<const float4*>(es + row * H + 4 * bcg);
      const float e[UPT] = {e4.x, e4.y, e4.z, e4.w, es[row * H + 32 + bcg]};
#pragma unroll
      for (int u = 0; u < UPT; ++u) {
        const uint64_t e2 = pack2(e[u], e[u]);
#pragma unroll
        for (int k = 0; k < KPT / 2; ++k) acc[k][u] = fma2(x[k], e2, acc[k][u]);
      }
    }
  }

  // backward and store_dw0 out of line, PAIRS pairs of features after others and acc in memory: what registers a call needs are lost to its
  // caller's loop (streaming, 16 windows of 40013 rows: 49.0 us a step with all six pairs at once, 47.3 with one)
  static constexpr int LEAN = KPT / 2 * UPT;
  template <int PAIRS>
  static __device__ __noinline__ void backward_lean(const float* xb, const float* es, uint64_t* acc) {
    const SplitWarp lanes;
#pragma unroll 1
    for (int k = 0; k < KPT / 2; k += PAIRS) {
      uint64_t a[PAIRS][UPT];
#pragma unroll
      for (int i = 0; i < PAIRS * UPT; ++i) a[i / UPT][i % UPT] = acc[k * UPT + i];
#pragma unroll 2
      for (int s = 0; s < ROWS / 2; ++s) {
        const int row = 2 * s + lanes.rsub;
        uint64_t x[PAIRS];
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) x[i] = lds64(xb + row * KP + lanes.kh * KPT + 2 * (k + i));
        const float4 e4 = *reinterpret_cast<const float4*>(es + row * H + 4 * lanes.bcg);
        const float e[UPT] = {e4.x, e4.y, e4.z, e4.w, es[row * H + 32 + lanes.bcg]};
#pragma unroll
        for (int u = 0; u < UPT; ++u)
#pragma unroll
          for (int i = 0; i < PAIRS; ++i) a[i][u] = fma2(x[i], pack2(e[u], e[u]), a[i][u]);
      }
#pragma unroll
      for (int i = 0; i < PAIRS * UPT; ++i) acc[k * UPT + i] = a[i / UPT][i % UPT];
    }
    __syncwarp();
  }
  static __device__ __noinline__ void store_dw0_lean(const uint64_t* acc, float* out) {
    const SplitWarp lanes;
#pragma unroll 1
    for (int k = 0; k < 3; ++k)
#pragma unroll 1
      for (int u = 0; u < UPT; ++u) {
        const uint64_t lo = acc[k * UPT + u], hi = acc[(k + 3) * UPT + u];
        float a, b;
        unpack2(add2(lanes.rsub ? hi : lo, __shfl_xor_sync(0xffffffffu, lanes.rsub ? lo : hi, 16)), a, b);
        const int unit = u < 4 ? 4 * lanes.bcg + u : 32 + lanes.bcg;
        out[2 * k * H + unit] = a;
        out[(2 * k + 1) * H + unit] = b;
      }
  }
};

}  // namespace mcmc_b200
