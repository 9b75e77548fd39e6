// FP32 product of rows and first-layer weights (24 features x 40 units) on the tensor core.
//
// The FFMA kernels' forward product keeps the FMA pipe busy for as long as everything else together; the tensor core
// does it beside them.  It takes TF32 operands and truncates its sums, so:
//   * every operand is the sum of three parts: a high one of SPLIT_X_BITS (rows) or SPLIT_W_BITS (weights) significant
//     bits, a middle one of 11 bits and the rest (at most 8): together all 24 bits of the float, whatever its exponent;
//   * the products of the high parts have 11 bits, so their sum over 24 features is exact for 99 % of the elements; it gets an
//     accumulator of its own, S0.  Everything else but rest x rest, 2^-5 of it, goes into a second one, S1, whose truncation is then
//     2^-5 of an ulp;
//   * z = S0 + S1 is one rounded FP32 addition.
// Measured on a B200 against 64 bits, N(0,1) rows x small weights: rms error 2.6e-8 of z's rms, for no unit more than
// 3.3e-8, mean error -7e-10 of |z| (a chain of 23 FMAs: 8.8e-8, 1.0e-7 and 0; even and odd features apart, as the gradient kernels
// without the tensor core add them: 6.9e-8); the same with features of very different scales.  With one, two or five features that are not zero
// 2.5e-8 (FMAs 2.5e-8, 3.1e-8, 4.5e-8), the largest error 6.2e-8 of the one term (5.9e-8).  Without middle x rest and rest x middle, 18
// MMAs: 4.4e-8 for all features, but 4.2e-8 for one, the largest 2.6e-7 of it.
// Gradients, losses and row losses are as far from 64 bits as with FFMA (0.99, 1.00 and 0.98 of the error): the tanh sets that.
// With plain halves of 11 bits and one accumulator the truncation's mean is 7e-8 of |z| in every row alike, and a gradient
// 7.5e-7 off instead of 6e-8: that is why the parts are cut like this.  High parts of 6 and 6 bits: mean -1.2e-9 to -1.9e-9;
// three bf16 parts and two thirds of the MMAs: mean -6e-9, gradients 1.1 to 2.8 times as far off.
// An MMA of 128 x 48 x 8 takes 24 to 29 cycles of a string of them, and 90 pass until the last result.
// Predictions and mean losses cut otherwise (forward.cu).
//
// Parts of infinities are not numbers, and products near the largest float overflow in one part and not in the other.  So
// values from 2^60 on, infinities and NaN (split_wide) take plain FFMA (SplitWarp::plain, fws_plain): then sums, signs and NaN
// are as before.
#pragma once
#include "chain.cuh"
#include "tc05.cuh"

namespace mcmc_b200 {

constexpr int SPLIT_X_BITS = 5, SPLIT_W_BITS = 6;
constexpr int SPLIT_K = 24, SPLIT_D = 22;
// tensor memory: the rows' three parts, [part][24] columns; the accumulators, S1 at column 0 and S0 at 40 (an MMA's N is a
// multiple of 16: eight more columns than units are written, into S0 before its first MMA clears it and behind S0)
constexpr int SPLIT_A_COLS = 3 * SPLIT_K, SPLIT_S0 = SPLIT_H, SPLIT_Z_COLS = SPLIT_S0 + 48;
// shared memory: the weights' three parts, K-major lines of 128 bytes (16-byte-chunk swizzle), a line per unit, and the
// eight lines behind the last part that the last MMAs read along (any finite values)
constexpr int SPLIT_B_PART = SPLIT_H * 128, SPLIT_B_BYTES = 3 * SPLIT_B_PART + 8 * 128;

// The high part is rounded, so that what is left has either sign; so is a weight's middle one, since what a product leaves out would
// otherwise have one sign for a weight in every row.  A row's middle part is everything left: the tensor core cuts it to 11
// bits itself, from which `rest` is counted
template <int BITS, bool WEIGHT>
__device__ __forceinline__ void split_parts(float v, float& high, float& mid, float& rest) {
  high = __uint_as_float((__float_as_uint(v) + (1u << (23 - BITS))) & ~((1u << (24 - BITS)) - 1u));
  const float r = v - high;
  const float cut = __uint_as_float((__float_as_uint(r) + (WEIGHT ? 0x1000u : 0u)) & 0xffffe000u);
  mid = WEIGHT ? cut : r;
  rest = r - cut;
}
__device__ __forceinline__ float split_round(float v) {  // to TF32
  return __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u);
}
// values whose parts would not add up to what FFMA makes of them
__device__ __forceinline__ bool split_wide(float v) { return (__float_as_uint(v) & 0x7fffffffu) >= 0x5d800000u; }

__device__ __forceinline__ float split_max(float m, float a, float b) {  // of the magnitudes; NaN if one is
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(a), "f"(b));
  return r;
}

// byte offset of features k .. k + 3 (k a multiple of 4) of unit n in a part of the weights
__device__ __forceinline__ uint32_t split_b_off(int n, int k) { return (uint32_t)(n * 128 + (((k >> 2) ^ (n & 7)) << 4)); }

// the parts of weight v, at shared address `dst` of the high one; a value that split_wide finds stays whole (the sum of the
// parts is the weight either way).  Returns whether it is one
__device__ __forceinline__ bool split_store_weight(uint32_t dst, float v) {
  float high, mid, rest;
  split_parts<SPLIT_W_BITS, true>(v, high, mid, rest);
  const bool wide = split_wide(v);
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst), "f"(wide ? v : high) : "memory");
  asm volatile("st.shared.f32 [%0+%2], %1;" ::"r"(dst), "f"(wide ? 0.f : mid), "n"(SPLIT_B_PART) : "memory");
  asm volatile("st.shared.f32 [%0+%2], %1;" ::"r"(dst), "f"(wide ? 0.f : rest), "n"(2 * SPLIT_B_PART) : "memory");
  return wide;
}

// features 8 j .. 8 j + 7 of this thread's row (v[7] of j = 2 must be zero: column 23 is the target) to tensor memory
template <int BITS = SPLIT_X_BITS>
__device__ __forceinline__ void split_store_row(uint32_t a_t, int j, const float (&v)[8]) {
  // (split_parts of two values at a time)
  constexpr uint32_t HALF = 1u << (23 - BITS), KEEP = ~((1u << (24 - BITS)) - 1u);
  const uint64_t minus1 = pack2(-1.f, -1.f);
  float p[3][8];
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    p[0][i] = __uint_as_float((__float_as_uint(v[i]) + HALF) & KEEP);
    p[0][i + 1] = __uint_as_float((__float_as_uint(v[i + 1]) + HALF) & KEEP);
    const uint64_t r = fma2(pack2(p[0][i], p[0][i + 1]), minus1, pack2(v[i], v[i + 1]));
    unpack2(r, p[1][i], p[1][i + 1]);
    const uint64_t cut = pack2(__uint_as_float(__float_as_uint(p[1][i]) & 0xffffe000u),
                               __uint_as_float(__float_as_uint(p[1][i + 1]) & 0xffffe000u));
    unpack2(fma2(cut, minus1, r), p[2][i], p[2][i + 1]);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q)
    tc_st8(a_t + q * SPLIT_K + 8 * j, make_float4(p[q][0], p[q][1], p[q][2], p[q][3]),
           make_float4(p[q][4], p[q][5], p[q][6], p[q][7]));
}

// The 24 MMAs of a 128-row tile, by a converged warp (`on` in one lane): all products but rest x rest, smallest first.
// (As a loop they take 150 cycles each, for want of operands that are constants apart; a predicate that keeps one from being issued
// costs as much as the MMA)
__device__ __forceinline__ void split_issue(uint32_t z_t, uint32_t a_t, uint32_t b_smem, uint32_t on) {
  constexpr uint32_t IDESC = umma_idesc_tf32(128, 48, 0, 0);
  const uint64_t b0 = umma_desc_k128(b_smem);
  constexpr int NP = 8, XP[NP] = {2, 1, 2, 0, 1, 1, 0, 0}, WP[NP] = {1, 2, 0, 2, 1, 0, 1, 0};
#pragma unroll
  for (int q = 0; q < NP; ++q)
#pragma unroll
    for (int kb = 0; kb < 3; ++kb)
      tc_mma_tf32_ts_if(z_t + (q == NP - 1 ? SPLIT_S0 : 0), a_t + XP[q] * SPLIT_K + kb * 8,
                        umma_desc_advance(b0, WP[q] * (SPLIT_B_PART >> 4) + kb * 2), IDESC, q % (NP - 1) > 0 || kb > 0 ? 1u : 0u, on);
}

}  // namespace mcmc_b200
