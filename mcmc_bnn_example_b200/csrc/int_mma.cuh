// Sums over rows of features x dL/dz, 24 x 40 of them, exact on the integer tensor core: the FP32 kernels' backward pass.
//
// By FFMA it was half of a tile's instructions.  TF32 or bf16 parts, as the forward product has them (split_mma.cuh), are no way for it: the
// tensor core cuts off every addition in the same direction, and over thousands of rows that adds up.  Its integer form adds exactly.
//   * One factor becomes an integer of 32 bits, round(x 2^31 / X), X a power of two per feature; the other likewise with a power of
//     two B for all of them.  On the chip (resident_fp32.cu) they are the feature and dL/dz, streaming (grad_fp32_int.cu) the feature x dL/dpred
//     and 1 - h^2.  Either is four signed bytes (adding 0x808080 and flipping the lower bytes' top bits makes the digits), which
//     is how memory holds it: no byte has to be moved.
//   * One tcgen05.mma kind::i8 multiplies all 4 x 4 bytes of 32 rows, a warp's: M = 96 lines (byte a of feature k is line 4 k + a;
//     the instruction's other 32 read whatever follows, and nobody reads their sums), N = 160 columns (byte b of unit j is column 4 j + b).
//     Sums stay below 2^31 for 128,000 rows (127 x 128 x 128,000); their order is of no consequence.
//   * Whoever reads them weighs them by 2^(8 a + 8 b) in FP32: the first rounding after those of the integers.
// On the chip X is bounded by the rows' largest value, where that is less than 2^8 over the mean binary exponent (int_scale_exp); B is 2^5 over the mean
// exponent of dL/dpred: a normal distribution ends at half of that, and what lies beyond is an outlier.  A warp that has one takes
// FFMA, as infinities and NaN do.  So does one with INT_FEW rows far below the mean, of which integers would have fewer bits than a float: behind a first tile with residuals a
// thousand times theirs, gradients of a feature that is only there were 1e-5 off (FFMA and now 1e-7).  So an integer of dL/dz is off by 2^-29 of their rms.
// Gradients' error against 64 bits, on the chip / by FFMA: N(0,1) features 0.95 to 1.00 of it over 1000 to 58368 rows, feature by feature 0.86 to 0.98; t-distributed, lognormal, constant,
// zero-one and differently scaled features, targets with outliers, ordered rows 0.8 to 1.02, in the mean 0.96.  (Streaming: grad_fp32_int.cu.)  With 2^8 in the place of 2^5, and
// 30 bits instead of 31, it was 1.1 to 1.7 times as large for 100 rows.
// Operands lie in shared memory without a swizzle, rows as K: groups of 8 rows, in them 16 bytes of a row (four values), row after row.
// An MMA of 128 x 160 x 32 takes 81 cycles (one B200).
#pragma once
#include "split_mma.cuh"

namespace mcmc_b200 {

constexpr int INT_X_ROW = SPLIT_K * 4, INT_E_ROW = SPLIT_H * 4;          // bytes of a row
constexpr int INT_X_WARP = 32 * INT_X_ROW, INT_E_WARP = 32 * INT_E_ROW;  // ... and of 32
constexpr int INT_ACC_COLS = INT_E_ROW, INT_LINES = INT_X_ROW;
constexpr float INT_TOP = 2126008811.f;      // 0.99 x 2^31: the bound of scaled values
constexpr float INT_LOW = 1048576.f;         // 2^-6 of their mean exponent, which 0.5 % of normal ones are below: of 32 rows five once in a million
constexpr int INT_FEW = 5;
// sums of a unit's 96 lines side by side; four floats more keep readers of neighbouring units apart
constexpr int INT_S_STR = INT_LINES + 4, INT_S_FLOATS = SPLIT_H * INT_S_STR;

__device__ __forceinline__ uint64_t int_x_desc(uint32_t smem) { return umma_desc(smem, 8 * INT_X_ROW, 128, 0); }
__device__ __forceinline__ uint64_t int_e_desc(uint32_t smem) { return umma_desc(smem, 8 * INT_E_ROW, 128, 0); }
// instruction: S32 sums of S8 x S8, M = 128, N = 160, both operands with rows as K outermost
constexpr uint32_t INT_IDESC = (2u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                               ((uint32_t)(INT_ACC_COLS >> 3) << 17) | ((128u >> 4) << 24);
__device__ __forceinline__ void int_mma_if(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(INT_IDESC), "r"(accumulate), "r"(on)
      : "memory");
}

// The four signed bytes of round(x * scale), two values at a time.  Conversions would take the pipe of the tanh, 8 cycles each; this is
// done by additions: high = x scale + INT_HI is that number in units of 512, INT_HI + INT_LO - high the rest's offset, and the low bits of
// both floats are integers.  Their offsets go, and 0x808080 comes (digits from -128 on), in one addition.
constexpr float INT_HI = 6442450944.f, INT_LO = 12582912.f;   // 1.5 x 2^32, 1.5 x 2^23
__device__ __forceinline__ uint2 int_digits2_of(uint64_t hi, uint64_t lo) {
  float h0, h1, l0, l1;
  unpack2(hi, h0, h1);
  unpack2(lo, l0, l1);
  constexpr uint32_t OFF = 0x808080u - (0x80000000u + 0x4b400000u);
  return make_uint2(((__float_as_uint(h0) << 9) + __float_as_uint(l0) + OFF) ^ 0x808080u,
                    ((__float_as_uint(h1) << 9) + __float_as_uint(l1) + OFF) ^ 0x808080u);
}
__device__ __forceinline__ uint2 int_digits2(uint64_t x, uint64_t scale) {
  const uint64_t hi = fma2(x, scale, pack2(INT_HI, INT_HI));
  return int_digits2_of(hi, fma2(x, scale, fma2(hi, pack2(-1.f, -1.f), pack2(INT_HI + INT_LO, INT_HI + INT_LO))));
}
__device__ __forceinline__ uint2 int_digits2(uint64_t x) {  // of values that have been scaled
  const uint64_t hi = add2(x, pack2(INT_HI, INT_HI));
  return int_digits2_of(hi, add2(x, fma2(hi, pack2(-1.f, -1.f), pack2(INT_HI + INT_LO, INT_HI + INT_LO))));
}

// Statistics behind a scale: a value's contribution; sums of them over at most 2^12 - 1 values
__device__ __forceinline__ uint32_t int_stat(float v) {
  const uint32_t e = (__float_as_uint(v) >> 23) & 255u;
  return e - 1u < 254u ? e | 1u << 20 : 0u;
}
constexpr int INT_ROOM_X = 8, INT_ROOM_E = 5;   // (see above)
// Biased exponent of the power of two that bounds the range: 2^room over the mean of the exponents.  INT_NONE: nothing is known of the
// values, or scales and their products might leave the range of a float: then only zeros are in range, all else is an outlier (2^126 as a scale)
constexpr int INT_NONE = 32;
__device__ __forceinline__ int int_scale_exp(uint32_t stat, int room) {
  const float n = (float)(stat >> 20);
  return n > 0.f ? (int)__fdividef((float)(stat & 0xfffffu) + 0.5f * n, n) + room : INT_NONE;
}
// the same for the largest magnitude, whose bits these are
__device__ __forceinline__ int int_max_exp(uint32_t bits) { return (int)((bits + 0x30000u) >> 23) + 1; }
template <int MOST = 60>
__device__ __forceinline__ int int_range_exp(int e) { return e >= 147 - MOST && e <= 127 + MOST ? e : INT_NONE; }
// the smallest of several, as the largest of these words; 0 where there is none.  (Kept within what int_range_exp allows: values for which that is
// no range are out of it)
__device__ __forceinline__ uint32_t int_stat_word(int e) { return 1024u - (uint32_t)min(max(e, 87), 187); }
__device__ __forceinline__ int int_stat_exp(uint32_t word) { return word ? (int)(1024u - word) : INT_NONE; }
__device__ __forceinline__ float int_scale(int e) { return __int_as_float((127 + 31 + 127 - e) << 23); }    // 2^31 / 2^(e - 127)
__device__ __forceinline__ float int_unscale(int e) { return __int_as_float((e - 31) << 23); }              // its inverse

// features 4 c .. 4 c + 3 of row `row` of 32
__device__ __forceinline__ uint32_t int_x_off(int row, int c) { return (uint32_t)((row >> 3) * (8 * INT_X_ROW) + c * 128 + (row & 7) * 16); }
__device__ __forceinline__ void int_store_x4(uint32_t dst, float4 x, float4 scale) {
  const uint2 a = int_digits2(pack2(x.x, x.y), pack2(scale.x, scale.y)), b = int_digits2(pack2(x.z, x.w), pack2(scale.z, scale.w));
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(a.x), "r"(a.y), "r"(b.x), "r"(b.y) : "memory");
}

// Sums of NU units (columns 4 j, ... + 3 at `t`), line 32 q + lane of the accumulator with q the warp's quarter, times `f` over 2^INT_READ_SHIFT.  Of at most 2^9
// rows, so that the two upper bytes' fit an integer.  Of the two lower ones' 2 bits are cut off, 2^-36 of the largest product X B.  (Cut off at the
// upper one's unit, 2^-30 of it and always downwards, they were as much as all other roundings of the integers, and more where a CTA has few rows
// with a feature)
constexpr int INT_READ_SHIFT = 2;
template <int NU>
__device__ __forceinline__ void int_read_out(uint32_t t, float f, float (&out)[NU]) {
  float a[4 * NU];
#pragma unroll
  for (int i = 0; i < NU / 2; ++i) tc_ld8(t + 8 * i, a + 8 * i);
  tc_wait_ld();
#pragma unroll
  for (int j = 0; j < NU; ++j) {
    const int v0 = __float_as_int(a[4 * j]), v1 = __float_as_int(a[4 * j + 1]), v2 = __float_as_int(a[4 * j + 2]),
              v3 = __float_as_int(a[4 * j + 3]);
    out[j] = fmaf((float)(v3 * 256 + v2), 16384.f, (float)(v1 * 64 + (v0 >> 2))) * f;
  }
}
// ... of any number of rows, without the factor
template <int NU>
__device__ __forceinline__ void int_read_out_long(uint32_t t, float (&out)[NU]) {
  float a[4 * NU];
#pragma unroll
  for (int i = 0; i < NU / 2; ++i) tc_ld8(t + 8 * i, a + 8 * i);
  tc_wait_ld();
#pragma unroll
  for (int j = 0; j < NU; ++j) {
    const float s = fmaf((float)__float_as_int(a[4 * j + 1]), 256.f, (float)__float_as_int(a[4 * j]));
    out[j] = fmaf((float)__float_as_int(a[4 * j + 3]), 16777216.f, fmaf((float)__float_as_int(a[4 * j + 2]), 65536.f, s));
  }
}
// the sum over a feature's four lines
__device__ __forceinline__ float int_sum4(const float* s, int k, int unit) {
  const float4 v = *reinterpret_cast<const float4*>(s + unit * INT_S_STR + 4 * k);
  return ((v.x + v.y) + v.z) + v.w;
}

}  // namespace mcmc_b200
