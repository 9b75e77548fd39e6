// Shared device-side definitions of the HMC hot path: launch parameter
// blocks, the fused leapfrog prologue, likelihood terms and the PTX wrappers
// (mbarrier, bulk copies, tcgen05) used by the gradient kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <utility>

namespace mcmc_b200 {

// Rows of the repacked dataset: 22 features, a constant 1 (so that the hidden
// bias is row 22 of W0 and db0 is row 22 of dW0), and the target y.
constexpr int KP = 24;          // floats per repacked row (96 bytes)
constexpr int COL_ONE = 22;
constexpr int COL_Y = 23;
constexpr int MAX_SLICES = 1024;

enum GradMode : int {
  MODE_EVAL = 0,   // evaluate at w_in as it is (the reference's eps = 0 call, main.h:85-99)
  MODE_FIRST = 1,  // half kick with the carried gradient, drift (MOM_CORRECTION = 2)
  MODE_NEXT = 2    // full kick with the gradient of the previous step, drift
};

struct LikParams {
  int kind;          // 0 Student-t, 1 Gaussian
  float inv_scale;   // 1 / scale
  float df;          // Student-t degrees of freedom
  float norm;        // log-normaliser
  float g_scale;     // (df + 1) / scale  (Student-t)  |  1 / scale (Gaussian)
  float l_scale;     // -(df + 1) / 2     (Student-t)  |  -1/2      (Gaussian)
  float inv_df;
};

struct PriorParams {
  float neg_inv_s2;  // -1 / s^2   (PRIOR_SCALE_NEG_RECP2)
  float inv_s;       // 1 / s
  float norm;        // PRIOR_LOSS_NORMALIZATION
};

// One launch of a gradient kernel: grid = (slices, windows).
struct GradParams {
  // data
  const float* xaug;        // [windows][rows_pad][KP]
  long long window_stride;  // floats between windows in xaug
  int data_window0;         // first data window this launch covers
  int n_rows;               // valid rows per window
  int n_tiles;              // rows_pad / tile rows
  int P, Pp;                // parameters, padded to a multiple of 4
  // state in / out ([windows][Pp], indexed by blockIdx.y)
  const float* w_in;
  const float* m_in;
  float* w_out;
  float* m_out;
  const float* g_carried;   // MODE_FIRST
  const float* partial_in;  // MODE_NEXT: [windows][slices_in][Pp] likelihood-gradient partials
  int slices_in;            // slots per window in partial_in (stride, and count when nslot_in is null)
  const int* nslot_in;      // optional [windows]: slots of partial_in that are in use
  // persistent (one CTA per SM) kernels: which tile ranges this launch's CTAs own
  const int* seg_ptr;       // [ctas + 1] first segment of each CTA
  const int4* segs;         // {window, first tile, end tile, slot}
  int slices_out;           // slots per window in partial_out / ll_out
  const double* red_in;     // MODE_NEXT with row sharding: [windows][Pp + 4] all-reduced sums
  float* partial_out;       // [windows][slices][Pp]
  double* ll_out;           // [windows][slices]
  const float* eps;         // [windows] or null
  float eps_scalar;
  int mode;
  int no_loss;              // 1: a step inside a trajectory, whose losses nobody reads (ll_out may be zero, row_loss is null)
  float* row_loss;          // optional [windows][rows_pad]
  long long row_loss_stride;
  LikParams lik;
  PriorParams prior;
  int* status;              // device error word (bounded waits that ran out)
  int data_fresh;           // 1: xaug was written by the launch directly before this one in the stream, so
                            // no row may be fetched ahead of the programmatic-dependency wait
  // self-test: 102 adds a wait for MMAs that nothing ends (streaming FP32 kernels with the tensor core), 103 to 105 one inside a segment (grad_fp32_int.cu)
  int test_code;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Dynamic shared memory from its first 1024-byte boundary on.  The offset is added to the array itself: a pointer rounded up as an
// integer loses its address space, and every access through it becomes a generic one.
__device__ __forceinline__ unsigned char* smem_align1024(unsigned char* raw) {
  return raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
}

// ---- reference tanh (kernel_helpers.h:32-44): 2*sigmoid(2x)-1 on ex2/rcp
// approximations, identity below the cut-off -------------------------------
__device__ __forceinline__ float tanh_ref(float x) {
  float e, d, s;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -2.88539008177792681472f));
  asm("add.ftz.f32 %0, %1, %2;" : "=f"(d) : "f"(1.f), "f"(e));
  // (ftz: d >= 1, and a result that would be denormal comes out as -1 either way)
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(d));
  return fabsf(x) < 0.0048176045529544353485f ? x : fmaf(s, 2.f, -1.f);
}
// one MUFU op; absolute error about 5e-4, inside the TF32 mode's tolerance
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// d(log-lik)/d(prediction) of a row, and its log-likelihood
__device__ __forceinline__ float lik_grad(const LikParams& lk, float y, float pred) {
  const float d = (y - pred) * lk.inv_scale;
  return lk.kind == 0 ? __fdividef(d * lk.g_scale, fmaf(d, d, lk.df)) : d * lk.g_scale;
}
__device__ __forceinline__ float lik_loss(const LikParams& lk, float y, float pred) {
  const float d = (y - pred) * lk.inv_scale, d2 = d * d;
  return lk.kind == 0 ? lk.l_scale * log1pf(d2 * lk.inv_df) - lk.norm : fmaf(lk.l_scale, d2, -lk.norm);
}
// per-row log-likelihood and d(log-lik)/d(prediction)
// (mcmc_step_ffma.h:289-301 for Student-t)
__device__ __forceinline__ void lik_terms(const LikParams& lk, float y, float pred, float& loss,
                                          float& dy) {
  float d = (y - pred) * lk.inv_scale;
  float d2 = d * d;
  if (lk.kind == 0) {
    loss = lk.l_scale * log1pf(d2 * lk.inv_df) - lk.norm;
    dy = __fdividef(d * lk.g_scale, d2 + lk.df);
  } else {
    loss = fmaf(lk.l_scale, d2, -lk.norm);
    dy = d * lk.g_scale;
  }
}

// Fused leapfrog update of N parameters of window `win`: p0, p0 + step, ... below `limit`
// (apply_leapfrog_step, mcmc_step_ffma.h:106-120; load_weights_bias :122-152):
// every CTA of the window recomputes the same values from the same inputs in
// the same order, slice 0 stores them.
// All of a thread's loads come before its stores: one parameter after the other, a store between the loads of two of them
// kept the second's from being issued early, and eight of them were eight trips to L2 in a row (FP32, 16 windows of 40013
// rows: 82 us a step instead of 79; 128 units TF32, 8 x 1,048,576 rows: 541 instead of 530).
template <int N>
__device__ __forceinline__ void leapfrog_params(const GradParams& g, int win, int p0, int step, int limit, bool store,
                                                float (&w)[N]) {
  const size_t o = (size_t)win * g.Pp + p0;
  const float eps = g.eps ? g.eps[win] : g.eps_scalar;
  float grad[N], m[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    w[i] = grad[i] = m[i] = 0.f;
    if (p0 + i * step < limit) w[i] = __ldcg(g.w_in + o + i * step);
  }
  if (g.mode == MODE_EVAL) return;
  float kick;
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (p0 + i * step < limit) m[i] = __ldcg(g.m_in + o + i * step);
  if (g.mode == MODE_FIRST) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (p0 + i * step < limit) grad[i] = __ldcg(g.g_carried + o + i * step);
    kick = 0.5f;
  } else {
    if (g.red_in) {
      const double* r = g.red_in + (size_t)win * (g.Pp + 4) + p0;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (p0 + i * step < limit) grad[i] = (float)__ldcg(r + i * step);
    } else {
      const float* pi = g.partial_in + (size_t)win * g.slices_in * g.Pp + p0;
      const int ns = g.nslot_in ? g.nslot_in[win] : g.slices_in;
      for (int s = 0; s < ns; ++s)
#pragma unroll
        for (int i = 0; i < N; ++i)
          if (p0 + i * step < limit) grad[i] += __ldcg(pi + (size_t)s * g.Pp + i * step);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) grad[i] = fmaf(w[i], g.prior.neg_inv_s2, grad[i]);  // prior gradient at the previous point
    kick = 1.f;
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    m[i] = fmaf(eps * kick, grad[i], m[i]);
    w[i] = fmaf(eps, m[i], w[i]);
  }
  if (store) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (p0 + i * step < limit) {
        g.w_out[o + i * step] = w[i];
        g.m_out[o + i * step] = m[i];
      }
  }
}

// ---- mbarrier / bulk-copy wrappers --------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// try_wait that lets the hardware suspend the thread for up to `hint_ns` until the phase completes
__device__ __forceinline__ bool mbar_try_wait_hint(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
// Bounded wait: the thread sleeps in hardware on the barrier in slices of 20 us and gives up after
// `slices` of them (default 2^16, about 1.3 s), records the code in the status word and returns false;
// the kernel then finishes with whatever it has, so a lost copy or MMA can never hang the GPU.
constexpr uint32_t MBAR_WAIT_SLICES = 1u << 16;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status, int code,
                                          uint32_t slices = MBAR_WAIT_SLICES) {
  if (mbar_try_wait(bar, parity)) return true;
  for (uint32_t i = 0; i < slices; ++i) {
    if (mbar_try_wait_hint(bar, parity, 20000u)) return true;
  }
  if (status) atomicExch(status, code);
  return false;
}
// contiguous global -> shared copy through the bulk-copy engine
__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src, uint32_t bytes,
                                         uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst_smem)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// block-wide sum of doubles in a fixed order (deterministic); blockDim.x <= 1024
__device__ __forceinline__ double block_sum_f64(double v, double* scratch /* >= 32 */) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) scratch[w] = v;
  __syncthreads();
  double t = 0.0;
  const int nw = (blockDim.x + 31) >> 5;
  for (int i = 0; i < nw; ++i) t += scratch[i];
  return t;
}

// Packed FP32 pairs (sm_100 executes fma/mul on two floats per instruction)
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// tanh_ref of two values, its arithmetic packed
__device__ __forceinline__ uint64_t tanh_ref2(uint64_t x) {
  float x0, x1, e0, e1, d0, d1, s0, s1, t0, t1;
  uint64_t m, d, t;
  unpack2(x, x0, x1);
  m = mul2(x, pack2(-2.88539008177792681472f, -2.88539008177792681472f));
  unpack2(m, e0, e1);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e0));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e1));
  d = add2(pack2(1.f, 1.f), pack2(e0, e1));
  unpack2(d, d0, d1);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s0) : "f"(d0));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s1) : "f"(d1));
  t = fma2(pack2(s0, s1), pack2(2.f, 2.f), pack2(-1.f, -1.f));
  unpack2(t, t0, t1);
  return pack2(fabsf(x0) < 0.0048176045529544353485f ? x0 : t0, fabsf(x1) < 0.0048176045529544353485f ? x1 : t1);
}

// ---- programmatic dependent launch -----------------------------------------
// The chain is a string of short dependent launches (gradient, partial sum, accept).  A kernel
// launched with the programmatic-serialization attribute may start while its predecessor is still
// draining: its CTAs are scheduled as the predecessor's CTAs exit, do their private set-up (barriers,
// tensor-memory allocation, first row tiles — nothing the predecessor writes) and then block in
// pdl_wait() until the predecessor has completed and its writes are visible.  Every kernel of the
// chain calls pdl_trigger() (lets ITS successor start early) and pdl_wait() before it touches
// anything a predecessor produced, and writes global memory only after the wait.  Without the launch
// attribute both calls do nothing.  MCMC_B200_NO_PDL=1 turns the attribute off.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline bool pdl_enabled() {
  static const bool on = [] {
    const char* e = getenv("MCMC_B200_NO_PDL");
    return !(e && e[0] == '1');
  }();
  return on;
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_chain_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                       cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace mcmc_b200
