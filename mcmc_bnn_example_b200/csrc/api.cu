// C-ABI of the library (declared in include/mcmc_b200.h): context and buffer
// management, launch sequencing of the gradient / accept kernels, CUDA-graph
// replay of whole HMC iterations, the optional NCCL allreduce for row sharding.
// Host-side counterpart of the reference's main_loop / Network / mcmc_step
// (include/mcmc/main.h:48-76, :117-308; mcmc_step_ffma.h:395-427).
#include <cuda.h>
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <limits>
#include <mutex>
#include <random>
#include <string>
#include <vector>

#include "../../include/mcmc_b200.h"
#include "chain.cuh"
#include "common.cuh"
#include "philox.h"
#include "refstream.cuh"

using namespace mcmc_b200;

#define API extern "C" __attribute__((visibility("default")))

static thread_local std::string g_last_error;

static int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}
// for the other translation units of the library
void mcmc_b200_set_last_error(const std::string& msg) { g_last_error = msg; }

#define CK(call)                                                                              \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess)                                                                    \
      return fail(MCMC_B200_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));    \
  } while (0)

// ---- NCCL through dlopen: no link-time dependency, and the copy already
// loaded into the process (for instance by torch) is the one that is used ----
namespace {
struct NcclUniqueId { char internal[128]; };
typedef void* NcclComm;
struct NcclApi {
  void* handle = nullptr;
  int (*GetUniqueId)(NcclUniqueId*) = nullptr;
  int (*CommInitRank)(NcclComm*, int, NcclUniqueId, int) = nullptr;
  int (*AllReduce)(const void*, void*, size_t, int, int, NcclComm, cudaStream_t) = nullptr;
  int (*AllGather)(const void*, void*, size_t, int, NcclComm, cudaStream_t) = nullptr;
  int (*CommDestroy)(NcclComm) = nullptr;
  const char* (*GetErrorString)(int) = nullptr;
  bool ok = false;
};
NcclApi g_nccl;

bool nccl_load(std::string* why) {
  if (g_nccl.ok) return true;
  const char* env = getenv("MCMC_B200_NCCL_LIB");
  const char* names[] = {env, "libnccl.so.2", "libnccl.so"};
  for (const char* n : names) {
    if (!n) continue;
    g_nccl.handle = dlopen(n, RTLD_NOW | RTLD_GLOBAL);
    if (g_nccl.handle) break;
  }
  if (!g_nccl.handle) {
    *why = std::string("dlopen(libnccl.so.2) failed: ") + dlerror();
    return false;
  }
  g_nccl.GetUniqueId = (int (*)(NcclUniqueId*))dlsym(g_nccl.handle, "ncclGetUniqueId");
  g_nccl.CommInitRank = (int (*)(NcclComm*, int, NcclUniqueId, int))dlsym(g_nccl.handle, "ncclCommInitRank");
  g_nccl.AllReduce = (int (*)(const void*, void*, size_t, int, int, NcclComm, cudaStream_t))dlsym(
      g_nccl.handle, "ncclAllReduce");
  g_nccl.AllGather = (int (*)(const void*, void*, size_t, int, NcclComm, cudaStream_t))dlsym(g_nccl.handle,
                                                                                         "ncclAllGather");
  g_nccl.CommDestroy = (int (*)(NcclComm))dlsym(g_nccl.handle, "ncclCommDestroy");
  g_nccl.GetErrorString = (const char* (*)(int))dlsym(g_nccl.handle, "ncclGetErrorString");
  if (!g_nccl.GetUniqueId || !g_nccl.CommInitRank || !g_nccl.AllReduce || !g_nccl.CommDestroy) {
    *why = "NCCL symbols missing";
    return false;
  }
  g_nccl.ok = true;
  return true;
}
constexpr int kNcclFloat64 = 8;
constexpr int kNcclChar = 0;
constexpr int kNcclSum = 0;
}  // namespace

constexpr int HB_FLOATS = 3076;  // P of the widest model, rounded up
struct HostBlock {
  double scalars[2];
  int status;
  float log_acpt;  // out: the drop-in accept ratio
  int fwd_status;  // a wait of a forward pass that ran out
  int pad[1];
  float w[HB_FLOATS], m[HB_FLOATS], g[HB_FLOATS];  // in: position, momentum, gradient
  float w_out[HB_FLOATS], m_out[HB_FLOATS], g_out[HB_FLOATS];
};

// Page-locking takes milliseconds, so the blocks of destroyed contexts are kept for the next ones: at most
// HB_CHUNK of them, one allocation, returned when the process ends.  Any thread may take and give.
constexpr int HB_CHUNK = 16;
static std::mutex g_hb_mutex;
static HostBlock* g_hb_chunk = nullptr;
static unsigned g_hb_used = 0;  // bit i: block i of the chunk is taken
static HostBlock* host_block_take() {
  std::lock_guard<std::mutex> lock(g_hb_mutex);
  if (!g_hb_chunk) {
    void* p = nullptr;
    if (cudaHostAlloc(&p, sizeof(HostBlock) * HB_CHUNK, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) return nullptr;
    g_hb_chunk = static_cast<HostBlock*>(p);
  }
  for (int i = 0; i < HB_CHUNK; ++i)
    if (!(g_hb_used >> i & 1u)) {
      g_hb_used |= 1u << i;
      return g_hb_chunk + i;
    }
  void* p = nullptr;  // more contexts than that at once: a block of its own
  return cudaHostAlloc(&p, sizeof(HostBlock), cudaHostAllocMapped | cudaHostAllocPortable) == cudaSuccess
             ? static_cast<HostBlock*>(p) : nullptr;
}
static void host_block_give(HostBlock* b) {
  std::lock_guard<std::mutex> lock(g_hb_mutex);
  if (b >= g_hb_chunk && b < g_hb_chunk + HB_CHUNK) g_hb_used &= ~(1u << (b - g_hb_chunk));
  else cudaFreeHost(b);
}

struct mcmc_b200_ctx {
  mcmc_b200_config cfg;
  int device = 0, W = 0, P = 0, Pp = 0;
  long long rows = 0, rows_pad = 0;
  int num_sms = 0, ctas_per_sm = 1;
  bool use_red = false, use_red_x = false;  // sum partial slots with a separate small launch
  int slices = 1;      // CTAs per window in chain launches
  int slices_x = 1;    // CTAs for single-window explicit calls
  int tile_rows = 64;
  cudaStream_t stream = nullptr;
  cudaStream_t copies = nullptr;  // predict_mean: rows and means of a block beside the pass over another
  cudaEvent_t copy_events[3] = {};
  // dataset
  float* xaug = nullptr;
  std::vector<char> window_set;
  CUtensorMap tmaps[2] = {};  // 32-byte-chunk swizzle; 128 units: and 16-byte-chunk swizzle
  // persistent kernels (TF32; FP32 with 40 units) have work tables: chain launches and single-window launches
  bool table = false;
  int *tab_seg_ptr = nullptr, *tab_nslot = nullptr, *xtab_seg_ptr = nullptr, *xtab_nslot = nullptr;
  int4 *tab_segs = nullptr, *xtab_segs = nullptr;
  int tab_ctas = 0, xtab_ctas = 0;
  bool tab_ints = false, xtab_ints = false;   // FP32: its segments are for grad_fp32_int.cu
  // chain state
  float *wbuf[2] = {}, *mbuf[2] = {}, *w_cur = nullptr, *g_cur = nullptr, *m0 = nullptr;
  float* partial[2] = {};
  double* llp[2] = {};
  double *red = nullptr, *ll_cur = nullptr, *lp_cur = nullptr;
  float* eps = nullptr;
  int *iter = nullptr, *n_accept = nullptr;
  long long* gwin = nullptr;
  float* samples = nullptr;
  float *tr_mom = nullptr, *tr_log_u = nullptr, *tr_eps = nullptr;
  double* tr_log_acpt = nullptr;
  int* tr_accept = nullptr;
  int* status = nullptr;
  std::vector<long long> h_gwin;
  bool bootstrapped = false;
  int iters_done = 0;
  // explicit-state scratch (one window)
  float *xw[2] = {}, *xm[2] = {}, *xg = nullptr, *xpartial[2] = {}, *g_out = nullptr, *row_loss = nullptr;
  double *xllp[2] = {}, *xred = nullptr, *scalars = nullptr;
  // bound dataset of the drop-in mcmc_step
  const float *bound_x = nullptr, *bound_y = nullptr;
  // graph of one HMC iteration
  cudaGraphExec_t graph_exec = nullptr;
  bool graph_tried = false;
  // row sharding
  NcclComm comm = nullptr;
  int nranks = 1, rank = 0;
  // ... with the one-shot all-reduce over peer memory instead of the NCCL call
  bool oneshot = false;
  void* os_block = nullptr;                 // this rank's receive buffer + flags (one allocation, IPC-exported)
  std::vector<void*> os_peer_blocks;        // the peers' blocks as mapped here (null at [rank])
  std::vector<void*> os_base;               // every rank's block as seen from here (own block at [rank])
  unsigned int *os_seq = nullptr, *os_done = nullptr;
  unsigned int os_poll_limit = 1u << 22;    // polls of about 0.1 us .. 1 us each
  long long launches = 0;
  // whole iterations in one cooperative launch (resident.cuh): plans and message buffers of the chain launches
  // and of the single-window explicit calls, for contexts that may have such launches at all (res_try); a plan is made
  // when the first call wants it
  bool res_try = false, res_asked = false, res_x_asked = false, res_ok = false, res_x_ok = false;
  ResidentParams res, res_x;
  int res_cluster = 1, res_x_cluster = 1;  // CTAs per cluster
  int refuse = 0;  // self-test: the next such launches that are answered as too large
  int test_code = 0;       // self-test: ForwardParams, GradParams
  int refuse_forward = 0;  // self-test: which of the next forward launches of predict_mean is answered so
  // host block the kernels of the explicit host-pointer calls read and write directly (mapped, page-locked)
  HostBlock* hb = nullptr;
  // small device arrays are cut from zeroed slabs
  char* slab = nullptr;
  size_t slab_left = 0;
  float* stage = nullptr;  // upload staging for one window: [rows][D] then [rows]
  // forward-only pass over the stored samples: scratch that grows on demand and is kept (no allocation per call)
  float* fwd_x = nullptr;
  float* fwd_out = nullptr;
  double* fwd_partial = nullptr;
  size_t fwd_x_cap = 0, fwd_out_cap = 0, fwd_partial_cap = 0;
  // the reference's random streams: host-computed log accept draws, indexed by iteration
  float* ref_log_u = nullptr;
  int ref_cap = 0, ref_filled = 0;
  std::vector<void*> allocs;
};

// Device memory of the context.  Small arrays share zeroed slabs: a context has some forty of them, and an
// allocator call each (they synchronise the device) was most of the time to create one.
constexpr size_t SLAB_BYTES = 1u << 20, SLAB_MAX = 16u << 10;
static int dalloc(mcmc_b200_ctx* c, void** p, size_t bytes, bool zero = true) {
  bytes = (std::max<size_t>(bytes, 16) + 255) / 256 * 256;
  const bool small = bytes <= SLAB_MAX;
  if (small && bytes <= c->slab_left) {
    *p = c->slab;
    c->slab += bytes;
    c->slab_left -= bytes;
    return MCMC_B200_OK;
  }
  const size_t take = small ? SLAB_BYTES : bytes;
  cudaError_t e = cudaMalloc(p, take);
  if (e != cudaSuccess) {
    cudaGetLastError();  // (not the error of the next launch)
    return fail(MCMC_B200_ERR_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  }
  c->allocs.push_back(*p);
  if (zero || small) {
    // waited for here: what fills the array next may be queued on another stream
    e = cudaMemsetAsync(*p, 0, take, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, std::string("cudaMemset: ") + cudaGetErrorString(e));
  }
  if (small) {
    c->slab = (char*)*p + bytes;
    c->slab_left = take - bytes;
  }
  return MCMC_B200_OK;
}
#define DA(ptr, bytes)                                                   \
  do {                                                                   \
    int r_ = dalloc(c, (void**)&(ptr), (bytes));                         \
    if (r_ != MCMC_B200_OK) { mcmc_b200_destroy(c); return r_; }         \
  } while (0)

API const char* mcmc_b200_last_error(void) { return g_last_error.c_str(); }
API int mcmc_b200_has_tf32(void) { return tf32_supported(40); }

API void mcmc_b200_config_reference(mcmc_b200_config* cfg) {
  memset(cfg, 0, sizeof(*cfg));
  cfg->D = 22; cfg->H = 40;
  cfg->likelihood = MCMC_B200_LIK_STUDENT_T;
  cfg->precision = MCMC_B200_PREC_FP32;
  cfg->lik_scale = 100.0; cfg->lik_df = 2.2; cfg->prior_scale = 200.0;
  cfg->leapfrog_steps = 1000; cfg->burn_in = 100; cfg->adapt_steps = 100; cfg->sample_capacity = 800;
  cfg->eps0 = 0.01; cfg->target_rate = 0.2; cfg->decrement = 0.1; cfg->increment = 0.01;
  cfg->seed = 0; cfg->trace_iters = 0; cfg->slices = 0;
  cfg->rng_streams = MCMC_B200_RNG_PHILOX;
}
API void mcmc_b200_config_baseline(mcmc_b200_config* cfg) {
  mcmc_b200_config_reference(cfg);
  cfg->likelihood = MCMC_B200_LIK_GAUSSIAN;
  cfg->lik_scale = 1.0; cfg->lik_df = 0.0; cfg->prior_scale = 1.0;
  cfg->leapfrog_steps = 10; cfg->burn_in = 0; cfg->adapt_steps = 0;
  cfg->eps0 = 1e-3;
}

static LikParams make_lik(const mcmc_b200_config& cfg) {
  LikParams l;
  const double pi = 3.14159265358979323846;
  l.kind = cfg.likelihood;
  l.inv_scale = (float)(1.0 / cfg.lik_scale);
  if (cfg.likelihood == MCMC_B200_LIK_STUDENT_T) {
    l.df = (float)cfg.lik_df;
    l.inv_df = (float)(1.0 / cfg.lik_df);
    l.norm = (float)(log(fabs(cfg.lik_scale)) + 0.5 * log(cfg.lik_df) + 0.5 * log(pi) +
                     lgamma(0.5 * cfg.lik_df) - lgamma(0.5 * (cfg.lik_df + 1.0)));
    l.g_scale = (float)((cfg.lik_df + 1.0) / cfg.lik_scale);
    l.l_scale = (float)(-0.5 * (cfg.lik_df + 1.0));
  } else {
    l.df = 0.f;
    l.inv_df = 0.f;
    l.norm = (float)(0.5 * log(2.0 * pi) + log(cfg.lik_scale));
    l.g_scale = (float)(1.0 / cfg.lik_scale);
    l.l_scale = -0.5f;
  }
  return l;
}
static PriorParams make_prior(const mcmc_b200_config& cfg) {
  PriorParams p;
  const double pi = 3.14159265358979323846;
  p.neg_inv_s2 = (float)(-1.0 / (cfg.prior_scale * cfg.prior_scale));
  p.inv_s = (float)(1.0 / cfg.prior_scale);
  p.norm = (float)(0.5 * log(2.0 * pi) + log(cfg.prior_scale));
  return p;
}

static int make_tensor_map(mcmc_b200_ctx* c) {
  typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                               CUtensorMapFloatOOBfill);
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qres;
  CK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
  if (!fn || qres != cudaDriverEntryPointSuccess)
    return fail(MCMC_B200_ERR_CUDA, "cuTensorMapEncodeTiled not available");
  // [W * rows_pad][24] floats; the box is 32 floats wide so that a staged row
  // is a full 128-byte swizzle span: columns 24..31 are out of bounds and
  // arrive as zeros without being read.
  cuuint64_t gdim[2] = {(cuuint64_t)KP, (cuuint64_t)((long long)c->W * c->rows_pad)};
  cuuint64_t gstride[1] = {(cuuint64_t)(KP * sizeof(float))};
  cuuint32_t box[2] = {32, (cuuint32_t)(c->cfg.H == 128 ? WIDE_TILE : TF32_TILE)};
  cuuint32_t estr[2] = {1, 1};
  // 32-byte-chunk swizzle: the layout the tensor core wants for MN-major TF32 operands; 16-byte-chunk: K-major ones
  const CUtensorMapSwizzle swizzle[2] = {CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_SWIZZLE_128B};
  for (int k = 0; k < (c->cfg.H == 128 ? 2 : 1); ++k) {
    CUresult r = ((EncodeFn)fn)(&c->tmaps[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, c->xaug, gdim, gstride, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle[k], CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
      char b[96];
      snprintf(b, sizeof b, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
      return fail(MCMC_B200_ERR_CUDA, b);
    }
  }
  return MCMC_B200_OK;
}

// Cuts the flattened (window, tile) list of a launch into one contiguous range per CTA and each
// range into per-window segments; slot = the segment's index among its window's segments.
struct WorkPlan {
  std::vector<int> seg_ptr, nslot;
  std::vector<int4> segs;
  bool ints = false;  // FP32: sums over rows by integers
};
static void plan_work_table(int windows, long long tiles_per_window, int max_ctas, int chunks_per_window, double seg_cost,
                            WorkPlan& plan);
static int upload_work_table(mcmc_b200_ctx* c, const WorkPlan& plan, int** d_seg_ptr, int4** d_segs, int** d_nslot,
                             int* n_ctas, int* max_slots);

static cudaError_t launch_resident(mcmc_b200_ctx* c, int cluster, const ResidentParams& g, cudaStream_t st,
                                   int* max_clusters = nullptr) {
  if (!max_clusters && c->refuse > 0) {
    --c->refuse;
    return cudaErrorCooperativeLaunchTooLarge;
  }
  return (c->cfg.precision == MCMC_B200_PREC_TF32 ? launch_resident_tf32 : launch_resident_fp32)(
      cluster, c->tmaps, g, st, max_clusters);
}
static cudaError_t launch_resident_eval(mcmc_b200_ctx* c, const ResidentEvalParams& g, cudaStream_t st) {
  if (c->refuse > 0) {
    --c->refuse;
    return cudaErrorCooperativeLaunchTooLarge;
  }
  return (c->cfg.precision == MCMC_B200_PREC_TF32 ? launch_resident_eval_tf32 : launch_resident_eval_fp32)(c->tmaps, g, st);
}
// Clusters of 1 << i CTAs that can be resident.  Asked once per device and kernel, and only when a plan wants to know:
// the first question loads the kernel, which costs milliseconds.
static int resident_max_clusters(mcmc_b200_ctx* c, int i) {
  static std::mutex mutex;
  static int known[2][64][4];
  static bool asked[2][64][4] = {};
  const int k = c->cfg.precision == MCMC_B200_PREC_TF32, d = c->device & 63;
  std::lock_guard<std::mutex> lock(mutex);
  if (!asked[k][d][i]) {
    if (launch_resident(c, 1 << i, c->res, nullptr, &known[k][d][i]) != cudaSuccess) {
      cudaGetLastError();
      known[k][d][i] = 0;
    }
    asked[k][d][i] = true;
  }
  return known[k][d][i];
}

// What a plan counts on at most: the clusters of 1, 2, 4 and 8 CTAs that every B200 measured holds at once.  So a plan
// follows from precision, windows and rows alone, and a chain has the same bits on every GPU that holds as many.
constexpr int RES_CLUSTERS[4] = {148, 74, 33, 15};

// How a window is dealt to clusters when `windows` of them share the GPU (resident.cuh); available(i): clusters of 1 << i
// CTAs that can be resident.  False when the rows do not fit.
//   * one cluster per window, of the most CTAs (8, 4, 2, 1) that every window can have, if that holds the rows: the
//     exchange then never leaves the cluster;
//   * rows that one cluster of 8 cannot hold: as many clusters of 8 as every window can have (up to 16) while each
//     CTA still has at least four 32-row units (below that the step is all exchange and more CTAs only add to it).  FP32:
//     as many as leave it at most four, since a fifth unit costs its scheduler a second round.
//   * FP32 chains of more than RES_SPREAD units on one cluster: on several, if that leaves a CTA four units or one had 15 or 16
//     (explicit calls keep one cluster: a call is as long as its launch and copies).
// us a step by clusters, TF32: 4096 rows 4.2 (1), 4.2 (8); 4097 rows 3.9 (4, taken), 4.0 (5); 6000 rows 4.2 (3), 4.1 (5, taken),
// 4.1 (6), 4.6 (15); 16384 rows 5.4 (4), 4.5 (8), 4.8 (15, taken): the rule is not the best one there (8 and 15 clusters both give a CTA two
// 128-row tiles).  FP32, one cluster and several: 2048 rows 5.1, 5.2 (2); 2560 5.56, 5.46 (3); 3000 5.77, 5.49; 4096 6.81, 5.51 (4); four
// windows of 4096 6.83, 6.23 (3 each, six units a CTA); seven of 2100, 3000 and 4096 5.55, 5.80, 6.83 and 6.09, 6.21, 6.39 (2 each).  Several:
// 4097 rows 5.55 (5), 16384 6.3, 30000 6.6, 58368 8.3 (15); four units against five when tiles took twice as long: 6000 rows 6.7 (6), 8.1 (5).
// Against one launch per step (one B200, 1 to 148 windows of 100 to 61440 rows that fit, 10-step iterations): 1.13 (FP32, one window of
// 4096 rows when it took 8.2 us a step; 58368 rows 9.9 and 14.6) to 3.2 times as fast, so every window that fits goes this way.
constexpr int RES_SPREAD = 80;
template <typename F>
static bool resident_plan(long long rows, int windows, int num_sms, bool fp32, bool chain, F available, int* cluster, int* clusters) {
  const long long units = (rows + 31) / 32;
  auto count = [&](int i) { return std::min(RES_CLUSTERS[i], available(i)); };
  if ((long long)windows * ((units + RES_UNITS - 1) / RES_UNITS) > num_sms) return false;
  const long long share = windows <= RES_CLUSTERS[3] / 2 ? std::min<long long>(count(3) / windows, RES_MAX_CLUSTERS) : 1;
  const bool spread = fp32 && chain && units > RES_SPREAD && share > 1 && (share >= (units + 31) / 32 || units > 112);
  for (int i = 3; i >= 0 && !spread; --i)
    if (units <= (long long)RES_UNITS << i && windows <= RES_CLUSTERS[i] && windows <= count(i)) {
      *cluster = 1 << i;
      *clusters = 1;
      return true;
    }
  const long long need = (units + 8 * RES_UNITS - 1) / (8 * RES_UNITS);
  if (need * windows > RES_CLUSTERS[3]) return false;
  const long long have = std::min<long long>(count(3) / windows, RES_MAX_CLUSTERS);
  if (need > have) return false;
  *cluster = 8;
  *clusters = (int)std::max(need, std::min(have, (units + (fp32 ? 31 : 0)) / 32));
  return true;
}

// 16-byte words of one rank and cluster through L2 (resident.cuh: STR)
static size_t resident_words_stride(int P, int cluster) {
  const size_t words = (size_t)(P + 5) / 3;
  return ((words + cluster - 1) / cluster + 7) / 8 * 8;
}

// enough for any plan of the context: only windows of several clusters of eight send such words
static size_t resident_msg_bytes(const mcmc_b200_ctx* c, int windows) {
  const int clusters = std::min(RES_CLUSTERS[3] / windows, RES_MAX_CLUSTERS);
  if (clusters < 2 || c->rows <= (c->cfg.precision == MCMC_B200_PREC_FP32 ? RES_SPREAD : 8 * RES_UNITS) * 32) return 0;
  return (size_t)2 * windows * clusters * 8 * resident_words_stride(c->P, 8) * 16;
}

// Prepares the resident launches of a context and allocates their message buffers.  A fixed `slices` asks for bits
// that do not depend on what shares the launch: such contexts keep one launch per step.
static int resident_setup(mcmc_b200_ctx* c) {
  const char* off = getenv("MCMC_B200_NO_MULTISTEP");
  if ((off && off[0] == '1') || c->cfg.slices > 0 || c->cfg.H != 40)
    return MCMC_B200_OK;
  c->res_try = true;
  for (int k = 0; k < 2; ++k) {
    ResidentParams& g = k ? c->res_x : c->res;
    memset(&g, 0, sizeof g);
    g.windows = k ? 1 : c->W;
    if (g.windows > RES_CLUSTERS[0]) continue;
    g.n_rows = (int)c->rows;
    g.rows_pad = (int)c->rows_pad;
    g.Pp = c->Pp;
    g.xaug = c->xaug;
    g.lik = make_lik(c->cfg);
    g.prior = make_prior(c->cfg);
    g.status = c->status;
    g.wait_ticks = RES_WAIT_TICKS;
    int r = dalloc(c, (void**)&g.seq, (size_t)g.windows * 4);
    const size_t bytes = resident_msg_bytes(c, g.windows);
    if (r == MCMC_B200_OK && bytes > 0) r = dalloc(c, (void**)&g.msg, bytes);
    if (r) return r;
  }
  return MCMC_B200_OK;
}

// Leapfrog steps of one resident launch: about a tenth of a second, so that other work on the GPU gets its turn.
// Longer trajectories take one launch per step.
static int resident_max_steps(const mcmc_b200_ctx* c) { return c->cfg.precision == MCMC_B200_PREC_TF32 ? 20000 : 10000; }

// Whether trajectories of L steps are resident launches: those of the chain, or of the explicit calls (x)
static bool use_resident(mcmc_b200_ctx* c, bool x, int L) {
  if (!c->res_try || c->comm || c->oneshot || L > resident_max_steps(c)) return false;
  bool &asked = x ? c->res_x_asked : c->res_asked, &ok = x ? c->res_x_ok : c->res_ok;
  if (!asked) {
    ResidentParams& g = x ? c->res_x : c->res;
    ok = resident_plan(c->rows, g.windows, c->num_sms, c->cfg.precision == MCMC_B200_PREC_FP32, !x,
                       [&](int i) { return resident_max_clusters(c, i); }, x ? &c->res_x_cluster : &c->res_cluster, &g.clusters);
    asked = true;
  }
  return ok;
}

API int mcmc_b200_resident_plan(mcmc_b200_ctx* c, int explicit_calls, int* ctas_per_cluster, int* clusters) {
  if (!c || !ctas_per_cluster || !clusters) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CK(cudaSetDevice(c->device));
  const bool x = explicit_calls != 0, on = use_resident(c, x, x ? 1 : c->cfg.leapfrog_steps);
  *ctas_per_cluster = !on ? 0 : x ? c->res_x_cluster : c->res_cluster;
  *clusters = !on ? 0 : x ? c->res_x.clusters : c->res.clusters;
  return MCMC_B200_OK;
}

API int mcmc_b200_plan_resident_for(int precision, int windows, int64_t rows, int num_sms, const int32_t available[4],
                                    int32_t* ctas_per_cluster, int32_t* clusters) {
  if ((precision != MCMC_B200_PREC_FP32 && precision != MCMC_B200_PREC_TF32) || windows < 1 || rows < 1 || num_sms < 1 ||
      !available || !ctas_per_cluster || !clusters)
    return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  int C = 0, K = 0;
  if (!resident_plan(rows, windows, num_sms, precision == MCMC_B200_PREC_FP32, true, [&](int i) { return available[i]; }, &C, &K))
    C = K = 0;
  *ctas_per_cluster = C;
  *clusters = K;
  return MCMC_B200_OK;
}
API int mcmc_b200_plan_resident(int windows, int64_t rows, int num_sms, const int32_t available[4],
                                int32_t* ctas_per_cluster, int32_t* clusters) {
  return mcmc_b200_plan_resident_for(MCMC_B200_PREC_TF32, windows, rows, num_sms, available, ctas_per_cluster, clusters);
}

// What a segment costs besides its tiles, in tiles.
// TF32 (a tile is 0.53 us): 25-window step 0.5135 ms (8) -> 0.5063 (11) -> 0.5035 (14), flat up to 24; 13 windows 0.284 -> 0.282;
// 50, 100 and 200 windows unchanged within 0.5 %
// FP32, 40 units (a tile is 1.4 us): 200 windows of 2000 rows 45.1 us a step (3), 46.6 (5, 8, 12); 100 of 10000 rows 89.5, 90.1,
// 93.4, 97.7; 25 of 58368 rows 123.0 (3, 5), 125.1
// ... by integers (1.1 us): 200 of 4000 rows 71.3 (3), 69.5 (4.5), 69.3 (6), 60 of 8000 43.9, 41.8, 41.1, 40 of 20000 62.8, 60.9, 59.8 (9:
// 60.0), 25 of 58368 101.6, 100.1, 99.5 (9: 99.3)
constexpr double TF32_SEG_COST = 14.0, FP32_SEG_COST = 3.0, FP32_INT_SEG_COST = 6.0;
constexpr int FP32_START = 3;  // FP32 without a table: a CTA

// CTAs per window of the FP32 kernel without a table.  All CTAs of a launch take the same time: what counts is how many rounds
// of the GPU they make, and how many tiles the longest CTA of a round has; a CTA's start and end cost FP32_START tiles.
// The fewest that come to the least: partial vectors have to be summed.
static int fp32_slices(int windows, long long n_tiles, long long capacity) {
  long long best = 0, at = 1;
  for (long long k = 1; k <= std::min<long long>(n_tiles, MAX_SLICES) && (k == 1 || k * windows <= 4 * capacity); ++k) {
    const long long cost = (k * windows + capacity - 1) / capacity * ((n_tiles + k - 1) / k + FP32_START);
    if (k == 1 || cost < best) {
      best = cost;
      at = k;
    }
  }
  return (int)at;
}

// FP32, 40 units: whether the kernel without the tensor core is the faster one.  Its CTAs are light and there are three to an SM, the other
// kernel has one, and every segment costs it 5 us whatever its rows.  Few tiles in all: fp32_few_tiles.  Else both times are estimated, us:
//   with: 2 + 1.53 x the longest CTA's tiles, a segment counted as FP32_SEG_COST more (off by 1.7 % on average);
//   without: (6 + 5.4 x a CTA's tiles) x rounds of the GPU + 0.2 x slices.  The last round of several is shorter, and so is one that gives
//   every SM the same one or two CTAs (2.7 %).
// Measured with 20 to 2000 windows of 1 to 16 tiles, 189 shapes: what the rule takes is 0.04 % slower on average than the faster kernel,
// 2.1 % at most (444 windows of 10 tiles: 60.9 us a step, 59.7 with the tensor core).  Without / with: 200 windows of 6 tiles 22.7 / 24.7,
// 400 of 6 39.3 / 41.6, 888 of 8 96.0 / 101.3, 2000 of 10 262 / 272; 149 of 6 22.5 / 22.0, 250 of 5 32.3 / 25.4, 600 of 7 71.5 / 68.3,
// 888 of 12 137 / 135
static bool fp32_plain_faster(int windows, long long tiles, int num_sms, const WorkPlan& plan) {
  if (windows * tiles <= num_sms) return false;
  double longest = 0;
  for (size_t b = 0; b + 1 < plan.seg_ptr.size(); ++b) {
    double t = 0;
    for (int i = plan.seg_ptr[b]; i < plan.seg_ptr[b + 1]; ++i) t += plan.segs[i].z - plan.segs[i].y + FP32_SEG_COST;
    longest = std::max(longest, t);
  }
  const long long capacity = 3ll * num_sms;
  const int k = fp32_slices(windows, tiles, capacity);
  const long long full = (long long)k * windows / capacity, rest = (long long)k * windows % capacity;
  double rounds = full;
  if (rest && full) rounds += std::min(1.0, 0.26 / (full * full) + (double)rest / capacity);
  else if (rest) rounds = rest % num_sms == 0 ? 0.78 : 1.0;
  return (6.0 + 5.4 * ((tiles + k - 1) / k)) * rounds + 0.2 * k <= 2.0 + 1.53 * longest;
}

// FP32, 40 units: whether the sums over rows go by integers (grad_fp32_int.cu): a tile takes 1.1 us then instead of 1.39, a segment
// 5 us instead of 3.  us a step, integers and FFMA, by tiles of a segment in the mean: 1 x 100000 rows (5) 18.5, 17.4; 200 x 2000 (9) 44.7, 43.4;
// 4 x 58368 (12) 28.1, 26.9; 200 x 3000 (14) 57.6, 58.4; 60 x 8000 (18) 42.9, 44.1; 200 x 4000 (18) 69.5, 74.0; 6 x 58368 (18) 30.6, 34.8;
// 149 x 5000 (20) 61.1, 68.2; 1 x 400000 (21) 34.9, 39.8; 16 x 40013 (31) 47.1, 57.1; 30 x 62000 (82) 122, 145
// These are both kernels' times, when the line was drawn, with the FFMA kernel's table; the other one gets its own afterwards (FP32_INT_SEG_COST: 60 x 8000
// 41.4, 200 x 4000 66.9, 6 x 58368 31.1, 16 x 40013 46.8).
static void plan_ints(int windows, long long tiles, int num_sms, int slices, WorkPlan& plan) {
  plan.ints = windows * tiles >= 16 * (long long)plan.segs.size();
  if (plan.ints) plan_work_table(windows, tiles, num_sms, slices, FP32_INT_SEG_COST, plan);
}

// The work table of a launch over `windows` windows; false: that of the FP32 kernel without one.  With fixed `slices` FP32 has a table
// always (40 units): bits must not depend on the number of windows.
static bool plan_gradient(bool tf32, int H, int windows, long long tiles, int num_sms, int slices, WorkPlan& plan) {
  if (!tf32 && (H != SPLIT_H || (slices == 0 && fp32_few_tiles(windows * tiles)))) return false;
  plan_work_table(windows, tiles, num_sms, slices, tf32 ? TF32_SEG_COST : FP32_SEG_COST, plan);
  if (tf32) return true;
  if (slices == 0 && fp32_plain_faster(windows, tiles, num_sms, plan)) return false;
  plan_ints(windows, tiles, num_sms, slices, plan);
  return true;
}

API int mcmc_b200_create(const mcmc_b200_config* cfg, int device, int n_windows, int64_t rows,
                         mcmc_b200_ctx** out) {
  if (!cfg || !out || n_windows < 1 || rows < 1) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  if (cfg->D != 22) return fail(MCMC_B200_ERR_UNSUPPORTED, "only D = 22 is built");
  if (cfg->H != 40 && cfg->H != 128) return fail(MCMC_B200_ERR_UNSUPPORTED, "only H = 40 or 128 is built");
  if (cfg->precision == MCMC_B200_PREC_TF32 && !tf32_supported(cfg->H))
    return fail(MCMC_B200_ERR_UNSUPPORTED, "the TF32 path is not built for this hidden width");
  if (cfg->leapfrog_steps < 1 || cfg->lik_scale <= 0 || cfg->prior_scale <= 0)
    return fail(MCMC_B200_ERR_INVALID, "bad sampler/model constants");
  if (cfg->rng_streams != MCMC_B200_RNG_PHILOX && cfg->rng_streams != MCMC_B200_RNG_REFERENCE)
    return fail(MCMC_B200_ERR_INVALID, "rng_streams must be MCMC_B200_RNG_PHILOX or MCMC_B200_RNG_REFERENCE");
  if (n_windows > 65535) return fail(MCMC_B200_ERR_INVALID, "at most 65535 windows per context");
  {
    // the kernels index rows of the whole context with 32-bit integers (TMA coordinates, tile numbers)
    const long long rp = (rows + TF32_TILE - 1) / TF32_TILE * TF32_TILE;
    if (rows > 0x7fffffffLL - TF32_TILE || rp * (long long)n_windows > 0x7fffffffLL)
      return fail(MCMC_B200_ERR_INVALID, "rows per window x windows must stay below 2^31 rows per context");
  }
  int ndev = 0;
  cudaError_t e0 = cudaGetDeviceCount(&ndev);
  if (e0 != cudaSuccess || ndev == 0)
    return fail(MCMC_B200_ERR_CUDA, "no CUDA device: this library has no CPU path");
  if (device < 0 || device >= ndev) return fail(MCMC_B200_ERR_INVALID, "device ordinal out of range");
  CK(cudaSetDevice(device));
  int cc_major = 0, sm_count = 0;  // (two attributes: the whole property record takes milliseconds)
  CK(cudaDeviceGetAttribute(&cc_major, cudaDevAttrComputeCapabilityMajor, device));
  CK(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
  if (cc_major != 10)
    return fail(MCMC_B200_ERR_UNSUPPORTED, "kernels are built for sm_100a (B200) only");

  mcmc_b200_ctx* c = new mcmc_b200_ctx();
  c->cfg = *cfg;
  c->device = device;
  c->W = n_windows;
  c->rows = rows;
  c->rows_pad = (rows + TF32_TILE - 1) / TF32_TILE * TF32_TILE;
  c->P = cfg->D * cfg->H + 2 * cfg->H + 1;
  c->Pp = (c->P + 3) / 4 * 4;
  c->num_sms = sm_count;
  const bool tf32 = cfg->precision == MCMC_B200_PREC_TF32;
  c->tile_rows = tf32 ? TF32_TILE : fp32_tile_rows(cfg->H);
  const long long n_tiles = c->rows_pad / c->tile_rows;
  c->window_set.assign(n_windows, 0);
  c->h_gwin.assign(n_windows, 0);
  cudaError_t es = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
  if (es != cudaSuccess) { delete c; return fail(MCMC_B200_ERR_CUDA, "cudaStreamCreate failed"); }
  WorkPlan plan;
  c->table = plan_gradient(tf32, cfg->H, n_windows, n_tiles, sm_count, cfg->slices, plan);
  c->ctas_per_sm = c->table ? 1 : std::max(1, fp32_max_ctas_per_sm(cfg->H));
  if (c->table) {
    // persistent kernels: by default every CTA gets an equal share of the launch's tiles, so where a
    // window is cut depends on how many windows share the launch.  cfg.slices > 0 instead cuts every
    // window into that many fixed chunks (whole chunks per CTA): a window's result is then bit-identical
    // wherever and with whatever else it runs, at some cost in load balance.
    int r_ = upload_work_table(c, plan, &c->tab_seg_ptr, &c->tab_segs, &c->tab_nslot, &c->tab_ctas, &c->slices);
    c->tab_ints = plan.ints;
    if (r_ == MCMC_B200_OK) {
      WorkPlan one;
      plan_work_table(1, n_tiles, c->num_sms, cfg->slices, tf32 ? TF32_SEG_COST : FP32_SEG_COST, one);
      if (!tf32) plan_ints(1, n_tiles, c->num_sms, cfg->slices, one);
      r_ = upload_work_table(c, one, &c->xtab_seg_ptr, &c->xtab_segs, &c->xtab_nslot, &c->xtab_ctas, &c->slices_x);
      c->xtab_ints = one.ints;
    }
    if (r_ != MCMC_B200_OK) { mcmc_b200_destroy(c); return r_; }
  } else {
    const long long capacity = (long long)c->num_sms * c->ctas_per_sm;
    long long s = cfg->slices > 0 ? cfg->slices : fp32_slices(n_windows, n_tiles, capacity);
    if (s > n_tiles) s = n_tiles;
    if (s > MAX_SLICES) s = MAX_SLICES;
    c->slices = (int)s;
    long long sx = cfg->slices > 0 ? cfg->slices : fp32_slices(1, n_tiles, capacity);
    if (sx > n_tiles) sx = n_tiles;
    if (sx > MAX_SLICES) sx = MAX_SLICES;
    c->slices_x = (int)sx;
  }

  // many slots per window (few windows per GPU): one small launch sums them once per step instead of
  // every CTA of the next launch summing all of them in its prologue
  c->use_red = c->slices > 4;
  c->use_red_x = c->slices_x > 4;
  const size_t W = n_windows, Pp = c->Pp, P = c->P;
  DA(c->xaug, W * c->rows_pad * KP * sizeof(float));
  for (int i = 0; i < 2; ++i) {
    DA(c->wbuf[i], W * Pp * 4);
    DA(c->mbuf[i], W * Pp * 4);
    DA(c->partial[i], W * c->slices * Pp * 4);
    DA(c->llp[i], W * c->slices * 8);
    DA(c->xw[i], Pp * 4);
    DA(c->xm[i], Pp * 4);
    DA(c->xpartial[i], (size_t)c->slices_x * Pp * 4);
    DA(c->xllp[i], (size_t)c->slices_x * 8);
  }
  DA(c->w_cur, W * Pp * 4);
  DA(c->g_cur, W * Pp * 4);
  DA(c->m0, W * Pp * 4);
  DA(c->red, W * (Pp + 4) * 8);
  DA(c->xred, (Pp + 4) * 8);
  DA(c->ll_cur, W * 8);
  DA(c->lp_cur, W * 8);
  DA(c->eps, W * 4);
  DA(c->iter, W * 4);
  DA(c->n_accept, W * 4);
  DA(c->gwin, W * 8);
  DA(c->status, 4);
  DA(c->xg, Pp * 4);
  DA(c->g_out, Pp * 4);
  DA(c->row_loss, (size_t)c->rows_pad * 4);
  DA(c->scalars, 4 * 8);
  if (cfg->sample_capacity > 0) {
    int r_ = dalloc(c, (void**)&c->samples, W * (size_t)cfg->sample_capacity * P * 4, false);
    if (r_ != MCMC_B200_OK) { mcmc_b200_destroy(c); return r_; }
  }
  if (cfg->trace_iters > 0) {
    const size_t K = cfg->trace_iters;
    DA(c->tr_mom, W * K * P * 4);
    DA(c->tr_log_u, W * K * 4);
    DA(c->tr_log_acpt, W * K * 8);
    DA(c->tr_accept, W * K * 4);
    DA(c->tr_eps, W * K * 4);
  }
  if (tf32) {
    int r_ = make_tensor_map(c);
    if (r_ != MCMC_B200_OK) { mcmc_b200_destroy(c); return r_; }
  }
  {
    int r_ = resident_setup(c);
    if (r_ != MCMC_B200_OK) { mcmc_b200_destroy(c); return r_; }
  }
  c->hb = host_block_take();
  if (!c->hb) {
    mcmc_b200_destroy(c);
    return fail(MCMC_B200_ERR_NOMEM, "cudaHostAlloc failed");
  }
  memset(c->hb, 0, sizeof(HostBlock));
  std::vector<float> e(W, (float)cfg->eps0);
  cudaError_t e_end = cudaMemcpyAsync(c->eps, e.data(), W * 4, cudaMemcpyHostToDevice, c->stream);
  if (e_end == cudaSuccess) e_end = cudaStreamSynchronize(c->stream);
  if (e_end != cudaSuccess) {
    mcmc_b200_destroy(c);
    return fail(MCMC_B200_ERR_CUDA, std::string("context set-up: ") + cudaGetErrorString(e_end));
  }
  *out = c;
  return MCMC_B200_OK;
}

// Host-only planner of the persistent kernels' work table: which (window, tile range, slot) segments each
// CTA owns.  Pure arithmetic (no CUDA): also exported for inspection and CPU tests.
static void plan_work_table(int windows, long long tiles_per_window, int max_ctas, int chunks_per_window, double seg_cost,
                            WorkPlan& plan) {
  std::vector<int>&seg_ptr = plan.seg_ptr, &nslot = plan.nslot;
  std::vector<int4>& segs = plan.segs;
  const long long T = (long long)windows * tiles_per_window;
  seg_ptr.clear();
  segs.clear();
  nslot.assign(windows, 0);
  long long G;
  if (chunks_per_window > 0) {
    long long cpw = std::min<long long>(std::min<long long>(chunks_per_window, tiles_per_window), MAX_SLICES);
    const long long NC = (long long)windows * cpw;
    G = std::min<long long>(max_ctas, NC);
    seg_ptr.assign(G + 1, 0);
    for (long long b = 0; b < G; ++b) {
      seg_ptr[b] = (int)segs.size();
      for (long long ch = b * NC / G; ch < (b + 1) * NC / G; ++ch) {
        const long long w = ch / cpw, k = ch % cpw;
        segs.push_back(make_int4((int)w, (int)(k * tiles_per_window / cpw), (int)((k + 1) * tiles_per_window / cpw),
                                 (int)k));
        nslot[w] = (int)cpw;
      }
    }
  } else {
    // Contiguous ranges of the flattened (window, tile) list, balanced by COST rather than by tile
    // count: every segment a CTA starts (a new window inside its range) costs a fixed prologue + drain +
    // read-out, worth about `seg_cost` tiles.  A CTA whose range crosses a window boundary therefore
    // gets fewer tiles than one that stays inside a window.  The smallest per-CTA budget that covers
    // all tiles with at most max_ctas CTAs is found by bisection over a greedy walk.
    const long long tpw = tiles_per_window;
    const long long Gmax = std::max<long long>(1, std::min<long long>(max_ctas, T));
    auto walk = [&](double budget_per_cta, bool emit) -> long long {
      long long pos = 0, used = 0;
      while (pos < T) {
        if (emit) seg_ptr.push_back((int)segs.size());
        double budget = budget_per_cta;
        bool first = true;
        while (pos < T) {
          long long can = (long long)std::floor(budget - seg_cost + 1e-9);
          if (can < 1) {
            if (!first) break;
            can = 1;  // a CTA always takes at least one tile
          }
          const long long w = pos / tpw;
          const long long take = std::min(can, (w + 1) * tpw - pos);
          if (emit)
            segs.push_back(make_int4((int)w, (int)(pos - w * tpw), (int)(pos + take - w * tpw), nslot[w]++));
          pos += take;
          budget -= seg_cost + (double)take;
          first = false;
        }
        if (++used > 4 * Gmax + 16) break;  // cannot happen for a budget >= the lower bound
      }
      return used;
    };
    double lo = (double)T / (double)Gmax, hi = (double)T / (double)Gmax + seg_cost * ((double)(T / Gmax) / tpw + 3.0) + 2.0;
    while (walk(hi, false) > Gmax) hi *= 1.5;
    for (int it = 0; it < 48; ++it) {
      const double mid = 0.5 * (lo + hi);
      if (walk(mid, false) <= Gmax) hi = mid; else lo = mid;
    }
    G = walk(hi, true);
  }
  seg_ptr.resize(G + 1);
  seg_ptr[G] = (int)segs.size();
}

static int upload_work_table(mcmc_b200_ctx* c, const WorkPlan& plan, int** d_seg_ptr, int4** d_segs, int** d_nslot,
                             int* n_ctas, int* max_slots) {
  const std::vector<int>&seg_ptr = plan.seg_ptr, &nslot = plan.nslot;
  const std::vector<int4>& segs = plan.segs;
  const long long G = (long long)seg_ptr.size() - 1;
  int ms = 1;
  for (int n : nslot) ms = std::max(ms, n);
  int r = dalloc(c, (void**)d_seg_ptr, seg_ptr.size() * sizeof(int), false);
  if (r == MCMC_B200_OK) r = dalloc(c, (void**)d_segs, segs.size() * sizeof(int4), false);
  if (r == MCMC_B200_OK) r = dalloc(c, (void**)d_nslot, nslot.size() * sizeof(int), false);
  if (r != MCMC_B200_OK) return r;
  CK(cudaMemcpy(*d_seg_ptr, seg_ptr.data(), seg_ptr.size() * sizeof(int), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(*d_segs, segs.data(), segs.size() * sizeof(int4), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(*d_nslot, nslot.data(), nslot.size() * sizeof(int), cudaMemcpyHostToDevice));
  *n_ctas = (int)G;
  *max_slots = ms;
  return MCMC_B200_OK;
}

API int mcmc_b200_plan_work_table_for(int precision, int H, int windows, int64_t tiles_per_window, int num_sms, int slices,
                                      int32_t* seg_ptr_out, int seg_ptr_capacity, int32_t* segs_out,
                                      int segs_capacity, int32_t* n_ctas, int32_t* n_segs) {
  if (windows < 1 || tiles_per_window < 1 || num_sms < 1 || slices < 0 || !n_ctas || !n_segs ||
      (precision != MCMC_B200_PREC_FP32 && precision != MCMC_B200_PREC_TF32))
    return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  WorkPlan plan;
  if (!plan_gradient(precision == MCMC_B200_PREC_TF32, H, windows, tiles_per_window, num_sms, slices, plan)) {
    *n_ctas = *n_segs = 0;
    return MCMC_B200_OK;
  }
  const std::vector<int>& seg_ptr = plan.seg_ptr;
  const std::vector<int4>& segs = plan.segs;
  *n_ctas = (int32_t)seg_ptr.size() - 1;
  *n_segs = (int32_t)segs.size();
  if (seg_ptr_out) {
    if ((int)seg_ptr.size() > seg_ptr_capacity) return fail(MCMC_B200_ERR_INVALID, "seg_ptr_out too small");
    for (size_t i = 0; i < seg_ptr.size(); ++i) seg_ptr_out[i] = seg_ptr[i];
  }
  if (segs_out) {
    if ((int)segs.size() > segs_capacity) return fail(MCMC_B200_ERR_INVALID, "segs_out too small");
    for (size_t i = 0; i < segs.size(); ++i) {
      segs_out[4 * i] = segs[i].x;
      segs_out[4 * i + 1] = segs[i].y;
      segs_out[4 * i + 2] = segs[i].z;
      segs_out[4 * i + 3] = segs[i].w;
    }
  }
  return MCMC_B200_OK;
}
API int mcmc_b200_plan_work_table(int windows, int64_t tiles_per_window, int max_ctas, int slices,
                                  int32_t* seg_ptr_out, int seg_ptr_capacity, int32_t* segs_out,
                                  int segs_capacity, int32_t* n_ctas, int32_t* n_segs) {
  return mcmc_b200_plan_work_table_for(MCMC_B200_PREC_TF32, SPLIT_H, windows, tiles_per_window, max_ctas, slices, seg_ptr_out,
                                       seg_ptr_capacity, segs_out, segs_capacity, n_ctas, n_segs);
}

API void mcmc_b200_destroy(mcmc_b200_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  if (c->copies) cudaStreamSynchronize(c->copies);
  if (c->graph_exec) cudaGraphExecDestroy(c->graph_exec);
  for (void* p : c->os_peer_blocks)
    if (p) cudaIpcCloseMemHandle(p);
  if (c->comm && g_nccl.ok) g_nccl.CommDestroy(c->comm);
  for (void* p : c->allocs) cudaFree(p);
  if (c->hb) host_block_give(c->hb);
  for (cudaEvent_t e : c->copy_events)
    if (e) cudaEventDestroy(e);
  if (c->copies) cudaStreamDestroy(c->copies);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

API int mcmc_b200_num_params(const mcmc_b200_ctx* c) { return c ? c->P : -1; }
API void* mcmc_b200_stream(mcmc_b200_ctx* c) { return c ? (void*)c->stream : nullptr; }

static int finish_status(mcmc_b200_ctx* c);
static int check_status(mcmc_b200_ctx* c) {
  CK(cudaMemcpyAsync(&c->hb->status, c->status, 4, cudaMemcpyDeviceToHost, c->stream));
  return finish_status(c);
}
// waits for the context's stream and reports the status word that has arrived in the host block
static int finish_status(mcmc_b200_ctx* c) {
  CK(cudaStreamSynchronize(c->stream));
  const int st = c->hb->status;
  if (st != 0) {
    // resident launches have done nothing since the report (resident.cuh): none of their words is awaited any more.
    // (Some may be queued on a caller's stream.)
    cudaDeviceSynchronize();
    c->hb->status = 0;
    for (int k = 0; k < 2; ++k)
      if (k ? c->res_x_ok : c->res_ok) {
        const ResidentParams& g = k ? c->res_x : c->res;
        if (g.msg) cudaMemsetAsync(g.msg, 0, resident_msg_bytes(c, g.windows), c->stream);
        cudaMemsetAsync(g.seq, 0, (size_t)g.windows * 4, c->stream);
      }
    cudaMemsetAsync(c->status, 0, 4, c->stream);
    cudaStreamSynchronize(c->stream);
    char b[96];
    snprintf(b, sizeof b, "device-side wait ran out (code %d)", st);
    return fail(MCMC_B200_ERR_TIMEOUT, b);
  }
  return MCMC_B200_OK;
}

API int mcmc_b200_synchronize(mcmc_b200_ctx* c) {
  if (!c) return fail(MCMC_B200_ERR_INVALID, "null context");
  CK(cudaSetDevice(c->device));
  return check_status(c);
}

API int mcmc_b200_philox_device(mcmc_b200_ctx* c, const uint32_t ctr[4], const uint32_t key[2], int n,
                                uint32_t* raw_out, float* normals_out, float* uniform_out) {
  if (!c || !ctr || !key || n < 1 || n > 4096 || !raw_out || !normals_out || !uniform_out)
    return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CK(cudaSetDevice(c->device));
  // scratch of this call: the single-window row-loss buffer is at least 128 floats and is free between calls
  if ((size_t)n * 5 + 1 > (size_t)c->rows_pad) return fail(MCMC_B200_ERR_INVALID, "n too large for this context");
  uint32_t* raw = reinterpret_cast<uint32_t*>(c->row_loss);
  float* normals = c->row_loss + 4 * (size_t)n;
  float* uni = normals + n;
  cudaError_t e = launch_philox_probe(ctr, key, n, raw, normals, uni, c->stream);
  c->launches++;
  if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
  CK(cudaMemcpyAsync(raw_out, raw, (size_t)n * 16, cudaMemcpyDeviceToHost, c->stream));
  CK(cudaMemcpyAsync(normals_out, normals, (size_t)n * 4, cudaMemcpyDeviceToHost, c->stream));
  CK(cudaMemcpyAsync(uniform_out, uni, 4, cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  return MCMC_B200_OK;
}

API int mcmc_b200_selftest_wait_timeout(mcmc_b200_ctx* c, int limit_us) {
  if (!c || limit_us < 20 || limit_us > 1000000) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CK(cudaSetDevice(c->device));
  cudaError_t e = launch_wait_probe(c->status, (unsigned int)(limit_us / 20), c->stream);
  c->launches++;
  if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
  return check_status(c);
}

API int mcmc_b200_set_window_data(mcmc_b200_ctx* c, int window, int64_t global_window, const float* x,
                                  const float* y, int is_device) {
  if (!c || !x || !y || window < 0 || window >= c->W) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CK(cudaSetDevice(c->device));
  const size_t nx = (size_t)c->rows * c->cfg.D, ny = (size_t)c->rows;
  const float *dx = x, *dy = y;
  if (!is_device) {
    if (!c->stage) {
      int r = dalloc(c, (void**)&c->stage, (nx + ny) * 4, false);
      if (r) return r;
    }
    CK(cudaMemcpyAsync(c->stage, x, nx * 4, cudaMemcpyHostToDevice, c->stream));
    CK(cudaMemcpyAsync(c->stage + nx, y, ny * 4, cudaMemcpyHostToDevice, c->stream));
    dx = c->stage;
    dy = c->stage + nx;
  }
  cudaError_t e = launch_repack(dx, dy, c->xaug + (size_t)window * c->rows_pad * KP, c->rows, c->rows_pad,
                                c->cfg.D, c->stream);
  c->launches++;
  if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
  c->h_gwin[window] = global_window;
  c->window_set[window] = 1;
  CK(cudaMemcpyAsync(c->gwin + window, &c->h_gwin[window], 8, cudaMemcpyHostToDevice, c->stream));
  CK(cudaStreamSynchronize(c->stream));  // the caller's buffers are free again on return
  if (window == 0) { c->bound_x = nullptr; c->bound_y = nullptr; }
  return MCMC_B200_OK;
}

// ---- launch helpers ------------------------------------------------------
static GradParams base_grad_params(mcmc_b200_ctx* c) {
  GradParams g;
  memset(&g, 0, sizeof g);
  g.xaug = c->xaug;
  g.window_stride = c->rows_pad * KP;
  g.n_rows = (int)c->rows;
  g.n_tiles = (int)(c->rows_pad / c->tile_rows);
  g.P = c->P;
  g.Pp = c->Pp;
  g.lik = make_lik(c->cfg);
  g.prior = make_prior(c->cfg);
  g.status = c->status;
  g.test_code = c->test_code;
  return g;
}

// `single` selects the single-window work table / slot count (explicit-state calls)
static int launch_grad(mcmc_b200_ctx* c, GradParams g, bool single, cudaStream_t st) {
  cudaError_t e;
  const int slots = single ? c->slices_x : c->slices;
  g.slices_in = slots;
  g.slices_out = slots;
  if (c->table) {
    g.nslot_in = single ? c->xtab_nslot : c->tab_nslot;
    g.seg_ptr = single ? c->xtab_seg_ptr : c->tab_seg_ptr;
    g.segs = single ? c->xtab_segs : c->tab_segs;
    const int ctas = single ? c->xtab_ctas : c->tab_ctas;
    e = c->cfg.precision == MCMC_B200_PREC_TF32 ? launch_grad_tf32(c->cfg.H, c->tmaps, g, ctas, st)
                                                : (single ? c->xtab_ints : c->tab_ints) ? launch_grad_fp32_int(g, ctas, st)
                                                                                        : launch_grad_fp32_split(g, ctas, st);
  } else {
    e = launch_grad_fp32(c->cfg.H, g, slots, single ? 1 : c->W, st);
  }
  c->launches++;
  if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, std::string("gradient kernel launch: ") + cudaGetErrorString(e));
  return MCMC_B200_OK;
}

static int allreduce(mcmc_b200_ctx* c, double* buf, size_t count, cudaStream_t st) {
  int r = g_nccl.AllReduce(buf, buf, count, kNcclFloat64, kNcclSum, c->comm, st);
  if (r != 0)
    return fail(MCMC_B200_ERR_NCCL, std::string("ncclAllReduce: ") +
                                        (g_nccl.GetErrorString ? g_nccl.GetErrorString(r) : "error"));
  return MCMC_B200_OK;
}

// this rank's sums and their all-reduce over peer memory in one launch (row sharding, one window)
static size_t oneshot_block_bytes(const mcmc_b200_ctx* c) {
  return (size_t)2 * c->nranks * (c->Pp + 4) * 2 * sizeof(uint2);  // [2 halves][nranks][Pp + 4][2 words]
}
static int oneshot_allreduce(mcmc_b200_ctx* c, const float* partial, const double* llp, cudaStream_t st) {
  OneShotParams p;
  memset(&p, 0, sizeof p);
  p.partial = partial;
  p.ll_partial = llp;
  p.slices = c->slices;
  p.nslot = c->tab_nslot;
  p.P = c->P;
  p.Pp = c->Pp;
  p.red = c->red;
  p.rank = c->rank;
  p.nranks = c->nranks;
  for (int k = 0; k < c->nranks; ++k) p.peer_words[k] = reinterpret_cast<uint2*>(c->os_base[k]);
  p.local_words = reinterpret_cast<const uint2*>(c->os_block);
  p.seq = c->os_seq;
  p.done = c->os_done;
  p.poll_limit = c->os_poll_limit;
  p.status = c->status;
  cudaError_t e = launch_oneshot_allreduce(p, st);
  c->launches++;
  if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, std::string("one-shot all-reduce launch: ") + cudaGetErrorString(e));
  return MCMC_B200_OK;
}

static AcceptParams base_accept_params(mcmc_b200_ctx* c) {
  AcceptParams a;
  memset(&a, 0, sizeof a);
  a.P = c->P;
  a.Pp = c->Pp;
  a.prior = make_prior(c->cfg);
  a.seed = c->cfg.seed;
  a.ref_streams = c->cfg.rng_streams == MCMC_B200_RNG_REFERENCE;
  a.ref_log_u = c->ref_log_u;
  a.ref_cap = c->ref_cap > 0 ? c->ref_cap : 1;
  return a;
}

// ---- the reference's random streams (main.h:207-216, :235-239): the libraries' own engines ----------
static float refstream_log_uniform(uint64_t seed) {
  // main.h:235-239: a fresh engine per draw, U(FLT_MIN, 1), log() evaluated in double and narrowed
  std::default_random_engine engine;
  engine.seed((std::default_random_engine::result_type)seed);
  std::uniform_real_distribution<float> accept_draw(std::numeric_limits<float>::min(), 1.0f);
  return (float)log((double)accept_draw(engine));
}
API uint32_t mcmc_b200_refstream_engine(uint64_t n_discard) {
  thrust::default_random_engine engine;
  engine.discard(n_discard);
  return (uint32_t)engine();
}
API uint32_t mcmc_b200_refstream_engine0(uint64_t seed) {
  std::default_random_engine engine;
  engine.seed((std::default_random_engine::result_type)seed);
  return (uint32_t)engine();
}
API float mcmc_b200_refstream_log_uniform(uint64_t seed) { return refstream_log_uniform(seed); }

static void drop_graph(mcmc_b200_ctx* c);
// makes the log accept draws of iterations [0, upto) available on the device (absolute iteration index)
static int refstream_fill(mcmc_b200_ctx* c, int upto) {
  if (c->cfg.rng_streams != MCMC_B200_RNG_REFERENCE || upto <= c->ref_filled) return MCMC_B200_OK;
  if (upto > c->ref_cap) {
    const int cap = std::max(upto + 64, c->cfg.burn_in + c->cfg.sample_capacity + 64);
    float* nb = nullptr;
    int r = dalloc(c, (void**)&nb, (size_t)cap * 4, true);  // (the old buffer stays in the context's free list)
    if (r) return r;
    CK(cudaStreamSynchronize(c->stream));
    c->ref_log_u = nb;
    c->ref_cap = cap;
    c->ref_filled = 0;
    drop_graph(c);  // the captured accept launch holds the old pointer
  }
  std::vector<float> h((size_t)(upto - c->ref_filled));
  for (int it = c->ref_filled; it < upto; ++it)
    h[(size_t)(it - c->ref_filled)] = refstream_log_uniform(c->cfg.seed + REF_DRAWS_PER_ITER * (uint64_t)it + 961);
  CK(cudaMemcpyAsync(c->ref_log_u + c->ref_filled, h.data(), h.size() * 4, cudaMemcpyHostToDevice, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  c->ref_filled = upto;
  return MCMC_B200_OK;
}

API int mcmc_b200_refstream_momentum_device(mcmc_b200_ctx* c, uint64_t first_n, int count, float* out) {
  if (!c || !out || count < 1 || (long long)count > c->rows_pad)
    return fail(MCMC_B200_ERR_INVALID, "bad arguments (count is limited to the context's padded row count)");
  CK(cudaSetDevice(c->device));
  cudaError_t e = launch_refstream_momentum(first_n, count, c->row_loss, c->stream);
  c->launches++;
  if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
  CK(cudaMemcpyAsync(out, c->row_loss, (size_t)count * 4, cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  return MCMC_B200_OK;
}

static void fill_chain_accept(mcmc_b200_ctx* c, AcceptParams& a, int mode, int L) {
  a.mode = mode;
  a.slices = c->slices;
  a.nslot = c->tab_nslot;
  const int last = (mode == ACC_BOOTSTRAP) ? 0 : (L - 1) & 1;
  a.partial = c->partial[last];
  a.ll_partial = c->llp[last];
  a.red_in = (c->comm || c->use_red || c->oneshot) ? c->red : nullptr;
  a.w_new = (mode == ACC_BOOTSTRAP) ? c->wbuf[0] : c->wbuf[L & 1];
  a.m_new = (mode == ACC_BOOTSTRAP) ? c->mbuf[0] : c->mbuf[L & 1];
  a.m0 = c->m0;
  a.w_cur = c->w_cur;
  a.g_cur = c->g_cur;
  a.ll_cur = c->ll_cur;
  a.lp_cur = c->lp_cur;
  a.eps = c->eps;
  a.iter = c->iter;
  a.n_accept = c->n_accept;
  a.gwin = c->gwin;
  a.w_start = c->wbuf[0];
  a.m_start = c->mbuf[0];
  a.samples = c->samples;
  a.sample_capacity = c->samples ? c->cfg.sample_capacity : 0;
  a.burn_in = c->cfg.burn_in;
  a.adapt_steps = c->cfg.adapt_steps;
  a.log_target = (float)log(c->cfg.target_rate);
  a.dec_adj = -(float)c->cfg.decrement / (1.f + (float)c->cfg.decrement);
  a.inc_adj = (float)c->cfg.increment;
  a.trace_iters = c->cfg.trace_iters;
  a.tr_mom = c->tr_mom;
  a.tr_log_u = c->tr_log_u;
  a.tr_log_acpt = c->tr_log_acpt;
  a.tr_accept = c->tr_accept;
  a.tr_eps = c->tr_eps;
}

// queue one gradient evaluation for all windows (+ the allreduce when sharded); s: step of the trajectory
static int chain_grad(mcmc_b200_ctx* c, int mode, int s, cudaStream_t st) {
  GradParams g = base_grad_params(c);
  g.mode = mode;
  g.no_loss = mode != MODE_EVAL && s < c->cfg.leapfrog_steps - 1;
  g.w_in = c->wbuf[s & 1];
  g.m_in = c->mbuf[s & 1];
  g.w_out = c->wbuf[(s + 1) & 1];
  g.m_out = c->mbuf[(s + 1) & 1];
  g.g_carried = c->g_cur;
  g.partial_in = c->partial[(s + 1) & 1];
  const bool red = c->comm || c->use_red || c->oneshot;
  g.red_in = (red && mode == MODE_NEXT) ? c->red : nullptr;
  g.partial_out = c->partial[s & 1];
  g.ll_out = c->llp[s & 1];
  g.eps = c->eps;
  int r = launch_grad(c, g, false, st);
  if (r) return r;
  if (c->oneshot) return oneshot_allreduce(c, c->partial[s & 1], c->llp[s & 1], st);
  if (red) {
    cudaError_t e = launch_reduce_partials(c->partial[s & 1], c->llp[s & 1], c->slices, c->tab_nslot, c->P,
                                           c->Pp, c->red, c->W, c->num_sms, st);
    c->launches++;
    if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
    if (c->comm) {
      r = allreduce(c, c->red, (size_t)c->W * (c->Pp + 4), st);
      if (r) return r;
    }
  }
  return MCMC_B200_OK;
}

// Up to n_iter HMC iterations in cooperative launches that keep the rows on the chip; returns how many were queued.  A
// launch that is refused (not all of its CTAs fit into what the stream or the process may use) has done nothing: the
// caller goes on with one launch per step, and an error of another kind shows up there again.
static int resident_chain(mcmc_b200_ctx* c, int n_iter, cudaStream_t st) {
  ResidentParams g = c->res;
  g.mode = RES_CHAIN;
  g.n_steps = c->cfg.leapfrog_steps;
  g.a = base_accept_params(c);
  fill_chain_accept(c, g.a, ACC_ITERATE, g.n_steps);
  const int per_launch = resident_max_steps(c) / g.n_steps;
  int done = 0;
  for (; done < n_iter; done += g.n_iter) {
    g.n_iter = std::min(per_launch, n_iter - done);
    if (launch_resident(c, c->res_cluster, g, st) != cudaSuccess) {
      cudaGetLastError();
      break;
    }
    c->launches++;
  }
  return done;
}

static int queue_iteration(mcmc_b200_ctx* c, cudaStream_t st) {
  const int L = c->cfg.leapfrog_steps;
  for (int s = 0; s < L; ++s) {
    int r = chain_grad(c, s == 0 ? MODE_FIRST : MODE_NEXT, s, st);
    if (r) return r;
  }
  AcceptParams a = base_accept_params(c);
  fill_chain_accept(c, a, ACC_ITERATE, L);
  cudaError_t e = launch_accept(a, c->W, st);
  c->launches++;
  if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
  return MCMC_B200_OK;
}

static int bootstrap(mcmc_b200_ctx* c) {
  for (int w = 0; w < c->W; ++w)
    if (!c->window_set[w]) return fail(MCMC_B200_ERR_INVALID, "a window has no data yet");
  // main.h:52,182-185: the chain starts at w = 0
  const size_t n = (size_t)c->W * c->Pp * 4;
  CK(cudaMemsetAsync(c->wbuf[0], 0, n, c->stream));
  CK(cudaMemsetAsync(c->mbuf[0], 0, n, c->stream));
  CK(cudaMemsetAsync(c->iter, 0, (size_t)c->W * 4, c->stream));
  CK(cudaMemsetAsync(c->n_accept, 0, (size_t)c->W * 4, c->stream));
  std::vector<float> e(c->W, (float)c->cfg.eps0);
  CK(cudaMemcpyAsync(c->eps, e.data(), (size_t)c->W * 4, cudaMemcpyHostToDevice, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  int r = chain_grad(c, MODE_EVAL, 0, c->stream);
  if (r) return r;
  AcceptParams a = base_accept_params(c);
  fill_chain_accept(c, a, ACC_BOOTSTRAP, 1);
  cudaError_t er = launch_accept(a, c->W, c->stream);
  c->launches++;
  if (er != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(er));
  c->bootstrapped = true;
  c->iters_done = 0;
  return MCMC_B200_OK;
}

// The captured iteration graph bakes in the launch sequence (with or without the partial-sum and
// all-reduce launches, one launch per step or one per iteration): whatever changes that sequence drops it.
static void drop_graph(mcmc_b200_ctx* c) {
  if (c->graph_exec) cudaGraphExecDestroy(c->graph_exec);
  c->graph_exec = nullptr;
  c->graph_tried = false;
}

API int mcmc_b200_reset_chain(mcmc_b200_ctx* c) {
  if (!c) return fail(MCMC_B200_ERR_INVALID, "null context");
  CK(cudaSetDevice(c->device));
  CK(cudaStreamSynchronize(c->stream));
  drop_graph(c);
  c->bootstrapped = false;
  c->iters_done = 0;
  return MCMC_B200_OK;
}

API int mcmc_b200_run_chain_async(mcmc_b200_ctx* c, int n_iter) {
  if (!c || n_iter < 0) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CK(cudaSetDevice(c->device));
  if (!c->bootstrapped) {
    int r = bootstrap(c);
    if (r) return r;
  }
  if (n_iter == 0) return MCMC_B200_OK;
  {
    int r = refstream_fill(c, c->iters_done + n_iter);
    if (r) return r;
  }
  if (use_resident(c, false, c->cfg.leapfrog_steps)) {
    const int done = resident_chain(c, n_iter, c->stream);
    c->iters_done += done;
    n_iter -= done;
    if (n_iter == 0) return MCMC_B200_OK;
  }
  // One HMC iteration (L gradient launches + the accept kernel) is captured
  // once and replayed: launch cost stays off the critical path.
  if (!c->graph_tried) {
    c->graph_tried = true;
    const long long launches_before = c->launches;
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      int r = queue_iteration(c, c->stream);
      e = cudaStreamEndCapture(c->stream, &graph);
      if (r == MCMC_B200_OK && e == cudaSuccess && graph) {
        e = cudaGraphInstantiate(&c->graph_exec, graph, 0);
        if (e != cudaSuccess) c->graph_exec = nullptr;
      }
      if (graph) cudaGraphDestroy(graph);
    }
    cudaGetLastError();
    c->launches = launches_before;
  }
  const long long per_iter =
      (long long)c->cfg.leapfrog_steps * ((c->comm || c->use_red || c->oneshot) ? 2 : 1) + 1;
  for (int i = 0; i < n_iter; ++i) {
    if (c->graph_exec) {
      CK(cudaGraphLaunch(c->graph_exec, c->stream));
      c->launches += per_iter;
    } else {
      int r = queue_iteration(c, c->stream);
      if (r) return r;
    }
  }
  c->iters_done += n_iter;
  return MCMC_B200_OK;
}

API int mcmc_b200_run_chain(mcmc_b200_ctx* c, int n_iter) {
  int r = mcmc_b200_run_chain_async(c, n_iter);
  if (r) return r;
  return check_status(c);
}

API int mcmc_b200_chain_info(mcmc_b200_ctx* c, int window, int32_t* iterations, int32_t* accepted,
                             float* eps) {
  if (!c || window < 0 || window >= c->W) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CK(cudaSetDevice(c->device));
  CK(cudaStreamSynchronize(c->stream));
  if (iterations) CK(cudaMemcpy(iterations, c->iter + window, 4, cudaMemcpyDeviceToHost));
  if (accepted) CK(cudaMemcpy(accepted, c->n_accept + window, 4, cudaMemcpyDeviceToHost));
  if (eps) CK(cudaMemcpy(eps, c->eps + window, 4, cudaMemcpyDeviceToHost));
  return MCMC_B200_OK;
}

API int mcmc_b200_get_state(mcmc_b200_ctx* c, int window, float* w, float* grad, double* loglik,
                            double* logprior) {
  if (!c || window < 0 || window >= c->W) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CK(cudaSetDevice(c->device));
  CK(cudaStreamSynchronize(c->stream));
  const size_t o = (size_t)window * c->Pp;
  if (w) CK(cudaMemcpy(w, c->w_cur + o, (size_t)c->P * 4, cudaMemcpyDeviceToHost));
  if (grad) CK(cudaMemcpy(grad, c->g_cur + o, (size_t)c->P * 4, cudaMemcpyDeviceToHost));
  if (loglik) CK(cudaMemcpy(loglik, c->ll_cur + window, 8, cudaMemcpyDeviceToHost));
  if (logprior) CK(cudaMemcpy(logprior, c->lp_cur + window, 8, cudaMemcpyDeviceToHost));
  return MCMC_B200_OK;
}

API int mcmc_b200_get_samples(mcmc_b200_ctx* c, int window, int first, int count, float* out) {
  if (!c || !out || window < 0 || window >= c->W || first < 0 || count < 0 || !c->samples ||
      first + count > c->cfg.sample_capacity)
    return fail(MCMC_B200_ERR_INVALID, "bad arguments or no sample storage");
  CK(cudaSetDevice(c->device));
  CK(cudaStreamSynchronize(c->stream));
  const size_t P = c->P;
  CK(cudaMemcpy(out, c->samples + ((size_t)window * c->cfg.sample_capacity + first) * P,
                (size_t)count * P * 4, cudaMemcpyDeviceToHost));
  return MCMC_B200_OK;
}

API int mcmc_b200_get_trace(mcmc_b200_ctx* c, int window, int first, int count, float* momenta,
                            float* log_u, double* log_acpt, int32_t* accepted, float* eps) {
  if (!c || window < 0 || window >= c->W || first < 0 || count < 0 ||
      first + count > c->cfg.trace_iters)
    return fail(MCMC_B200_ERR_INVALID, "bad arguments or trace not enabled");
  CK(cudaSetDevice(c->device));
  CK(cudaStreamSynchronize(c->stream));
  const size_t K = c->cfg.trace_iters, P = c->P, o = (size_t)window * K + first;
  if (momenta) CK(cudaMemcpy(momenta, c->tr_mom + o * P, (size_t)count * P * 4, cudaMemcpyDeviceToHost));
  if (log_u) CK(cudaMemcpy(log_u, c->tr_log_u + o, (size_t)count * 4, cudaMemcpyDeviceToHost));
  if (log_acpt) CK(cudaMemcpy(log_acpt, c->tr_log_acpt + o, (size_t)count * 8, cudaMemcpyDeviceToHost));
  if (accepted) CK(cudaMemcpy(accepted, c->tr_accept + o, (size_t)count * 4, cudaMemcpyDeviceToHost));
  if (eps) CK(cudaMemcpy(eps, c->tr_eps + o, (size_t)count * 4, cudaMemcpyDeviceToHost));
  return MCMC_B200_OK;
}

// ---- checkpoint / resume ------------------------------------------------------
// The reference keeps its samples in device memory and loses them, with the chain state, when the
// process ends (main.h:183,277-283,295).  Every random draw here is a pure function of (seed, global
// window, iteration), so a chain resumed from a checkpoint continues bit-identically where sums are added in the same
// order (same windows, rows and resident plan, or a fixed `slices`).
namespace {
struct CkptHeader {
  char magic[8];          // "MCB2CKPT"
  uint32_t version, header_bytes;
  int32_t W, P, Pp, D, H, likelihood, precision, leapfrog_steps, burn_in, adapt_steps, sample_capacity,
      trace_iters, iters_done, slices, rng_streams;
  int64_t rows;
  uint64_t seed;
  uint64_t payload_bytes;
};
struct CkptField {
  void* dev;
  size_t bytes;
};
std::vector<CkptField> ckpt_fields(mcmc_b200_ctx* c) {
  const size_t W = c->W, Pp = c->Pp, P = c->P, S = c->cfg.sample_capacity, K = c->cfg.trace_iters;
  std::vector<CkptField> f = {
      {c->wbuf[0], W * Pp * 4}, {c->mbuf[0], W * Pp * 4}, {c->w_cur, W * Pp * 4}, {c->g_cur, W * Pp * 4},
      {c->m0, W * Pp * 4},      {c->ll_cur, W * 8},       {c->lp_cur, W * 8},     {c->eps, W * 4},
      {c->iter, W * 4},         {c->n_accept, W * 4},     {c->gwin, W * 8}};
  if (c->samples) f.push_back({c->samples, W * S * P * 4});
  if (K > 0) {
    f.push_back({c->tr_mom, W * K * P * 4});
    f.push_back({c->tr_log_u, W * K * 4});
    f.push_back({c->tr_log_acpt, W * K * 8});
    f.push_back({c->tr_accept, W * K * 4});
    f.push_back({c->tr_eps, W * K * 4});
  }
  return f;
}
CkptHeader ckpt_header(mcmc_b200_ctx* c) {
  CkptHeader h;
  memset(&h, 0, sizeof h);
  memcpy(h.magic, "MCB2CKPT", 8);
  h.version = 2;
  h.header_bytes = sizeof(CkptHeader);
  h.W = c->W; h.P = c->P; h.Pp = c->Pp; h.D = c->cfg.D; h.H = c->cfg.H;
  h.likelihood = c->cfg.likelihood; h.precision = c->cfg.precision;
  h.leapfrog_steps = c->cfg.leapfrog_steps; h.burn_in = c->cfg.burn_in; h.adapt_steps = c->cfg.adapt_steps;
  h.sample_capacity = c->cfg.sample_capacity; h.trace_iters = c->cfg.trace_iters;
  h.iters_done = c->iters_done; h.slices = c->slices; h.rng_streams = c->cfg.rng_streams;
  h.rows = c->rows; h.seed = c->cfg.seed;
  for (const CkptField& f : ckpt_fields(c)) h.payload_bytes += f.bytes;
  return h;
}
}  // namespace

API int mcmc_b200_checkpoint_size(mcmc_b200_ctx* c, uint64_t* bytes) {
  if (!c || !bytes) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  const CkptHeader h = ckpt_header(c);
  *bytes = sizeof(CkptHeader) + h.payload_bytes;
  return MCMC_B200_OK;
}

API int mcmc_b200_checkpoint_save(mcmc_b200_ctx* c, void* host_buf, uint64_t bytes) {
  if (!c || !host_buf) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  if (!c->bootstrapped) return fail(MCMC_B200_ERR_INVALID, "nothing to save: the chain has not started");
  CK(cudaSetDevice(c->device));
  int r = check_status(c);  // synchronises; a chain that timed out is not worth saving
  if (r) return r;
  const CkptHeader h = ckpt_header(c);
  if (bytes < sizeof(CkptHeader) + h.payload_bytes) return fail(MCMC_B200_ERR_INVALID, "buffer too small");
  memcpy(host_buf, &h, sizeof h);
  char* p = static_cast<char*>(host_buf) + sizeof h;
  for (const CkptField& f : ckpt_fields(c)) {
    CK(cudaMemcpy(p, f.dev, f.bytes, cudaMemcpyDeviceToHost));
    p += f.bytes;
  }
  return MCMC_B200_OK;
}

API int mcmc_b200_checkpoint_load(mcmc_b200_ctx* c, const void* host_buf, uint64_t bytes) {
  if (!c || !host_buf || bytes < sizeof(CkptHeader)) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CkptHeader h;
  memcpy(&h, host_buf, sizeof h);
  const CkptHeader want = ckpt_header(c);
  if (memcmp(h.magic, want.magic, 8) != 0 || h.version != want.version || h.header_bytes != sizeof h)
    return fail(MCMC_B200_ERR_INVALID, "not a checkpoint of this library version");
  if (h.W != want.W || h.P != want.P || h.Pp != want.Pp || h.D != want.D || h.H != want.H ||
      h.likelihood != want.likelihood || h.precision != want.precision ||
      h.leapfrog_steps != want.leapfrog_steps || h.burn_in != want.burn_in ||
      h.adapt_steps != want.adapt_steps || h.sample_capacity != want.sample_capacity ||
      h.trace_iters != want.trace_iters || h.rows != want.rows || h.seed != want.seed ||
      h.rng_streams != want.rng_streams ||
      h.payload_bytes != want.payload_bytes)
    return fail(MCMC_B200_ERR_INVALID, "checkpoint was written by a context with a different configuration");
  if (bytes < sizeof h + h.payload_bytes) return fail(MCMC_B200_ERR_INVALID, "truncated checkpoint");
  for (int w = 0; w < c->W; ++w)
    if (!c->window_set[w]) return fail(MCMC_B200_ERR_INVALID, "upload every window's data before resuming");
  CK(cudaSetDevice(c->device));
  CK(cudaStreamSynchronize(c->stream));
  const char* p = static_cast<const char*>(host_buf) + sizeof h;
  const std::vector<CkptField> fields = ckpt_fields(c);
  // the stored global window ids must be the ones this context was given: chains are keyed by them
  {
    size_t off = 0;
    for (const CkptField& f : fields) {
      if (f.dev == c->gwin) break;
      off += f.bytes;
    }
    if (memcmp(p + off, c->h_gwin.data(), (size_t)c->W * 8) != 0)
      return fail(MCMC_B200_ERR_INVALID, "checkpoint belongs to other global windows");
  }
  for (const CkptField& f : fields) {
    CK(cudaMemcpy(f.dev, p, f.bytes, cudaMemcpyHostToDevice));
    p += f.bytes;
  }
  c->bootstrapped = true;
  c->iters_done = h.iters_done;
  return MCMC_B200_OK;
}

// ---- explicit-state calls (one window) -------------------------------------
// explicit_steps in one launch where the window's rows fit on the chip.  Pointers may be device memory or the mapped
// host block; the parameters of an evaluation come from the host by value (w_host).  False: the launch was refused and
// nothing has been done (see resident_chain).
static bool resident_steps(mcmc_b200_ctx* c, int data_window, int L, float eps, const float* w0, const float* m0,
                          const float* g0, float* w_last, float* m_last, float* g_out, float* zero_out,
                          float* row_loss, float* prior_loss, double* scalars, cudaStream_t st, bool eval_only,
                          const float* w_host = nullptr) {
  ResidentParams g = c->res_x;
  g.mode = eval_only ? RES_EVAL : RES_STEPS;
  g.n_steps = L;
  g.n_iter = 1;
  g.data_window0 = data_window;
  g.status_host = &c->hb->status;
  g.w0 = w0;
  g.m0 = m0;
  g.g0 = g0;
  g.eps_scalar = eps;
  g.w_out = w_last;
  g.m_out = m_last;
  g.g_out = g_out;
  g.zero_out = zero_out;
  g.row_loss = row_loss;
  g.prior_loss = prior_loss;
  g.scalars = scalars;
  cudaError_t e = cudaErrorCooperativeLaunchTooLarge;
  if (!w_host) {
    e = launch_resident(c, c->res_x_cluster, g, st);
  } else if (c->res_x_cluster == 8) {  // one window has clusters of eight on every GPU that holds one of them
    ResidentEvalParams v;
    static_cast<ResidentParams&>(v) = g;
    memcpy(v.w_val, w_host, (size_t)c->P * 4);
    e = launch_resident_eval(c, v, st);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  c->launches++;
  return true;
}

API int mcmc_b200_selftest_resident_wait(mcmc_b200_ctx* c, int code, int limit_us) {
  const bool steps = code >= 621 && code <= 624;
  if (!c || limit_us < 40 || limit_us > 10000 ||
      (code != 603 && code != 611 && code != 901 &&
       (c->cfg.precision != MCMC_B200_PREC_FP32 || (!steps && code != 612 && code != 613))))
    return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CK(cudaSetDevice(c->device));
  if (c->W != 1 || !c->window_set[0] || !use_resident(c, true, 1) || (code == 603 && c->res_x.clusters < 2))
    return fail(MCMC_B200_ERR_INVALID, "needs one window with data whose rows (603: more than 4096) fit on the chip");
  if (steps && resident_one_tile((int)c->rows, c->res_x.clusters, c->res_x_cluster))
    return fail(MCMC_B200_ERR_INVALID, "needs more than a tile of rows in a CTA");
  if (code == 901) {
    cudaError_t e = launch_wait_probe(c->status, (unsigned int)(limit_us / 20), c->stream);
    c->launches++;
    if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
  }
  const std::vector<float> w(c->P, 0.f);
  if (code != 603) {
    c->res_x.test_code = steps ? code - 10 : code;
    c->res_x.wait_ticks = (unsigned int)limit_us / 33;
    const int r = steps ? mcmc_b200_leapfrog(c, 0, 3, 0.f, w.data(), w.data(), w.data(), nullptr, nullptr, nullptr, nullptr, nullptr)
                        : mcmc_b200_potential_and_grad(c, 0, w.data(), nullptr, nullptr, nullptr, nullptr);
    c->res_x.test_code = 0;
    c->res_x.wait_ticks = RES_WAIT_TICKS;
    return r;
  }
  int r = refstream_fill(c, c->iters_done + 1);
  if (r) return r;
  const bool chain = c->bootstrapped && use_resident(c, false, c->cfg.leapfrog_steps);
  ResidentParams& g = chain ? c->res : c->res_x;
  g.missing = 1;
  g.wait_ticks = (unsigned int)limit_us / 33;
  const bool done = chain ? resident_chain(c, 1, c->stream) == 1
                          : resident_steps(c, 0, 1, 0.f, nullptr, nullptr, nullptr, nullptr, nullptr, c->hb->g_out,
                                           nullptr, nullptr, nullptr, c->hb->scalars, c->stream, true, w.data());
  g.missing = 0;
  g.wait_ticks = RES_WAIT_TICKS;
  if (!done) return fail(MCMC_B200_ERR_CUDA, "the launch was refused");
  return check_status(c);
}

static int explicit_steps(mcmc_b200_ctx* c, int data_window, int L, float eps, const float* w0, const float* m0, const float* g0,
                          float* w_last, float* m_last, float* g_out, float* row_loss, float* prior_loss, cudaStream_t st,
                          bool eval_only, bool data_fresh = false);
API int mcmc_b200_selftest_kernel_wait(mcmc_b200_ctx* c, int code) {
  if (!c || ((code < 102 || code > 105) && code != 402)) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CK(cudaSetDevice(c->device));
  int r;
  if (code == 402) {
    if (c->cfg.sample_capacity < 1) return fail(MCMC_B200_ERR_INVALID, "needs sample storage");
    const std::vector<float> x(c->cfg.D, 0.f);
    float out;
    c->test_code = code;
    r = mcmc_b200_predict_mean(c, 0, x.data(), 1, 0, 1, &out);
  } else {
    if (c->cfg.precision != MCMC_B200_PREC_FP32 || !c->table || !c->window_set[0])
      return fail(MCMC_B200_ERR_INVALID, "needs an FP32 context of 40 units with a work table, and data");
    if (code != 102 && !c->xtab_ints) return fail(MCMC_B200_ERR_INVALID, "needs segments of 16 tiles in the mean");
    CK(cudaMemsetAsync(c->xw[0], 0, (size_t)c->P * 4, c->stream));
    c->test_code = code;
    r = explicit_steps(c, 0, 1, 0.f, c->xw[0], c->xm[0], c->xg, nullptr, nullptr, c->g_out, nullptr, nullptr, c->stream, true);
    if (r == MCMC_B200_OK) r = check_status(c);
  }
  c->test_code = 0;
  return r;
}

API int mcmc_b200_selftest_refuse_forward(mcmc_b200_ctx* c, int nth) {
  if (!c || nth < 0) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  c->refuse_forward = nth;
  return MCMC_B200_OK;
}

API int mcmc_b200_selftest_refuse_resident(mcmc_b200_ctx* c, int launches) {
  if (!c || launches < 0) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  c->refuse = launches;
  return MCMC_B200_OK;
}

// L leapfrog steps from (w0, m0, g0) on device; results in xw/xm[L&1], g_out, scalars.
static int explicit_steps(mcmc_b200_ctx* c, int data_window, int L, float eps, const float* w0,
                          const float* m0, const float* g0, float* w_last, float* m_last,
                          float* g_out, float* row_loss, float* prior_loss, cudaStream_t st,
                          bool eval_only, bool data_fresh) {
  const int S = c->slices_x;
  for (int s = 0; s < L; ++s) {
    GradParams g = base_grad_params(c);
    g.data_window0 = data_window;
    g.data_fresh = (data_fresh && s == 0) ? 1 : 0;  // a repack was queued directly before the first launch
    g.mode = eval_only ? MODE_EVAL : (s == 0 ? MODE_FIRST : MODE_NEXT);
    g.w_in = s == 0 ? w0 : c->xw[s & 1];
    g.m_in = s == 0 ? m0 : c->xm[s & 1];
    const bool last = s == L - 1;
    g.w_out = (last && w_last) ? w_last : c->xw[(s + 1) & 1];
    g.m_out = (last && m_last) ? m_last : c->xm[(s + 1) & 1];
    g.g_carried = g0;
    g.partial_in = c->xpartial[(s + 1) & 1];
    const bool red = c->comm || c->use_red_x;
    g.red_in = (red && g.mode == MODE_NEXT) ? c->xred : nullptr;
    g.partial_out = c->xpartial[s & 1];
    g.ll_out = c->xllp[s & 1];
    g.eps = nullptr;
    g.eps_scalar = eps;
    g.no_loss = !last;
    g.row_loss = last ? row_loss : nullptr;
    g.row_loss_stride = 0;
    int r = launch_grad(c, g, true, st);
    if (r) return r;
    if (red) {
      cudaError_t e = launch_reduce_partials(c->xpartial[s & 1], c->xllp[s & 1], S, c->xtab_nslot, c->P, c->Pp,
                                             c->xred, 1, c->num_sms, st);
      c->launches++;
      if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
      if (c->comm) {
        r = allreduce(c, c->xred, (size_t)(c->Pp + 4), st);
        if (r) return r;
      }
    }
  }
  AcceptParams a = base_accept_params(c);
  a.mode = ACC_FINALIZE;
  a.slices = S;
  a.nslot = c->xtab_nslot;
  a.partial = c->xpartial[(L - 1) & 1];
  a.ll_partial = c->xllp[(L - 1) & 1];
  a.red_in = (c->comm || c->use_red_x) ? c->xred : nullptr;
  a.w_new = eval_only ? w0 : ((w_last) ? w_last : c->xw[L & 1]);
  a.g_out = g_out;
  a.prior_loss_out = prior_loss;
  a.scalars_out = c->scalars;
  cudaError_t e = launch_accept(a, 1, st);
  c->launches++;
  if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
  return MCMC_B200_OK;
}

API int mcmc_b200_potential_and_grad(mcmc_b200_ctx* c, int window, const float* w, double* loglik,
                                     double* logprior, float* grad, float* row_loss) {
  if (!c || !w || window < 0 || window >= c->W) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  if (!c->window_set[window]) return fail(MCMC_B200_ERR_INVALID, "window has no data yet");
  CK(cudaSetDevice(c->device));
  // One launch and one wait, no copies: gradient and sums through the mapped host block, the parameters with the launch.
  // Every cluster wants all of them, and read from the host block they were some 260 reads over PCIe for one cluster and
  // 4,000 for fifteen: 32.9 us instead of 30.0 for 1000 rows (FP32), 68.7 instead of 62.0 for 58368 (TF32, row losses).
  if (use_resident(c, true, 1) &&
      resident_steps(c, window, 1, 0.f, nullptr, nullptr, nullptr, nullptr, nullptr, c->hb->g_out, nullptr,
                     row_loss ? c->row_loss : nullptr, nullptr, c->hb->scalars, c->stream, true, w)) {
    if (row_loss)
      CK(cudaMemcpyAsync(row_loss, c->row_loss, (size_t)c->rows * 4, cudaMemcpyDeviceToHost, c->stream));
    int r = finish_status(c);
    if (r) return r;
    if (grad) memcpy(grad, c->hb->g_out, (size_t)c->P * 4);
    if (loglik) *loglik = c->hb->scalars[0];
    if (logprior) *logprior = c->hb->scalars[1];
    return MCMC_B200_OK;
  }
  CK(cudaMemcpyAsync(c->xw[0], w, (size_t)c->P * 4, cudaMemcpyHostToDevice, c->stream));
  int r = explicit_steps(c, window, 1, 0.f, c->xw[0], c->xm[0], c->xg, nullptr, nullptr, c->g_out,
                         row_loss ? c->row_loss : nullptr, nullptr, c->stream, true);
  if (r) return r;
  double sc[2];
  CK(cudaMemcpyAsync(sc, c->scalars, 16, cudaMemcpyDeviceToHost, c->stream));
  if (grad) CK(cudaMemcpyAsync(grad, c->g_out, (size_t)c->P * 4, cudaMemcpyDeviceToHost, c->stream));
  if (row_loss)
    CK(cudaMemcpyAsync(row_loss, c->row_loss, (size_t)c->rows * 4, cudaMemcpyDeviceToHost, c->stream));
  r = check_status(c);
  if (r) return r;
  if (loglik) *loglik = sc[0];
  if (logprior) *logprior = sc[1];
  return MCMC_B200_OK;
}

API int mcmc_b200_leapfrog(mcmc_b200_ctx* c, int window, int L, float eps, const float* w_prev,
                           const float* mom_prev, const float* grad_prev, float* w_next,
                           float* mom_next, float* grad_cur, double* loglik, double* logprior) {
  if (!c || !w_prev || !mom_prev || !grad_prev || L < 1 || window < 0 || window >= c->W)
    return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  if (!c->window_set[window]) return fail(MCMC_B200_ERR_INVALID, "window has no data yet");
  CK(cudaSetDevice(c->device));
  const size_t n = (size_t)c->P * 4;
  HostBlock* h = c->hb;
  if (use_resident(c, true, L) &&
      (memcpy(h->w, w_prev, n), memcpy(h->m, mom_prev, n), memcpy(h->g, grad_prev, n),
       resident_steps(c, window, L, eps, h->w, h->m, h->g, h->w_out, h->m_out, h->g_out, nullptr, nullptr, nullptr,
                      h->scalars, c->stream, false))) {
    int r = finish_status(c);
    if (r) return r;
    if (w_next) memcpy(w_next, h->w_out, n);
    if (mom_next) memcpy(mom_next, h->m_out, n);
    if (grad_cur) memcpy(grad_cur, h->g_out, n);
    if (loglik) *loglik = h->scalars[0];
    if (logprior) *logprior = h->scalars[1];
    return MCMC_B200_OK;
  }
  CK(cudaMemcpyAsync(c->xw[0], w_prev, n, cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(c->xm[0], mom_prev, n, cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(c->xg, grad_prev, n, cudaMemcpyHostToDevice, c->stream));
  int r = explicit_steps(c, window, L, eps, c->xw[0], c->xm[0], c->xg, nullptr, nullptr, c->g_out, nullptr,
                         nullptr, c->stream, false);
  if (r) return r;
  double sc[2];
  CK(cudaMemcpyAsync(sc, c->scalars, 16, cudaMemcpyDeviceToHost, c->stream));
  if (w_next) CK(cudaMemcpyAsync(w_next, c->xw[L & 1], n, cudaMemcpyDeviceToHost, c->stream));
  if (mom_next) CK(cudaMemcpyAsync(mom_next, c->xm[L & 1], n, cudaMemcpyDeviceToHost, c->stream));
  if (grad_cur) CK(cudaMemcpyAsync(grad_cur, c->g_out, n, cudaMemcpyDeviceToHost, c->stream));
  r = check_status(c);
  if (r) return r;
  if (loglik) *loglik = sc[0];
  if (logprior) *logprior = sc[1];
  return MCMC_B200_OK;
}

API int mcmc_b200_mcmc_step(mcmc_b200_ctx* c, const float* x, const float* y, const float* weights_prev,
                            float* weights_next, const float* mom_prev, float* mom_next,
                            const float* grad_prev, float* grad_cur, float* grad_next,
                            float* loss_values, int L, float eps, void* stream) {
  if (!c || !x || !y || !weights_prev || !weights_next || !mom_prev || !mom_next || !grad_prev ||
      !grad_cur || L < 1)
    return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  if (c->W != 1) return fail(MCMC_B200_ERR_INVALID, "mcmc_step needs a context with one window");
  CK(cudaSetDevice(c->device));
  cudaStream_t st = (cudaStream_t)stream;
  bool repacked = false;
  if (x != c->bound_x || y != c->bound_y) {
    // first use of this dataset (or the first call after mcmc_b200_rebind_data): repack it
    // (io.h:82-85 is where the reference uploads it)
    cudaError_t e = launch_repack(x, y, c->xaug, c->rows, c->rows_pad, c->cfg.D, st);
    c->launches++;
    if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
    c->bound_x = x;
    c->bound_y = y;
    c->window_set[0] = 1;
    repacked = true;
  }
  if (use_resident(c, true, L) &&
      resident_steps(c, 0, L, eps, weights_prev, mom_prev, grad_prev, weights_next, mom_next, grad_cur, grad_next,
                     loss_values, loss_values ? loss_values + c->rows : nullptr, c->scalars, st, false))
    return MCMC_B200_OK;
  int r = explicit_steps(c, 0, L, eps, weights_prev, mom_prev, grad_prev, weights_next, mom_next, grad_cur,
                         loss_values, loss_values ? loss_values + c->rows : nullptr, st, false, repacked);
  if (r) return r;
  if (grad_next) CK(cudaMemsetAsync(grad_next, 0, (size_t)c->P * 4, st));
  return MCMC_B200_OK;
}

API int mcmc_b200_rebind_data(mcmc_b200_ctx* c) {
  if (!c) return fail(MCMC_B200_ERR_INVALID, "null context");
  c->bound_x = nullptr;
  c->bound_y = nullptr;
  return MCMC_B200_OK;
}

API int mcmc_b200_log_acpt(mcmc_b200_ctx* c, const float* prev_loss, const float* new_loss,
                           int64_t n_loss, const float* prev_mom, const float* new_mom,
                           const float* grad_cur, float eps, void* stream, float* out) {
  if (!c || !prev_loss || !new_loss || !prev_mom || !new_mom || !grad_cur || !out)
    return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  CK(cudaSetDevice(c->device));
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = launch_log_acpt(prev_loss, new_loss, n_loss, prev_mom, new_mom, grad_cur, c->P, eps,
                                  &c->hb->log_acpt, st);
  c->launches++;
  if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
  CK(cudaStreamSynchronize(st));
  // (the losses may come from a trajectory that has given up)
  if (*reinterpret_cast<volatile int*>(&c->hb->status) != 0) return finish_status(c);
  *out = c->hb->log_acpt;
  return MCMC_B200_OK;
}

// grows a cached scratch buffer (kept for the life of the context; the old one stays in the free list)
template <typename T>
static int fwd_reserve(mcmc_b200_ctx* c, T** buf, size_t* cap, size_t need) {
  if (need <= *cap) return MCMC_B200_OK;
  T* nb = nullptr;
  int r = dalloc(c, (void**)&nb, need * sizeof(T), false);
  if (r) return r;
  *buf = nb;
  *cap = need;
  return MCMC_B200_OK;
}

// waits for a forward pass; a wait of its kernel that ran out is reported through the mapped host block
static int forward_finish(mcmc_b200_ctx* c) {
  CK(cudaStreamSynchronize(c->stream));
  const int code = *reinterpret_cast<volatile int*>(&c->hb->fwd_status);
  if (code == 0) return MCMC_B200_OK;
  c->hb->fwd_status = 0;
  char b[96];
  snprintf(b, sizeof b, "device-side wait ran out (code %d)", code);
  return fail(MCMC_B200_ERR_TIMEOUT, b);
}

// the stream and events of copies that run beside the context's work, made when first wanted
static int copy_stream(mcmc_b200_ctx* c) {
  if (!c->copies) CK(cudaStreamCreateWithFlags(&c->copies, cudaStreamNonBlocking));
  for (cudaEvent_t& e : c->copy_events)
    if (!e) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  return MCMC_B200_OK;
}

// Rows cut[k] .. cut[k + 1], k < 3: copied, predicted, their means copied back; `blocks`: copies on a stream of their own
static int predict_queue(mcmc_b200_ctx* c, ForwardParams a, const int64_t* cut, bool blocks, const float* xs, float* out) {
  const int H = c->cfg.H;
  const size_t D = c->cfg.D;
  auto rows = [&](int k) { return cut[k + 1] - cut[k]; };
  cudaStream_t copies = blocks ? c->copies : c->stream;
  for (int k = 0; k < 3 && rows(k) > 0; ++k) {
    a.n = rows(k);
    a.x = c->fwd_x + cut[k] * D;
    float* sum = c->fwd_out + cut[k];
    CK(cudaMemcpyAsync(c->fwd_x + cut[k] * D, xs + cut[k] * D, a.n * D * 4, cudaMemcpyHostToDevice, copies));
    if (blocks) {
      CK(cudaEventRecord(c->copy_events[k], copies));
      CK(cudaStreamWaitEvent(c->stream, c->copy_events[k], 0));
    }
    cudaError_t e = c->refuse_forward > 0 && --c->refuse_forward == 0 ? cudaErrorLaunchOutOfResources
                                                                      : launch_forward(H, a, c->num_sms, false, c->stream);
    if (e == cudaSuccess) e = launch_forward_finish_predict(H, a, c->num_sms, sum, c->stream);
    if (e == cudaSuccess) c->launches += 2;
    if (e == cudaSuccess && blocks) e = cudaEventRecord(c->copy_events[k], c->stream);
    if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
  }
  for (int k = 0; k < 3 && rows(k) > 0; ++k) {
    if (blocks) CK(cudaStreamWaitEvent(copies, c->copy_events[k], 0));
    CK(cudaMemcpyAsync(out + cut[k], c->fwd_out + cut[k], rows(k) * 4, cudaMemcpyDeviceToHost, copies));
  }
  return MCMC_B200_OK;
}

API int mcmc_b200_predict_mean(mcmc_b200_ctx* c, int window, const float* xs, int64_t n, int first,
                               int count, float* out) {
  if (!c || !xs || !out || n < 1 || window < 0 || window >= c->W || first < 0 || count < 1 ||
      !c->samples || first + count > c->cfg.sample_capacity)
    return fail(MCMC_B200_ERR_INVALID, "bad arguments or no sample storage");
  CK(cudaSetDevice(c->device));
  const int H = c->cfg.H;
  const size_t D = c->cfg.D;
  ForwardParams a;
  memset(&a, 0, sizeof a);
  a.x_stride = D;
  a.n = n;
  a.samples = c->samples + ((size_t)window * c->cfg.sample_capacity + first) * c->P;
  a.count = count;
  a.lik = make_lik(c->cfg);
  a.status = &c->hb->fwd_status;
  a.test_code = c->test_code;
  int r = fwd_reserve(c, &c->fwd_x, &c->fwd_x_cap, (size_t)n * D);
  if (r == MCMC_B200_OK) r = fwd_reserve(c, &c->fwd_out, &c->fwd_out_cap, (size_t)n);
  if (r) return r;
  // The rows come from pageable memory, through the driver's buffers, at 17 GB/s while the caller waits: 0.3 ms for 58368 of them,
  // as long as the pass over 230 samples.  So a block is copied beside the pass over the one before it; a first short one,
  // since nothing runs beside its copy.  That takes six launches instead of two, some 12 us, which the passes have to hide: where rows x
  // samples x units are few, one block is faster.  us a call in one block / in three: 40 units, 8192 rows x 16 90 / 104, x 200 128 / 132;
  // 12288 x 75 132 / 131, x 150 159 / 148; 16384 x 50 137 / 141, x 100 163 / 155; 58368 x 16 356 / 346, x 24 367 / 350, x 800 1370 / 1190;
  // 100000 x 16 559 / 577, x 50 647 / 624.  128 units, 12288 x 16 128 / 124, x 32 146 / 135; 16384 x 24 152 / 155; 58368 x 8 376 / 364
  const int64_t tile = forward_rows(H);
  const bool blocks = n >= 12288 && (double)n * count * H >= 50e6;
  int64_t cut[4] = {0, n, n, n};
  if (blocks) {
    cut[1] = n / 8 / tile * tile;
    cut[2] = n / 2 / tile * tile;
    r = copy_stream(c);
    if (r) return r;
    // a caller may have queued on the context's stream what fills `xs`
    CK(cudaEventRecord(c->copy_events[0], c->stream));
    CK(cudaStreamWaitEvent(c->copies, c->copy_events[0], 0));
  }
  auto rows = [&](int k) { return cut[k + 1] - cut[k]; };
  size_t sums = 0, most = 0;  // a row's sums from several CTAs, or one where there is no memory for more
  for (int k = 0; k < 3 && rows(k) > 0; ++k) {
    a.n = rows(k);
    sums = std::max<size_t>(sums, (size_t)forward_slots(H, c->num_sms, a) * a.n);
    most = std::max<size_t>(most, a.n);
  }
  r = fwd_reserve(c, &c->fwd_partial, &c->fwd_partial_cap, sums);
  if (r == MCMC_B200_ERR_NOMEM && sums > most) {
    a.whole = 1;
    r = fwd_reserve(c, &c->fwd_partial, &c->fwd_partial_cap, most);
  }
  if (r) return r;
  a.partial = c->fwd_partial;
  r = predict_queue(c, a, cut, blocks, xs, out);
  if (r) {  // the caller gets `xs` and `out` back: nothing may still read the one or write the other
    if (blocks) cudaStreamSynchronize(c->copies);
    cudaStreamSynchronize(c->stream);
    return r;
  }
  if (blocks) CK(cudaStreamSynchronize(c->copies));
  return forward_finish(c);
}

API int mcmc_b200_final_loss(mcmc_b200_ctx* c, int window, int first, int count, double* mean_loglik,
                             double* mean_logprior) {
  if (!c || window < 0 || window >= c->W || first < 0 || count < 1 || !c->samples ||
      first + count > c->cfg.sample_capacity)
    return fail(MCMC_B200_ERR_INVALID, "bad arguments or no sample storage");
  if (!c->window_set[window]) return fail(MCMC_B200_ERR_INVALID, "window has no data yet");
  CK(cudaSetDevice(c->device));
  // all samples against the window's rows in one launch (FP32 forward pass, no gradient)
  const int tiles = (int)forward_tiles(c->cfg.H, c->rows);
  int r = fwd_reserve(c, &c->fwd_partial, &c->fwd_partial_cap, (size_t)tiles * count + 2 * (size_t)count);
  if (r) return r;
  const float* xw = c->xaug + (size_t)window * c->rows_pad * KP;
  const float* smp = c->samples + ((size_t)window * c->cfg.sample_capacity + first) * c->P;
  ForwardParams a;
  memset(&a, 0, sizeof a);
  a.x = xw;
  a.x_stride = KP;
  a.y = xw + COL_Y;
  a.y_stride = KP;
  a.n = c->rows;
  a.samples = smp;
  a.count = count;
  a.lik = make_lik(c->cfg);
  a.partial = c->fwd_partial;
  double* d_ll = c->fwd_partial + (size_t)tiles * count;
  double* d_lp = d_ll + count;
  a.status = &c->hb->fwd_status;
  cudaError_t e = launch_forward(c->cfg.H, a, c->num_sms, true, c->stream);
  if (e == cudaSuccess)
    e = launch_forward_finish_loss(c->fwd_partial, tiles, count, smp, c->P, make_prior(c->cfg), d_ll, d_lp, c->stream);
  c->launches += 2;
  if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
  std::vector<double> h(2 * (size_t)count);
  CK(cudaMemcpyAsync(h.data(), d_ll, h.size() * 8, cudaMemcpyDeviceToHost, c->stream));
  r = forward_finish(c);
  if (r) return r;
  double sa = 0, sb = 0;
  for (int s = 0; s < count; ++s) { sa += h[s]; sb += h[count + s]; }  // main.h:100-113: running means
  if (mean_loglik) *mean_loglik = sa / count;
  if (mean_logprior) *mean_logprior = sb / count;
  return MCMC_B200_OK;
}

API int mcmc_b200_nccl_unique_id(unsigned char id[128]) {
  std::string why;
  if (!nccl_load(&why)) return fail(MCMC_B200_ERR_NCCL, why);
  NcclUniqueId u;
  int r = g_nccl.GetUniqueId(&u);
  if (r != 0) return fail(MCMC_B200_ERR_NCCL, "ncclGetUniqueId failed");
  memcpy(id, u.internal, 128);
  return MCMC_B200_OK;
}

API int mcmc_b200_enable_row_sharding(mcmc_b200_ctx* c, const unsigned char id[128], int rank, int nranks) {
  if (!c || !id || nranks < 1 || rank < 0 || rank >= nranks) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  if (c->bootstrapped) return fail(MCMC_B200_ERR_INVALID, "enable row sharding before the chain starts");
  std::string why;
  if (!nccl_load(&why)) return fail(MCMC_B200_ERR_NCCL, why);
  CK(cudaSetDevice(c->device));
  NcclUniqueId u;
  memcpy(u.internal, id, 128);
  int r = g_nccl.CommInitRank(&c->comm, nranks, u, rank);
  if (r != 0) {
    c->comm = nullptr;
    return fail(MCMC_B200_ERR_NCCL, std::string("ncclCommInitRank: ") +
                                        (g_nccl.GetErrorString ? g_nccl.GetErrorString(r) : "error"));
  }
  c->rank = rank;
  c->nranks = nranks;
  drop_graph(c);         // a graph captured before this call has neither the sums nor the all-reduce in it
  return MCMC_B200_OK;
}

// Sets up the peer-memory all-reduce on top of an existing row-sharding communicator: one allocation per
// rank (receive slots + flags), its CUDA IPC handle gathered over the communicator, every peer's block
// mapped into this process.  `fake_peers` (self-test only): no communicator, the "peers" are further
// blocks of THIS GPU that nothing ever writes.
static int oneshot_setup(mcmc_b200_ctx* c, bool fake_peers) {
  if (c->nranks > ONESHOT_MAX_RANKS) return fail(MCMC_B200_ERR_INVALID, "too many ranks for the one-shot all-reduce");
  const size_t block = oneshot_block_bytes(c);
  int r = dalloc(c, &c->os_block, fake_peers ? block * c->nranks : block, true);
  if (r) return r;
  r = dalloc(c, (void**)&c->os_seq, 8, true);
  if (r) return r;
  c->os_done = c->os_seq + 1;
  std::vector<char*> base(c->nranks, nullptr);
  c->os_peer_blocks.assign(c->nranks, nullptr);
  if (fake_peers) {
    for (int k = 0; k < c->nranks; ++k) base[k] = static_cast<char*>(c->os_block) + (size_t)k * block;
  } else {
    cudaIpcMemHandle_t mine;
    CK(cudaIpcGetMemHandle(&mine, c->os_block));
    char* dh = nullptr;
    r = dalloc(c, (void**)&dh, sizeof(mine) * c->nranks, true);
    if (r) return r;
    CK(cudaMemcpy(dh + sizeof(mine) * c->rank, &mine, sizeof(mine), cudaMemcpyHostToDevice));
    if (!g_nccl.AllGather) return fail(MCMC_B200_ERR_NCCL, "ncclAllGather missing");
    int nr = g_nccl.AllGather(dh + sizeof(mine) * c->rank, dh, sizeof(mine), kNcclChar, c->comm, c->stream);
    if (nr != 0) return fail(MCMC_B200_ERR_NCCL, "ncclAllGather of the IPC handles failed");
    CK(cudaStreamSynchronize(c->stream));
    std::vector<cudaIpcMemHandle_t> all(c->nranks);
    CK(cudaMemcpy(all.data(), dh, sizeof(mine) * c->nranks, cudaMemcpyDeviceToHost));
    for (int k = 0; k < c->nranks; ++k) {
      if (k == c->rank) { base[k] = static_cast<char*>(c->os_block); continue; }
      void* p = nullptr;
      cudaError_t e = cudaIpcOpenMemHandle(&p, all[k], cudaIpcMemLazyEnablePeerAccess);
      if (e != cudaSuccess)
        return fail(MCMC_B200_ERR_CUDA, std::string("cudaIpcOpenMemHandle (peer access between the GPUs is "
                                                    "required): ") + cudaGetErrorString(e));
      c->os_peer_blocks[k] = p;
      base[k] = static_cast<char*>(p);
    }
  }
  c->os_base.assign(base.begin(), base.end());
  if (!fake_peers) {
    // nobody may send before every rank has zeroed and mapped its block: one tiny all-reduce as the barrier
    int nr = g_nccl.AllReduce(c->red, c->red, 1, kNcclFloat64, kNcclSum, c->comm, c->stream);
    if (nr != 0) return fail(MCMC_B200_ERR_NCCL, "set-up barrier failed");
    CK(cudaStreamSynchronize(c->stream));
  }
  c->oneshot = true;
  drop_graph(c);
  return MCMC_B200_OK;
}

API int mcmc_b200_enable_oneshot_allreduce(mcmc_b200_ctx* c) {
  if (!c) return fail(MCMC_B200_ERR_INVALID, "null context");
  if (!c->comm) return fail(MCMC_B200_ERR_INVALID, "call mcmc_b200_enable_row_sharding first");
  if (c->bootstrapped) return fail(MCMC_B200_ERR_INVALID, "enable it before the chain starts");
  if (c->oneshot) return MCMC_B200_OK;
  if (c->W != 1) return fail(MCMC_B200_ERR_INVALID, "row sharding is for contexts with one window");
  CK(cudaSetDevice(c->device));
  return oneshot_setup(c, false);
}

API int mcmc_b200_selftest_oneshot_timeout(mcmc_b200_ctx* c, int polls) {
  if (!c || polls < 1 || polls > (1 << 24)) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  if (c->comm || c->oneshot || c->bootstrapped || c->W != 1)
    return fail(MCMC_B200_ERR_INVALID, "needs a fresh one-window context without row sharding");
  CK(cudaSetDevice(c->device));
  // two "ranks" of which only this one ever sends: the wait for the other one must run out
  c->nranks = 2;
  c->rank = 0;
  int r = oneshot_setup(c, true);
  if (r) return r;
  c->os_poll_limit = (unsigned int)polls;
  CK(cudaMemsetAsync(c->partial[0], 0, (size_t)c->slices * c->Pp * 4, c->stream));
  r = oneshot_allreduce(c, c->partial[0], c->llp[0], c->stream);
  // back to an unsharded context whatever happened
  c->oneshot = false;
  c->nranks = 1;
  c->os_poll_limit = 1u << 22;
  drop_graph(c);
  if (r) return r;
  return check_status(c);
}

API int mcmc_b200_time_allreduce(mcmc_b200_ctx* c, int reps, float* us_per_call) {
  if (!c || reps < 1 || !us_per_call) return fail(MCMC_B200_ERR_INVALID, "bad arguments");
  if (!c->comm) return fail(MCMC_B200_ERR_INVALID, "row sharding is not enabled");
  CK(cudaSetDevice(c->device));
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  auto once = [&]() -> int {
    if (c->oneshot) return oneshot_allreduce(c, c->partial[0], c->llp[0], c->stream);
    cudaError_t e = launch_reduce_partials(c->partial[0], c->llp[0], c->slices, c->tab_nslot, c->P, c->Pp, c->red,
                                           c->W, c->num_sms, c->stream);
    c->launches++;
    if (e != cudaSuccess) return fail(MCMC_B200_ERR_CUDA, cudaGetErrorString(e));
    return allreduce(c, c->red, (size_t)c->W * (c->Pp + 4), c->stream);
  };
  for (int i = 0; i < 5; ++i) { int r = once(); if (r) return r; }
  CK(cudaEventRecord(e0, c->stream));
  for (int i = 0; i < reps; ++i) { int r = once(); if (r) return r; }
  CK(cudaEventRecord(e1, c->stream));
  CK(cudaEventSynchronize(e1));
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  *us_per_call = 1e3f * ms / reps;
  return check_status(c);
}

API int64_t mcmc_b200_launch_count(mcmc_b200_ctx* c, int reset) {
  if (!c) return -1;
  long long v = c->launches;
  if (reset) c->launches = 0;
  return v;
}

API int mcmc_b200_chain_geometry(mcmc_b200_ctx* c, int* slices, int* ctas_per_sm, int* tile_rows) {
  if (!c) return fail(MCMC_B200_ERR_INVALID, "null context");
  if (slices) *slices = c->slices;
  if (ctas_per_sm) *ctas_per_sm = c->ctas_per_sm;
  if (tile_rows) *tile_rows = c->tile_rows;
  return MCMC_B200_OK;
}
