// Launch parameter block of the accept kernel and the host-callable launchers
// shared between the translation units of the library.
#pragma once
#include "common.cuh"

namespace mcmc_b200 {

enum AcceptMode : int {
  ACC_BOOTSTRAP = 0,  // adopt the evaluated state as the chain's current state (main.h:191-202)
  ACC_ITERATE = 1,    // accept ratio, accept/reject, adaptation, store, next momentum
  ACC_FINALIZE = 2    // only assemble gradient and log-density sums for the caller
};

struct AcceptParams {
  int mode;
  int P, Pp;
  int slices;                // slots per window (stride, and count when nslot is null)
  const int* nslot;          // optional [windows]: slots in use
  const float* partial;      // [windows][slices][Pp] of the last gradient launch
  const double* ll_partial;  // [windows][slices]
  const double* red_in;      // row sharding: [windows][Pp + 4] all-reduced sums, else null
  const float* w_new;        // [windows][Pp] proposal position
  const float* m_new;        // [windows][Pp] proposal momentum (before the closing half kick)
  float* m0;                 // [windows][Pp] momentum drawn for the running iteration
  float* w_cur;              // [windows][Pp] chain state
  float* g_cur;              // [windows][Pp] full gradient at the chain state
  double* ll_cur;            // [windows]
  double* lp_cur;            // [windows]
  float* eps;                // [windows]
  int* iter;                 // [windows]
  int* n_accept;             // [windows]
  const long long* gwin;     // [windows] global window ids (random-stream keys)
  float* w_start;            // [windows][Pp] where the next iteration starts from
  float* m_start;            // [windows][Pp]
  float* samples;            // [windows][sample_capacity][P]
  int sample_capacity;
  int burn_in;
  int adapt_steps;
  float log_target, dec_adj, inc_adj;
  unsigned long long seed;
  // trace of the first trace_iters iterations
  int trace_iters;
  float* tr_mom;             // [windows][trace_iters][P]
  float* tr_log_u;           // [windows][trace_iters]
  double* tr_log_acpt;
  int* tr_accept;
  float* tr_eps;
  PriorParams prior;
  // ACC_FINALIZE outputs (single window)
  float* g_out;              // [P]
  float* prior_loss_out;     // optional [P]
  double* scalars_out;       // [2]: loglik, logprior
  const int* status_in;      // optional: device error word; when it is set the scalars come out as NaN
  // the reference's random streams instead of Philox (main.h:207-216, :235-239)
  int ref_streams;
  const float* ref_log_u;    // [ref_cap] host-computed log accept draws, indexed by iteration % ref_cap
  int ref_cap;
};

cudaError_t launch_accept(const AcceptParams& a, int windows, cudaStream_t st);
cudaError_t launch_repack(const float* x, const float* y, float* out, long long n_rows,
                          long long rows_pad, int D, cudaStream_t st);
cudaError_t launch_reduce_partials(const float* partial, const double* ll_partial, int slices,
                                   const int* nslot, int P, int Pp, double* red, int windows,
                                   int num_sms, cudaStream_t st);
// One-shot all-reduce over peer memory for row sharding (chain.cu): what every rank's launch needs
constexpr int ONESHOT_SLICE = 32;   // parameters per CTA
constexpr int ONESHOT_MAX_RANKS = 16;
struct OneShotParams {
  // this rank's partial vectors, as for reduce_partials
  const float* partial;
  const double* ll_partial;
  int slices;
  const int* nslot;
  int P, Pp;
  double* red;                  // [Pp + 4] result, identical bits on every rank
  int rank, nranks;
  // every rank's receive buffer (this rank's own at [rank]): [2 halves][nranks][Pp + 4][2] words of
  // {32 bits of payload, sequence number}
  uint2* peer_words[ONESHOT_MAX_RANKS];
  const uint2* local_words;
  unsigned int* seq;            // device counter of completed exchanges on this rank
  unsigned int* done;           // ticket of the CTAs of one launch
  unsigned int poll_limit;      // bounded wait: polls before giving up
  int* status;
};
cudaError_t launch_oneshot_allreduce(const OneShotParams& p, cudaStream_t st);
// forward-only pass over (samples x rows) (forward.cu)
struct ForwardParams {
  const float* x;          // rows, x_stride floats apart (22 for caller rows, 24 for the repacked dataset)
  long long x_stride;
  const float* y;          // LOSS only: targets, y_stride floats apart
  long long y_stride;
  long long n;             // rows
  const float* samples;    // [count][P]
  int count;
  LikParams lik;
  double* partial;         // PREDICT: [forward_slots][n]   LOSS: [row tiles][count]
  int whole;               // every CTA takes whole row tiles, so that a row has one sum
  int* status;             // where a bounded wait that runs out leaves its code
  int test_code;           // self-test: 402 adds a wait for MMAs that nothing ends
};
constexpr int SPLIT_H = 40;  // units of the gradient kernels with split_mma.cuh
// rows of a CTA's tile: four or three 128-row tiles (forward.cu)
__host__ __device__ constexpr int forward_rows(int H) { return H == 40 ? 512 : 384; }
__host__ __device__ inline long long forward_tiles(int H, long long n) { return (n + forward_rows(H) - 1) / forward_rows(H); }
int forward_slots(int H, int num_sms, const ForwardParams& a);
cudaError_t launch_forward(int H, const ForwardParams& a, int num_sms, bool loss, cudaStream_t st);
cudaError_t launch_forward_finish_predict(int H, const ForwardParams& a, int num_sms, float* out, cudaStream_t st);
cudaError_t launch_forward_finish_loss(const double* partial, int tiles, int count, const float* samples, int P,
                                       const PriorParams& prior, double* out_ll, double* out_lp, cudaStream_t st);
cudaError_t launch_philox_probe(const uint32_t ctr[4], const uint32_t key[2], int n, uint32_t* raw, float* normals,
                                float* uniform, cudaStream_t st);
cudaError_t launch_refstream_momentum(unsigned long long first_n, int count, float* out, cudaStream_t st);
cudaError_t launch_wait_probe(int* status, unsigned int slices, cudaStream_t st);
cudaError_t launch_log_acpt(const float* prev_loss, const float* new_loss, long long n_loss,
                            const float* prev_mom, const float* new_mom, const float* grad_cur, int P,
                            float eps, float* out, cudaStream_t st);

// One cooperative launch for whole iterations / trajectories / evaluations of windows that fit on the chip
// (resident.cuh)
enum ResidentMode : int {
  RES_CHAIN = 0,  // n_iter HMC iterations of n_steps leapfrog steps from the chain state in `a`
  RES_STEPS = 1,  // n_steps leapfrog steps from (w0, m0, g0)
  RES_EVAL = 2    // log density and gradient at w0
};
constexpr int RES_UNITS = 16;          // 32-row units per CTA
constexpr int RES_MAX_CLUSTERS = 16;   // clusters of one window
constexpr unsigned int RES_WAIT_TICKS = 15000;  // about half a second
struct ResidentParams {
  int mode, n_steps, n_iter;
  int windows, clusters;    // clusters per window
  int data_window0, n_rows, rows_pad, Pp;
  const float* xaug;        // [windows][rows_pad][KP] (FP32; TF32 goes through the tensor map)
  uint4* msg;               // [2][windows][ranks][clusters][words] cluster sums
  unsigned int* seq;        // [windows] last sequence number used
  LikParams lik;
  PriorParams prior;
  int* status;
  int* status_host;         // optional: the same code for the host to read without a copy; also one that was set before
  unsigned int wait_ticks;  // limit of the waits, in 2^16 cycles
  int missing;              // self-test: clusters of the last window that do not start
  int test_code;            // self-test: 611 adds a wait for rows that nothing ends, FP32: 612, 613, 614 one for MMAs, for an accumulator, for a scale
  // RES_STEPS / RES_EVAL (one window); all outputs but g_out and scalars are optional
  const float *w0, *m0, *g0;
  float eps_scalar;
  float *w_out, *m_out, *g_out, *zero_out, *row_loss, *prior_loss;
  double* scalars;          // [2] log-likelihood, log-prior
  AcceptParams a;           // RES_CHAIN
};
// RES_EVAL with the parameters themselves in place of w0 (a type of its own: 3.8 KB more in every launch of a trajectory
// cost 0.7 us)
struct ResidentEvalParams : ResidentParams {
  float w_val[964];
};
// The launch, for clusters of `cluster` CTAs (1, 2, 4, 8); or, when max_clusters is given, only the number of such
// clusters that can be resident at once
cudaError_t launch_resident_tf32(int cluster, const void* tmap, const ResidentParams& g, cudaStream_t st,
                                 int* max_clusters);
cudaError_t launch_resident_fp32(int cluster, const void* tmap, const ResidentParams& g, cudaStream_t st,
                                 int* max_clusters);
// ... in FP32 of windows whose CTAs have 128 rows at most
bool resident_one_tile(int rows, int clusters, int cluster);
// ... of one leapfrog step of a window, for clusters of eight
cudaError_t launch_resident_step_fp32(const void* tmap, const ResidentParams& g, cudaStream_t st);
cudaError_t launch_resident_fp32_ffma(int cluster, const void* tmap, const ResidentParams& g, cudaStream_t st,
                                      int* max_clusters);
// ... of an evaluation with its parameters, for clusters of eight
cudaError_t launch_resident_eval_tf32(const void* tmap, const ResidentEvalParams& g, cudaStream_t st);
cudaError_t launch_resident_eval_fp32(const void* tmap, const ResidentEvalParams& g, cudaStream_t st);

// gradient kernels
cudaError_t launch_grad_fp32(int H, const GradParams& g, int slices, int windows, cudaStream_t st);
int fp32_max_ctas_per_sm(int H);
// FP32, 40 units, the forward product on the tensor core: persistent, over the work table in `g`, or one window in `ctas` slices
cudaError_t launch_grad_fp32_split(const GradParams& g, int ctas, cudaStream_t st);
// ... the sums over rows there too
cudaError_t launch_grad_fp32_int(const GradParams& g, int ctas, cudaStream_t st);
// Launches of so few tiles are one latency after the other, of which that kernel has more: us a step of one window, without the tensor
// core and with it, 4 tiles 7.8 and 9.0, 24 9.1 and 9.2, 32 9.3 and 9.4, 40 10.2 and 9.7, 148 11.7 and 10.6
inline bool fp32_few_tiles(long long tiles) { return tiles <= 32; }
int fp32_tile_rows(int H);

// TF32 (tcgen05) path: persistent, one CTA per SM; `tmaps` are CUtensorMaps over the repacked dataset: one that stages a
// row tile with the 32-byte-chunk swizzle and, for 128 units, a second with the 16-byte-chunk swizzle
cudaError_t launch_grad_tf32(int H, const void* tmaps, const GradParams& g, int ctas, cudaStream_t st);
int tf32_supported(int H);
cudaError_t launch_grad_tf32_wide(const void* tmaps, const GradParams& g, int ctas, cudaStream_t st);
constexpr int TF32_TILE = 128;
constexpr int WIDE_TILE = 64;  // rows of a tile of the 128-unit kernel

}  // namespace mcmc_b200
