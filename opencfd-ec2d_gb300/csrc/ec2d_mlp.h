// ec2d_mlp.h -- internal declarations of the warm-start network (k_mlp.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <mutex>
#include <vector>

namespace ec2d {

constexpr int NIN = 7;        // x, y, log10 dw, M, AoA (deg), log10 Re, t/c
constexpr int NIN_PAD = 64;   // input columns as the GEMMs see them
constexpr int NOUT = 5;       // rho, rho u, rho v, E, log1p(nu_tilde Re)
constexpr int NOUT_PAD = 128; // output rows of the last weight matrix
constexpr int MAX_HIDDEN = 12;
constexpr float ADAM_B1 = 0.9f, ADAM_B2 = 0.999f, ADAM_EPS = 1e-8f;
constexpr int KSPLIT = 32;    // K splits of the weight-gradient GEMM

enum { EPI_F32 = 0, EPI_BIAS = 1, EPI_BIAS_SILU = 2, EPI_DSILU = 3, EPI_BF16 = 4 };

// epilogue of C[M x N] = A[M x K] . B[N x K]^T
struct Epi {
  int mode;                 // EPI_*
  const float *bias;        // [N] (bias modes)
  float *zout;              // pre-activation out (EPI_BIAS_SILU), [M x ldz]
  const float *zin;         // pre-activation in (EPI_DSILU), [M x ldz]
  int ldz;
  __nv_bfloat16 *hout;      // bf16 out (EPI_BIAS_SILU, EPI_DSILU, EPI_BF16)
  float *fout;              // fp32 out (EPI_BIAS, EPI_F32)
  int ldc;
  long long split_stride;   // EPI_F32: offset between the K-split partial tiles
};

// tcgen05 (TMEM accumulator) GEMM, k_gemm_tc.cu: M % 128 == 0, N % 64 == 0,
// (K / ksplit) % 64 == 0.  err: device flag set if an mbarrier wait timed out.
void launch_gemm_tc(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, int M, int N, int K,
                    int ksplit, const Epi &e, int *err, cudaStream_t s);

// ---- the network at width 256 in fused kernels (k_mlp_fused.cu) ----
enum { FUSED_GATHER = 0, FUSED_STAGED = 1, FUSED_ROWS = 2 };  // where a tile's inputs come from
struct FusedArgs {
  int nlin, ntiles, mode, B;
  long long n;                          // samples (gather) or feature rows
  unsigned long long seed;
  const int *step;
  const float *feat, *targ, *nrm, *Y;
  const __nv_bfloat16 *X;               // staged inputs, row-major [B x NIN_PAD]
  const __nv_bfloat16 *wk[MAX_HIDDEN + 1], *wtk[MAX_HIDDEN + 1];  // packed weights and their transposes
  const float *bias[MAX_HIDDEN + 1];
  __nv_bfloat16 *H[MAX_HIDDEN], *dz[MAX_HIDDEN], *Xt, *dO;        // blocks of 128 rows (core-matrix layout)
  float *lrow, *pred;                   // squared error per row; predictions
  int *err;
};
struct PackArgs {
  int nlin;
  float b1, b2, eps;  // Adam
  float *w[MAX_HIDDEN + 1], *b[MAX_HIDDEN + 1], *mw[MAX_HIDDEN + 1], *vw[MAX_HIDDEN + 1], *mb[MAX_HIDDEN + 1],
      *vb[MAX_HIDDEN + 1], *gw[MAX_HIDDEN + 1], *gb[MAX_HIDDEN + 1];
  __nv_bfloat16 *wb[MAX_HIDDEN + 1], *wt[MAX_HIDDEN + 1], *wk[MAX_HIDDEN + 1], *wtk[MAX_HIDDEN + 1];
};
void launch_mlp_forward(const FusedArgs &a, cudaStream_t s);
void launch_mlp_train_tile(const FusedArgs &a, cudaStream_t s);
void launch_mlp_dw(const FusedArgs &a, float *part, long long unit_stride, int ks, int rows, cudaStream_t s);
void launch_mlp_reduce(const PackArgs &p, const float *part, long long unit_stride, int ks, const int *step, float lr,
                       int adam, cudaStream_t s);
void launch_mlp_bias(const FusedArgs &a, const PackArgs &p, float *cpart, int nb, const int *step, float lr, int adam,
                     float *loss, cudaStream_t s);
void launch_mlp_pack(const PackArgs &p, cudaStream_t s);

#ifdef __CUDACC__
// minibatch row k of a training step: hash(step, k) mod n
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ long long gather_row(unsigned long long seed, int step, unsigned k, long long n) {
  const unsigned long long h = mix64(seed ^ mix64(((unsigned long long)step << 32) | k));
  return (long long)(h % (unsigned long long)n);
}
#endif

struct Layer {
  float *w = nullptr, *b = nullptr;    // FP32 masters [out x in], [out]
  float *mw = nullptr, *vw = nullptr, *mb = nullptr, *vb = nullptr;  // Adam moments
  float *gw = nullptr, *gb = nullptr;  // gradients
  __nv_bfloat16 *wb = nullptr, *wt = nullptr;  // BF16 copy and its transpose
  __nv_bfloat16 *wk = nullptr, *wtk = nullptr;  // packed for the fused kernels (width 256)
};

constexpr int HOST_SLOTS = 4;  // chunks of a host prediction on the device

// Standardised rows that a host or the GEMM path's gather hands over (up to cap_stage
// rows); buffers of the GEMM path for batches of up to cap_batch rows; and of the fused
// training pass (width 256; up to cap_fused rows): activations and dZ in 128-row blocks,
// partial weight gradients of every layer.  Each set is replaced as a whole.
struct StageBuf {
  __nv_bfloat16 *X = nullptr;
  float *Y = nullptr;
};
struct BatchBuf {
  __nv_bfloat16 *H[MAX_HIDDEN] = {}, *dOut = nullptr, *dA = nullptr, *dB = nullptr, *T1 = nullptr, *T2 = nullptr;
  float *Z[MAX_HIDDEN] = {}, *out = nullptr, *part = nullptr, *cpart = nullptr, *lpart = nullptr;
};
struct FusedBuf {
  __nv_bfloat16 *Xt = nullptr, *Ht[MAX_HIDDEN] = {}, *dZt[MAX_HIDDEN] = {}, *dOt = nullptr;
  float *fpart = nullptr, *fcpart = nullptr, *lrow = nullptr;
};

struct Net : StageBuf, BatchBuf, FusedBuf {
  int device = 0, width = 256, nlin = 7;
  unsigned long long seed = 0;
  cudaStream_t stream = nullptr;
  Layer L[MAX_HIDDEN + 1];
  float *nrm = nullptr;  // feature mean[NIN], std[NIN], target mean[NOUT], std[NOUT]
  int *d_step = nullptr;
  int *d_err = nullptr;   // set by a tcgen05 GEMM whose mbarrier wait timed out
  int gemm_kind = 1;      // 1: tcgen05 GEMMs (default), 0: mma.sync GEMMs
  float *d_loss = nullptr;
  double *d_moments = nullptr;
  int cap_stage = 0, cap_batch = 0, cap_fused = 0;
  std::vector<void *> stage_mem, batch_mem, fused_mem;  // the memory of the sets
  // a second stream for the biases of the fused pass
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  // predictions for host rows: a ring of chunks on the device, kept with the net (at
  // most HOST_SLOTS chunks, 15 MB); one call at a time uses it
  std::mutex host_mu;
  float *host_in = nullptr, *host_out = nullptr;
  long long host_cap = 0;  // rows of the ring
  cudaStream_t copy = nullptr;
  cudaEvent_t ev_in[HOST_SLOTS] = {}, ev_out[HOST_SLOTS] = {};
  // samples (device): features n x NIN, targets n x NOUT
  float *feat = nullptr, *targ = nullptr;
  long long nsamp = 0, cap_samp = 0;
  cudaGraphExec_t train_graph = nullptr;  // one training step (gather, forward, backward, Adam)
  int graph_batch = 0, graph_kind = -1;
  float graph_lr = 0.0f;
  std::vector<void *> owned;

  int init(int dev, int hidden, int width, unsigned long long seed);
  void destroy();
  int layer_in(int l) const;
  int layer_out(int l) const;
  void refresh_bf16();
  void gemm(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, int M, int N, int K, int ksplit,
            const Epi &e);
  int ensure_stage(int B);
  int ensure_batch(int B);
  bool fused() const { return width == 256 && gemm_kind == 1; }
  int ensure_fused(int B);
  FusedArgs fused_args(int B, int mode) const;
  PackArgs pack_args() const;
  void fused_pass(int B, int mode, bool adam, float lr);  // forward, backward and (adam) the update
  void forward(int B);
  void backward(int B);
  void adam(float lr);
  void gather(int B);
  void train_step(int B, float lr);  // minibatch, forward, backward, Adam
  void drop_graph();
  int fit_normalization();
  int reserve_samples(long long n);
  int predict(const float *feat, long long n, float *pred);
  int predict_host(const float *feat, long long n, float *pred);  // rows in host memory
  int check_err();  // 0, or 1 if a tcgen05 wait timed out since the last call
};

}  // namespace ec2d
