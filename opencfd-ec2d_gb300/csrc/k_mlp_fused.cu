// k_mlp_fused.cu -- the warm-start network (k_mlp.cu) at width 256 in three
// kernels per training step and one per prediction, on the 5th-generation
// tensor cores.
//
//   k_mlp_tile     a CTA takes 128 rows through every layer: the inputs are
//                  gathered and standardised, each layer's activations stay in
//                  shared memory as the next layer's A operand, and in
//                  training the loss gradient goes back through the layers the
//                  same way.  The pre-activations a backward layer needs are
//                  formed again by a second MMA from the stored activations
//                  (two bytes per value) instead of being stored themselves
//                  (four bytes written and read).
//   k_mlp_dw       the weight gradients dZ^T H of all layers, split over the
//                  batch
//   k_mlp_reduce   sums the splits in order, Adam, and the bf16 copies
// What bounds k_mlp_tile is the SiLU: an exponential and a reciprocal per value
// on the special-function unit (16 a cycle and SM: 4,096 cycles per 128 x 256
// tile), against 2,100 cycles of MMA, so the MMAs of a layer follow its
// epilogue 64 columns behind.  Before, every layer was a GEMM launch whose
// operands and FP32 pre-activations went through HBM, and the weight gradient
// needed both operands transposed.
//
// Measured (GB300, 6 hidden layers): a training step of 16,384 rows 742 -> 168
// us (tile kernel 88 us, weight gradients 27, reduce 17, and beside those two the column
// sums 24 and the bias update 13; each alone, ncu), 46 -> 194 TFLOP/s;
// predictions of 300,007 rows 2.9 -> 0.43 ms in the kernel.  The training tile
// kernel is bound by the weights its 128 CTAs each read from L2 (310 MB a step).
//
// Arithmetic is that of the separate kernels (k_gemm_tc.cu, k_mlp.cu): BF16
// operands, FP32 accumulation over K in steps of 16 in the same order, the
// same splits of the batch summed in the same order, so a training run gives
// the same weights (below z = -87 SiLU is about -1e-36 here and rounds to -0 there).
//
// Layout.  Activations (and dZ) of 128 rows x 256 columns are a block of 8 x 8
// core matrices of 128 contiguous bytes (8 rows of 16 bytes): row group r / 8
// at 4,096 bytes, column group c / 8 at 128 bytes.  The block is the K-major
// operand of the layer products (rows are M, columns K) and, read with the
// other strides, the MN-major operand of the weight gradient (columns are M or
// N, rows K), so nothing is ever transposed, and it moves between shared and
// global memory as one bulk copy.  Weights are packed the same way per 32 of K
// by the kernel that updates them.
//
// Every wait is bounded: one that runs out sets *err and `dead`, after which
// no role waits or issues any more, and the CTA leaves through the common exit.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "ec2d_mlp.h"

namespace ec2d {
namespace fused {

constexpr int W = 256, TILE_B = 128 * W * 2, SMALL_B = 128 * 16 * 2;  // bytes of a 128-row block, of a 16-column one
constexpr int STAGE_B = W * 32 * 2;  // a weight chunk: 256 rows x 32 of K
constexpr int WAIT_LIMIT = 1 << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t a, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t a) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t a, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, unsigned bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ void bulk_store(void *dst, uint32_t src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ bool wait(uint32_t a, unsigned parity, volatile int *dead, int *err) {
  for (int it = 0; it < WAIT_LIMIT; it++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, "
        "p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity & 1u)
        : "memory");
    if (done) return true;
    if (*dead) return false;
  }
  *dead = 1;
  atomicExch(err, 1);
  return false;
}
// shared-memory operand descriptor, no swizzle (see k_gemm_tc.cu)
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)((lbo >> 4) & 0x3FFF) << 16 |
         (uint64_t)((sbo >> 4) & 0x3FFF) << 32 | (uint64_t)1 << 46;
}
// instruction descriptor, kind::f16, BF16 operands, FP32 accumulators; mn: both
// operands MN-major
__host__ __device__ constexpr uint32_t idesc(int M, int N, bool mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (mn ? (1u << 15) | (1u << 16) : 0u) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t id, bool acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(a), "l"(b), "r"(id), "r"((uint32_t)acc)
      : "memory");
}
__device__ __forceinline__ void commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t (&v)[32], uint32_t a) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(a));
}
__device__ __forceinline__ void tmem_ld16(uint32_t (&v)[16], uint32_t a) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(a));
}

// n / d for d >= 1, rounded to nearest but for rare ties: the quotient by the
// approximate reciprocal, corrected by its exact remainder (Markstein, IBM J.
// Res. Dev. 34, 1990).  d is at most 2^126 here (exp_neg), so 1/d is normal.
__device__ __forceinline__ float quotient(float n, float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = n * r;
  return fmaf(fmaf(-q, d, n), r, q);
}
// exp(-z) as k_mlp.cu forms it, held below 2^126 (SiLU is 0 to 36 digits there)
__device__ __forceinline__ float exp_neg(float z) { return fminf(__expf(-z), 0x1p126f); }
// (z itself where the denominator is 1: also keeps infinities)
__device__ __forceinline__ float silu(float z) {
  const float d = 1.0f + exp_neg(z);
  return d == 1.0f ? z : quotient(z, d);
}
__device__ __forceinline__ float dsilu(float z) {
  const float s = quotient(1.0f, 1.0f + exp_neg(z));
  return s * (1.0f + z * (1.0f - s));
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ void sts16(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// The three forms of the tile kernel.
//   FORM_TRAIN   forward, loss gradient and backward of tile blockIdx.x
//   FORM_ONE     forward of tiles blockIdx.x, + gridDim.x, ... with predictions out, a
//                CTA per SM: sixteen epilogue warps on one tile, the MMAs of a
//                layer 64 columns behind the epilogue of the last (with eight warps alone
//                a layer took 8,000 cycles)
//   FORM_TWO     the same with two CTAs per SM of eight epilogue warps, one accumulator
//                and a short weight ring each: one CTA's MMAs run under the other's
//                epilogue.  A tile took 53,900 cycles in FORM_ONE, with the special-function
//                unit 46 % and the issue slots 49 % busy.  For more tiles than
//                SMs; up to that a tile alone is faster in FORM_ONE.
enum { FORM_TRAIN, FORM_ONE, FORM_TWO };
template <int FORM>
struct Form {
  static constexpr bool TRAIN = FORM == FORM_TRAIN, TWO = FORM == FORM_TWO;
  static constexpr int EW = TWO ? 8 : 16, ECOL = 64 / (EW / 4);  // epilogue warps; columns of each 64 a warp takes
  static constexpr int NSTAGE = TWO ? 2 : 5, COLS = TWO ? W : 2 * W;  // weight ring; TMEM columns
  static constexpr int THREADS = 32 * (EW + 2);
  static constexpr int S_A = 0, S_E = S_A + TILE_B, S_X = S_E + (TRAIN ? TILE_B : 0), S_O = S_X + SMALL_B,
                       S_W = S_O + (TRAIN ? SMALL_B : 0), S_END = S_W + NSTAGE * STAGE_B;
};

// Warps 0 to EW - 1: inputs and epilogues (warp w: rows 32 (w % 4) .. of the tile,
// columns ECOL (w / 4) .. of each 64); then one warp for the bulk copies and one for
// MMAs and TMEM.
template <int FORM>
__global__ void __launch_bounds__(Form<FORM>::THREADS, Form<FORM>::TWO ? 2 : 1)
    k_mlp_tile(const __grid_constant__ FusedArgs a) {
  using C = Form<FORM>;
  constexpr bool TRAIN = C::TRAIN;
  constexpr int EW = C::EW, ECOL = C::ECOL, NSTAGE = C::NSTAGE, S_A = C::S_A, S_E = C::S_E, S_X = C::S_X, S_O = C::S_O,
                S_W = C::S_W, NACC = C::COLS / W;  // accumulators
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t bars[2 * NSTAGE + 4 + 4];
  __shared__ uint32_t tmem_sh;
  __shared__ int dead_sh;
  volatile int *dead = &dead_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t s0 = smem_u32(smem), b0 = smem_u32(bars);
  auto wfull = [&](int s) { return b0 + 8u * s; };
  auto wempty = [&](int s) { return b0 + 8u * (NSTAGE + s); };
  auto afull = [&](int c) { return b0 + 8u * (2 * NSTAGE + c); };
  const uint32_t accfull = b0 + 8u * (2 * NSTAGE + 4), hfull = accfull + 8, hdone = accfull + 16, efree = accfull + 24;
  const int nl = a.nlin;
  if (warp == EW + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)), "n"(C::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < 2 * NSTAGE; s++) mbar_init(b0 + 8u * s, 1);
    for (int c = 0; c < 4; c++) mbar_init(afull(c), EW);
    for (int c = 0; c < 4; c++) mbar_init(accfull + 8u * c, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    dead_sh = 0;
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_sh;
  const int step_tiles = TRAIN ? a.ntiles : (int)gridDim.x;

  if (warp == EW) {
    // ---- weights through the ring; stored activations for the backward MMAs
    if (lane == 0) {
      int s = 0;
      unsigned use = 0;  // rounds of the ring
      auto put = [&](const void *src, unsigned bytes) {
        if (!wait(wempty(s), (use & 1u) ^ 1u, dead, a.err)) return;
        mbar_expect(wfull(s), bytes);
        bulk_load(s0 + S_W + s * STAGE_B, src, bytes, wfull(s));
        if (++s == NSTAGE) { s = 0; use++; }
      };
      // layer l forward (B rows: its outputs), its chunks of K
      auto put_w = [&](int l) {
        if (l == 0) { put(a.wk[0], W * 16 * 2); return; }
        const unsigned bytes = (l < nl - 1 ? W : 16) * 32 * 2;
        for (int c = 0; c < W / 32; c++) put(reinterpret_cast<const uint8_t *>(a.wk[l]) + (size_t)c * bytes, bytes);
      };
      auto put_wt = [&](int l) {  // transposed (B rows: its inputs)
        if (l == nl - 1) { put(a.wtk[l], W * 16 * 2); return; }
        for (int c = 0; c < W / 32; c++) put(reinterpret_cast<const uint8_t *>(a.wtk[l]) + (size_t)c * STAGE_B, STAGE_B);
      };
      for (int t = blockIdx.x; t < a.ntiles && !*dead; t += step_tiles) {
        for (int l = 0; l < nl; l++) put_w(l);
        if (TRAIN) {
          wait(hdone, 0, dead, a.err);
          int n = 0;
          for (int l = nl - 1; l >= 1; l--) {
            if (l >= 2) {  // H of layer l - 2, operand of the pre-activations of layer l - 1
              if (n > 0) wait(efree, (n - 1) & 1u, dead, a.err);
              if (*dead) break;
              mbar_expect(hfull, TILE_B);
              bulk_load(s0 + S_E, reinterpret_cast<const uint8_t *>(a.H[l - 2]) + (size_t)t * TILE_B, TILE_B, hfull);
              n++;
            }
            put_wt(l);
            put_w(l - 1);
          }
        }
      }
    }
  } else if (warp == EW + 1) {
    // ---- MMAs
    if (lane == 0) {
      int s = 0;
      unsigned use = 0, gen = 0;
      // one product: A from `abase` (K of 256 in the block layout, or 16), N
      // columns, weights from the ring; ready(c): waits for 64 columns of A
      auto product = [&](uint32_t abase, bool k16, int N, uint32_t col, auto ready) {
        const uint32_t id = idesc(128, N, false);
        for (int c = 0; c < (k16 ? 1 : W / 32); c++) {
          if ((c & 1) == 0 && !ready(c >> 1)) return;
          if (!wait(wfull(s), use & 1u, dead, a.err)) return;
          fence_after();
          const uint32_t sb = s0 + S_W + s * STAGE_B;
          if (k16) {
            mma(tmem + col, sdesc(abase, 128, 256), sdesc(sb, 128, 256), id, false);
          } else {
#pragma unroll
            for (int k = 0; k < 2; k++)
              mma(tmem + col, sdesc(abase + (4 * c + 2 * k) * 128, 128, 4096), sdesc(sb + k * 256, 128, 512), id,
                  c > 0 || k > 0);
          }
          commit(wempty(s));
          if (++s == NSTAGE) { s = 0; use++; }
        }
      };
      for (int t = blockIdx.x; t < a.ntiles && !*dead; t += step_tiles) {
        for (int l = 0; l < nl; l++, gen++) {
          // (one accumulator: only once the epilogue has read all of it)
          if (C::TWO)
            for (int c = 0; c < 4; c++) wait(afull(c), gen & 1u, dead, a.err);
          product(s0 + (l == 0 ? S_X : S_A), l == 0, l < nl - 1 ? W : 16, (l % NACC) * W,
                  [&](int c) { return C::TWO ? !*dead : wait(afull(c), gen & 1u, dead, a.err); });
          // the chunks of A that a one-chunk product did not wait for
          if (!C::TWO && l == 0)
            for (int c = 1; c < 4; c++) wait(afull(c), gen & 1u, dead, a.err);
          commit(accfull);
        }
        if (TRAIN) {
          unsigned n = 0;
          for (int l = nl - 1; l >= 1; l--, gen++) {
            // dH of layer l - 1: all of dZ is there and the epilogue has read
            // both accumulators of the layer before
            for (int c = 0; c < 4; c++) wait(afull(c), gen & 1u, dead, a.err);
            product(s0 + (l == nl - 1 ? S_O : S_A), l == nl - 1, W, 0, [](int) { return true; });
            // pre-activations of layer l - 1
            if (l >= 2) wait(hfull, n++ & 1u, dead, a.err);
            product(s0 + (l >= 2 ? S_E : S_X), l < 2, W, W, [](int) { return true; });
            if (l >= 2) commit(efree);
            commit(accfull);
          }
        }
      }
    }
  } else {
    // ---- inputs and epilogues
    const int r = (warp & 3) * 32 + lane, h = warp >> 2;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t arow = s0 + S_A + (r >> 3) * 4096 + (r & 7) * 16;
    unsigned acc = 0;  // accumulators waited for
    auto ready = [&](int c) {
      fence_before();
      proxy_fence();
      __syncwarp();
      if (lane == 0) mbar_arrive(afull(c));
    };
    auto epi_barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * EW) : "memory"); };
    auto stores_read = [&] {  // the last bulk store has read its shared memory
      if (TRAIN) {
        if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        epi_barrier();
      }
    };
    auto store_tile = [&](void *dst, uint32_t src, unsigned bytes) {
      epi_barrier();
      if (tid == 0) bulk_store(dst, src, bytes);
    };
    // (after a wait that gave up every role runs on without waiting, so that the
    // barriers among the epilogue warps stay matched)
    for (int t = blockIdx.x; t < a.ntiles && (TRAIN || !*dead); t += step_tiles) {
      const long long row = (long long)t * 128 + r;
      long long src = row;
      if (h == 0) {
        // standardised inputs: 7 features, zeros to 16 columns
        uint32_t v[4];
        if (a.mode == FUSED_STAGED) {
          const uint4 *x = reinterpret_cast<const uint4 *>(a.X + (size_t)row * NIN_PAD);
          const uint4 q = x[0];
          v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
          if (a.mode == FUSED_GATHER) src = gather_row(a.seed, *a.step, (unsigned)row, a.n);
          float f[8];
#pragma unroll
          for (int c = 0; c < 8; c++)
            f[c] = (c < NIN && src < a.n) ? (a.feat[src * NIN + c] - a.nrm[c]) / a.nrm[NIN + c] : 0.0f;
#pragma unroll
          for (int k = 0; k < 4; k++) v[k] = pack2(f[2 * k], f[2 * k + 1]);
        }
        const uint32_t x = s0 + S_X + (r >> 3) * 256 + (r & 7) * 16;
        sts16(x, v[0], v[1], v[2], v[3]);
        sts16(x + 128, 0, 0, 0, 0);
      }
      for (int c = 0; c < 4; c++) ready(c);
      if (TRAIN) store_tile(reinterpret_cast<uint8_t *>(a.Xt) + (size_t)t * SMALL_B, s0 + S_X, SMALL_B);
      for (int l = 0; l < nl - 1; l++) {
        wait(accfull, acc++, dead, a.err);
        fence_after();
        stores_read();
        const float *bias = a.bias[l];
#pragma unroll 1
        for (int c = 0; c < 4; c++) {
          const int col = c * 64 + h * ECOL;
          uint32_t v[ECOL];
          if constexpr (ECOL == 32) tmem_ld32(v, lane_base + (l % NACC) * W + col);
          else tmem_ld16(v, lane_base + (l % NACC) * W + col);
          ld_wait();
#pragma unroll
          for (int p = 0; p < ECOL / 8; p++) {
            float z[8];
#pragma unroll
            for (int k = 0; k < 8; k += 4) {
              const float4 b = __ldg(reinterpret_cast<const float4 *>(bias + col + 8 * p + k));
              z[k] = silu(__uint_as_float(v[8 * p + k]) + b.x);
              z[k + 1] = silu(__uint_as_float(v[8 * p + k + 1]) + b.y);
              z[k + 2] = silu(__uint_as_float(v[8 * p + k + 2]) + b.z);
              z[k + 3] = silu(__uint_as_float(v[8 * p + k + 3]) + b.w);
            }
            sts16(arow + (col / 8 + p) * 128, pack2(z[0], z[1]), pack2(z[2], z[3]), pack2(z[4], z[5]), pack2(z[6], z[7]));
          }
          ready(c);
        }
        if (TRAIN) store_tile(reinterpret_cast<uint8_t *>(a.H[l]) + (size_t)t * TILE_B, s0 + S_A, TILE_B);
      }
      // outputs
      wait(accfull, acc++, dead, a.err);
      fence_after();
      if (h == 0) {
        uint32_t v[16];
        tmem_ld16(v, lane_base + ((nl - 1) % NACC) * W);
        ld_wait();
        if (!TRAIN) {
          if (row < a.n)
#pragma unroll
            for (int c = 0; c < NOUT; c++)
              a.pred[row * NOUT + c] =
                  (__uint_as_float(v[c]) + a.bias[nl - 1][c]) * a.nrm[2 * NIN + NOUT + c] + a.nrm[2 * NIN + c];
        } else {
          // squared error of the row and its gradient, as k_loss
          float l = 0.0f, g[8] = {};
#pragma unroll
          for (int c = 0; c < NOUT; c++) {
            const float y = a.mode == FUSED_STAGED
                                ? a.Y[row * NOUT + c]
                                : (a.targ[src * NOUT + c] - a.nrm[2 * NIN + c]) / a.nrm[2 * NIN + NOUT + c];
            const float e = (__uint_as_float(v[c]) + a.bias[nl - 1][c]) - y;
            l += e * e;
            g[c] = 2.0f * e / (float)(a.B * NOUT);
          }
          a.lrow[row] = l;
          const uint32_t o = s0 + S_O + (r >> 3) * 256 + (r & 7) * 16;
          sts16(o, pack2(g[0], g[1]), pack2(g[2], g[3]), pack2(g[4], g[5]), pack2(g[6], g[7]));
          sts16(o + 128, 0, 0, 0, 0);
        }
      }
      if (TRAIN) {
        // every stored H has reached memory before the copies that read it
        if (tid == 0) {
          asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
          asm volatile("fence.proxy.async;" ::: "memory");
          mbar_arrive(hdone);
        }
        for (int c = 0; c < 4; c++) ready(c);
        store_tile(reinterpret_cast<uint8_t *>(a.dO) + (size_t)t * SMALL_B, s0 + S_O, SMALL_B);
        for (int l = nl - 1; l >= 1; l--) {
          wait(accfull, acc++, dead, a.err);
          fence_after();
          stores_read();
          const float *bias = a.bias[l - 1];
#pragma unroll 1
          for (int c = 0; c < 4; c++) {
            const int col = c * 64 + h * ECOL;
            uint32_t v[16], z[16];  // (ECOL)
            tmem_ld16(v, lane_base + col);
            tmem_ld16(z, lane_base + W + col);
            ld_wait();
#pragma unroll
            for (int p = 0; p < ECOL / 8; p++) {
              float d[8];
#pragma unroll
              for (int k = 0; k < 8; k += 4) {
                const float4 b = __ldg(reinterpret_cast<const float4 *>(bias + col + 8 * p + k));
                const int q = 8 * p + k;
                d[k] = __uint_as_float(v[q]) * dsilu(__uint_as_float(z[q]) + b.x);
                d[k + 1] = __uint_as_float(v[q + 1]) * dsilu(__uint_as_float(z[q + 1]) + b.y);
                d[k + 2] = __uint_as_float(v[q + 2]) * dsilu(__uint_as_float(z[q + 2]) + b.z);
                d[k + 3] = __uint_as_float(v[q + 3]) * dsilu(__uint_as_float(z[q + 3]) + b.w);
              }
              sts16(arow + (col / 8 + p) * 128, pack2(d[0], d[1]), pack2(d[2], d[3]), pack2(d[4], d[5]), pack2(d[6], d[7]));
            }
            ready(c);
          }
          store_tile(reinterpret_cast<uint8_t *>(a.dz[l - 1]) + (size_t)t * TILE_B, s0 + S_A, TILE_B);
        }
      }
    }
    if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  if (*dead)  // copies and MMAs in flight end before the shared memory is given up
    for (int k = 0; k < 1000; k++) __nanosleep(1000);
  if (warp == EW + 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(C::COLS) : "memory");
}

// ---- weight gradients -------------------------------------------------------
// Unit u = 2 layer + half: 128 rows (half) of dW of the layer; split
// blockIdx.x of the batch.  Hidden layers: dZ^T H of the layer before (N =
// 256); layer 0: dZ^T X (N = 16); the last layer transposed, H^T dO (N = 16).
// Both operands are read MN-major from the 128-row blocks: 64 batch rows (K)
// per stage.  Partial sums go out four columns at a time, [N / 4][128][4].
constexpr int DW_A = 64 * 128 * 2, DW_B = 64 * W * 2, DW_STAGE = DW_A + DW_B, DW_NS = 2;
__global__ void __launch_bounds__(192, 2) k_mlp_dw(const __grid_constant__ FusedArgs a, float *__restrict__ part,
                                                   long long unit_stride, int rows) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t bars[2 * DW_NS + 1];
  __shared__ uint32_t tmem_sh;
  __shared__ int dead_sh;
  volatile int *dead = &dead_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t s0 = smem_u32(smem), b0 = smem_u32(bars);
  auto full = [&](int s) { return b0 + 8u * s; };
  auto empty = [&](int s) { return b0 + 8u * (DW_NS + s); };
  const uint32_t done = b0 + 8u * 2 * DW_NS;
  const int l = blockIdx.y >> 1, half = blockIdx.y & 1, nl = a.nlin, last = nl - 1;
  const bool wide = l > 0 && l < last;
  const uint8_t *A = reinterpret_cast<const uint8_t *>(l < last ? a.dz[l] : a.H[l - 1]);
  const uint8_t *B = reinterpret_cast<const uint8_t *>(l == 0 ? a.Xt : l == last ? a.dO : a.H[l - 1]);
  const int r0 = blockIdx.x * rows, nst = rows / 64;
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(&tmem_sh)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < 2 * DW_NS + 1; s++) mbar_init(b0 + 8u * s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    dead_sh = 0;
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_sh;
  if (warp == 4 && lane == 0) {
    for (int k = 0; k < nst && !*dead; k++) {
      const int s = k % DW_NS, row = r0 + 64 * k;
      if (!wait(empty(s), ((k / DW_NS) & 1) ^ 1, dead, a.err)) break;
      const size_t t = row / 128, g = (row % 128) / 8;  // block and its first row group
      mbar_expect(full(s), DW_A + (wide ? DW_B : 64 * 16 * 2));
      for (int q = 0; q < 8; q++)
        bulk_load(s0 + s * DW_STAGE + q * 2048, A + t * TILE_B + (g + q) * 4096 + half * 2048, 2048, full(s));
      if (wide) bulk_load(s0 + s * DW_STAGE + DW_A, B + t * TILE_B + g * 4096, DW_B, full(s));
      else bulk_load(s0 + s * DW_STAGE + DW_A, B + t * SMALL_B + g * 256, 64 * 16 * 2, full(s));
    }
  } else if (warp == 5 && lane == 0) {
    const uint32_t id = idesc(128, wide ? W : 16, true), kb = wide ? 4096 : 256;
    for (int k = 0; k < nst && !*dead; k++) {
      const int s = k % DW_NS;
      if (!wait(full(s), (k / DW_NS) & 1, dead, a.err)) break;
      fence_after();
      const uint32_t sa = s0 + s * DW_STAGE, sb = sa + DW_A;
#pragma unroll
      for (int q = 0; q < 4; q++)  // 16 batch rows: two row groups
        mma(tmem, sdesc(sa + q * 2 * 2048, 2048, 128), sdesc(sb + q * 2 * kb, kb, 128), id, k > 0 || q > 0);
      commit(empty(s));
    }
    commit(done);
  } else if (warp < 4) {
    if (wait(done, 0, dead, a.err) && !*dead) {
      fence_after();
      const int row = warp * 32 + lane;
      const uint32_t base = tmem + ((uint32_t)(warp * 32) << 16);
      float4 *out = reinterpret_cast<float4 *>(part + blockIdx.y * unit_stride + (size_t)blockIdx.x * 128 * W) + row;
      if (wide) {
#pragma unroll 1
        for (int c = 0; c < W; c += 32) {
          uint32_t v[32];
          tmem_ld32(v, base + c);
          ld_wait();
#pragma unroll
          for (int q = 0; q < 8; q++)
            out[(size_t)(c / 4 + q) * 128] = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                                         __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
        }
      } else {
        uint32_t v[16];
        tmem_ld16(v, base);
        ld_wait();
#pragma unroll
        for (int q = 0; q < 4; q++)
          out[(size_t)q * 128] = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                             __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
      }
    }
  }
  fence_before();
  __syncthreads();
  if (*dead)
    for (int k = 0; k < 1000; k++) __nanosleep(1000);
  if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
}

// Adam on one weight with the roundings of k_adam as it is compiled (checked
// bit for bit); p1, p2: 1 - b^t
__device__ __forceinline__ float adam1(const PackArgs &p, float w, float &m, float &v, float gr, float p1, float p2,
                                       float lr) {
  const float mk = __fmaf_rn(1.0f - p.b1, gr, __fmul_rn(p.b1, m));
  const float vk = __fmaf_rn(__fmul_rn(1.0f - p.b2, gr), gr, __fmul_rn(p.b2, v));
  m = mk;
  v = vk;
  const float mh = mk / p1, vh = vk / p2;
  return __fsub_rn(w, __fdiv_rn(__fmul_rn(lr, mh), __fadd_rn(sqrtf(vh), p.eps)));
}
// the bf16 copies of weight (r, c) of layer l: row-major, transposed, and packed
// for the two products
__device__ __forceinline__ void put_bf16(const PackArgs &p, int l, int r, int c, float w) {
  const __nv_bfloat16 h = __float2bfloat16_rn(w);
  const int ni = l == 0 ? NIN_PAD : W, no = l == p.nlin - 1 ? NOUT_PAD : W;
  p.wb[l][(size_t)r * ni + c] = h;
  p.wt[l][(size_t)c * no + r] = h;
  if (l == 0) {
    if (c < 16) p.wk[0][(r >> 3) * 128 + (c >> 3) * 64 + (r & 7) * 8 + (c & 7)] = h;
  } else if (l < p.nlin - 1) {
    p.wk[l][(c >> 5) * (W * 32) + (r >> 3) * 256 + ((c >> 3) & 3) * 64 + (r & 7) * 8 + (c & 7)] = h;
    p.wtk[l][(r >> 5) * (W * 32) + (c >> 3) * 256 + ((r >> 3) & 3) * 64 + (c & 7) * 8 + (r & 7)] = h;
  } else if (r < 16) {
    p.wk[l][(c >> 5) * (16 * 32) + (r >> 3) * 256 + ((c >> 3) & 3) * 64 + (r & 7) * 8 + (c & 7)] = h;
    p.wtk[l][(c >> 3) * 128 + (r >> 3) * 64 + (c & 7) * 8 + (r & 7)] = h;
  }
}
__global__ void k_mlp_pack(const __grid_constant__ PackArgs p) {
  const int l = blockIdx.y, ni = l == 0 ? NIN_PAD : W, no = l == p.nlin - 1 ? NOUT_PAD : W;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < ni * no) put_bf16(p, l, k / ni, k % ni, p.w[l][k]);
}

// the splits of every unit summed in order; the gradient out, and (adam) the
// update.  A block has 32 rows x 32 columns of a unit's partial tiles: summed as
// they lie (four columns of a row per thread, 512 contiguous bytes per 32
// rows), then turned in shared memory so that the weights, their moments and
// the gradient are read and written along rows of the weight matrix.
__global__ void __launch_bounds__(256) k_mlp_reduce(const __grid_constant__ PackArgs p, const float *__restrict__ part,
                                                    long long unit_stride, int ks, const int *__restrict__ step, float lr,
                                                    int adam) {
  __shared__ float tile[32][33];  // [row of the unit][column]
  const int l = blockIdx.y >> 1, half = blockIdx.y & 1, last = p.nlin - 1;
  const int cols = l > 0 && l < last ? W : 16;
  const int r0 = (blockIdx.x & 3) * 32, c0 = (blockIdx.x >> 2) * 32;
  if (c0 >= cols) return;
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  if (c0 + 4 * q < cols) {
    const float4 *src = reinterpret_cast<const float4 *>(part + blockIdx.y * unit_stride) + (c0 / 4 + q) * 128 + r0 + lane;
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 16
    for (int z = 0; z < ks; z++) {
      const float4 v = __ldcg(src + (size_t)z * (128 * W / 4));
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    tile[lane][4 * q] = s.x; tile[lane][4 * q + 1] = s.y; tile[lane][4 * q + 2] = s.z; tile[lane][4 * q + 3] = s.w;
  }
  float p1 = 1.0f, p2 = 1.0f;
  if (adam) {
    const float t = (float)*step;
    p1 = 1.0f - powf(p.b1, t);
    p2 = 1.0f - powf(p.b2, t);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; k++) {
    // lanes along a row of the weights: the unit's columns, or its rows where the
    // unit is the transposed product
    const int a = q + 8 * k, i = l == last ? lane : a, j = l == last ? a : lane;  // unit row, column
    if (c0 + j >= cols) continue;
    const int r = l == last ? c0 + j : half * 128 + r0 + i, c = l == last ? half * 128 + r0 + i : c0 + j;
    const size_t at = (size_t)r * (l == 0 ? NIN_PAD : W) + c;
    const float g = tile[i][j];
    p.gw[l][at] = g;
    if (adam) {
      float m = p.mw[l][at], v = p.vw[l][at];
      const float w = adam1(p, p.w[l][at], m, v, g, p1, p2, lr);
      p.mw[l][at] = m; p.vw[l][at] = v; p.w[l][at] = w;
      put_bf16(p, l, r, c, w);
    }
  }
}

// column sums of dZ (bias gradients): 256-row partials in row order, one warp
// per layer and 256 rows, a lane's 8 columns of a row group being 128
// contiguous bytes
__global__ void __launch_bounds__(32) k_mlp_colsum(const __grid_constant__ FusedArgs a, float *__restrict__ cpart, int nb) {
  const int l = blockIdx.y, lane = threadIdx.x;
  const bool last = l == a.nlin - 1;
  if (last && lane >= 2) return;
  const uint8_t *src = reinterpret_cast<const uint8_t *>(last ? a.dO : a.dz[l]) + lane * 128;
  const int stride = last ? 256 : 4096;
  float s[8] = {};
#pragma unroll 4
  for (int g = 0; g < 32; g++) {
    const uint4 *q = reinterpret_cast<const uint4 *>(src + (size_t)(blockIdx.x * 32 + g) * stride);
    uint4 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = __ldg(q + k);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const uint32_t w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
      for (int c = 0; c < 4; c++) {
        s[2 * c] += __uint_as_float(w[c] << 16);
        s[2 * c + 1] += __uint_as_float(w[c] & 0xffff0000u);
      }
    }
  }
  float *o = cpart + ((size_t)l * nb + blockIdx.x) * W + lane * 8;
#pragma unroll
  for (int c = 0; c < 8; c++) o[c] = s[c];
}
// their sums in order and Adam on the biases; block nlin: the loss of the batch
// (the tree over 256 rows and the sum over blocks of k_loss, k_loss_final)
__global__ void __launch_bounds__(256) k_mlp_bias(const __grid_constant__ PackArgs p, const float *__restrict__ cpart,
                                                  int nb, const int *__restrict__ step, float lr, int adam,
                                                  const float *__restrict__ lrow, int B, float *__restrict__ loss) {
  const int l = blockIdx.x, c = threadIdx.x;
  if (l == p.nlin) {
    // a warp per 256 rows: the tree of k_loss (row t takes row t + s for s = 128,
    // 64, 32 in the lane's registers, then across lanes)
    __shared__ float sums[8];
    const int lane = c & 31, w = c >> 5;
    double total = 0.0;
    for (int k0 = 0; k0 < nb; k0 += 8) {
      if (k0 + w < nb) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = lrow[(size_t)(k0 + w) * 256 + 32 * k + lane];
#pragma unroll
        for (int h = 4; h > 0; h >>= 1)
#pragma unroll
          for (int k = 0; k < h; k++) v[k] += v[k + h];
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) v[0] += __shfl_down_sync(0xffffffffu, v[0], s);
        if (lane == 0) sums[w] = v[0];
      }
      __syncthreads();
      if (c == 0)
        for (int k = 0; k < min(8, nb - k0); k++) total += sums[k];
      __syncthreads();
    }
    if (c == 0) *loss = (float)(total / ((double)B * NOUT));
    return;
  }
  const int n = l == p.nlin - 1 ? 16 : W;
  if (c >= n) return;
  float s = 0.0f;
#pragma unroll 8
  for (int z = 0; z < nb; z++) s += cpart[((size_t)l * nb + z) * W + c];
  p.gb[l][c] = s;
  if (adam) {
    const float t = (float)*step;
    float m = p.mb[l][c], v = p.vb[l][c];
    p.b[l][c] = adam1(p, p.b[l][c], m, v, s, 1.0f - powf(p.b1, t), 1.0f - powf(p.b2, t), lr);
    p.mb[l][c] = m;
    p.vb[l][c] = v;
  }
}

}  // namespace fused

int fused_tiles_per_wave() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}
template <int FORM>
static void launch_tile(const FusedArgs &a, int grid, cudaStream_t s) {
  using C = fused::Form<FORM>;
  cudaFuncSetAttribute(fused::k_mlp_tile<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::S_END);
  fused::k_mlp_tile<FORM><<<grid, C::THREADS, C::S_END, s>>>(a);
}
void launch_mlp_forward(const FusedArgs &a, cudaStream_t s) {
  const int sms = fused_tiles_per_wave();
  if (a.ntiles <= sms) launch_tile<fused::FORM_ONE>(a, a.ntiles, s);
  else launch_tile<fused::FORM_TWO>(a, a.ntiles < 2 * sms ? a.ntiles : 2 * sms, s);
}
void launch_mlp_train_tile(const FusedArgs &a, cudaStream_t s) { launch_tile<fused::FORM_TRAIN>(a, a.ntiles, s); }
void launch_mlp_dw(const FusedArgs &a, float *part, long long unit_stride, int ks, int rows, cudaStream_t s) {
  const int sm = fused::DW_NS * fused::DW_STAGE;
  cudaFuncSetAttribute(fused::k_mlp_dw, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  fused::k_mlp_dw<<<dim3(ks, 2 * a.nlin), 192, sm, s>>>(a, part, unit_stride, rows);
}
void launch_mlp_reduce(const PackArgs &p, const float *part, long long unit_stride, int ks, const int *step, float lr,
                       int adam, cudaStream_t s) {
  fused::k_mlp_reduce<<<dim3(4 * fused::W / 32, 2 * p.nlin), 256, 0, s>>>(p, part, unit_stride, ks, step, lr, adam);
}
void launch_mlp_bias(const FusedArgs &a, const PackArgs &p, float *cpart, int nb, const int *step, float lr, int adam,
                     float *loss, cudaStream_t s) {
  fused::k_mlp_colsum<<<dim3(nb, a.nlin), 32, 0, s>>>(a, cpart, nb);
  fused::k_mlp_bias<<<p.nlin + 1, 256, 0, s>>>(p, cpart, nb, step, lr, adam, a.lrow, a.B, loss);
}
void launch_mlp_pack(const PackArgs &p, cudaStream_t s) {
  fused::k_mlp_pack<<<dim3(fused::W * fused::W / 256, p.nlin), 256, 0, s>>>(p);
}

}  // namespace ec2d
