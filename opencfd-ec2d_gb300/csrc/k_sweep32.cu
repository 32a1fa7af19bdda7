// k_sweep32.cu -- the LU-SGS operator (du_LU_SGS_2D, sub_LU_SGS.f90:4-108) in
// FP32, for the mixed-precision mode in which the sweeps only precondition:
// the residual stays FP64, Res is rounded to float when the records are built,
// U stays FP64 and receives U += (double)dU in a separate all-cells kernel.
//
// The Gauss-Seidel order is the reference's, one CTA per block, thread j owns
// row j, the next three cells' records are in flight by cp.async.  Two forms
// with the same arithmetic, term by term (dU is the same to the bit):
//   k_push32         a cell, once updated, forms the terms it adds to its two
//                    downstream neighbours: the next cell's stays in the
//                    thread, the next row's moves by shuffle, or from a warp's
//                    last row to the next warp through an inbox whose words are
//                    their own flags (as in k_sweep_push.cu).  Warps run at
//                    their own pace, a few cells apart; no CTA barrier.
//   k_lusgs_sweep32  a cell pulls its neighbours' states through a
//                    double-buffered shared slot, one CTA barrier per plane;
//                    where the inboxes do not fit shared memory.
// What bounds the sweep is the chain of about 20 dependent FP32 operations and
// one reciprocal per cell (some 150 cycles) and what cannot be put beside it: a step
// is about 90 instructions of one warp at four cycles each.  Flat plate, 2 x 96 x 96
// cells, with the record builder and the update: 93 us (152 with the barrier per
// plane, 123 with branches in a step, the inbox read at its end and the records
// converted by conversion instructions, which occupy the FP64 pipe); 24 x 24 cells 35 us.
// Records by bulk copy in windows that lag with the rows, and dU stored in the warps'
// order, measured the same.
// One difference in arithmetic, not in the operator: the flux difference of comput_DFn
// (sub_LU_SGS.f90:117-138), F_n(U + dU) - F_n(U), is evaluated in the
// algebraically identical increment form
//     du = (d(rho u) - u d(rho)) / (rho + d(rho)),  dv likewise,
//     dp = (gamma-1) (dE - (d(rho u) u' + rho u du + d(rho v) v' + rho v dv) / 2),
//     dF_0 = d(rho) un' + rho dun,        dF_1 = d(rho u) un' + rho u dun + dp n1,
//     dF_2 = d(rho v) un' + rho v dun + dp n2,
//     dF_3 = (dE + dp) un' + (E + p) dun, dF_m = dU_m un' + U_m dun (m >= 4),
// with un' = u' n1 + v' n2 and dun = du n1 + dv n2.  In float, F_n(U + dU)
// - F_n(U) would cancel to zero once |dU| < 6e-8 |U| and stall convergence;
// here every term is an increment times an O(1) state, so the rounding error
// stays relative to dU.  The producer of a state computes du, dv, u', v', dp
// (they do not depend on the face normal) and ships them with dU and its base
// state; the consumer forms un', dun with its own face normal, which already
// carries the factor +-0.5 s of the reference (the flux is linear in n).
#include <algorithm>

#include "ec2d_dev.cuh"
#include "ec2d_internal.h"

namespace ec2d {

namespace {

constexpr int TILE = EC2D_TILE;

constexpr int pad4(int n) { return (n + 3) / 4 * 4; }

// record (floats), identical for both passes:
//  A        Res (forward) or the forward dU (backward)
//  B        base state of the cell: rho, rho u, rho v, E + p, U_5.., then u, v
//  CI, CJ   0.5 Lc_nb (+ Lv_nb when viscous) of the upstream neighbours
//  N1I..N2J face normals of face i / j times the signed 0.5 s of the reference
//           (push form: of the terms the cell gives to its downstream
//           neighbours instead of those it takes from the upstream ones)
//  IA, IA5  1/alfa and, for the SA row, 1/(alfa + Lvi + Lvj)
template <int NV>
struct R32 {
  static constexpr int A = 0, B = NV, BU = 2 * NV, BV = 2 * NV + 1, CI = 2 * NV + 2, CJ = CI + 1, N1I = CI + 2,
                       N2I = CI + 3, N1J = CI + 4, N2J = CI + 5, IA = CI + 6, IA5 = CI + 7;
  static constexpr int NF = pad4(CI + 8);
  static constexpr int BYTES = NF * 4;
  static_assert(BYTES % 16 == 0, "records are whole 16-byte units");
};

// shipped state: dU, base (rho, rho u, rho v, E + p, U_5..), u', v', du, dv, dp
template <int NV>
struct S32 {
  static constexpr int D = 0, B = NV, UP = 2 * NV, VP = UP + 1, DU = UP + 2, DV = UP + 3, DP = UP + 4;
  static constexpr int S = pad4(DP + 1);
};

template <int NV, bool PUSH>
__global__ void __launch_bounds__(TILE) k_lusgs_prep32(Lvl L, double alfa1, int force) {
  using RC = R32<NV>;
  int bk, i, j;
  if (!core_ij(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  if (i < 1 || i > b.nx - 1 || j < 1 || j > b.ny - 1) return;
  const CaseDev &c = L.cs[b.cas];
  const long long F = L.F, P = b.P;
  const long long id = fidx(b, i, j);
  const double gm1 = c.gamma - 1.0;
  const double *g = L.geo, *lc = L.lc;
  const bool visc = L.visc != 0;
  const size_t cell = (size_t)b.cell0 + (size_t)(j - 1) * (b.nx - 1) + (i - 1);
  // the two records are assembled in registers and written 16 bytes at a time
  float rf[RC::NF], rb[RC::NF];
#pragma unroll
  for (int k = RC::CI + 8; k < RC::NF; k++) rf[k] = rb[k] = 0.0f;
  double vol = g[G_VOL * F + id];
  double Lv = lc[L_VI * F + id] + lc[L_VJ * F + id];
  double alfa = vol * rcp(lc[L_DT * F + id]) + 1.0 * (lc[L_CI * F + id] + lc[L_CJ * F + id]) + vol * alfa1;
  if (visc) alfa += 2.0 * Lv;
  double ia = rcp(alfa), ia5 = (NV == 5) ? rcp(alfa + Lv) : ia;
  double U[NV];
#pragma unroll
  for (int m = 0; m < NV; m++) U[m] = L.U[m * F + id];
  double r = rcp(U[0]), u = U[1] * r, v = U[2] * r;
  double p = gm1 * (U[3] - 0.5 * (U[1] * u + U[2] * v));
#pragma unroll
  for (int m = 0; m < NV; m++) {
    rf[RC::A + m] = to<float>((force && m < 4) ? L.res[m * F + id] + L.qf[m * F + id] : L.res[m * F + id]);
    rb[RC::A + m] = 0.0f;
  }
  float *rr[2] = {rf, rb};
#pragma unroll
  for (int pass = 0; pass < 2; pass++) {
    float *q = rr[pass];
    q[RC::B + 0] = to<float>(U[0]);
    q[RC::B + 1] = to<float>(U[1]);
    q[RC::B + 2] = to<float>(U[2]);
    q[RC::B + 3] = to<float>(U[3] + p);
#pragma unroll
    for (int m = 4; m < NV; m++) q[RC::B + m] = to<float>(U[m]);
    q[RC::BU] = to<float>(u);
    q[RC::BV] = to<float>(v);
    q[RC::IA] = to<float>(ia);
    q[RC::IA5] = to<float>(ia5);
#pragma unroll
    for (int dir = 0; dir < 2; dir++) {  // 0: i-neighbour, 1: j-neighbour
      const bool fwd = pass == 0;
      const long long step = dir == 0 ? 1 : P;
      // the cell that takes the term, the one that gives it
      const bool up = fwd != PUSH;  // the other cell has the smaller index
      const long long other = up ? id - step : id + step, taker = PUSH ? other : id, nb = PUSH ? id : other;
      const bool has = dir == 0 ? (up ? i > 1 : i < b.nx - 1) : (up ? j > 1 : j < b.ny - 1);
      double cc = 0.0, hh = 0.0, n1 = 0.0, n2 = 0.0;
      if (has) {
        cc = 0.5 * lc[(dir == 0 ? L_CI : L_CJ) * F + nb];
        if (visc) cc += lc[(dir == 0 ? L_VI : L_VJ) * F + nb];
        // forward: +0.5 s of the taking cell's face; backward: -0.5 s of the
        // giving cell's face with the taking cell's normal (sub_LU_SGS.f90:87-88,95-96)
        hh = 0.5 * g[(dir == 0 ? G_SI : G_SJ) * F + (fwd ? taker : nb)];
        if (!fwd) hh = -hh;
        n1 = g[(dir == 0 ? G_NI1 : G_NJ1) * F + taker];
        n2 = g[(dir == 0 ? G_NI2 : G_NJ2) * F + taker];
      }
      q[dir == 0 ? RC::CI : RC::CJ] = to<float>(cc);
      q[dir == 0 ? RC::N1I : RC::N1J] = to<float>(hh * n1);
      q[dir == 0 ? RC::N2I : RC::N2J] = to<float>(hh * n2);
    }
  }
  char *base = reinterpret_cast<char *>(L.rec);
  float4 *wf = reinterpret_cast<float4 *>(base + cell * RC::BYTES);
  float4 *wb = reinterpret_cast<float4 *>(base + ((size_t)L.ncell + cell) * RC::BYTES);
#pragma unroll
  for (int k = 0; k < RC::NF / 4; k++) {
    wf[k] = make_float4(rf[4 * k], rf[4 * k + 1], rf[4 * k + 2], rf[4 * k + 3]);
    wb[k] = make_float4(rb[4 * k], rb[4 * k + 1], rb[4 * k + 2], rb[4 * k + 3]);
  }
}

// the term a cell gives a downstream neighbour: dF_n(its state, scaled normal) +
// cc dU
template <int NV>
__device__ __forceinline__ void dterm(const float *s, float n1, float n2, float cc, float *x) {
  using SL = S32<NV>;
  const float unp = s[SL::UP] * n1 + s[SL::VP] * n2;
  const float dun = s[SL::DU] * n1 + s[SL::DV] * n2;
  const float dp = s[SL::DP];
  x[0] = s[SL::D + 0] * unp + s[SL::B + 0] * dun + cc * s[SL::D + 0];
  x[1] = s[SL::D + 1] * unp + s[SL::B + 1] * dun + dp * n1 + cc * s[SL::D + 1];
  x[2] = s[SL::D + 2] * unp + s[SL::B + 2] * dun + dp * n2 + cc * s[SL::D + 2];
  x[3] = (s[SL::D + 3] + dp) * unp + s[SL::B + 3] * dun + cc * s[SL::D + 3];
#pragma unroll
  for (int m = 4; m < NV; m++) x[m] = s[SL::D + m] * unp + s[SL::B + m] * dun + cc * s[SL::D + m];
}
// the state of a cell that its terms need, from dU (in st) and the record
template <int NV>
__device__ __forceinline__ void shipped_state(float *st, const float *cur, float gm1) {
  using SL = S32<NV>;
  using RC = R32<NV>;
#pragma unroll
  for (int m = 0; m < NV; m++) st[SL::B + m] = cur[RC::B + m];
  const float rho = cur[RC::B + 0], m1 = cur[RC::B + 1], m2 = cur[RC::B + 2];
  const float u = cur[RC::BU], v = cur[RC::BV];
  const float dr = st[SL::D + 0], dm1 = st[SL::D + 1], dm2 = st[SL::D + 2], dE = st[SL::D + 3];
  float rr;  // 1 / (rho + d rho): the approximate reciprocal (an FP32 preconditioner)
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rr) : "f"(rho + dr));
  const float du = (dm1 - u * dr) * rr, dv = (dm2 - v * dr) * rr;
  const float up = u + du, vp = v + dv;
  st[SL::UP] = up;
  st[SL::VP] = vp;
  st[SL::DU] = du;
  st[SL::DV] = dv;
  st[SL::DP] = gm1 * (dE - 0.5f * (dm1 * up + m1 * du + dm2 * vp + m2 * dv));
}

// acc += dF_n(shipped state, scaled normal) + cc dU_nb
template <int NV>
__device__ __forceinline__ void dflux(const float *s, float n1, float n2, float cc, float *acc) {
  using SL = S32<NV>;
  float unp = s[SL::UP] * n1 + s[SL::VP] * n2;
  float dun = s[SL::DU] * n1 + s[SL::DV] * n2;
  float dp = s[SL::DP];
  acc[0] += s[SL::D + 0] * unp + s[SL::B + 0] * dun + cc * s[SL::D + 0];
  acc[1] += s[SL::D + 1] * unp + s[SL::B + 1] * dun + dp * n1 + cc * s[SL::D + 1];
  acc[2] += s[SL::D + 2] * unp + s[SL::B + 2] * dun + dp * n2 + cc * s[SL::D + 2];
  acc[3] += (s[SL::D + 3] + dp) * unp + s[SL::B + 3] * dun + cc * s[SL::D + 3];
#pragma unroll
  for (int m = 4; m < NV; m++) acc[m] += s[SL::D + m] * unp + s[SL::B + m] * dun + cc * s[SL::D + m];
}

__device__ __forceinline__ void cp16(void *dst, const void *src) {
  unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_ring() { asm volatile("cp.async.wait_group 3;" ::: "memory"); }
// record buffers per thread: the record of the cell three planes ahead is in
// flight while the current one is computed (an FP32 plane is short next to
// the L2 latency)
constexpr int RING32 = 4;
__device__ __forceinline__ void cp_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <int NV>
__device__ __forceinline__ void fetch32(char *dst, const char *src) {
#pragma unroll
  for (int k = 0; k < R32<NV>::BYTES; k += 16) cp16(dst + k, src + k);
}

// One pass of a row, forward (FWD) or backward.
template <int NV, bool fwd>
__device__ __forceinline__ void sweep32_pass(const Lvl &L, float *shf, char *rec, const char *recF, const char *recB,
                                             char *recBw, float *st, const BlkDev &bd, int R, int rl, int j,
                                             bool row_ok, float gm1) {
  using SL = S32<NV>;
  using RC = R32<NV>;
  constexpr int S = SL::S;
  const int nx = bd.nx, ny = bd.ny, rows = ny - 1, ni = nx - 1;
  const char *rsrc = fwd ? recF : recB;
  // record of the k-th visited cell: forward i = 1 + k, backward i = ni - k
  auto src = [&](int k) { return rsrc + (size_t)(fwd ? k : ni - 1 - k) * RC::BYTES; };
  for (int q = 0; q < RING32 - 1; q++) {
    if (row_ok && q < ni) fetch32<NV>(rec + q * RC::BYTES, src(q));
    cp_commit();
  }
  int k = 0;
  for (int pp = 2; pp <= nx + ny - 2; pp++) {
    const int p = fwd ? pp : nx + ny - pp;
    const int i = p - j;
    const int buf = p & 1;
    if (row_ok && i >= 1 && i <= ni) {
      const float4 *cur4 = reinterpret_cast<const float4 *>(rec + (k % RING32) * RC::BYTES);
      if (k + RING32 - 1 < ni) fetch32<NV>(rec + ((k + RING32 - 1) % RING32) * RC::BYTES, src(k + RING32 - 1));
      cp_commit();
      cp_wait_ring();
      // the whole record into registers with 16-byte shared loads at once
      float cur[RC::NF];
#pragma unroll
      for (int q = 0; q < RC::NF / 4; q++) {
        const float4 v = cur4[q];
        cur[4 * q] = v.x; cur[4 * q + 1] = v.y; cur[4 * q + 2] = v.z; cur[4 * q + 3] = v.w;
      }
      float acc[NV];
#pragma unroll
      for (int m = 0; m < NV; m++) acc[m] = fwd ? cur[RC::A + m] : 0.0f;
      if (fwd ? (i > 1) : (i < ni)) dflux<NV>(st, cur[RC::N1I], cur[RC::N2I], cur[RC::CI], acc);
      if (fwd ? (j > 1) : (j < rows)) {
        const float4 *s4 = reinterpret_cast<const float4 *>(shf + ((size_t)(buf ^ 1) * (R + 2) + (fwd ? rl : rl + 2)) * S);
        float sn[S];
#pragma unroll
        for (int m = 0; m < S / 4; m++) {
          float4 v = s4[m];
          sn[4 * m] = v.x; sn[4 * m + 1] = v.y; sn[4 * m + 2] = v.z; sn[4 * m + 3] = v.w;
        }
        dflux<NV>(sn, cur[RC::N1J], cur[RC::N2J], cur[RC::CJ], acc);
      }
      const float ia = cur[RC::IA], ia5 = cur[RC::IA5];
#pragma unroll
      for (int m = 0; m < NV; m++) {
        float inv = (NV == 5 && m == 4) ? ia5 : ia;
        st[SL::D + m] = fwd ? acc[m] * inv : cur[RC::A + m] + acc[m] * inv;
      }
      shipped_state<NV>(st, cur, gm1);  // for the two downstream neighbours
      float4 *own = reinterpret_cast<float4 *>(shf + ((size_t)buf * (R + 2) + rl + 1) * S);
#pragma unroll
      for (int m = 0; m < S / 4; m++) own[m] = make_float4(st[4 * m], st[4 * m + 1], st[4 * m + 2], st[4 * m + 3]);
      // forward: the forward dU becomes the A field of this cell's backward
      // record; backward: the final dU replaces it there, and k_apply32
      // widens it to FP64 afterwards (FP64 instructions hold a warp for
      // about 64 cycles each, so they stay off the wavefront)
      float *w = reinterpret_cast<float *>(recBw + (size_t)(i - 1) * RC::BYTES);
      static_assert(RC::A == 0 && SL::D == 0, "A and D open the record and the slot");
#pragma unroll
      for (int m = 0; m + 3 < NV; m += 4)
        reinterpret_cast<float4 *>(w)[m / 4] = make_float4(st[m], st[m + 1], st[m + 2], st[m + 3]);
#pragma unroll
      for (int m = NV / 4 * 4; m < NV; m++) w[m] = st[m];
      k++;
    }
    __syncthreads();
  }
  cp_wait0();
}

template <int NV>
__global__ void __launch_bounds__(1024) k_lusgs_sweep32(Lvl L) {
  using SL = S32<NV>;
  using RC = R32<NV>;
  constexpr int S = SL::S;
  extern __shared__ __align__(16) float shf[];  // [2][rows+2][S] slots, then [blockDim][RING32] records
  const BlkDev bd = L.blk[blockIdx.x];
  const int rows = bd.ny - 1, ni = bd.nx - 1;
  const int rl = threadIdx.x;
  const int j = rl + 1;
  const int R = blockDim.x;
  const bool row_ok = j <= rows;
  const float gm1 = (float)(L.cs[bd.cas].gamma - 1.0);
  char *rec = reinterpret_cast<char *>(shf + (size_t)2 * (R + 2) * S) + (size_t)threadIdx.x * RING32 * RC::BYTES;
  const char *recF = reinterpret_cast<const char *>(L.rec) + ((size_t)bd.cell0 + (size_t)(j - 1) * ni) * RC::BYTES;
  const char *recB = recF + (size_t)L.ncell * RC::BYTES;
  char *recBw = reinterpret_cast<char *>(L.rec) + ((size_t)L.ncell + bd.cell0 + (size_t)(j - 1) * ni) * RC::BYTES;
  float st[S];
#pragma unroll
  for (int m = 0; m < S; m++) st[m] = 0.0f;
  sweep32_pass<NV, true>(L, shf, rec, recF, recB, recBw, st, bd, R, rl, j, row_ok, gm1);
  sweep32_pass<NV, false>(L, shf, rec, recF, recB, recBw, st, bd, R, rl, j, row_ok, gm1);
}

// ---- push form ----------------------------------------------------------------
constexpr unsigned FULL = 0xffffffffu;
constexpr int WAIT32 = 1 << 18;  // polls of an inbox before the wait gives up
// an inbox word nothing has been written to: a NaN no arithmetic produces
constexpr unsigned EMPTY32 = 0x7fc9e37bu;
// records per thread: those of the next PRING32 - 2 cells are in flight (an FP32
// cell takes a third of the L2 latency); padded so that the 16-byte reads of
// eight neighbouring threads meet eight different groups of banks
constexpr int PRING32 = 8;
template <int NV>
constexpr int ring_bytes() { return PRING32 * R32<NV>::BYTES + 16; }
static_assert(ring_bytes<4>() % 32 == 16 && ring_bytes<5>() % 32 == 16 && ring_bytes<6>() % 32 == 16, "odd multiples of 16 bytes");
__device__ __forceinline__ void cp_wait_push() { asm volatile("cp.async.wait_group %0;" ::"n"(PRING32 - 3) : "memory"); }
__device__ __forceinline__ float4 box_read4(unsigned a) {
  float4 v;
  asm volatile("ld.volatile.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void box_write4_if(bool p, unsigned a, float x, float y, float z, float w) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p st.volatile.shared.v4.f32 [%0], {%1, %2, %3, %4};\n\t}" ::"r"(a),
               "f"(x), "f"(y), "f"(z), "f"(w), "r"((int)p)
               : "memory");
}
__device__ __forceinline__ void stg4_if(bool p, float *a, float x, float y, float z, float w) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p st.global.v4.f32 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(a), "f"(x),
               "f"(y), "f"(z), "f"(w), "r"((int)p)
               : "memory");
}
__device__ __forceinline__ void stg_if(bool p, float *a, float x) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}" ::"l"(a), "f"(x), "r"((int)p)
               : "memory");
}
__device__ __forceinline__ void cp16_if(bool p, unsigned d, const char *src) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p cp.async.cg.shared.global [%0], [%1], 16;\n\t}" ::"r"(d), "l"(src),
               "r"((int)p)
               : "memory");
}
constexpr int PUSH32_THREADS = 352;  // the rings of as many rows fill the shared memory
template <int NV>
constexpr int box_words() { return NV == 4 ? 4 : 8; }

template <int NV, bool FWD>
__device__ __forceinline__ void push32_pass(const Lvl &L, const BlkDev &bd, int bk, char *rec, unsigned box, unsigned out,
                                            const char *src_row, char *dst_row, int j0, float gm1) {
  using SL = S32<NV>;
  using RC = R32<NV>;
  constexpr int SB = box_words<NV>();
  const int lane = threadIdx.x & 31, ni = bd.nx - 1, rows = bd.ny - 1;
  const int last = min(31, rows - j0);  // the warp's last row
  const bool row_ok = lane <= last;
  const int lag = FWD ? lane : last - lane;
  // the inbox serves the warp's first row in the order of the pass; the last one
  // feeds the next warp
  const bool has_box = FWD ? j0 > 1 : j0 + 32 <= rows, has_out = FWD ? j0 + 32 <= rows : j0 > 1;
  const bool first = lane == (FWD ? 0 : last), sends = has_out && !L.silent_band_edge && lane == (FWD ? last : 0);
  const int from = FWD ? (lane + 31) & 31 : (lane + 1) & 31;
  auto src = [&](int k) { return src_row + (ptrdiff_t)(FWD ? k : ni - 1 - k) * RC::BYTES; };
  const unsigned ring = (unsigned)__cvta_generic_to_shared(rec);
  // (k below PRING32 - 2: requested before the first step)
  auto fetch = [&](int k, int from_k = PRING32 - 2) {
    const bool go = row_ok && k >= from_k && k < ni;
    const unsigned d = ring + (unsigned)(k & (PRING32 - 1)) * RC::BYTES;
    const char *p = src(k);
#pragma unroll
    for (int b = 0; b < RC::BYTES; b += 16) cp16_if(go, d + b, p + b);
    cp_commit();
  };
  auto read = [&](float (&c)[RC::NF], int k) {
    const float4 *p = reinterpret_cast<const float4 *>(rec + (k & (PRING32 - 1)) * RC::BYTES);
#pragma unroll
    for (int q = 0; q < RC::NF / 4; q++) {
      const float4 v = p[q];
      c[4 * q] = v.x; c[4 * q + 1] = v.y; c[4 * q + 2] = v.z; c[4 * q + 3] = v.w;
    }
  };
  int gave_up = -1;
  // the inbox entry of step t: read in the middle of the step before (peek), and
  // again at its end while a word of it is empty (poll)
  float in[NV];
#pragma unroll
  for (int m = 0; m < NV; m++) in[m] = 0.0f;
  auto peek = [&](int t) {
    if (!has_box) return;
    const unsigned p = box + 4u * SB * (unsigned)min(t, ni - 1);
    const float4 v = box_read4(p);
    in[0] = v.x; in[1] = v.y; in[2] = v.z; in[3] = v.w;
    if (NV > 4) {
      const float4 w = box_read4(p + 16u);
      in[4 < NV ? 4 : 0] = w.x;
      if (NV > 5) in[NV - 1] = w.y;
    }
  };
  auto poll = [&](int t) {
    if (!has_box || t >= ni || gave_up >= 0) return;
    for (int n = 0;; n++) {
      bool empty = false;
#pragma unroll
      for (int m = 0; m < NV; m++) empty |= __float_as_uint(in[m]) == EMPTY32;
      if (!empty) break;  // (one word for the whole warp: every lane finds the same)
      if (n == WAIT32) { gave_up = t; break; }
      peek(t);
    }
  };
  float st[SL::S], own[NV], down[NV];  // the cell's state; the terms for the next cell and the next row
#pragma unroll
  for (int m = 0; m < SL::S; m++) st[m] = 0.0f;
#pragma unroll
  for (int m = 0; m < NV; m++) own[m] = down[m] = 0.0f;
  float c0[RC::NF], c1[RC::NF];
  // records of the row's first visits; visit k + PRING32 - 2 is requested in visit
  // k, one group a step, so that the record of visit k + 1 has landed at the
  // end of visit k
  for (int k = 0; k < PRING32 - 2; k++) fetch(k, 0);
  cp_wait_push();
  read(c0, 0);
  peek(0);
  poll(0);
  // no branch but the poll: what a lane may not keep or store is selected or
  // predicated, so that the loads of the next step are issued among the arithmetic
  auto step = [&](int t, float (&cur)[RC::NF], float (&next)[RC::NF]) {
    const int k = t - lag;
    const bool act = row_ok && (unsigned)k < (unsigned)ni;
    float nb[NV];
#pragma unroll
    for (int m = 0; m < NV; m++) nb[m] = __shfl_sync(FULL, down[m], from);
#pragma unroll
    for (int m = 0; m < NV; m++) nb[m] = first ? in[m] : nb[m];
    fetch(k + PRING32 - 2);
    cp_wait_push();
    read(next, max(k + 1, 0));
    peek(t + 1);
    const float ia = cur[RC::IA], ia5 = cur[RC::IA5];
    float dn[NV];
#pragma unroll
    for (int m = 0; m < NV; m++) {
      float acc = FWD ? cur[RC::A + m] : 0.0f;
      acc += own[m];
      acc += nb[m];
      const float inv = (NV == 5 && m == 4) ? ia5 : ia;
      dn[m] = FWD ? acc * inv : cur[RC::A + m] + acc * inv;
    }
    float x[NV], y[NV];
#pragma unroll
    for (int m = 0; m < NV; m++) st[SL::D + m] = dn[m];
    shipped_state<NV>(st, cur, gm1);
    dterm<NV>(st, cur[RC::N1J], cur[RC::N2J], cur[RC::CJ], y);
    dterm<NV>(st, cur[RC::N1I], cur[RC::N2I], cur[RC::CI], x);
#pragma unroll
    for (int m = 0; m < NV; m++) {
      down[m] = act ? y[m] : down[m];
      own[m] = act ? x[m] : own[m];
    }
    const bool send = sends && act;
    const unsigned o = out + 4u * SB * (unsigned)k;
    box_write4_if(send, o, down[0], down[1], down[2], down[3]);
    if (NV > 4) box_write4_if(send, o + 16u, down[4 < NV ? 4 : 0], down[NV - 1], 0.0f, 0.0f);
    // forward: the A field of the backward record; backward: the final dU
    // replaces it there (k_apply32 widens it afterwards)
    float *w = reinterpret_cast<float *>(dst_row + (ptrdiff_t)(FWD ? k : ni - 1 - k) * RC::BYTES);
    stg4_if(act, w, dn[0], dn[1], dn[2], dn[3]);
#pragma unroll
    for (int m = 4; m < NV; m++) stg_if(act, w + m, dn[m]);
    poll(t + 1);
  };
  const int steps = ni + last;
  for (int t = 0; t < steps; t += 2) {
    step(t, c0, c1);
    step(t + 1, c1, c0);
  }
  cp_wait0();
  if (gave_up >= 0 && lane == 0)
    set_status(L.status + 4 * bd.cas, 4, bk, FWD ? gave_up + 1 : ni - gave_up, j0);
}

template <int NV>
__global__ void __launch_bounds__(PUSH32_THREADS, 1) k_push32(Lvl L) {
  using RC = R32<NV>;
  extern __shared__ __align__(16) char sh[];  // rings [thread], inboxes [warp][column][SB]
  const BlkDev bd = L.blk[blockIdx.x];
  const int rows = bd.ny - 1, ni = bd.nx - 1, w = threadIdx.x >> 5, j0 = 32 * w + 1, j = threadIdx.x + 1;
  const float gm1 = (float)(L.cs[bd.cas].gamma - 1.0);
  char *rec = sh + (size_t)threadIdx.x * ring_bytes<NV>();
  float *boxes = reinterpret_cast<float *>(sh + (size_t)blockDim.x * ring_bytes<NV>());
  const size_t words = (size_t)ni * box_words<NV>();
  float *box = boxes + w * words;
  const unsigned mine = (unsigned)__cvta_generic_to_shared(box), step = 4u * (unsigned)words;
  auto clear = [&] {
    for (size_t t = threadIdx.x & 31; t < words; t += 32) box[t] = __uint_as_float(EMPTY32);
  };
  const int jr = min(j, rows);  // record pointers of idle rows stay in the array
  char *recF = reinterpret_cast<char *>(L.rec) + ((size_t)bd.cell0 + (size_t)(jr - 1) * ni) * RC::BYTES;
  char *recB = recF + (size_t)L.ncell * RC::BYTES;
  clear();
  __syncthreads();  // every inbox empty before any warp writes into one
  if (j0 <= rows) {
    push32_pass<NV, true>(L, bd, blockIdx.x, rec, mine, mine + step, recF, recB, j0, gm1);
    __syncwarp();
    clear();
  }
  __syncthreads();  // and again before the backward pass (the others wait for the last warp anyway)
  if (j0 <= rows) push32_pass<NV, false>(L, bd, blockIdx.x, rec, mine, mine - step, recB, recB, j0, gm1);
}

// dU (FP32, in the backward records) -> U += dU in FP64, or -> L.du
// (NS_Time_advance_LU_SGS, sub_NS_singlegrid.f90:203-211)
template <int NV>
__global__ void __launch_bounds__(TILE) k_apply32(Lvl L, int update) {
  using RC = R32<NV>;
  int2 t = L.tiles[blockIdx.x];
  const BlkDev &b = L.blk[t.x];
  int W = b.nx + 3, lin = t.y + threadIdx.x;
  if (lin >= W * (b.ny + 3)) return;
  int i = lin % W - 1, j = lin / W - 1;
  if (i < 1 || i > b.nx - 1 || j < 1 || j > b.ny - 1) return;
  const long long F = L.F, id = fidx(b, i, j);
  const size_t cell = (size_t)b.cell0 + (size_t)(j - 1) * (b.nx - 1) + (i - 1);
  const float *rb = reinterpret_cast<const float *>(reinterpret_cast<const char *>(L.rec) +
                                                    ((size_t)L.ncell + cell) * RC::BYTES);
  // an updating sweep keeps no DU, as the FP64 sweep (the reference reads DU
  // only inside du_LU_SGS_2D and the update after it)
#pragma unroll
  for (int m = 0; m < NV; m++) {
    const double d = to_double(rb[RC::A + m]);
    if (update) L.U[m * F + id] += d;
    else L.du[m * F + id] = d;
  }
}

template <int NV>
size_t smem32(int rows) {
  int th = ((rows + 31) / 32) * 32;
  return (size_t)2 * (th + 2) * S32<NV>::S * sizeof(float) + (size_t)th * RING32 * R32<NV>::BYTES;
}

// shared memory of the push form; it serves blocks whose inboxes fit
template <int NV>
size_t push32_smem(int rows, int cols) {
  const int th = ((rows + 31) / 32) * 32;
  return (size_t)th * ring_bytes<NV>() + (size_t)(th / 32) * cols * box_words<NV>() * sizeof(float);
}

template <int NV>
void sweep32_nv(const Lvl &L, double alfa1, int mode, int max_rows, int max_cols, cudaStream_t s) {
  const int update = mode & LUSGS_UPDATE, force = mode & LUSGS_FORCE;
  const int th = ((max_rows + 31) / 32) * 32;
  const size_t push = push32_smem<NV>(max_rows, max_cols), pull = smem32<NV>(max_rows);
  if (th <= PUSH32_THREADS && push <= 227 * 1024) {
    k_lusgs_prep32<NV, true><<<L.nctiles, TILE, 0, s>>>(L, alfa1, force);
    if (push > 48 * 1024) cudaFuncSetAttribute(k_push32<NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)push);
    k_push32<NV><<<L.nblk, th, push, s>>>(L);
  } else {
    k_lusgs_prep32<NV, false><<<L.nctiles, TILE, 0, s>>>(L, alfa1, force);
    if (pull > 48 * 1024)
      cudaFuncSetAttribute(k_lusgs_sweep32<NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pull);
    k_lusgs_sweep32<NV><<<L.nblk, th, pull, s>>>(L);
  }
  k_apply32<NV><<<L.ntiles, TILE, 0, s>>>(L, update);
}

}  // namespace

size_t lusgs32_smem(int nv, int rows) {
  return nv == 4 ? smem32<4>(rows) : nv == 5 ? smem32<5>(rows) : smem32<6>(rows);
}

void launch_lusgs_fast32(const Lvl &L, double alfa1, int mode, int max_rows, int max_cols, cudaStream_t s) {
  if (L.nvar == 4) sweep32_nv<4>(L, alfa1, mode, max_rows, max_cols, s);
  else if (L.nvar == 5) sweep32_nv<5>(L, alfa1, mode, max_rows, max_cols, s);
  else sweep32_nv<6>(L, alfa1, mode, max_rows, max_cols, s);
}

}  // namespace ec2d
