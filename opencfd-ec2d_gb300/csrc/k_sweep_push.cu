// k_sweep_push.cu -- the LU-SGS wavefront (du_LU_SGS_2D, sub_LU_SGS.f90:4-108)
// with eight lanes per row, in push form: a cell, once updated, forms the
// terms it adds to its two downstream neighbours and hands over those.
//
// The Gauss-Seidel order is the reference's, as in k_sweep.cu.  What bounds
// the sweep is the chain between two cells of a row: a warp's FP64
// instruction takes 64 cycles on this part whether or not the next one
// depends on it, and a value that passes from the FP64 pipe through another
// one (a shuffle, a select) and back costs about 50 more than that pipe's own
// latency (measured).  So the FP64 instructions and the crossings per cell
// set the time, and everything else has to fit in their shadow.  What keeps
// them few (4 variables: 6 FP64 instructions and 3 crossings; 15 and 5 when a
// cell pulled its neighbours' states):
//  * the records hold the face normals, dissipation coefficients and constant
//    terms already multiplied by 1/alfa of the cell that receives the term,
//    and the constant term with U added, so the new state is the sum of the
//    own row's term and the neighbouring row's: one addition;
//  * in a half row of four lanes, one instruction with per-lane operands forms
//    m = s1 a + s2 b with (a, b) the scaled normal (lanes 0, 2), minus the
//    momenta themselves (lane 1) or (gamma - 1) / 2 times the normal (lane 3),
//    and then z = m / rho + k: w = u_n + cc, p' = 2 E - |rho u|^2 / rho, u_n
//    and (gamma - 1) u_n / 2.  Two exchanges give every lane w and p' =
//    2 p / (gamma - 1), and its term of variable q is s_q w + p' g_q with g =
//    (0, n1, n2, u_n) (gamma - 1) / 2: (rho, rho u, rho v, E) w plus the
//    pressure terms of F_n;
//  * 1/rho is formed on the integer and FP32 pipes while the FP64 pipe forms m
//    (recip).
// The first half row (lanes 0-3) serves the next cell of the own row: its
// accumulator starts from that cell's constant term and stays in the lane.
// The second half serves the same column of the next row: its four sums move
// to that row's first half by one shuffle, or, at the edge of a warp, as four
// 8-byte words to the next warp's inbox.  A warp holds four rows and runs at
// its own pace: no CTA barrier, no cluster barrier per plane.  The inbox has
// a word per column and variable that starts as a fixed NaN pattern (EMPTY);
// the word is its own flag, so the receiver polls the words it needs and no
// fence or second location is involved.  Every wait is bounded (PWAIT polls,
// some ten milliseconds); one that gives up records status 4 for the case.
// Loads and stores share a queue with the shuffles, so records come by bulk
// copies of 16 cells (loads into registers three cells ahead cost 150 cycles
// per cell), and what has to be stored goes out behind the shuffles.
//
// Measured (GB300, 2,070 MHz, events, with the launch; the pull form before it in
// brackets): 2 x 96 x 96 cells 174 us (339), 940 cycles per plane (1,840), 256 x 64 one
// block 266 us (564), 64 x 16 72 us (147); 4 x 128 x 128 with the SA row 348 us
// (622), with the SST rows 337 us (749).  Of a plane 6 x 64 cycles are FP64 and 3 x 75
// crossings; the reciprocal's chain is as long as the two instructions of m, and a row of
// warps adds half a cell per warp at its start.  With two FP64 Newton instructions for
// the reciprocal 2 x 96 x 96 took 200 us.  Bands of 8 to 16 rows per CTA measure
// the same.
#include <algorithm>

#include "ec2d_dev.cuh"
#include "ec2d_internal.h"

namespace ec2d {

constexpr int TILE = EC2D_TILE;

// The records, arrays of one entry per cell (block after block, i fastest), in
// doubles.  Per pass two half records, own row's face and neighbouring row's
// face, of the coefficients of the term the cell RECEIVES through that face,
// all scaled by 1/alfa of the cell:
//   N1, N2   +-0.5 s n of the face        G1, G2  (gamma - 1) / 2 times these
//   C        0.5 Lc + Lv of the upstream neighbour
//   A..A+3   constant terms: own half, forward: U + (Res + K)/alfa; backward:
//            the forward sweep's result (written by it); other half, forward:
//            0; backward: K of the downstream neighbours
//   Z        0
// K = -sum over the upstream neighbours of F_n(U_nb, s) + cc U_nb (mean flow)
// or F_n(U_nb, s) (turbulence variables).  A missing neighbour's coefficients
// are zero.  Without the update of U the constant terms hold no U, and an
// array of U follows.  Turbulence variables t (NV = 5: nu~; 6: k, omega), per
// pass:
//   AT  (Res + K)/alfa, backward: K/alfa   UT  U
//   DT  backward: the forward sweep's dU   RT  alfa / (alfa + Lv) of the SA row
constexpr int HREC = 10, TREC = 8, UREC = 4;
enum { H_N1 = 0, H_N2 = 1, H_G1 = 2, H_G2 = 3, H_C = 4, H_A = 5, H_Z = 9 };
enum { T_AT = 0, T_UT = 2, T_DT = 4, T_RT = 6 };
__host__ __device__ __forceinline__ double *half_rec(double *rec, size_t ncell, int pass, int half) {
  return rec + (size_t)(2 * pass + half) * ncell * HREC;
}
__host__ __device__ __forceinline__ double *turb_rec(double *rec, size_t ncell, int pass) {
  return rec + 4 * ncell * HREC + (size_t)pass * ncell * TREC;
}
__host__ __device__ __forceinline__ double *u_rec(double *rec, size_t ncell, int nv) {
  return rec + 4 * ncell * HREC + (nv > 4 ? 2 * ncell * TREC : 0);
}
// doubles per cell and pass that the record array must hold
int push_record(int nv) { return (4 * HREC + (nv > 4 ? 2 * TREC : 0) + UREC + 1) / 2; }

template <int NV>
__device__ __forceinline__ void face_term(const double *U, double n1, double n2, double cc, double gm1, double *K) {
  const double r = recip(U[0]);
  const double un = (U[1] * n1 + U[2] * n2) * r;
  const double p = gm1 * fma(-half(fma(U[1], U[1], U[2] * U[2])), r, U[3]);
  const double w = un + cc;
  K[0] = fma(-U[0], w, K[0]);
  K[1] = fma(-U[1], w, fma(-p, n1, K[1]));
  K[2] = fma(-U[2], w, fma(-p, n2, K[2]));
  K[3] = fma(-U[3], w, fma(-p, un, K[3]));
#pragma unroll
  for (int m = 4; m < NV; m++) K[m] = fma(-U[m], un, K[m]);
}

// the records of both passes, all cells at once (force: Res + QF in place of
// Res, see k_lusgs_prep).  Bound by FP64 issue on large levels (65 k cells 29 us) and by one
// cell's chain on small ones: 100 instructions per cell at NV = 4 (ncu), with reciprocals
// and halves off the FP64 pipe and every term folded into an FMA.
template <int NV, bool update>
__global__ void __launch_bounds__(TILE) k_push_prep(Lvl L, double alfa1, int force) {
  int bk, i, j;
  if (!core_ij(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  if (i < 1 || i > b.nx - 1 || j < 1 || j > b.ny - 1) return;
  const CaseDev &c = L.cs[b.cas];
  const long long F = L.F, P = b.P;
  const long long id = fidx(b, i, j);
  const double gm1 = c.gm1, hg = half(gm1);
  const double *g = L.geo, *lc = L.lc;
  const bool visc = L.visc != 0;
  const size_t cell = (size_t)b.cell0 + (size_t)(j - 1) * (b.nx - 1) + (i - 1);
  const double vol = g[G_VOL * F + id];
  const double Lv = lc[L_VI * F + id] + lc[L_VJ * F + id];
  double alfa = fma(vol, recip(lc[L_DT * F + id]), fma(vol, alfa1, lc[L_CI * F + id] + lc[L_CJ * F + id]));
  if (visc) alfa += pow2<1>(Lv);
  const double ia = recip(alfa);
  const double ni1 = g[G_NI1 * F + id], ni2 = g[G_NI2 * F + id], nj1 = g[G_NJ1 * F + id], nj2 = g[G_NJ2 * F + id];
  double u[NV], res[NV];
#pragma unroll
  for (int m = 0; m < NV; m++) {
    u[m] = L.U[m * F + id];
    res[m] = L.res[m * F + id];
    if (force && m < 4) res[m] = res[m] + L.qf[m * F + id];
  }
#pragma unroll
  for (int pass = 0; pass < 2; pass++) {
    const bool fwd = pass == 0;
    double r[2][HREC];
    double K[NV];
#pragma unroll
    for (int m = 0; m < NV; m++) K[m] = 0.0;
#pragma unroll
    for (int dir = 0; dir < 2; dir++) {  // 0: i-neighbour, 1: j-neighbour
      const long long step = dir == 0 ? 1 : P;
      const long long nb = fwd ? id - step : id + step;
      const bool has = dir == 0 ? (fwd ? i > 1 : i < b.nx - 1) : (fwd ? j > 1 : j < b.ny - 1);
      double cc = 0.0, s1 = 0.0, s2 = 0.0;
      if (has) {
        double Un[NV];
#pragma unroll
        for (int m = 0; m < NV; m++) Un[m] = L.U[m * F + nb];
        cc = half(lc[(dir == 0 ? L_CI : L_CJ) * F + nb]);
        if (visc) cc += lc[(dir == 0 ? L_VI : L_VJ) * F + nb];
        cc *= ia;
        // forward: +0.5 s of this cell's face; backward: -0.5 s of the
        // neighbour's face with this cell's normal (the reference pairs the
        // normal of face i with the length of face i+1, sub_LU_SGS.f90:87-88,95-96)
        const double h2 = half(g[(dir == 0 ? G_SI : G_SJ) * F + (fwd ? id : nb)]), hh = (fwd ? h2 : -h2) * ia;
        s1 = hh * (dir == 0 ? ni1 : nj1);
        s2 = hh * (dir == 0 ? ni2 : nj2);
        face_term<NV>(Un, s1, s2, cc, gm1, K);
      }
      double *h = r[dir];
      h[H_N1] = s1; h[H_N2] = s2;
      h[H_G1] = hg * s1; h[H_G2] = hg * s2;
      h[H_C] = cc;
      h[H_Z] = 0.0;
    }
#pragma unroll
    for (int m = 0; m < 4; m++) {
      r[0][H_A + m] = fwd ? fma(res[m], ia, K[m]) + (update ? u[m] : 0.0) : 0.0;
      r[1][H_A + m] = fwd ? 0.0 : K[m];
    }
#pragma unroll
    for (int dir = 0; dir < 2; dir++) {
      double2 *w = reinterpret_cast<double2 *>(half_rec(L.rec, L.ncell, pass, dir) + cell * HREC);
#pragma unroll
      for (int q = 0; q < HREC / 2; q++) w[q] = make_double2(r[dir][2 * q], r[dir][2 * q + 1]);
    }
    if (NV > 4) {
      double2 *w = reinterpret_cast<double2 *>(turb_rec(L.rec, L.ncell, pass) + cell * TREC);
      constexpr int m5 = NV - 1;  // the second variable's index (the first again for NV = 5)
      auto at = [&](int m) { return fwd ? fma(res[m], ia, K[m]) : K[m]; };
      w[T_AT / 2] = make_double2(at(4 < NV ? 4 : 0), at(m5));
      w[T_UT / 2] = make_double2(u[4 < NV ? 4 : 0], u[m5]);
      w[T_DT / 2] = make_double2(0.0, 0.0);
      w[T_RT / 2] = make_double2(NV == 5 ? alfa * recip(alfa + Lv) : 0.0, 0.0);
    }
  }
  if (!update) {
    double2 *w = reinterpret_cast<double2 *>(u_rec(L.rec, L.ncell, NV) + cell * UREC);
    w[0] = make_double2(u[0], u[1]);
    w[1] = make_double2(u[2], u[3]);
  }
}

constexpr unsigned FULL = 0xffffffffu;
constexpr int PROWS = 4;            // rows per warp
constexpr int PWARPS = 8;           // most warps per CTA
constexpr int PWAIT = 1 << 18;      // polls of an inbox before the wait gives up
// an inbox word nothing has been written to: a quiet NaN with a payload that
// no arithmetic produces (the hardware's NaN is 0x7fffffffffffffff)
constexpr unsigned long long EMPTY = 0x7ff8ec2d0e3b7a19ull;
__device__ __forceinline__ unsigned hi_of(unsigned long long v) { return (unsigned)(v >> 32); }

template <int NV>
constexpr int inbox_words() { return NV == 4 ? 4 : NV; }

__device__ __forceinline__ unsigned push_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void push_cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned push_remote(unsigned local, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ unsigned long long inbox_read(unsigned a) {
  unsigned long long v;
  asm volatile("ld.relaxed.cluster.shared::cta.b64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}
// 2 x on the integer pipe (of a normal number below 2^1022; infinities and NaNs
// are left as they are)
__device__ __forceinline__ double twice(double x) {
  const int h = __double2hiint(x);
  return __hiloint2double((h & 0x7ff00000) < 0x7fe00000 ? h + 0x00100000 : h, __double2loint(x));
}

// Records reach a warp through shared memory: a ring of two chunks of PCH
// cells per stream (each of its four rows' own half, the half of the row each
// of them feeds, the turbulence and U entries of the rows, and backward the
// other half of a last row, which has no upstream row), copied by one bulk
// copy per stream and chunk, completion on the warp's mbarrier.
constexpr int PCH = 16, PRING = 2 * PCH;
template <int NV, bool update>
struct PRing {
  static constexpr int EDGE = 2 * PROWS;                          // stream of the edge row
  static constexpr int T = (EDGE + 1) * PRING * HREC;             // [row][PRING][TREC]
  static constexpr int U = T + (NV > 4 ? PROWS * PRING * TREC : 0);  // [row][PRING][UREC]
  static constexpr int N = U + (update ? 0 : PROWS * PRING * UREC);
};
__device__ __forceinline__ double lds(unsigned a) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double2 lds2(unsigned a) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void stg_if(bool p, double *a, double v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p st.global.f64 [%0], %1;\n\t}" ::"l"(a), "d"(v),
               "r"((int)p)
               : "memory");
}

// to an inbox of this CTA (local) or of another one of the cluster
__device__ __forceinline__ void inbox_write_if(bool local, bool remote, unsigned a, double x) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %2, 0;\n\tsetp.ne.s32 q, %3, 0;\n\t"
      "@p st.relaxed.cluster.shared::cta.b64 [%0], %1;\n\t"
      "@q st.relaxed.cluster.shared::cluster.b64 [%0], %1;\n\t}" ::"r"(a),
      "l"(__double_as_longlong(x)), "r"((int)local), "r"((int)remote)
      : "memory");
}

// what a lane reads for one step, one step ahead
struct PSet {
  double2 n;         // the lane's pair of face coefficients
  double c, a, g;    // cc (or 0), constant term, pressure coefficient
  double e;          // backward, a row without an upstream row: K of the cell itself
  double u;          // without the update: U of the next cell
  double at, ut, dt, rt;
};

struct PWarp {
  int lane, q, r, j, j0, rows, ni;  // j0: the warp's first row
  bool own, row_ok;
  unsigned box, out;   // this pass's inbox of the warp, the inbox it writes to
  bool has_box, has_out, local;  // local: the warp it writes to is in this CTA
  unsigned ring, mbar, phase;  // record ring, its mbarrier and chunk count
};

template <int NV, bool update, bool FWD>
__device__ __forceinline__ void push_pass(const Lvl &L, const BlkDev &bd, PWarp &W, int bk) {
  using RG = PRing<NV, update>;
  constexpr int SB = inbox_words<NV>();
  constexpr int PASS = FWD ? 0 : 1;
  const int q = W.q, ni = W.ni, lag = FWD ? W.r : PROWS - 1 - W.r;
  const long long F = L.F;
  const int tq = NV == 6 ? (q & 1) : 0;
  // a row with no upstream row, and the lanes that take the inbox
  const bool edge = W.own && (FWD ? W.j == 1 : W.j == W.rows);
  const bool boxed = W.own && W.has_box && (FWD ? W.r == 0 : W.r == PROWS - 1), first = edge || boxed;
  const int from = FWD ? (W.lane - 4) & 31 : (W.lane + 12) & 31;
  const bool sends = !W.own && W.has_out && W.row_ok && (FWD ? W.r == PROWS - 1 : W.r == 0);
  const int gl = W.lane & ~7, hl = W.lane & ~3;
  const bool is_p = q == 1, is_g = q == 3;

  // chunk c: visits PCH c .. of every stream; lane s copies stream s.  Kept
  // short: every warp issues at the same steps, and a path of dependent cells
  // that runs down the rows meets that step in every warp
  const bool warp_edge = !FWD && W.j0 + PROWS > W.rows;
  int rec = 0;  // doubles per entry of the lane's stream; 0: no stream
  const double *src = nullptr;
  unsigned dst = W.ring, per_cell = 8u * (2 * PROWS * HREC + (warp_edge ? HREC : 0) + (NV > 4 ? PROWS * TREC : 0) +
                                         (update ? 0 : PROWS * UREC));
  {
    auto row = [&](int j) { return (size_t)bd.cell0 + (size_t)(min(max(j, 1), W.rows) - 1) * ni; };
    const int s = W.lane, r = s & (PROWS - 1);
    if (s < 2 * PROWS) {  // own halves, then the halves of the rows fed
      rec = HREC;
      const int h = s / PROWS;
      src = half_rec(L.rec, L.ncell, PASS, h) + row(W.j0 + r + (h ? (FWD ? 1 : -1) : 0)) * HREC;
      dst += 8u * s * PRING * HREC;
    } else if (s == RG::EDGE) {
      rec = warp_edge ? HREC : 0;
      src = half_rec(L.rec, L.ncell, PASS, 1) + row(W.rows) * HREC;
      dst += 8u * s * PRING * HREC;
    } else if (NV > 4 && s >= 12 && s < 16) {
      rec = TREC;
      src = turb_rec(L.rec, L.ncell, PASS) + row(W.j0 + r) * TREC;
      dst += 8u * (RG::T + r * PRING * TREC);
    } else if (!update && s >= 16 && s < 20) {
      rec = UREC;
      src = u_rec(L.rec, L.ncell, NV) + row(W.j0 + r) * UREC;
      dst += 8u * (RG::U + r * PRING * UREC);
    }
  }
  auto issue = [&](int c) {
    const int n = min(PCH, ni - c * PCH);
    if (n <= 0) return;
    __syncwarp();
    const int cell = FWD ? c * PCH : ni - c * PCH - n;         // first cell of the chunk
    const int slot = (c & 1) * PCH + (FWD ? 0 : PCH - n);      // its place in the ring
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.eq.s32 p, %4, 0;\n\tsetp.ne.u32 q, %2, 0;\n\t"
        "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%3], %5;\n\t"
        "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(
            dst + 8u * rec * slot),
        "l"(src + (size_t)rec * cell), "r"(8u * rec * n), "r"(W.mbar), "r"(W.lane), "r"(per_cell * n)
        : "memory");
  };
  int gave_up = -1;
  auto arrived = [&](int c) {
    if (c * PCH >= ni) return;
    unsigned done = 0;
    for (int n = 0; n < PWAIT && !done; n++)
      asm volatile(
          "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(done)
          : "r"(W.mbar), "r"(W.phase & 1u)
          : "memory");
    if (!done && gave_up < 0) gave_up = c * PCH;
    W.phase++;
    __syncwarp();
  };
  issue(0);
  // the lane's fields within its stream's entries
  const unsigned ring = W.ring + 8u * (W.r + (W.own ? 0 : PROWS)) * PRING * HREC;
  const unsigned rn = ring + 8u * (is_g ? H_G1 : H_N1), rc = ring + 8u * (q < 2 ? H_C : H_Z);
  const unsigned ra = ring + 8u * (H_A + q), rg = ring + 8u * (q == 1 ? H_G1 : q == 2 ? H_G2 : H_Z);
  const unsigned re = W.ring + 8u * (RG::EDGE * PRING * HREC + H_A + q);
  const unsigned rt_ = W.ring + 8u * (RG::T + W.r * PRING * TREC + tq), ru = W.ring + 8u * (RG::U + W.r * PRING * UREC + q);
  // ring entry of visit k
  auto at = [&](int k) { return (unsigned)((k & (PRING - 1)) ^ (FWD ? 0 : PCH - 1)); };
  // the fields for step t: of visit k + 1 for the first half rows, k for the others
  auto load = [&](PSet &s, int t) {
    const int k = t - lag;
    const unsigned e = at(W.own ? k + 1 : k), o = 8u * HREC * e;
    s.n = lds2(rn + o);
    s.c = lds(rc + o);
    s.a = lds(ra + o);
    s.g = lds(rg + o);
    if (!FWD) s.e = lds(re + 8u * HREC * at(k));
    if (!update) s.u = lds(ru + 8u * UREC * e);
    if (NV > 4) {
      const unsigned ot = rt_ + 8u * TREC * e;
      const double a = lds(ot + 8u * T_AT);
      s.at = W.own ? a : 0.0;
      s.ut = lds(ot + 8u * T_UT);
      if (!FWD) s.dt = lds(ot + 8u * T_DT);
      if (NV == 5) s.rt = lds(ot + 8u * T_RT - 8u * tq);
    }
  };
  arrived(0);
  PSet s0{}, s1{};
  double acc = 0.0, acct = 0.0, ucur = 0.0, ut = 0.0, dtf = 0.0, rt = 0.0;
  if (W.own) {
    const unsigned e = at(0);
    acc = lds(ra + 8u * HREC * e);
    if (!update) ucur = lds(ru + 8u * UREC * e);
    if (NV > 4) {
      const unsigned ot = rt_ + 8u * TREC * e;
      acct = lds(ot + 8u * T_AT);
      ut = lds(ot + 8u * T_UT);
      if (!FWD) dtf = lds(ot + 8u * T_DT);
      if (NV == 5) rt = lds(ot + 8u * T_RT - 8u * tq);
    }
  }
  load(s0, 0);
  const unsigned box = W.box + 8u * q, boxt = W.box + 8u * (4 + tq);
  const unsigned out = W.out + 8u * q;
  // results of the first half rows: forward into the backward records,
  // backward into U (or dU)
  const int jo = min(W.j, W.rows);
  double *wp, *wpt;
  long long ws, wst;
  if (FWD) {
    const size_t c0 = (size_t)bd.cell0 + (size_t)(jo - 1) * ni;
    wp = half_rec(L.rec, L.ncell, 1, 0) + c0 * HREC + H_A + q;
    wpt = turb_rec(L.rec, L.ncell, 1) + c0 * TREC + T_DT + tq;
    ws = HREC; wst = TREC;
  } else {
    const long long id = bd.off + (long long)(jo + 2) * bd.P + 2 + ni;
    wp = (update ? L.U : L.du) + q * F + id;
    wpt = (update ? L.U : L.du) + (4 + tq) * F + id;
    ws = wst = -1;
  }
  wp -= (long long)lag * ws;
  wpt -= (long long)lag * wst;

  // hold: a row's first half keeps its start value until the row begins
  auto step = [&](int t, const PSet &cur, PSet &next, bool hold) {
    const int k = t - lag;
    const bool act = W.row_ok && (unsigned)k < (unsigned)ni;
    // the inbox words of this step (read in the shadow of the last step's FMA)
    unsigned long long v = 0, vt = 0;
    {
      const unsigned o = 8u * SB * (unsigned)min(t, ni - 1);
      v = inbox_read(box + o);
      if (NV > 4) vt = inbox_read(boxt + o);
      const bool need = W.has_box && t < ni && gave_up < 0;
      auto empty = [&] { return need && (hi_of(v) == hi_of(EMPTY) || (NV > 4 && hi_of(vt) == hi_of(EMPTY))); };
      if (__any_sync(FULL, empty())) {
        for (int n = 0; __any_sync(FULL, empty()); n++) {
          if (n == PWAIT) { gave_up = t; break; }
          v = inbox_read(box + o);
          if (NV > 4) vt = inbox_read(boxt + o);
        }
      }
    }
    double other = __shfl_sync(FULL, acc, from);
    double othert = NV > 4 ? __shfl_sync(FULL, acct, from) : 0.0;
    // the last step's terms to the next warp: after the shuffles, so that
    // nothing above waits for the FMA that forms them
    {
      const bool go = sends && (unsigned)(k - 1) < (unsigned)ni;
      const unsigned o = out + 8u * SB * (unsigned)(k - 1);
      inbox_write_if(go && W.local, go && !W.local, o, acc);
      if (NV > 4) inbox_write_if(go && q < NV - 4 && W.local, go && q < NV - 4 && !W.local, o + 32u, acct);
    }
    if (first) {
      other = edge ? (FWD ? 0.0 : cur.e) : __longlong_as_double((long long)v);
      othert = edge ? 0.0 : __longlong_as_double((long long)vt);
    }
    // the new state of the cell (first half row)
    const double dn = acc + other;
    const double st = update ? dn : ucur + dn;
    double dnt = 0.0, stt = 0.0;
    if (NV > 4) {
      const double a = acct + othert;
      dnt = FWD ? (NV == 5 ? a * rt : a) : (NV == 5 ? fma(a, rt, dtf) : a + dtf);
      stt = ut + dnt;
    }
    const double v0 = __shfl_sync(FULL, st, gl), v1 = __shfl_sync(FULL, st, gl + 1);
    const double v2 = __shfl_sync(FULL, st, gl + 2), v3 = __shfl_sync(FULL, st, gl + 3);
    const double x = __shfl_sync(FULL, st, gl + q);
    // m and z with the lane's operands; lane 1 forms 2 p' = 2 E - (m1^2 +
    // m2^2) / rho, the doubling and the sign on the integer pipe
    const double a1 = is_p ? neg(v1) : cur.n.x, a2 = is_p ? neg(v2) : cur.n.y;
    const double kz = is_p ? twice(v3) : cur.c;
    const double m = fma(v1, a1, v2 * a2);
    const double rd = recip(v0);
    // the next step's fields and this step's results, in the shadow of the
    // longest stretch of FP64 instructions
    load(next, t + 1);
    stg_if(act && W.own, wp, FWD || !update ? dn : st);
    if (NV > 4) stg_if(act && W.own && q < NV - 4, wpt, FWD || !update ? dnt : stt);
    wp += ws;
    if (NV > 4) wpt += wst;
    const double z = fma(m, rd, kz);
    const double w = __shfl_sync(FULL, z, hl), pr = __shfl_sync(FULL, z, hl + 1);
    const double nacc = fma(x, w, fma(pr, is_g ? z : cur.g, cur.a));
    double nacct = 0.0;
    if (NV > 4) {
      const double un = __shfl_sync(FULL, z, hl + 2);
      const double T2 = __shfl_sync(FULL, stt, gl + tq), D2 = __shfl_sync(FULL, dnt, gl + tq);
      nacct = fma(cur.c, D2, fma(T2, un, cur.at));
    }
    if (!hold || act || !W.own) {
      acc = nacc;
      acct = nacct;
      if (!update) ucur = cur.u;
      if (NV > 4) { ut = cur.ut; dtf = cur.dt; rt = cur.rt; }
    }
  };
  // chunk c is needed from step PCH c - 2 on (the fields of step t + 1 are
  // read in step t, one visit ahead in the first half rows), and its place in
  // the ring is free once no row reads chunk c - 2 (lags of up to three steps)
  step(0, s0, s1, true);
  step(1, s1, s0, true);
  step(2, s0, s1, true);
  step(3, s1, s0, false);
  // (one step more than the last row's cells: it sends that row's last terms)
  for (int t = 4; t < ni + PROWS; t += 2) {
    const int ph = t & (PCH - 1);
    if (ph == 4) issue(t / PCH + 1);
    if (ph == PCH - 2) arrived(t / PCH + 1);
    step(t, s0, s1, false);
    step(t + 1, s1, s0, false);
  }
  if (gave_up >= 0 && W.lane == 0)
    set_status(L.status + 4 * bd.cas, 4, bk, FWD ? min(gave_up, ni - 1) + 1 : max(ni - gave_up, 1), min(W.j0, W.rows));
}

// R = 4 x warps rows per CTA, CS CTAs (a cluster) per block
template <int NV, bool update>
__global__ void __launch_bounds__(32 * PWARPS, 1) k_push_sweep(Lvl L, int CS) {
  using RG = PRing<NV, update>;
  constexpr int SB = inbox_words<NV>();
  // record rings [warp][RG::N], inboxes [warp][column][SB]
  extern __shared__ __align__(16) unsigned long long shm[];
  __shared__ __align__(8) unsigned long long mbar[PWARPS];
  const int nw = blockDim.x >> 5, wi = threadIdx.x >> 5;
  const unsigned rank = CS > 1 ? push_rank() : 0u;
  const int bk = blockIdx.x / CS;
  const BlkDev bd = L.blk[bk];  // by value: no re-reads after global stores
  PWarp W;
  W.lane = threadIdx.x & 31;
  W.q = W.lane & 3;
  W.r = W.lane >> 3;
  W.own = !((W.lane >> 2) & 1);
  W.rows = bd.ny - 1;
  W.ni = bd.nx - 1;
  const int gw = (int)rank * nw + wi;  // warp number within the block
  W.j0 = gw * PROWS + 1;
  W.j = W.j0 + W.r;
  W.row_ok = W.j <= W.rows;
  W.out = 0;
  W.local = true;
  const int words = W.ni * SB;
  unsigned long long *inbox = shm + (size_t)nw * RG::N, *mine = inbox + (size_t)wi * words;
  auto barrier = [&] {
    if (CS > 1) push_cluster_barrier();
    else __syncthreads();
  };
  auto clear = [&] {
    for (int t = W.lane; t < words; t += 32) mine[t] = EMPTY;
  };
  clear();
  W.mbar = (unsigned)__cvta_generic_to_shared(mbar + wi);
  W.phase = 0;
  if (W.lane == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(W.mbar), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  barrier();  // every inbox empty before any warp writes into one
  const bool used = W.j0 <= W.rows, up = gw > 0, down = W.j0 + PROWS <= W.rows;
  W.ring = (unsigned)__cvta_generic_to_shared(shm) + 8u * RG::N * (unsigned)wi;
  W.box = (unsigned)__cvta_generic_to_shared(mine);
  auto send_to = [&](int w) {  // the inbox of warp w of this block
    const unsigned a = (unsigned)__cvta_generic_to_shared(inbox + (size_t)(w % nw) * words);
    W.local = w / nw == (int)rank;
    W.out = W.local ? a : push_remote(a, (unsigned)(w / nw));
  };
  // forward: from the warp above (lower j) to the one below; backward: the
  // other way round, once every warp has done its forward pass and emptied its
  // inbox again (the others wait for the last one anyway)
  if (used) {
    W.has_box = up;
    W.has_out = down && !L.silent_band_edge;
    if (down) send_to(gw + 1);
    push_pass<NV, update, true>(L, bd, W, bk);
    // the forward results, written by this warp, are read by its bulk copies
    asm volatile("fence.proxy.async;" ::: "memory");
    __syncwarp();
    clear();
  }
  barrier();
  if (used) {
    W.has_box = down;
    W.has_out = up && !L.silent_band_edge;
    if (up) send_to(gw - 1);
    push_pass<NV, update, false>(L, bd, W, bk);
  }
  barrier();  // no CTA leaves while a neighbour may still write into it
}

static void (*push_kernel(int nv, int update))(Lvl, int) {
  if (nv == 4) return update ? k_push_sweep<4, true> : k_push_sweep<4, false>;
  if (nv == 5) return update ? k_push_sweep<5, true> : k_push_sweep<5, false>;
  return update ? k_push_sweep<6, true> : k_push_sweep<6, false>;
}

struct PushShape {
  int CS, nw;
  size_t smem;
};
static size_t ring_doubles(int nv, int update) {
  return nv == 4 ? (update ? PRing<4, true>::N : PRing<4, false>::N) : (update ? PRing<6, true>::N : PRing<6, false>::N);
}
static PushShape push_shape(int max_rows, int max_cols, int rmax, int nv, int update) {
  PushShape p;
  const int warps = (max_rows + PROWS - 1) / PROWS;
  p.nw = std::max(1, std::min((rmax + PROWS - 1) / PROWS, PWARPS));
  p.CS = (warps + p.nw - 1) / p.nw;
  p.nw = (warps + p.CS - 1) / p.CS;
  p.smem = p.nw * (ring_doubles(nv, update) + (size_t)max_cols * (nv == 4 ? 4 : nv)) * sizeof(double);
  return p;
}
static void push_attributes(const PushShape &p, int nv, int update) {
  auto kern = push_kernel(nv, update);
  if (p.smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
  if (p.CS > 8) cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}
static cudaLaunchConfig_t push_config(const Lvl &L, const PushShape &p, cudaLaunchAttribute *attr, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(L.nblk * p.CS);
  cfg.blockDim = dim3(32 * p.nw);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// bands of at most rmax rows (rounded up to whole warps of four): at most 16
// CTAs per block, an SM for every CTA (with fewer, the one-lane sweep's lower
// FP64 instruction count per cell wins) and the inboxes in shared memory
bool push_fits(const Lvl &L, int update, int max_rows, int max_cols, int rmax) {
  static const int nsm = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
  }();
  const PushShape p = push_shape(max_rows, max_cols, rmax, L.nvar, update);
  if (max_rows < 1 || p.CS > 16 || p.smem > 226 * 1024 || (long long)L.nblk * p.CS > nsm) return false;
  if (p.CS <= 8) return true;
  // a non-portable cluster size: launchable only if the device can place one
  push_attributes(p, L.nvar, update);
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = push_config(L, p, attr, nullptr);
  int n = 0;
  const bool ok = cudaOccupancyMaxActiveClusters(&n, push_kernel(L.nvar, update), &cfg) == cudaSuccess && n >= 1;
  cudaGetLastError();  // a refused query leaves no error behind
  return ok;
}

void launch_push_prep(const Lvl &L, double alfa1, int update, int force, cudaStream_t s) {
  auto go = [&](auto kern) { kern<<<L.nctiles, TILE, 0, s>>>(L, alfa1, force); };
  if (L.nvar == 4) update ? go(k_push_prep<4, true>) : go(k_push_prep<4, false>);
  else if (L.nvar == 5) update ? go(k_push_prep<5, true>) : go(k_push_prep<5, false>);
  else update ? go(k_push_prep<6, true>) : go(k_push_prep<6, false>);
}

void launch_push(const Lvl &L, int update, int max_rows, int max_cols, int rmax, cudaStream_t s) {
  const PushShape p = push_shape(max_rows, max_cols, rmax, L.nvar, update);
  push_attributes(p, L.nvar, update);
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = push_config(L, p, attr, s);
  cudaLaunchKernelEx(&cfg, push_kernel(L.nvar, update), L, p.CS);
}

}  // namespace ec2d
