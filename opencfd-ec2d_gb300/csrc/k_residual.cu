// k_residual.cu -- the residual of sub_Residual.f90 on the GPU.
//
// One residual evaluation of a mesh level (Comput_Residual_one_mesh,
// sub_Residual.f90:13-107) is a chain of launches over all blocks of all cases:
//   k_prim      primitives d,u,v,T,p (+c, Sutherland mu)       comput_duvtpckw + get_viscous
//   k_flux_i/j  reconstruction + Riemann flux + viscous stress  Residual_FVM face loops
//   k_res       flux differences, spectral radii, time step    Residual_FVM:460-468, comput_Lvc, comput_dt
//   k_norm_*    max / RMS residual norms, deterministic order  sub_Residual.f90:72-106
// Work is distributed by EC2D_TILE-item tiles of each block's extended index
// range [-1,nx+1] x [-1,ny+1] (k_prim: the primitives of both ghost layers)
// or of its core range [0,nx] x [0,ny] (the face, residual and norm kernels,
// core_ij); a kernel maps the tile item to (i,j) and keeps the items that lie
// in its own index range.
#include "ec2d_dev.cuh"
#include "ec2d_internal.h"
#include "ec2d_mixed.cuh"

#include <type_traits>

namespace ec2d {

constexpr int TILE = EC2D_TILE;

__device__ __forceinline__ bool tile_ij(const Lvl &L, int &bk, int &i, int &j) {
  int2 t = L.tiles[blockIdx.x];
  bk = t.x;
  const BlkDev &b = L.blk[bk];
  int W = b.nx + 3, H = b.ny + 3;
  int lin = t.y + threadIdx.x;
  if (lin >= W * H) return false;
  i = lin % W - 1;
  j = lin / W - 1;
  return true;
}

// M (here and below): a context with FP32 parts, whose arithmetic keeps its order of
// operations (ec2d_mixed.cuh)
struct Prim { double u, v, T, p, sT; };
template <bool M>
__device__ __forceinline__ Prim primitives(const CaseDev &c, double d, double ru, double rv, double E) {
  Prim w;
  if constexpr (M) {
    const double rd = rcp(d);
    w.u = ru * rd;
    w.v = rv * rd;
    w.T = (E - 0.5 * d * (w.u * w.u + w.v * w.v)) * (rd * c.rCv);
    w.p = c.p00 * d * w.T;
    w.sT = w.T > 0.0 ? sqrt_p(w.T) : sqrt(w.T);  // the reference's sqrt, NaN for T < 0
  } else {
    const double rd = recip(d);
    w.u = ru * rd;
    w.v = rv * rd;
    const double e = E - half(fma(ru, w.u, rv * w.v));
    w.T = e * (rd * c.rCv);
    w.p = e * c.gm1;
    w.sT = root_t(w.T);
  }
  return w;
}
template <bool M>
__device__ __forceinline__ double sutherland(const CaseDev &c, const Prim &w) {  // T^1.5 = T sqrt(T)
  if constexpr (M) return c.rRe * (1.0 + c.Tsb) * (w.T * w.sT) * rcp(c.Tsb + w.T);
  else return c.mu0 * (w.T * w.sT) * recip(c.Tsb + w.T);
}

// comput_duvtpckw (sub_Residual.f90:114-152) + get_viscous (:670-689) + Amu_t=0
// (:172); 14 FP64 instructions per viscous cell of an FP64 context instead of 29 (1.05 M
// cells: 36 us instead of 68)
template <bool M>
__global__ void __launch_bounds__(TILE) k_prim(Lvl L) {
  int bk, i, j;
  if (!tile_ij(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  const CaseDev &c = L.cs[b.cas];
  long long id = fidx(b, i, j);
  const long long F = L.F;
  const double d = L.U[id];
  const Prim w = primitives<M>(c, d, L.U[F + id], L.U[2 * F + id], L.U[3 * F + id]);
  L.q[Q_D * F + id] = d;
  L.q[Q_U * F + id] = w.u;
  L.q[Q_V * F + id] = w.v;
  L.q[Q_T * F + id] = w.T;
  L.q[Q_P * F + id] = w.p;
  bool interior = (i >= 1 && i <= b.nx - 1 && j >= 1 && j <= b.ny - 1);
  if (interior) {
    if (!at_least(w.T, 1.0e-5)) set_status(L.status + 4 * b.cas, 3, bk, i, j);
    L.q[Q_C * F + id] = w.sT * c.rMa;
  }
  if (L.visc) {
    if (i >= 0 && i <= b.nx && j >= 0 && j <= b.ny) L.amu[id] = sutherland<M>(c, w);
    if (!L.keep_amut) L.amut[id] = 0.0;
  }
}

__device__ __forceinline__ bool in_fdm_core(const BlkDev &b, int i, int j) {
  return b.fdm && (i >= LFDM + 2 && i <= b.nx - LFDM - 1) && (j >= LFDM + 2 && j <= b.ny - LFDM - 1);
}

// Limited slopes of a large level's cells, two planes per direction and variable (to the
// upper face, to the lower).  The limiter belongs to the cell, so the two faces of a
// direction share it: 96 FP64 instructions per cell here and 8 per face for the states,
// against 2 x 80 where each face forms both of its sides.  M: the planes
// hold the states themselves, with the bits that the faces form (batch of 16 airfoils,
// 0.6 M cells on the finest level: 3.49 -> 3.32 ms per V-cycle).
// The planes' traffic (256 bytes per cell) hides behind the FP64 pipe, but the launch
// pays only on large levels (slope_level).
// The planes are memory that holds nothing between the primitives and the fluxes: the
// array of the sweep records, or, where a level has none (more rows than a CTA's sweep
// takes) or a smaller one, eight planes for one direction at a time: the turbulence rows
// of the face fluxes, and the mean-flow rows of Res, which k_res and the FDM patch
// fill over every interior cell.  Taking turns costs 2 x 1024 x 512 cells 0.8 % of an
// RK3 step and 0.3 M cells 2 % of a residual against planes of their own.
__device__ __forceinline__ double *slope_planes(const Lvl &L, bool iface, int m) {
  if (L.slope) return L.slope + ((iface ? 0 : 8) + 2 * m) * L.F;
  return m == 0 ? L.fi + 4 * L.F : m == 1 ? L.fj + 4 * L.F : L.res + (2 * m - 4) * L.F;
}
template <bool M>
__global__ void __launch_bounds__(TILE) k_slopes(Lvl L, int dirs) {
  int bk, i, j;
  if (!core_ij(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  const long long F = L.F, id = fidx(b, i, j);
#pragma unroll
  for (int dir = 0; dir < 2; dir++) {
    if (!(dirs & (dir == 0 ? SLOPES_I : SLOPES_J))) continue;
    if (dir == 0 ? j < 1 || j > b.ny - 1 || i < 0 || i > b.nx : i < 1 || i > b.nx - 1 || j < 0 || j > b.ny) continue;
    const long long st = dir == 0 ? 1 : b.P;
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int pl = m == 0 ? Q_D : m == 1 ? Q_U : m == 2 ? Q_V : Q_P;
      const double *q = L.q + pl * F + id;
      const double u = q[0];
      double a, c;
      if constexpr (M) mixed::muscl3_states(q[-st], u, q[st], a, c);
      else muscl3_slopes(u - q[-st], q[st] - u, a, c);
      double *sp = slope_planes(L, dir == 0, m) + id;
      sp[0] = a;
      sp[F] = c;
    }
  }
}

// inviscid flux of a face from the states before and after it, F = -s (flux)
template <bool M, typename T>
__device__ __forceinline__ void inviscid_states(const Lvl &L, const CaseDev &c, const T *UL, const T *UR, T n1, T n2, T s, T *F) {
  if constexpr (M) {
    T QL[4] = {UL[0], UL[1] * n1 + UL[2] * n2, -UL[1] * n2 + UL[2] * n1, UL[3]};
    T QR[4] = {UR[0], UR[1] * n1 + UR[2] * n2, -UR[1] * n2 + UR[2] * n1, UR[3]};
    T Fl[4];
    mixed::face_flux(L.flux, QL, QR, Fl, to<T>(c.gamma), to<T>(c.ggm1));
    F[0] = -Fl[0] * s;
    F[1] = -(Fl[1] * n1 - Fl[2] * n2) * s;
    F[2] = -(Fl[1] * n2 + Fl[2] * n1) * s;
    F[3] = -Fl[3] * s;
  } else {
    face_flux(L.flux, UL, UR, n1, n2, s, F, gas(c));
  }
}
// the same with the reconstruction
template <bool M, typename T>
__device__ __forceinline__ void inviscid(const Lvl &L, const CaseDev &c, int scheme, T S0[4][4], T n1, T n2, T s, T *F) {
  T UL[4], UR[4];
  if constexpr (M) mixed::reconstruct(L.recon, scheme, S0, to<T>(c.gamma), UL, UR);
  else reconstruct(L.recon, scheme, S0, gas(c), UL, UR);
  inviscid_states<M>(L, c, UL, UR, n1, n2, s, F);
}
// viscous terms of a face, added to F.  across: from the cell before the face to the
// one after; along: the sum over both cells of the differences between their
// neighbours beside the face's ends.  g: the face's four metric planes; ml, tl and
// mr, tr: laminar and eddy viscosity before and after the face (eddy: the latter
// are not zero by the level's model); lo, hi: a face on the block's first or last
// line, which takes the interior cell's.
template <typename T>
struct FaceDiff { T xu, xv, xT, yu, yv, yT, us, vs; };
template <bool M, bool IFACE, typename T>
__device__ __forceinline__ void viscous(const CaseDev &c, const double *g, long long F, const FaceDiff<T> &D, T ml, T mr,
                                        bool eddy, T tl, T tr, bool lo, bool hi, T n1, T n2, T s, T *Fo) {
  if constexpr (M) {
    // (the laminar product fused, the eddy one rounded: the order is part of the results)
    T Amu1, Amk1;
    const T Cp = to<T>(c.Cp), rPr = to<T>(c.rPr), rPrT = (T)(1.0 / PrT);
    if (lo) {
      Amu1 = mr + tr;
      Amk1 = Cp * fma(mr, rPr, tr * rPrT);
    } else if (hi) {
      Amu1 = ml + tl;
      Amk1 = Cp * fma(ml, rPr, tl * rPrT);
    } else {
      // the two families of faces add the viscosities in their own order
      if (IFACE) Amu1 = mixed::scaled<-1>(ml + mr + tl + tr);
      else Amu1 = mixed::scaled<-1>(mr + ml + tr + tl);
      Amk1 = mixed::scaled<-1>(Cp * fma(ml + mr, rPr, (tl + tr) * rPrT));
    }
    const T yu = mixed::scaled<-2>(D.yu), yv = mixed::scaled<-2>(D.yv), yT = mixed::scaled<-2>(D.yT);
    mixed::viscous_face_m(to<T>(g[0]), to<T>(g[F]), to<T>(g[2 * F]), to<T>(g[3 * F]), IFACE ? D.xu : yu, IFACE ? D.xv : yv,
                          IFACE ? D.xT : yT, IFACE ? yu : D.xu, IFACE ? yv : D.xv, IFACE ? yT : D.xT, Amu1, Amk1,
                          mixed::scaled<-1>(D.us), mixed::scaled<-1>(D.vs), n1, n2, s, Fo[1], Fo[2], Fo[3]);
  } else {
    const double h = half(s);
    double mu = ((lo ? mr : ml) + (hi ? ml : mr)) * h, k = mu * c.kpr;
    if (eddy) {
      const double mt = ((lo ? tr : tl) + (hi ? tl : tr)) * h;
      k = fma(mt, c.kprt, k);
      mu += mt;
    }
    viscous_face_m(g[0], g[F], g[2 * F], g[3 * F], IFACE ? D.xu : D.yu, IFACE ? D.xv : D.yv, IFACE ? D.xT : D.yT,
                   IFACE ? D.yu : D.xu, IFACE ? D.yv : D.xv, IFACE ? D.yT : D.xT, mu, k, D.us, D.vs, n1, n2, Fo[1],
                   Fo[2], Fo[3]);
  }
}
// the differences from u(k), v(k), T(k) at cell k; r: the cell after the face, st: to the
// cell before it, ot: along the face
template <bool M, typename T, typename Fu, typename Fv, typename FT>
__device__ __forceinline__ FaceDiff<T> face_diff(long long r, long long st, long long ot, Fu u, Fv v, FT t) {
  const long long l = r - st, n = r + ot, z = r - ot;
  auto along = [&](auto &q) -> T {
    if constexpr (M) return q(n - st) + q(n) - q(z - st) - q(z);
    else return (q(n - st) - q(z - st)) + (q(n) - q(z));
  };
  return {u(r) - u(l), v(r) - v(l), t(r) - t(l), along(u), along(v), along(t), u(r) + u(l), v(r) + v(l)};
}

// The face kernels are bound by the issue of FP64 instructions (one per 16 to 19
// cycles and SM; memory traffic is a tenth of the time): a viscous MUSCL3 / AUSM+
// face takes about 166 of them (reconstruction 80, flux 44, viscous terms 42; 97 from
// the cells' slopes) where the formulas written out with divides, rotations and
// floating-point selects take 273 (M, ec2d_mixed.cuh).  65 k cells take 27 us per
// direction between events instead of 39, 1.05 M cells with the slopes 205 (and 195 for
// both directions' slopes) instead of 600, HLLC with characteristic WENO3 on 131 x
// 59 cells 22 instead of 41, most of them the chain of one face.  In FP32 the
// values are converted on the integer pipes (to<float>), not by the FP64 pipe.
// IFACE: face loop in i of Residual_FVM (sub_Residual.f90:238-346), face (i,j),
// i=1..nx, j=1..ny-1, between cells (i-1,j) and (i,j); else in j (:352-455), face (i,j),
// i=1..nx-1, j=1..ny, between cells (i,j-1) and (i,j).
// SLOPES: from the cells' limited slopes (k_slopes).
template <bool M, bool IFACE, bool SLOPES, typename T>
__global__ void __launch_bounds__(TILE) k_flux(Lvl L) {
  int bk, i, j;
  if (!core_ij(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  if (i < 1 || i > b.nx - !IFACE || j < 1 || j > b.ny - IFACE) return;
  if (in_fdm_core(b, i, j)) return;
  const CaseDev &c = L.cs[b.cas];
  const long long F = L.F, st = IFACE ? 1 : b.P, id = fidx(b, i, j);
  const T s = to<T>(L.geo[(IFACE ? G_SI : G_SJ) * F + id]), n1 = to<T>(L.geo[(IFACE ? G_NI1 : G_NJ1) * F + id]),
          n2 = to<T>(L.geo[(IFACE ? G_NI2 : G_NJ2) * F + id]);
  T Fl[4];
  if constexpr (SLOPES) {
    double UL[4], UR[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int pl = m == 0 ? Q_D : m == 1 ? Q_U : m == 2 ? Q_V : Q_P;
      const double *sp = slope_planes(L, IFACE, m) + id;
      UL[m] = M ? sp[-st] : L.q[pl * F + id - st] + sp[-st];
      UR[m] = M ? sp[F] : L.q[pl * F + id] - sp[F];
    }
    inviscid_states<M>(L, c, UL, UR, n1, n2, s, Fl);
  } else {
    T S0[4][4];
    int scheme = L.scheme;
    if (L.recon == Recon_Original) {
      if (!IFACE) scheme = L.gscheme;  // the reference passes the global Iflag_Scheme here (sub_Residual.f90:367)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const long long q = id + (k - 2) * st;
        S0[k][0] = to<T>(L.q[Q_D * F + q]); S0[k][1] = to<T>(L.q[Q_U * F + q]);
        S0[k][2] = to<T>(L.q[Q_V * F + q]); S0[k][3] = to<T>(L.q[Q_P * F + q]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++)
#pragma unroll
        for (int m = 0; m < 4; m++) S0[k][m] = to<T>(L.U[m * F + id + (k - 2) * st]);
    }
    inviscid<M>(L, c, scheme, S0, n1, n2, s, Fl);
  }
  if (L.visc) {
    const double *uu = L.q + Q_U * F, *vv = L.q + Q_V * F, *TT = L.q + Q_T * F;
    auto u = [=](long long k) { return to<T>(uu[k]); };
    auto v = [=](long long k) { return to<T>(vv[k]); };
    auto t = [=](long long k) { return to<T>(TT[k]); };
    const bool eddy = M || L.turb != Turb_NONE || L.keep_amut;
    T tl = T(0), tr = T(0);
    if (eddy) { tl = to<T>(L.amut[id - st]); tr = to<T>(L.amut[id]); }
    viscous<M, IFACE>(c, L.geo + (IFACE ? G_VIP : G_VJP) * F + id, F, face_diff<M, T>(id, st, IFACE ? b.P : 1, u, v, t),
                      to<T>(L.amu[id - st]), to<T>(L.amu[id]), eddy, tl, tr, (IFACE ? i : j) == 1,
                      IFACE ? i == b.nx : j == b.ny, n1, n2, s, Fl);
  }
  double *out = IFACE ? L.fi : L.fj;
#pragma unroll
  for (int m = 0; m < 4; m++) out[m * F + id] = to_double(Fl[m]);
}

// Norm reductions.  max |Res| is reduced on the bit patterns: for
// non-negative doubles the order of the patterns as signed 64-bit integers is
// the order of the values, so the maxima run on the integer pipes (an FP64
// warp instruction holds its sub-partition for 64 cycles on this part) and
// are exact in any order.  Sums of Res^2 run in a fixed tree order.
__device__ __forceinline__ long long warp_max_bits(long long a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a = max(a, __shfl_xor_sync(0xffffffffu, a, o));
  return a;
}
__device__ __forceinline__ double warp_sum(double q) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
  return q;
}

// NV variables (4 or 8) reduced over a warp at once by a transposed
// butterfly: at each of the first log2(NV) exchanges a lane keeps half of the
// variables it carries and combines them with its partner's copies, so one
// instruction serves several variables (four sums take 2 + 1 + 3 FP64 adds per
// lane instead of 4 x 5, eight take 4 + 2 + 1 + 2 instead of 8 x 5).  Lane l
// ends with the warp's value of variable l / (32 / NV); every lane of that
// group holds the same bits (each exchange adds the same two operands on both
// sides), and the order of the operations is fixed.
struct OpMax { __device__ long long operator()(long long a, long long b) const { return max(a, b); } };
struct OpAdd { __device__ double operator()(double a, double b) const { return a + b; } };
template <int NV, typename T, typename Op>
__device__ __forceinline__ T warp_reduce_vars(const T (&v)[NV], Op op) {
  static_assert(NV == 4 || NV == 8, "four or eight variables");
  constexpr int R = NV == 4 ? 2 : 3;  // exchanges that halve the variables
  const int lane = threadIdx.x & 31;
  T c[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) c[k] = v[k];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int o = 16 >> r, n = NV >> (r + 1);  // lanes o apart; variables kept
    const bool hi = lane & o;
#pragma unroll
    for (int k = 0; k < NV / 2; k++) {
      if (k < n) {
        const T keep = hi ? c[n + k] : c[k], send = hi ? c[k] : c[n + k];
        c[k] = op(keep, __shfl_xor_sync(0xffffffffu, send, o));
      }
    }
  }
#pragma unroll
  for (int o = 32 / NV / 2; o > 0; o >>= 1) c[0] = op(c[0], __shfl_xor_sync(0xffffffffu, c[0], o));
  return c[0];
}

// one warp's max |Res| bits and sum Res^2 of NV variables into the CTA's
// shared arrays (column w)
template <int NV, int NW>
__device__ __forceinline__ void warp_partials(bool act, const double *vres, int nv, long long (*smax)[NW],
                                              double (*ssum)[NW]) {
  long long a[NV];
  double q[NV];
#pragma unroll
  for (int m = 0; m < NV; m++) {
    // variables past the sixth are zero at compile time (no FP64 work)
    const double r = (m < 6 && act && m < nv) ? vres[m < 6 ? m : 0] : 0.0;
    a[m] = __double_as_longlong(fabs(r));
    q[m] = m < 6 ? r * r : 0.0;
  }
  const long long am = warp_reduce_vars<NV>(a, OpMax());
  const double qs = warp_reduce_vars<NV>(q, OpAdd());
  const int lane = threadIdx.x & 31, g = lane / (32 / NV);
  if (lane % (32 / NV) == 0 && g < nv) {
    smax[g][threadIdx.x >> 5] = am;
    ssum[g][threadIdx.x >> 5] = qs;
  }
}

// one CTA's partials: per variable the max |Res| and sum Res^2 of its cells
// (NT threads in the CTA)
template <int NT = TILE>
__device__ __forceinline__ void tile_partials(const Lvl &L, bool act, const double *vres) {
  __shared__ long long smax[6][NT / 32];
  __shared__ double ssum[6][NT / 32];
  const int nv = L.nvar;
  if (nv <= 4) warp_partials<4, NT / 32>(act, vres, nv, smax, ssum);
  else warp_partials<8, NT / 32>(act, vres, nv, smax, ssum);
  __syncthreads();
  if (threadIdx.x < 6) {
    const int m = threadIdx.x;
    long long a = 0;
    double q = 0.0;
    if (m < nv)
      for (int k = 0; k < NT / 32; k++) { a = max(a, smax[m][k]); q += ssum[m][k]; }
    L.npart[(size_t)blockIdx.x * 12 + m] = __longlong_as_double(a);
    L.npart[(size_t)blockIdx.x * 12 + 6 + m] = q;
  }
}

// per case and quantity (max[6], rms[6]) from the tile partials: one warp per
// (case, quantity), lanes over tiles with four loads in flight per lane (four
// accumulators in a fixed order), then the warp tree
__device__ __forceinline__ void final_norm(const Lvl &L, int cs, int m) {
  const int lane = threadIdx.x & 31;
  const int nt = L.case_ntile[cs];
  const double *p = L.npart + (size_t)L.case_tile0[cs] * 12 + m;
  double out = 0.0;
  if (m < 6) {
    long long a[4] = {0, 0, 0, 0};
    for (int t = lane; t < nt; t += 128) {
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (t + 32 * k < nt) a[k] = max(a[k], __double_as_longlong(p[(size_t)(t + 32 * k) * 12]));
    }
    out = __longlong_as_double(warp_max_bits(max(max(a[0], a[1]), max(a[2], a[3]))));
  } else {
    double q[4] = {0.0, 0.0, 0.0, 0.0};
    for (int t = lane; t < nt; t += 128) {
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (t + 32 * k < nt) q[k] += p[(size_t)(t + 32 * k) * 12];
    }
    const double s = warp_sum((q[0] + q[1]) + (q[2] + q[3]));
    out = (m - 6 < L.nvar) ? sqrt(s / (1.0 * L.case_ncell[cs])) : 0.0;
  }
  if (lane == 0) L.norms[cs * 12 + m] = out;
}

// viscous spectral radii of a cell (comput_Lvc)
template <bool M>
__device__ __forceinline__ void viscous_radii(const CaseDev &c, const double *g, long long F, double d, double amu, bool eddy,
                                              double amut, double &Lvi, double &Lvj) {
  double m;
  if constexpr (M) {
    m = c.gamma * rcp(d) * (amu * c.rPr + amut * (1.0 / PrT));
  } else {
    m = amu * c.gpr;
    if (eddy) m = fma(amut, c.gprt, m);
    m *= recip(d);
  }
  Lvi = m * g[G_VI2 * F];
  Lvj = m * g[G_VJ2 * F];
}

// flux differences (sub_Residual.f90:460-468), comput_Lvc (sub_NS_singlegrid.f90:352-388)
// and comput_dt (sub_NS_singlegrid.f90:324-348) for interior cells
// NORM: also the tile's partial norms of Res (the work of k_norm_partial,
// same cells, same reduction tree, so the norms are bit-identical); only when
// no later kernel of the residual stage changes Res (no FDM patch, no
// dual-time term)
// post: RES_ADD_FORCE (Res += QF once the norms are taken), RES_FORCE_FN
// (QF -= Res), RES_SET_UN (Un = U over 0..nx, 0..ny): the multigrid steps
// that follow a residual evaluation, done in the same pass
template <bool M, bool NORM, bool FINAL>
__global__ void __launch_bounds__(TILE) k_res(Lvl L, int post) {
  int bk, i, j;
  bool act = core_ij(L, bk, i, j);
  if (act) {
    const BlkDev &b0 = L.blk[bk];
    if ((post & RES_SET_UN) && i >= 0 && i <= b0.nx && j >= 0 && j <= b0.ny) {
      const long long id = fidx(b0, i, j);
#pragma unroll
      for (int m = 0; m < 4; m++) L.un[m * L.F + id] = L.U[m * L.F + id];
    }
    act = i >= 1 && i <= b0.nx - 1 && j >= 1 && j <= b0.ny - 1;
  }
  if (!NORM && !act) return;
  double vres[6] = {0, 0, 0, 0, 0, 0};
  if (act) {
    const BlkDev &b = L.blk[bk];
    const CaseDev &c = L.cs[b.cas];
    const long long F = L.F, P = b.P;
    long long id = fidx(b, i, j);
    bool fdm = b.fdm && (i >= LFDM + 1 && i <= b.nx - LFDM - 1) && (j >= LFDM + 1 && j <= b.ny - LFDM - 1);
    if (!fdm) {
#pragma unroll
      for (int m = 0; m < 4; m++) {
        double r = L.fi[m * F + id + 1] - L.fi[m * F + id] + L.fj[m * F + id + P] - L.fj[m * F + id];
        vres[m] = r;
        if (post & (RES_ADD_FORCE | RES_FORCE_FN)) {
          const double qf = L.qf[m * F + id];
          if (post & RES_FORCE_FN) L.qf[m * F + id] = qf - r;
          if (post & RES_ADD_FORCE) r = r + qf;
        }
        L.res[m * F + id] = r;
      }
    }
    if (NORM)
#pragma unroll
      for (int m = 4; m < 6; m++)
        if (m < L.nvar) vres[m] = L.res[m * F + id];  // constant indices: vres stays in registers
    const double *g = L.geo + id;
    const double s0 = g[G_VOL * F];
    const double si = g[G_SIA * F], ni1 = g[G_NI1A * F], ni2 = g[G_NI2A * F];
    const double sj = g[G_SJA * F], nj1 = g[G_NJ1A * F], nj2 = g[G_NJ2A * F];
    double uu = L.q[Q_U * F + id], vv = L.q[Q_V * F + id], cc = L.q[Q_C * F + id], d = L.q[Q_D * F + id];
    double uni = uu * ni1 + vv * ni2, unj = uu * nj1 + vv * nj2;
    double Lci = (fabs(uni) + cc) * si, Lcj = (fabs(unj) + cc) * sj;
    double Lvi = 0.0, Lvj = 0.0;
    if (L.visc) {
      const bool eddy = L.turb != Turb_NONE || L.keep_amut;
      viscous_radii<M>(c, g, F, d, L.amu[id], eddy, eddy ? L.amut[id] : 0.0, Lvi, Lvj);
    }
    L.lc[L_CI * F + id] = Lci;
    L.lc[L_CJ * F + id] = Lcj;
    L.lc[L_VI * F + id] = Lvi;
    L.lc[L_VJ * F + id] = Lvj;
    double dt;
    if (c.local_dt == 0) dt = c.dt_global;
    else {
      double sum = Lci + Lcj;
      if (L.visc) sum += Lvi + Lvj;
      dt = c.CFL * s0 * (M ? rcp(sum) : recip(sum));
      if (above(dt, c.dtmax)) dt = c.dtmax;
      if (below(dt, c.dtmin)) dt = c.dtmin;
    }
    L.lc[L_DT * F + id] = dt;
  }
  if (NORM) {
    tile_partials(L, act, vres);
    if (FINAL) {
      // the last CTA to finish reduces every tile's partials (few cases)
      __shared__ int last;
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) last = atomicAdd(L.nctr, 1u) == gridDim.x - 1;
      __syncthreads();
      if (last) {
        __threadfence();
        const int w = threadIdx.x >> 5;
        for (int k = w; k < L.ncase * 12; k += TILE / 32) final_norm(L, k / 12, k % 12);
        if (threadIdx.x == 0) *L.nctr = 0u;
      }
    }
  }
}

// ---- the residual of a level in one kernel --------------------------------
// k_residual_tile does the work of k_prim, k_flux_i, k_flux_j and k_res for a
// 2-D tile of RTX x RTY cells: the primitives (and Sutherland mu) of the tile
// and its two-cell halo go into shared memory, every i- and j-face of the
// tile's cells is reconstructed and fluxed from there (the faces on the
// tile's edges are evaluated by both tiles that share them), and each thread
// forms its cell's residual, spectral radii, time step and norm partials.
// Nothing but U, the geometry and the outputs touches HBM, and one launch
// replaces four.  It serves levels without a turbulence model or a
// finite-difference patch, in FP64; the face, reconstruction and viscous
// arithmetic is the same code as the chain's.
constexpr int RTX = RES_TILE_X, RTY = RES_TILE_Y;  // cells per tile
constexpr int RGX = RTX + 4, RGY = RTY + 4;        // tile + two halo cells on each side
constexpr int RGN = RGX * RGY;
constexpr int RNT = RES_TILE_THREADS;
// one thread per face of the tile, per halo cell and per cell: every FP64
// chain of a phase runs side by side (on the small multigrid levels the
// kernel is as long as one thread's chain)
static_assert((RTX + 1) * RTY + RTX * (RTY + 1) <= RNT && RGN <= RNT && RTX * RTY <= RNT, "a thread per item");

template <bool M, bool NORM, bool FINAL>
__global__ void __launch_bounds__(RNT) k_residual_tile(Lvl L, const int4 *rt, int post) {
  __shared__ double sd[RGN], su[RGN], sv[RGN], sp[RGN], sT[RGN], sc[RGN], smu[RGN];
  __shared__ double sU[4][RGN];
  __shared__ double fi[4][RTY][RTX + 1], fj[4][RTY + 1][RTX];
  const int4 t4 = rt[blockIdx.x];
  const int bk = t4.x, i0 = t4.y, j0 = t4.z;
  const BlkDev &b = L.blk[bk];
  const CaseDev &c = L.cs[b.cas];
  const long long F = L.F;
  const int nx = b.nx, ny = b.ny;
  const int i1 = min(i0 + RTX - 1, nx - 1), j1 = min(j0 + RTY - 1, ny - 1);  // last cells of the tile
  auto R = [&](int i, int j) { return (j - j0 + 2) * RGX + (i - i0 + 2); };
  // (1) primitives over the tile and its halo (comput_duvtpckw + get_viscous,
  // as k_prim), within the block's extended range -1..nx+1 x -1..ny+1
  for (int t = threadIdx.x; t < RGN; t += RNT) {
    const int i = i0 - 2 + t % RGX, j = j0 - 2 + t / RGX;
    if (i < -1 || i > nx + 1 || j < -1 || j > ny + 1) continue;
    const long long id = fidx(b, i, j);
    const double d = L.U[id], ru = L.U[F + id], rv = L.U[2 * F + id], E = L.U[3 * F + id];
    const Prim w = primitives<M>(c, d, ru, rv, E);
    sd[t] = d; su[t] = w.u; sv[t] = w.v; sT[t] = w.T; sp[t] = w.p;
    sc[t] = w.sT * c.rMa;
    sU[0][t] = d; sU[1][t] = ru; sU[2][t] = rv; sU[3][t] = E;
    const bool own = i >= i0 && i <= i1 && j >= j0 && j <= j1;
    if (own && !at_least(w.T, 1.0e-5)) set_status(L.status + 4 * b.cas, 3, bk, i, j);
    if (L.visc) {
      const double mu = sutherland<M>(c, w);
      smu[t] = mu;
      // Amu over 0..nx x 0..ny as k_prim leaves it: the tile's cells, and the
      // block's ghost lines next to them when the tile is on the block's edge
      const bool wi = (i >= i0 && i <= i1) || (i == 0 && i0 == 1) || (i == nx && i1 == nx - 1);
      const bool wj = (j >= j0 && j <= j1) || (j == 0 && j0 == 1) || (j == ny && j1 == ny - 1);
      if (wi && wj) { L.amu[id] = mu; L.amut[id] = 0.0; }
    }
  }
  __syncthreads();
  // (2) faces: i-faces i0..i1+1 of rows j0..j1, j-faces j0..j1+1 of columns i0..i1
  const int nfi = (i1 - i0 + 2) * (j1 - j0 + 1), nfj = (i1 - i0 + 1) * (j1 - j0 + 2);
  for (int t = threadIdx.x; t < nfi + nfj; t += RNT) {
    const bool ifc = t < nfi;
    int i, j;
    if (ifc) { i = i0 + t % (i1 - i0 + 2); j = j0 + t / (i1 - i0 + 2); }
    else { const int u = t - nfi; i = i0 + u % (i1 - i0 + 1); j = j0 + u / (i1 - i0 + 1); }
    const long long id = fidx(b, i, j);
    const int r = R(i, j), st = ifc ? 1 : RGX;  // stencil stride in the tile's shared arrays
    const double s = L.geo[(ifc ? G_SI : G_SJ) * F + id];
    const double n1 = L.geo[(ifc ? G_NI1 : G_NJ1) * F + id], n2 = L.geo[(ifc ? G_NI2 : G_NJ2) * F + id];
    double S0[4][4];
    int scheme = L.scheme;
    if (L.recon == Recon_Original) {
      if (!ifc) scheme = L.gscheme;  // the global Iflag_Scheme in the j direction (sub_Residual.f90:367)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int q = r + (k - 2) * st;
        S0[k][0] = sd[q]; S0[k][1] = su[q]; S0[k][2] = sv[q]; S0[k][3] = sp[q];
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++)
#pragma unroll
        for (int m = 0; m < 4; m++) S0[k][m] = sU[m][r + (k - 2) * st];
    }
    double Fl[4];
    inviscid<M>(L, c, scheme, S0, n1, n2, s, Fl);
    if (L.visc) {
      auto u = [&](long long k) { return su[k]; };
      auto v = [&](long long k) { return sv[k]; };
      auto t = [&](long long k) { return sT[k]; };
      const FaceDiff<double> D = face_diff<M, double>(r, st, ifc ? RGX : 1, u, v, t);
      const double ml = smu[r - st], mr = smu[r], *g = L.geo + id;
      if (ifc) viscous<M, true>(c, g + G_VIP * F, F, D, ml, mr, false, 0.0, 0.0, i == 1, i == nx, n1, n2, s, Fl);
      else viscous<M, false>(c, g + G_VJP * F, F, D, ml, mr, false, 0.0, 0.0, j == 1, j == ny, n1, n2, s, Fl);
    }
#pragma unroll
    for (int m = 0; m < 4; m++) (ifc ? fi[m][j - j0][i - i0] : fj[m][j - j0][i - i0]) = Fl[m];
  }
  __syncthreads();
  // (3) the cell of this thread: flux differences, radii, time step (k_res)
  const int tx = threadIdx.x % RTX, ty = threadIdx.x / RTX;
  const int i = i0 + tx, j = j0 + ty;
  const bool act = threadIdx.x < RTX * RTY && i <= i1 && j <= j1;
  if (post & RES_SET_UN) {
    // Un = U over 0..nx x 0..ny: the tile's cells and the ghost lines at
    // the block's edges next to them
    for (int t = threadIdx.x; t < RGN; t += RNT) {
      const int ii = i0 - 2 + t % RGX, jj = j0 - 2 + t / RGX;
      const bool wi = (ii >= i0 && ii <= i1) || (ii == 0 && i0 == 1) || (ii == nx && i1 == nx - 1);
      const bool wj = (jj >= j0 && jj <= j1) || (jj == 0 && j0 == 1) || (jj == ny && j1 == ny - 1);
      if (wi && wj) {
        const long long id = fidx(b, ii, jj);
#pragma unroll
        for (int m = 0; m < 4; m++) L.un[m * F + id] = sU[m][t];
      }
    }
  }
  double vres[6] = {0, 0, 0, 0, 0, 0};
  if (act) {
    const long long id = fidx(b, i, j);
    const int r = R(i, j);
#pragma unroll
    for (int m = 0; m < 4; m++) {
      double rr = fi[m][ty][tx + 1] - fi[m][ty][tx] + fj[m][ty + 1][tx] - fj[m][ty][tx];
      vres[m] = rr;
      if (post & (RES_ADD_FORCE | RES_FORCE_FN)) {
        const double qf = L.qf[m * F + id];
        if (post & RES_FORCE_FN) L.qf[m * F + id] = qf - rr;
        if (post & RES_ADD_FORCE) rr = rr + qf;
      }
      L.res[m * F + id] = rr;
    }
    const double *g = L.geo + id;
    const double s0 = g[G_VOL * F];
    const double si = g[G_SIA * F], ni1 = g[G_NI1A * F], ni2 = g[G_NI2A * F];
    const double sj = g[G_SJA * F], nj1 = g[G_NJ1A * F], nj2 = g[G_NJ2A * F];
    const double uu = su[r], vv = sv[r], cc = sc[r], d = sd[r];
    const double uni = uu * ni1 + vv * ni2, unj = uu * nj1 + vv * nj2;
    const double Lci = (fabs(uni) + cc) * si, Lcj = (fabs(unj) + cc) * sj;
    double Lvi = 0.0, Lvj = 0.0;
    if (L.visc) viscous_radii<M>(c, g, F, d, smu[r], false, 0.0, Lvi, Lvj);
    L.lc[L_CI * F + id] = Lci;
    L.lc[L_CJ * F + id] = Lcj;
    L.lc[L_VI * F + id] = Lvi;
    L.lc[L_VJ * F + id] = Lvj;
    double dt;
    if (c.local_dt == 0) dt = c.dt_global;
    else {
      double sum = Lci + Lcj;
      if (L.visc) sum += Lvi + Lvj;
      dt = c.CFL * s0 * (M ? rcp(sum) : recip(sum));
      if (above(dt, c.dtmax)) dt = c.dtmax;
      if (below(dt, c.dtmin)) dt = c.dtmin;
    }
    L.lc[L_DT * F + id] = dt;
  }
  if (NORM) {
    tile_partials<RNT>(L, act, vres);
    if (FINAL) {
      __shared__ int last;
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) last = atomicAdd(L.nctr, 1u) == gridDim.x - 1;
      __syncthreads();
      if (last) {
        __threadfence();
        const int w = threadIdx.x >> 5;
        for (int k = w; k < L.ncase * 12; k += RNT / 32) final_norm(L, k / 12, k % 12);
        if (threadIdx.x == 0) *L.nctr = 0u;
      }
    }
  }
}

// per-tile partial norms of Res (max |Res| and sum Res^2 per variable)
__global__ void __launch_bounds__(TILE) k_norm_partial(Lvl L) {
  int bk, i, j;
  double vres[6] = {0, 0, 0, 0, 0, 0};
  bool act = false;
  if (core_ij(L, bk, i, j)) {
    const BlkDev &b = L.blk[bk];
    if (i >= 1 && i <= b.nx - 1 && j >= 1 && j <= b.ny - 1) {
      act = true;
      long long id = fidx(b, i, j);
#pragma unroll
      for (int m = 0; m < 6; m++)
        if (m < L.nvar) vres[m] = L.res[m * L.F + id];
    }
  }
  tile_partials(L, act, vres);
}

// per-case reduction of the tile partials, one CTA per case and quantity: a thread
// takes one of the 128 partial results that a warp of final_norm keeps, in the same order
__global__ void __launch_bounds__(128) k_norm_final(Lvl L) {
  __shared__ double acc[128];
  const int cs = blockIdx.x / 12, m = blockIdx.x % 12, nt = L.case_ntile[cs];
  const double *p = L.npart + (size_t)L.case_tile0[cs] * 12 + m;
  if (m < 6) {
    long long a = 0;
#pragma unroll 8
    for (int t = threadIdx.x; t < nt; t += 128) a = max(a, __double_as_longlong(p[(size_t)t * 12]));
    acc[threadIdx.x] = __longlong_as_double(a);
  } else {
    double q = 0.0;
#pragma unroll 8
    for (int t = threadIdx.x; t < nt; t += 128) q += p[(size_t)t * 12];
    acc[threadIdx.x] = q;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const double *r = acc + threadIdx.x;
  double out;
  if (m < 6) {
    long long b = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) b = max(b, __double_as_longlong(r[32 * k]));
    out = __longlong_as_double(warp_max_bits(b));
  } else {
    const double s = warp_sum((r[0] + r[32]) + (r[64] + r[96]));
    out = (m - 6 < L.nvar) ? sqrt(s / (1.0 * L.case_ncell[cs])) : 0.0;
  }
  if (threadIdx.x == 0) L.norms[cs * 12 + m] = out;
}

// set-up, and when a context gets or loses its FP32 parts: the viscous metric
// coefficients (G_VIP..G_VJS) of the i-faces (i = 1..nx, j =
// 1..ny-1) and j-faces (i = 1..nx-1, j = 1..ny) from the cell centres, with the
// stencils of Residual_FVM (sub_Residual.f90:313-330, 419-436), and the cell
// metric factors of the spectral radii
__global__ void __launch_bounds__(TILE) k_face_metrics(Lvl L) {
  int bk, i, j;
  if (!tile_ij(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  const long long F = L.F, P = b.P, id = fidx(b, i, j);
  const double *x1 = L.geo + G_X1 * F, *y1 = L.geo + G_Y1 * F;
  double *g = L.geo + id;
  // fi, fj: the factors of the differences in i and j (1/4 of those along the face)
  auto put = [&](int to, int nrm, double A, double B, double C, double D, double fi, double fj) {
    const double n1 = g[nrm * F], n2 = g[(nrm + 1) * F];
    g[to * F] = L.mixed ? A : fi * (A * n1 - C * n2);
    g[(to + 1) * F] = L.mixed ? B : fj * (D * n2 - B * n1);
    g[(to + 2) * F] = L.mixed ? C : fi * (A * n2 + C * n1);
    g[(to + 3) * F] = L.mixed ? D : fj * (B * n2 + D * n1);
  };
  if (i >= 1 && i <= b.nx && j >= 1 && j <= b.ny - 1) {
    const long long w = id - 1, nN = id + P, nS = id - P;
    const double Dix = x1[id] - x1[w], Diy = y1[id] - y1[w];
    const double Djx = (x1[nN - 1] + x1[nN] - x1[nS - 1] - x1[nS]) * 0.25;
    const double Djy = (y1[nN - 1] + y1[nN] - y1[nS - 1] - y1[nS]) * 0.25;
    const double Ds = 1.0 / (Dix * Djy - Djx * Diy);
    const double A = Djy * Ds, B = Diy * Ds, C = Djx * Ds, D = Dix * Ds;
    put(G_VIP, G_NI1, A, B, C, D, 1.0, 0.25);
  }
  if (i >= 1 && i <= b.nx - 1 && j >= 1 && j <= b.ny) {
    const long long s = id - P;
    const double Dix = (x1[s + 1] + x1[id + 1] - x1[s - 1] - x1[id - 1]) * 0.25;
    const double Diy = (y1[s + 1] + y1[id + 1] - y1[s - 1] - y1[id - 1]) * 0.25;
    const double Djx = x1[id] - x1[s], Djy = y1[id] - y1[s];
    const double Ds = 1.0 / (Dix * Djy - Djx * Diy);
    const double A = Djy * Ds, B = Diy * Ds, C = Djx * Ds, D = Dix * Ds;
    put(G_VJP, G_NJ1, A, B, C, D, 0.25, 1.0);
  }
  if (i >= 1 && i <= b.nx - 1 && j >= 1 && j <= b.ny - 1) {
    // comput_Lvc (sub_NS_singlegrid.f90:352-388): face metrics averaged over
    // the cell's two faces of each family
    const double *gg = L.geo;
    const double si = 0.5 * (gg[G_SI * F + id] + gg[G_SI * F + id + 1]);
    const double sj = 0.5 * (gg[G_SJ * F + id] + gg[G_SJ * F + id + P]);
    const double rs0 = 1.0 / gg[G_VOL * F + id];
    g[G_SIA * F] = si;
    g[G_NI1A * F] = 0.5 * (gg[G_NI1 * F + id] + gg[G_NI1 * F + id + 1]);
    g[G_NI2A * F] = 0.5 * (gg[G_NI2 * F + id] + gg[G_NI2 * F + id + 1]);
    g[G_SJA * F] = sj;
    g[G_NJ1A * F] = 0.5 * (gg[G_NJ1 * F + id] + gg[G_NJ1 * F + id + P]);
    g[G_NJ2A * F] = 0.5 * (gg[G_NJ2 * F + id] + gg[G_NJ2 * F + id + P]);
    g[G_VI2 * F] = si * si * rs0;
    g[G_VJ2 * F] = sj * sj * rs0;
  }
}
void launch_face_metrics(const Lvl &L, cudaStream_t s) { k_face_metrics<<<L.ntiles, TILE, 0, s>>>(L); }

// f(std::integral_constant<bool, M>): with the level's kind of arithmetic
template <typename Fn>
static void by_kind(const Lvl &L, Fn f) {
  if (L.mixed) f(std::true_type());
  else f(std::false_type());
}
void launch_prim(const Lvl &L, cudaStream_t s) {
  by_kind(L, [&](auto M) { k_prim<M.value><<<L.ntiles, TILE, 0, s>>>(L); });
}
// A level takes the slopes pass if its faces are MUSCL3 on the primitives and in FP64: from
// 262,144 cells, in contexts with FP32 parts from 65,536, whose faces save twice as much.  2 x 1024 x 512 cells in FP64: slopes 195 us, faces 2 x 217 (205
// since), the RK3 step 2.26 -> 2.07 ms; with the pass everywhere a RANS step of 66 k cells
// is 1 % slower, a V-cycle of 18 k cells 0.7 %, 16 k cells of an airfoil 0.9 %.  With FP32 sweeps
// an SA residual of 131 k cells 271 -> 254 us, of 66 k 162 -> 158, of 33 k 105 -> 103, of
// 16 k 74.2 -> 74.9; a V-cycle of 18 k cells 0.4 % slower.
int slope_level(const Lvl &L, long long cells) {
  if (L.recon != Recon_Original || L.scheme != Scheme_MUSCL3 || L.gscheme != Scheme_MUSCL3) return 0;
  return cells >= SLOPE_CELLS ? 2 : cells >= SLOPE_CELLS_MIXED ? 1 : 0;
}
bool takes_slopes(const Lvl &L) { return L.slopes == 2 || (L.slopes == 1 && L.mixed); }
void launch_slopes(const Lvl &L, int dirs, cudaStream_t s) {
  by_kind(L, [&](auto M) { k_slopes<M.value><<<L.nctiles, TILE, 0, s>>>(L, dirs); });
}
template <bool IFACE>
static void launch_flux(const Lvl &L, bool fp32, cudaStream_t s) {
  if (fp32) k_flux<true, IFACE, false, float><<<L.nctiles, TILE, 0, s>>>(L);
  else if (takes_slopes(L)) by_kind(L, [&](auto M) { k_flux<M.value, IFACE, true, double><<<L.nctiles, TILE, 0, s>>>(L); });
  else by_kind(L, [&](auto M) { k_flux<M.value, IFACE, false, double><<<L.nctiles, TILE, 0, s>>>(L); });
}
void launch_flux_i(const Lvl &L, bool fp32, cudaStream_t s) { launch_flux<true>(L, fp32, s); }
void launch_flux_j(const Lvl &L, bool fp32, cudaStream_t s) { launch_flux<false>(L, fp32, s); }
// with_norms: the tile partials inside k_res; with few cases of few tiles the last CTA of
// k_res also forms the per-case norms (norms_fused_final() tells the caller).  A warp of
// that CTA takes three quantities of a case, a round of loads per 128 tiles each, while the rest
// of the chip stands idle: 2 us at 144 tiles, 70 us at the 8242 tiles of 1.05 M cells, where
// a CTA per quantity (k_norm_final) takes 5 us; they cross near 1000 tiles.
bool norms_fused_final(const Lvl &L) { return L.ncase <= 8 && L.nctiles <= 1024; }
void launch_res(const Lvl &L, bool with_norms, int post, cudaStream_t s) {
  by_kind(L, [&](auto M) {
    if (!with_norms) k_res<M.value, false, false><<<L.nctiles, TILE, 0, s>>>(L, post);
    else if (norms_fused_final(L)) k_res<M.value, true, true><<<L.nctiles, TILE, 0, s>>>(L, post);
    else k_res<M.value, true, false><<<L.nctiles, TILE, 0, s>>>(L, post);
  });
}
// Lr: the level with npart, case_tile0, case_ntile and nctr of the 2-D tile list
void launch_residual_tile(const Lvl &Lr, const int4 *rt, int ntiles, bool with_norms, int post, cudaStream_t s) {
  by_kind(Lr, [&](auto M) {
    if (!with_norms) k_residual_tile<M.value, false, false><<<ntiles, RNT, 0, s>>>(Lr, rt, post);
    else if (norms_fused_final(Lr)) k_residual_tile<M.value, true, true><<<ntiles, RNT, 0, s>>>(Lr, rt, post);
    else k_residual_tile<M.value, true, false><<<ntiles, RNT, 0, s>>>(Lr, rt, post);
  });
}
void launch_norms(const Lvl &L, bool partials, cudaStream_t s) {
  if (partials) k_norm_partial<<<L.nctiles, TILE, 0, s>>>(L);
  k_norm_final<<<L.ncase * 12, 128, 0, s>>>(L);
}

}  // namespace ec2d
