// ec2d_mixed.cuh -- the face physics of contexts with FP32 parts (FP32 LU-SGS
// sweeps, FP32 faces of the coarse levels).
//
// Where a residual is rounded to FP32, a difference in its last FP64 bit can move the
// rounded value by 2^-24: single cells' increments change by 6e-8 and the
// largest residual after a few cycles by up to 6e-8 (measured on a batched polar
// and a three-level flat plate, in one start in three by more than 1e-9).  So that the results of
// mixed-precision runs stay what they were, bit for bit, these contexts keep the order of
// operations of the formulas written out, and FP64 contexts use the
// shorter one of ec2d_dev.cuh.  Both are compared with the oracle to the same
// bounds.  A viscous AUSM+ face takes 273 FP64 instructions (298 with every power of two
// on the FP64 pipe; 343 -> 322 us per direction of a batched polar) against 166 there.
#pragma once
#include "ec2d_dev.cuh"

namespace ec2d {
namespace mixed {

// The face physics below is written once for the arithmetic type T: double
// is the reference's arithmetic (every literal T(x) is then the same double
// constant), float serves the FP32 coarse multigrid levels.

// x 2^K and comparisons, in FP64 on the integer pipes: only where that leaves the compiler's
// choice of the product that it fuses with a sum as it was (residuals compared bit for bit;
// the split Mach numbers and Roe's 0.5 / a^2 are not among them).
template <int K>
__device__ __forceinline__ double scaled(double x) { return pow2<K>(x); }
template <int K>
__device__ __forceinline__ float scaled(float x) { return x * (K >= 0 ? (float)(1 << (K & 31)) : 1.0f / (float)(1 << (-K & 31))); }
__device__ __forceinline__ bool less(double x, double y) { return below(x, y); }  // y of clear sign bit
__device__ __forceinline__ bool less(float x, float y) { return x < y; }
__device__ __forceinline__ bool outside_one(double m) { return at_least(fabs(m), 1.0); }  // |m| >= 1
__device__ __forceinline__ bool outside_one(float m) { return fabsf(m) >= 1.0f; }
__device__ __forceinline__ bool not_negative(double x) { return at_least(x, 0.0) || __double_as_longlong(x) << 1 == 0; }
__device__ __forceinline__ bool not_negative(float x) { return x >= 0.0f; }
__device__ __forceinline__ double max0(double x) { return above(x, 0.0) ? x : 0.0; }  // fmax(0, x)
__device__ __forceinline__ float max0(float x) { return fmaxf(0.0f, x); }
__device__ __forceinline__ double min0(double x) { return above(neg(x), 0.0) ? x : 0.0; }
__device__ __forceinline__ float min0(float x) { return fminf(0.0f, x); }

// ---- reconstruction, sub_Residual.f90:477-659 --------------------------------
template <typename T>
__device__ __forceinline__ T minmod(T a, T b) {
  if (a * b <= T(0.0)) return T(0.0);
  return (fabs(a) <= fabs(b)) ? a : b;
}

// scheme_fP (sub_Residual.f90:591-623): left state at the face between u2 and u3
template <typename T>
__device__ __forceinline__ T scheme_fp(T u1, T u2, T u3, T u4, int flag) {
  const T ep = T(1.0e-6), k3 = T(1.0) / T(3.0);
  switch (flag) {
    case Scheme_UD1: return u2;
    case Scheme_UD3: return (-u1 + T(5.0) * u2 + T(2.0) * u3) / T(6.0);
    case Scheme_NND2: return u2 + T(0.5) * minmod(u2 - u1, u3 - u2);
    case Scheme_WENO3: {
      T IS1 = (u2 - u1) * (u2 - u1), IS2 = (u3 - u2) * (u3 - u2);
      T e1 = T(1.0e-6) + IS1, e2 = T(1.0e-6) + IS2;
      T a1 = T(1.0) / (T(3.0) * (e1 * e1)), a2 = T(2.0) / (T(3.0) * (e2 * e2));
      T w1 = a1 / (a1 + a2), w2 = a2 / (a1 + a2);
      return w1 * (-u1 / T(2.0) + T(3.0) * u2 / T(2.0)) + w2 * (u2 / T(2.0) + u3 / T(2.0));
    }
    case Scheme_MUSCL2:  // k=1, b=2
      return u2 + T(0.25) * ((T(1.0) - T(1.0)) * minmod(u2 - u1, T(2.0) * (u3 - u2)) + (T(1.0) + T(1.0)) * minmod(u3 - u2, T(2.0) * (u2 - u1)));
    case Scheme_MUSCL3: {
      T up = u3 - u2, um = u2 - u1;
      T s = (scaled<1>(up) * um + ep) * rcp(up * up + um * um + ep);
      return u2 + scaled<-2>(s) * ((T(1.0) - k3 * s) * um + (T(1.0) + k3 * s) * up);
    }
    case Scheme_OMUSCL2: {
      T r1 = (u2 - u1 + ep) / (u3 - u2 + ep), r2 = (u3 - u2 + ep) / (u4 - u3 + ep);
      T f1 = T(0.8) - T(0.175) / r2 + T(0.375) * r1;
      T f = fmax(T(0.0), fmin(fmin(T(2.0), f1), T(2.0) * r1));
      return u2 + T(0.5) * f * (u3 - u2);
    }
  }
  return T(0.0);
}
// scheme_fm (sub_Residual.f90:626-659): right state at the face between u2 and u3
template <typename T>
__device__ __forceinline__ T scheme_fm(T u1, T u2, T u3, T u4, int flag) {
  const T ep = T(1.0e-6), k3 = T(1.0) / T(3.0);
  switch (flag) {
    case Scheme_UD1: return u3;
    case Scheme_UD3: return (T(2.0) * u2 + T(5.0) * u3 - u4) / T(6.0);
    case Scheme_NND2: return u3 - T(0.5) * minmod(u3 - u2, u4 - u3);
    case Scheme_WENO3: {
      T IS1 = (u3 - u4) * (u3 - u4), IS2 = (u2 - u3) * (u2 - u3);
      T e1 = T(1.0e-6) + IS1, e2 = T(1.0e-6) + IS2;
      T a1 = T(1.0) / (T(3.0) * (e1 * e1)), a2 = T(2.0) / (T(3.0) * (e2 * e2));
      T w1 = a1 / (a1 + a2), w2 = a2 / (a1 + a2);
      return w1 * (-u4 / T(2.0) + T(3.0) * u3 / T(2.0)) + w2 * (u3 / T(2.0) + u2 / T(2.0));
    }
    case Scheme_MUSCL2: {  // k=1/3, b=1
      const T k = T(1.0) / T(3.0);
      return u3 - T(0.25) * ((T(1.0) - k) * minmod(u4 - u3, (u3 - u2)) + (T(1.0) + k) * minmod(u3 - u2, (u4 - u3)));
    }
    case Scheme_MUSCL3: {
      T up = u4 - u3, um = u3 - u2;
      T s = (scaled<1>(up) * um + ep) * rcp(up * up + um * um + ep);
      return u3 - scaled<-2>(s) * ((T(1.0) - k3 * s) * up + (T(1.0) + k3 * s) * um);
    }
    case Scheme_OMUSCL2: {
      T r1 = (u4 - u3 + ep) / (u3 - u2 + ep), r2 = (u3 - u2 + ep) / (u2 - u1 + ep);
      T f1 = T(0.8) - T(0.175) / r2 + T(0.375) * r1;
      T f = fmax(T(0.0), fmin(fmin(T(2.0), f1), T(2.0) * r1));
      return u3 - T(0.5) * f * (u3 - u2);
    }
  }
  return T(0.0);
}

// MUSCL3 states of cell u2 towards its upper and its lower face, the bits of scheme_fp and
// scheme_fm there: the fused products are written out as the compiler chooses them in those
__device__ __forceinline__ void muscl3_states(double u1, double u2, double u3, double &hi, double &lo) {
  const double ep = 1.0e-6, k3 = 1.0 / 3.0;
  const double up = u3 - u2, um = u2 - u1;
  const double s = fma(scaled<1>(up), um, ep) * rcp(fma(um, um, up * up) + ep);
  const double q = scaled<-2>(s), a = fma(-k3, s, 1.0), b = fma(k3, s, 1.0);
  hi = fma(q, fma(a, um, b * up), u2);
  lo = fma(-q, fma(a, up, b * um), u2);
}

// conservative (rho, rho u, rho v, E) -> primitive (rho, u, v, p), as at the
// end of Reconstuction_conservative/Characteristic (sub_Residual.f90:526-527)
template <typename T>
__device__ __forceinline__ void cons_to_prim(const T Q[4], T W[4], T gm1) {
  W[0] = Q[0];
  W[1] = Q[1] / W[0];
  W[2] = Q[2] / W[0];
  W[3] = (Q[3] - (W[1] * Q[1] + W[2] * Q[2]) * T(0.5)) * gm1;
}

// S0[k][m]: stencil points k = i-2..i+1 (or j-2..j+1), variable m.
// Reconstuction_original/conservative/Characteristic (sub_Residual.f90:505-586)
template <typename T>
__device__ __forceinline__ void reconstruct(int recon, int scheme, T S0[4][4], T gamma,
                                            T UL[4], T UR[4]) {
  if (recon == Recon_Original) {
#pragma unroll
    for (int m = 0; m < 4; m++) {
      UL[m] = scheme_fp(S0[0][m], S0[1][m], S0[2][m], S0[3][m], scheme);
      UR[m] = scheme_fm(S0[0][m], S0[1][m], S0[2][m], S0[3][m], scheme);
    }
    return;
  }
  T gm1 = gamma - T(1.0);
  if (recon == Recon_Conservative) {
    T QL[4], QR[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      QL[m] = scheme_fp(S0[0][m], S0[1][m], S0[2][m], S0[3][m], scheme);
      QR[m] = scheme_fm(S0[0][m], S0[1][m], S0[2][m], S0[3][m], scheme);
    }
    cons_to_prim(QL, UL, gm1);
    cons_to_prim(QR, UR, gm1);
    return;
  }
  // characteristic: project on the left eigenvectors at the arithmetic
  // mid-state, limit each characteristic variable, project back
  T Uh[4];
#pragma unroll
  for (int m = 0; m < 4; m++) Uh[m] = T(0.5) * (S0[1][m] + S0[2][m]);
  T d1 = Uh[0], u1 = Uh[1] / d1, v1 = Uh[2] / d1;
  T p1 = (Uh[3] - (Uh[1] * u1 + Uh[2] * v1) * T(0.5)) * gm1;
  T c1 = sqrt(gamma * p1 / d1);
  T V2 = (u1 * u1 + v1 * v1) * T(0.5);
  T tmp1 = gm1 / c1, tmp3 = gm1 / (c1 * c1), tmp5 = T(1.0) / (T(2.0) * c1), tmp0 = T(1.0) / tmp3;
  const T Sm[4][4] = {{V2 - tmp0, -u1, -v1, T(1.0)},
                           {-v1, T(0.0), T(1.0), T(0.0)},
                           {-u1 - V2 * tmp1, T(1.0) + tmp1 * u1, tmp1 * v1, -tmp1},
                           {-u1 + V2 * tmp1, T(1.0) - tmp1 * u1, -tmp1 * v1, tmp1}};
  T V0[4][4];
#pragma unroll
  for (int k = 0; k < 4; k++)
#pragma unroll
    for (int m = 0; m < 4; m++)
      V0[k][m] = Sm[m][0] * S0[k][0] + Sm[m][1] * S0[k][1] + Sm[m][2] * S0[k][2] + Sm[m][3] * S0[k][3];
  T VL[4], VR[4];
#pragma unroll
  for (int m = 0; m < 4; m++) {
    VL[m] = scheme_fp(V0[0][m], V0[1][m], V0[2][m], V0[3][m], scheme);
    VR[m] = scheme_fm(V0[0][m], V0[1][m], V0[2][m], V0[3][m], scheme);
  }
  const T S1[4][4] = {{-tmp3, T(0.0), -tmp5, tmp5},
                           {-tmp3 * u1, T(0.0), T(0.5) - u1 * tmp5, T(0.5) + u1 * tmp5},
                           {-tmp3 * v1, T(1.0), -v1 * tmp5, v1 * tmp5},
                           {-tmp3 * V2, v1, (c1 * u1 - V2 - tmp0) * tmp5, (c1 * u1 + V2 + tmp0) * tmp5}};
  T QL[4], QR[4];
#pragma unroll
  for (int m = 0; m < 4; m++) {
    QL[m] = S1[m][0] * VL[0] + S1[m][1] * VL[1] + S1[m][2] * VL[2] + S1[m][3] * VL[3];
    QR[m] = S1[m][0] * VR[0] + S1[m][1] * VR[1] + S1[m][2] * VR[2] + S1[m][3] * VR[3];
  }
  cons_to_prim(QL, UL, gm1);
  cons_to_prim(QR, UR, gm1);
}

// ---- 1-D face fluxes on rotated primitive states (rho, u_n, u_t, p) ----------
// Flux_Roe_1D, sub_flux_split.f90:265-324 (Harten entropy fix, delta = 0.1)
template <typename T>
__device__ __forceinline__ void flux_roe(const T *QL, const T *QR, T *F, T gamma, T ggm1) {
  const T delt = T(0.1);
  T dl = QL[0], uul = QL[1], vvl = QL[2], pl = QL[3];
  T dr = QR[0], uur = QR[1], vvr = QR[2], pr = QR[3];
  T gm1 = gamma - T(1.0);
  const T rdl = rcp(dl), rdr = rcp(dr);
  T hl = ggm1 * pl * rdl + T(0.5) * (uul * uul + vvl * vvl);
  T hr = ggm1 * pr * rdr + T(0.5) * (uur * uur + vvr * vvr);
  T Fl0 = dl * uul, Fl1 = dl * uul * uul + pl, Fl2 = dl * uul * vvl, Fl3 = uul * dl * hl;
  T Fr0 = dr * uur, Fr1 = dr * uur * uur + pr, Fr2 = dr * uur * vvr, Fr3 = uur * dr * hr;
  T tmpp = sqrt_p(dr * rdl);
  T inv = rcp(T(1.0) + tmpp);
  T avd = scaled<-2>(dl) * (T(1.0) + tmpp) * (T(1.0) + tmpp);
  T avu = (uul + tmpp * uur) * inv;
  T avv = (vvl + tmpp * vvr) * inv;
  T avh = (hl + tmpp * hr) * inv;
  T ava = sqrt_p(gm1 * (avh - T(0.5) * (avu * avu + avv * avv)));
  T l0 = fabs(avu - ava), l1 = fabs(avu), l3 = fabs(avu + ava);
  const T i2d = T(1.0) / (T(2.0) * delt);
  if (less(l0, delt)) l0 = (l0 * l0 + delt * delt) * i2d;
  if (less(l1, delt)) l1 = (l1 * l1 + delt * delt) * i2d;
  T l2 = l1;
  if (less(l3, delt)) l3 = (l3 * l3 + delt * delt) * i2d;
  T ia = rcp(ava);
  T i2aa = T(0.5) * ia * ia;
  T dp = pr - pl;
  T a0 = (avd * ava * (-uur + uul) + dp) * i2aa;
  T a1 = dr - dl - dp * (ia * ia);
  T a2 = avd * (vvr - vvl) * ia;
  T a3 = (avd * ava * (uur - uul) + dp) * i2aa;
  F[0] = T(0.5) * (Fl0 + Fr0) - T(0.5) * (l0 * a0 + l1 * a1 + l3 * a3);
  F[1] = T(0.5) * (Fl1 + Fr1) - T(0.5) * (l0 * a0 * (avu - ava) + l1 * a1 * avu + l3 * a3 * (avu + ava));
  F[2] = T(0.5) * (Fl2 + Fr2) - T(0.5) * (l0 * a0 * avv + l1 * a1 * avv + l2 * a2 + l3 * a3 * avv);
  F[3] = T(0.5) * (Fl3 + Fr3) - T(0.5) * (l0 * a0 * (avh - avu * ava) + l1 * a1 * T(0.5) * (avu * avu + avv * avv) +
                                    l2 * a2 * avv + l3 * a3 * (avh + avu * ava));
}

// Flux_Ausm_1Da (AUSM+), sub_flux_split.f90:195-261
template <typename T>
__device__ __forceinline__ void flux_ausm(const T *QL, const T *QR, T *F, T gamma, T ggm1) {
  T dl = QL[0], uul = QL[1], vvl = QL[2], pl = QL[3];
  T dr = QR[0], uur = QR[1], vvr = QR[2], pr = QR[3];
  const T rdl = rcp(dl), rdr = rcp(dr);
  const T prl = pl * rdl, prr = pr * rdr;  // p / rho
  T hl = ggm1 * prl + T(0.5) * (uul * uul + vvl * vvl);
  T hr = ggm1 * prr + T(0.5) * (uur * uur + vvr * vvr);
  T al = sqrt_p(gamma * prl), ar = sqrt_p(gamma * prr);
  T a = scaled<-1>(al + ar);
  T ia = rcp(a);
  T Ml = uul * ia, Mr = uur * ia;
  T Mp4, Mm4, Pp5, Pm5;
  T ml2 = Ml * Ml - T(1.0), mr2 = Mr * Mr - T(1.0);
  if (outside_one(Ml)) { Mp4 = T(0.5) * (Ml + fabs(Ml)); Pp5 = T(0.5) * (Ml + fabs(Ml)) / Ml; }
  else { Mp4 = T(0.25) * (Ml + T(1.0)) * (Ml + T(1.0)) + T(0.125) * ml2 * ml2;
         Pp5 = T(0.25) * (Ml + T(1.0)) * (Ml + T(1.0)) * (T(2.0) - Ml) + T(3.0) * Ml * ml2 * ml2 / T(16.0); }
  if (outside_one(Mr)) { Mm4 = T(0.5) * (Mr - fabs(Mr)); Pm5 = T(0.5) * (Mr - fabs(Mr)) / Mr; }
  else { Mm4 = -T(0.25) * (Mr - T(1.0)) * (Mr - T(1.0)) - T(0.125) * mr2 * mr2;
         Pm5 = T(0.25) * (Mr - T(1.0)) * (Mr - T(1.0)) * (T(2.0) + Mr) - T(3.0) * Mr * mr2 * mr2 / T(16.0); }
  T M = Mp4 + Mm4;
  T xm = dl * a * max0(M) + dr * a * min0(M);
  T dm = not_negative(M) ? a * fabs(M) * dl : a * fabs(M) * dr;
  T p = pl * Pp5 + pr * Pm5;
  F[0] = xm;  // 0.5 xm (1 + 1) - 0.5 dm (1 - 1): the same value for finite xm, dm
  const T hx = scaled<-1>(xm), hd = scaled<-1>(dm);
  F[1] = hx * (uul + uur) - hd * (uur - uul) + p;
  F[2] = hx * (vvl + vvr) - hd * (vvr - vvl);
  F[3] = hx * (hl + hr) - hd * (hr - hl);
}

// Flux_Van_Leer_1Da, sub_flux_split.f90:139-189
template <typename T>
__device__ __forceinline__ void flux_vanleer(const T *QL, const T *QR, T *F, T gamma) {
  T dl = QL[0], uul = QL[1], vvl = QL[2], pl = QL[3];
  T dr = QR[0], uur = QR[1], vvr = QR[2], pr = QR[3];
  T gm1 = gamma - T(1.0);
  T al = sqrt(gamma * pl / dl), ar = sqrt(gamma * pr / dr);
  T Ml = uul / al, Mr = uur / ar;
  T fp0 = 0, fp1 = 0, fp2 = 0, fp3 = 0, fm0 = 0, fm1 = 0, fm2 = 0, fm3 = 0;
  if (Ml >= T(1.0)) {
    fp0 = dl * uul; fp1 = dl * uul * uul + pl; fp2 = dl * uul * vvl;
    fp3 = uul * (gamma * pl / gm1 + T(0.5) * dl * (uul * uul + vvl * vvl));
  } else if (fabs(Ml) < T(1.0)) {
    T tmp0 = dl * al * (T(0.25) * (T(1.0) + Ml) * (T(1.0) + Ml));
    T w = gm1 * uul + T(2.0) * al;
    fp0 = tmp0; fp1 = tmp0 * w / gamma; fp2 = tmp0 * vvl;
    fp3 = tmp0 * (w * w * T(0.5) / (gamma * gamma - T(1.0)) + T(0.5) * (vvl * vvl));
  }
  if (Mr >= T(1.0)) {
  } else if (fabs(Mr) < T(1.0)) {
    T tmp0 = dr * ar * (-T(0.25) * (Mr - T(1.0)) * (Mr - T(1.0)));
    T w = gm1 * uur - T(2.0) * ar;
    fm0 = tmp0; fm1 = tmp0 * w / gamma; fm2 = tmp0 * vvr;
    fm3 = tmp0 * (w * w * T(0.5) / (gamma * gamma - T(1.0)) + T(0.5) * (vvr * vvr));
  } else if (Mr <= -T(1.0)) {
    fm0 = dr * uur; fm1 = dr * uur * uur + pr; fm2 = dr * uur * vvr;
    fm3 = uur * (gamma * pr / gm1 + T(0.5) * dr * (uur * uur + vvr * vvr));
  }
  F[0] = fp0 + fm0; F[1] = fp1 + fm1; F[2] = fp2 + fm2; F[3] = fp3 + fm3;
}

// Flux_steger_warming_1Da, sub_flux_split.f90:99-136
template <typename T>
__device__ __forceinline__ void flux_sw(const T *QL, const T *QR, T *F, T gamma) {
  T dl = QL[0], uul = QL[1], vvl = QL[2], pl = QL[3];
  T dr = QR[0], uur = QR[1], vvr = QR[2], pr = QR[3];
  T al = sqrt(gamma * pl / dl), ar = sqrt(gamma * pr / dr);
  T gm1 = gamma - T(1.0);
  T tmp1 = T(2.0) * gm1, tmp3 = (T(3.0) - gamma) / (T(2.0) * gm1);
  T E1P = (uul + fabs(uul)) * T(0.5), E2P = (uul - al + fabs(uul - al)) * T(0.5), E3P = (uul + al + fabs(uul + al)) * T(0.5);
  T t0 = dl / (T(2.0) * gamma);
  T p0 = t0 * (tmp1 * E1P + E2P + E3P);
  T p1 = t0 * (tmp1 * E1P * uul + E2P * (uul - al) + E3P * (uul + al));
  T p2 = t0 * (tmp1 * E1P * vvl + E2P * vvl + E3P * vvl);
  T p3 = t0 * (E1P * gm1 * (uul * uul + vvl * vvl) + E2P * ((uul - al) * (uul - al) + vvl * vvl) * T(0.5) +
                    E3P * ((uul + al) * (uul + al) + vvl * vvl) * T(0.5) + tmp3 * al * al * (E2P + E3P));
  T E1M = (uur - fabs(uur)) * T(0.5), E2M = (uur - ar - fabs(uur - ar)) * T(0.5), E3M = (uur + ar - fabs(uur + ar)) * T(0.5);
  t0 = dr / (T(2.0) * gamma);
  T m0 = t0 * (tmp1 * E1M + E2M + E3M);
  T m1 = t0 * (tmp1 * E1M * uur + E2M * (uur - ar) + E3M * (uur + ar));
  T m2 = t0 * (tmp1 * E1M * vvr + E2M * vvr + E3M * vvr);
  T m3 = t0 * (E1M * gm1 * (uur * uur + vvr * vvr) + E2M * ((uur - ar) * (uur - ar) + vvr * vvr) * T(0.5) +
                    E3M * ((uur + ar) * (uur + ar) + vvr * vvr) * T(0.5) + tmp3 * ar * ar * (E2M + E3M));
  F[0] = p0 + m0; F[1] = p1 + m1; F[2] = p2 + m2; F[3] = p3 + m3;
}

// Flux_HLL_HLLC_1D, sub_flux_split.f90:16-93
template <typename T>
__device__ __forceinline__ void flux_hll(const T *QL, const T *QR, T *F, T gamma, bool hllc) {
  T dl = QL[0], uul = QL[1], vvl = QL[2], pl = QL[3];
  T dr = QR[0], uur = QR[1], vvr = QR[2], pr = QR[3];
  T gm1 = gamma - T(1.0);
  T UL[4] = {dl, dl * uul, dl * vvl, pl / gm1 + dl * (uul * uul + vvl * vvl) * T(0.5)};
  T UR[4] = {dr, dr * uur, dr * vvr, pr / gm1 + dr * (uur * uur + vvr * vvr) * T(0.5)};
  T al = sqrt(gamma * pl / dl), ar = sqrt(gamma * pr / dr);
  T p_pvrs = T(0.5) * (pl + pr) - (uur - uul) * (dl + dr) * (al + ar) * T(0.125);
  T p_star = fmax(T(0.0), p_pvrs);
  T g2 = (gamma + T(1.0)) / (T(2.0) * gamma);
  T qql = (p_star <= pl) ? T(1.0) : sqrt(T(1.0) + g2 * (p_star / pl - T(1.0)));
  T qqr = (p_star <= pr) ? T(1.0) : sqrt(T(1.0) + g2 * (p_star / pr - T(1.0)));
  T Sl = uul - al * qql, Sr = uur + ar * qqr;
  T Fl[4] = {UL[1], UL[1] * uul + pl, UL[2] * uul, uul * (UL[3] + pl)};
  T Fr[4] = {UR[1], UR[1] * uur + pr, UR[2] * uur, uur * (UR[3] + pr)};
  if (!hllc) {
    if (Sl >= 0) { for (int m = 0; m < 4; m++) F[m] = Fl[m]; }
    else if (Sr <= 0) { for (int m = 0; m < 4; m++) F[m] = Fr[m]; }
    else { T inv = T(1.0) / (Sr - Sl);
      for (int m = 0; m < 4; m++) F[m] = (Sr * Fl[m] - Sl * Fr[m] + Sl * Sr * (UR[m] - UL[m])) * inv; }
    return;
  }
  T S_star = (pr - pl + dl * uul * (Sl - uul) - dr * uur * (Sr - uur)) / (dl * (Sl - uul) - dr * (Sr - uur));
  if (Sl >= 0) { for (int m = 0; m < 4; m++) F[m] = Fl[m]; return; }
  if (Sr <= 0) { for (int m = 0; m < 4; m++) F[m] = Fr[m]; return; }
  if (S_star >= 0) {
    T tmpl = dl * (Sl - uul) / (Sl - S_star);
    T tmp = UL[3] / dl + (S_star - uul) * (S_star + pl / (dl * (Sl - uul)));
    F[0] = Fl[0] + Sl * (tmpl - UL[0]);
    F[1] = Fl[1] + Sl * (tmpl * S_star - UL[1]);
    F[2] = Fl[2] + Sl * (tmpl * vvl - UL[2]);
    F[3] = Fl[3] + Sl * (tmpl * tmp - UL[3]);
  } else {
    T tmpr = dr * (Sr - uur) / (Sr - S_star);
    T tmp = UR[3] / dr + (S_star - uur) * (S_star + pr / (dr * (Sr - uur)));
    F[0] = Fr[0] + Sr * (tmpr - UR[0]);
    F[1] = Fr[1] + Sr * (tmpr * S_star - UR[1]);
    F[2] = Fr[2] + Sr * (tmpr * vvr - UR[2]);
    F[3] = Fr[3] + Sr * (tmpr * tmp - UR[3]);
  }
}

template <typename T>
__device__ __forceinline__ void face_flux(int iflux, const T *QL, const T *QR, T *F, T gamma, T ggm1) {
  switch (iflux) {
    case Flux_Roe: flux_roe(QL, QR, F, gamma, ggm1); return;
    case Flux_Ausm: flux_ausm(QL, QR, F, gamma, ggm1); return;
    case Flux_VanLeer: flux_vanleer(QL, QR, F, gamma); return;
    case Flux_SW: flux_sw(QL, QR, F, gamma); return;
    case Flux_HLL: flux_hll(QL, QR, F, gamma, false); return;
    case Flux_HLLC: flux_hll(QL, QR, F, gamma, true); return;
  }
  F[0] = F[1] = F[2] = F[3] = T(0.0);
}

// the same from the face's precomputed inverse Jacobian (A, B, C, D) =
// (Djy, Diy, Djx, Dix) / (Dix Djy - Djx Diy): u_x = Diu A - Dju B,
// u_y = Dju D - Diu C
template <typename T>
__device__ __forceinline__ void viscous_face_m(T A, T B, T C, T D, T Diu, T Div, T DiT, T Dju, T Djv, T DjT,
                                               T Amu1, T Amk1, T u1, T v1, T n1, T n2, T s, T &F2, T &F3, T &F4) {
  T ux = fma(Diu, A, -Dju * B), vx = fma(Div, A, -Djv * B), Tx = fma(DiT, A, -DjT * B);
  T uy = fma(Dju, D, -Diu * C), vy = fma(Djv, D, -Div * C), Ty = fma(DjT, D, -DiT * C);
  T t11 = ((T(4.0) / T(3.0)) * ux - (T(2.0) / T(3.0)) * vy) * Amu1;
  T t22 = ((T(4.0) / T(3.0)) * vy - (T(2.0) / T(3.0)) * ux) * Amu1;
  T t12 = (uy + vx) * Amu1;
  T E1 = u1 * t11 + v1 * t12 + Amk1 * Tx, E2 = u1 * t12 + v1 * t22 + Amk1 * Ty;
  F2 += (t11 * n1 + t12 * n2) * s;
  F3 += (t12 * n1 + t22 * n2) * s;
  F4 += (E1 * n1 + E2 * n2) * s;
}

}  // namespace mixed
}  // namespace ec2d
