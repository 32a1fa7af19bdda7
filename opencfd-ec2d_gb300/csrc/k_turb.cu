// k_turb.cu -- turbulence-model residual rows (Spalart-Allmaras,
// sub_turbulence_SA.f90; k-omega SST, sub_turbulence_SST.f90), the ghost
// eddy viscosity at walls (Amut_boundary), the finite-difference WENO5 patch
// (sub_Finite_Difference.f90) and the dual-time source term.  Contexts with FP32
// parts take the face and residual kernels of k_turb_mixed.cu.
#include "ec2d_dev.cuh"
#include "ec2d_internal.h"

namespace ec2d {

constexpr int TILE = EC2D_TILE;

__device__ __forceinline__ bool tile_xy(const Lvl &L, int &bk, int &i, int &j) {
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

// ---- Spalart-Allmaras (sub_turbulence_SA.f90:4-175) -------------------------
namespace sa {
constexpr double sigma = 2.0 / 3.0, Cv1 = 7.1, Cb1 = 0.1355, Cb2 = 0.622, kap = 0.41;
constexpr double Cw2 = 0.3, Cw3 = 2.0, Ct3 = 1.3, Ct4 = 0.5;
}

// eddy viscosity over 0..nx, 0..ny (sub_turbulence_SA.f90:25-32)
__global__ void k_sa_mut(Lvl L) {
  int bk, i, j;
  if (!tile_xy(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  if (i < 0 || i > b.nx || j < 0 || j > b.ny) return;
  const long long F = L.F;
  long long id = fidx(b, i, j);
  double vt = L.U[4 * F + id], d = L.q[Q_D * F + id];
  double X = d * vt * rcp(L.amu[id]);
  double X3 = X * X * X;
  double fv1 = X3 * rcp(X3 + sa::Cv1 * sa::Cv1 * sa::Cv1);
  L.amut[id] = fv1 * d * vt;
}

// Amut_boundary (sub_turbulence_SA.f90:180-220): mirror the eddy viscosity
// into the first ghost layer of wall subfaces; one CTA per block
__global__ void k_amut_boundary(Lvl L) {
  const BlkDev &b = L.blk[blockIdx.x];
  for (int ks = 0; ks < b.nsub; ks++) {
    const SubDev s = L.sub[b.sub0 + ks];
    if (s.neighb != BC_Wall) continue;
    if (s.face == 1 || s.face == 3) {
      for (int j = s.jst + threadIdx.x; j <= s.jend - 1; j += blockDim.x) {
        if (s.face == 1) L.amut[fidx(b, 0, j)] = -L.amut[fidx(b, 1, j)];
        else L.amut[fidx(b, b.nx, j)] = -L.amut[fidx(b, b.nx - 1, j)];
      }
    } else {
      for (int i = s.ist + threadIdx.x; i <= s.iend - 1; i += blockDim.x) {
        if (s.face == 2) L.amut[fidx(b, i, 0)] = -L.amut[fidx(b, i, 1)];
        else L.amut[fidx(b, i, b.ny)] = -L.amut[fidx(b, i, b.ny - 1)];
      }
    }
    __syncthreads();
  }
}

// nu~ face fluxes: first-order upwind convection and the (1+cb2)/sigma
// diffusion, i faces (sub_turbulence_SA.f90:43-73) and j faces (:87-114);
// planes 4/5 of fi, fj hold Fluxv and fluxv2
__global__ void k_sa_faces(Lvl L) {
  int bk, i, j;
  if (!tile_xy(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  const long long F = L.F, P = b.P;
  long long id = fidx(b, i, j);
  const double *vt = L.U + 4 * F, *d = L.q + Q_D * F, *uu = L.q + Q_U * F, *vv = L.q + Q_V * F;
  const double *amu = L.amu;
  const double c0 = 0.5 * (1.0 + sa::Cb2) / sa::sigma;
  const double nu = amu[id] * recip(d[id]);
  if (i >= 1 && i <= b.nx && j >= 1 && j <= b.ny - 1) {
    long long w = id - 1, nN = id + P, nS = id - P;
    double s0 = L.geo[G_SI * F + id], n1 = L.geo[G_NI1 * F + id], n2 = L.geo[G_NI2 * F + id];
    double vn1 = uu[w] * n1 + vv[w] * n2, vn2 = uu[id] * n1 + vv[id] * n2;
    const double vf = fma(pos_part(vn1), vt[w], neg_part(vn2) * vt[id]) * s0;
    const double v0 = c0 * ((vt[id] + nu) + fma(amu[w], recip(d[w]), vt[w]));
    // the normal derivative by the face's coefficients formed at set-up (k_face_metrics)
    const double *gm = L.geo + id;
    double Div = vt[id] - vt[w];
    double Djv = (vt[nN - 1] - vt[nS - 1]) + (vt[nN] - vt[nS]);
    double g = fma(Div, gm[G_VIP * F], Djv * gm[G_VIQ * F]) * s0;
    L.fi[4 * F + id] = fma(v0, g, -vf);
    L.fi[5 * F + id] = g;
  }
  if (i >= 1 && i <= b.nx - 1 && j >= 1 && j <= b.ny) {
    long long s = id - P;
    double s0 = L.geo[G_SJ * F + id], n1 = L.geo[G_NJ1 * F + id], n2 = L.geo[G_NJ2 * F + id];
    double vn1 = uu[s] * n1 + vv[s] * n2, vn2 = uu[id] * n1 + vv[id] * n2;
    const double vf = fma(pos_part(vn1), vt[s], neg_part(vn2) * vt[id]) * s0;
    const double v0 = c0 * ((vt[id] + nu) + fma(amu[s], recip(d[s]), vt[s]));
    const double *gm = L.geo + id;
    double Div = (vt[s + 1] - vt[s - 1]) + (vt[id + 1] - vt[id - 1]);
    double Djv = vt[id] - vt[s];
    double g = fma(Div, gm[G_VJP * F], Djv * gm[G_VJQ * F]) * s0;
    L.fj[4 * F + id] = fma(v0, g, -vf);
    L.fj[5 * F + id] = g;
  }
}

// (a / b)^(1/6), b >= 64: w = (b / a)^(-1/6) to about 2^-19 in FP32, then one step of
// Householder's third-order iteration for w^-6 = b / a.  The float w has exact squares,
// so the relative error stays below 0.84 eps (0.73 in 4e6 samples; 0.78 of cbrt(sqrt(a / b)));
// 9 FP64 instructions against about 40 of those functions, which serve the rest of the range.
__device__ __forceinline__ double sixth_root(double a, double ra, double b) {
  if (!(at_least(b, 64.0) && below(b, 1.0e37))) return cbrt(sqrt(a * recip(b)));
  const double q = b * ra, w = to_double(exp2f(log2f(to<float>(q)) * (-1.0f / 6.0f)));
  const double w2 = w * w, e = fma(-q, w2 * w2 * w2, 1.0);
  return fma(w, e * fma(e, 7.0 / 72.0, 1.0 / 6.0), w);
}

// Bound by FP64 issue like every kernel of this file (65 k cells are 14 warps per
// SM): quotients by rcp, signs and halves by integers.
// Res(5): flux differences with the cb2 cross term and the production /
// destruction source (sub_turbulence_SA.f90:77-82, 118-124, 129-168)
__global__ void k_sa_res(Lvl L) {
  int bk, i, j;
  if (!tile_xy(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  if (i < 1 || i > b.nx - 1 || j < 1 || j > b.ny - 1) return;
  const long long F = L.F, P = b.P;
  long long id = fidx(b, i, j);
  const double *x1 = L.geo + G_X1 * F, *y1 = L.geo + G_Y1 * F, *uu = L.q + Q_U * F, *vv = L.q + Q_V * F;
  double vt = L.U[4 * F + id], d = L.q[Q_D * F + id], amu = L.amu[id];
  const double ramu = recip(amu);
  double v0 = (vt + amu * recip(d)) * (sa::Cb2 / sa::sigma);
  const double r = (L.fi[4 * F + id + 1] - L.fi[4 * F + id]) + (L.fj[4 * F + id + P] - L.fj[4 * F + id]) -
                   v0 * ((L.fi[5 * F + id + 1] - L.fi[5 * F + id]) + (L.fj[5 * F + id + P] - L.fj[5 * F + id]));
  // the halves of the central differences cancel in the quotients
  const double Dix = x1[id + 1] - x1[id - 1], Diy = y1[id + 1] - y1[id - 1];
  const double Djx = x1[id + P] - x1[id - P], Djy = y1[id + P] - y1[id - P];
  const double Ds = recip(Dix * Djy - Djx * Diy);
  const double Diu = uu[id + 1] - uu[id - 1], Div = vv[id + 1] - vv[id - 1];
  const double Dju = uu[id + P] - uu[id - P], Djv = vv[id + P] - vv[id - P];
  const double S = fabs(((Div * Djy - Djv * Diy) - (Dju * Dix - Diu * Djx)) * Ds);
  double dw = L.geo[G_DW * F + id];
  double X = d * vt * ramu;
  double X3 = X * X * X;
  double fv1 = X3 * recip(X3 + sa::Cv1 * sa::Cv1 * sa::Cv1);
  double fv2 = 1.0 - X * recip(1.0 + X * fv1);
  double kd = sa::kap * dw;
  const double rkd2 = recip(kd * kd);  // 1 / (kappa d)^2
  double S1 = fmax(S + fv2 * vt * rkd2, (double)0.3f * S);  // 0.3 is a single-precision literal
  double rr = fmin(vt * recip(S1) * rkd2, 10.0);
  double r2 = rr * rr, r6 = r2 * r2 * r2;
  double g = rr + sa::Cw2 * (r6 - rr);
  double g2 = g * g, g6 = g2 * g2 * g2;
  constexpr double c36 = sa::Cw3 * sa::Cw3 * sa::Cw3 * sa::Cw3 * sa::Cw3 * sa::Cw3;
  const double fw = g * sixth_root(1.0 + c36, 1.0 / (1.0 + c36), g6 + c36);
  // exp(-X^2 / 2) is zero from X^2 = 1492 on, in most of a boundary layer
  const double X2 = X * X, ft2 = at_least(X2, 1492.0) ? 0.0 : sa::Ct3 * exp(-sa::Ct4 * X2);
  const double Cw1 = sa::Cb1 / (sa::kap * sa::kap) + (1.0 + sa::Cb2) / sa::sigma;
  double q = vt * recip(dw);
  double Q = sa::Cb1 * (1.0 - ft2) * S1 * vt - (Cw1 * fw - sa::Cb1 * ft2 / (sa::kap * sa::kap)) * (q * q);
  L.res[4 * F + id] = r + Q * L.geo[G_VOL * F + id];
}

void launch_sa(const Lvl &L, cudaStream_t s) {
  k_sa_mut<<<L.ntiles, TILE, 0, s>>>(L);
  k_amut_boundary<<<L.nblk, 128, 0, s>>>(L);
  if (L.mixed) { launch_sa_rows_mixed(L, s); return; }
  k_sa_faces<<<L.ntiles, TILE, 0, s>>>(L);
  k_sa_res<<<L.ntiles, TILE, 0, s>>>(L);
}
void launch_amut_boundary(const Lvl &L, cudaStream_t s) { k_amut_boundary<<<L.nblk, 128, 0, s>>>(L); }

// ---- k-omega SST (sub_turbulence_SST.f90:6-271) -----------------------------
namespace sst {
constexpr double sk1 = 0.85, sw1 = 0.5, beta1 = 0.075, Cw1 = 0.533;
constexpr double sk2 = 1.0, sw2 = 0.856, beta2 = 0.0828, Cw2 = 0.440;
constexpr double a1 = 0.31, betas = 0.09;
}
// scratch planes in L.tb
enum { T_AMUS = 0, T_AMUTS = 1, T_F1 = 2, T_QK = 3, T_QW = 4 };
static_assert(T_QW + 1 == SST_PLANES, "planes of the SST scratch");
// k and omega, in two of the planes that the mean-flow fluxes fill after the model
enum { FI_K = 0, FI_W = 1 };

// cell pass (sub_turbulence_SST.f90:53-121): eddy viscosity, blending f1 and
// the k/omega sources; Amu is scaled by Re for the model and scaled back
// (x*Re/Re, as the reference does at :85 and :259)
__global__ void k_sst_cell(Lvl L) {
  int bk, i, j;
  if (!tile_xy(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  if (i < 0 || i > b.nx || j < 0 || j > b.ny) return;
  const CaseDev &c = L.cs[b.cas];
  const long long F = L.F, P = b.P;
  const double Re = c.Re;
  long long id = fidx(b, i, j);
  const double *x1 = L.geo + G_X1 * F, *y1 = L.geo + G_Y1 * F, *uu = L.q + Q_U * F, *vv = L.q + Q_V * F;
  const double *d = L.q + Q_D * F, *U5 = L.U + 4 * F, *U6 = L.U + 5 * F;
  const double dc = d[id], rd = recip_any(dc), K = U5[id] * rd, W = U6[id] * rd;
  // k and omega of every cell that a face reads
  L.fi[FI_K * F + id] = K;
  L.fi[FI_W * F + id] = W;
  if (i < 1 || i > b.nx - 1 || j < 1 || j > b.ny - 1) return;
  // central differences (their halves cancel in the quotients)
  const double Dix = x1[id + 1] - x1[id - 1], Diy = y1[id + 1] - y1[id - 1];
  const double Djx = x1[id + P] - x1[id - P], Djy = y1[id + P] - y1[id - P];
  const double Ds = recip(Dix * Djy - Djx * Diy);
  const double re = recip_any(d[id + 1]), rw = recip_any(d[id - 1]), rn = recip_any(d[id + P]), rs = recip_any(d[id - P]);
  const double Diu = uu[id + 1] - uu[id - 1], Div = vv[id + 1] - vv[id - 1];
  const double Dju = uu[id + P] - uu[id - P], Djv = vv[id + P] - vv[id - P];
  const double Dik = U5[id + 1] * re - U5[id - 1] * rw, Diw = U6[id + 1] * re - U6[id - 1] * rw;
  const double Djk = U5[id + P] * rn - U5[id - P] * rs, Djw = U6[id + P] * rn - U6[id - P] * rs;
  const double omega = ((Div * Djy - Djv * Diy) - (Dju * Dix - Diu * Djx)) * Ds;
  const double kx = Dik * Djy - Djk * Diy, wx = Diw * Djy - Djw * Diy;
  const double ky = Djk * Dix - Dik * Djx, wy = Djw * Dix - Diw * Djx;
  const double rRe = c.rRe, amu = L.amu[id], amus = amu * Re;
  const double dw = L.geo[G_DW * F + id], rdw = recip_any(dw), rW = recip_any(W);
  const double c009 = (double)0.09f;  // single-precision literal (sub_turbulence_SST.f90:87,96)
  const double t2 = 500.0 * amu * rRe * rd * rW * (rdw * rdw);
  const double kw = root(fabs(K)) * rW * rdw * recip(c009 * Re);
  const double arg2 = fmax(pow2<1>(kw), t2);
  const double f2 = tanh_pos(arg2 * arg2);
  const double dK = dc * K;
  double amuts = fmin(fmin(dK * rW, sst::a1 * dK * Re * recip_any(f2 * fabs(omega))), 100000.0);
  const double Kws = (kx * wx + ky * wy) * (Ds * Ds) * dc * (2.0 * sst::sw2) * recip_any(W + 1.0e-20);
  const double CD = fmax(Kws, 1.0e-20);
  const double arg3 = fmax(kw, t2);
  const double arg1 = fmin(arg3, 4.0 * sst::sw2 * dK * recip_any(CD * (dw * dw)));
  double a1s = arg1 * arg1;
  double f1 = tanh_pos(a1s * a1s);
  const double om2 = omega * omega, g1 = 1.0 - f1;
  double Pk = amuts * om2;
  double Pk0 = fmin(Pk, 20.0 * sst::betas * K * W * (Re * Re));
  double Qk = Pk0 * rRe - sst::betas * dK * W * Re;
  double Cw = f1 * sst::Cw1 + g1 * sst::Cw2;
  double beta = f1 * sst::beta1 + g1 * sst::beta2;
  double Qw = (Cw * dc * om2 + g1 * Kws) * rRe - beta * dc * (W * W) * Re;
  L.tb[T_AMUS * F + id] = amus;
  L.tb[T_AMUTS * F + id] = amuts;
  L.tb[T_F1 * F + id] = f1;
  L.tb[T_QK * F + id] = Qk;
  L.tb[T_QW * F + id] = Qw;
}

// k and omega come from planes that k_sst_cell fills once per cell, and the normal
// derivatives from the set-up coefficients, where each face divided twelve times by the
// density and formed its Jacobian: the four kernels of the model on 65 k cells take
// 55 us instead of 125.
// k and omega face fluxes, i faces (sub_turbulence_SST.f90:129-182) and j
// faces (:198-248); planes 4/5 of fi and fj
__global__ void k_sst_faces(Lvl L) {
  int bk, i, j;
  if (!tile_xy(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  const CaseDev &c = L.cs[b.cas];
  const long long F = L.F, P = b.P;
  long long id = fidx(b, i, j);
  const double *uu = L.q + Q_U * F, *vv = L.q + Q_V * F, *K = L.fi + FI_K * F, *W = L.fi + FI_W * F;
  const double *amus = L.tb + T_AMUS * F, *amuts = L.tb + T_AMUTS * F, *g = L.geo + id;
  const double f1 = L.tb[T_F1 * F + id];
  const double sk = f1 * sst::sk1 + (1.0 - f1) * sst::sk2;
  const double sw = f1 * sst::sw1 + (1.0 - f1) * sst::sw2;
  // convection of the upwind side and diffusion along the normal (metric coefficients
  // of k_face_metrics); cl, cr: the cells of the viscosity, the interior one
  // twice at a block's ends
  auto face = [&](long long o, long long cl, long long cr, double s, double n1, double n2, double Dk, double Dw, double *f) {
    const double un1 = uu[o] * n1 + vv[o] * n2, un2 = uu[id] * n1 + vv[id] * n2;
    const double up = pos_part(un1) * s, um = neg_part(un2) * s;
    const double ms = amus[cl] + amus[cr], mt = amuts[cl] + amuts[cr], sr = half(s) * c.rRe;
    f[4 * F + id] = fma(fma(sk, mt, ms) * sr, Dk, -fma(up, K[o], um * K[id]));
    f[5 * F + id] = fma(fma(sw, mt, ms) * sr, Dw, -fma(up, W[o], um * W[id]));
  };
  if (i >= 1 && i <= b.nx && j >= 1 && j <= b.ny - 1) {
    const long long w = id - 1, nN = id + P, nS = id - P;
    const double p = g[G_VIP * F], q = g[G_VIQ * F];
    const double Djk = (K[nN - 1] - K[nS - 1]) + (K[nN] - K[nS]), Djw = (W[nN - 1] - W[nS - 1]) + (W[nN] - W[nS]);
    face(w, i == 1 ? id : w, i == b.nx ? w : id, g[G_SI * F], g[G_NI1 * F], g[G_NI2 * F],
         fma(K[id] - K[w], p, Djk * q), fma(W[id] - W[w], p, Djw * q), L.fi);
  }
  if (i >= 1 && i <= b.nx - 1 && j >= 1 && j <= b.ny) {
    const long long s = id - P;
    const double p = g[G_VJP * F], q = g[G_VJQ * F];
    const double Dik = (K[s + 1] - K[s - 1]) + (K[id + 1] - K[id - 1]), Diw = (W[s + 1] - W[s - 1]) + (W[id + 1] - W[id - 1]);
    face(s, j == 1 ? id : s, j == b.ny ? s : id, g[G_SJ * F], g[G_NJ1 * F], g[G_NJ2 * F],
         fma(Dik, p, (K[id] - K[s]) * q), fma(Diw, p, (W[id] - W[s]) * q), L.fj);
  }
}

// Res(5:6) and the rescaled viscosities (sub_turbulence_SST.f90:186-191, 254-262)
__global__ void k_sst_res(Lvl L) {
  int bk, i, j;
  if (!tile_xy(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  if (i < 1 || i > b.nx - 1 || j < 1 || j > b.ny - 1) return;
  const CaseDev &c = L.cs[b.cas];
  const long long F = L.F, P = b.P;
  long long id = fidx(b, i, j);
  double vol = L.geo[G_VOL * F + id];
  double r5 = L.fi[4 * F + id + 1] - L.fi[4 * F + id];
  double r6 = L.fi[5 * F + id + 1] - L.fi[5 * F + id];
  r5 = r5 + L.fj[4 * F + id + P] - L.fj[4 * F + id] + L.tb[T_QK * F + id] * vol;
  r6 = r6 + L.fj[5 * F + id + P] - L.fj[5 * F + id] + L.tb[T_QW * F + id] * vol;
  L.res[4 * F + id] = r5;
  L.res[5 * F + id] = r6;
  L.amu[id] = L.tb[T_AMUS * F + id] * c.rRe;
  L.amut[id] = L.tb[T_AMUTS * F + id] * c.rRe;
}

void launch_sst(const Lvl &L, cudaStream_t s) {
  if (L.mixed) {
    launch_sst_rows_mixed(L, s);
  } else {
    k_sst_cell<<<L.ntiles, TILE, 0, s>>>(L);
    k_sst_faces<<<L.ntiles, TILE, 0, s>>>(L);
    k_sst_res<<<L.ntiles, TILE, 0, s>>>(L);
  }
  k_amut_boundary<<<L.nblk, 128, 0, s>>>(L);
}

// ---- finite-difference patch (sub_Finite_Difference.f90:4-275) --------------
// scratch planes in L.fdm: 0-7 i-direction split fluxes (fp 0-3, fm 4-7),
// 8-15 j-direction, 16-19 i fluxes, 20-23 j fluxes, 24-29 viscous Ev1/Ev2
enum { D_SPI = 0, D_SPJ = 8, D_FI = 16, D_FJ = 20, D_EV1 = 24, D_EV2 = 27 };

// split_Steger_Warming, sub_Finite_Difference.f90:154-202
// An eigenvalue goes to one of the two parts by its sign, so the halves (E + |E|)/2
// and E - E+ are selects.
__device__ __forceinline__ void split_sw(double d, double u, double v, double cc, double A1, double A2,
                                         const CaseDev &c, double *fp, double *fm) {
  const double w = fma(A1, A1, A2 * A2), rss = rroot(w), cs = cc * (w * rss);
  const double c1 = cc * (A1 * rss), c2 = cc * (A2 * rss);
  const double t0 = half(d * c.rg), E1 = A1 * u + A2 * v, E2 = E1 - cs, E3 = E1 + cs;
  const double e1 = E1 * (t0 * pow2<1>(c.gm1)), e2 = E2 * t0, e3 = E3 * t0;
  const double uc1 = u - c1, uc2 = u + c1, vc1 = v - c2, vc2 = v + c2;
  const double W2 = (half(3.0 - c.gamma) * c.rgm1) * (cc * cc);
  const double h1 = half(fma(u, u, v * v)), h2 = fma(half(uc1), uc1, fma(half(vc1), vc1, W2)),
               h3 = fma(half(uc2), uc2, fma(half(vc2), vc2, W2));
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const double a = k ? neg_part(e1) : pos_part(e1), p = k ? neg_part(e2) : pos_part(e2),
                 q = k ? neg_part(e3) : pos_part(e3);
    double *f = k ? fm : fp;
    f[0] = a + p + q;
    f[1] = fma(a, u, fma(p, uc1, q * uc2));
    f[2] = fma(a, v, fma(p, vc1, q * vc2));
    f[3] = fma(a, h1, fma(p, h2, q * h3));
  }
}
enum { M_KX = 0, M_KY = 1, M_IX = 2, M_IY = 3, M_JAC = 4 };

__global__ void k_fdm_split(Lvl L) {
  int bk, i, j;
  if (!tile_xy(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  if (!b.fdm || i < 1 || i > b.nx - 1 || j < 1 || j > b.ny - 1) return;
  const CaseDev &c = L.cs[b.cas];
  const long long F = L.F;
  long long id = fidx(b, i, j);
  double d = L.q[Q_D * F + id], u = L.q[Q_U * F + id], v = L.q[Q_V * F + id], cc = L.q[Q_C * F + id];
  const double rJ = recip(L.met[M_JAC * F + id]);
  double fp[4], fm[4];
  // blockIdx.y: 0 the i-direction split, 1 the j-direction split (two threads per cell)
  const int dir = blockIdx.y;
  const int mx = dir == 0 ? M_KX : M_IX, my = dir == 0 ? M_KY : M_IY, out = dir == 0 ? D_SPI : D_SPJ;
  split_sw(d, u, v, cc, L.met[mx * F + id] * rJ, L.met[my * F + id] * rJ, c, fp, fm);
  for (int m = 0; m < 4; m++) { L.fdm[(out + m) * F + id] = fp[m]; L.fdm[(out + 4 + m) * F + id] = fm[m]; }
}

// fp_weno5 at point k from v[k-2..k+2] = a, b, c, d, e; fm_weno5 is the same with the
// points in reverse (sub_Finite_Difference.f90:207-275).  The reference forms the
// weights as a_k = C_k / (ep + S_k)^2 and W_k = a_k / sum(a); over the common
// denominator D_0 D_1 D_2 (D_k = (ep + S_k)^2) they are
// W_0 : W_1 : W_2 = 3 D_1 D_2 : 6 D_0 D_2 : D_0 D_1.  Smoothness indicators and
// candidate values are written in the first and second differences of v,
//   S_0 = d3^2 + s3 (4/3 s3 - d3),  S_1 = d3^2 + s2 (4/3 s2 - d3),  S_2 = d2^2 + s1 (4/3 s1 + d2),
//   q_0 - c = d3/2 - s3/6,  q_1 - c = d3/2 - s2/6,  q_2 - c = d2/2 + s1/3,
// 30 FP64 instructions per value; written out from the five values with an IEEE
// divide it took 60, and the 65 k cells of a 513 x 129 block took 203 us with
// split and residual, three launches (110 us now).  D_k >= 1e-12, so numerator and denominator stay above
// 1e-36, and they overflow only for smoothness indicators beyond about 1e50, far
// from any split flux of this solver.
__device__ __forceinline__ double weno5(double a, double b, double c, double d, double e) {
  const double ep = 1.0e-6, t = 4.0 / 3.0;
  const double d1 = b - a, d2 = c - b, d3 = d - c, d4 = e - d;
  const double s1 = d2 - d1, s2 = d3 - d2, s3 = d4 - d3;
  const double c3 = fma(d3, d3, ep), c2 = fma(d2, d2, ep);
  double D0 = fma(s3, fma(t, s3, -d3), c3), D1 = fma(s2, fma(t, s2, -d3), c3), D2 = fma(s1, fma(t, s1, d2), c2);
  D0 *= D0;
  D1 *= D1;
  D2 *= 3.0 * D2;
  const double E0 = pow2<1>(D0), q = D0 * D1, sixth = 1.0 / 6.0;
  const double h = half(d3), p0 = fma(-sixth, s3, h), p1 = fma(-sixth, s2, h), p2 = fma(2.0 * sixth, s1, half(d2));
  return fma(fma(D2, fma(D1, p0, E0 * p1), q * p2), recip(fma(D2, D1 + E0, q)), c);
}

// WENO5 half-point fluxes (sub_Finite_Difference.f90:37-77) and the central
// viscous tensors Ev1/Ev2 (:87-117); indices are FDM cells = FVM cells.
// blockIdx.y picks the part: 0 the i-direction fluxes, 1 the j-direction
// fluxes, 2 the viscous tensors, so a cell's three independent chains run
// on three threads.
__global__ void k_fdm_flux(Lvl L) {
  const int part = blockIdx.y;
  int bk, i, j;
  if (!tile_xy(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  int nxF = b.nx - 1, nyF = b.ny - 1;
  if (!b.fdm || i < 1 || i > nxF || j < 1 || j > nyF) return;
  const CaseDev &c = L.cs[b.cas];
  const long long F = L.F, P = b.P;
  long long id = fidx(b, i, j);
  if (part == 0 && j >= LFDM && j <= nyF - LFDM && i >= LFDM && i <= nxF - LFDM) {
    for (int m = 0; m < 4; m++) {
      const double *fp = L.fdm + (D_SPI + m) * F, *fm = L.fdm + (D_SPI + 4 + m) * F;
      double h1 = weno5(fp[id - 2], fp[id - 1], fp[id], fp[id + 1], fp[id + 2]);
      double h2 = weno5(fm[id + 3], fm[id + 2], fm[id + 1], fm[id], fm[id - 1]);
      L.fdm[(D_FI + m) * F + id] = -(h1 + h2);
    }
  }
  if (part == 1 && i >= LFDM && i <= nxF - LFDM && j >= LFDM && j <= nyF - LFDM) {
    for (int m = 0; m < 4; m++) {
      const double *fp = L.fdm + (D_SPJ + m) * F, *fm = L.fdm + (D_SPJ + 4 + m) * F;
      double h1 = weno5(fp[id - 2 * P], fp[id - P], fp[id], fp[id + P], fp[id + 2 * P]);
      double h2 = weno5(fm[id + 3 * P], fm[id + 2 * P], fm[id + P], fm[id], fm[id - P]);
      L.fdm[(D_FJ + m) * F + id] = -(h1 + h2);
    }
  }
  if (part == 2 && L.visc && i >= 2 && i <= nxF - 1 && j >= 2 && j <= nyF - 1) {
    const double *uu = L.q + Q_U * F, *vv = L.q + Q_V * F, *TT = L.q + Q_T * F;
    double mu0 = L.amu[id] + L.amut[id];
    double Ak0 = c.kpr * L.amu[id] + c.kprt * L.amut[id];
    double ui = half(uu[id + 1] - uu[id - 1]), vi = half(vv[id + 1] - vv[id - 1]), Ti = half(TT[id + 1] - TT[id - 1]);
    double uj = half(uu[id + P] - uu[id - P]), vj = half(vv[id + P] - vv[id - P]), Tj = half(TT[id + P] - TT[id - P]);
    double Akx = L.met[M_KX * F + id], Aky = L.met[M_KY * F + id], Aix = L.met[M_IX * F + id], Aiy = L.met[M_IY * F + id];
    const double rJ = recip(L.met[M_JAC * F + id]);
    double ux = ui * Akx + uj * Aix, vx = vi * Akx + vj * Aix, Tx = Ti * Akx + Tj * Aix;
    double uy = ui * Aky + uj * Aiy, vy = vi * Aky + vj * Aiy, Ty = Ti * Aky + Tj * Aiy;
    double t11 = (4.0 / 3.0 * ux - 2.0 / 3.0 * vy) * mu0, t22 = (4.0 / 3.0 * vy - 2.0 / 3.0 * ux) * mu0;
    double t12 = (uy + vx) * mu0;
    double E1 = uu[id] * t11 + vv[id] * t12 + Ak0 * Tx, E2 = uu[id] * t12 + vv[id] * t22 + Ak0 * Ty;
    L.fdm[(D_EV1 + 0) * F + id] = (Akx * t11 + Aky * t12) * rJ;
    L.fdm[(D_EV1 + 1) * F + id] = (Akx * t12 + Aky * t22) * rJ;
    L.fdm[(D_EV1 + 2) * F + id] = (Akx * E1 + Aky * E2) * rJ;
    L.fdm[(D_EV2 + 0) * F + id] = (Aix * t11 + Aiy * t12) * rJ;
    L.fdm[(D_EV2 + 1) * F + id] = (Aix * t12 + Aiy * t22) * rJ;
    L.fdm[(D_EV2 + 2) * F + id] = (Aix * E1 + Aiy * E2) * rJ;
  }
}

// FDM residual (sub_Finite_Difference.f90:121-145) with the viscous half-point
// averages added to the inviscid fluxes
__global__ void k_fdm_res(Lvl L) {
  int bk, i, j;
  if (!tile_xy(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  int nxF = b.nx - 1, nyF = b.ny - 1;
  if (!b.fdm || i < LFDM + 1 || i > nxF - LFDM || j < LFDM + 1 || j > nyF - LFDM) return;
  const long long F = L.F, P = b.P;
  long long id = fidx(b, i, j);
  for (int m = 0; m < 4; m++) {
    const double *fi = L.fdm + (D_FI + m) * F, *fj = L.fdm + (D_FJ + m) * F;
    double r = (fi[id] - fi[id - 1]) + (fj[id] - fj[id - P]);
    if (L.visc && m >= 1) {  // differences of the half-point averages
      const double *e1 = L.fdm + (D_EV1 + m - 1) * F, *e2 = L.fdm + (D_EV2 + m - 1) * F;
      r += half((e1[id + 1] - e1[id - 1]) + (e2[id + P] - e2[id - P]));
    }
    L.res[m * F + id] = r;
  }
}

void launch_fdm(const Lvl &L, cudaStream_t s) {
  if (L.mixed) { launch_fdm_mixed(L, s); return; }
  k_fdm_split<<<dim3(L.ntiles, 2), TILE, 0, s>>>(L);
  k_fdm_flux<<<dim3(L.ntiles, L.visc ? 3 : 2), TILE, 0, s>>>(L);
  k_fdm_res<<<L.ntiles, TILE, 0, s>>>(L);
}

// dual-time source (sub_Residual.f90:55-65)
__global__ void k_dual(Lvl L, double sfac) {
  int bk, i, j;
  if (!tile_xy(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  if (i < 1 || i > b.nx - 1 || j < 1 || j > b.ny - 1) return;
  const long long F = L.F;
  long long id = fidx(b, i, j);
  double vol = L.geo[G_VOL * F + id];
  for (int m = 0; m < L.nvar; m++)
    L.res[m * F + id] = L.res[m * F + id] - (3.0 * L.U[m * F + id] - 4.0 * L.un[m * F + id] + L.un1[m * F + id]) * vol * sfac;
}
void launch_dual_term(const Lvl &L, double sfac, cudaStream_t s) { k_dual<<<L.ntiles, TILE, 0, s>>>(L, sfac); }

}  // namespace ec2d
