// ec2d_dev.cuh -- device data layout and the pointwise physics of the
// GB300-native OpenCFD-EC2D core.
//
// Layout in HBM (one allocation per field kind and mesh level, all blocks of
// all cases of a context side by side):
//   every 2-D quantity of block b lives in a "frame" of (nx+5) x (ny+5)
//   doubles, row-major with i fastest, origin at (i,j) = (-2,-2):
//       idx(i,j) = off_b + (j+2)*P_b + (i+2),   P_b = nx+5
//   so cell, node and face arrays of the reference (whose index ranges all lie
//   in [-2, nx+2] x [-2, ny+2]) share one index map.  A multi-variable field
//   is NV such planes, plane stride F = total frame size of the level, so the
//   variable index is the slowest (structure of arrays) and warps read
//   consecutive i with unit stride.
#pragma once
#include <cstdint>

namespace ec2d {

constexpr int LAP = 2;
constexpr int LFDM = 4;
constexpr double PrT = 0.9;
constexpr int SST_PLANES = 5;  // scratch planes of the SST model

enum { Scheme_UD1 = 0, Scheme_NND2 = 1, Scheme_UD3 = 2, Scheme_WENO3 = 3,
       Scheme_MUSCL2 = 4, Scheme_MUSCL3 = 5, Scheme_OMUSCL2 = 6 };
enum { Flux_SW = 1, Flux_HLL = 2, Flux_HLLC = 3, Flux_Roe = 4, Flux_VanLeer = 5, Flux_Ausm = 6 };
enum { Recon_Original = 0, Recon_Conservative = 1, Recon_Characteristic = 2 };
enum { BC_Wall = -10, BC_Farfield = -20, BC_Symmetry = -30, BC_Inlet = -40, BC_Outlet = -50 };
enum { Time_Euler1 = 1, Time_RK3 = 3, Time_LU_SGS = 0, Time_Dual = -1 };
enum { Turb_NONE = 0, Turb_BL = 1, Turb_SA = 2, Turb_SST = 3 };

// primitive planes in Lvl::q
enum { Q_D = 0, Q_U = 1, Q_V = 2, Q_T = 3, Q_P = 4, Q_C = 5, NQ = 6 };
// geometry planes in Lvl::geo
// G_VI*, G_VJ*: the metric coefficients of the viscous terms of an i- or j-face,
// formed at set-up (k_face_metrics) from the cell centres: with the face-local
// inverse Jacobian (A, B, C, D) = (Djy, Diy, Djx, Dix) / (Dix Djy - Djx Diy) and
// the unit normal n, P = A n1 - C n2, Q = D n2 - B n1, R = A n2 + C n1, S = B n2 +
// D n1 (see viscous_face_m); G_SIA..G_NJ2A: the cell's face
// length and normal averaged over its two i- (j-) faces, G_VI2 / G_VJ2 their
// squared length over the cell volume (the metric factors of comput_Lvc)
enum { G_VOL = 0, G_SI = 1, G_SJ = 2, G_NI1 = 3, G_NI2 = 4, G_NJ1 = 5, G_NJ2 = 6,
       G_X = 7, G_Y = 8, G_X1 = 9, G_Y1 = 10, G_DW = 11,
       G_VIP = 12, G_VIQ = 13, G_VIR = 14, G_VIS = 15, G_VJP = 16, G_VJQ = 17, G_VJR = 18, G_VJS = 19,
       G_SIA = 20, G_NI1A = 21, G_NI2A = 22, G_SJA = 23, G_NJ1A = 24, G_NJ2A = 25, G_VI2 = 26, G_VJ2 = 27,
       NG = 28 };
// spectral-radius / time-step planes in Lvl::lc
enum { L_CI = 0, L_CJ = 1, L_VI = 2, L_VJ = 3, L_DT = 4, NL = 5 };

struct BlkDev {
  int nx, ny, P, cas;       // node counts, frame pitch, owning case (0-based)
  long long off;            // frame offset in every plane of the level
  int fdm;                  // 1: finite-difference interior (FDM.in)
  int nsub, sub0;           // subfaces [sub0, sub0+nsub) in Lvl::sub
  int tile0;                // first extended-range tile of this block
  int lsub0, lsubn;         // fine-mesh wall faces (forces), unused on coarse levels
  int cell0;                // dense index of cell (1,1) among the level's interior cells
  int nphase;               // barrier phases of the physical boundary conditions
};

struct SubDev {
  int face, ist, iend, jst, jend, neighb, orient;
  int phase, nitem;         // physical BC: barrier phase within the block, work items
  int nbk;                  // level-global index of the neighbour block (-1: physical)
  int nface, nist, niend, njst, njend;  // the neighbour subface it reads
  int nP;                   // the neighbour block's frame pitch and offset (halo copy)
  long long noff;
  int nrm0;                 // far-field / symmetry: first node's entry in Lvl::bcn (-1: none)
};

struct CaseDev {
  double gamma, Ma, Re, Pr, Cv, Cp, cosA, sinA, p00, Tsb, Twall, p_outlet;
  double vt_inf, Kt_inf, Wt_inf, CFL, dtmax, dtmin, dt_global, T_inf;
  double xaxis, yaxis;
  double rPr, rCv, rMa, rRe;  // 1/Pr, 1/Cv, 1/Ma, 1/Re
  double rgm1;                // 1/(gamma - 1)
  double gm1, rg;             // gamma - 1, 1/gamma
  double kpr, kprt;           // Cp/Pr, Cp/Pr_t
  double mu0;                 // (1 + Tsb)/Re
  double gpr, gprt;           // gamma/Pr, gamma/Pr_t
  double ggm1;                // gamma/(gamma - 1)
  int local_dt, pad;
};

// Everything a kernel needs about one mesh level, passed by value.
struct Lvl {
  int nblk, nvar, scheme, gscheme, flux, recon, visc, turb, level, time_method;
  int ncase, ntiles;
  long long F;              // plane stride (doubles)
  const BlkDev *blk;
  const SubDev *sub;
  const CaseDev *cs;
  const int2 *tiles;        // (block, first linear index) of the extended window's tiles
  const int2 *ctiles;       // the same over the core window (core_ij)
  int nctiles;
  double *U, *q, *amu, *amut, *res, *lc, *du, *geo, *un, *deltu, *qf, *un1;
  double *fi, *fj;          // face-flux scratch, 6 planes each (before the fluxes also slopes, k and omega)
  double *tb;               // turbulence scratch planes
  int slopes;               // MUSCL3 slopes once per cell (k_slopes): 0 no, 1 where the context has FP32 parts, 2 always
  double *slope;            // their 16 planes, in rec; null: 8 planes of fi, fj and res for a direction at a time
  double *met;              // FDM metrics Akx,Aky,Aix,Aiy,Ajac
  double *fdm;              // FDM scratch planes
  double *lu;               // LU-SGS pre-pass planes (4 NV + 10)
  double *rec;              // LU-SGS per-cell sweep records, [2 passes][ncell][lusgs_planes(NV)] (null: rows too many)
  double2 *bcn;             // unit normals of the far-field and symmetry boundary nodes
  int ncell;                // interior cells of the level (all blocks of all cases)
  double *npart;            // norm partials: per tile 2*6 doubles
  double *norms;            // per case: max[6], rms[6]
  const int *case_tile0, *case_ntile, *case_ncell;  // per case: first tile, tiles, interior cells
  unsigned *nctr;           // tiles of k_res done (the last one reduces the partials)
  int *status;              // per case: code, block, i, j
  int silent_band_edge;     // test hook: band edges of the banded wavefronts send nothing
  int mixed;                // a context with FP32 parts: arithmetic of ec2d_mixed.cuh
  int keep_amut;            // coarse level: amut is restricted from the finer level, not zeroed
};

// Items (cells, faces or nodes of a block's padded index range) per tile of
// the level's tile list, and threads per CTA of the kernels that walk it.
// Most of those kernels are chains of FP64 operations on this part, so their
// time is the chain length times the warps that share a sub-partition: 128
// gives every warp of the 2 x 48 x 48 and 2 x 24 x 24 multigrid levels its
// own sub-partition, where 256 put two on each.
constexpr int EC2D_TILE = 128;

__host__ __device__ __forceinline__ long long fidx(const BlkDev &b, int i, int j) {
  return b.off + (long long)(j + 2) * b.P + (i + 2);
}

// Tiles of a level come in two windows per block.  The extended window
// (Lvl::tiles, i = -1..nx+1, j = -1..ny+1) reaches the second ghost layer,
// where the primitives and the explicit updates are formed.  The core window
// (Lvl::ctiles, i = 0..nx, j = 0..ny) holds every face, every interior cell
// and the range of Set_Un: the face, residual, norm and record kernels walk
// it.  On two blocks of 97 x 97 nodes the extended window takes 158 tiles and
// the core window 152, so those kernels give no SM of the 152 a second CTA
// (whose warps would share sub-partitions and double the FP64 chain time).
__device__ __forceinline__ bool core_ij(const Lvl &L, int &bk, int &i, int &j) {
  const int2 t = L.ctiles[blockIdx.x];
  bk = t.x;
  const BlkDev &b = L.blk[bk];
  const int W = b.nx + 1, lin = t.y + (int)threadIdx.x;
  if (lin >= W * (b.ny + 1)) return false;
  i = lin % W;
  j = lin / W;
  return true;
}

// Reciprocal on the face and wavefront paths.  FP64: the hardware's
// approximate reciprocal (relative error e below 2^-19.9, measured over 4e7
// mantissas) refined by one third-order step of the series
// 1/x = r / (1 - e) = r (1 + e + e^2 + ...), e = 1 - x r taken exactly by an
// fma; the neglected e^3 is below 2^-59, so the result is within an ulp of
// the quotient in four dependent FP64 operations, against nine times that
// for a divide; a / b becomes a * rcp(b).  FP32: the division.
template <typename T>
__device__ __forceinline__ T rcp(T x);
template <>
__device__ __forceinline__ double rcp<double>(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
template <>
__device__ __forceinline__ float rcp<float>(float x) { return 1.0f / x; }

// 1/sqrt(x), x > 0, FP64: the hardware's approximate reciprocal square root
// (|x y^2 - 1| below 2^-19, measured over 4e7 samples) refined by one
// third-order step of the series (1 - e)^(-1/2) = 1 + e/2 + 3e^2/8 + ...,
// e = 1 - x y^2; within an ulp of 1/sqrt(x), and x times it within two ulps
// of sqrt(x) (measured), in six dependent FP64 operations.
__device__ __forceinline__ double rsqrt_d(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y * y, 1.0);
  return fma(y, e * fma(0.375, e, 0.5), y);
}
// sqrt(x), x > 0, on the face and primitive paths: FP64 x * rsqrt_d(x)
// (within two ulps of the rounded root, seven FP64 operations against about
// ten for the correctly rounded one); FP32 the square root
template <typename T>
__device__ __forceinline__ T sqrt_p(T x);
template <>
__device__ __forceinline__ double sqrt_p<double>(double x) { return x * rsqrt_d(x); }
template <>
__device__ __forceinline__ float sqrt_p<float>(float x) { return sqrtf(x); }

// FP64 arithmetic of the face, primitive and turbulence kernels.  An SM completes
// one FP64 warp instruction per 16 to 19 cycles, and each holds its sub-partition
// for 64, while that sub-partition could issue an integer or FP32 instruction
// every cycle: whatever needs no FP64 pipe is done beside it.
//   * reciprocals and reciprocal roots are formed in FP32 and integers altogether (a
//     divide takes about nine FP64 instructions, the hardware's 20-bit approximation with
//     a third-order step three for a reciprocal and five for a root);
//   * negation, powers of two and comparisons are integer operations.
// x 2^K, K in -3..1: exact; zeros, infinities and NaNs stay what they are, and so
// do values below 2^-1019
template <int K>
__device__ __forceinline__ double pow2(double x) {
  const int h = __double2hiint(x);
  const unsigned e = (unsigned)h & 0x7ff00000u;
  return __hiloint2double(e - 0x00400000u < 0x7fa00000u ? h + K * 0x00100000 : h, __double2loint(x));
}
__device__ __forceinline__ double half(double x) { return pow2<-1>(x); }
__device__ __forceinline__ double neg(double x) {
  return __hiloint2double(__double2hiint(x) ^ (int)0x80000000, __double2loint(x));
}
// Conversions between double and float, rounded to nearest even: a conversion
// instruction occupies the FP64 pipe as an FP64 instruction does (64 to 100 cycles), so
// values within the float's normal range are converted by integer operations.
template <typename T>
__device__ __forceinline__ T to(double x);
template <>
__device__ __forceinline__ double to<double>(double x) { return x; }
template <>
__device__ __forceinline__ float to<float>(double x) {
  const long long i = __double_as_longlong(x);
  const unsigned hi = (unsigned)(i >> 32), a = hi & 0x7fffffffu;
  const long long r = i + 0x0fffffffll + ((i >> 29) & 1);
  // 2^-126 <= |x| < 2^127, or zero
  if (a - 0x38100000u < 0x47e00000u - 0x38100000u)
    return __uint_as_float((((unsigned)(r >> 29) - (896u << 23)) & 0x7fffffffu) | (hi & 0x80000000u));
  return (i << 1) == 0 ? __uint_as_float(hi) : (float)x;
}
__device__ __forceinline__ double to_double(double x) { return x; }
__device__ __forceinline__ double to_double(float x) {
  const unsigned i = __float_as_uint(x), a = i & 0x7fffffffu;
  if (a - 0x00800000u < 0x7f800000u - 0x00800000u)
    return __hiloint2double((int)(((a >> 3) + (896u << 20)) | (i & 0x80000000u)), (int)(i << 29));
  return a == 0 ? __hiloint2double((int)i, 0) : (double)x;
}
// sign bit clear; x < y, x >= y and x > y for any x and a y of clear sign bit (false
// for a NaN x)
__device__ __forceinline__ bool sign_clear(double x) { return __double2hiint(x) >= 0; }
__device__ __forceinline__ bool below(double x, double y) {
  const long long i = __double_as_longlong(x);
  return i < __double_as_longlong(y) && (unsigned long long)i <= 0xfff0000000000000ull;
}
__device__ __forceinline__ bool at_least(double x, double y) {
  const long long i = __double_as_longlong(x);
  return i >= __double_as_longlong(y) && i <= 0x7ff0000000000000ll;
}
__device__ __forceinline__ bool above(double x, double y) {
  const long long i = __double_as_longlong(x);
  return i > __double_as_longlong(y) && i <= 0x7ff0000000000000ll;
}

// 1/x without the FP64 pipe.  In FP32: x's mantissa as a float and the float of its
// remaining bits, the approximate reciprocal r of the first, and the correction r
// (e + e^2), e = 1 - x r, added to r's double as an integer: 43 bits (FULL = false).
// Then a Newton step in integers: with the mantissas as 53-bit integers X and R the
// remainder 2^105 - X R is below 2^62, so it is known from the product modulo 2^64, and R
// times it, shifted, is added: half an ulp and 2^-17 more.  NaN for zero, subnormal,
// infinite or NaN x and from 2^1022.
template <bool FULL>
__device__ __forceinline__ double reciprocal(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const float xf = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | 0x3f800000u);
  const float xl = fmaf(__uint_as_float(((lo >> 6) & 0x7fffffu) | 0x3f800000u), 0x1p-23f, -0x1p-23f);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(xf));  // in (0.5, 1]
  const float e = fmaf(-xl, r, fmaf(-xf, r, 1.0f));
  // the correction in units of 2^-43, rounded by the float that has its last bit there
  const int q = __float_as_int(fmaf(r * 0x1p43f, fmaf(e, e, e), 0x1.8p23f)) - 0x4b400000;
  const unsigned rb = __float_as_uint(r), ex = hi & 0x7ff00000u;
  // 1/x of the mantissa as a double's bits with the float's exponent bias (units of
  // 2^-53 below 1, so that the sum is right on both sides of 1)
  unsigned long long y = (((unsigned long long)(rb >> 3) << 32) | (rb << 29)) + (unsigned long long)((long long)q << 10);
  if (FULL) {
    const unsigned Rl = (unsigned)y, Rh = (unsigned)(y >> 32) - (125u << 20);  // 2^53 r
    const unsigned Xh = (hi & 0xfffffu) | 0x100000u;                           // 2^52 x
    const unsigned ph = __umulhi(lo, Rl) + lo * Rh + Xh * Rl;  // bits 32 to 63 of X R
    const int c = (__mulhi((int)~ph, (int)__funnelshift_l(Rl, Rh, 9)) + (1 << 17)) >> 18;
    y += (unsigned long long)(long long)c;
  }
  const unsigned bias = ((1023u - 127u) << 20) + 0x3ff00000u - ex + (hi & 0x80000000u);
  return __hiloint2double(ex - 0x00100000u < 0x7fc00000u ? (int)((unsigned)(y >> 32) + bias) : 0x7ff80000, (int)(unsigned)y);
}
__device__ __forceinline__ double rcp_seed(double x) { return reciprocal<false>(x); }
// 1/sqrt(x) the same way: the exponent made even, r the FP32 approximate reciprocal root
// of the mantissa m in [1, 4), e = 1 - m r^2, and r (1 + e/2 + 3/8 e^2).  FULL = false: e in
// FP32, 43 bits.  FULL: with A = 2^24 r and X the 53-bit mantissa, e is -X A^2 modulo 2^96 (known
// to 2^-67 from four 32-bit products), r e/2 is A times it, shifted; only the term
// in e^2 is FP32: half an ulp and 2^-8 more.
// NaN for negative, infinite or NaN x; for zero (and subnormal x) NaN or, ZERO, 1,
// so that x times the root is zero.
template <bool ZERO, bool FULL>
__device__ __forceinline__ double rsqrt_x(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned odd = (hi & 0x00100000u) ? 0u : 1u;  // biased exponent even: mantissa in [2, 4)
  const float xf = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | (odd ? 0x40000000u : 0x3f800000u));
  const float ul = odd ? 0x1p-22f : 0x1p-23f;
  const float xl = fmaf(__uint_as_float(((lo >> 6) & 0x7fffffu) | 0x3f800000u), ul, -ul);
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(xf));  // in (0.5, 1]
  const float r2 = r * r, r2l = fmaf(r, r, -r2);
  const float e = fmaf(-xl, r2, fmaf(-xf, r2l, fmaf(-xf, r2, 1.0f)));
  const unsigned rb = __float_as_uint(r);
  unsigned long long y = ((unsigned long long)(rb >> 3) << 32) | (rb << 29);  // 2^53 r
  if (FULL) {
    const unsigned A = rb - (125u << 23), Xh = (hi & 0xfffffu) | 0x100000u;
    const unsigned long long S = (unsigned long long)A * A;
    const unsigned Sl = (unsigned)S, Sh = (unsigned)(S >> 32);
    // bits 32 to 95 of X A^2: 2^(68 - odd) (1 - e) modulo 2^64
    const unsigned long long M = (unsigned long long)Xh * Sl + (unsigned long long)lo * Sh + __umulhi(lo, Sl) +
                                 ((unsigned long long)(Xh * Sh) << 32);
    const long long E = -(long long)M;
    const long long c = (long long)(int)A * (int)(E >> 32) + (long long)__umulhi(A, (unsigned)E);  // 2^(8 - odd) r e/2
    const int q = __float_as_int(fmaf(r * (odd ? 0x1.8p58f : 0x1.8p59f), e * e, 0x1.8p23f)) - 0x4b400000;  // r 3/8 e^2
    const int sh = 8 - (int)odd;
    y += (unsigned long long)((c + q + (1 << (sh - 1))) >> sh);
  } else {
    const int q = __float_as_int(fmaf(r * 0x1p43f, e * fmaf(0.375f, e, 0.5f), 0x1.8p23f)) - 0x4b400000;
    y += (unsigned long long)((long long)q << 10);
  }
  // x = m 4^k with k = (exponent - odd) / 2 of the unbiased exponent
  const int k = ((int)(hi >> 20) - 1023 - (int)odd) >> 1;
  const unsigned bias = ((1023u - 127u) << 20) - ((unsigned)k << 20);
  const int out = ZERO && (hi & 0x7ff00000u) == 0 ? 0x3ff00000 : 0x7ff80000;
  return __hiloint2double(hi - 0x00100000u < 0x7fe00000u ? (int)((unsigned)(y >> 32) + bias) : out, (int)(unsigned)y);
}

__device__ __forceinline__ double recip(double x) { return reciprocal<true>(x); }
// 1/x where x may be zero or infinite: by the divide there
__device__ __forceinline__ double recip_any(double x) {
  return ((unsigned)__double2hiint(x) & 0x7ff00000u) - 0x00100000u < 0x7fc00000u ? recip(x) : 1.0 / x;
}
// a / b, y = rcp_seed(b): from q = a y the remainder a - b q, exact by an fma, gives the
// quotient's last bits (the rounded quotient in all of 8e8 samples): three FP64 instructions,
// and one seed serves every quotient by b.  NaN for infinite a.
__device__ __forceinline__ double quot(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}
// the same with infinities (of a, or of the quotient), picked by an integer compare
__device__ __forceinline__ double quot_any(double a, double b, double y) {
  const double q = a * y, r = fma(fma(-b, q, a), y, q);
  return ((unsigned)__double2hiint(q) & 0x7ff00000u) == 0x7ff00000u ? q : r;
}
// max(x, 0) and min(x, 0) by the sign (a NaN goes to one of them)
__device__ __forceinline__ double pos_part(double x) { return __double2hiint(x) >= 0 ? x : 0.0; }
__device__ __forceinline__ double neg_part(double x) { return __double2hiint(x) < 0 ? x : 0.0; }

// 1/sqrt(x), x > 0
__device__ __forceinline__ double rroot(double x) { return rsqrt_x<false, true>(x); }
// sqrt(x) = x / sqrt(x), within an ulp of the rounded root
__device__ __forceinline__ double root(double x) { return x * rsqrt_x<true, true>(x); }
// the square root function where x is not a positive normal number (T < 0: NaN)
__device__ __forceinline__ double root_t(double x) {
  return (unsigned)__double2hiint(x) - 0x00100000u < 0x7fe00000u ? root(x) : sqrt(x);
}
// sqrt(a / b) = |a| / sqrt(a b): no reciprocal; to two ulps
__device__ __forceinline__ double root_ratio(double a, double b) { return fabs(a) * rsqrt_x<true, true>(a * b); }

// the rounded quotient and root in three FP64 instructions where the operands are of
// ordinary size (2^-400 to 2^400), by the divide and the square root function elsewhere
__device__ __forceinline__ bool ordinary(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) - ((1023u - 400u) << 20) < (800u << 20);
}
__device__ __forceinline__ double div_r(double a, double b) {
  return ordinary(a) && ordinary(b) ? quot(a, b, rcp_seed(b)) : a / b;
}
// (from g = x y, y to 43 bits, the remainder x - g^2, exact by an fma, gives the last bits)
__device__ __forceinline__ double sqrt_r(double x) {
  if (!(ordinary(x) && sign_clear(x))) return sqrt(x);
  const double y = rsqrt_x<false, false>(x), g = x * y;
  return fma(half(y), fma(-g, g, x), g);
}
// tanh(x), x >= 0: 1 from 22 on, as the function gives it
__device__ __forceinline__ double tanh_pos(double x) { return at_least(x, 22.0) ? 1.0 : tanh(x); }

// the gas constants of a case in the arithmetic of a face
struct Gas {
  double g, gm1, ggm1, rgm1, rg;  // gamma, gamma - 1, gamma / (gamma - 1), 1 / (gamma - 1), 1 / gamma
};
__device__ __forceinline__ Gas gas(const CaseDev &c) {
  return {c.gamma, c.gm1, c.ggm1, c.rgm1, c.rg};
}

// The face physics of FP64 contexts (ec2d_mixed.cuh: of contexts with FP32 parts).

// ---- reconstruction, sub_Residual.f90:477-659 --------------------------------
// zero where a b <= 0, else the one of smaller magnitude, by integer compares
__device__ __forceinline__ double minmod(double a, double b) {
  const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  const long long ax = x & 0x7fffffffffffffffll, ay = y & 0x7fffffffffffffffll, inf = 0x7ff0000000000000ll;
  if (ax > inf || ay > inf) return b;  // a NaN: as the comparisons of doubles take it
  if ((x ^ y) < 0 || ax == 0 || ay == 0) return 0.0;
  return ax <= ay ? a : b;
}

// scheme_fP and scheme_fm (sub_Residual.f90:591-659): the left and right state
// at the face between u2 and u3.  Both sides in one pass over the three
// differences; every scheme is u2 (u3) plus a correction, in the same formulas as the
// reference with one reciprocal in place of its divides.
__device__ __forceinline__ void scheme_pair(double u1, double u2, double u3, double u4, int flag, double &l, double &r) {
  const double ep = 1.0e-6, k3 = 1.0 / 3.0;
  const double d1 = u2 - u1, d2 = u3 - u2, d3 = u4 - u3;
  switch (flag) {
    case Scheme_UD1: l = u2; r = u3; return;
    case Scheme_UD3:
      l = (-u1 + 5.0 * u2 + 2.0 * u3) * (1.0 / 6.0);
      r = (2.0 * u2 + 5.0 * u3 - u4) * (1.0 / 6.0);
      return;
    case Scheme_NND2:
      l = u2 + half(minmod(d1, d2));
      r = u3 - half(minmod(d2, d3));
      return;
    case Scheme_WENO3: {
      // weights a_1 / (a_1 + a_2), a_2 / (a_1 + a_2) with a_1 = 1 / (3 q_1), a_2 = 2 / (3 q_2)
      // over the common denominator q_2 + 2 q_1, q_k = (ep + d_k^2)^2 >= 1e-12
      const double e1 = fma(d1, d1, ep), e2 = fma(d2, d2, ep), e3 = fma(d3, d3, ep);
      const double q1 = pow2<1>(e1 * e1), q2 = e2 * e2, q3 = pow2<1>(e3 * e3);
      l = fma(half(fma(q1, d2, q2 * d1)), recip(q1 + q2), u2);
      r = fma(-(half(fma(q3, d2, q2 * d3))), recip(q3 + q2), u3);
      return;
    }
    case Scheme_MUSCL2: {  // left: k = 1, b = 2; right: k = 1/3, b = 1
      l = u2 + half(minmod(d2, pow2<1>(d1)));
      const double k = 1.0 / 3.0, m = minmod(d3, d2);
      r = u3 - pow2<-2>((1.0 - k) * m + (1.0 + k) * minmod(d2, d3));
      return;
    }
    case Scheme_MUSCL3: {
      // s ((1 - k s) um + (1 + k s) up) / 4 = s ((um + up) + k s (up - um)) / 4, van
      // Albada's s = (2 up um + ep) / (up^2 + um^2 + ep); on the right up and um change
      // places
      const double e2 = fma(d2, d2, ep), t2 = pow2<1>(d2);
      double s = fma(t2, d1, ep) * recip(fma(d1, d1, e2));
      l = fma(pow2<-2>(s), fma(k3 * s, d2 - d1, u3 - u1), u2);
      s = fma(t2, d3, ep) * recip(fma(d3, d3, e2));
      r = fma(-(pow2<-2>(s)), fma(k3 * s, d2 - d3, u4 - u2), u3);
      return;
    }
    case Scheme_OMUSCL2: {
      double r1 = (d1 + ep) / (d2 + ep), r2 = (d2 + ep) / (d3 + ep);
      double f1 = 0.8 - 0.175 / r2 + 0.375 * r1;
      double f = fmax(0.0, fmin(fmin(2.0, f1), 2.0 * r1));
      l = u2 + 0.5 * f * d2;
      r1 = (d3 + ep) / (d2 + ep);
      r2 = (d2 + ep) / (d1 + ep);
      f1 = 0.8 - 0.175 / r2 + 0.375 * r1;
      f = fmax(0.0, fmin(fmin(2.0, f1), 2.0 * r1));
      r = u3 - 0.5 * f * d2;
      return;
    }
  }
  l = r = 0.0;
}

// The same MUSCL3 states from one cell: van Albada's s and both corrections depend on the
// cell's differences dm and dp alone.  a: to its upper face (left state u + a), b: to its
// lower face (right state u - b).
__device__ __forceinline__ void muscl3_slopes(double dm, double dp, double &a, double &b) {
  const double ep = 1.0e-6;
  const double s = fma(pow2<1>(dp), dm, ep) * recip(fma(dm, dm, fma(dp, dp, ep)));
  const double ks = (1.0 / 3.0) * s, sum = dm + dp, w = dp - dm;
  a = pow2<-2>(s) * fma(ks, w, sum);
  b = fma(half(s), sum, -a);  // s/4 (sum - ks w)
}

// conservative (rho, rho u, rho v, E) -> primitive (rho, u, v, p), as at the
// end of Reconstuction_conservative/Characteristic (sub_Residual.f90:526-527)
__device__ __forceinline__ void cons_to_prim(const double Q[4], double W[4], double gm1) {
  const double r = recip(Q[0]);
  W[0] = Q[0];
  W[1] = Q[1] * r;
  W[2] = Q[2] * r;
  W[3] = (Q[3] - half(fma(W[2], Q[2], W[1] * Q[1]))) * gm1;
}

// S0[k][m]: stencil points k = i-2..i+1 (or j-2..j+1), variable m.
// Reconstuction_original/conservative/Characteristic (sub_Residual.f90:505-586)
__device__ __forceinline__ void reconstruct(int recon, int scheme, double S0[4][4], const Gas &G, double UL[4], double UR[4]) {
  if (recon == Recon_Original) {
#pragma unroll
    for (int m = 0; m < 4; m++) scheme_pair(S0[0][m], S0[1][m], S0[2][m], S0[3][m], scheme, UL[m], UR[m]);
    return;
  }
  double QL[4], QR[4];
  if (recon == Recon_Conservative) {
#pragma unroll
    for (int m = 0; m < 4; m++) scheme_pair(S0[0][m], S0[1][m], S0[2][m], S0[3][m], scheme, QL[m], QR[m]);
    cons_to_prim(QL, UL, G.gm1);
    cons_to_prim(QR, UR, G.gm1);
    return;
  }
  // characteristic: project on the left eigenvectors at the arithmetic
  // mid-state, limit each characteristic variable, project back
  double Uh[4];
#pragma unroll
  for (int m = 0; m < 4; m++) Uh[m] = half(S0[1][m] + S0[2][m]);
  const double rd = recip(Uh[0]), u1 = Uh[1] * rd, v1 = Uh[2] * rd;
  const double p1 = (Uh[3] - half(fma(Uh[2], v1, Uh[1] * u1))) * G.gm1;
  // sound speed c1 and its inverse from c^2 = gamma p / rho
  const double c2 = G.g * p1 * rd;
  const double c1 = root(c2), ic = c1 * recip(c2);
  const double V2 = half(fma(v1, v1, u1 * u1));
  const double tmp1 = G.gm1 * ic, tmp3 = tmp1 * ic, tmp5 = half(ic), tmp0 = c2 * G.rgm1;
  const double a0 = V2 - tmp0, vt = V2 * tmp1, ut = tmp1 * u1, wt = tmp1 * v1;
  double V0[4][4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double *S = S0[k];
    V0[k][0] = fma(a0, S[0], fma(-u1, S[1], fma(-v1, S[2], S[3])));
    V0[k][1] = fma(-v1, S[0], S[2]);
    // the two acoustic rows share everything but a sign
    const double e = fma(vt, S[0], fma(-ut, S[1], fma(-wt, S[2], tmp1 * S[3])));
    const double o = fma(-u1, S[0], S[1]);
    V0[k][2] = o - e;
    V0[k][3] = o + e;
  }
  double VL[4], VR[4];
#pragma unroll
  for (int m = 0; m < 4; m++) scheme_pair(V0[0][m], V0[1][m], V0[2][m], V0[3][m], scheme, VL[m], VR[m]);
#pragma unroll
  for (int side = 0; side < 2; side++) {
    const double *V = side ? VR : VL;
    double *Q = side ? QR : QL;
    // back: with e = -tmp3 V0 (entropy), s = V2 + V3, d = (V3 - V2) tmp5
    const double e = -(tmp3 * V[0]), sum = V[2] + V[3], dif = (V[3] - V[2]) * tmp5, r0 = e + dif;
    Q[0] = r0;
    Q[1] = fma(u1, r0, half(sum));
    Q[2] = fma(v1, r0, V[1]);
    Q[3] = fma(V2, r0, fma(v1, V[1], fma(u1, half(sum), tmp0 * dif)));
  }
  cons_to_prim(QL, UL, G.gm1);
  cons_to_prim(QR, UR, G.gm1);
}

// ---- face fluxes -------------------------------------------------------------
// Roe and AUSM+ take the primitive states (rho, u, v, p) as they are and give
// F = -s (flux through the face with unit normal n and length s): the reference
// turns the states into the face's frame and the flux back, which multiplies
// out to the same sums (16 FP64 instructions less).
// Flux_Roe_1D, sub_flux_split.f90:265-324 (Harten entropy fix, delta = 0.1)
__device__ __forceinline__ double harten(double l) {
  const double delt = 0.1, i2d = 1.0 / (2.0 * delt);
  if (below(l, delt)) l = fma(l, l, delt * delt) * i2d;
  return l;
}
__device__ __forceinline__ void flux_roe(const double *L, const double *R, double n1, double n2, double s, double *F, const Gas &G) {
  const double dl = L[0], ul = L[1], vl = L[2], pl = L[3], dr = R[0], ur = R[1], vr = R[2], pr = R[3];
  const double unl = fma(vl, n2, ul * n1), unr = fma(vr, n2, ur * n1);
  const double hl = fma(G.ggm1 * pl, recip(dl), half(fma(vl, vl, ul * ul)));
  const double hr = fma(G.ggm1 * pr, recip(dr), half(fma(vr, vr, ur * ur)));
  // Roe averages: t = sqrt(rho_r / rho_l)
  const double t = root_ratio(dr, dl), t1 = t + 1.0, inv = recip(t1);
  const double ad = pow2<-2>(dl * (t1 * t1));
  const double au = fma(t, ur, ul) * inv, av = fma(t, vr, vl) * inv, ah = fma(t, hr, hl) * inv;
  const double an = fma(av, n2, au * n1), at = fma(av, n1, -(au * n2));  // normal and tangential
  const double k2 = half(fma(av, av, au * au));
  const double c2 = G.gm1 * (ah - k2);
  const double c = root(c2), ic2 = recip(c2), ic = c * ic2;
  const double l0 = harten(fabs(an - c)), l1 = harten(fabs(an)), l3 = harten(fabs(an + c));
  const double dp = pr - pl, du = ur - ul, dv = vr - vl;
  const double x = (ad * c) * (unr - unl), i2 = half(ic2);
  const double w0 = l0 * ((dp - x) * i2), w3 = l3 * ((dp + x) * i2), w1 = l1 * fma(-dp, ic2, dr - dl);
  const double w2 = l1 * (ad * fma(dv, n1, -(du * n2)) * ic);
  // with S = w0 + w1 + w3 and q = (w3 - w0) c the dissipation is (S, S u + q n1 - w2 n2,
  // S v + q n2 + w2 n1, (w0 + w3) h + q u_n + w1 |u|^2 / 2 + w2 u_t)
  const double w03 = w0 + w3, S = w03 + w1, q = (w3 - w0) * c;
  const double ml = dl * unl, mr = dr * unr, pp = (pl + pr) - q, hs = neg(half(s));
  F[0] = ((ml + mr) - S) * hs;
  F[1] = fma(ml, ul, fma(mr, ur, fma(-S, au, fma(pp, n1, w2 * n2)))) * hs;
  F[2] = fma(ml, vl, fma(mr, vr, fma(-S, av, fma(pp, n2, -(w2 * n1))))) * hs;
  F[3] = (fma(ml, hl, mr * hr) - fma(w03, ah, fma(q, an, fma(w1, k2, w2 * at)))) * hs;
}

// Flux_Ausm_1Da (AUSM+), sub_flux_split.f90:195-261.  Its sums 0.5 xm (f_l + f_r) -
// 0.5 dm (f_r - f_l) with dm = a |M| rho of the upwind side are xm times f of the
// upwind side, so only that side's enthalpy is formed.
__device__ __forceinline__ bool supersonic(double m) {  // 1 <= |m| < infinity
  return ((unsigned)__double2hiint(m) & 0x7fffffffu) - 0x3ff00000u < 0x40000000u;
}
// split Mach number and pressure of the left state; the right state's are -m4(-M)
// and p5(-M)
__device__ __forceinline__ void ausm_split(double m, double &m4, double &p5) {
  if (supersonic(m)) {
    m4 = sign_clear(m) ? m : 0.0;
    p5 = sign_clear(m) ? 1.0 : 0.0;
    return;
  }
  const double a = m + 1.0, q = pow2<-2>(a * a), r = fma(m, m, -1.0), w = r * r;
  m4 = fma(0.125, w, q);
  p5 = fma(0.1875 * m, w, q * (2.0 - m));
}
__device__ __forceinline__ void flux_ausm(const double *L, const double *R, double n1, double n2, double s, double *F, const Gas &G) {
  const double unl = fma(L[2], n2, L[1] * n1), unr = fma(R[2], n2, R[1] * n1);
  const double al = root_ratio(G.g * L[3], L[0]), ar = root_ratio(G.g * R[3], R[0]);
  const double a = half(al + ar), ia = recip(a);
  double m4, p5, n4, q5;
  ausm_split(unl * ia, m4, p5);
  ausm_split(-(unr * ia), n4, q5);
  const double M = m4 - n4;
  const bool left = sign_clear(M);
  const double d = left ? L[0] : R[0], u = left ? L[1] : R[1], v = left ? L[2] : R[2], c = left ? al : ar;
  const double ns = neg(s), xm = (a * M) * (d * ns), p = fma(L[3], p5, R[3] * q5) * ns;
  const double h = fma(c * c, G.rgm1, half(fma(v, v, u * u)));
  F[0] = xm;
  F[1] = fma(xm, u, p * n1);
  F[2] = fma(xm, v, p * n2);
  F[3] = xm * h;
}

// The other fluxes in the face's frame: rotated primitive states (rho, u_n, u_t, p).
// Flux_Van_Leer_1Da, sub_flux_split.f90:139-189
__device__ __forceinline__ void flux_vanleer(const double *QL, const double *QR, double *F, const Gas &G) {
  double dl = QL[0], uul = QL[1], vvl = QL[2], pl = QL[3];
  double dr = QR[0], uur = QR[1], vvr = QR[2], pr = QR[3];
  const double gamma = G.g, gm1 = G.gm1, rg = G.rg, rgg = recip(gamma * gamma - 1.0);
  double al = root_ratio(gamma * pl, dl), ar = root_ratio(gamma * pr, dr);
  double fp0 = 0, fp1 = 0, fp2 = 0, fp3 = 0, fm0 = 0, fm1 = 0, fm2 = 0, fm3 = 0;
  if (uul >= al) {
    fp0 = dl * uul; fp1 = dl * uul * uul + pl; fp2 = dl * uul * vvl;
    fp3 = uul * (G.ggm1 * pl + 0.5 * dl * (uul * uul + vvl * vvl));
  } else if (fabs(uul) < al) {
    const double Ml = uul * recip(al);
    double tmp0 = dl * al * (0.25 * (1.0 + Ml) * (1.0 + Ml));
    double w = gm1 * uul + 2.0 * al;
    fp0 = tmp0; fp1 = tmp0 * w * rg; fp2 = tmp0 * vvl;
    fp3 = tmp0 * 0.5 * (w * w * rgg + vvl * vvl);
  }
  if (uur >= ar) {
  } else if (fabs(uur) < ar) {
    const double Mr = uur * recip(ar);
    double tmp0 = dr * ar * (-0.25 * (Mr - 1.0) * (Mr - 1.0));
    double w = gm1 * uur - 2.0 * ar;
    fm0 = tmp0; fm1 = tmp0 * w * rg; fm2 = tmp0 * vvr;
    fm3 = tmp0 * 0.5 * (w * w * rgg + vvr * vvr);
  } else if (uur <= -ar) {
    fm0 = dr * uur; fm1 = dr * uur * uur + pr; fm2 = dr * uur * vvr;
    fm3 = uur * (G.ggm1 * pr + 0.5 * dr * (uur * uur + vvr * vvr));
  }
  F[0] = fp0 + fm0; F[1] = fp1 + fm1; F[2] = fp2 + fm2; F[3] = fp3 + fm3;
}

// Flux_steger_warming_1Da, sub_flux_split.f90:99-136
__device__ __forceinline__ void flux_sw(const double *QL, const double *QR, double *F, const Gas &G) {
  double dl = QL[0], uul = QL[1], vvl = QL[2], pl = QL[3];
  double dr = QR[0], uur = QR[1], vvr = QR[2], pr = QR[3];
  const double gamma = G.g, gm1 = G.gm1;
  double al = root_ratio(gamma * pl, dl), ar = root_ratio(gamma * pr, dr);
  double tmp1 = 2.0 * gm1, tmp3 = 0.5 * (3.0 - gamma) * G.rgm1;
  double E1P = (uul + fabs(uul)) * 0.5, E2P = (uul - al + fabs(uul - al)) * 0.5, E3P = (uul + al + fabs(uul + al)) * 0.5;
  double t0 = dl * 0.5 * G.rg;
  double p0 = t0 * (tmp1 * E1P + E2P + E3P);
  double p1 = t0 * (tmp1 * E1P * uul + E2P * (uul - al) + E3P * (uul + al));
  double p2 = t0 * (tmp1 * E1P * vvl + E2P * vvl + E3P * vvl);
  double p3 = t0 * (E1P * gm1 * (uul * uul + vvl * vvl) + E2P * ((uul - al) * (uul - al) + vvl * vvl) * 0.5 +
                    E3P * ((uul + al) * (uul + al) + vvl * vvl) * 0.5 + tmp3 * al * al * (E2P + E3P));
  double E1M = (uur - fabs(uur)) * 0.5, E2M = (uur - ar - fabs(uur - ar)) * 0.5, E3M = (uur + ar - fabs(uur + ar)) * 0.5;
  t0 = dr * 0.5 * G.rg;
  double m0 = t0 * (tmp1 * E1M + E2M + E3M);
  double m1 = t0 * (tmp1 * E1M * uur + E2M * (uur - ar) + E3M * (uur + ar));
  double m2 = t0 * (tmp1 * E1M * vvr + E2M * vvr + E3M * vvr);
  double m3 = t0 * (E1M * gm1 * (uur * uur + vvr * vvr) + E2M * ((uur - ar) * (uur - ar) + vvr * vvr) * 0.5 +
                    E3M * ((uur + ar) * (uur + ar) + vvr * vvr) * 0.5 + tmp3 * ar * ar * (E2M + E3M));
  F[0] = p0 + m0; F[1] = p1 + m1; F[2] = p2 + m2; F[3] = p3 + m3;
}

// Flux_HLL_HLLC_1D, sub_flux_split.f90:16-93
__device__ __forceinline__ void flux_hll(const double *QL, const double *QR, double *F, const Gas &G, bool hllc) {
  double dl = QL[0], uul = QL[1], vvl = QL[2], pl = QL[3];
  double dr = QR[0], uur = QR[1], vvr = QR[2], pr = QR[3];
  double UL[4] = {dl, dl * uul, dl * vvl, pl * G.rgm1 + dl * half(uul * uul + vvl * vvl)};
  double UR[4] = {dr, dr * uur, dr * vvr, pr * G.rgm1 + dr * half(uur * uur + vvr * vvr)};
  double al = root_ratio(G.g * pl, dl), ar = root_ratio(G.g * pr, dr);
  double p_pvrs = half(pl + pr) - (uur - uul) * (dl + dr) * pow2<-3>(al + ar);
  double p_star = fmax(0.0, p_pvrs);
  const double g2 = half((G.g + 1.0) * G.rg);
  double qql = (p_star <= pl) ? 1.0 : root(fma(g2, p_star * recip(pl) - 1.0, 1.0));
  double qqr = (p_star <= pr) ? 1.0 : root(fma(g2, p_star * recip(pr) - 1.0, 1.0));
  double Sl = uul - al * qql, Sr = uur + ar * qqr;
  double Fl[4] = {UL[1], UL[1] * uul + pl, UL[2] * uul, uul * (UL[3] + pl)};
  double Fr[4] = {UR[1], UR[1] * uur + pr, UR[2] * uur, uur * (UR[3] + pr)};
  if (!hllc) {
    if (Sl >= 0) { for (int m = 0; m < 4; m++) F[m] = Fl[m]; }
    else if (Sr <= 0) { for (int m = 0; m < 4; m++) F[m] = Fr[m]; }
    else { double inv = recip(Sr - Sl);
      for (int m = 0; m < 4; m++) F[m] = (Sr * Fl[m] - Sl * Fr[m] + Sl * Sr * (UR[m] - UL[m])) * inv; }
    return;
  }
  const double bl = dl * (Sl - uul), br = dr * (Sr - uur);
  double S_star = (pr - pl + bl * uul - br * uur) * recip(bl - br);
  if (Sl >= 0) { for (int m = 0; m < 4; m++) F[m] = Fl[m]; return; }
  if (Sr <= 0) { for (int m = 0; m < 4; m++) F[m] = Fr[m]; return; }
  // the star state of the side the face lies in
  const bool left = S_star >= 0;
  double U[4], Fs[4];
#pragma unroll
  for (int m = 0; m < 4; m++) { U[m] = left ? UL[m] : UR[m]; Fs[m] = left ? Fl[m] : Fr[m]; }
  const double u = left ? uul : uur, v = left ? vvl : vvr, p = left ? pl : pr, b = left ? bl : br, S = left ? Sl : Sr;
  // E / rho + (S* - u) (S* + p / b) over one reciprocal of rho b
  const double d = U[0], rdb = recip(d * b);
  const double ts = b * recip(S - S_star);
  const double e = U[3] * (b * rdb) + (S_star - u) * (S_star + p * (d * rdb));
  F[0] = Fs[0] + S * (ts - d);
  F[1] = Fs[1] + S * (ts * S_star - U[1]);
  F[2] = Fs[2] + S * (ts * v - U[2]);
  F[3] = Fs[3] + S * (ts * e - U[3]);
}

// F = -s (flux through the face with unit normal n and length s)
__device__ __forceinline__ void face_flux(int iflux, const double *L, const double *R, double n1, double n2, double s, double *F, const Gas &G) {
  if (iflux == Flux_Roe) { flux_roe(L, R, n1, n2, s, F, G); return; }
  if (iflux == Flux_Ausm) { flux_ausm(L, R, n1, n2, s, F, G); return; }
  const double QL[4] = {L[0], L[1] * n1 + L[2] * n2, -L[1] * n2 + L[2] * n1, L[3]};
  const double QR[4] = {R[0], R[1] * n1 + R[2] * n2, -R[1] * n2 + R[2] * n1, R[3]};
  double f[4] = {0.0, 0.0, 0.0, 0.0};
  switch (iflux) {
    case Flux_VanLeer: flux_vanleer(QL, QR, f, G); break;
    case Flux_SW: flux_sw(QL, QR, f, G); break;
    case Flux_HLL: flux_hll(QL, QR, f, G, false); break;
    case Flux_HLLC: flux_hll(QL, QR, f, G, true); break;
  }
  const double ns = neg(s);
  F[0] = f[0] * ns;
  F[1] = (f[1] * n1 - f[2] * n2) * ns;
  F[2] = (f[1] * n2 + f[2] * n1) * ns;
  F[3] = f[3] * ns;
}

// viscous stress and heat flux through a face from the face-local 2x2
// Jacobian of cell centres, sub_Residual.f90:313-343 / 419-450
__device__ __forceinline__ void viscous_face(double Dix, double Diy, double Djx, double Djy, double Diu, double Div,
                                             double DiT, double Dju, double Djv, double DjT, double Amu1, double Amk1,
                                             double u1, double v1, double n1, double n2, double s, double &F2,
                                             double &F3, double &F4) {
  double Ds = rcp(Dix * Djy - Djx * Diy);
  double ux = (Diu * Djy - Dju * Diy) * Ds, vx = (Div * Djy - Djv * Diy) * Ds, Tx = (DiT * Djy - DjT * Diy) * Ds;
  double uy = (-Diu * Djx + Dju * Dix) * Ds, vy = (-Div * Djx + Djv * Dix) * Ds, Ty = (-DiT * Djx + DjT * Dix) * Ds;
  double t11 = ((4.0 / 3.0) * ux - (2.0 / 3.0) * vy) * Amu1;
  double t22 = ((4.0 / 3.0) * vy - (2.0 / 3.0) * ux) * Amu1;
  double t12 = (uy + vx) * Amu1;
  double E1 = u1 * t11 + v1 * t12 + Amk1 * Tx, E2 = u1 * t12 + v1 * t22 + Amk1 * Ty;
  F2 += (t11 * n1 + t12 * n2) * s;
  F3 += (t12 * n1 + t22 * n2) * s;
  F4 += (E1 * n1 + E2 * n2) * s;
}

// The same from the face's four metric coefficients formed at set-up
// (G_VIP..G_VIS, k_face_metrics), which give the derivatives of a quantity q
// across the face and along it from its differences: d_n q = Diq P + Djq Q,
// d_t q = Djq S - Diq R (a factor 1/4 of the averaged differences is in the
// coefficients).  In the frame of the face the stress on it is
//   F_x = mu (d_n u - d_t v + n1 div / 3),  F_y = mu (d_n v + d_t u + n2 div / 3),
//   div = n1 (d_n u + d_t v) + n2 (d_n v - d_t u),
// the same sums as (t11 n1 + t12 n2, t12 n1 + t22 n2), and the work and heat
// u F_x + v F_y + k d_n T.  us, vs: the sums of the velocities of both sides; mu
// and k already hold the face length.
__device__ __forceinline__ void viscous_face_m(double P, double Q, double R, double S, double Diu, double Div, double DiT, double Dju, double Djv, double DjT, double mu, double k,
                                               double us, double vs, double n1, double n2, double &F2, double &F3, double &F4) {
  const double nu = fma(Diu, P, Dju * Q), nv = fma(Div, P, Djv * Q);
  const double tu = fma(Dju, S, -(Diu * R)), tv = fma(Djv, S, -(Div * R));
  const double d3 = fma(n1, nu + tv, n2 * (nv - tu)) * (1.0 / 3.0);
  const double fx = fma(n1, d3, nu - tv), fy = fma(n2, d3, nv + tu);
  F2 = fma(fx, mu, F2);
  F3 = fma(fy, mu, F3);
  F4 = fma(fma(us, fx, vs * fy), half(mu), F4);
  F4 = fma(fma(DiT, P, DjT * Q), k, F4);
}

// device-side error record (first error of a case wins)
__device__ __forceinline__ void set_status(int *st, int code, int blk, int i, int j) {
  if (atomicCAS(st, 0, code) == 0) { st[1] = blk; st[2] = i; st[3] = j; }
}

}  // namespace ec2d
