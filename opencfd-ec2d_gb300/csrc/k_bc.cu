// k_bc.cu -- ghost cells: physical boundary conditions (sub_boundary.f90:10-34,
// 306-581), block-interface halo copy and ghost-corner extrapolation
// (update_buffer_onemesh, sub_boundary.f90:45-153), and the nu~/k/omega
// clip (force_vt_kw, sub_NS_singlegrid.f90:30-60).
//
// Write order.  The reference runs every physical subface of every block in
// (block, subface) order, then per block its halo copies followed by its four
// ghost corners.  A physical subface loops over node indices ist..iend,
// jst..jend, so its end points write ghost rows that later subfaces read.
// The write sets of one subface never overlap its read set, halo copies read
// only interior cells, and corners read only the block's own ghosts.  Hence
// one cluster per block reproduces the reference exactly: subfaces of phase 1 in
// order with a barrier between them, all halo items of phase 2 in parallel,
// then the corners.  Physical subfaces whose read and write sets do not meet
// those of any earlier subface of the block share a barrier phase (the
// grouping is computed at set-up from the index rectangles).
#include "ec2d_dev.cuh"
#include "ec2d_internal.h"

namespace ec2d {

__device__ __forceinline__ void ghost_pair(int face, int i, int j, int k, int &i1, int &j1, int &i2, int &j2) {
  if (face == 1) { i1 = i + k - 1; j1 = j; i2 = i - k; j2 = j; }
  else if (face == 2) { i1 = i; j1 = j + k - 1; i2 = i; j2 = j - k; }
  else if (face == 3) { i1 = i - k; j1 = j; i2 = i + k - 1; j2 = j; }
  else { i1 = i; j1 = j - k; i2 = i; j2 = j + k - 1; }
}

// the nvar variables of a cell, all loads in flight before the first use (a store between
// them would hold each load back: the compiler cannot tell the two cells apart)
struct Cell { double v[6]; };
__device__ __forceinline__ Cell load_cell(const Lvl &L, long long id) {
  Cell c;
#pragma unroll
  for (int m = 0; m < 6; m++) c.v[m] = m < L.nvar ? L.U[m * L.F + id] : 0.0;
  return c;
}
__device__ __forceinline__ void store_cell(const Lvl &L, long long id, const Cell &c) {
#pragma unroll
  for (int m = 0; m < 6; m++)
    if (m < L.nvar) L.U[m * L.F + id] = c.v[m];
}

// boundary_wall, sub_boundary.f90:306-386
__device__ __forceinline__ void bc_wall(const Lvl &L, const BlkDev &b, const CaseDev &c, const SubDev &s, int i, int j,
                                        int k) {
  int i1, j1, i2, j2;
  ghost_pair(s.face, i, j, k, i1, j1, i2, j2);
  const long long a = fidx(b, i1, j1);
  const double dw = L.nvar == 6 ? L.geo[G_DW * L.F + a] : 0.0;
  const Cell A = load_cell(L, a);
  Cell G = A;
  if (c.Twall <= 0) {
    G.v[1] = -A.v[1];
    G.v[2] = -A.v[2];
  } else {
    const double d1 = A.v[0];
    double u1 = A.v[1] / d1, v1 = A.v[2] / d1;
    double p1 = (A.v[3] - 0.5 * d1 * (u1 * u1 + v1 * v1)) * (c.gamma - 1.0);
    double T1 = c.gamma * c.Ma * c.Ma * p1 / d1;
    double p2 = p1, T2 = 2.0 * c.Twall - T1, u2 = -u1, v2 = -v1;
    double d2 = c.gamma * c.Ma * c.Ma * p2 / T2;
    G.v[0] = d2;
    G.v[1] = d2 * u2;
    G.v[2] = d2 * v2;
    G.v[3] = p2 / (c.gamma - 1.0) + 0.5 * d2 * (u2 * u2 + v2 * v2);
  }
  if (L.nvar == 5) G.v[4] = 0.0;
  if (L.nvar == 6) {
    const double beta1 = 0.075;
    const double d1 = A.v[0];
    double d2 = G.v[0];
    double r2 = G.v[1], r3 = G.v[2];
    double T2 = (G.v[3] - 0.5 * (r2 * r2 + r3 * r3) / d2) / (c.Cv * d2);
    double Amu2 = (1.0 + c.Tsb) * sqrt(T2 * T2 * T2) / (c.Tsb + T2);
    double wt = 60.0 * Amu2 / (d2 * beta1 * (dw * dw) * c.Re * c.Re);
    G.v[4] = -A.v[4];
    G.v[5] = (d1 + d2) * wt - A.v[5];
  }
  store_cell(L, fidx(b, i2, j2), G);
}

// Symmetry_or_slidewall, sub_boundary.f90:391-451.  The reflection
// U - 2 (U.n) n does not depend on the sign of n, so the far-field edge
// normal serves.
__device__ __forceinline__ void bc_symmetry(const Lvl &L, const BlkDev &b, const SubDev &s, int i, int j, int k,
                                            double2 nrm) {
  int i1, j1, i2, j2;
  ghost_pair(s.face, i, j, k, i1, j1, i2, j2);
  Cell C = load_cell(L, fidx(b, i1, j1));
  const double n1 = nrm.x, n2 = nrm.y;
  const double Vn = C.v[1] * n1 + C.v[2] * n2;
  C.v[1] = C.v[1] - 2.0 * Vn * n1;
  C.v[2] = C.v[2] - 2.0 * Vn * n2;
  store_cell(L, fidx(b, i2, j2), C);
}

// Outward unit normal of a boundary node's edge, as boundary_Farfield_inlet_outlet
// (sub_boundary.f90:484-497) and Symmetry_or_slidewall (:400-412) form it: the
// edge from node (i,j) to (i,j+1) on faces 1 and 3, to (i+1,j) on faces 2 and
// 4, rotated by the face's sign.  Geometry only, so it is evaluated once at
// set-up (k_bc_normals), in separately rounded operations: the far-field
// inflow/outflow switch is a sign test on u.n.
__device__ __forceinline__ double2 edge_normal(const Lvl &L, const BlkDev &b, int face, int i, int j) {
  const long long F = L.F;
  const double *x = L.geo + G_X * F, *y = L.geo + G_Y * F;
  const long long p0 = fidx(b, i, j), p1 = (face == 1 || face == 3) ? fidx(b, i, j + 1) : fidx(b, i + 1, j);
  const double dx = __dsub_rn(x[p1], x[p0]), dy = __dsub_rn(y[p1], y[p0]);
  const double sl = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
  if (face == 1 || face == 4) return make_double2(__ddiv_rn(-dy, sl), __ddiv_rn(dx, sl));
  return make_double2(__ddiv_rn(dy, sl), __ddiv_rn(-dx, sl));
}

// boundary_Farfield_inlet_outlet, sub_boundary.f90:457-581.  The state is
// formed by reciprocal-multiply and a refined reciprocal square root (each
// within an ulp or two of the reference's divides and square root).  The
// inflow / outflow switch is a comparison of the normal Mach number with 0
// and +-1: where the fast value lies within its error bound of a threshold,
// the switch is decided on the value the reference computes, in separately
// rounded correctly rounded operations, so every cell takes the reference's
// branch.  Every ghost layer takes the same interior state and normal (the
// reference recomputes the same values per layer), so the ghost state is
// formed once and written to all LAP layers.
__device__ __forceinline__ void bc_farfield(const Lvl &L, const BlkDev &b, const CaseDev &c, const SubDev &s, int i, int j,
                                            double2 nrm) {
  const double gamma = c.gamma, gm1 = gamma - 1.0;
  const double n1 = nrm.x, n2 = nrm.y;
  int i1, j1;
  if (s.face == 1 || s.face == 2) { i1 = i; j1 = j; }
  else if (s.face == 3) { i1 = i - 1; j1 = j; }
  else { i1 = i; j1 = j - 1; }
  long long a = fidx(b, i1, j1);
  const Cell A = load_cell(L, a);
  const double d1 = A.v[0], m1 = A.v[1], m2 = A.v[2], E1 = A.v[3];
  const double rd = rcp(d1);
  const double u1 = m1 * rd, v1 = m2 * rd;
  const double p1 = (E1 - 0.5 * d1 * (u1 * u1 + v1 * v1)) * gm1;
  const double c2 = gamma * p1 * rd;
  const double rc = rsqrt_d(c2);  // 1 / c1
  const double c1 = c2 * rc;
  double Ma_n = (u1 * n1 + v1 * n2) * rc;
  // a few ulps of |u| / c bound the fast value's error; the test itself is in FP32 with
  // twice that bound, and 1e-6 about +-1
  const float Mf = fabsf(to<float>(Ma_n));
  const float tol = 2.0e-12f * (fabsf(to<float>(u1)) + fabsf(to<float>(v1))) * to<float>(rc);
  if (!(Mf > tol) || fabsf(Mf - 1.0f) <= 1.0e-6f) {
    const double ux = __ddiv_rn(m1, d1), vx = __ddiv_rn(m2, d1);
    const double ke = __dmul_rn(__dmul_rn(0.5, d1), __dadd_rn(__dmul_rn(ux, ux), __dmul_rn(vx, vx)));
    const double px = __dmul_rn(__dsub_rn(E1, ke), gm1);
    const double cx = __dsqrt_rn(__ddiv_rn(__dmul_rn(gamma, px), d1));
    Ma_n = __ddiv_rn(__dadd_rn(__dmul_rn(ux, n1), __dmul_rn(vx, n2)), cx);
  }
  const bool out = at_least(Ma_n, 0.0) || __double_as_longlong(Ma_n) << 1 == 0;  // Ma_n >= 0
  Cell C = A;
  double *G = C.v;
  const int type = s.neighb;
  if (type == BC_Outlet || (type == BC_Farfield && out)) {
    if (!(above(Ma_n, 1.0) || c.p_outlet < 0 || type == BC_Farfield)) {
      const double pb = c.p_outlet;
      const double db = d1 + (c.p_outlet - p1) * (rc * rc);
      const double t = (p1 - c.p_outlet) * (rd * rc);
      const double ub = u1 + t * n1, vb = v1 + t * n2;
      const double p2 = 2.0 * pb - p1, d2 = 2.0 * db - d1, u2 = 2.0 * ub - u1, v2 = 2.0 * vb - v1;
      G[0] = d2; G[1] = d2 * u2; G[2] = d2 * v2;
      G[3] = p2 * c.rgm1 + 0.5 * d2 * (u2 * u2 + v2 * v2);
    }
  } else {
    const double d_inf = 1.0, u_inf = c.cosA, v_inf = c.sinA, p_inf = c.p00;
    if (c.p_outlet < 0 || at_least(neg(Ma_n), 1.0)) {
      G[0] = d_inf; G[1] = d_inf * u_inf; G[2] = d_inf * v_inf;
      G[3] = p_inf / gm1 + 0.5 * d_inf * (u_inf * u_inf + v_inf * v_inf);
    } else {
      const double pb = 0.5 * (p1 + p_inf - d1 * c1 * ((u_inf - u1) * n1 + (v_inf - v1) * n2));
      const double db = d_inf + (pb - p_inf) * (rc * rc);
      const double t = (p_inf - pb) * (rd * rc);
      const double ub = u_inf - t * n1, vb = v_inf - t * n2;
      const double p2 = 2.0 * pb - p1, d2 = 2.0 * db - d1, u2 = 2.0 * ub - u1, v2 = 2.0 * vb - v1;
      G[0] = d2; G[1] = d2 * u2; G[2] = d2 * v2;
      G[3] = p2 * c.rgm1 + 0.5 * d2 * (u2 * u2 + v2 * v2);
    }
    if (L.nvar == 5) G[4] = c.vt_inf / c.Re;
    else if (L.nvar == 6) { G[4] = d_inf * c.Kt_inf; G[5] = d_inf * c.Wt_inf; }
  }
  for (int k = 1; k <= LAP; k++) {
    int i2, j2;
    if (s.face == 1) { i2 = i - k; j2 = j; }
    else if (s.face == 2) { i2 = i; j2 = j - k; }
    else if (s.face == 3) { i2 = i + k - 1; j2 = j; }
    else { i2 = i; j2 = j + k - 1; }
    store_cell(L, fidx(b, i2, j2), C);
  }
}

// U_average_conner, sub_boundary.f90:595-612: the corner ghost cell i4 takes
// rho, u, v, T extrapolated from its neighbours i1, i3 across the corner of
// i2.  One warp per corner; lanes 0..2 form the primitives of i1, i2, i3 side
// by side (the divisions by rho as reciprocal-multiplies), lane 0 combines.
__device__ __forceinline__ void corner(const Lvl &L, const CaseDev &c, long long i1, long long i2, long long i3,
                                       long long i4) {
  const int lane = threadIdx.x & 31;
  // lanes past the third repeat it
  const Cell A = load_cell(L, lane == 0 ? i1 : lane == 1 ? i2 : i3);
  const double d = A.v[0], rd = rcp(d), uu = A.v[1] * rd, v = A.v[2] * rd;
  const double T = (A.v[3] - (uu * A.v[1] + v * A.v[2]) * 0.5) * (rd * c.rCv);
  auto across = [](double x) {
    const double x2 = __shfl_sync(0xffffffffu, x, 1), x3 = __shfl_sync(0xffffffffu, x, 2);
    return x + x3 - x2;  // of lane 0
  };
  const double d4 = across(d), uu4 = across(uu), v4 = across(v), T4 = across(T);
  Cell C;
  C.v[0] = d4;
  C.v[1] = d4 * uu4;
  C.v[2] = d4 * v4;
  C.v[3] = d4 * (c.Cv * T4 + (uu4 * uu4 + v4 * v4) * 0.5);
  if (L.nvar > 4) {
    C.v[4] = across(A.v[4]);
    C.v[5] = across(A.v[5]);
  }
  if (lane == 0) store_cell(L, i4, C);
}

// phases: 1 physical BCs, 2 halo copy, 4 corners
constexpr int BC_SMEM_SUBS = 32;  // subfaces of a block staged in shared memory
// A block's boundary is served by a cluster of CTAs whose warps take its items in turn,
// with a cluster barrier between phases.  On one SM the FP64 instructions of a
// far-field phase queue up (some 60 per item, one warp instruction per 16 to 19 cycles:
// twelve warps of a 97 x 97 plate 6 us); on eight SMs a phase costs one item's chain.
// Measured per call between events (5 us of them the launch), 512 threads on one SM
// against eight CTAs: 1025 x 513 54 and 21 us, 16 cases of 385 x 97 22 and 18; 97 x 97
// 20.4 and 18.5, the chain of a far-field item (some 45 FP64 instructions of 64 cycles)
// once per phase.  From 152 blocks on the blocks fill the chip and a cluster has
// BC_CTAS_MANY CTAs.
constexpr int BC_THREADS = 256, BC_CTAS = 8, BC_CTAS_MANY = 2;

// every global write of the cluster's threads before is seen by them after
__device__ __forceinline__ void bc_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

__global__ void __launch_bounds__(BC_THREADS) k_bc(Lvl L, int phases, int CS) {
  const int bk = blockIdx.x / CS, rank = blockIdx.x % CS;  // the cluster is blocks bk CS .. bk CS + CS - 1
  // the cluster's warps in turn over its CTAs; the items of a phase's subfaces go to
  // them subface by subface, each starting at the warp after the last one's
  const int lane = threadIdx.x & 31, gw = (threadIdx.x >> 5) * CS + rank, nw = CS * (BC_THREADS / 32), step = nw * 32;
  auto after = [&](int w, int n) {
    w -= ((n + 31) >> 5) & (nw - 1);
    return w < 0 ? w + nw : w;
  };
  const BlkDev &b = L.blk[bk];
  // the block's subface table (global beyond 32 entries) and its case in shared memory,
  // copied in words by all threads: the items of every phase read them
  __shared__ SubDev ssub[BC_SMEM_SUBS];
  __shared__ CaseDev c;
  const int nsub = b.nsub;
  {
    static_assert(sizeof(SubDev) % 8 == 0 && sizeof(CaseDev) % 8 == 0, "copied in words");
    constexpr int SW = sizeof(SubDev) / 8, CW = sizeof(CaseDev) / 8;
    const long long *ps = reinterpret_cast<const long long *>(L.sub + b.sub0),
                    *pc = reinterpret_cast<const long long *>(L.cs + b.cas);
    long long *ds = reinterpret_cast<long long *>(ssub), *dc = reinterpret_cast<long long *>(&c);
    for (int t = threadIdx.x; t < CW; t += BC_THREADS) dc[t] = pc[t];
    for (int t = threadIdx.x; t < min(nsub, BC_SMEM_SUBS) * SW; t += BC_THREADS) ds[t] = ps[t];
    __syncthreads();
  }
  auto sub = [&](int ks) -> const SubDev & { return ks < BC_SMEM_SUBS ? ssub[ks] : L.sub[b.sub0 + ks]; };
  if (phases & 1) {
    // subfaces of one phase touch disjoint cells (grouped at set-up in
    // subface order): their items are spread over the cluster together
    for (int ph = 0; ph < b.nphase; ph++) {
      int w = gw;  // this warp's place after the warps of the subfaces before
      for (int ks = 0; ks < nsub; ks++) {
        const SubDev &s = sub(ks);
        if (s.neighb >= 0 || s.phase != ph) continue;
        const int ni = s.iend - s.ist + 1, nj = s.jend - s.jst + 1, n = s.nitem;
        for (int u = w * 32 + lane; u < n; u += step) {
          const bool ff = s.neighb == BC_Farfield || s.neighb == BC_Inlet || s.neighb == BC_Outlet;
          const int k = ff ? 1 : u % LAP + 1, r = ff ? u : u / LAP;  // ghost layer, node
          int i = s.ist, j = s.jst;
          if (nj == 1) i += r;
          else if (ni == 1) j += r;
          else { i += r % ni; j += r / ni; }
          if (ff) bc_farfield(L, b, c, s, i, j, L.bcn[s.nrm0 + r]);
          else if (s.neighb == BC_Wall) bc_wall(L, b, c, s, i, j, k);
          else if (s.neighb == BC_Symmetry) bc_symmetry(L, b, s, i, j, k, L.bcn[s.nrm0 + r]);
        }
        w = after(w, n);
      }
      bc_barrier();
    }
  }
  if (phases & 2) {
    int w = gw;
    for (int ks = 0; ks < nsub; ks++) {
      const SubDev &s = sub(ks);
      if (s.neighb < 0) continue;
      int n1 = s.iend - s.ist + s.jend - s.jst;
      for (int t = w * 32 + lane; t < n1 * LAP; t += step) {
        int l = t % LAP + 1, k = t / LAP + 1;
        int k1 = (s.orient == 2) ? k : n1 + 1 - k;
        int si, sj;
        if (s.nface == 1) { si = s.nist + l - 1; sj = s.njst + k1 - 1; }
        else if (s.nface == 2) { si = s.nist + k1 - 1; sj = s.njst + l - 1; }
        else if (s.nface == 3) { si = s.niend - LAP - 1 + l; sj = s.njst + k1 - 1; }
        else { si = s.nist + k1 - 1; sj = s.njend - LAP - 1 + l; }
        int di, dj;
        if (s.face == 1) { di = s.ist - LAP - 1 + l; dj = s.jst + k - 1; }
        else if (s.face == 2) { di = s.ist + k - 1; dj = s.jst - LAP - 1 + l; }
        else if (s.face == 3) { di = s.iend + l - 1; dj = s.jst + k - 1; }
        else { di = s.ist + k - 1; dj = s.jend + l - 1; }
        long long src = s.noff + (long long)(sj + 2) * s.nP + (si + 2), dst = fidx(b, di, dj);
        store_cell(L, dst, load_cell(L, src));
      }
      w = after(w, n1 * LAP);
    }
    bc_barrier();
  }
  if (phases & 4) {
    int nx = b.nx, ny = b.ny;
    const int w = gw;  // a warp per corner, on different SMs
    if (w == 0) corner(L, c, fidx(b, 1, 0), fidx(b, 1, 1), fidx(b, 0, 1), fidx(b, 0, 0));
    else if (w == 1) corner(L, c, fidx(b, 1, ny), fidx(b, 1, ny - 1), fidx(b, 0, ny - 1), fidx(b, 0, ny));
    else if (w == 2) corner(L, c, fidx(b, nx - 1, 0), fidx(b, nx - 1, 1), fidx(b, nx, 1), fidx(b, nx, 0));
    else if (w == 3) corner(L, c, fidx(b, nx - 1, ny), fidx(b, nx - 1, ny - 1), fidx(b, nx, ny - 1), fidx(b, nx, ny));
  }
}

void launch_bc(const Lvl &L, int phases, cudaStream_t s) {
  const int CS = L.nblk < 152 ? BC_CTAS : BC_CTAS_MANY;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(L.nblk * CS);
  cfg.blockDim = dim3(BC_THREADS);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CS; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_bc, L, phases, CS);
}

// force_vt_kw: negative nu~, k and omega of the interior cells become 1e-10
__global__ void __launch_bounds__(EC2D_TILE) k_clip(Lvl L) {
  int bk, i, j;
  if (!core_ij(L, bk, i, j)) return;
  const BlkDev &b = L.blk[bk];
  if (i < 1 || i > b.nx - 1 || j < 1 || j > b.ny - 1) return;
  const long long id = fidx(b, i, j);
  for (int m = 4; m < L.nvar; m++)
    if (L.U[m * L.F + id] < 0) L.U[m * L.F + id] = 1.0e-10;
}
void launch_clip(const Lvl &L, cudaStream_t s) {
  if (L.nvar >= 5) k_clip<<<L.nctiles, EC2D_TILE, 0, s>>>(L);
}

// set-up: the edge normals of every far-field and symmetry node (grid y: block)
__global__ void __launch_bounds__(256) k_bc_normals(Lvl L) {
  const BlkDev &b = L.blk[blockIdx.y];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  for (int ks = 0; ks < b.nsub; ks++) {
    const SubDev &s = L.sub[b.sub0 + ks];
    const int ni = s.iend - s.ist + 1, nn = ni * (s.jend - s.jst + 1);
    if (s.nrm0 < 0 || t >= nn) continue;
    L.bcn[s.nrm0 + t] = edge_normal(L, b, s.face, s.ist + t % ni, s.jst + t / ni);
  }
}
void launch_bc_normals(const Lvl &L, int max_nodes, cudaStream_t s) {
  if (max_nodes > 0) k_bc_normals<<<dim3((max_nodes + 255) / 256, L.nblk), 256, 0, s>>>(L);
}

}  // namespace ec2d
