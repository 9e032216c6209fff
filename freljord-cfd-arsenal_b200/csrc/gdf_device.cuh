// gdf_device.cuh -- the per-item device code of the GDF P2 step: one face
// quadrature point, vertex, cell or face per call, in the reference's
// arithmetic order. The single-problem kernels (gdf_kernels.cu) and the
// ensemble's persistent stage kernel (gdf_ensemble.cu) both run these.
#pragma once

#include <cuda_runtime.h>

#include "../../include/gdf.h"
#include "gdf_charlim.cuh"
#include "gdf_kernels.cuh"
#include "gdf_mlp.cuh"
#include "gdf_vertex.cuh"

#include <mutex>

namespace gdf {

// Grid-independent basis tables (one copy per device and module; each
// translation unit that launches kernels fills its own with
// upload_basis_once before its first launch on a device).
static __constant__ Basis c_basis;

// ------------------------------------------------------------ live slots --
__host__ __device__ constexpr int LI(int n, int d) {
  return n < 5 ? n * 6 + d
               : n == 5 ? 30 + (d <= 6 ? d : 7)
                        : n == 6 ? 38 + (d <= 5 ? d : (d == 7 ? 6 : 7)) : 46 + d;
}
static __constant__ unsigned char c_live_n[NLIVE] = {0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 1, 1, 2, 2, 2, 2, 2, 2,
                                              3, 3, 3, 3, 3, 3, 4, 4, 4, 4, 4, 4, 5, 5, 5, 5, 5, 5,
                                              5, 5, 6, 6, 6, 6, 6, 6, 6, 6, 7, 7, 7, 7, 7, 7};
static __constant__ unsigned char c_live_d[NLIVE] = {0, 1, 2, 3, 4, 5, 0, 1, 2, 3, 4, 5, 0, 1, 2, 3, 4, 5,
                                              0, 1, 2, 3, 4, 5, 0, 1, 2, 3, 4, 5, 0, 1, 2, 3, 4, 5,
                                              6, 8, 0, 1, 2, 3, 4, 5, 7, 9, 0, 1, 2, 3, 4, 5};

// variable and mode of live slot s (the order of c_live_n / c_live_d)
__host__ __device__ constexpr int slot_n(int s) { return s < 30 ? s / 6 : s < 38 ? 5 : s < 46 ? 6 : 7; }
__host__ __device__ constexpr int slot_d(int s) {
  return s < 30 ? s % 6 : s < 38 ? (s - 30 <= 6 ? s - 30 : 8) : s < 46 ? (s - 38 <= 5 ? s - 38 : (s == 44 ? 7 : 9)) : s - 46;
}
// structural zeros of the volume basis derivatives: phixG vanishes for
// modes 1, 3, 6, 10 and phiyG for modes 1, 2, 4, 7 (get_basis.f90)
__host__ __device__ constexpr bool px_zero(int d) { return d == 0 || d == 2 || d == 5 || d == 9; }
__host__ __device__ constexpr bool py_zero(int d) { return d == 0 || d == 1 || d == 3 || d == 6; }

__device__ __forceinline__ long long gtid() { return (long long)blockIdx.x * blockDim.x + threadIdx.x; }

// ------------------------------------------------------------- set_bc ----
// set_bc.f90:5-27. Ghost (i,j) takes the value of (mapx(i), mapy(j)): the
// x pass first and then the y pass over full rows make every corner ghost
// the image of an interior cell under both maps. zeroB also clears the
// ghost Bx/By modes, as div_free_Balsara.f90:11 leaves them.
__host__ __device__ __forceinline__ long long set_bc_items(const Consts& K) {
  return (2LL * (K.nx + 2) + 2LL * K.ny) * NLIVE;
}
__device__ __forceinline__ void set_bc_item(const Consts& K, double* __restrict__ U, int zeroB, long long t) {
  const long long nper = 2LL * (K.nx + 2) + 2LL * K.ny;
  const int k = (int)(t / nper);
  const long long q = t - (long long)k * nper;
  int i, j;
  if (q < K.nx + 2) { i = (int)q; j = 0; }
  else if (q < 2LL * (K.nx + 2)) { i = (int)(q - (K.nx + 2)); j = K.ny + 1; }
  else if (q < 2LL * (K.nx + 2) + K.ny) { i = 0; j = (int)(q - 2LL * (K.nx + 2)) + 1; }
  else { i = K.nx + 1; j = (int)(q - 2LL * (K.nx + 2) - K.ny) + 1; }
  int si = i, sj = j;
  if (i == 0) si = (K.bc_l == GDF_BC_PERIODIC) ? K.nx : 1;
  else if (i == K.nx + 1) si = (K.bc_r == GDF_BC_PERIODIC) ? 1 : K.nx;
  if (j == 0) sj = (K.bc_d == GDF_BC_PERIODIC) ? K.ny : 1;
  else if (j == K.ny + 1) sj = (K.bc_u == GDF_BC_PERIODIC) ? 1 : K.ny;
  const int n = c_live_n[k], d = c_live_d[k];
  const long long off = K.plane * (d + 10 * n);
  double v = U[off + si + (long long)K.nx2 * sj];
  if (zeroB && (n == 5 || n == 6)) v = 0.0;
  U[off + i + (long long)K.nx2 * j] = v;
}

// ---------------------------------------------------- face Riemann -------
// Lh.f90:72-265 and LhEz.f90:6-31 for one face quadrature point.
// DIR 0: x face (i = 0..Nx, j = 1..Ny) between cells (i,j) and (i+1,j).
// DIR 1: y face (i = 1..Nx, j = 0..Ny) between cells (i,j) and (i,j+1).
template <int DIR>
__host__ __device__ __forceinline__ long long face_items(const Consts& K) {
  return DIR == 0 ? (long long)(K.nx + 1) * NG * K.ny : (long long)K.nx * NG * (K.ny + 1);
}
// One face quadrature point from the modes of its two cells, read through
// mL(n, d) (the cell on the low side) and mR(n, d) (the high side); o is the
// face's offset in its plane. The arithmetic is that of Lh.f90:72-265 and
// LhEz.f90:6-31 whichever memory the modes come from.
template <int DIR, class DIV, class ML, class MR>
__device__ __forceinline__ bool face_point(const Consts& K, ML mL, MR mR, int g, double* __restrict__ Fh_out,
                                           double* __restrict__ Ez_out, long long o) {
  double uL[NE], uR[NE];
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    double a = 0.0, b = 0.0;
#pragma unroll
    for (int d = 0; d < NP; ++d) {
      if (!live_mode(n, d)) continue;
      const double pl = DIR == 0 ? c_basis.phiGR[g][d] : c_basis.phiGU[g][d];
      const double pr = DIR == 0 ? c_basis.phiGL[g][d] : c_basis.phiGD[g][d];
      // the face basis is 1 for mode 1, and for mode 2 (x faces) or 3 (y
      // faces) 1 on the low cell's face and -1 on the high cell's
      // (get_basis.f90): those products are exact (x * 1 == x, x * -1 == -x for
      // every double) and written out
      const int du = DIR == 0 ? 1 : 2;
      if (d == 0) {
        a = a + mL(n, d);
        b = b + mR(n, d);
      } else if (d == du) {
        a = a + mL(n, d);
        b = b + (-mR(n, d));
      } else {
        a = a + mL(n, d) * pl;
        b = b + mR(n, d) * pr;
      }
    }
    uL[n] = a;
    uR[n] = b;
  }
  SideOf<DIV> L, R;
  unsigned bad = 0;
  make_side(K.P, uL, L, bad);
  make_side(K.P, uR, R, bad);
  double Fh[NE], fL[NE], fR[NE];
  face_flux_sides(K.P, L, R, DIR, Fh, fL, fR, bad);
  const long long fp = DIR == 0 ? K.fxplane : K.fyplane;
#pragma unroll
  for (int n = 0; n < NE; ++n) Fh_out[(n * NG + g) * fp + o] = Fh[n];
  double ez;
  if (DIR == 0) {
    if (K.ez_fhat) {
      ez = -Fh[6];
    } else {
      const double S = fmax2(fabs(L.u), fabs(R.u));
      ez = -0.5 * (fL[6] + fR[6] - S * (uR[6] - uL[6]));
    }
  } else {
    if (K.ez_fhat) {
      ez = Fh[5];
    } else {
      const double S = fmax2(fabs(L.v), fabs(R.v));
      ez = 0.5 * (fL[5] + fR[5] - S * (uR[5] - uL[5]));
    }
  }
  Ez_out[g * fp + o] = ez;
  return !bad;
}

// Face f (in plane order) at point g; false where an operand left rdiv's ranges.
template <int DIR, class DIV>
__device__ __forceinline__ bool face_solve(const Consts& K, const double* __restrict__ U, double* __restrict__ Fh_out,
                                        double* __restrict__ Ez_out, long long f, int g) {
  const int nf = DIR == 0 ? K.nx + 1 : K.nx;
  const int i0 = (int)(f % nf), j0 = (int)(f / nf);
  long long cL, cR;
  if (DIR == 0) {
    cL = i0 + (long long)K.nx2 * (j0 + 1);
    cR = cL + 1;
  } else {
    cL = (i0 + 1) + (long long)K.nx2 * j0;
    cR = cL + K.nx2;
  }
  const long long pl = K.plane;
  return face_point<DIR, DIV>(
      K, [&](int n, int d) { return U[pl * (d + 10 * n) + cL]; }, [&](int n, int d) { return U[pl * (d + 10 * n) + cR]; },
      g, Fh_out, Ez_out, f);
}

// A face whose operands leave rdiv's ranges is solved again with IEEE divisions
// (out of line: rare, and its code stays out of the instruction cache).
template <int DIR>
static __device__ __noinline__ void face_refused(const Consts& K, const double* __restrict__ U,
                                                 double* __restrict__ Fh_out, double* __restrict__ Ez_out, long long f,
                                                 int g) {
  face_solve<DIR, IeeeDiv>(K, U, Fh_out, Ez_out, f, g);
}
template <int DIR>
__device__ __forceinline__ void face_at(const Consts& K, const double* __restrict__ U, double* __restrict__ Fh_out,
                                        double* __restrict__ Ez_out, long long f, int g) {
  if (!face_solve<DIR, SharedRcp>(K, U, Fh_out, Ez_out, f, g)) face_refused<DIR>(K, U, Fh_out, Ez_out, f, g);
}

// the same from an item number, faces of a row fastest, then its points (the
// ensemble's tiles)
template <int DIR>
__device__ __forceinline__ void face_item(const Consts& K, const double* __restrict__ U, double* __restrict__ Fh_out,
                                          double* __restrict__ Ez_out, long long item) {
  const int nf = DIR == 0 ? K.nx + 1 : K.nx;
  const long long r = item / nf;
  face_at<DIR>(K, U, Fh_out, Ez_out, item - r * nf + (r / NG) * nf, (int)(r % NG));
}

// ------------------------------------------------------- vertex Ez -------
// LhEz.f90:34-69: corner traces of the four cells around vertex (i,j),
// i = 0..Nx, j = 0..Ny, and the 2-D Riemann solver.
// Lane q of four (see gdf_vertex.cuh). Corner values of modes 1, 2,
// 3 and 5 are +-1 (get_basis.f90: 1, x, y and x y at the corner): their products
// are exact and written as sign changes.
template <int FLUX, class DIV>
__device__ __forceinline__ bool vertex_lane_as(const Consts& K, const double* __restrict__ U, long long item, int q,
                                               double& Ez) {
  const int i = (int)(item % (K.nx + 1));
  const int j = (int)(item / (K.nx + 1));
  const bool xr = !(q & 1), yu = q < 2;      // the cell is right of, above the vertex
  const long long c = i + xr + (long long)K.nx2 * (j + yu);
  const int sx = xr ? (int)0x80000000 : 0, sy = yu ? (int)0x80000000 : 0;
  double u[NE], phi[NP];
  // in registers: a choice among the tables inside the sums is a branch that
  // keeps one variable's loads from starting before the last one's sum
#pragma unroll
  for (int d = 0; d < NP; ++d) {
    const double ru = c_basis.phiRU[d], lu = c_basis.phiLU[d], rd = c_basis.phiRD[d], ld = c_basis.phiLD[d];
    phi[d] = xr ? (yu ? ld : lu) : (yu ? rd : ru);
  }
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    double a = 0;
#pragma unroll
    for (int d = 0; d < NP; ++d) {
      if (!live_mode(n, d)) continue;
      const double v = U[K.plane * (d + 10 * n) + c];
      if (d == 0) a = a + v;
      else if (d == 1 || d == 2 || d == 4)
        a = a + __hiloint2double(__double2hiint(v) ^ (d == 1 ? sx : d == 2 ? sy : sx ^ sy), __double2loint(v));
      else
        a = a + v * phi[d];
    }
    u[n] = a;
  }
  return vertex_quad<FLUX, DIV>(K.P, u, Ez);
}
template <int FLUX>
static __device__ __noinline__ double vertex_refused(const Consts& K, const double* __restrict__ U, long long item, int q) {
  double Ez;
  vertex_lane_as<FLUX, IeeeDiv>(K, U, item, q, Ez);
  return Ez;
}
template <int FLUX>
__device__ __forceinline__ void vertex_lane(const Consts& K, const double* __restrict__ U, double* __restrict__ EzV,
                                            long long item, int q) {
  const bool live = q == 0 && item < K.vplane;
  if (item >= K.vplane) item = K.vplane - 1;   // the whole warp takes part
  double Ez;
  if (!vertex_lane_as<FLUX, SharedRcp>(K, U, item, q, Ez)) Ez = vertex_refused<FLUX>(K, U, item, q);
  if (live) EzV[item] = Ez;
}
// for any solver
__device__ __forceinline__ void vertex_at(const Consts& K, const double* __restrict__ U, double* __restrict__ EzV,
                                          long long item, int q) {
  switch (K.P.flux) {
    case 1: return vertex_lane<1>(K, U, EzV, item, q);
    case 2: return vertex_lane<2>(K, U, EzV, item, q);
    case 3: return vertex_lane<3>(K, U, EzV, item, q);
    default: return vertex_lane<4>(K, U, EzV, item, q);
  }
}

// ------------------------------------------------ residual + combine -----
// Lh.f90:11-68 (volume), :268-304 (surface, mass) and the RK3.f90 stage
// combine for one cell of the whole (Nx+2)x(Ny+2) array (ghost cells have
// du = 0, as Lh leaves them). stage 0 writes du instead (gdf_lh).
constexpr int CELL_BS = 64;

// A thread's 52 staged modes, two by two at ms[2*(CELL_BS*(k/2) + tid) + k%2]
// (one 128-bit load per pair).
constexpr int CELL_SLOTS = NLIVE;

// The point values and fluxes of the volume term take a third of the residual's
// operations, the 52 sums du the rest: they hold 104 registers, which is what
// keeps the kernel at 8 warps per SM. Sums keep the reference's order (the 25
// points with b fastest, then x faces, then y faces, then the mass matrix); what
// is shared between points or modes is shared before a sum, never across one: a face flux times lambda
// (modes 3 and 5, or 2 and 5) or times P2 (modes 6 and 9, or 4 and 8), one
// reciprocal per point for u, v, w, known reciprocals for the mass matrix.
// The instruction cache decides much of the rest: eight warps at different places
// of a long straight line evict each other's code. So the surface sums are one
// copy per direction (not unrolled over the points) and the divisions behind
// rdiv out of line.
// Blast 2048^2: 3.80 ms per launch, 6.09 at first (5.66 with the surface sums
// unrolled, 4.27 with the fallback divisions inline); rotor 512^2 319 us, 448 at
// first. (Keeping a column's parts in shared memory, forming the next point's
// values beside this one's primitives, and the mass matrix and the combination
// as a loop over the slots in shared memory were each slower.)
// ms: the block's CELL_SLOTS * CELL_BS doubles, 16-byte aligned (blockDim.x ==
// CELL_BS).
__device__ __forceinline__ void cell_item(const Consts& K, const double* __restrict__ U, double* __restrict__ U0,
                                          double* __restrict__ UI, const double* __restrict__ Fxh,
                                          const double* __restrict__ Fyh, double* __restrict__ duout,
                                          const Scal* __restrict__ sc, int stage, long long item, double* ms) {
  const int tid = threadIdx.x;
  const int i = (int)(item % K.nx2);
  const int j = (int)(item / K.nx2);
  const bool interior = i >= 1 && i <= K.nx && j >= 1 && j <= K.ny;
  auto at = [&](int k) -> double& { return ms[2 * (CELL_BS * (k >> 1) + tid) + (k & 1)]; };
  auto pair = [&](int k) { return reinterpret_cast<const double2*>(ms)[CELL_BS * (k >> 1) + tid]; };   // k even
  double du[NLIVE];
#pragma unroll
  for (int k = 0; k < NLIVE; ++k) du[k] = 0.0;
  if (interior) {
#pragma unroll
    for (int n = 0; n < NE; ++n)
#pragma unroll
      for (int d = 0; d < NP; ++d)
        if (live_mode(n, d)) at(LI(n, d)) = U[item + K.plane * (d + 10 * n)];
    {
      // the surface term reads the fluxes of the cell's four faces after the
      // volume loop: ask for them in L2 now, so the loads that follow the
      // volume work do not wait on DRAM
      const long long px = (i - 1) + 1 + (long long)(K.nx + 1) * (j - 1);
      const long long py = (i - 1) + (long long)K.nx * j;
#pragma unroll 1
      for (int q = 0; q < NE * NG; ++q) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(Fxh + q * K.fxplane + px - 1));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(Fyh + q * K.fyplane + py));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(Fyh + q * K.fyplane + py - K.nx));
      }
    }
    // volume term
#pragma unroll 1
    for (int a = 0; a < NG; ++a) {
#pragma unroll 1
      for (int b = 0; b < NG; ++b) {
        const double* f = c_basis.phiG[a][b];
        double v[NE];
#pragma unroll
        for (int n = 0; n < NE; ++n) {
          double m[8];
          const int nl = (n == 5 || n == 6) ? 8 : 6;
#pragma unroll
          for (int k = 0; k < nl; k += 2) {
            const double2 q = pair(LI(n, 0) + k);
            m[k] = q.x;
            m[k + 1] = q.y;
          }
          double acc = 0.0 + m[0];
#pragma unroll
          for (int d = 1; d < NP; ++d)
            if (live_mode(n, d)) acc = acc + m[LI(n, d) - LI(n, 0)] * f[d];
          v[n] = acc;
        }
        const double rho = v[0];
        unsigned bad = 0;
        const Rcp rr = rcp_of(rho, bad);
        double u = rdiv(v[1], rr, bad), vv = rdiv(v[2], rr, bad), w = rdiv(v[3], rr, bad);
        if (bad) {   // an operand out of rdiv's range: the IEEE division itself
          u = ieee_div(v[1], rho);
          vv = ieee_div(v[2], rho);
          w = ieee_div(v[3], rho);
        }
        const double E = v[4], B1 = v[5], B2 = v[6], B3 = v[7];
        const double BB = sq(B1) + sq(B2) + sq(B3);
        const double p = K.P.gamma1 * (E - 0.5 * rho * (sq(u) + sq(vv) + sq(w)) - 0.5 * BB);
        const double S = p + 0.5 * BB;
        const double T = E + S;
        const double Kc = u * B1 + vv * B2 + w * B3;
        double Fx[NE], Fy[NE];
        Fx[0] = v[1];
        Fx[1] = rho * sq(u) + S - sq(B1);
        Fx[2] = rho * u * vv - B1 * B2;
        Fx[3] = rho * u * w - B1 * B3;
        Fx[4] = T * u - Kc * B1;
        Fx[5] = 0.0;
        Fx[6] = u * B2 - vv * B1;
        Fx[7] = u * B3 - w * B1;
        Fy[0] = v[2];
        Fy[1] = rho * u * vv - B1 * B2;
        Fy[2] = rho * sq(vv) + S - sq(B2);
        Fy[3] = rho * vv * w - B2 * B3;
        Fy[4] = T * vv - Kc * B2;
        Fy[5] = vv * B1 - u * B2;
        Fy[6] = 0.0;
        Fy[7] = vv * B3 - w * B2;
        const double coef = 0.25 * c_basis.w[a] * c_basis.w[b];
        // du(d,n) += coef*(Fx*phixG + Fy*phiyG); a product with an exact zero
        // (phixG of modes 1,3,6,10, phiyG of modes 1,2,4,7, Fx(6), Fy(7))
        // contributes +-0 and is left out
#pragma unroll
        for (int d = 1; d < NP; ++d)
#pragma unroll
          for (int n = 0; n < NE; ++n) {
            if (!live_mode(n, d)) continue;
            const bool hx = n != 5 && !px_zero(d);
            const bool hy = n != 6 && !py_zero(d);
            if (hx && hy)
              du[LI(n, d)] = du[LI(n, d)] + coef * (Fx[n] * K.phix[a][b][d] + Fy[n] * K.phiy[a][b][d]);
            else if (hx)
              du[LI(n, d)] = du[LI(n, d)] + coef * (Fx[n] * K.phix[a][b][d]);
            else if (hy)
              du[LI(n, d)] = du[LI(n, d)] + coef * (Fy[n] * K.phiy[a][b][d]);
          }
      }
    }
    // surface terms in the reference order (x faces, then y faces), a point at
    // a time for all variables (one copy of the code per direction: unrolled
    // over the points and variables the kernel did not fit the instruction
    // cache). q1 the flux on the high face, q0 on the low one; the face basis is
    // the same on both up to the sign of the modes odd in the face's direction
    // (get_basis.f90), 1 for mode 1, +-1 for the slope across the face, and at
    // the middle point zero for the modes odd along it.
    const long long ox = (i - 1) + 1 + (long long)(K.nx + 1) * (j - 1);  // Fxhat(i,j)
    const long long oy = (i - 1) + (long long)K.nx * j;                  // Fyhat(i,j)
    auto faces = [&](const double* F, long long pl, long long o, long long low, const double* cw,
                     const double (*fb)[NP], bool x) {
      const int across = x ? 1 : 2, along = x ? 2 : 1, across2 = x ? 3 : 5, along2 = x ? 5 : 3;
#pragma unroll 1
      for (int g = 0; g < NG; ++g) {
        const double c = cw[g];
        const double* f = fb[g];
        const double* G = F + g * pl + o;
        double q1[NE], q0[NE];
#pragma unroll
        for (int n = 0; n < NE; ++n) {
          q1[n] = G[n * NG * pl];
          q0[n] = G[n * NG * pl - low];
        }
#pragma unroll
        for (int n = 0; n < NE; ++n) {
          auto add = [&](int d, double t) { du[LI(n, d)] = du[LI(n, d)] - c * t; };
          add(0, q1[n] - q0[n]);
          add(across, q1[n] + q0[n]);
          add(across2, q1[n] * f[across2] - q0[n] * f[across2]);
          const double s1 = q1[n] * f[along2], s0 = q0[n] * f[along2];
          add(along2, s1 - s0);
          // Bx's mode 9, By's 8
          if (n == 5 && x) add(8, s1 + s0);
          if (n == 6 && !x) add(7, s1 + s0);
          if (n == 5 && x) add(6, q1[n] * f[6] + q0[n] * f[6]);
          if (n == 6 && !x) add(9, q1[n] * f[9] + q0[n] * f[9]);
        }
        if (g != 2) {
#pragma unroll
          for (int n = 0; n < NE; ++n) {
            auto add = [&](int d, double t) { du[LI(n, d)] = du[LI(n, d)] - c * t; };
            const double l1 = q1[n] * f[along], l0 = q0[n] * f[along];
            add(along, l1 - l0);
            add(4, l1 + l0);
            if (n == 5 && !x) {
              add(6, q1[n] * f[6] - q0[n] * f[6]);
              add(8, q1[n] * f[8] - q0[n] * f[8]);
            }
            if (n == 6 && x) {
              add(7, q1[n] * f[7] - q0[n] * f[7]);
              add(9, q1[n] * f[9] - q0[n] * f[9]);
            }
          }
        }
      }
    };
    faces(Fxh, K.fxplane, ox, 1, K.cxw, c_basis.phiGR, true);
    faces(Fyh, K.fyplane, oy, K.nx, K.cyw, c_basis.phiGU, false);
    // mm(1) = 1 (get_basis.f90): x / 1 == x
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      unsigned bad = 0;
      double q[NP];
#pragma unroll
      for (int d = 1; d < NP; ++d)
        if (live_mode(n, d)) q[d] = rdiv(du[LI(n, d)], Rcp{c_basis.mm[d], c_basis.rmm[d]}, bad);
#pragma unroll
      for (int d = 1; d < NP; ++d)
        if (live_mode(n, d)) du[LI(n, d)] = bad ? ieee_div(du[LI(n, d)], c_basis.mm[d]) : q[d];
    }
  }
  if (stage == 0) {
    if (interior) {
#pragma unroll
      for (int n = 0; n < NE; ++n)
#pragma unroll
        for (int d = 0; d < NP; ++d)
          if (live_mode(n, d)) duout[item + K.plane * (d + 10 * n)] = du[LI(n, d)];
    }
    return;
  }
  // the stage's combination, a variable at a time: its loads are all under way
  // before its first store
  const double dt = sc->dt;
  double na[NP], nb[NP];
  auto fetch = [&](int n) {
#pragma unroll
    for (int d = 0; d < NP; ++d) {
      if (!live_mode(n, d)) continue;
      const long long c = item + K.plane * (d + 10 * n);
      na[d] = stage == 1 ? U[c] : UI[c];
      nb[d] = stage == 1 ? 0.0 : U0[c];
    }
  };
  fetch(0);
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    double a[NP], b[NP];
#pragma unroll
    for (int d = 0; d < NP; ++d)
      if (live_mode(n, d)) { a[d] = na[d]; b[d] = nb[d]; }
    if (n + 1 < NE) fetch(n + 1);
#pragma unroll
    for (int d = 0; d < NP; ++d) {
      if (!live_mode(n, d)) continue;
      const long long c = item + K.plane * (d + 10 * n);
      const double v = a[d] + dt * du[LI(n, d)];
      if (stage == 1) {
        U0[c] = a[d];
        UI[c] = v;
      } else if (stage == 2) {
        UI[c] = (3.0 / 4.0) * b[d] + (1.0 / 4.0) * v;
      } else {
        UI[c] = (1.0 / 3.0) * b[d] + (2.0 / 3.0) * v;
      }
    }
  }
}

// The same for two lanes to a cell, lane r of a half warp's sixteen cells and its
// partner sixteen lanes on: lane 0 has the sums of rho, m_x, E and Bx, lane 1
// those of m_z, m_y, B3 and By. Each forms its four variables at a point, takes
// the other four from its partner and forms the point's primitives and fluxes
// for both; so 52 sums become 26 (PAIR_SLOTS), a thread's code and its chain of
// dependent operations halve, and twice the warps run, for 15% more operations.
// Operations and their order are those of cell_item; a sum of one lane that the
// other one's variables do not have adds zeros.
// A whole warp comes here together. phix, phiy: K's tables, or the caller's copy.
constexpr int PAIR_BS = 128, PAIR_SLOTS = 26;
__device__ __forceinline__ double flip_if(double v, bool neg) {
  return __hiloint2double(__double2hiint(v) ^ (neg ? (int)0x80000000 : 0), __double2loint(v));
}
__device__ __forceinline__ void cell_pair(const Consts& K, const double* __restrict__ U, double* __restrict__ U0,
                                          double* __restrict__ UI, const double* __restrict__ Fxh,
                                          const double* __restrict__ Fyh, double* __restrict__ duout,
                                          const Scal* __restrict__ sc, int stage, long long item, int r, double* ms,
                                          const double (*phix)[NG][NP], const double (*phiy)[NG][NP]) {
  const int tid = threadIdx.x;
  const bool live = item < K.plane;
  if (!live) item = K.plane - 1;
  const int i = (int)(item % K.nx2);
  const int j = (int)(item / K.nx2);
  const bool interior = live && i >= 1 && i <= K.nx && j >= 1 && j <= K.ny;
  // own variable k is number vn(k); its modes start at sum 6 k, the last one has two more: 7 and 9 of Bx, 8 and 10 of By
  const int vn[4] = {r ? 3 : 0, r ? 2 : 1, r ? 7 : 4, r ? 6 : 5};
  const int e0 = r ? 7 : 6, e1 = r ? 9 : 8;
  auto mode_of = [&](int k, int q) { return K.plane * ((q < 6 ? q : q == 6 ? e0 : e1) + 10 * vn[k]); };   // q: 0..7
  auto at = [&](int s) -> double& { return ms[2 * (PAIR_BS * (s >> 1) + tid) + (s & 1)]; };
  auto pair = [&](int s) { return reinterpret_cast<const double2*>(ms)[PAIR_BS * (s >> 1) + tid]; };   // s even
  double du[PAIR_SLOTS];
#pragma unroll
  for (int s = 0; s < PAIR_SLOTS; ++s) du[s] = 0.0;
  if (__any_sync(0xffffffffu, interior)) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int q = 0; q < (k == 3 ? 8 : 6); ++q) at(6 * k + q) = U[item + mode_of(k, q)];
#pragma unroll 1
    for (int a = 0; a < NG; ++a) {
#pragma unroll 1
      for (int b = 0; b < NG; ++b) {
        const double* f = c_basis.phiG[a][b];
        const double f6 = f[6], f7 = f[7], f8 = f[8], f9 = f[9];
        const double fe0 = r ? f7 : f6, fe1 = r ? f9 : f8;
        double m[4], o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          double t[8];
#pragma unroll
          for (int q = 0; q < (k == 3 ? 8 : 6); q += 2) {
            const double2 z = pair(6 * k + q);
            t[q] = z.x;
            t[q + 1] = z.y;
          }
          double acc = 0.0 + t[0];
#pragma unroll
          for (int q = 1; q < 6; ++q) acc = acc + t[q] * f[q];
          if (k == 3) {
            acc = acc + t[6] * fe0;
            acc = acc + t[7] * fe1;
          }
          m[k] = acc;
          o[k] = __shfl_xor_sync(0xffffffffu, acc, 16);
        }
        const double rho = r ? o[0] : m[0], mx = r ? o[1] : m[1], my = r ? m[1] : o[1], mz = r ? m[0] : o[0];
        const double E = r ? o[2] : m[2], B1 = r ? o[3] : m[3], B2 = r ? m[3] : o[3], B3 = r ? m[2] : o[2];
        unsigned bad = 0;
        const Rcp rr = rcp_of(rho, bad);
        double u = rdiv(mx, rr, bad), vv = rdiv(my, rr, bad), w = rdiv(mz, rr, bad);
        if (bad) {   // an operand out of rdiv's range: the IEEE division itself
          u = ieee_div(mx, rho);
          vv = ieee_div(my, rho);
          w = ieee_div(mz, rho);
        }
        const double BB = sq(B1) + sq(B2) + sq(B3);
        const double p = K.P.gamma1 * (E - 0.5 * rho * (sq(u) + sq(vv) + sq(w)) - 0.5 * BB);
        const double S = p + 0.5 * BB;
        double Fx[4], Fy[4];
        // rho | m_z;  E | B3: T u - K B1 | u B3 - w B1, so a product with u (or v) less one with B1 (or B2)
        const double ru = rho * u, rv = rho * vv;
        Fx[0] = r ? ru * w - B1 * B3 : mx;
        Fy[0] = r ? rv * w - B2 * B3 : my;
        // m_x | m_y
        const double cross = ru * vv - B1 * B2;
        const double un = r ? vv : u, Bn = r ? B2 : B1;
        const double along = rho * sq(un) + S - sq(Bn);
        Fx[1] = r ? cross : along;
        Fy[1] = r ? along : cross;
        const double P1 = r ? B3 : E + S, P2 = r ? w : u * B1 + vv * B2 + w * B3;
        Fx[2] = P1 * u - P2 * B1;
        Fy[2] = P1 * vv - P2 * B2;
        // Bx | By
        const double ez = u * B2 - vv * B1;
        Fx[3] = r ? ez : 0.0;
        Fy[3] = r ? 0.0 : -ez;
        const double coef = 0.25 * c_basis.w[a] * c_basis.w[b];
        const double* px = phix[a][b];
        const double* py = phiy[a][b];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          double* d = du + 6 * k;
          d[1] = d[1] + coef * (Fx[k] * px[1]);
          d[2] = d[2] + coef * (Fy[k] * py[2]);
          d[3] = d[3] + coef * (Fx[k] * px[3]);
          d[4] = d[4] + coef * (Fx[k] * px[4] + Fy[k] * py[4]);
          d[5] = d[5] + coef * (Fy[k] * py[5]);
        }
        const double g0 = coef * (Fx[3] * px[7]), g1 = coef * (Fy[3] * py[8]);   // By's mode 8 | Bx's mode 9
        du[24] = du[24] + (r ? g0 : 0.0);
        du[25] = du[25] + (r ? 0.0 : g1);
      }
    }
  }
  if (!interior) {   // a ghost cell beside the others of its warp
#pragma unroll
    for (int s = 0; s < PAIR_SLOTS; ++s) du[s] = 0.0;
  } else {
    const long long ox = (i - 1) + 1 + (long long)(K.nx + 1) * (j - 1);  // Fxhat(i,j)
    const long long oy = (i - 1) + (long long)K.nx * j;                  // Fyhat(i,j)
    auto faces = [&](const double* F, long long pl, long long o, long long low, const double* cw,
                     const double (*fb)[NP], bool x) {
      const int across = x ? 1 : 2, along = x ? 2 : 1, across2 = x ? 3 : 5, along2 = x ? 5 : 3;
      // Bx's modes 7, 9 are odd across an x face and even across a y face, By's 8 and 10 the other way round
      const bool odd = (r == 0) == x;
      const double* G[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) G[k] = F + vn[k] * NG * pl + o;
#pragma unroll 1
      for (int g = 0; g < NG; ++g) {
        const double c = cw[g];
        const double* f = fb[g];
        const double f6 = f[6], f7 = f[7], f8 = f[8], f9 = f[9];
        const double fe0 = r ? f7 : f6, fe1 = r ? f9 : f8;
        double q1[4], q0[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          q1[k] = G[k][g * pl];
          q0[k] = G[k][g * pl - low];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          auto add = [&](int d, double t) { du[6 * k + d] = du[6 * k + d] - c * t; };
          add(0, q1[k] - q0[k]);
          add(across, q1[k] + q0[k]);
          add(across2, q1[k] * f[across2] - q0[k] * f[across2]);
          add(along2, q1[k] * f[along2] - q0[k] * f[along2]);
          if (g != 2) {
            const double l1 = q1[k] * f[along], l0 = q0[k] * f[along];
            add(along, l1 - l0);
            add(4, l1 + l0);
          }
          // the modes even across the face are odd along it, so zero at the middle point
          if (k == 3 && (odd || g != 2)) {
            add(6, q1[k] * fe0 + flip_if(q0[k] * fe0, !odd));
            add(7, q1[k] * fe1 + flip_if(q0[k] * fe1, !odd));
          }
        }
      }
    };
    faces(Fxh, K.fxplane, ox, 1, K.cxw, c_basis.phiGR, true);
    faces(Fyh, K.fyplane, oy, K.nx, K.cyw, c_basis.phiGU, false);
    // mm(1) = 1 (get_basis.f90): x / 1 == x
    const double m6 = c_basis.mm[6], m7 = c_basis.mm[7], m8 = c_basis.mm[8], m9 = c_basis.mm[9];
    const double r6 = c_basis.rmm[6], r7 = c_basis.rmm[7], r8 = c_basis.rmm[8], r9 = c_basis.rmm[9];
    const Rcp me0 = {r ? m7 : m6, r ? r7 : r6}, me1 = {r ? m9 : m8, r ? r9 : r8};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      unsigned bad = 0;
      double q[8];
#pragma unroll
      for (int d = 1; d < (k == 3 ? 8 : 6); ++d)
        q[d] = rdiv(du[6 * k + d], d < 6 ? Rcp{c_basis.mm[d], c_basis.rmm[d]} : d == 6 ? me0 : me1, bad);
#pragma unroll
      for (int d = 1; d < (k == 3 ? 8 : 6); ++d)
        du[6 * k + d] = bad ? ieee_div(du[6 * k + d], d < 6 ? c_basis.mm[d] : d == 6 ? me0.b : me1.b) : q[d];
    }
  }
  if (stage == 0) {
    if (interior) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int q = 0; q < (k == 3 ? 8 : 6); ++q) duout[item + mode_of(k, q)] = du[6 * k + q];
    }
    return;
  }
  if (!live) return;
  // the stage's combination, a variable at a time: its loads are all under way
  // before its first store
  const double dt = sc->dt;
  double na[8], nb[8];
  auto fetch = [&](int k) {
#pragma unroll
    for (int q = 0; q < (k == 3 ? 8 : 6); ++q) {
      const long long c = item + mode_of(k, q);
      na[q] = stage == 1 ? U[c] : UI[c];
      nb[q] = stage == 1 ? 0.0 : U0[c];
    }
  };
  fetch(0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    double a[8], b[8];
#pragma unroll
    for (int q = 0; q < (k == 3 ? 8 : 6); ++q) { a[q] = na[q]; b[q] = nb[q]; }
    if (k < 3) fetch(k + 1);
#pragma unroll
    for (int q = 0; q < (k == 3 ? 8 : 6); ++q) {
      const long long c = item + mode_of(k, q);
      const double v = a[q] + dt * du[6 * k + q];
      if (stage == 1) {
        U0[c] = a[q];
        UI[c] = v;
      } else if (stage == 2) {
        UI[c] = (3.0 / 4.0) * b[q] + (1.0 / 4.0) * v;
      } else {
        UI[c] = (1.0 / 3.0) * b[q] + (2.0 / 3.0) * v;
      }
    }
  }
}

// --------------------------------------------------- face-B update -------
// LhEz.f90:71-96 (dEz1 on x faces, dEz2 on y faces) and the face-B stage
// combine of RK3.f90. stage 0 writes dEz only (gdf_lhez).
__device__ __forceinline__ void bface_item(const Consts& K, const double* __restrict__ EzRL,
                                           const double* __restrict__ EzUD, const double* __restrict__ EzV,
                                           double* __restrict__ BX, double* __restrict__ BX0,
                                           double* __restrict__ BXI, double* __restrict__ BY,
                                           double* __restrict__ BY0, double* __restrict__ BYI,
                                           double* __restrict__ dez1, double* __restrict__ dez2,
                                           const Scal* __restrict__ sc, int stage, long long item) {
  const long long nbx = K.fxplane;
  double dez[3];
  long long o, fp;
  double *B, *B0, *BI, *dout;
  if (item < nbx) {
    const int i = (int)(item % (K.nx + 1));
    const int j = (int)(item / (K.nx + 1)) + 1;
    o = item;
    fp = K.fxplane;
    const double v1 = EzV[i + (long long)(K.nx + 1) * j];
    const double v0 = EzV[i + (long long)(K.nx + 1) * (j - 1)];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double acc = 0.0;
#pragma unroll
      for (int g = 0; g < NG; ++g) acc = acc + 0.5 * c_basis.w[g] * EzRL[g * fp + o] * K.EzyG[g][d];
      dez[d] = (acc - v1 * c_basis.EzU[d] / K.hy + v0 * c_basis.EzD[d] / K.hy) / c_basis.mmE[d];
    }
    B = BX; B0 = BX0; BI = BXI; dout = dez1;
  } else {
    const long long k = item - nbx;
    const int i = (int)(k % K.nx) + 1;
    const int j = (int)(k / K.nx);
    o = k;
    fp = K.fyplane;
    const double v1 = EzV[i + (long long)(K.nx + 1) * j];
    const double v0 = EzV[(i - 1) + (long long)(K.nx + 1) * j];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double acc = 0.0;
#pragma unroll
      for (int g = 0; g < NG; ++g) acc = acc - 0.5 * c_basis.w[g] * EzUD[g * fp + o] * K.EzxG[g][d];
      dez[d] = (acc + v1 * c_basis.EzR[d] / K.hx - v0 * c_basis.EzL[d] / K.hx) / c_basis.mmE[d];
    }
    B = BY; B0 = BY0; BI = BYI; dout = dez2;
  }
  if (stage == 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) dout[o + fp * d] = dez[d];
    return;
  }
  const double dt = sc->dt;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const long long c = o + fp * d;
    if (stage == 1) {
      const double b = B[c];
      B0[c] = b;
      const double bi = b + dt * dez[d];
      BI[c] = bi;
      B[c] = bi;
    } else if (stage == 2) {
      const double v = BI[c] + dt * dez[d];
      const double bii = (3.0 / 4.0) * B0[c] + (1.0 / 4.0) * v;
      BI[c] = bii;
      B[c] = bii;
    } else {
      const double v = BI[c] + dt * dez[d];
      B[c] = (1.0 / 3.0) * B0[c] + (2.0 / 3.0) * v;
    }
  }
}

// ------------------------------------------- learned-indicator features ---
// Per cell (ghosts included) the first six P2 modes of rho (copied), of the
// pressure and of |B|^2 (L2 projections with a 3x3 Gauss rule, in FP32):
// 18 floats per cell, QM[(q*6 + d) * plane + cell], q = rho, p, |B|^2.
// These feed the troubled-cell network; the FP64 solver state is untouched.
constexpr int QMODES = 18;

__device__ __forceinline__ float basis10(int d, float x, float y) {
  switch (d) {
    case 0: return 1.f;
    case 1: return x;
    case 2: return y;
    case 3: return x * x - (1.f / 3.f);
    case 4: return x * y;
    case 5: return y * y - (1.f / 3.f);
    case 6: return x * x * x - 0.6f * x;
    case 7: return (x * x - (1.f / 3.f)) * y;
    case 8: return x * (y * y - (1.f / 3.f));
    default: return y * y * y - 0.6f * y;
  }
}

__device__ __forceinline__ void qmodes_item(const Consts& K, const double* __restrict__ S, float* __restrict__ QM,
                                            long long c) {
  const float gx[3] = {-0.7745966692414834f, 0.f, 0.7745966692414834f};
  const float gw[3] = {5.f / 9.f, 8.f / 9.f, 5.f / 9.f};
  const float mmf[6] = {1.f, 1.f / 3.f, 1.f / 3.f, 4.f / 45.f, 1.f / 9.f, 4.f / 45.f};
  float m[NE][NP];
#pragma unroll
  for (int n = 0; n < NE; ++n)
#pragma unroll
    for (int d = 0; d < NP; ++d) m[n][d] = live_mode(n, d) ? (float)S[c + K.plane * (d + 10 * n)] : 0.f;
  float pm[6], bm[6];
#pragma unroll
  for (int d = 0; d < 6; ++d) { pm[d] = 0.f; bm[d] = 0.f; }
  const float g1 = (float)K.P.gamma1;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      float v[NE];
#pragma unroll
      for (int n = 0; n < NE; ++n) {
        float x = 0.f;
#pragma unroll
        for (int d = 0; d < NP; ++d)
          if (live_mode(n, d)) x += m[n][d] * basis10(d, gx[a], gx[b]);
        v[n] = x;
      }
      const float rho = v[0];
      const float b2 = v[5] * v[5] + v[6] * v[6] + v[7] * v[7];
      const float kin = (v[1] * v[1] + v[2] * v[2] + v[3] * v[3]) / rho;
      const float pr = g1 * (v[4] - 0.5f * kin - 0.5f * b2);
      const float wq = gw[a] * gw[b] * 0.25f;
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        const float ph = basis10(d, gx[a], gx[b]);
        pm[d] += wq * ph * pr;
        bm[d] += wq * ph * b2;
      }
    }
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    QM[(long long)d * K.plane + c] = m[0][d];
    QM[(long long)(6 + d) * K.plane + c] = pm[d] / mmf[d];
    QM[(long long)(12 + d) * K.plane + c] = bm[d] / mmf[d];
  }
}

// The 90 inputs of interior cell (i, j): for the cell and its neighbours
// (i+1,j), (i-1,j), (i,j+1), (i,j-1), the 6 modes of rho, p, |B|^2, each
// quantity scaled by the largest |mean| over the five cells, with the
// cell's own mean subtracted from the means; clamped to [-8, 8].
constexpr int NFEAT = 90;
__device__ __forceinline__ void gather_features(const Consts& K, const float* __restrict__ QM, long long c,
                                                float* out /* 90 */) {
  const long long nb[5] = {c, c + 1, c - 1, c + K.nx2, c - K.nx2};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    float sc = 0.f;
#pragma unroll
    for (int k = 0; k < 5; ++k) sc = fmaxf(sc, fabsf(QM[(long long)(q * 6) * K.plane + nb[k]]));
    sc = sc + 1e-30f;
    const float inv = 1.f / sc;
    const float mean_c = QM[(long long)(q * 6) * K.plane + c];
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        float v = QM[(long long)(q * 6 + d) * K.plane + nb[k]];
        if (d == 0) v -= mean_c;
        out[(k * 3 + q) * 6 + d] = fminf(8.f, fmaxf(-8.f, v * inv));
      }
  }
}


// ------------------------------------------------------------ limiter ----
// TVB_Limiter_P2.f90:16-121 (characteristic TVB, Jacobi over cells), with
// KXRCF_Detector.f90 as gate, pp_Limiter.f90, and div_free_Balsara.f90:13-79
// fused, for one interior cell. S is the pre-limit state (ghosts as the
// reference leaves them), D receives the limited state.
constexpr int LIM_BS = 64;
// dynamic shared memory of a learned-mode limiter block: X, W1t, W2t, H1
// tiles (BF16) and the LIM_BS logits
constexpr size_t LIMIT_SMEM_LEARNED = (size_t)(LIM_BS + MLP_H) * MLP_LDX * 2 + (size_t)(MLP_H + LIM_BS) * MLP_LDH * 2 +
                                      LIM_BS * sizeof(float);

__device__ __forceinline__ void matvec8(const double* A, const double* x, double* y) {
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) acc = acc + A[r + 8 * k] * x[k];
    y[r] = acc;
  }
}

// One face of KXRCF_Detector.f90:187-224 for one variable: I gains
// h1 w(g) (own trace - neighbour's trace) at the five points in order. AX 0: the
// right face (low: the left), 1: the upper (lower). m and k are the modes of the
// cell and of its neighbour, cubic the variable's live cubic modes (0 none, 1
// those of Bx, 2 those of By). The sums keep mode order; the tables' +-1
// entries and the zeros at the middle point are not multiplied.
template <int AX>
__device__ __forceinline__ void kxrcf_face(const double* m, const double* k, bool low, int cubic, double h1,
                                           double& I) {
  auto flip = [](double x, bool neg) { return neg ? -x : x; };   // the odd modes' sign on a low face
  auto trace = [&](const double* q, bool neg, int g) {
    const double* f = AX == 0 ? c_basis.phiGR[g] : c_basis.phiGU[g];
    const bool mid = g == 2;
    double v = 0.0 + q[0];
    if (AX == 0) v = v + flip(q[1], neg);
    else if (!mid) v = v + q[1] * f[1];
    if (AX == 1) v = v + flip(q[2], neg);
    else if (!mid) v = v + q[2] * f[2];
    v = v + q[3] * f[3];
    if (!mid) v = v + flip(q[4] * f[4], neg);
    v = v + q[5] * f[5];
    if (cubic == 1 && (AX == 0 || !mid)) {
      v = v + flip(q[6] * f[6], AX == 0 && neg);
      v = v + flip(q[7] * f[8], AX == 0 && neg);
    } else if (cubic == 2 && (AX == 1 || !mid)) {
      v = v + flip(q[6] * f[7], AX == 1 && neg);
      v = v + flip(q[7] * f[9], AX == 1 && neg);
    }
    return v;
  };
#pragma unroll
  for (int g = 0; g < NG; ++g) I = I + h1 * c_basis.w[g] * (trace(m, low, g) - trace(k, !low, g));
}

// KXRCF_Detector.f90:187-236 for cell c (interior): flagged when some |I(n)| /
// (pow L uinf(n)) reaches Ck, I the jump of the inflow faces, uinf the largest
// |value| of the cell at its 25 Gauss points. That maximum lies between two
// bounds that cost a few operations: the root mean square over the points (the
// basis is orthogonal) and the sum of |mode| max |phi|. Where a bound decides
// (with a margin of 1e-9, far above rounding) the points are not evaluated.
// One variable at a time, so that a cell's 52 modes are never held and the
// gating pass fits 128 registers. What bounded the detector was its loads, some
// 2,000 per cell (every face point re-read both cells' modes), at 8 warps per
// SM: the gating pass took 277 us on the rotor 512^2 after 100 steps, 177 with
// each face's modes read once, 126 as it is.
static __device__ bool kxrcf_flag(const Consts& K, const double* __restrict__ S, long long c) {
  const long long pl = K.plane;
  const bool r = S[c + 1 + pl * 10] < 0, l = S[c - 1 + pl * 10] > 0;            // uh(i+1,j,1,2) < 0: right side inflow
  const bool u = S[c + K.nx2 + pl * 20] < 0, w = S[c - K.nx2 + pl * 20] > 0;
  double Lij = 1e-12;
#pragma unroll
  for (int g = 0; g < 4 * NG; ++g) {
    const int side = g / NG;
    if (side == 0 ? r : side == 1 ? l : side == 2 ? u : w) Lij = Lij + (side < 2 ? K.hy : K.hx);
  }
  const double pL = K.pow_hxhy * Lij;
  const double cd = K.ck * pL;
  // squares are compared where theirs neither over- nor underflow
  const bool tame = cd > 1e-100 && cd < 1e100;
#pragma unroll 1
  for (int n = 0; n < NE; ++n) {
    const int cubic = n == 5 ? 1 : n == 6 ? 2 : 0;
    const double* Sn = S + c + pl * (10 * n);
    const long long x0 = pl * (cubic == 2 ? 7 : 6), x1 = pl * (cubic == 2 ? 9 : 8);
    auto load = [&](const double* q, double* m) {
#pragma unroll
      for (int d = 0; d < 6; ++d) m[d] = q[pl * d];
      m[6] = cubic ? q[x0] : 0.0;
      m[7] = cubic ? q[x1] : 0.0;
    };
    double m[8], k[8], I = 0.0;
    load(Sn, m);
    if (r) { load(Sn + 1, k); kxrcf_face<0>(m, k, false, cubic, K.hy1, I); }
    if (l) { load(Sn - 1, k); kxrcf_face<0>(m, k, true, cubic, K.hy1, I); }
    if (u) { load(Sn + K.nx2, k); kxrcf_face<1>(m, k, false, cubic, K.hx1, I); }
    if (w) { load(Sn - K.nx2, k); kxrcf_face<1>(m, k, true, cubic, K.hx1, I); }
    // a zero integral gives the ratio 0 (the denominator is positive)
    if (I == 0.0) {
      if (0.0 >= K.ck) return true;
      continue;
    }
    double up = fabs(m[0]), ms = m[0] * m[0];
#pragma unroll
    for (int d = 1; d < 6; ++d) {
      up = up + fabs(m[d]) * c_basis.ppM[d];
      ms = ms + m[d] * m[d] * c_basis.mm[d];
    }
    const int d6 = cubic == 2 ? 7 : 6, d7 = cubic == 2 ? 9 : 8;
    if (cubic) {
      up = up + fabs(m[6]) * c_basis.ppM[d6] + fabs(m[7]) * c_basis.ppM[d7];
      ms = ms + m[6] * m[6] * c_basis.mm[d6] + m[7] * m[7] * c_basis.mm[d7];
    }
    const double a = fabs(I);
    if (a > cd * (up + 1e-12) * (1.0 + 1e-9)) return true;
    if (tame && (a < cd * 1e-12 * (1.0 - 1e-9) || (ms < 1e200 && a * a < cd * cd * ms * (1.0 - 1e-8)))) continue;
    double uinf = 0.0;
#pragma unroll 1
    for (int q = 0; q < NG * NG; ++q) {
      const double* f = &c_basis.phiG[0][0][0] + NP * q;
      double v = 0.0;
#pragma unroll
      for (int d = 0; d < 6; ++d) v = v + m[d] * f[d];
      if (cubic) {
        v = v + m[6] * f[d6];
        v = v + m[7] * f[d7];
      }
      if (fabs(v) + 1e-12 > uinf) uinf = fabs(v) + 1e-12;
    }
    if (dv(a, pL * uinf) >= K.ck) return true;
  }
  return false;
}

__device__ __forceinline__ void divfree_item(const Consts& K, double* __restrict__ D, const double* __restrict__ BX,
                                             const double* __restrict__ BY, long long item);

// calculate_tq of pp_Limiter.f90:101-126
static __device__ double pp_tq(const Consts& K, const double* ubar, const double* uq) {
  double ta = 0.0, tb = 1.0;
  double ut[NE];
  // bisection on [0,1] to width 1e-14 ends after at most 47 halvings
#pragma unroll 1
  for (int it = 0; it < 64 && tb - ta > 1e-14; ++it) {
    const double tq = 0.5 * (ta + tb);
#pragma unroll
    for (int n = 0; n < NE; ++n) ut[n] = tq * uq[n] + (1 - tq) * ubar[n];
    if (pressure(K.P.gamma, ut) < 1e-12) tb = tq; else ta = tq;
  }
  return ta;
}

// pp_Limiter.f90:58-72: the share of u_q - u_bar that keeps the pressure of
// one point with pq < 0 positive
static __device__ double pp_point(const Consts& K, const double* ubar, const double* uq) {
  const double tq = pp_tq(K, ubar, uq);
  double n1 = 0.0, n2 = 0.0;
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    const double sqv = tq * uq[n] + (1 - tq) * ubar[n];
    n1 = n1 + sq(sqv - ubar[n]);
    n2 = n2 + sq(uq[n] - ubar[n]);
  }
  return sqrt(n1) / sqrt(n2);
}

// Bound on |u_q - u_bar| over the 50 GLL-mixed points for variable n:
// sum_d |m_d| max_q |phi_d(q)|, inflated to cover the rounding of the point
// sums (relative error < 2.3e-15 of |u_bar| + the bound).
__device__ __forceinline__ double pp_spread_of(double b, double mean) {
  return b * (1.0 + 1e-12) + 1e-12 * fabs(mean);
}
__device__ __forceinline__ double pp_spread(const Consts& K, const double (*m)[NP], int n) {
  double b = 0.0;
#pragma unroll
  for (int d = 1; d < NP; ++d)
    if (live_mode(n, d)) b = b + fabs(m[n][d]) * c_basis.ppM[d];
  return pp_spread_of(b, m[n][0]);
}

// Whether pp_Limiter.f90 leaves a cell alone: the density part acts only if
// some point has |rho_bar - rho_q| > rho_bar - 1e-13, the pressure part only
// if some point has a negative pressure. Where the bounds of pp_spread rule
// both out (with margins far above rounding) the point evaluations would
// change nothing.
__device__ __forceinline__ bool pp_rho_safe(double mean, double spread) {
  return spread < (mean - 1e-13) * (1.0 - 1e-12);
}
// a lower bound of the pressure at every point, from the variables' means and
// spreads; positive beyond rounding: no point has pq < 0
__device__ __forceinline__ bool pp_pressure_safe(const double* mean, const double* spread) {
  const double rho_lo = mean[0] - spread[0];
  if (!(rho_lo > 0.0)) return false;
  const double e_lo = mean[4] - spread[4];
  auto top = [&](int n) { return sq(fabs(mean[n]) + spread[n]); };
  const double k_hi = 0.5 * (top(1) + top(2) + top(3)) / rho_lo * (1.0 + 1e-12);
  const double b_hi = 0.5 * (top(5) + top(6) + top(7)) * (1.0 + 1e-12);
  const double p_lo = e_lo - k_hi - b_hi;
  return p_lo > 1e-10 * (fabs(e_lo) + k_hi + b_hi);
}
__device__ __forceinline__ bool pp_pressure_safe(const Consts& K, const double (*m)[NP]) {
  double mean[NE], spread[NE];
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    mean[n] = m[n][0];
    spread[n] = pp_spread(K, m, n);
  }
  return pp_pressure_safe(mean, spread);
}
__device__ __forceinline__ bool pp_quiet(const Consts& K, const double (*m)[NP]) {
  return pp_rho_safe(m[0][0], pp_spread(K, m, 0)) && pp_pressure_safe(K, m);
}

// pp_Limiter.f90:10-81 for one cell's modes (in place), by one thread: the
// ensemble's persistent stage kernel, whose limiter phase has no pass of its
// own for these cells (elsewhere pp_item_warp takes them).
static __device__ void pp_cell(const Consts& K, double (*m)[NP]) {
  const double epsilon = 1e-13;
  double eta = 1.0;
  const double rb = m[0][0];
  if (!pp_rho_safe(rb, pp_spread(K, m, 0))) {
#pragma unroll 1
    for (int a = 0; a < NG; ++a)
#pragma unroll 1
      for (int b = 0; b < NG; ++b)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          double rq = 0.0;
#pragma unroll
          for (int d = 0; d < NP; ++d)
            if (live_mode(0, d)) rq = rq + m[0][d] * c_basis.phiGLL[s][a][b][d];
          const double eta1 = fabs((rb - epsilon) / (rb - rq));
          if (eta1 < 1) eta = eta1;
        }
    if (eta < 1) {
      const double f = 0.5 * eta;
#pragma unroll
      for (int d = 1; d < NP; ++d) m[0][d] = f * m[0][d];
    }
  }
  if (pp_pressure_safe(K, m)) return;   // eta stays 1: nothing changes
  double ubar[NE];
#pragma unroll
  for (int n = 0; n < NE; ++n) ubar[n] = m[n][0];
  eta = 1.0;
  double eta1 = 1.0;
#pragma unroll 1
  for (int a = 0; a < NG; ++a)
#pragma unroll 1
    for (int b = 0; b < NG; ++b)
#pragma unroll 1
      for (int s = 0; s < 2; ++s) {
        double uq[NE];
#pragma unroll
        for (int n = 0; n < NE; ++n) {
          double acc = 0.0;
#pragma unroll
          for (int d = 0; d < NP; ++d)
            if (live_mode(n, d)) acc = acc + m[n][d] * c_basis.phiGLL[s][a][b][d];
          uq[n] = acc;
        }
        if (pressure(K.P.gamma, uq) < 0) eta1 = pp_point(K, ubar, uq);
        if (eta1 < eta) eta = eta1;
      }
  if (eta < 1) eta = 0.5 * eta;
#pragma unroll
  for (int n = 0; n < NE; ++n)
#pragma unroll
    for (int d = 1; d < NP; ++d) m[n][d] = eta * m[n][d];
}

// The 50 GLL-mixed points of pp_Limiter.f90 in its loop order, p = 2*(5*a +
// b) + s, transposed ([mode][point]) so that 32 lanes at 32 points read 32
// banks.
constexpr int PP_POINTS = 2 * NG * NG;
constexpr int PP_BS = 128;   // four cells per block
__device__ __forceinline__ void pp_stage_points(double* sb /* [NP * PP_POINTS] */) {
  for (int k = threadIdx.x; k < NP * PP_POINTS; k += blockDim.x) {
    const int d = k / PP_POINTS, p = k - d * PP_POINTS;
    sb[k] = c_basis.phiGLL[p & 1][p / (2 * NG)][(p >> 1) % NG][d];
  }
}

// pp_Limiter.f90:10-81 for one cell whose limited modes are in D, by one
// warp: a lane per point in two rounds, instead of one thread walking 50
// points of which each one with a negative pressure costs 47 dependent
// bisection steps. The density part keeps the last eta1 < 1 in point order
// (the highest lane of the later round that has one); the pressure part's
// running minimum is the same in any order. Then the div-free
// reconstruction where the limiter fuses it. sm: the warp's NLIVE doubles.
__device__ __forceinline__ void pp_item_warp(const Consts& K, double* __restrict__ D, const double* __restrict__ BX,
                                             const double* __restrict__ BY, int divfree, long long item,
                                             const double* sb, double* sm) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int i = (int)(item % K.nx) + 1, j = (int)(item / K.nx) + 1;
  const long long c = i + (long long)K.nx2 * j, pl = K.plane;
  for (int s = lane; s < NLIVE; s += 32) sm[s] = D[c + pl * (c_live_d[s] + 10 * c_live_n[s])];
  __syncwarp();
  const double epsilon = 1e-13, rb = sm[0];
  bool changed = false;
  double spread = 0.0;
#pragma unroll
  for (int d = 1; d < NP; ++d)
    if (live_mode(0, d)) spread = spread + fabs(sm[LI(0, d)]) * c_basis.ppM[d];
  if (!pp_rho_safe(rb, pp_spread_of(spread, rb))) {
    double eta = 1.0;
#pragma unroll 1
    for (int r = 1; r >= 0; --r) {
      const int p = lane + 32 * r;
      double eta1 = 1.0;
      if (p < PP_POINTS) {
        double rq = 0.0;
#pragma unroll
        for (int d = 0; d < NP; ++d)
          if (live_mode(0, d)) rq = rq + sm[LI(0, d)] * sb[d * PP_POINTS + p];
        eta1 = fabs((rb - epsilon) / (rb - rq));
      }
      const unsigned hit = __ballot_sync(full, eta1 < 1);
      if (hit) {
        eta = __shfl_sync(full, eta1, 31 - __clz(hit));
        break;
      }
    }
    if (eta < 1) {
      changed = true;
      const double f = 0.5 * eta;
      __syncwarp();
      if (lane >= 1 && lane < 6) sm[lane] = f * sm[lane];
      __syncwarp();
    }
  }
  double eta = 1.0;
#pragma unroll 1
  for (int r = 0; r < 2; ++r) {
    const int p = lane + 32 * r;
    if (p >= PP_POINTS) break;
    double uq[NE], ubar[NE];
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      double acc = 0.0;
#pragma unroll
      for (int d = 0; d < NP; ++d)
        if (live_mode(n, d)) acc = acc + sm[LI(n, d)] * sb[d * PP_POINTS + p];
      uq[n] = acc;
      ubar[n] = sm[LI(n, 0)];
    }
    if (pressure(K.P.gamma, uq) < 0) {
      const double eta1 = pp_point(K, ubar, uq);
      if (eta1 < eta) eta = eta1;
    }
  }
  __syncwarp();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double e = __shfl_xor_sync(full, eta, o);
    if (e < eta) eta = e;
  }
  if (eta < 1) {
    changed = true;
    eta = 0.5 * eta;
  }
  // modes 2.. of every variable scaled (eta = 1: by nothing)
  if (changed)
    for (int s = lane; s < NLIVE; s += 32) {
      const int n = c_live_n[s], d = c_live_d[s];
      if (d == 0 || (divfree && (n == 5 || n == 6))) continue;
      D[c + pl * (d + 10 * n)] = eta * sm[s];
    }
  if (divfree && lane == 0) divfree_item(K, D, BX, BY, item);
  __syncwarp();
}

__device__ __forceinline__ void lim_load(const Consts& K, const double* __restrict__ S, long long c, double (*m)[NP]) {
#pragma unroll
  for (int n = 0; n < NE; ++n)
#pragma unroll
    for (int d = 0; d < NP; ++d) m[n][d] = live_mode(n, d) ? S[c + K.plane * (d + 10 * n)] : 0.0;
}

// One interior cell (item < nx*ny). LIM_INFER: called by every thread of a
// LIM_BS-thread block on LIM_BS consecutive items (those past nx*ny idle),
// with lsm the block's LIMIT_SMEM_LEARNED bytes of dynamic shared memory.
// LM (the detector mode): LIM_PLAIN, the reference's detectors; LIM_INFER,
// the learned gate with inference (the first stage of a step: the block runs
// the network on its cells and stores each probability in pnet);
// LIM_PNET, the learned gate on the step's stored probabilities (stages 2
// and 3: the network sees the step's stage-1 pre-limit state).
constexpr int LIM_PLAIN = 0, LIM_INFER = 1, LIM_PNET = 2;
// Limiter of one interior cell in three pieces, composed by limit_item:
//   lim_gate    decides the gate (detector, sticky KXRCF flag, learned
//               probability); LIM_INFER runs the network for the block first
//               (block-cooperative)
//   lim_tvb     characteristic TVB limiting of a gated cell
//   lim_finish  positivity limiter, div-free reconstruction, store, flags
template <int LM>
__device__ __forceinline__ bool lim_gate(const Consts& K, const double* __restrict__ S, int32_t* __restrict__ trouble,
                                         const MlpDev* __restrict__ net, const float* __restrict__ QM,
                                         float* __restrict__ pnet, float t_lo, float t_hi, long long item,
                                         unsigned char* lsm, bool valid, long long c, int32_t& word) {
  float p_net = 0.f;
  if (LM == LIM_INFER) {
    // the learned indicator for the block's 64 cells on the tensor cores
    __nv_bfloat16* Xs = reinterpret_cast<__nv_bfloat16*>(lsm);
    __nv_bfloat16* W1t = Xs + LIM_BS * MLP_LDX;
    __nv_bfloat16* W2t = W1t + MLP_H * MLP_LDX;
    __nv_bfloat16* H1 = W2t + MLP_H * MLP_LDH;
    float* zz = reinterpret_cast<float*>(H1 + LIM_BS * MLP_LDH);
    const int tid = threadIdx.x;
    // weights: 16-byte rows pieces (W1t rows 12 x 16 B, W2t rows 8 x 16 B)
    const uint4* g1 = reinterpret_cast<const uint4*>(net->W1t);
    const uint4* g2 = reinterpret_cast<const uint4*>(net->W2t);
    for (int k = tid; k < MLP_H * (MLP_INP / 8); k += LIM_BS) {
      const int r = k / (MLP_INP / 8), q = k % (MLP_INP / 8);
      *reinterpret_cast<uint4*>(W1t + r * MLP_LDX + 8 * q) = g1[k];
    }
    for (int k = tid; k < MLP_H * (MLP_H / 8); k += LIM_BS) {
      const int r = k / (MLP_H / 8), q = k % (MLP_H / 8);
      *reinterpret_cast<uint4*>(W2t + r * MLP_LDH + 8 * q) = g2[k];
    }
    float f[MLP_INP];
    if (valid) {
      gather_features(K, QM, c, f);
    } else {
#pragma unroll
      for (int k = 0; k < NFEAT; ++k) f[k] = 0.f;
    }
#pragma unroll
    for (int k = NFEAT; k < MLP_INP; ++k) f[k] = 0.f;
#pragma unroll
    for (int q = 0; q < MLP_INP / 8; ++q) {
      uint4 v;
      __nv_bfloat162 a = __floats2bfloat162_rn(f[8 * q], f[8 * q + 1]);
      __nv_bfloat162 b = __floats2bfloat162_rn(f[8 * q + 2], f[8 * q + 3]);
      __nv_bfloat162 cc = __floats2bfloat162_rn(f[8 * q + 4], f[8 * q + 5]);
      __nv_bfloat162 d = __floats2bfloat162_rn(f[8 * q + 6], f[8 * q + 7]);
      v.x = *reinterpret_cast<uint32_t*>(&a);
      v.y = *reinterpret_cast<uint32_t*>(&b);
      v.z = *reinterpret_cast<uint32_t*>(&cc);
      v.w = *reinterpret_cast<uint32_t*>(&d);
      *reinterpret_cast<uint4*>(Xs + tid * MLP_LDX + 8 * q) = v;
    }
    __syncthreads();
    mlp_infer_tiles(Xs, W1t, W2t, net->b1, net->b2, net->w3, net->b3, H1, zz, LIM_BS);
    p_net = 1.f / (1.f + expf(-zz[tid]));
    if (valid) pnet[item] = p_net;
  } else if (LM == LIM_PNET) {
    if (valid) p_net = pnet[item];
  }
  if (!valid) return false;
  word = 0;
  bool gate = true;
  if (K.detector == GDF_DETECT_KXRCF) {
    // a set sticky flag stays set whatever the detector finds
    gate = (K.sticky && trouble[item] != 0) || kxrcf_flag(K, S, c);
    trouble[item] = gate ? 1 : 0;
    if (gate) word |= (1 << 24);
  } else if (LM != LIM_PLAIN) {
    // confident network answers decide; KXRCF decides in the uncertain band
    if (p_net >= t_hi) gate = true;
    else if (p_net >= t_lo) gate = kxrcf_flag(K, S, c);
    else gate = false;
    if (gate) word |= (1 << 24);
  }
  return gate;
}

// TVB_Limiter_P1.f90:19-90: characteristic minmod of the two slopes only;
// a changed variable keeps its limited slopes and loses every higher mode
static __device__ __noinline__ void lim_tvb_p1(const Consts& K, const double* __restrict__ S, long long c,
                                              double (*m)[NP], int32_t& word) {
  const long long pl = K.plane;
  const double rhoij = m[0][0];
  const double u1 = m[1][0] / rhoij, u2 = m[2][0] / rhoij, u3 = dv(m[3][0], rhoij);
  const double Eij = m[4][0], B1 = m[5][0], B2 = m[6][0], B3 = m[7][0];
  double R[64], L[64];
  double DR[NE], DL[NE], D1[NE], t1[NE], t2[NE], tu[NE], mod[NE], Xm[NE], Ym[NE];
  unsigned change = 0;
  eigenmatrix(K.P, 0, rhoij, u1, u2, u3, Eij, B1, B2, B3, R, L);
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    DR[n] = S[c + 1 + pl * (10 * n)] - m[n][0];
    DL[n] = m[n][0] - S[c - 1 + pl * (10 * n)];
    D1[n] = m[n][1];
  }
  matvec8(L, DR, t1);
  matvec8(L, DL, t2);
  matvec8(L, D1, tu);
#pragma unroll
  for (int k = 0; k < NE; ++k) mod[k] = minmod1(tu[k], t1[k], t2[k], K.Mh2x);
  matvec8(R, mod, Xm);
#pragma unroll
  for (int d = 0; d < NE; ++d)
    if (fabs(Xm[d] - D1[d]) > 1e-6) change |= 1u << d;
  eigenmatrix(K.P, 1, rhoij, u1, u2, u3, Eij, B1, B2, B3, R, L);
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    DR[n] = S[c + K.nx2 + pl * (10 * n)] - m[n][0];
    DL[n] = m[n][0] - S[c - K.nx2 + pl * (10 * n)];
    D1[n] = m[n][2];
  }
  matvec8(L, DR, t1);
  matvec8(L, DL, t2);
  matvec8(L, D1, tu);
#pragma unroll
  for (int k = 0; k < NE; ++k) mod[k] = minmod1(tu[k], t1[k], t2[k], K.Mh2y);
  matvec8(R, mod, Ym);
#pragma unroll
  for (int d = 0; d < NE; ++d)
    if (fabs(Ym[d] - D1[d]) > 1e-6) change |= 1u << d;
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    if (change & (1u << n)) {
#pragma unroll
      for (int d = 3; d < NP; ++d) m[n][d] = 0.0;
      m[n][1] = Xm[n];
      m[n][2] = Ym[n];
    }
  }
  word |= (int32_t)change;
}

// One direction of TVB_Limiter_P2.f90's characteristic part
// (:24-55 x, :57-90 y): the face slopes Dp (mean to + face) and Dm (- face
// to mean) limited against the mean differences DR, DL in the
// characteristic variables of the cell mean (minmod with the bound Mh2),
// back in conserved variables as Yp, Ym: the general path behind
// char_limit_sparse. The left eigenvectors are built
// and used in the four products with L before the right ones are built, so
// one 8x8 matrix is live at a time; the products and sums are those of
// eigenmatrix's R and L. With the identity fallback of eigenmatrix.f90:
// 397-404 (either matrix summing above 1e4 in absolute value) both
// matrices are the identity, and the products are taken with it.
__device__ __forceinline__ void char_limit_dir(const Consts& K, int dir, double rho, double u1, double u2,
                                               double u3, double E, double B1, double B2, double B3,
                                               const double* DR, const double* DL, const double* Dp,
                                               const double* Dm, double Mh2, double* Yp, double* Ym) {
  EigFrame f;
  eigen_frame(K.P, dir, rho, u1, u2, u3, E, B1, B2, B3, f);
  double t1[NE], t2[NE], tp[NE], tm[NE];
  double sl = 0.0;
  {
    double L[64];
    eigen_left(dir, f, rho, u1, u2, u3, B1, B2, B3, L);
    if (K.P.eig_identity) {
#pragma unroll
      for (int q = 0; q < 64; ++q) sl = sl + fabs(L[q]);
    }
    matvec8(L, DR, t1);
    matvec8(L, DL, t2);
    matvec8(L, Dp, tp);
    matvec8(L, Dm, tm);
  }
  double R[64];
  eigen_right(dir, f, rho, u1, u2, u3, B1, B2, B3, R);
  if (K.P.eig_identity) {
    double sr = 0.0;
#pragma unroll
    for (int q = 0; q < 64; ++q) sr = sr + fabs(R[q]);
    if (sr > 1e4 || sl > 1e4) {
#pragma unroll
      for (int q = 0; q < 64; ++q) R[q] = (q % 9 == 0) ? 1.0 : 0.0;
      matvec8(R, DR, t1);
      matvec8(R, DL, t2);
      matvec8(R, Dp, tp);
      matvec8(R, Dm, tm);
    }
  }
  double mod[NE];
#pragma unroll
  for (int k = 0; k < NE; ++k) mod[k] = minmod1(tp[k], t1[k], t2[k], Mh2);
  matvec8(R, mod, Yp);
#pragma unroll
  for (int k = 0; k < NE; ++k) mod[k] = minmod1(tm[k], t1[k], t2[k], Mh2);
  matvec8(R, mod, Ym);
}

// Operands of one direction for cell c: mean differences to the + and -
// neighbours (stride st) and the two face slopes of modes 2+dir, 4+2*dir.
__device__ __forceinline__ void tvb_operands(const Consts& K, const double* __restrict__ S, long long c, int dir,
                                             double* DR, double* DL, double* Dp, double* Dm) {
  const long long pl = K.plane, st = dir ? K.nx2 : 1;
  const double c23 = 2.0 / 3.0;
  const double* lo = S + c + pl * (1 + dir);
  const double* hi = S + c + pl * (3 + 2 * dir);
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    const long long o = pl * (10 * n);
    const double m0 = S[c + o], m1 = lo[o], m2 = hi[o];
    DR[n] = S[c + st + o] - m0;
    DL[n] = m0 - S[c - st + o];
    Dp[n] = m1 + c23 * m2;
    Dm[n] = m1 - c23 * m2;
  }
}
// which variables one direction's limited slopes change (TVB_Limiter_P2.f90:
// 45-52, 78-85), and the modes they give: res[n] = the slope, res[8 + n] = the
// quadratic mode
__device__ __forceinline__ unsigned tvb_change(const Consts& K, const double* Dp, const double* Dm, const double* Yp,
                                               const double* Ym, double* res) {
  unsigned change = 0;
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    if (fabs(Yp[n] - Dp[n]) > 1e-6 || fabs(Ym[n] - Dm[n]) > 1e-6) change |= 1u << n;
    res[n] = 0.5 * (Yp[n] + Ym[n]);
    res[NE + n] = K.tvb_slope * (Yp[n] - Ym[n]);
  }
  return change;
}
// both directions through the general path (cells char_limit_sparse refuses)
static __device__ __noinline__ unsigned tvb_general(const Consts& K, const double* __restrict__ S, long long c,
                                                    double* res) {
  double m[NE];
#pragma unroll
  for (int n = 0; n < NE; ++n) m[n] = S[c + K.plane * (10 * n)];
  const double u1 = m[1] / m[0], u2 = m[2] / m[0], u3 = m[3] / m[0];
  unsigned change = 0;
#pragma unroll 1
  for (int dir = 0; dir < 2; ++dir) {
    double DR[NE], DL[NE], Dp[NE], Dm[NE], Yp[NE], Ym[NE];
    tvb_operands(K, S, c, dir, DR, DL, Dp, Dm);
    const bool z = dir == 1 && K.eig_y_zero_w;
    if (dir == 0)
      char_limit_dir(K, 0, m[0], u1, u2, u3, m[4], m[5], m[6], m[7], DR, DL, Dp, Dm, K.Mh2x, Yp, Ym);
    else
      char_limit_dir(K, 1, m[0], u1, u2, z ? 0.0 : u3, m[4], m[5], m[6], z ? 0.0 : m[7], DR, DL, Dp, Dm, K.Mh2y, Yp,
                     Ym);
    change |= tvb_change(K, Dp, Dm, Yp, Ym, res + 2 * NE * dir);
  }
  return change;
}

// both directions through one copy of char_limit_sparse; false where it refuses
template <class DIV>
__device__ __forceinline__ bool tvb_sparse(const Consts& K, const double* __restrict__ S, long long c, double* res,
                                           unsigned& change) {
  unsigned bad = 0;
  change = 0;
  double m[NE];
#pragma unroll
  for (int n = 0; n < NE; ++n) m[n] = S[c + K.plane * (10 * n)];
  const auto rr = DIV::by(m[0], bad);
  const double u1 = DIV::div(m[1], rr, bad), u2 = DIV::div(m[2], rr, bad), u3 = DIV::div(m[3], rr, bad);
#pragma unroll 1
  for (int dir = 0; dir < 2; ++dir) {
    double DR[NE], DL[NE], Dp[NE], Dm[NE], Yp[NE], Ym[NE];
    tvb_operands(K, S, c, dir, DR, DL, Dp, Dm);
    const bool z = dir == 1 && K.eig_y_zero_w;
    const Minmod mm{dir ? K.Mh2y : K.Mh2x};
    bad |= (unsigned)!char_limit_sparse<DIV>(K.P, dir, m[0], u1, u2, z ? 0.0 : u3, m[4], m[5], m[6], z ? 0.0 : m[7],
                                             rr, DR, DL, Dp, Dm, mm, Yp, Ym);
    change |= tvb_change(K, Dp, Dm, Yp, Ym, res + 2 * NE * dir);
  }
  return !bad;
}
// the cells tvb_sparse<SharedRcp> refuses
static __device__ __noinline__ unsigned tvb_refused(const Consts& K, const double* __restrict__ S, long long c,
                                                    double* res) {
  unsigned change;
  return tvb_sparse<IeeeDiv>(K, S, c, res, change) ? change : tvb_general(K, S, c, res);
}

// TVB_Limiter_P2.f90:24-90: the limited slopes and quadratic modes of cell c
// in both directions (res[dir][slope 8, quadratic 8]); returns the changed
// variables.
__device__ __forceinline__ unsigned tvb_slopes(const Consts& K, const double* __restrict__ S, long long c,
                                               double* res) {
  unsigned change;
  return tvb_sparse<SharedRcp>(K, S, c, res, change) ? change : tvb_refused(K, S, c, res);
}

// the modes of the changed variables from tvb_slopes (TVB_Limiter_P2.f90:92-121)
__device__ __forceinline__ void tvb_apply(unsigned change, const double* res, double (*m)[NP]) {
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    if (change & (1u << n)) {
#pragma unroll
      for (int d = 6; d < NP; ++d) m[n][d] = 0.0;
      m[n][4] = 0.0;
      m[n][1] = res[n];
      m[n][2] = res[2 * NE + n];
      m[n][3] = res[NE + n];
      m[n][5] = res[3 * NE + n];
    }
  }
}

// the limiter of a gated cell whose modes m are loaded
__device__ __forceinline__ void lim_tvb(const Consts& K, const double* __restrict__ S, long long c,
                                        double (*m)[NP], int32_t& word) {
  if (K.tvb_p1) {
    lim_tvb_p1(K, S, c, m, word);
    return;
  }
  double res[4 * NE];
  const unsigned change = tvb_slopes(K, S, c, res);
  tvb_apply(change, res, m);
  word |= (int32_t)change;
}

// the cell's flag word (its byte of this stage and gate bit) and the health of
// its means
__device__ __forceinline__ void lim_flags(int32_t* __restrict__ flags, int stage, Scal* __restrict__ sc, long long item,
                                          int32_t word, double rho, double E) {
  if (flags) {
    int32_t w = (word & 0xff) << (8 * (stage - 1));
    if (word & (1 << 24)) w |= (1 << (23 + stage));
    if (stage <= 1) flags[item] = w; else flags[item] |= w;
  }
  if (!(rho > 0.0) || !isfinite(E)) atomicOr(&sc->status, 1);
}

// Cells left to a later pass: list entries are tag + item.
template <class T>
struct LimList {
  T* list;
  int32_t* count;
  T tag;
};

// Appends the gated cells among the calling warp's active lanes to the list
// (one atomic per warp); true for a gated cell.
template <class T>
__device__ __forceinline__ bool lim_defer(bool gate, long long item, const LimList<T>& l) {
  const unsigned act = __activemask();
  const unsigned bal = __ballot_sync(act, gate);
  if (!gate) return false;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(bal) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(l.count, __popc(bal));
  base = __shfl_sync(bal, base, leader);
  l.list[base + __popc(bal & ((1u << lane) - 1u))] = l.tag + (T)item;
  return true;
}

// PPD: a cell the positivity limiter may change is stored as it is and listed
// in pp (pp_item_warp limits and finishes it in a pass of its own); otherwise
// it is limited here.
template <bool PPD>
__device__ __forceinline__ void lim_finish(const Consts& K, double* __restrict__ D, const double* __restrict__ BX,
                                           const double* __restrict__ BY, int32_t* __restrict__ flags, int stage,
                                           int divfree, Scal* __restrict__ sc, long long item, int i, int j,
                                           long long c, double (*m)[NP], int32_t word,
                                           const LimList<long long>& pp) {
  const long long pl = K.plane;
  if (K.pp) {
    if (PPD) {
      if (lim_defer(!pp_quiet(K, m), item, pp)) divfree = 0;
    } else {
      pp_cell(K, m);
    }
  }
  if (divfree) {
    // div_free_Balsara.f90:30-75 from the four face polynomials
    const long long fxp = K.fxplane, fyp = K.fyplane;
    const long long ox = i + (long long)(K.nx + 1) * (j - 1);
    const long long oy = (i - 1) + (long long)K.nx * j;
    const double a0R = BX[ox], a1R = BX[ox + fxp], a2R = BX[ox + 2 * fxp];
    const double a0L = BX[ox - 1], a1L = BX[ox - 1 + fxp], a2L = BX[ox - 1 + 2 * fxp];
    const double b0U = BY[oy], b1U = BY[oy + fyp], b2U = BY[oy + 2 * fyp];
    const double b0D = BY[oy - K.nx], b1D = BY[oy - K.nx + fyp], b2D = BY[oy - K.nx + 2 * fyp];
    const double rxy = K.rxy, ryx = K.ryx;
    const double c16 = 1.0 / 6.0, c115 = 1.0 / 15.0, c14 = 1.0 / 4.0, c12 = 1.0 / 2.0;
#pragma unroll
    for (int d = 0; d < NP; ++d) { m[5][d] = 0.0; m[6][d] = 0.0; }
    m[5][0] = c12 * (a0R + a0L) + c16 * rxy * (b1U - b1D);
    m[5][1] = c12 * (a0R - a0L) + c115 * rxy * (b2U - b2D);
    m[5][2] = c12 * (a1R + a1L);
    m[5][3] = -c14 * rxy * (b1U - b1D);
    m[5][4] = c12 * (a1R - a1L);
    m[5][5] = c12 * (a2R + a2L);
    m[5][6] = -c16 * rxy * (b2U - b2D);
    m[5][8] = c12 * (a2R - a2L);
    m[6][0] = c12 * (b0U + b0D) + c16 * ryx * (a1R - a1L);
    m[6][2] = c12 * (b0U - b0D) + c115 * ryx * (a2R - a2L);
    m[6][1] = c12 * (b1U + b1D);
    m[6][5] = -c14 * ryx * (a1R - a1L);
    m[6][4] = c12 * (b1U - b1D);
    m[6][3] = c12 * (b2U + b2D);
    m[6][9] = -c16 * ryx * (a2R - a2L);
    m[6][7] = c12 * (b2U - b2D);
  }
#pragma unroll
  for (int n = 0; n < NE; ++n)
#pragma unroll
    for (int d = 0; d < NP; ++d)
      if (live_mode(n, d)) D[c + pl * (d + 10 * n)] = m[n][d];
  lim_flags(flags, stage, sc, item, word, m[0][0], m[4][0]);
}

// One interior cell of the limiter in one pass (the ensemble's persistent stage
// kernel).
template <int LM>
__device__ __forceinline__ void limit_item(const Consts& K, const double* __restrict__ S, double* __restrict__ D,
                                           const double* __restrict__ BX, const double* __restrict__ BY,
                                           int32_t* __restrict__ flags, int32_t* __restrict__ trouble, int stage,
                                           int divfree, Scal* __restrict__ sc, const MlpDev* __restrict__ net,
                                           const float* __restrict__ QM, float* __restrict__ pnet,
                                           float t_lo, float t_hi, long long item, unsigned char* lsm) {
  const bool valid = item < (long long)K.nx * K.ny;
  const int i = valid ? (int)(item % K.nx) + 1 : 1;
  const int j = valid ? (int)(item / K.nx) + 1 : 1;
  const long long c = i + (long long)K.nx2 * j;
  double m[NE][NP];
  int32_t word = 0;
  const bool gate = lim_gate<LM>(K, S, trouble, net, QM, pnet, t_lo, t_hi, item, lsm, valid, c, word);
  if (!valid) return;
  lim_load(K, S, c, m);
  if (gate) lim_tvb(K, S, c, m, word);
  lim_finish<false>(K, D, BX, BY, flags, stage, divfree, sc, item, i, j, c, m, word, LimList<long long>{});
}

// The gating pass: a gated cell is only listed in defer (limit_tvb_item
// finishes it over full warps, so the characteristic limiter never runs beside
// idle lanes); an ungated one is finished here, a variable at a time: its modes
// copied to D, the bounds of the positivity limiter gathered on the way, the
// cell left to pp where they do not rule it out.
template <int LM, class T>
__device__ __forceinline__ void limit_gate_item(const Consts& K, const double* __restrict__ S, double* __restrict__ D,
                                                const double* __restrict__ BX, const double* __restrict__ BY,
                                                int32_t* __restrict__ flags, int32_t* __restrict__ trouble, int stage,
                                                int divfree, Scal* __restrict__ sc, const MlpDev* __restrict__ net,
                                                const float* __restrict__ QM, float* __restrict__ pnet, float t_lo,
                                                float t_hi, long long item, unsigned char* lsm,
                                                const LimList<T>& defer, const LimList<long long>& pp) {
  const bool valid = item < (long long)K.nx * K.ny;
  const int i = valid ? (int)(item % K.nx) + 1 : 1;
  const int j = valid ? (int)(item / K.nx) + 1 : 1;
  const long long c = i + (long long)K.nx2 * j, pl = K.plane;
  int32_t word = 0;
  const bool gate = lim_gate<LM>(K, S, trouble, net, QM, pnet, t_lo, t_hi, item, lsm, valid, c, word);
  if (!valid) return;
  if (lim_defer(gate, item, defer)) return;
  double mean[NE], spread[NE];
#pragma unroll
  for (int n = 0; n < NE; ++n) {
    double b = 0.0;
#pragma unroll
    for (int d = 0; d < NP; ++d) {
      if (!live_mode(n, d)) continue;
      const double v = S[c + pl * (d + 10 * n)];
      D[c + pl * (d + 10 * n)] = v;
      if (d == 0) mean[n] = v;
      else b = b + fabs(v) * c_basis.ppM[d];
    }
    spread[n] = pp_spread_of(b, mean[n]);
  }
  if (K.pp && lim_defer(!(pp_rho_safe(mean[0], spread[0]) && pp_pressure_safe(mean, spread)), item, pp)) divfree = 0;
  if (divfree) divfree_item(K, D, BX, BY, item);
  lim_flags(flags, stage, sc, item, word, mean[0], mean[4]);
}

// A cell of the limiting pass: one that limit_gate_item listed, or with
// GDF_DETECT_ALL any. The detector bit is the one lim_gate
// sets (KXRCF and the learned gate set it; GDF_DETECT_ALL does not). The modes
// are loaded after the characteristic part, which needs few of them.
__device__ __forceinline__ void limit_tvb_item(const Consts& K, const double* __restrict__ S, double* __restrict__ D,
                                               const double* __restrict__ BX, const double* __restrict__ BY,
                                               int32_t* __restrict__ flags, int stage, int divfree,
                                               Scal* __restrict__ sc, long long item,
                                               const LimList<long long>& pp) {
  const int i = (int)(item % K.nx) + 1;
  const int j = (int)(item / K.nx) + 1;
  const long long c = i + (long long)K.nx2 * j;
  double m[NE][NP];
  int32_t word = K.detector != GDF_DETECT_ALL ? (1 << 24) : 0;
  if (K.tvb_p1) {
    lim_load(K, S, c, m);
    lim_tvb_p1(K, S, c, m, word);
  } else {
    double res[4 * NE];
    const unsigned change = tvb_slopes(K, S, c, res);
    lim_load(K, S, c, m);
    tvb_apply(change, res, m);
    word |= (int32_t)change;
  }
  lim_finish<true>(K, D, BX, BY, flags, stage, divfree, sc, item, i, j, c, m, word, pp);
}

// Face-B TVB limiter of TVB_Limiter_P2.f90:128-187 (applied when enabled):
// S holds the limited cell state with ghosts set, pre div-free.
__device__ __forceinline__ double minmodB(double a, double b, double c, double Mh2) {
  if (fabs(a) <= Mh2) return a;
  const double s = (sgn1(a) + sgn1(b) + sgn1(c)) / 3.0;
  if (fabs(s) == 1) return s * fmin2(fmin2(fabs(a), fabs(b)), fabs(c));
  return 0.0;
}

__device__ __forceinline__ void faceb_item(const Consts& K, const double* __restrict__ S, double* __restrict__ BX,
                                           double* __restrict__ BY, long long item) {
  const long long pl = K.plane;
  const double c23 = 2.0 / 3.0, c25 = 2.0 / 5.0;
  (void)c25;
  if (item < K.fxplane) {
    const int i = (int)(item % (K.nx + 1));
    const int j = (int)(item / (K.nx + 1)) + 1;
    const long long cL = i + (long long)K.nx2 * j, cR = cL + 1;
    const long long s6 = pl * 50;  // Bx slots start at d + 10*5
    // aRM(i,j,d) (d = 2,3) of cell i and aLM(i+1,j,d) of cell i+1
    const double aRM2 = S[cL + s6 + pl * 2] + S[cL + s6 + pl * 4];
    const double aRM3 = S[cL + s6 + pl * 5] + S[cL + s6 + pl * 8];
    const double aLM2 = S[cR + s6 + pl * 2] - S[cR + s6 + pl * 4];
    const double aLM3 = S[cR + s6 + pl * 5] - S[cR + s6 + pl * 8];
    BX[item + K.fxplane] = minmodB(BX[item + K.fxplane], aRM2, aLM2, K.Mh2x_b);
    BX[item + 2 * K.fxplane] = minmodB(BX[item + 2 * K.fxplane], aRM3, aLM3, K.Mh2x_b);
    (void)c23;
  } else if (item < K.fxplane + K.fyplane) {
    const long long k = item - K.fxplane;
    const int i = (int)(k % K.nx) + 1;
    const int j = (int)(k / K.nx);
    const long long cD = i + (long long)K.nx2 * j, cU = cD + K.nx2;
    const long long s7 = pl * 60;
    const double bUM2 = S[cD + s7 + pl * 1] + S[cD + s7 + pl * 4];
    const double bUM3 = S[cD + s7 + pl * 3] + S[cD + s7 + pl * 7];
    const double bDM2 = S[cU + s7 + pl * 1] - S[cU + s7 + pl * 4];
    const double bDM3 = S[cU + s7 + pl * 3] - S[cU + s7 + pl * 7];
    BY[k + K.fyplane] = minmodB(BY[k + K.fyplane], bUM2, bDM2, K.Mh2y_b);
    BY[k + 2 * K.fyplane] = minmodB(BY[k + 2 * K.fyplane], bUM3, bDM3, K.Mh2y_b);
  }
}

// div_free_Balsara.f90:13-79 on its own (used after the face-B limiter)
__device__ __forceinline__ void divfree_item(const Consts& K, double* __restrict__ D, const double* __restrict__ BX,
                                             const double* __restrict__ BY, long long item) {
  const int i = (int)(item % K.nx) + 1;
  const int j = (int)(item / K.nx) + 1;
  const long long c = i + (long long)K.nx2 * j;
  const long long pl = K.plane, fxp = K.fxplane, fyp = K.fyplane;
  const long long ox = i + (long long)(K.nx + 1) * (j - 1);
  const long long oy = (i - 1) + (long long)K.nx * j;
  const double a0R = BX[ox], a1R = BX[ox + fxp], a2R = BX[ox + 2 * fxp];
  const double a0L = BX[ox - 1], a1L = BX[ox - 1 + fxp], a2L = BX[ox - 1 + 2 * fxp];
  const double b0U = BY[oy], b1U = BY[oy + fyp], b2U = BY[oy + 2 * fyp];
  const double b0D = BY[oy - K.nx], b1D = BY[oy - K.nx + fyp], b2D = BY[oy - K.nx + 2 * fyp];
  const double rxy = K.rxy, ryx = K.ryx;
  const double c16 = 1.0 / 6.0, c115 = 1.0 / 15.0, c14 = 1.0 / 4.0, c12 = 1.0 / 2.0;
  double* X = D + c + pl * 50;
  double* Y = D + c + pl * 60;
  X[0] = c12 * (a0R + a0L) + c16 * rxy * (b1U - b1D);
  X[pl * 1] = c12 * (a0R - a0L) + c115 * rxy * (b2U - b2D);
  X[pl * 2] = c12 * (a1R + a1L);
  X[pl * 3] = -c14 * rxy * (b1U - b1D);
  X[pl * 4] = c12 * (a1R - a1L);
  X[pl * 5] = c12 * (a2R + a2L);
  X[pl * 6] = -c16 * rxy * (b2U - b2D);
  X[pl * 8] = c12 * (a2R - a2L);
  Y[0] = c12 * (b0U + b0D) + c16 * ryx * (a1R - a1L);
  Y[pl * 2] = c12 * (b0U - b0D) + c115 * ryx * (a2R - a2L);
  Y[pl * 1] = c12 * (b1U + b1D);
  Y[pl * 5] = -c14 * ryx * (a1R - a1L);
  Y[pl * 4] = c12 * (b1U - b1D);
  Y[pl * 3] = c12 * (b2U + b2D);
  Y[pl * 9] = -c16 * ryx * (a2R - a2L);
  Y[pl * 7] = c12 * (b2U - b2D);
}

// --------------------------------------------------------- dt -----------
// calculate_dt.f90:11-25: per-block maxima of |u_n +- c_f| over the cell
// averages, then one block folds them and advances t (RK3.f90:60-71).
constexpr int DT_BS = 256;

__device__ __forceinline__ double max_ign_nan(double a, double b) {
  if (b != b) return a;
  if (a != a) return b;
  return b > a ? b : a;
}

// calculate_dt.f90:15-22 for interior cell `item`: the largest |fast
// speeds| of its average in x (ax) and y (ay); flags a non-positive density
// or non-finite energy in sc->status.
__device__ __forceinline__ void dt_cell_speeds(const Consts& K, const double* __restrict__ U, long long item,
                                               double& ax, double& ay, Scal* __restrict__ sc) {
  const int i = (int)(item % K.nx) + 1;
  const int j = (int)(item / K.nx) + 1;
  const long long c = i + (long long)K.nx2 * j;
  double Uv[NE];
#pragma unroll
  for (int n = 0; n < NE; ++n) Uv[n] = U[c + K.plane * (10 * n)];
  double a1, a2;
  fast_speeds(K.P, Uv, 0, a1, a2);
  if (fabs(a1) > ax || fabs(a2) > ax) ax = fmax2(fabs(a1), fabs(a2));
  fast_speeds(K.P, Uv, 1, a1, a2);
  if (fabs(a1) > ay || fabs(a2) > ay) ay = fmax2(fabs(a1), fabs(a2));
  if (!(Uv[0] > 0.0) || !isfinite(Uv[4])) atomicOr(&sc->status, 1);
}

// calculate_dt.f90:23-25 and RK3.f90:60-71 from the grid maxima: mode 0
// sets dt only (gdf_dt); mode 1 takes a time step (t, dt, active, steps).
__device__ __forceinline__ void dt_advance(const Consts& K, double ax, double ay, Scal* __restrict__ sc, int mode) {
  double dt = K.cfl / (ax / K.hx + ay / K.hy);
  if (mode == 0) {
    sc->dt = dt;
    return;
  }
  double t = sc->t;
  if (!(t < sc->tend)) {
    sc->active = 0;
    return;
  }
  if (t + dt >= sc->tend) {
    dt = sc->tend - t;
    t = sc->tend;
  } else {
    t = t + dt;
  }
  if (K.dt_floor_stop && dt < 1e-7) t = sc->tend;
  if (!(dt > 0.0) || !isfinite(dt)) sc->status |= 1;
  sc->dt = dt;
  sc->t = t;
  sc->active = 1;
  sc->steps += 1;
}

// Fills this module's c_basis on the current device (the tables do not
// depend on the configuration). always: on every call (handle creation:
// survives a reset of the device between handles); otherwise once per
// device and process. Returns a cudaError_t.
static inline cudaError_t upload_basis_once(const Consts& K, bool always = false) {
  static std::mutex mu;
  static bool done[256] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 256) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(mu);
  if (done[dev] && !always) return cudaSuccess;
  Basis B;
  basis_of(K, B);
  e = cudaMemcpyToSymbol(c_basis, &B, sizeof(Basis));
  if (e == cudaSuccess) done[dev] = true;
  return e;
}

}  // namespace gdf

