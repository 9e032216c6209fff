// The vertex solvers (LF, HLL, HLLC and HLLD_Flux_2D.f90) with four lanes to a
// vertex: lane 0 has the upper right cell's corner state, 1 the upper left one's, 2
// the lower right, 3 the lower left.
//
// An HLLD vertex is four states (primitives, two directions' speeds and fluxes) and
// four one-dimensional solves, some 2,500 double operations of which 92 are
// divisions and 40 square roots. One thread for all of it needed 168 registers
// with IEEE divisions, spilled with shared reciprocals, and ran a straight line
// of code four times as long. Here each lane reads one corner, forms what its
// two solves need and does one of the solves:
//   lane 0  upper  x solve  right RU (own)    left LU (lane 1)
//   lane 1  left   y solve  upper LU (own)    lower LD (lane 3)
//   lane 2  right  y solve  upper RU (lane 0) lower RD (own)
//   lane 3  lower  x solve  right RD (lane 2) left LD (own)
// so each lane sends one direction's values to one lane and takes another's.
// Blast 2048^2 (HLLD) 0.99 ms per launch, 1.31 with one thread per vertex; rotor
// 512^2 92 us, 107 before; HLL at k = 3, 480 x 240 36 us, 56 before.
#pragma once
#include "gdf_physics.cuh"

namespace gdf {

// What a solve takes of one side, in the frame of its normal: the component
// along the normal (n) and the one beside it in the plane (s); Fn, Fs are the
// fluxes of the normal momentum and of the field component s.
struct VHalf {
  double rho, mn, ms, Bn, Bs, un, us, Fn, Fs;
};

GDF_HD void vertex_halves(const Phys& P, const Side& s, VHalf& x, VHalf& y) {
  double Fx[NE], Fy[NE];
  side_flux_hard(P, s, Fx, Fy);
  x = {s.rho, s.U[1], s.U[2], s.B1, s.B2, s.u, s.v, Fx[1], Fx[6]};
  y = {s.rho, s.U[2], s.U[1], s.B2, s.B1, s.v, s.u, Fy[2], Fy[5]};
}

// hllcd_flux's flux of the field component s, the only one the vertex takes
// (x solves: -Ez, y solves: Ez). Nothing else of hllcd_flux enters it; the two
// directions' operations are the same up to the order of an addition's operands.
template <bool HLLD, class DIV>
GDF_HD double vertex_solve(const Phys& P, const VHalf& R, const VHalf& L, double SR, double SL, unsigned& bad) {
  if (SR < 0) return R.Fs;
  if (SL > 0) return L.Fs;
  const auto rS = DIV::by(SR - SL, bad);
  const double U0 = DIV::div(SR * R.rho - SL * L.rho + L.mn - R.mn, rS, bad);
  const double Un = DIV::div(SR * R.mn - SL * L.mn + L.Fn - R.Fn, rS, bad);
  const double Us = DIV::div(SR * R.Bs - SL * L.Bs + L.Fs - R.Fs, rS, bad);
  const double Sstar = DIV::div(Un, DIV::by(U0, bad), bad);
  if (HLLD) {
    const double Bsb = DIV::div(SR * R.Bn - SL * L.Bn, rS, bad);
    const double dR = SR - R.un, dL = SL - L.un;
    const double eR = SR - Sstar, eL = SL - Sstar;
    const auto reR = DIV::by(eR, bad), reL = DIV::by(eL, bad);
    const double rhoRs = DIV::div(R.rho * dR, reR, bad);
    const double rhoLs = DIV::div(L.rho * dL, reL, bad);
    const auto rrR = DIV::by(rhoRs, bad), rrL = DIV::by(rhoLs, bad);
    const double SRs = Sstar + DIV::root(DIV::div(sq(Bsb), rrR, bad));
    const double SLs = Sstar - DIV::root(DIV::div(sq(Bsb), rrL, bad));
    if ((fabs(Bsb) > P.hlld_eps) && (SRs - SLs > P.hlld_eps) && !(SLs > 0) && !(SRs < 0)) {
      const double AR = R.rho * sq(dR) - Bsb * R.Bn;
      const double AL = L.rho * sq(dL) - Bsb * L.Bn;
      const double CR = R.rho * dR * (R.Bn - Bsb);
      const double CL = L.rho * dL * (L.Bn - Bsb);
      const double DR = R.rho * dR * eR - sq(Bsb) + 1e-15;
      const double DL = L.rho * dL * eL - sq(Bsb) + 1e-15;
      const double BRs = DIV::div(AR * R.Bs + CR * R.us, DIV::by(DR, bad), bad);
      const double BLs = DIV::div(AL * L.Bs + CL * L.us, DIV::by(DL, bad), bad);
      const double mRs = DIV::div(R.ms * dR + R.Bn * R.Bs - Bsb * BRs, reR, bad);
      const double mLs = DIV::div(L.ms * dL + L.Bn * L.Bs - Bsb * BLs, reL, bad);
      const double uRs = DIV::div(mRs, rrR, bad);
      const double uLs = DIV::div(mLs, rrL, bad);
      const double sL = DIV::root(fabs(rhoLs)), sR = DIV::root(fabs(rhoRs));
      const double sg = sgn1(Bsb);
      const double sLR = DIV::root(fabs(rhoLs * rhoRs));
      const double Bss = DIV::div(sL * BLs + sR * BRs + sg * sLR * (uRs - uLs), DIV::by(sL + sR, bad), bad);
      if (Sstar > 0) return L.Fs + SL * (Us - L.Bs) + SLs * (Bss - Us);
      return R.Fs + SR * (Us - R.Bs) + SRs * (Bss - Us);
    }
    if ((fabs(Bsb) > P.hlld_eps) && (SRs - SLs > P.hlld_eps)) {
      if (SLs > 0) return L.Fs + SL * (Us - L.Bs);
      return R.Fs + SR * (Us - R.Bs);
    }
  }
  return Sstar > 0 ? L.Fs + SL * (Us - L.Bs) : R.Fs + SR * (Us - R.Bs);
}

// hll1_cm: the same flux component (f) and the normal field component (b)
template <class DIV>
GDF_HD void vertex_hll(const VHalf& R, const VHalf& L, double SR, double SL, double& f, double& b, unsigned& bad) {
  if (SR < 0) {
    f = R.Fs; b = R.Bn;
  } else if (SL > 0) {
    f = L.Fs; b = L.Bn;
  } else {
    const auto rS = DIV::by(SR - SL, bad);
    f = DIV::div(SR * L.Fs - SL * R.Fs + SL * SR * (R.Bs - L.Bs), rS, bad);
    b = DIV::div(SR * R.Bn - SL * L.Bn, rS, bad);
  }
}

// one corner's speeds: the largest and smallest in x, then in y
template <class DIV>
GDF_HD void vertex_corner(const Phys& P, const double* U, VHalf& x, VHalf& y, double* S, unsigned& bad) {
  SideOf<DIV> s;
  make_side(P, U, s, bad);
  side_speeds(P, s, 0, S[0], S[1], bad);
  side_speeds(P, s, 1, S[2], S[3], bad);
  vertex_halves(P, s, x, y);
}

// S: the four corners' speeds, extreme over them in vertex_ez's order
GDF_HD double vertex_speed(int k, const double* a) {
  return (k & 1) ? fmin2(fmin2(fmin2(a[0], a[1]), a[2]), a[3]) : fmax2(fmax2(fmax2(a[0], a[1]), a[2]), a[3]);
}

// Ez of the vertex from the speeds SR, SL, SU, SD and the solves' fluxes (upper, left, right, lower)
GDF_HD double vertex_pick(const double* S, const double* f) {
  const double fU = f[0], fL = f[1], fR = f[2], fD = f[3];
  if (S[1] > 0) return fL;
  if (S[0] < 0) return fR;
  if (S[3] > 0) return -fD;
  if (S[2] < 0) return -fU;
  return 0.25 * (fR + fL + -fU + -fD);
}

// HLL: S as above, the solves' fluxes and fields, the corners' fields B1, B2 (RU, LU, RD, LD)
template <class DIV>
GDF_HD double vertex_pick_hll(const double* S, const double* f, const double* b, const double* B1, const double* B2,
                              unsigned& bad) {
  const double SR = S[0], SL = S[1], SU = S[2], SD = S[3];
  const double EzUs = -f[0], EzLs = f[1], EzRs = f[2], EzDs = -f[3];
  const double BxUs = b[0], ByLs = b[1], ByRs = b[2], BxDs = b[3];
  if (SL > 0) return EzLs;
  if (SR < 0) return EzRs;
  if (SD > 0) return EzDs;
  if (SU < 0) return EzUs;
  // the corner Ez values are never assigned in the reference and taken as 0 (vertex_ez)
  const double z = 0.0;
  const auto rden = DIV::by(2 * (SR - SL) * (SU - SD), bad);
  const double BxSS = DIV::div(2 * SR * SU * B1[0] - 2 * SL * SU * B1[1] + 2 * SL * SD * B1[3] - 2 * SR * SD * B1[2] -
                             SR * (z - z) + SL * (z - z) - (SR - SL) * (EzUs - EzDs), rden, bad);
  const double BySS = DIV::div(2 * SR * SU * B2[0] - 2 * SL * SU * B2[1] + 2 * SL * SD * B2[3] - 2 * SR * SD * B2[2] +
                             SU * (z - z) - SD * (z - z) + (SU - SD) * (EzRs - EzLs), rden, bad);
  return 0.25 * (EzRs + EzLs + EzUs + EzDs) - 0.25 * SU * (BxUs - BxSS) - 0.25 * SD * (BxDs - BxSS) +
         0.25 * SR * (ByRs - BySS) + 0.25 * SL * (ByLs - BySS);
}

// LF: one corner's |u|, |v|, Ez (calculate_Ez.f90), B1, B2, and the vertex from the four
// corners' (v[c] is corner c's)
template <class DIV>
GDF_HD void vertex_corner_lf(const double* U, double* v, unsigned& bad) {
  const auto rr = DIV::by(U[0], bad);
  const double u1 = DIV::div(U[1], rr, bad), u2 = DIV::div(U[2], rr, bad);
  v[0] = fabs(u1);
  v[1] = fabs(u2);
  v[2] = u2 * U[5] - u1 * U[6];
  v[3] = U[5];
  v[4] = U[6];
}
GDF_HD double vertex_pick_lf(const double (*v)[5]) {
  const double ax = fmax2(fmax2(fmax2(v[0][0], v[1][0]), v[2][0]), v[3][0]);
  const double ay = fmax2(fmax2(fmax2(v[0][1], v[1][1]), v[2][1]), v[3][1]);
  return 0.25 * (v[0][2] + v[1][2] + v[2][2] + v[3][2]) - 0.25 * ay * (0.5 * (v[0][3] + v[1][3]) - 0.5 * (v[2][3] + v[3][3])) +
         0.25 * ax * (0.5 * (v[0][4] + v[2][4]) - 0.5 * (v[1][4] + v[3][4]));
}

#if defined(__CUDACC__)
// A whole warp comes here together, eight vertices (with a mask of its own for
// each four lanes the warp runs them one after another: 2.9 ms on the blast 2048^2). U: the lane's corner state. The Ez of the vertex (in each lane)
// is in Ez; false, in the whole warp, when an operand of any lane left DIV's range.
// FLUX: Phys::flux, 1 LF, 2 HLL, 3 HLLC, 4 HLLD.
template <int FLUX, class DIV>
__device__ __forceinline__ bool vertex_quad(const Phys& P, const double* U, double& Ez) {
  const int lane = threadIdx.x & 31, q = lane & 3, base = lane & ~3;
  unsigned bad = 0;
  if (FLUX == 1) {
    double mine[5], v[4][5];
    vertex_corner_lf<DIV>(U, mine, bad);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int k = 0; k < 5; ++k) v[c][k] = __shfl_sync(0xffffffffu, mine[k], base + c);
    Ez = vertex_pick_lf(v);
    return !__any_sync(0xffffffffu, bad);
  }
  VHalf x, y;
  double S[4];
  vertex_corner<DIV>(P, U, x, y, S, bad);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    double a[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) a[c] = __shfl_sync(0xffffffffu, S[k], base + c);
    S[k] = vertex_speed(k, a);
  }
  const bool isx = q == 0 || q == 3;
  const bool own_right = q < 2;                            // own corner is the solve's right (upper) side
  const int from = base + ((0x2031 >> (4 * q)) & 3);       // lanes 1, 3, 0, 2
  VHalf R, L;
  auto trade = [&](double vx, double vy, double& r, double& l) {
    const double mine = isx ? vx : vy;
    const double other = __shfl_sync(0xffffffffu, isx ? vy : vx, from);   // a lane sends the direction it does not solve
    r = own_right ? mine : other;
    l = own_right ? other : mine;
  };
  trade(x.rho, y.rho, R.rho, L.rho);
  trade(x.mn, y.mn, R.mn, L.mn);
  trade(x.ms, y.ms, R.ms, L.ms);
  trade(x.Bn, y.Bn, R.Bn, L.Bn);
  trade(x.Bs, y.Bs, R.Bs, L.Bs);
  trade(x.un, y.un, R.un, L.un);
  trade(x.us, y.us, R.us, L.us);
  trade(x.Fn, y.Fn, R.Fn, L.Fn);
  trade(x.Fs, y.Fs, R.Fs, L.Fs);
  double F, B = 0;
  if (FLUX == 2) vertex_hll<DIV>(R, L, isx ? S[0] : S[2], isx ? S[1] : S[3], F, B, bad);
  else F = vertex_solve<FLUX == 4, DIV>(P, R, L, isx ? S[0] : S[2], isx ? S[1] : S[3], bad);
  double f[4], b[4], B1[4], B2[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    f[c] = __shfl_sync(0xffffffffu, F, base + c);
    if (FLUX == 2) {
      b[c] = __shfl_sync(0xffffffffu, B, base + c);
      B1[c] = __shfl_sync(0xffffffffu, U[5], base + c);
      B2[c] = __shfl_sync(0xffffffffu, U[6], base + c);
    }
  }
  if (FLUX == 2) Ez = vertex_pick_hll<DIV>(S, f, b, B1, B2, bad);
  else Ez = vertex_pick(S, f);
  return !__any_sync(0xffffffffu, bad);
}
#endif

}  // namespace gdf
