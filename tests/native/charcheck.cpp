// Host build of the characteristic limiter (gdf_charlim.cuh) and of the general
// path it stands in for: eigen_left / eigen_right, the matrix products summed
// from zero in column order, minmod1, the identity fallback.
#include "../../freljord-cfd-arsenal_b200/csrc/gdf_charlim.cuh"

using namespace gdf;

static void matvec(const double* A, const double* x, double* y) {
  for (int r = 0; r < 8; ++r) {
    double acc = 0.0;
    for (int k = 0; k < 8; ++k) acc = acc + A[r + 8 * k] * x[k];
    y[r] = acc;
  }
}
static double minmod_beta(double a, double b, double c, double Mh2, double beta) {
  if (fabs(a) <= Mh2) return a;
  const double s = (sgn1(a) + sgn1(b) + sgn1(c)) / 3.0;
  if (fabs(s) == 1) return s * fmin2(fmin2(fabs(a), beta * fabs(b)), beta * fabs(c));
  return 0.0;
}

extern "C" {
// n quotients: q = rdiv's, returns how many operands raised the flag
int cc_div(int n, const double* a, const double* b, double* q) {
  int flagged = 0;
  for (int k = 0; k < n; ++k) {
    unsigned bad = 0;
    const Rcp r = rcp_of(b[k], bad);
    q[k] = rdiv(a[k], r, bad);
    if (bad) {
      ++flagged;
      q[k] = a[k] / b[k];
    }
  }
  return flagged;
}
// prm = {gamma_flux, Mh2, beta}, iprm = {dir, eig_p_typo, eig_identity, with beta, IEEE division};
// prim = rho, u1..3, E, B1..3; x = DR, DL, Dp, Dm (8 each). out: fast Yp, Ym,
// general Yp, Ym. Returns 1 where the fast path answered.
int cc_limit(const double* prm, const int* iprm, const double* prim, const double* x, double* out) {
  Phys P{};
  P.gflux = prm[0];
  P.eig_p_typo = iprm[1];
  P.eig_identity = iprm[2];
  set_eig_consts(P);
  const double *DR = x, *DL = x + 8, *Dp = x + 16, *Dm = x + 24;
  unsigned bad = 0;
  const Rcp rr = rcp_of(prim[0], bad);
  bool ok;
  if (iprm[4])
    ok = iprm[3] ? char_limit_sparse<IeeeDiv>(P, iprm[0], prim[0], prim[1], prim[2], prim[3], prim[4], prim[5], prim[6],
                                              prim[7], IeeeDiv::by(prim[0], bad), DR, DL, Dp, Dm,
                                              MinmodBeta{prm[1], prm[2]}, out, out + 8)
                 : char_limit_sparse<IeeeDiv>(P, iprm[0], prim[0], prim[1], prim[2], prim[3], prim[4], prim[5], prim[6],
                                              prim[7], IeeeDiv::by(prim[0], bad), DR, DL, Dp, Dm, Minmod{prm[1]}, out,
                                              out + 8);
  else
  if (iprm[3])
    ok = char_limit_sparse<SharedRcp>(P, iprm[0], prim[0], prim[1], prim[2], prim[3], prim[4], prim[5], prim[6], prim[7], rr, DR, DL,
                         Dp, Dm, MinmodBeta{prm[1], prm[2]}, out, out + 8);
  else
    ok = char_limit_sparse<SharedRcp>(P, iprm[0], prim[0], prim[1], prim[2], prim[3], prim[4], prim[5], prim[6], prim[7], rr, DR, DL,
                         Dp, Dm, Minmod{prm[1]}, out, out + 8);
  double R[64], L[64], t1[8], t2[8], tp[8], tm[8], mod[8];
  eigenmatrix(P, iprm[0], prim[0], prim[1], prim[2], prim[3], prim[4], prim[5], prim[6], prim[7], R, L);
  matvec(L, DR, t1);
  matvec(L, DL, t2);
  matvec(L, Dp, tp);
  matvec(L, Dm, tm);
  auto mm = [&](double a, double b, double c) {
    return iprm[3] ? minmod_beta(a, b, c, prm[1], prm[2]) : minmod1(a, b, c, prm[1]);
  };
  for (int k = 0; k < 8; ++k) mod[k] = mm(tp[k], t1[k], t2[k]);
  matvec(R, mod, out + 16);
  for (int k = 0; k < 8; ++k) mod[k] = mm(tm[k], t1[k], t2[k]);
  matvec(R, mod, out + 24);
  return ok && !bad;
}
}
