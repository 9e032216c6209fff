// Host build of the four-lane vertex solver (csrc/gdf_vertex.cuh): the lanes one
// after another, against vertex_ez.
#include "../../freljord-cfd-arsenal_b200/csrc/gdf_vertex.cuh"

using namespace gdf;

template <int FLUX, class DIV>
static double four(const Phys& P, const double* U, unsigned& bad) {
  if (FLUX == 1) {
    double v[4][5];
    for (int c = 0; c < 4; ++c) vertex_corner_lf<DIV>(U + 8 * c, v[c], bad);
    return vertex_pick_lf(v);
  }
  VHalf x[4], y[4];
  double s[4][4], S[4], f[4], b[4], B1[4], B2[4];
  for (int c = 0; c < 4; ++c) {
    vertex_corner<DIV>(P, U + 8 * c, x[c], y[c], s[c], bad);
    B1[c] = U[8 * c + 5];
    B2[c] = U[8 * c + 6];
  }
  for (int k = 0; k < 4; ++k) {
    const double a[4] = {s[0][k], s[1][k], s[2][k], s[3][k]};
    S[k] = vertex_speed(k, a);
  }
  auto solve = [&](int i, const VHalf& R, const VHalf& L, double SR, double SL) {
    if (FLUX == 2) vertex_hll<DIV>(R, L, SR, SL, f[i], b[i], bad);
    else f[i] = vertex_solve<FLUX == 4, DIV>(P, R, L, SR, SL, bad);
  };
  solve(0, x[0], x[1], S[0], S[1]);
  solve(1, y[1], y[3], S[2], S[3]);
  solve(2, y[0], y[2], S[2], S[3]);
  solve(3, x[2], x[3], S[0], S[1]);
  return FLUX == 2 ? vertex_pick_hll<DIV>(S, f, b, B1, B2, bad) : vertex_pick(S, f);
}
template <int FLUX>
static double run(const Phys& P, const double* U, int& shared) {
  unsigned bad = 0, any = 0;
  const double v = four<FLUX, SharedRcp>(P, U, bad);
  shared = !bad;
  return bad ? four<FLUX, IeeeDiv>(P, U, any) : v;
}

// U: n vertices x 4 corners (RU, LU, RD, LD) x 8; how[i]: 1 if shared reciprocals took it
extern "C" void vertex_four(double gamma, double gflux, double eps, int flux, long long n, const double* U, double* got,
                            double* want, int* how) {
  Phys P = {};
  P.gamma = gamma; P.gamma1 = gamma - 1; P.gflux = gflux; P.hlld_eps = eps; P.flux = flux;
  for (long long i = 0; i < n; ++i) {
    const double* V = U + 32 * i;
    got[i] = flux == 1 ? run<1>(P, V, how[i]) : flux == 2 ? run<2>(P, V, how[i]) : flux == 3 ? run<3>(P, V, how[i]) : run<4>(P, V, how[i]);
    want[i] = vertex_ez(P, V, V + 8, V + 16, V + 24);
  }
}
