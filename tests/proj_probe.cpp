// Test infrastructure: the bound below which the pair kernel keeps a pair without the projection filter
// (DevGeom::proj_lo), against the filter itself, on pairs placed where it is closest to rejecting them (built by
// tests/test_projection_bound.py with g++ -ffp-contract=off).
#include <cmath>
#include <cstdint>
#include <random>

#include "clm_build_steps.cuh"

namespace {

// The cell of a point.  The border-case shift belongs to real particles, which lie in the unit cell but for rounding: a
// point that it would move is a real particle only within a few units of the face.
template <int N> int cell_at(const clm::DevGeom<double>& d, const double* x, bool real) {
  for (int k = 0; k < N && real; k++) {
    const double tol = 32.0 * std::ldexp(1.0, -53) * (std::fabs(d.cbmin[k]) + std::fabs(d.cbmax[k]));
    const double lo = d.cbmin[k] + d.cs[k] * d.lcell, hi = d.cbmin[k] + d.cs[k] * (d.nc[k] - d.lcell);
    real = x[k] >= lo - tol && x[k] <= hi + tol;
  }
  return clm::cell_of<double, N>(d, x, real);
}

template <int N> int run(int kind, const double* Mcol, const double* origin, double cutoff, int lcell, int n, int64_t* out) {
  double M[3][3] = {};
  for (int i = 0; i < N; i++)
    for (int j = 0; j < N; j++) M[i][j] = (kind != clm::TRICLINIC && i != j) ? 0.0 : Mcol[j * N + i];
  clm::Geometry<double> g;
  double o[3] = {0, 0, 0};
  if (origin)
    for (int i = 0; i < N; i++) o[i] = origin[i];
  const int st = clm::make_geometry<double>(g, N, kind, M, cutoff, lcell, kind == clm::NONPERIODIC ? o : nullptr);
  if (st) return st;
  clm::DevGeom<double> d;
  clm::fill_devgeom<double>(g, 1, d);
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  for (int k = 0; k < 4; k++) out[k] = 0;
  const double r0 = std::sqrt(d.proj_lo);
  for (int t = 0; t < n; t++) {
    double x[3] = {0, 0, 0}, y[3] = {0, 0, 0}, u[3], s = 0;
    for (int k = 0; k < N; k++) {
      // on a face of a cell (within a few units), or anywhere
      const double c = std::floor(U(rng) * (d.nc[k] - 2)) + 1.0;
      x[k] = d.cbmin[k] + d.cs[k] * (U(rng) < 0.6 ? c : c + U(rng));
      const int steps = (int)(U(rng) * 7) - 3;
      for (int q = 0; q < std::abs(steps); q++) x[k] = std::nextafter(x[k], steps < 0 ? -1e300 : 1e300);
    }
    // along the line between two cell centres, where the projection is the distance, or near it
    const double noise = U(rng) < 0.5 ? 0.0 : std::pow(10.0, -9.0 * U(rng));
    for (int k = 0; k < N; k++) {
      u[k] = d.cs[k] * ((int)(U(rng) * (2 * lcell + 1)) - lcell) + noise * (U(rng) - 0.5);
      s += u[k] * u[k];
    }
    if (s == 0) continue;
    const double r = r0 * (1.0 - (U(rng) < 0.7 ? 4.0 * U(rng) * std::ldexp(1.0, -53) : U(rng) * 1e-6));
    for (int k = 0; k < N; k++) y[k] = x[k] + u[k] * (r / std::sqrt(s));
    double dx[3];
    for (int k = 0; k < N; k++) dx[k] = x[k] - y[k];
    double d2 = dx[0] * dx[0];
    for (int k = 1; k < N; k++) d2 += dx[k] * dx[k];
    const int ci = cell_at<N>(d, x, true), cj = cell_at<N>(d, y, U(rng) < 0.5);
    if (ci < 0 || cj < 0 || ci == cj || d2 > d.proj_lo) continue;
    int a[3], b[3];
    clm::cart_of(ci, d.nc, N, a);
    clm::cart_of(cj, d.nc, N, b);
    bool near = true;
    for (int k = 0; k < N; k++) near = near && std::abs(a[k] - b[k]) <= lcell;
    if (!near) continue;
    double ca[3], cb[3];
    clm::cell_center<double, N>(d, a, ca);
    clm::cell_center<double, N>(d, b, cb);
    out[0]++;
    out[1] += d2 > d.thr_lo ? 1 : 0;
    if (!clm::projection_pass<double, N>(d, ca, cb, x, y)) out[2]++;
    if (!clm::projection_pass<double, N>(d, cb, ca, y, x)) out[2]++;
  }
  out[3] = d.proj_lo > (double)d.thr_lo;
  return 0;
}

}  // namespace

extern "C" int proj_probe(int dim, int kind, const double* Mcol, const double* origin, double cutoff, int lcell, int n,
                          int64_t* out) {
  return dim == 3 ? run<3>(kind, Mcol, origin, cutoff, lcell, n, out) : run<2>(kind, Mcol, origin, cutoff, lcell, n, out);
}
