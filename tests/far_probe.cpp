// Test infrastructure: the FP32 distance of cell offsets and the histogram bin the pair kernel takes from it, against
// the Float64 distance of the coordinates, for boxes near and far from the origin (built by tests/test_far_bins.py with
// g++ -ffp-contract=off).
#include <cmath>
#include <cstdint>
#include <random>
#include <vector>

#include "clm_build_steps.cuh"

namespace {

template <int N> int run(const double* side, double origin, double cutoff, int lcell, int n, int nbins, int64_t* out) {
  double M[3][3] = {}, o[3] = {0, 0, 0};
  for (int i = 0; i < N; i++) {
    M[i][i] = side[i];
    o[i] = i == 1 ? -0.3 * origin : origin;
  }
  clm::Geometry<double> g;
  const int st = clm::make_geometry<double>(g, N, clm::NONPERIODIC, M, cutoff, lcell, o);
  if (st) return st;
  clm::DevGeom<double> d;
  clm::fill_devgeom<double>(g, 0, d);
  const float err = (float)(clm::offset_distance_error(g) * 1.001);
  std::vector<double> edges((size_t)nbins + 1);
  std::vector<float> ef((size_t)nbins + 1);
  for (int b = 0; b <= nbins; b++) ef[(size_t)b] = (float)(edges[(size_t)b] = 0.9 * cutoff * std::pow(10.0, 4.0 * (b - nbins) / nbins));
  std::mt19937_64 rng(11);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  for (int k = 0; k < 4; k++) out[k] = 0;
  for (int t = 0; t < n; t++) {
    double x[3] = {0, 0, 0}, y[3] = {0, 0, 0}, u[3], s = 0;
    // half of the distances within a millionth of an edge
    const double r0 = U(rng) < 0.5 ? edges[(size_t)(1 + (int)(U(rng) * nbins))] * (1.0 + 1e-6 * (U(rng) - 0.5))
                                   : cutoff * std::pow(10.0, -5.0 * U(rng));
    for (int k = 0; k < N; k++) {
      x[k] = o[k] + side[k] * (0.1 + 0.8 * U(rng));
      u[k] = U(rng) - 0.5;
      s += u[k] * u[k];
    }
    for (int k = 0; k < N; k++) y[k] = x[k] + u[k] * (r0 / std::sqrt(s));
    const int ci = clm::cell_of<double, N>(d, x, true), cj = clm::cell_of<double, N>(d, y, true);
    if (ci < 0 || cj < 0) continue;
    double px[2], py[2], pz[2];
    float4 off[2], xq[2];
    int code[2], a[3], b[3];
    clm::gather_copy<double, N>(d, d.shift, x, 0, 0, d.zero_code, ci, px, py, pz, off, xq, code);
    clm::gather_copy<double, N>(d, d.shift, y, 1, 1, d.zero_code, cj, px, py, pz, off, xq, code);
    clm::cart_of(ci, d.nc, N, a);
    clm::cart_of(cj, d.nc, N, b);
    // as the kernel stages the candidate and takes the distance
    const float oi[3] = {off[0].x, off[0].y, off[0].z};
    const float oj[3] = {off[1].x, off[1].y, off[1].z};
    float dv[3] = {0, 0, 0};
    double dx[3] = {0, 0, 0};
    for (int k = 0; k < N; k++) {
      dv[k] = oi[k] - (oj[k] + d.csf[k] * (float)(b[k] - a[k]));
      dx[k] = x[k] - y[k];
    }
    const float rf = std::sqrt(std::fma(dv[2], dv[2], std::fma(dv[1], dv[1], dv[0] * dv[0])));
    const double r = std::sqrt(clm::xadd(clm::xadd(dx[0] * dx[0], dx[1] * dx[1]), dx[2] * dx[2]));
    out[0]++;
    if (std::fabs((double)rf - r) > err + 4.0 * std::ldexp(1.0, -24) * r) out[1]++;
    const int lo = clm::first_edge_at_or_above(ef.data(), nbins, rf);
    const bool again = clm::near_edge(ef.data(), nbins, lo, rf, err);
    if (!again && lo != clm::first_edge_at_or_above(edges.data(), nbins, r)) out[2]++;
    out[3] += again ? 1 : 0;
  }
  return 0;
}

}  // namespace

extern "C" int far_probe(int dim, const double* side, double origin, double cutoff, int lcell, int n, int nbins, int64_t* out) {
  return dim == 3 ? run<3>(side, origin, cutoff, lcell, n, nbins, out) : run<2>(side, origin, cutoff, lcell, n, nbins, out);
}
