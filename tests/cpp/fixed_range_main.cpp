// The fixed-point functions of FP64 stepping (fk_fixed.cuh) over every
// argument that the stepping kernels hand them, for a build that stops at
// undefined arithmetic: positions in the range of the problem functions and on
// its edges, and, as the kernels form the results before they know, positions
// outside it (large, infinite, NaN), which to_pos must refuse.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>
#include <vector>

#include "../../spac_gb300/csrc/fk_fixed.cuh"

using namespace fk::fx;

static double sink = 0;

static void functions(double x, double y) {
  i64 X, Y, ux, uy;
  const bool ok = to_pos(x, X) & to_pos(y, Y);
  const bool in = x >= -0.375 && x < 1.375 && y >= -0.375 && y < 1.375;
  if (ok != in) {
    std::printf("to_pos(%a, %a): %d\n", x, y, ok);
    std::exit(1);
  }
  FrankeArgs f;
  FrankeTerms b;
  franke_args(X, Y, f);
  franke_terms(tables(), f, b);
  franke_grad(f, b, ux, uy);
  sink += to_double(franke_lap(tables(), f), -54) + to_double(franke_u(b), -60) + to_double(franke_lap_terms(f, b), -54) +
          to_double(ux, -58) + to_double(uy, -58);
  const u64 a = aniso_a(tables(), X, Y);
  AnisoOut o;
  aniso_step(tables(), X, Y, a, o);
  aniso_grad(X, Y, o, ux, uy);
  sink += to_double(o.f, -51) + to_double(o.mc, 0u, -54) + to_double(ux, -54) + to_double(uy, -54) + aniso_sigma(a);
}

int main() {
  std::mt19937_64 rng(3);
  std::uniform_real_distribution<double> U(0, 1);
  std::vector<double> v = {0.0, -0.0, 1e-300, -1e-300, 0.5, 1.0, -0.375, std::nextafter(-0.375, -1), 1.375, std::nextafter(1.375, 0),
                           2.0, std::nextafter(2.0, 0), -2.0, 3.0, -7.5, 1e9, -1e300, std::numeric_limits<double>::infinity(),
                           -std::numeric_limits<double>::infinity(), std::numeric_limits<double>::quiet_NaN(), 2.0 / 9, 7.0 / 9,
                           4.0 / 9, 3.0 / 9, -1.0 / 9};
  for (int i = -64; i < 64; ++i) v.push_back(i / 32.0);
  for (double x : v)
    for (double y : v) functions(x, y);
  for (int i = 0; i < 300000; ++i) {
    const double w = i % 3 == 0 ? 1.0 : (i % 3 == 1 ? 1.75 : 4.0), lo = i % 3 == 0 ? 0.0 : (i % 3 == 1 ? -0.375 : -2.0);
    functions(lo + w * U(rng), lo + w * U(rng));
  }
  for (int i = 0; i < 300000; ++i) {
    const u32 a = i < 64 ? (i < 32 ? 1u << i : ~(1u << (i - 32))) : static_cast<u32>(rng()), b = static_cast<u32>(rng());
    double z0, z1;
    i64 k0, k1;
    normal_pair(tables(), a, b, z0, z1);
    normal_pair_fx(tables(), a, b, k0, k1);
    sink += z0 + z1 + static_cast<double>(k0 % 1024) + static_cast<double>(k1 % 1024);
    sink += exp_core(tables(), (U(rng) - 0.9) * std::ldexp(1.0, i % 8)) * 1e-60;
  }
  std::printf("ok %g\n", sink);
  return 0;
}
