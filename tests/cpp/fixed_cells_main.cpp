// Errors of the fixed-point problem functions of FP64 stepping (fk_fixed.cuh)
// against long double, cell by cell over the range of positions that they
// accept, beside those of the FP64 forms that they replace, with the fused
// multiply-adds that a GPU compiler forms and sines rounded correctly.  One
// line per cell of 1/8 and function: name, the cell's lower left corner, rms,
// mean and largest error, then the FP64 form's.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../spac_gb300/csrc/fk_fixed.cuh"

using namespace fk::fx;
typedef long double ld;

constexpr int kFuns = 11;
const char* kNames[kFuns] = {"u", "ux", "uy", "lap", "lap_terms", "a", "sigma", "f", "mc", "Ux", "Uy"};

template <typename T>
static void forms(double x, double y, ld (&o)[kFuns]) {
  auto fm = [](T a, T b, T c) { return std::fma(a, b, c); };
  auto sn = [](double v) { return T(sinl(acosl(-1.0L) * ((ld)v - rintl((ld)v / 2) * 2))); };  // sin(pi v)
  const T px = x, py = y;
  const T a = fm(9, px, -2), b = fm(9, py, -2), c = fm(9, px, 1), d = fm(9, py, 1), p = fm(9, px, -7), q = fm(9, py, -3),
          r = fm(9, px, -4), t = fm(9, py, -7);
  const T s1 = fm(a, a, b * b), s3 = fm(p, p, q * q), s4 = fm(r, r, t * t);
  const T e1 = std::exp(T(-0.25) * s1), e2 = std::exp(fm(T(-1) / 49, c * c, T(-1) / 10 * d)), e3 = std::exp(T(-0.25) * s3), e4 = std::exp(-s4);
  const T u = fm(T(-1) / 5, e4, fm(T(0.5), e3, fm(T(0.75), e1, T(0.75) * e2)));
  const T ux = fm(T(18) / 5 * r, e4, fm(T(-2.25) * p, e3, fm(T(-27) / 98 * c, e2, T(-3.375) * a * e1)));
  const T uy = fm(T(18) / 5 * t, e4, fm(T(-2.25) * q, e3, fm(T(-27) / 40, e2, T(-3.375) * b * e1)));
  const T lap = fm(fm(T(-324) / 5, s4, T(324) / 5), e4,
                   fm(fm(T(10.125), s3, T(-40.5)), e3,
                      fm(fm(T(486) / 4802, c * c, -(T(243) / 98 - T(243) / 400)), e2, fm(T(15.1875), s1, T(-60.75)) * e1)));
  const T av = fm(T(0.5) * sn(2 * x), sn(2 * y), 1);
  const T k = fm(px, py, 1), mc = fm(py, py, fm(px, px, 1)), bx = py - T(0.5), by = T(0.5) - px;
  const T Ux = fm(ux, k, u * py), Uy = fm(uy, k, u * px), L = fm(lap, k, 2 * fm(ux, py, uy * px));
  const ld v[kFuns] = {u, ux, uy, lap, lap, av, std::sqrt(2 * av), -fm(-mc, u * k, fm(by, Uy, fm(av, L, bx * Ux))), mc, Ux, Uy};
  for (int j = 0; j < kFuns; ++j) o[j] = v[j];
}

static void fixed(double x, double y, ld (&o)[kFuns]) {
  i64 X, Y, ux, uy, gx, gy;
  if (!to_pos(x, X) || !to_pos(y, Y)) std::abort();
  FrankeArgs fa;
  FrankeTerms ft;
  franke_args(X, Y, fa);
  franke_terms(tables(), fa, ft);
  franke_grad<61>(fa, ft, ux, uy);
  const u64 a62 = aniso_a(tables(), X, Y);
  AnisoParts<55, 59> s;
  aniso_step(tables(), X, Y, a62, s);
  aniso_grad<60>(X, Y, s, gx, gy);
  const ld v[kFuns] = {to_double(franke_u<62>(ft), -62), to_double(ux, -61), to_double(uy, -61), to_double(franke_lap<56>(tables(), fa), -56),
                       to_double(franke_lap_terms<56>(fa, ft), -56), to_double(a62, 0u, -62), aniso_sigma(a62), to_double(s.f, -55),
                       to_double(s.mc, 0u, -59), to_double(gx, -60), to_double(gy, -60)};
  for (int j = 0; j < kFuns; ++j) o[j] = v[j];
}

int main(int argc, char**) {
  std::mt19937_64 rng(11);
  std::uniform_real_distribution<double> U(0, 1);
  const int cells = 14, n = argc > 1 ? 40000 : 1500;
  for (int ci = 0; ci < cells; ++ci)
    for (int cj = 0; cj < cells; ++cj) {
      const double x0 = -0.375 + 0.125 * ci, y0 = -0.375 + 0.125 * cj;
      struct {
        ld s2 = 0, s = 0, m = 0;
        void add(ld v) {
          s2 += v * v;
          s += v;
          m = fmaxl(m, fabsl(v));
        }
      } A[kFuns], D[kFuns];
      for (int i = 0; i < n; ++i) {
        const double x = x0 + 0.125 * U(rng), y = y0 + 0.125 * U(rng);
        ld e[kFuns], k[kFuns], v[kFuns];
        forms<ld>(x, y, e);
        forms<double>(x, y, k);
        fixed(x, y, v);
        for (int j = 0; j < kFuns; ++j) {
          A[j].add(v[j] - e[j]);
          D[j].add(k[j] - e[j]);
        }
      }
      for (int j = 0; j < kFuns; ++j)
        std::printf("%s %.3f %.3f %.4Lg %.4Lg %.4Lg %.4Lg %.4Lg %.4Lg\n", kNames[j], x0, y0, sqrtl(A[j].s2 / n), A[j].s / n, A[j].m,
                    sqrtl(D[j].s2 / n), D[j].s / n, D[j].m);
    }
  return 0;
}
