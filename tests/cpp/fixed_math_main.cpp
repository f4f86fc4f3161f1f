// Errors of the fixed-point functions of FP64 stepping (fk_fixed.cuh) against
// long double, on seeded samples and on the ends of their ranges.  Prints
// one line "name max_error" each.
#include <cmath>
#include <cstdio>
#include <random>

#include "../../spac_gb300/csrc/fk_fixed.cuh"

using namespace fk::fx;
typedef long double ld;

static void put(const char* name, ld e) { std::printf("%s %.6Lg\n", name, e); }

int main() {
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> U(0, 1);
  const ld pi = acosl(-1.0L);
  // e^v: relative error in units of 2^-53
  ld e = 0;
  auto try_exp = [&](double v) {
    const ld x = expl((ld)v);
    e = fmaxl(e, fabsl((ld)exp_core(tables(), v) - x) / x * 9007199254740992.0L);
  };
  for (int i = 0; i < 1000000; ++i) try_exp(-100 + 110 * U(rng));
  for (int i = 0; i < 200000; ++i) try_exp((U(rng) - 0.5) * std::ldexp(1.0, -(i % 60)));
  for (int j = -8192; j < 2048; ++j) {
    try_exp(j * 0.6931471805599453 / 1024);
    try_exp(std::nextafter(j * 0.6931471805599453 / 1024, -1e9));
  }
  try_exp(255.99);
  try_exp(-255.99);
  put("exp_ulp", e);
  // -ln u: absolute
  e = 0;
  auto try_log = [&](u32 a) {
    int ex;
    const u64 l = neg_log(tables(), a, ex);
    e = fmaxl(e, fabsl(l * ldexpl(1, ex - 1) + logl(((ld)a + 0.5L) * ldexpl(1, -32))));
  };
  for (int i = 0; i < 1000000; ++i) try_log((u32)rng());
  for (int i = 0; i < 32; ++i)
    for (int d = -3; d < 4; ++d) {
      try_log((u32)(1ull << i) + d);
      try_log(~((u32)(1ull << i) + d));
    }
  for (u32 j = 0; j < 512; ++j)
    for (int d = -2; d < 3; ++d) try_log((j << 22 | 1u << 31) + d);
  put("neg_log_abs", e);
  // cos, sin: absolute
  e = 0;
  auto try_sc = [&](u32 b) {
    u64 c, s;
    sincos_quadrant(tables(), b, c, s);
    const ld t = 2 * pi * ((ld)(b & 0x3fffffffu) + 0.5L) * ldexpl(1, -32);
    e = fmaxl(e, fmaxl(fabsl(c * ldexpl(1, -63) - cosl(t)), fabsl(s * ldexpl(1, -63) - sinl(t))));
  };
  for (int i = 0; i < 1000000; ++i) try_sc((u32)rng());
  for (u32 j = 0; j < 1024; ++j) {
    try_sc(j << 20);
    try_sc((j << 20) | 0xfffffu);
    try_sc((j << 20) | 0x7ffffu);
    try_sc((j << 20) | 0x80000u);
  }
  put("sincos_abs", e);
  // square root: relative in units of 2^-53
  e = 0;
  for (int i = 0; i < 1000000; ++i) {
    const u64 L = (rng() >> (i % 60)) | 1u;
    int ex;
    const u64 r = sqrt_norm(L, -58, ex);
    const ld x = sqrtl((ld)L * ldexpl(1, -58));
    e = fmaxl(e, fabsl((ld)r * ldexpl(1, ex) - x) / x * 9007199254740992.0L);
  }
  put("sqrt_ulp", e);
  // normal pair: absolute, and the FP64 forms' beside it
  e = 0;
  ld f = 0, e2 = 0, f2 = 0, efx = 0;
  const int n = 1000000;
  for (int i = 0; i < n; ++i) {
    const u32 a = i < 64 ? (i < 32 ? 1u << i : ~(1u << (i - 32))) : (u32)rng(), b = (u32)rng();
    double z0, z1;
    normal_pair(tables(), a, b, z0, z1);
    const ld u1 = ((ld)a + 0.5L) * ldexpl(1, -32), u2 = ((ld)b + 0.5L) * ldexpl(1, -32), r = sqrtl(-2 * logl(u1));
    const ld x0 = r * cosl(2 * pi * u2), x1 = r * sinl(2 * pi * u2);
    const double du1 = (a + 0.5) * 2.3283064365386962890625e-10, du2 = (b + 0.5) * 2.3283064365386962890625e-10;
    const double dr = std::sqrt(-2.0 * std::log(du1));
    const ld d0 = dr * std::cos(6.283185307179586 * du2), d1 = dr * std::sin(6.283185307179586 * du2);
    i64 k0, k1;
    normal_pair_fx(tables(), a, b, k0, k1);
    efx = fmaxl(efx, fmaxl(fabsl(k0 * ldexpl(1, -53) - x0), fabsl(k1 * ldexpl(1, -53) - x1)));
    const ld m = fmaxl(fabsl(z0 - x0), fabsl(z1 - x1)), k = fmaxl(fabsl(d0 - x0), fabsl(d1 - x1));
    e = fmaxl(e, m);
    f = fmaxl(f, k);
    e2 += m * m;
    f2 += k * k;
  }
  put("normal_fx_abs", efx);
  put("normal_abs", e);
  put("normal_abs_fp64", f);
  put("normal_rms", sqrtl(e2 / n));
  put("normal_rms_fp64", sqrtl(f2 / n));
  // Franke function and the anisotropic problem: rms over the square and the
  // largest error, against the FP64 forms' own
  struct Acc {
    ld s2 = 0, m = 0;
    void add(ld v) { s2 += v * v; m = fmaxl(m, fabsl(v)); }
  } A[16], D[16];
  const int np = 300000;
  for (int i = 0; i < np; ++i) {
    const double lo = i & 1 ? -0.375 : 0.0, w = i & 1 ? 1.75 : 1.0;
    const double x = lo + w * U(rng), y = lo + w * U(rng);
    i64 X, Y;
    if (!to_pos(x, X) || !to_pos(y, Y)) return 1;
    struct R { ld u, ux, uy, lap, a, s, f, mc, Ux, Uy; };
    auto ref = [&](auto one) {
      typedef decltype(one) T;
      const T px = x, py = y;
      const T a = 9 * px - 2, b = 9 * py - 2, c = 9 * px + 1, d = 9 * py + 1, p = 9 * px - 7, q = 9 * py - 3, r = 9 * px - 4, t = 9 * py - 7;
      const T s1 = a * a + b * b, s3 = p * p + q * q, s4 = r * r + t * t;
      const T e1 = std::exp(-s1 / 4), e2 = std::exp(T(-1) / 49 * (c * c) - d / 10), e3 = std::exp(-s3 / 4), e4 = std::exp(-s4);
      R o;
      const T u = T(0.75) * e1 + T(0.75) * e2 + T(0.5) * e3 - T(1) / 5 * e4;
      const T ux = T(-3.375) * a * e1 - T(27) / 98 * c * e2 - T(2.25) * p * e3 + T(18) / 5 * r * e4;
      const T uy = T(-3.375) * b * e1 - T(27) / 40 * e2 - T(2.25) * q * e3 + T(18) / 5 * t * e4;
      const T lap = (T(15.1875) * s1 - T(60.75)) * e1 + (T(486) / 4802 * (c * c) - (T(243) / 98 - T(243) / 400)) * e2 +
                    (T(10.125) * s3 - T(40.5)) * e3 + (T(324) / 5 - T(324) / 5 * s4) * e4;
      const T av = 1 + T(0.5) * std::sin(2 * T(pi) * px) * std::sin(2 * T(pi) * py);
      const T k = 1 + px * py, mc = 1 + px * px + py * py, bx = py - T(0.5), by = T(0.5) - px;
      const T Ux = ux * k + u * py, Uy = uy * k + u * px, L = lap * k + 2 * (ux * py + uy * px);
      o.u = u; o.ux = ux; o.uy = uy; o.lap = lap; o.a = av; o.s = std::sqrt(2 * av); o.mc = mc; o.Ux = Ux; o.Uy = Uy;
      o.f = -(av * L + bx * Ux + by * Uy - mc * (u * k));
      return o;
    };
    const R E = ref((ld)0), F = ref(0.0);
    FrankeArgs fa;
    FrankeTerms ft;
    franke_args(X, Y, fa);
    franke_terms(tables(), fa, ft);
    i64 ux, uy, gx, gy;
    franke_grad(fa, ft, ux, uy);
    const u64 a62 = aniso_a(tables(), X, Y);
    AnisoOut o;
    aniso_step(tables(), X, Y, a62, o);
    aniso_grad(X, Y, o, gx, gy);
    const ld v[11] = {to_double(franke_lap(tables(), fa), -54), to_double(franke_u(ft), -60), ux * ldexpl(1, -58), uy * ldexpl(1, -58),
                      franke_lap_terms(fa, ft) * ldexpl(1, -54), to_double(a62, 0u, -62), aniso_sigma(a62), to_double(o.f, -51),
                      to_double(o.mc, 0u, -54), gx * ldexpl(1, -54), gy * ldexpl(1, -54)};
    const ld e[11] = {E.lap, E.u, E.ux, E.uy, E.lap, E.a, E.s, E.f, E.mc, E.Ux, E.Uy};
    const ld k[11] = {F.lap, F.u, F.ux, F.uy, F.lap, F.a, F.s, F.f, F.mc, F.Ux, F.Uy};
    for (int j = 0; j < 11; ++j) {
      A[j].add(v[j] - e[j]);
      D[j].add(k[j] - e[j]);
    }
  }
  const char* names[11] = {"lap", "u", "ux", "uy", "lap_terms", "a", "sigma", "f", "mc", "Ux", "Uy"};
  for (int j = 0; j < 11; ++j)
    std::printf("%s %.3Lg %.3Lg\n%s_max %.3Lg %.3Lg\n", names[j], sqrtl(A[j].s2 / np), sqrtl(D[j].s2 / np), names[j], A[j].m, D[j].m);
  return 0;
}
