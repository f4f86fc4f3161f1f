// Error of the normal pair of FP64 stepping (fk_fixed.cuh) against long
// double, by the size of its radius, beside that of the FP64 forms that it
// replaces: first the largest rounding, in units of 2^-55, of the pair as the
// lane groups add it, then one line per power of two of the radius: its exponent, rms and largest error of the fixed-point pair and of
// the FP64 pair.
#include <cmath>
#include <cstdio>
#include <random>

#include "../../spac_gb300/csrc/fk_fixed.cuh"

using namespace fk::fx;
typedef long double ld;

int main() {
  std::mt19937_64 rng(17);
  const ld pi = acosl(-1.0L);
  struct {
    ld s2[2] = {0, 0}, m[2] = {0, 0};
    long n = 0;
  } B[32];
  ld fx = 0;
  for (int i = 0; i < 1200000; ++i) {
    // words of every size, and words that leave a u next to 1 of every distance
    const u32 w = static_cast<u32>(rng()) >> (i % 32), a = i & 32 ? w : ~w, b = static_cast<u32>(rng());
    double z0, z1;
    normal_pair(tables(), a, b, z0, z1);
    const ld u1 = ((ld)a + 0.5L) * ldexpl(1, -32), u2 = ((ld)b + 0.5L) * ldexpl(1, -32);
    const ld r = sqrtl(-2 * log1pl(u1 - 1)), x0 = r * cosl(2 * pi * u2), x1 = r * sinl(2 * pi * u2);
    const double du1 = (a + 0.5) * 2.3283064365386962890625e-10, du2 = (b + 0.5) * 2.3283064365386962890625e-10;
    const double dr = std::sqrt(-2.0 * std::log(du1));
    const double d0 = dr * std::cos(6.283185307179586 * du2), d1 = dr * std::sin(6.283185307179586 * du2);
    u64 m0, m1;
    u32 n0, n1;
    int ez;
    normal_parts(tables(), a, b, m0, m1, n0, n1, ez);
    fx = fmaxl(fx, fabsl(normal_fx<55>(m0, n0, ez) - ldexpl(n0 ? -(ld)m0 : (ld)m0, ez + 55)));
    fx = fmaxl(fx, fabsl(normal_fx<55>(m1, n1, ez) - ldexpl(n1 ? -(ld)m1 : (ld)m1, ez + 55)));
    auto& c = B[16 + (int)floorl(log2l(r))];
    ++c.n;
    const ld e[2] = {fmaxl(fabsl(z0 - x0), fabsl(z1 - x1)), fmaxl(fabsl(d0 - x0), fabsl(d1 - x1))};
    for (int k = 0; k < 2; ++k) {
      c.s2[k] += e[k] * e[k];
      c.m[k] = fmaxl(c.m[k], e[k]);
    }
  }
  std::printf("fx %.4Lg\n", fx);
  for (int j = 0; j < 32; ++j)
    if (B[j].n >= 200)
      std::printf("%d %.4Lg %.4Lg %.4Lg %.4Lg\n", j - 16, sqrtl(B[j].s2[0] / B[j].n), B[j].m[0], sqrtl(B[j].s2[1] / B[j].n), B[j].m[1]);
  return 0;
}
