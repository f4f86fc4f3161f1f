// 64-bit fixed-point building blocks of FP64 stepping.
//
// FP64 arithmetic runs at 1/64 of the FP32 rate on this part (two lanes per
// SM and cycle: one FP64 warp instruction every 16 cycles), so a path step
// written in FP64 is bound by that pipe alone: about 225 such instructions
// per step for the Franke problem, 3,600 cycles, while the other pipes idle.
// The functions here compute the step's transcendental and polynomial parts
// on the integer pipes in 64-bit fixed point.  Fixed point has absolute units,
// so a single small operand may hold fewer digits than a double would; units
// (2^-55 to 2^-80) and the order of products and cuts are chosen so that no
// result is further off than the FP64 form's, wherever in the range: normals
// for every size of the radius, source terms in every 1/8 x 1/8 cell of the
// positions (against long double, tests/cpp/fixed_normals_main.cpp and
// fixed_cells_main.cpp).  A 64 x 64 product's upper half is three
// 32 x 32 -> 64 multiply-adds, about 8 of the 64 issue slots that one FP64
// instruction takes.
//
// The methods are the usual table-driven ones (P. T. P. Tang, ACM TOMS 1989
// and 1990, for exp and log: a table at the leading bits and a short Taylor
// polynomial for the rest), with exact integer argument reduction.  Tables
// are built at compile time by integer arithmetic from a few mathematical
// constants.
//
// Host and device give the same bits (the square root's seed excepted, whose
// error the iteration removes).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define FX_FN __host__ __device__ __forceinline__
#else
#define FX_FN inline
#endif

namespace fk {
namespace fx {

typedef uint64_t u64;
typedef int64_t i64;
typedef uint32_t u32;

// ------------------------------------------------------------ products -----
FX_FN u32 mulhi32(u32 a, u32 b) { return static_cast<u32>((static_cast<u64>(a) * b) >> 32); }
// (a b) >> 64 for a, b < 2^63, low by less than 2 units (the product of the
// low words is dropped).
FX_FN u64 mulhi(u64 a, u64 b) {
  const u32 ah = static_cast<u32>(a >> 32), al = static_cast<u32>(a), bh = static_cast<u32>(b >> 32), bl = static_cast<u32>(b);
  u64 t = static_cast<u64>(ah) * bl;
  t += static_cast<u64>(al) * bh;
  return static_cast<u64>(ah) * bh + (t >> 32);
}
// (a b) >> S, 32 < S < 64, for a < 2^63, b < 2^63 (1 + 2^-19) and a result below 2^64:
// low by less than 2 units, or (R = 1) rounded to nearest.
template <int S, int R = 0>
FX_FN u64 mulshr(u64 a, u64 b) {
  const u32 ah = static_cast<u32>(a >> 32), al = static_cast<u32>(a), bh = static_cast<u32>(b >> 32), bl = static_cast<u32>(b);
  u64 t = static_cast<u64>(ah) * bl + (static_cast<u64>(mulhi32(al, bl)) + (static_cast<u64>(R) << (S - 33)));
  t += static_cast<u64>(al) * bh;
  return ((static_cast<u64>(ah) * bh) << (64 - S)) + (t >> (S - 32));
}
// a^2 >> 63 for a < 2^63.5, rounded to nearest.
FX_FN u64 sqr63(u64 a) {
  const u32 ah = static_cast<u32>(a >> 32), al = static_cast<u32>(a);
  return ((static_cast<u64>(ah) * ah) << 1) + ((static_cast<u64>(ah) * al + ((mulhi32(al, al) >> 1) + (1u << 29))) >> 30);
}
// a^2 >> 64 for a < 2^63, low by less than 2 units.
FX_FN u64 sqrhi(u64 a) {
  const u32 ah = static_cast<u32>(a >> 32), al = static_cast<u32>(a);
  return static_cast<u64>(ah) * ah + ((static_cast<u64>(ah) * al) >> 31);
}
// Sums that may wrap (arguments outside a function's range, whose results are not
// used, and partial sums whose total is in range).
FX_FN i64 addw(i64 a, i64 b) { return static_cast<i64>(static_cast<u64>(a) + static_cast<u64>(b)); }
FX_FN i64 subw(i64 a, i64 b) { return static_cast<i64>(static_cast<u64>(a) - static_cast<u64>(b)); }
// v >> K, rounded to nearest
template <int K>
FX_FN i64 rshr(i64 v) { return K == 0 ? v : addw(v, (1ll << K) >> 1) >> K; }
FX_FN i64 shlw(i64 a, int k) { return static_cast<i64>(static_cast<u64>(a) << k); }
// Signed: (a b) >> 64 and (a b) >> S (32 < S < 64) for |a|, |b| < 2^62, low by less than 2 units
// or (R = 1) rounded to nearest.
FX_FN i64 smulhi(i64 a, i64 b) {
  const int ah = static_cast<int>(a >> 32), bh = static_cast<int>(b >> 32);
  const i64 al = static_cast<i64>(static_cast<u32>(a)), bl = static_cast<i64>(static_cast<u32>(b));
  const i64 t = addw(ah * bl, al * bh);
  return static_cast<i64>(ah) * bh + (t >> 32);
}
template <int S, int R = 0>
FX_FN i64 smulshr(i64 a, i64 b) {
  const int ah = static_cast<int>(a >> 32), bh = static_cast<int>(b >> 32);
  const i64 al = static_cast<i64>(static_cast<u32>(a)), bl = static_cast<i64>(static_cast<u32>(b));
  const i64 t = addw(addw(ah * bl, al * bh), static_cast<i64>(static_cast<u64>(mulhi32(static_cast<u32>(a), static_cast<u32>(b))) +
                                                                     (static_cast<u64>(R) << (S - 33))));
  return addw(shlw(static_cast<i64>(ah) * bh, 64 - S), t >> (S - 32));
}
FX_FN int clz64(u64 v) {
#ifdef __CUDA_ARCH__
  return __clzll(static_cast<long long>(v));
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}

// v >> k and v << k, 0 for k > 63 and for negative k (the PTX shifts clamp, C++ ones do not)
FX_FN u64 shr64(u64 v, int k) {
#ifdef __CUDA_ARCH__
  u64 r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(k));
  return r;
#else
  return static_cast<u32>(k) > 63u ? 0 : v >> k;
#endif
}
FX_FN u64 shl64(u64 v, int k) {
#ifdef __CUDA_ARCH__
  u64 r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(k));
  return r;
#else
  return static_cast<u32>(k) > 63u ? 0 : v << k;
#endif
}

// ------------------------------------------------------------- tables ------
constexpr u64 kLn2_64 = 0xB17217F7D1CF79ACull;  // ln 2 * 2^64
constexpr u64 kLn2_59 = 0x058B90BFBE8E7BCDull;  // ln 2 * 2^59

struct alignas(16) LogEntry {
  u64 ln;   // ln(c / 2^15) * 2^64: 0 in the last interval, next to u = 1
  u64 c;    // reciprocal of the interval's middle, 16 bits
};
struct alignas(16) SinCosEntry {
  u64 c, s;  // cos, sin of the cell's middle * 2^63
};
struct alignas(16) Tables {
  u64 exp2[1024];       // 2^(j/1024) * 2^62
  u64 exp2m1[1024];     // (2^(i / 2^20) - 1) * 2^64
  SinCosEntry sc[1024]; // angle (j + 1/2) / 4096 of a turn
  LogEntry log[512];    // y in [1 + j/512, 1 + (j+1)/512)
};

// exact upper half of a 64 x 64 product (compile time)
constexpr u64 cmulhi(u64 a, u64 b) {
  const u64 ah = a >> 32, al = a & 0xffffffffu, bh = b >> 32, bl = b & 0xffffffffu;
  const u64 m = ah * bl + ((al * bl) >> 32), n = al * bh + (m & 0xffffffffu);
  return ah * bh + (m >> 32) + (n >> 32);
}
constexpr Tables make_tables() {
  Tables t{};
  // 2^(2^-i) * 2^63, i = 1 .. 10
  constexpr u64 root[10] = {0xB504F333F9DE6484ull, 0x9837F0518DB8A96Full, 0x8B95C1E3EA8BD6E7ull, 0x85AAC367CC487B15ull,
                            0x82CD8698AC2BA1D7ull, 0x8164D1F3BC030773ull, 0x80B1ED4FD999AB6Cull, 0x8058D7D2D5E5F6B1ull,
                            0x802C6436D0E04F51ull, 0x8016302F17467628ull};
  for (int j = 0; j < 1024; ++j) {
    u64 v = 1ull << 63;  // Q1.63; each factor below 2 keeps the product below 2
    for (int i = 0; i < 10; ++i)
      if ((j >> (9 - i)) & 1) {
        const u64 p = cmulhi(v, root[i]);  // Q2.62
        v = (p << 1) | 1u;                 // (middle of the dropped bit)
      }
    t.exp2[j] = v >> 1;
    const u64 x = static_cast<u64>(j) * (kLn2_64 >> 20) + ((static_cast<u64>(j) * (kLn2_64 & 0xfffffu)) >> 20);
    const u64 x2 = cmulhi(x, x), x3 = cmulhi(x2, x), x4 = cmulhi(x3, x);
    t.exp2m1[j] = x + x2 / 2 + x3 / 6 + x4 / 24;
  }
  // cos and sin of 2^-i of a turn * 2^64, i = 3 .. 13, then angle (2j + 1) / 8192 from its binary digits
  constexpr u64 cr[11] = {0xB504F333F9DE6484ull, 0xEC835E79946A3145ull, 0xFB14BE7FBAE58156ull, 0xFEC46D1E89292CF0ull,
                            0xFFB10F1BCB6BEF1Dull, 0xFFEC4304266865D9ull, 0xFFFB10B4DC96DABCull, 0xFFFEC42C7454926Bull,
                            0xFFFFB10B10E80E95ull, 0xFFFFEC42C3773236ull, 0xFFFFFB10B0D19F76ull};
  constexpr u64 sr[11] = {0xB504F333F9DE6484ull, 0x61F78A9ABAA58B47ull, 0x31F17078D34C156Dull, 0x1917A6BC29B42BE2ull,
                            0x0C8FB2F886EC09F3ull, 0x0648557DE8D99F7Eull, 0x03243A3F9BD8F08Dull, 0x01921F0FE6700712ull,
                            0x00C90FC5F66525D2ull, 0x006487EABB991CB6ull, 0x003243F655D966C1ull};
  for (int j = 0; j < 1024; ++j) {
    const int a = 2 * j + 1;  // of 8192ths of a turn, below 2048
    u64 c = 0, s = 0;
    bool one = true;  // (cos 0 = 1 does not fit 64 fractional bits)
    for (int i = 0; i < 11; ++i)
      if ((a >> (10 - i)) & 1) {
        if (one) {
          c = cr[i];
          s = sr[i];
          one = false;
        } else {
          const u64 cn = cmulhi(c, cr[i]) - cmulhi(s, sr[i]);
          s = cmulhi(s, cr[i]) + cmulhi(c, sr[i]);
          c = cn;
        }
      }
    t.sc[j].c = c >> 1;
    t.sc[j].s = s >> 1;
  }
  for (int j = 0; j < 512; ++j) {
    const u64 d = 1025 + 2 * static_cast<u64>(j);  // middle of the interval: d / 1024
    u64 c = ((1ull << 27) / d + 1) >> 1;           // 2^16 / (d / 1024), rounded
    if (j == 511) c = 1ull << 15;                  // exactly 1/2: -ln u is exact near u = 1
    // ln(c / 2^15) = 2 atanh((c - 2^15) / (c + 2^15)), the series in 2^-65: at most 1/3, and few terms where it is small
    const u64 num = c - 32768, den = c + 32768;
    u64 x = 0, r = num;
    for (int b = 0; b < 65; ++b) {
      r <<= 1;
      x <<= 1;
      if (r >= den) {
        r -= den;
        x |= 1;
      }
    }
    const u64 x2 = cmulhi(x, x) >> 2;
    u64 p = x, sum = 0;
    for (int k = 1; k < 60 && p; k += 2) {
      sum += p / k;
      p = cmulhi(p, x2);
    }
    t.log[j].ln = sum;  // 2 sum 2^-65
    t.log[j].c = c;
  }
  return t;
}
// The tables in global memory (device) or static storage (host).  The path
// kernel's warp mode copies them to shared memory: a gather of 32 lanes over
// 64 cache lines costs a warp that runs alone about 130 cycles there, and ten
// of them made up 40 % of its step.
#ifdef __CUDACC__
static __device__ const Tables kTablesDev = make_tables();
#endif
#ifndef __CUDA_ARCH__
static constexpr Tables kTablesHost = make_tables();
#endif
FX_FN const Tables* tables() {
#ifdef __CUDA_ARCH__
  return &kTablesDev;
#else
  return &kTablesHost;
#endif
}

// ------------------------------------------------- conversions -------------
FX_FN u64 bits_of(double v) {
#ifdef __CUDA_ARCH__
  return static_cast<u64>(__double_as_longlong(v));
#else
  u64 u;
  std::memcpy(&u, &v, 8);
  return u;
#endif
}
FX_FN double from_bits(u64 u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(static_cast<long long>(u));
#else
  double v;
  std::memcpy(&v, &u, 8);
  return v;
#endif
}
// mag 2^e2 with the given sign (0 or 1), rounded to nearest, on the integer
// pipes; mag = 0 gives 2^(e2 - 1).
FX_FN double to_double(u64 mag, u32 sign, int e2) {
  const int n = clz64(mag | 1);
  const u64 m = mag << n;
  const u64 b = (static_cast<u64>(1085 - n + e2) << 52) + (m >> 11) + ((m >> 10) & 1);
  return from_bits(b | (static_cast<u64>(sign) << 63));
}
FX_FN double to_double(i64 v, int e2) {
  const i64 s = v >> 63;
  return to_double(static_cast<u64>(subw(v ^ s, s)), static_cast<u32>(s) & 1u, e2);
}

// -------------------------------------------------------------- exp --------
// 2^(N / 2^20) e^z for the low 20 bits of N and z 2^64 < 2^45, times 2^62;
// relative error below 2^-59.  Two tables of ten bits each, so that e^z needs
// two terms.
FX_FN u64 exp_frac(const Tables* tb, u32 N, u64 z) {
  const u32 j = (N >> 10) & 1023u, i = N & 1023u;
  const u64 T = tb->exp2[j], S = tb->exp2m1[i];
  const u32 zh = static_cast<u32>(z >> 13);       // z 2^51
  const u64 w = z + (mulhi32(zh, zh) >> 7);       // e^z - 1 = z + z^2 / 2
  return T + mulhi(T, S + w + ((static_cast<u64>(static_cast<u32>(S >> 22)) * static_cast<u32>(w >> 13)) >> 29));
}
// e^-v for v = V 2^-U >= 0 (V < 2^63, U = 55 or 57): the value is M 2^-62 2^-q, M in [2^62, 2^63 (1 + 2^-19)).
// n ln 2 / 2^20 lies above v by less than two of its steps; the rest z > 0.
template <int U>
FX_FN u64 exp_neg(const Tables* tb, u64 V, int& q) {
  const u32 n = mulhi32(static_cast<u32>(V >> 32), U == 57 ? 0x0B8AA3B2u : 0x2E2A8ECAu) + 2u;  // log2(e) 2^(84 - U)
  const u64 z = ((static_cast<u64>(n) * static_cast<u32>(kLn2_64 >> 32)) << 12) +
                ((static_cast<u64>(n) * static_cast<u32>(kLn2_64)) >> 20) - (V << (64 - U));
  q = static_cast<int>((n + 0xfffffu) >> 20);
  return exp_frac(tb, 0u - n, z);
}
// e^v for |v| < 256, relative error below 1.3 2^-53: the result's rounding, and
// the exponent's 2^-55.
FX_FN double exp_core(const Tables* tb, double v) {
  const u64 b = bits_of(v);
  const int e = static_cast<int>(b >> 52) & 0x7ff;
  const u64 m = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10;  // |v| = m 2^(e - 1085), m < 2^63
  const int s = 1030 - e;                                                 // >= 0 for |v| < 256: |v| 2^55 = m >> s
  const u64 V = s < 63 ? m >> s : 0;
  const bool neg = (b >> 63) != 0;
  const u32 n = mulhi32(static_cast<u32>(V >> 32), 0x2E2A8ECAu) + (neg ? 2u : 0u);
  const u64 nl = ((static_cast<u64>(n) * static_cast<u32>(kLn2_64 >> 32)) << 12) +
                 ((static_cast<u64>(n) * static_cast<u32>(kLn2_64)) >> 20);
  const u64 d = nl - (V << 9);
  const u32 N = neg ? 0u - n : n;
  u64 M = exp_frac(tb, N, neg ? d : 0ull - d);
  const int up = static_cast<int>(M >> 63);  // (z may carry the value over the next power of two)
  M >>= up;
  const int k = (static_cast<int>(N) >> 20) + up;
  return from_bits((static_cast<u64>(1022 + k) << 52) + (M >> 10) + ((M >> 9) & 1));
}

// --------------------------------------------------------- square root -----
// sqrt(A 2^e) for A in [2^62, 2^64) and even e: root 2^61 sqrt(A 2^-64) (in
// [2^60, 2^61]), the value being root 2^((e + 64) / 2 - 61); relative error
// below 2^-57.  Seed y ~ (A 2^-64)^-1/2 of 22 bits, h = 1 - a y^2 exactly,
// sqrt(a) = a y (1 + h/2 + 3 h^2 / 8 + O(2^-63)).
FX_FN u64 sqrt_core(u64 A) {
  const float af = static_cast<float>(static_cast<u32>(A >> 40)) * 5.9604644775390625e-8f;
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(af));
#else
  float y = 1.0f / std::sqrt(af);
#endif
  y = y < 1.99999988f ? y : 1.99999988f;
  y = y > 1.0f ? y : 1.0f;
#ifdef __CUDA_ARCH__
  const u32 yb = static_cast<u32>(__float_as_uint(y));
#else
  u32 yb;
  std::memcpy(&yb, &y, 4);
#endif
  const u32 Y = (yb & 0x7fffffu) | 0x800000u;  // y 2^23
  const u64 A1 = A >> 1;                       // a 2^63
  const i64 h = static_cast<i64>((1ull << 60) - mulhi(A1, (static_cast<u64>(Y) * Y) << 15));  // (1 - a y^2) 2^60
  const u64 g = mulhi(A1, static_cast<u64>(Y) << 39);                                         // a y 2^61
  const int hh = static_cast<int>(h >> 9);
  const i64 corr = (h >> 1) + 3 * static_cast<i64>((static_cast<u64>(static_cast<i64>(hh) * hh)) >> 45);  // (h/2 + 3h^2/8) 2^60
  const i64 sg = corr >> 63;
  const u64 d = mulshr<60>(g, static_cast<u64>((corr ^ sg) - sg));
  return g + static_cast<u64>((static_cast<i64>(d) ^ sg) - sg);
}
// sqrt(L 2^e) for L > 0: a root in [2^60, 2^61] and its exponent.
FX_FN u64 sqrt_norm(u64 L, int e, int& e_out) {
  const int n = clz64(L);
  u64 A = L << n;
  e -= n;
  if (e & 1) {
    A >>= 1;
    e += 1;
  }
  e_out = ((e + 64) >> 1) - 61;
  return sqrt_core(A);
}

// -------------------------------------------------- normal pair -------------
// l = -ln((a + 1/2) 2^-32) as l 2^59 (e = -58), for u >= 1/2 as l 2^64 (e = -63), in the
// last table cell before u = 1 as l 2^72 (e = -71) and for l < 2^-17 as l 2^80 (e = -79):
// the error of a radius sqrt(2 l) is that of l over it, and with one unit for
// all l a radius of 2^-5 has two, one of 2^-11 nine times the error that an FP64
// logarithm leaves it.
// Exact argument reduction: u = y 2^(30-n), y c - 1 an integer multiple of 2^-48.
FX_FN u64 neg_log(const Tables* tb, u32 a, int& e) {
  const u64 m = (static_cast<u64>(a) << 1) | 1u;
  const int n = clz64(m);
  const u64 Y = m << n;  // y 2^63, y in [1, 2)
  const u32 j = static_cast<u32>(Y >> 54) & 511u;
  const LogEntry t = tb->log[j];
  const u64 ln = t.ln, c = t.c;
  const i64 r = static_cast<i64>((Y >> 31) * c - (1ull << 48));  // (y c - 1) 2^48, |r| < 2^38.1
  const i64 sg = r >> 63;
  const u64 A = static_cast<u64>((r ^ sg) - sg) << 24;  // |r| 2^72
  const u64 r2 = sqrhi(A);                              // r^2 2^80 (exact in the last cell)
  const u32 rh = static_cast<u32>(A >> 32), q = static_cast<u32>(r2 >> 29);  // |r| 2^40, r^2 2^51
  const u32 r4 = mulhi32(q, q);                                              // r^4 2^70
  const u64 odd = ((static_cast<u64>(mulhi32(q, 0x55555555u)) * rh) >> 11) +
                  (static_cast<u64>(mulhi32(mulhi32(r4, rh), 0x33333334u)) << 2);    // |r|^3/3 + |r|^5/5, 2^-80
  const u64 even = (r2 >> 1) + (static_cast<u64>(r4) << 8);                          // r^2/2 + r^4/4
  const i64 h = ((static_cast<i64>(odd) ^ sg) - sg) - static_cast<i64>(even);        // log1p(r) - r, 2^-80
  const i64 l1p = ((static_cast<i64>(A) ^ sg) - sg) + (h >> 8);                      // log1p(r), 2^-72
  const bool half = n == 31, last = half && ln == 0, tiny = last && A < (1ull << 55);  // (there r < 0)
  e = tiny ? -79 : (last ? -71 : (half ? -63 : -58));
  const u64 base = half ? ln : static_cast<u64>(n - 31) * kLn2_59 + (ln >> 5);
  const u64 l = base - static_cast<u64>(l1p >> (last ? 0 : (half ? 8 : 13)));
  return tiny ? (A << 8) - static_cast<u64>(h) : l;
}

// cos and sin of the angle b + 1/2 (of 2^32) within its quadrant, times 2^63;
// absolute error below 2^-58 (the dropped theta^5 / 120 term is 2^-58.6).
FX_FN void sincos_quadrant(const Tables* tb, u32 b, u64& cs, u64& sn) {
  const u32 j = (b >> 20) & 1023u;
  const SinCosEntry t = tb->sc[j];
  const u64 C = t.c, S = t.s;
  // theta = 2 pi D 2^-33 from the cell's middle, |D| < 2^20, odd
  const int D = static_cast<int>(2u * (b & 0xfffffu) + 1u) - (1 << 20);
  const int sg = D >> 31;
  const u32 Da = static_cast<u32>((D ^ sg) - sg);
  const u64 hq = mulhi(static_cast<u64>(Da) * Da << 23, 0x4EF4F326F9177969ull);  // theta^2 / 2 * 2^83
  const u32 q = static_cast<u32>(hq >> 30);                                      // theta^2 / 2 * 2^53
  const u64 th = mulhi(static_cast<u64>(Da) << 43, 0x6487ED5110B4611Aull);       // theta 2^72 (2 pi 2^60)
  const u64 c1 = (hq >> 20) - (mulhi32(mulhi32(q, q), 0x2AAAAAABu) >> 11);       // (1 - cos theta) 2^63
  const u64 s1 = (th >> 9) - mulhi32(static_cast<u32>(th >> 30), mulhi32(q, 0x55555556u));  // sin |theta| 2^63
  const u64 cc = mulhi(C, c1 << 1), ss = mulhi(S, s1 << 1), sc = mulhi(S, c1 << 1), csn = mulhi(C, s1 << 1);
  const u64 m = static_cast<u64>(static_cast<i64>(sg));
  cs = C - cc - ((ss ^ m) - m);
  sn = S - sc + ((csn ^ m) - m);
}

// Box-Muller pair sqrt(-2 ln u1) (cos, sin)(2 pi u2), u = (word + 1/2) 2^-32:
// magnitudes m0, m1 times 2^e and signs; absolute error below 2^-56 for |z| of order 1.
FX_FN void normal_parts(const Tables* tb, u32 a, u32 b, u64& m0, u64& m1, u32& n0, u32& n1, int& e) {
  int el;
  const u64 l = neg_log(tb, a, el);
  const u64 rad = sqrt_norm(l, el, e);  // sqrt(2 l) = rad 2^e, rad in [2^60, 2^61]
  u64 c, s;
  sincos_quadrant(tb, b, c, s);
  const u32 quad = b >> 30;
  m0 = mulhi(rad, (quad & 1u) ? s : c);
  m1 = mulhi(rad, (quad & 1u) ? c : s);
  n0 = (quad ^ (quad >> 1)) & 1u;
  n1 = quad >> 1;
  e += 1;
}
FX_FN void normal_pair(const Tables* tb, u32 a, u32 b, double& z0, double& z1) {
  u64 m0, m1;
  u32 n0, n1;
  int e;
  normal_parts(tb, a, b, m0, m1, n0, n1, e);
  z0 = to_double(m0, n0, e);
  z1 = to_double(m1, n1, e);
}
// One of the pair's parts in 2^-U units, rounded to nearest (|z| < 6.8, so e <= -57; U <= 55).
template <int U>
FX_FN i64 normal_fx(u64 m, u32 n, int e) {
  const int s = -U - e < 63 ? -U - e : 63;
  const i64 k = -static_cast<i64>(n);
  return (static_cast<i64>((m + (1ull << (s - 1))) >> s) ^ k) - k;
}
template <int U = 53>
FX_FN void normal_pair_fx(const Tables* tb, u32 a, u32 b, i64& z0, i64& z1) {
  u64 m0, m1;
  u32 n0, n1;
  int e;
  normal_parts(tb, a, b, m0, m1, n0, n1, e);
  z0 = normal_fx<U>(m0, n0, e);
  z1 = normal_fx<U>(m1, n1, e);
}

// ------------------------------------------------------ Franke function ----
// Positions are 2^-59 units, in [-3/8, 11/8)^2, which holds the unit square and
// the serial driver's domain: there the sums of squares stay below 256.
// Elsewhere the FP64 forms run.
// A sum in fixed point has one absolute error, so it is as exact as the FP64
// form only if its unit lies below what the smallest sum of the range leaves
// there, and the factors of an exponential's polynomial (up to 256 of a square,
// 324 of the Laplacian's e4) must not meet an exponential that was cut to a
// unit before.  So the products are formed with the exponential's 62 digits,
// and cut after; results are 2^-56 (Laplacian), 2^-60 (gradient), 2^-62 (value)
// and 2^-55 units (source of the anisotropic problem).  Worst error of any 1/8
// x 1/8 cell of the range, in parts of the FP64 form's there (rms): value 0.56,
// gradient 0.55, Laplacian 0.59, source 0.57 (fixed_cells_main.cpp).
FX_FN bool to_pos(double v, i64& p) {
  const u64 b = bits_of(v);
  const int e = static_cast<int>(b >> 52) & 0x7ff;
  const u64 m = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10;  // |v| = m 2^(e - 1085)
  int s = 1026 - e;
  const bool small = s >= 3;  // |v| < 2
  s = small ? (s < 63 ? s : 63) : 3;
  const i64 sg = static_cast<i64>(b) >> 63;
  p = subw(static_cast<i64>(m >> s) ^ sg, sg);
  // -3/8 <= p 2^-59 < 11/8
  return small && static_cast<u32>(p >> 32) + 0x03000000u < 0x0E000000u;
}
constexpr u64 kOne55 = 1ull << 55;
// Squares of the four exponents, 2^-55 units.  One square per coordinate:
// (9x - k)^2 = (9x)^2 - 2k (9x) + k^2.
struct FrankeArgs {
  i64 X9, Y9;       // 9x, 9y (2^-59)
  u64 Gx, Gy;       // (9x)^2, (9y)^2
  u64 s1, s3, s4;   // a^2 + b^2, p^2 + q^2, r^2 + t^2 (one unit below zero at the least)
  u64 c2;           // (9x + 1)^2
  u64 v2;           // (9x + 1)^2 / 49 + (9y + 5) / 10 (2^-57): e2 = e^(4/10 - v2)
};
FX_FN u64 abs64(i64 v) {
  const i64 s = v >> 63;
  return static_cast<u64>(subw(v ^ s, s));
}
// (Unsigned sums: Gx + Gy passes 2^63 near the range's upper corner, and 9x does
// for the positions outside it, whose results are overwritten.)
FX_FN void franke_args(i64 X, i64 Y, FrankeArgs& f) {
  f.X9 = static_cast<i64>(9 * static_cast<u64>(X));
  f.Y9 = static_cast<i64>(9 * static_cast<u64>(Y));
  f.Gx = sqr63(abs64(f.X9));
  f.Gy = sqr63(abs64(f.Y9));
  const u64 S = f.Gx + f.Gy;
  const u64 x9 = static_cast<u64>(f.X9), y9 = static_cast<u64>(f.Y9);
  const u64 xq = static_cast<u64>(f.X9 >> 2), xe = static_cast<u64>(f.X9 >> 3);
  const u64 yq = static_cast<u64>(f.Y9 >> 2), ye = static_cast<u64>(f.Y9 >> 3);
  f.s1 = S - xq - yq + 8 * kOne55;
  f.s3 = S - (x9 - xe) - (yq + ye) + 58 * kOne55;
  f.s4 = S - static_cast<u64>(f.X9 >> 1) - (y9 - ye) + 65 * kOne55;
  f.c2 = f.Gx + xe + kOne55;
  f.v2 = mulhi(f.c2, 0x14E5E0A72F053978ull) + mulhi(static_cast<u64>(f.Y9 >> 1) + (5ull << 58), 0x0CCCCCCCCCCCCCCDull) + 1;
}
// d M 2^-(S + k): an exponential's polynomial d times the exponential M 2^-k, with
// the digits of M.  (Large d come with large k: where the product for S = 60 wraps,
// at d of 64, k is past 63.)
template <int S>
FX_FN i64 times_exp(i64 d, u64 M, int k) {
  const i64 sg = d >> 63;
  const u64 t = S == 64 ? mulhi(abs64(d), M) : mulshr<S < 64 ? S : 63>(abs64(d), M);
  const u64 r = shl64(shr64(t, k > 0 ? k : 0), k < 0 ? -k : 0);
  return subw(static_cast<i64>(r) ^ sg, sg);
}
// Laplacian of the Franke function, 2^-U units; each coefficient c is folded
// into its exponential's exponent as m ln 2 - ln c >= 0, the power of two into its scale:
// lap = 243/16 (s1 - 4) e1 + 81/8 (s3 - 4) e3 - 324/5 (s4 - 1) e4 + 486/4802 (c2 - 18.4975) e2
template <int U = 54>
FX_FN i64 franke_lap(const Tables* tb, const FrankeArgs& f) {
  int q1, q2, q3, q4;
  const u64 M1 = exp_neg<57>(tb, f.s1 + 0x001AAEF2D0FB10FCull, q1), M3 = exp_neg<57>(tb, f.s3 + 0x00EA481236F7D35Cull, q3);
  const u64 M4 = exp_neg<55>(tb, f.s4 + 0x005721FC55588EF9ull, q4), M2 = exp_neg<57>(tb, f.v2 + 0x0102319DC0F73A58ull, q2);
  i64 l = addw(times_exp<64>(static_cast<i64>(f.s1 - 4 * kOne55), M1, q1 - 7),
               times_exp<64>(static_cast<i64>(f.s3 - 4 * kOne55), M3, q3 - 7));
  l = subw(l, times_exp<60>(static_cast<i64>(f.s4 - kOne55), M4, q4 - 6));
  const i64 d2 = static_cast<i64>(f.c2 - 0x093FAE147AE147AEull), sg = d2 >> 63;
  const i64 t2 = static_cast<i64>(mulshr<63, 1>(abs64(d2), shr64(M2, q2)));
  return rshr<56 - U>(addw(l, subw(t2 ^ sg, sg)));
}
// b1 = 3/4 e1, b2 = 3/4 e2, b3 = e3 / 2, b4 = e4 / 5 in 2^-63, 2^-62, 2^-64 and 2^-65 units
// (u = b1 + b2 + b3 - b4), and the Laplacian's parts
// p = (s1 - 4) b1 + (s3 - 4) b3 (2^-61), p4 = (s4 - 1) b4 (2^-64).
struct FrankeTerms {
  u64 b1, b2, b3, b4;
  i64 p, p4;
};
FX_FN void franke_terms(const Tables* tb, const FrankeArgs& f, FrankeTerms& b) {
  int q1, q2, q3, q4;
  const u64 M1 = exp_neg<57>(tb, f.s1 + 0x00934B1089A6DC94ull, q1), M3 = exp_neg<57>(tb, f.s3 + 0x0162E42FEFA39EF3ull, q3);
  const u64 M4 = exp_neg<55>(tb, f.s4 + 0x00CE020FBF6C699Bull, q4), M2 = exp_neg<57>(tb, f.v2 + 0x01296273AC7DAEBAull, q2);
  b.b1 = shr64(M1, q1 - 1) + (shr64(M1, q1 - 2) & 1u);  // (rounded: its last digit counts 54 times in a gradient)
  b.b2 = shr64(M2, q2 - 1);
  b.b3 = shr64(M3, q3 - 2);
  b.b4 = shr64(M4, q4 - 3);
  b.p = addw(times_exp<64>(static_cast<i64>(f.s1 - 4 * kOne55), M1, q1 - 8),
             times_exp<64>(static_cast<i64>(f.s3 - 4 * kOne55), M3, q3 - 8));
  b.p4 = times_exp<60>(static_cast<i64>(f.s4 - kOne55), M4, q4 - 7);
}
// u, 2^-U units
template <int U = 60>
FX_FN i64 franke_u(const FrankeTerms& b) {
  return rshr<62 - U>(static_cast<i64>((b.b1 >> 1) + b.b2 + (b.b3 >> 2) - (b.b4 >> 3)));
}
// u_x and u_y, 2^-U units (g = 18/49):
// u_x = 9x (18 b4 - 9/2 (b1 + b3) - g b2) + 9 b1 - g b2 + 63/2 b3 - 72 b4
// u_y = 9y (18 b4 - 9/2 (b1 + b3)) + 9 b1 - 9/10 b2 + 27/2 b3 - 126 b4
// (sums in 2^-61, whose parts may wrap; below 4 in the end, 3.3 at the most)
template <int U = 58>
FX_FN void franke_grad(const FrankeArgs& f, const FrankeTerms& b, i64& ux, i64& uy) {
  const u64 gb = mulhi(b.b2, 0x5E0A72F05397829Dull);             // g b2, 2^-62
  const u64 nb = mulhi(b.b2, 0x7333333333333333ull) + 1;         // 9/10 b2, 2^-61
  // the brackets over 9/2, 2^-63, and 81/2 x, 81/2 y, 2^-55
  const i64 dy = static_cast<i64>(b.b4 - (b.b1 + ((b.b3 + 1) >> 1)));
  const i64 dx = subw(dy, static_cast<i64>(mulshr<63, 1>(b.b2, 0x14E5E0A72F053978ull)));
  const i64 ax = static_cast<i64>(9 * static_cast<u64>(f.X9 >> 3)) >> 2, ay = static_cast<i64>(9 * static_cast<u64>(f.Y9 >> 3)) >> 2;
  const u64 v = 2 * b.b1 + (b.b1 >> 2);
  const u64 vx = v - (gb >> 1) + 4 * b.b3 - (b.b3 >> 4) - 4 * b.b4 - (b.b4 >> 1);
  const u64 vy = v - nb + 2 * b.b3 - (b.b3 >> 2) - (b.b3 >> 4) - 8 * b.b4 + (b.b4 >> 3);
  ux = rshr<61 - U>(addw(smulshr<57, 1>(ax, dx), static_cast<i64>(vx)));
  uy = rshr<61 - U>(addw(smulshr<57, 1>(ay, dy), static_cast<i64>(vy)));
}
// Laplacian from the same terms, 2^-U units:
// 81/4 p - 324 p4 + (g^2 c2 - 9 g + 81/100) b2, 81/128 and 81/64 as sums of three halvings
template <int U = 54>
FX_FN i64 franke_lap_terms(const FrankeArgs& f, const FrankeTerms& b) {
  const i64 l = rshr<1>(addw(b.p, addw(b.p >> 2, b.p >> 6))), l4 = addw(b.p4, addw(b.p4 >> 2, b.p4 >> 6));  // 2^-56
  const i64 k = static_cast<i64>(mulshr<63>(f.c2, 0x451759AB57896FA2ull) - 0x04FE03C2FA5B8877ull);      // 2^-57
  return rshr<56 - U>(addw(subw(l, l4), smulshr<63, 1>(k, static_cast<i64>(b.b2))));
}

// -------------------------------------- the anisotropic problem's factors ----
// sin(2 pi x), 2^-63 units and its sign; x in 2^-59 units of a turn.
FX_FN u64 sin_turn(const Tables* tb, i64 X, u32& neg) {
  const u32 quad = static_cast<u32>(X >> 57) & 3u, j = static_cast<u32>(X >> 47) & 1023u;
  const SinCosEntry t = tb->sc[j];
  const u64 C = t.c, S = t.s;
  const i64 D = (X & ((1ll << 47) - 1)) - (1ll << 46);  // theta = 2 pi D 2^-59 from the cell's middle
  const i64 sg = D >> 63;
  const u64 th = mulhi(static_cast<u64>((D ^ sg) - sg) << 17, 0x6487ED5110B4611Aull);  // theta 2^72
  const u64 hq = sqrhi(th) << 2;                                                       // theta^2 / 2 * 2^83
  const u32 q = static_cast<u32>(hq >> 30);
  const u64 c1 = (hq >> 20) - (mulhi32(mulhi32(q, q), 0x2AAAAAABu) >> 11);
  const u64 s1 = (th >> 9) - mulhi32(static_cast<u32>(th >> 30), mulhi32(q, 0x55555556u));
  const u64 P = (quad & 1u) ? C : S, Q = (quad & 1u) ? S : C;
  const u64 m = static_cast<u64>((quad & 1u) ? ~sg : sg);
  neg = quad >> 1;
  return P - mulhi(P, c1 << 1) + ((mulhi(Q, s1 << 1) ^ m) - m);
}
// a = 1 + sin(2 pi x) sin(2 pi y) / 2, 2^-62 units
FX_FN u64 aniso_a(const Tables* tb, i64 X, i64 Y) {
  u32 nx, ny;
  const u64 sx = sin_turn(tb, X, nx), sy = sin_turn(tb, Y, ny);
  const u64 p = mulhi(sx, sy) >> 1;
  const u64 m = 0ull - static_cast<u64>(nx ^ ny);
  return (1ull << 62) + ((p ^ m) - m);
}
// v 2^62 of a double v in [2^-10, 2)
FX_FN u64 a_bits(double v) {
  const u64 b = bits_of(v);
  return ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10 >> ((1023 - static_cast<int>(b >> 52)) & 63);
}
FX_FN double aniso_sigma(u64 a62) {  // sqrt(2 a)
  int e;
  const u64 r = sqrt_norm(a62, -61, e);
  return to_double(r, 0u, e);
}
// The anisotropic problem at a point: source f (2^-UF units) of
// u = F q, q = 1 + xy, F the Franke function:
//   f = -(q (a lap F + b . grad F + c F) + 2 a (F_x y + F_y x) + F (y^2 - x^2 + (x - y) / 2)),
// b = (y - 1/2, 1/2 - x), c = -(1 + x^2 + y^2); and -c (2^-UM units).
template <int UF, int UM>
struct AnisoParts {
  i64 f;
  u64 mc;
  i64 F, Fx, Fy, q;  // 2^-61, 2^-60, 2^-60, 2^-60 units
};
typedef AnisoParts<51, 54> AnisoOut;
template <int UF, int UM>
FX_FN void aniso_step(const Tables* tb, i64 X, i64 Y, u64 a62, AnisoParts<UF, UM>& o) {
  FrankeArgs f;
  FrankeTerms b;
  franke_args(X, Y, f);
  franke_terms(tb, f, b);
  o.F = franke_u<61>(b);
  franke_grad<60>(f, b, o.Fx, o.Fy);
  const i64 lap = franke_lap_terms<55>(f, b);
  const i64 X61 = shlw(X, 2), Y61 = shlw(Y, 2), a61 = static_cast<i64>(a62 >> 1);
  o.q = addw(1ll << 60, smulshr<62>(X61, Y61));
  const u64 mc = (1ull << 59) + mulhi((f.Gx + f.Gy) >> 1, 0x6522C3F35BA78195ull);  // 2^-59
  o.mc = mc >> (59 - UM);
  const i64 adv = subw(addw(smulshr<63>(subw(Y61, 1ll << 60), o.Fx), smulshr<63>(subw(1ll << 60, X61), o.Fy)),
                       smulshr<62>(static_cast<i64>(mc), o.F));                // 2^-58
  const i64 inner = addw(smulshr<61, 1>(lap, a61), rshr<3>(adv));              // 2^-55
  const i64 t1 = smulshr<60, 1>(inner, o.q);                                   // 2^-55
  const i64 g = addw(smulshr<63>(o.Fx, Y61), smulshr<63>(o.Fy, X61));          // 2^-58
  const i64 t2 = smulshr<63, 1>(g, a61);                                       // 2 a g, 2^-55
  const i64 h = addw(smulshr<61>(static_cast<i64>(f.Gy - f.Gx) >> 1, 0x1948B0FCD6E9E065ll), subw(X, Y));  // 2^-60
  const i64 t3 = rshr<3>(smulshr<63>(o.F, h));                                 // 2^-55
  o.f = rshr<55 - UF>(subw(0, addw(addw(t1, t2), t3)));
}
// grad u = grad F q + F (y, x), 2^-U units
template <int U = 54, int UF, int UM>
FX_FN void aniso_grad(i64 X, i64 Y, const AnisoParts<UF, UM>& o, i64& ux, i64& uy) {
  ux = rshr<60 - U>(addw(smulshr<60, 1>(o.Fx, o.q), smulshr<62, 1>(o.F, shlw(Y, 2))));
  uy = rshr<60 - U>(addw(smulshr<60, 1>(o.Fy, o.q), smulshr<62, 1>(o.F, shlw(X, 2))));
}

}  // namespace fx
}  // namespace fk
