// acg_fx.cuh -- log-sum-exps of FP64 values in integer arithmetic.
//
// GB300 runs an FP64 instruction at 1/64 of the FP32 rate (2 lanes per clock and
// SM), so a CUDA exp() of a double, about 25 FP64 instructions, costs as much
// issue time as 1,600 integer ones.  Here exp(x) is formed on the integer pipes
// as 2^k f with f in 61 fraction bits, by the table-driven method of P. Tang
// ("Table-driven implementation of the exponential function in IEEE
// floating-point arithmetic", 1989) in fixed point:
//   n = round(64 x / ln 2) = 64 k + j,   r = x - n ln 2 / 64  (60 fraction bits,
//   formed modulo 2^64, exact but for the rounding of the constant at 2^-93),
//   f = 2^(j/64) (1 + r + r^2/2 + ... + r^6/720).
// The relative error of f is below 2.5e-16 (tests/test_fx_lse.py checks it
// against extended precision), about that of a correctly rounded double.
// Sums are kept relative to a power of two 2^K, K the largest k so far, as
// 96-bit fixed point (61 fraction bits): adding is exact but for the truncation
// at 2^-61 of the largest term, and rescaling is a shift.  A sum of 100,000
// values near 8 comes out within 4e-15 (an FP64 running sum: 1e-13).
// FP64 kernels before and after: vertex phase of R-MAT 18 with a 16/32 pattern
// 1,318 -> 357 us an iteration (then acg_vertex_fx.cu), source-side static pass
// 7,070 -> 1,392 us.
//
// The header compiles for the host as well (the tests run it there).
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define ACG_FX_HD __host__ __device__ __forceinline__
#define ACG_FX_SLOW static __host__ __device__ __noinline__
#else
#include <cmath>
#define ACG_FX_HD inline
#define ACG_FX_SLOW inline
#endif

namespace acg {

// round(2^(j / 64) 2^61)
#define ACG_FX_EXP_TABLE { \
    0x2000000000000000ull, 0x2059347cef00c1ddull, 0x20b361a62b0ae876ull, 0x210e8a30eb379012ull, \
    0x216ab0d9f3121ec5ull, 0x21c7d865a7a34404ull, 0x222603a024b6a14aull, 0x2285355d525bbf67ull, \
    0x22e57078faa2f5baull, 0x2346b7d6df96ea79ull, 0x23a90e62d17354f0ull, 0x240c7710c519ac77ull, \
    0x2470f4dceac470ceull, 0x24d68acbc4f9ba4bull, 0x253d3bea3fbdc258ull, 0x25a50b4dc8061680ull, \
    0x260dfc14636e2a5cull, 0x26781164c82dfe99ull, 0x26e34e6e7553954eull, 0x274fb669cb3fedd4ull, \
    0x27bd4c982468446bull, 0x282c1443ee5c53f1ull, 0x289c10c0c3125a06ull, 0x290d456b8279a028ull, \
    0x297fb5aa6c544e3bull, 0x29f364ed3a594d5aull, 0x2a6856ad3a9f03beull, 0x2ade8e6d6a4fb4ceull, \
    0x2b560fba90a852b2ull, 0x2bcede2b5a4290ddull, 0x2c48fd6074ab0964ull, 0x2cc47104aa444922ull, \
    0x2d413cccfe779921ull, 0x2dbf6478ca345de4ull, 0x2e3eebd1d8bee7baull, 0x2ebfd6ac84cf917full, \
    0x2f4228e7d6030db0ull, 0x2fc5e66d9e9cc421ull, 0x304b1332999c2516ull, 0x30d1b3368925d902ull, \
    0x3159ca845541b6b7ull, 0x31e35d322aee6c57ull, 0x326e6f619b8bc9e9ull, 0x32fb053fbc9c9f17ull, \
    0x3389230547e12039ull, 0x3418ccf6bbcac965ull, 0x34aa07647c4ab917ull, 0x353cd6aaf3fb7e88ull, \
    0x35d13f32b5a75abdull, 0x366745709e2bf5edull, 0x36feede5f6bc8dd5ull, 0x37983d209783a449ull, \
    0x383337bb0aa53844ull, 0x38cfe25cafa29694ull, 0x396e41b9df20d22aull, 0x3a0e5a940f12f71aull, \
    0x3ab031b9f7490e4cull, 0x3b53cc07b6650ae1ull, 0x3bf92e66f736bd73ull, 0x3ca05dcf167fec4eull, \
    0x3d495f454921b30bull, 0x3df437dcc2b44eeeull, 0x3ea0ecb6dc8a80cfull, 0x3f4f83033d21b05dull}
// round(2^(j / 1024) 2^61), j < 16
#define ACG_FX_EXP16_TABLE { \
    0x2000000000000000ull, 0x20058c0bc5d19d8aull, 0x200b190db43813d4ull, 0x2010a705f5df063bull, \
    0x201635f4b5797dacull, 0x201bc5da1dc1e9ecull, 0x202156b6597a22e1ull, 0x2026e889936b69dbull, \
    0x202c7b53f6666adbull, 0x20320f15ad433de0ull, 0x2037a3cee2e1682cull, 0x203d397fc227dd90ull, \
    0x2042d028760501b5ull, 0x204867c9296ea967ull, 0x204e006207621bdfull, 0x205399f33ae4140bull}

#ifdef __CUDACC__
static __device__ const uint64_t kFxExpDev[64] = ACG_FX_EXP_TABLE;
static __device__ const uint64_t kFxExp16Dev[16] = ACG_FX_EXP16_TABLE;
#endif
static const uint64_t kFxExpHost[64] = ACG_FX_EXP_TABLE;
static const uint64_t kFxExp16Host[16] = ACG_FX_EXP16_TABLE;

ACG_FX_HD uint64_t fx_exp_entry(int j) {
#ifdef __CUDA_ARCH__
  return __ldg(reinterpret_cast<const unsigned long long*>(kFxExpDev) + j);
#else
  return kFxExpHost[j];
#endif
}
ACG_FX_HD uint64_t fx_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
ACG_FX_HD double fx_double(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}
ACG_FX_HD int32_t fx_mulhi(int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
  return __mulhi(a, b);
#else
  return (int32_t)(((int64_t)a * b) >> 32);
#endif
}

// |x| below this (2^14) takes fx_add's integer path; the high word's bits
constexpr uint32_t kFxLimit = 0x40d00000u;

// exp(x) = 2^k f / 2^61 from x with 60 fraction bits modulo 2^64 (X) and
// n = 64 x / ln 2 rounded; f in (0.99, 2.02) 2^61.
ACG_FX_HD uint64_t fx_exp_core(uint64_t X, int n, int& k) {
  // r = x - n ln2 / 64: 92 fraction bits of ln2 / 64
  const int64_t r = (int64_t)(X - (uint64_t)(int64_t)n * 0x2c5c85fdf473deull) -
                    (((int64_t)n * (int64_t)0x6af278edll) >> 32);
  const uint64_t T = fx_exp_entry(n & 63);
  k = n >> 6;
  // |r| < 0.0075.  r^2 from the high 31 bits (rh, 38 fraction bits) and the
  // rest; the tail r^3/6 + ... + r^6/720 in 32 bits (its coefficients with 33
  // fraction bits, the last with 27)
  const int32_t rh = (int32_t)(r >> 22);
  const int32_t rl = (int32_t)((uint32_t)r & 0x3fffffu);
  const int64_t s1 = (int64_t)rh * rh;
  const int64_t r2 = (s1 >> 16) + (((int64_t)rh * rl) >> 37);
  int32_t u = 71582788 + fx_mulhi(rh, 186414);
  u = 357913941 + (fx_mulhi(rh, u) >> 6);
  u = 1431655765 + (fx_mulhi(rh, u) >> 6);
  const int32_t s = fx_mulhi(rh, u);  // 39 fraction bits
  const int64_t p = r + (r2 >> 1) + (((int64_t)(int32_t)(s1 >> 32) * s) >> 23);
  // T (1 + p)
  const int32_t ph = (int32_t)(p >> 32);
  const uint32_t pl = (uint32_t)p;
  const uint32_t Th = (uint32_t)(T >> 32), Tl = (uint32_t)T;
  const int64_t a = (int64_t)(int32_t)Th * ph;
  const int64_t b = (int64_t)((uint64_t)Th * pl) + (int64_t)Tl * ph;
  return T + ((uint64_t)a << 4) + (uint64_t)(b >> 28);
}

// exp(x) for a double, |x| < 2^14.
ACG_FX_HD uint64_t fx_exp(uint64_t bits, int& k) {
  const uint32_t hi = (uint32_t)(bits >> 32), lo = (uint32_t)bits;
  const uint32_t t = hi & 0x7fffffffu;
  // x as a float, truncated (exponent rebased from 1023 to 127; 0 below 2^-15,
  // where n is 0 whatever the value)
  uint32_t fb = ((hi << 3) | (lo >> 29)) - 0xc0000000u;
  fb = t < 0x3f000000u ? 0u : (fb | (hi & 0x80000000u));
  float xf;
  int n;
#ifdef __CUDA_ARCH__
  xf = __uint_as_float(fb);
  n = __float_as_int(__fmaf_rn(xf, 92.33248262f, 12582912.f)) - 0x4b400000;
#else
  std::memcpy(&xf, &fb, 4);
  n = (int)std::lrintf(xf * 92.33248262f);
#endif
  // x with 60 fraction bits, modulo 2^64
  const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
  const int c = (int)(t >> 20) - 1015;
  uint64_t X = c >= 0 ? m << c : (c > -53 ? m >> -c : 0ull);
  if ((int32_t)hi < 0) X = 0ull - X;
  return fx_exp_core(X, n, k);
}

// The same from a table of 2^(j / 1024), which leaves a shorter series
// (|r| < 4e-4: r + r^2 (1/2 + r/6 + r^2/24)) and half the instructions; kernels
// build it in shared memory (8 KB) with fx_table_entry.
constexpr int kFxTable = 1024;
ACG_FX_HD uint64_t fx_table_entry(int j) {
#ifdef __CUDA_ARCH__
  const uint64_t a = kFxExpDev[j >> 4], b = kFxExp16Dev[j & 15];
  const uint64_t hi = __umul64hi(a, b), lo = a * b;
#else
  const uint64_t a = kFxExpHost[j >> 4], b = kFxExp16Host[j & 15];
  const unsigned __int128 p = (unsigned __int128)a * b;
  const uint64_t hi = (uint64_t)(p >> 64), lo = (uint64_t)p;
#endif
  return (hi << 3) | (lo >> 61);
}
// n = 1024 x / ln 2 rounded
ACG_FX_HD uint64_t fx_exp_tab(uint64_t X, int n, const uint64_t* tab, int& k) {
  const int64_t r = (int64_t)(X - (uint64_t)(int64_t)n * 0x2c5c85fdf473dull) -
                    (((int64_t)n * (int64_t)0x735793c7ll) >> 31);
  const uint64_t T = tab[n & (kFxTable - 1)];
  k = n >> 10;
  const int32_t rh = (int32_t)(r >> 18);                          // 42 fraction bits
  const int32_t r2 = (int32_t)(((int64_t)rh * rh) >> 31);         // 53
  const int32_t c = 0x40000000 + fx_mulhi(rh, 349525) + fx_mulhi(r2, 43);  // 31
  const int64_t p = r + (((int64_t)r2 * c) >> 24);
  const int32_t ph = (int32_t)(p >> 32);
  const uint32_t pl = (uint32_t)p;
  const uint32_t Th = (uint32_t)(T >> 32), Tl = (uint32_t)T;
  const int64_t a = (int64_t)(int32_t)Th * ph;
  const int64_t b = (int64_t)((uint64_t)Th * pl) + (int64_t)Tl * ph;
  return T + ((uint64_t)a << 4) + (uint64_t)(b >> 28);
}

// exp(x) for x = X / 2^Q, 47 <= Q <= 54 and |x| < 2^14.
// c: 1024 / ln 2 with 64 - Q fraction bits (fx_scaled_factor).
ACG_FX_HD int32_t fx_scaled_factor(int Q) {
  return (int32_t)((6345039891169ull + (1ull << (Q - 33))) >> (Q - 32));  // 2^32 1024 / ln 2
}
ACG_FX_HD uint64_t fx_exp_scaled(int64_t X, int Q, int32_t c, const uint64_t* tab, int& k) {
  const int n = (int)(((int64_t)(int32_t)(X >> 32) * c + 0x80000000ll) >> 32);
  return fx_exp_tab((uint64_t)X << (60 - Q), n, tab, k);
}

// x with Q fraction bits, truncated toward zero, for |x| < 2^(60 - Q); +-2^60
// beyond that.
ACG_FX_HD int64_t fx_from_double(double x, int Q) {
  const uint64_t b = fx_bits(x);
  const uint32_t hi = (uint32_t)(b >> 32);
  const int sh = 1083 - Q - (int)((hi >> 20) & 0x7ffu);
  uint64_t v = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 8;
  v = sh < 0 ? 1ull << 60 : v >> (sh < 63 ? sh : 63);
  return (int32_t)hi < 0 ? -(int64_t)v : (int64_t)v;
}
// v / 2^Q rounded to a double.
ACG_FX_HD double fx_to_double(int64_t v, int Q) {
  const uint64_t sign = (uint64_t)v & 0x8000000000000000ull;
  uint64_t a = (uint64_t)(v < 0 ? -v : v);
  if (a == 0) return 0.0;
#ifdef __CUDA_ARCH__
  const int lz = __clzll((long long)a);
#else
  const int lz = __builtin_clzll(a);
#endif
  a <<= lz;
  // 53 bits, rounded half up; the leading one adds to the exponent field
  const uint64_t m = (a >> 11) + ((a >> 10) & 1u);
  return fx_double(sign | (((uint64_t)(1085 - lz - Q) << 52) + m));
}

// exp(x) as a double (within 4e-16 relative); CUDA's where |x| >= 700.
ACG_FX_HD double fx_expd(double x) {
  const uint64_t b = fx_bits(x);
  if (((uint32_t)(b >> 32) & 0x7fffffffu) >= 0x4085e000u) return exp(x);
  int k;
  uint64_t f = fx_exp(b, k);
#ifdef __CUDA_ARCH__
  const int lz = __clzll((long long)f);
#else
  const int lz = __builtin_clzll(f);
#endif
  f <<= lz;
  return fx_double(((uint64_t)(1024 + k - lz) << 52) + (f >> 11) + ((f >> 10) & 1u));
}

// A log-sum-exp state in four words.  Integer form (bit 31 of w[3] clear):
// w[0] = K, w[1..3] the 96-bit sum of exp(x) 2^(61 - K).  Wide form (bit set),
// entered where the sum is of values beyond +-2^24: w[0..1] the running maximum
// m, w[2..3] minus the sum of exp(x - m), both doubles.  Only fx_add, fx_add_far
// and fx_merge take a wide state; fx_add_term does not.
struct FxLse {
  uint32_t w[4];
};
ACG_FX_HD void fx_init(FxLse& a) {
  a.w[0] = 0xc0000000u;  // K = -2^30, below every k
  a.w[1] = a.w[2] = a.w[3] = 0u;
}
ACG_FX_HD bool fx_wide(const FxLse& a) { return (int32_t)a.w[3] < 0; }

// (m, s): the sum is s exp(m); (-inf, 0) where nothing was added.
ACG_FX_HD void fx_pair(const FxLse& a, double& m, double& s) {
  if (fx_wide(a)) {
    m = fx_double(((uint64_t)a.w[1] << 32) | a.w[0]);
    s = -fx_double(((uint64_t)a.w[3] << 32) | a.w[2]);
    return;
  }
  if ((a.w[1] | a.w[2] | a.w[3]) == 0u) {
    m = fx_double(0xfff0000000000000ull);
    s = 0.0;
    return;
  }
  // m = K ln 2 rounded; what the rounding leaves goes into s
  const double K = (double)(int32_t)a.w[0];
  m = K * 0x1.62e42fefa39efp-1;
#ifdef __CUDA_ARCH__
  const double d = __fma_rn(K, 0x1.62e42fefa39efp-1, -m) + K * 0x1.abc9e3b39803fp-56;
#else
  const double d = std::fma(K, 0x1.62e42fefa39efp-1, -m) + K * 0x1.abc9e3b39803fp-56;
#endif
  s = (double)a.w[3] * 8.0 + (double)(((uint64_t)a.w[2] << 32) | a.w[1]) * 0x1p-61;
  s += s * d;
}

// the sum shifted right by sh >= 0 bits
ACG_FX_HD void fx_shift(FxLse& a, uint32_t sh) {
  uint64_t lo = ((uint64_t)a.w[2] << 32) | a.w[1];
  uint64_t hi = a.w[3];
  if (sh >= 64) {
    lo = 0;  // at most 2^-3 of the largest term's last bit is left
    hi = 0;
  } else if (sh > 0) {
    lo = (lo >> sh) | (hi << (64 - sh));
    hi >>= sh;
  }
  a.w[1] = (uint32_t)lo;
  a.w[2] = (uint32_t)(lo >> 32);
  a.w[3] = (uint32_t)hi;
}

// add 2^k f / 2^61.  A larger term shifts the sum without a branch (some lane of
// a warp has a new largest term at almost every addition), by up to 31 bits;
// the first term and larger jumps take the branch.
ACG_FX_HD void fx_add_term(FxLse& a, int k, uint64_t f) {
  const int d = k - (int)a.w[0];
  if (d > 31) {
    fx_shift(a, (uint32_t)d);
  } else {
    const uint32_t up = d > 0 ? (uint32_t)d : 0u;
#ifdef __CUDA_ARCH__
    a.w[1] = __funnelshift_r(a.w[1], a.w[2], up);
    a.w[2] = __funnelshift_r(a.w[2], a.w[3], up);
    a.w[3] >>= up;
#else
    fx_shift(a, up);
#endif
  }
  a.w[0] = (uint32_t)(d > 0 ? k : (int)a.w[0]);
  const uint32_t dn = d < 0 ? (uint32_t)-d : 0u;
  f >>= dn < 63u ? dn : 63u;  // f < 2^63
#ifdef __CUDA_ARCH__
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, 0;"
      : "+r"(a.w[1]), "+r"(a.w[2]), "+r"(a.w[3]) : "r"((uint32_t)f), "r"((uint32_t)(f >> 32)));
#else
  const uint64_t lo = ((uint64_t)a.w[2] << 32) | a.w[1];
  const uint64_t t = lo + f;
  a.w[3] += t < lo;
  a.w[1] = (uint32_t)t;
  a.w[2] = (uint32_t)(t >> 32);
#endif
}

// x beyond +-2^24, or a wide state that x does not replace.  Values further apart
// than e^100 (nearly all, at this scale) need no exponential.
constexpr double kFxFar = 100.0;
ACG_FX_SLOW FxLse fx_add_wide(FxLse a, double x) {
  if (!(x > fx_double(0xfff0000000000000ull))) return a;  // NaN, -inf: nothing
  double m, s;
  fx_pair(a, m, s);
  const double d = x - m;
  if (s > 0.0 && d < -kFxFar) return a;
  if (!(s > 0.0) || d > kFxFar) {
    m = x;
    s = 1.0;
  } else if (d > 0.0) {
    s = s * exp(-d) + 1.0;
    m = x;
  } else {
    s += exp(d);
  }
  const uint64_t mb = fx_bits(m), sb = fx_bits(-s);
  a.w[0] = (uint32_t)mb;
  a.w[1] = (uint32_t)(mb >> 32);
  a.w[2] = (uint32_t)sb;
  a.w[3] = (uint32_t)(sb >> 32) | 0x80000000u;
  return a;
}

// Value x outside fx_add's range (|x| >= 2^14), or a state already wide.  Up to
// 2^24 the integer form holds it, n rounded from FP64 (the series' argument is
// formed modulo 2^64 as before).  A term more than e^-100 below the sum adds
// nothing, and a wide sum more than that below x is dropped for x: so one vertex
// far from everything leaves the state in integer form, or returns it there with
// the next ordinary value.
ACG_FX_SLOW FxLse fx_add_far(FxLse a, double x) {
  const uint64_t b = fx_bits(x);
  const uint32_t t = (uint32_t)(b >> 32) & 0x7fffffffu;
  if (t < 0x41700000u) {
    if (fx_wide(a) && x - fx_double(((uint64_t)a.w[1] << 32) | a.w[0]) > kFxFar)
      fx_init(a);  // (its scaled sum is below 2^33)
    if (!fx_wide(a)) {
#ifdef __CUDA_ARCH__
      const int n = __double2int_rn(x * 92.332482616893656877);
#else
      const int n = (int)std::lrint(x * 92.332482616893656877);
#endif
      const uint64_t m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
      const int c = (int)(t >> 20) - 1015;
      const uint64_t X = c >= 0 ? m << c : (c > -53 ? m >> -c : 0ull);
      int k;
      const uint64_t f = fx_exp_core((b >> 63) ? 0ull - X : X, n, k);
      fx_add_term(a, k, f);
      return a;
    }
  }
  return fx_add_wide(a, x);
}

ACG_FX_HD void fx_add(FxLse& a, double x) {
  const uint64_t b = fx_bits(x);
  const uint32_t hi = (uint32_t)(b >> 32);
  if ((hi & 0x7fffffffu) < kFxLimit && !fx_wide(a)) {
    int k;
    const uint64_t f = fx_exp(b, k);
    fx_add_term(a, k, f);
  } else if (hi != 0xfff00000u) {  // (-inf adds nothing)
    a = fx_add_far(a, x);
  }
}

// fx_add with a table of 2^(j / 1024) (tab): |x| < 2^9, else fx_add.
ACG_FX_HD void fx_add(FxLse& a, double x, const uint64_t* tab) {
  const uint64_t b = fx_bits(x);
  const uint32_t hi = (uint32_t)(b >> 32), t = hi & 0x7fffffffu;
  if (t < 0x40800000u && !fx_wide(a)) {
    // x as a float, and with 60 fraction bits modulo 2^64 (as fx_exp)
    uint32_t fb = ((hi << 3) | ((uint32_t)b >> 29)) - 0xc0000000u;
    fb = t < 0x3f000000u ? 0u : (fb | (hi & 0x80000000u));
    float xf;
    int n, k;
#ifdef __CUDA_ARCH__
    xf = __uint_as_float(fb);
    n = __float_as_int(__fmaf_rn(xf, 1477.31972f, 12582912.f)) - 0x4b400000;
#else
    std::memcpy(&xf, &fb, 4);
    n = (int)std::lrintf(xf * 1477.31972f);
#endif
    const uint64_t m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const int c = (int)(t >> 20) - 1015;
    uint64_t X = c >= 0 ? m << c : (c > -53 ? m >> -c : 0ull);
    if ((int32_t)hi < 0) X = 0ull - X;
    const uint64_t f = fx_exp_tab(X, n, tab, k);
    fx_add_term(a, k, f);
  } else if (hi != 0xfff00000u) {
    fx_add(a, x);
  }
}

// a += b
ACG_FX_SLOW FxLse fx_merge_wide(FxLse a, FxLse b) {
  double m, s, m2, s2;
  fx_pair(a, m, s);
  fx_pair(b, m2, s2);
  const double d = m2 - m;
  if (s2 == 0.0 || d < -kFxFar) return a;
  if (s == 0.0 || d > kFxFar) return b;
  if (d > 0.0) {
    s = s * exp(-d) + s2;
    m = m2;
  } else {
    s += s2 * exp(d);
  }
  const uint64_t mb = fx_bits(m), sb = fx_bits(-s);
  a.w[0] = (uint32_t)mb;
  a.w[1] = (uint32_t)(mb >> 32);
  a.w[2] = (uint32_t)sb;
  a.w[3] = (uint32_t)(sb >> 32) | 0x80000000u;
  return a;
}
ACG_FX_HD void fx_merge(FxLse& a, FxLse b) {
  if (fx_wide(a) || fx_wide(b)) {
    a = fx_merge_wide(a, b);
    return;
  }
  const int ka = (int)a.w[0], kb = (int)b.w[0];
  if (kb > ka) {
    fx_shift(a, (uint32_t)kb - (uint32_t)ka);
    a.w[0] = (uint32_t)kb;
  } else {
    fx_shift(b, (uint32_t)ka - (uint32_t)kb);
  }
  const uint64_t x = ((uint64_t)a.w[2] << 32) | a.w[1], y = ((uint64_t)b.w[2] << 32) | b.w[1];
  const uint64_t t = x + y;
  a.w[3] += b.w[3] + (t < x ? 1u : 0u);
  a.w[1] = (uint32_t)t;
  a.w[2] = (uint32_t)(t >> 32);
}

// ---- distances: sqrt(sum_k (x_k - y_k)^2) from fixed point
// A feature in units of 2^(a - W), |x| < 2^a, as h 2^LB + l: h signed, l LB bits.
// Differences of the parts need no carry.  For sums over up to KM features the
// parts are as wide as 64 bits allow: dh^2 and dl^2 (unsigned) below 2^64 / KM,
// dh dl (signed) below 2^63 / KM.
// A feature of at least 2^(a - W + 52) is exact, a smaller one rounded to half a
// unit.  Distances of less than 2^T units are left to FP64 (fx_small): from there
// on the result's error against extended precision is below FP64's own, whose
// differences, squares and sums round at every step.  In units of the last place,
// 17 features: N(0, 1) rms 0.29, largest 0.55 (FP64 0.50 and 2.4); pairs between
// 2^52 and 2^53 units, the outermost, 0.51 and 1.9 (FP64 0.56 and 2.4).  Up to four
// features leave FP64 less to round, so their limit is higher; a single one next to
// nothing: it stays in FP64.
template <int KM>
struct FxWindow {
  static constexpr int LB = KM <= 4 ? 31 : KM <= 8 ? 30 : 29;
  static constexpr int W = LB + (KM <= 2 ? 30 : KM <= 16 ? 29 : 28);
  static constexpr int T = KM <= 4 ? 53 : 52;
};
struct FxPart {
  int32_t h, l;
};
// x rounded to a multiple of the unit; *big is set where |x| >= 2^a (or rounds to
// it) or x is not finite.
template <int KM>
ACG_FX_HD FxPart fx_part(double x, int a, bool* big) {
  constexpr int W = FxWindow<KM>::W, LB = FxWindow<KM>::LB;
  const uint64_t b = fx_bits(x);
  const uint32_t hi = (uint32_t)(b >> 32);
  const int e = (int)((hi >> 20) & 0x7ffu);
  if (e >= a + 1023) *big = true;  // |x| >= 2^a, infinities, NaN
  // 53-bit mantissa in units of 2^(e - 1075), moved up to W bits: sh >= 0 below 2^a
  const uint64_t m = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << (W - 53);
  const int sh = a + 1022 - e;
  // to nearest, ties to even: with ties away from zero the errors of x and y add up
  // along their difference
  uint64_t v = sh <= 0 ? m : sh > 62 ? 0ull : (m + ((1ull << (sh - 1)) - 1u + ((m >> sh) & 1u))) >> sh;
  if (e == 0) v = 0;  // zero (a subnormal is far below any unit used)
  if ((v >> W) != 0) *big = true;
  const int64_t s = (int32_t)hi < 0 ? -(int64_t)v : (int64_t)v;
  FxPart p;
  p.h = (int32_t)(s >> LB);
  p.l = (int32_t)((uint32_t)s & ((1u << LB) - 1u));
  return p;
}

ACG_FX_HD float fx_rsqrt(float x) {
#ifdef __CUDA_ARCH__
  return rsqrtf(x);
#else
  return (float)(1.0 / std::sqrt((double)x));
#endif
}
ACG_FX_HD int32_t fx_f2i(float x) {
#ifdef __CUDA_ARCH__
  return __float2int_rn(x);
#else
  return (int32_t)std::lrintf(x);
#endif
}
ACG_FX_HD uint32_t fx_f2u(float x) {  // saturating
#ifdef __CUDA_ARCH__
  return __float2uint_rz(x);
#else
  return x >= 4294967296.f ? 0xffffffffu : (uint32_t)x;
#endif
}

// sqrt(sh 2^(2 LB) + sc 2^(LB + 1) + sl) 2^(a - W) rounded to a double, for sums
// that are not fx_small: a radicand of at least 2^(2 T).
// Two Newton steps from a single-precision reciprocal root: R0 (31 bits), then
// the residuals of 64 and of the next bits, each multiplied by the same
// reciprocal; the root carries 58 bits before its rounding, so it is nearly always
// the double nearest to that of the radicand.
template <int KM>
ACG_FX_HD bool fx_small(uint64_t sh) {
  return (sh >> (2 * (FxWindow<KM>::T - FxWindow<KM>::LB))) == 0;
}
template <int KM>
ACG_FX_HD double fx_root(uint64_t sh, int64_t sc, uint64_t sl, int a) {
  constexpr int W = FxWindow<KM>::W, LB = FxWindow<KM>::LB;
  // the radicand as hi 2^64 + lo
  const uint64_t c = (uint64_t)sc << (LB + 1);
  uint64_t lo = (sh << (2 * LB)) + c;
  uint64_t hi = (sh >> (64 - 2 * LB)) + (uint64_t)(sc >> (63 - LB)) + (lo < c ? 1u : 0u);
  lo += sl;
  hi += lo < sl ? 1u : 0u;
#ifdef __CUDA_ARCH__
  const int z = __clzll((long long)hi) & ~1;
#else
  const int z = __builtin_clzll(hi) & ~1;
#endif
  // (2 <= z <= 24) 2^z radicand in [2^126, 2^128): its upper 64 bits
  const uint64_t n = (hi << z) | (lo >> (64 - z));
  const float nf = (float)(uint32_t)(n >> 32);
  const float y = fx_rsqrt(nf);  // 2^-15 .. 2^-16
  const uint32_t r0 = fx_f2u(nf * y * 65536.f);
  const int64_t e0 = (int64_t)(n - (uint64_t)r0 * r0);
  const int32_t d0 = fx_f2i((float)(int32_t)(e0 >> 14) * y * 32768.f);
  const uint64_t r1 = ((uint64_t)r0 << 32) + ((uint64_t)(int64_t)d0 << 14);
  const uint32_t h1 = (uint32_t)(r1 >> 32), l1 = (uint32_t)r1;
  const int32_t e1 = (int32_t)(n - (uint64_t)h1 * h1 - (((uint64_t)h1 * l1) >> 31));
  const uint64_t r = r1 + (uint64_t)(int64_t)fx_f2i((float)e1 * y * 32768.f);
  // r 2^(-z / 2) 2^(a - W), r in [2^63, 2^64]; a carry out of r's 64 bits
  // cannot occur below the rounding (r <= 2^64 - 2^10 there)
  const uint64_t m = (r >> 11) + ((r >> 10) & 1u);
  return fx_double(((uint64_t)(1022 + 63 - (z >> 1) + a - W) << 52) + m);
}

}  // namespace acg
