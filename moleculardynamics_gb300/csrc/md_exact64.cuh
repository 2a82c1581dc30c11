// Correctly rounded FP64 products, quotients and square roots by integer
// operations.
//
// GB300's FP64 pipe takes 64 cycles of a scheduler for a warp-wide operation
// (1.25 TFLOP/s measured), and a division or a square root is eight to ten of
// them.  The integer pipes run at half to full rate, so a 53-bit product by
// 32 x 32 -> 64 multiplies costs about 25 issue slots, and a reciprocal or a
// square root about 45: the plain FP64 Lennard-Jones pair (one square root,
// three quotients, a dozen products, every one rounded as the reference
// rounds it) is evaluated here with the FP64 pipe left for the additions.
//
// Method: a seed of 22 bits from the FP32 approximation instruction, Newton
// steps in fixed point (the residual N - q B or N - q^2 is exact, taken modulo
// 2^64 once it is known to fit), and one exact test of the last residual
// against half a unit in the last place.  Quotients and roots of 53-bit
// numbers never lie halfway between two results, so the test is strict.
//
// Arguments and results are the bit patterns of positive normal doubles whose
// results are normal (no zero, subnormal, infinity or NaN): callers screen the
// range.  Everything but the two seeds is plain integer code, compiled for
// the host as well.
#pragma once
#include <stdint.h>

#include <cuda_runtime.h>

namespace mdgb {

constexpr uint64_t kMant52 = (1ull << 52) - 1;

__host__ __device__ __forceinline__ uint64_t wide32(uint32_t a, uint32_t b) {
  return (uint64_t)a * b;
}

// hi 2^64 + lo = a b, four 32 x 32 -> 64 multiply-adds
__host__ __device__ __forceinline__ void mul128(uint64_t a, uint64_t b, uint64_t& hi,
                                                uint64_t& lo) {
  const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32);
  const uint32_t bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
  const uint64_t p0 = wide32(al, bl);
  const uint64_t p1 = wide32(al, bh) + (p0 >> 32);
  const uint64_t p2 = wide32(ah, bl) + (uint32_t)p1;
  hi = wide32(ah, bh) + (p1 >> 32) + (p2 >> 32);
  lo = (p2 << 32) | (uint32_t)p0;
}

__host__ __device__ __forceinline__ uint64_t mant64(uint64_t a) {
  return (a & kMant52) | (1ull << 52);
}

// the bits of a double from its biased exponent and its mantissa with the
// leading one (which may have carried into 2^53)
__host__ __device__ __forceinline__ uint64_t pack64(uint32_t exponent, uint64_t m) {
  return m + ((uint64_t)((exponent - 1) << 20) << 32);
}

// a b
__host__ __device__ __forceinline__ uint64_t imul64(uint64_t a, uint64_t b) {
  uint64_t hi, lo;
  mul128(mant64(a), mant64(b) << 11, hi, lo);  // hi in [2^51, 2^53)
  const uint32_t big = (uint32_t)(hi >> 52);   // product of mantissas at least 2
  if (!big) {
    hi = (hi << 1) | (lo >> 63);
    lo <<= 1;
  }
  // above half a unit, or half and odd
  const uint64_t up = lo > (1ull << 63) - (hi & 1);
  return pack64((uint32_t)(a >> 52) + (uint32_t)(b >> 52) - 1023 + big, hi + up);
}

// the seed y of 22 bits as a 32-bit fraction (y in [0.5, 1): the true value
// lies in (0.5, 1], the approximation may fall just outside)
__host__ __device__ __forceinline__ uint32_t seed_fraction(uint32_t ybits) {
  const uint32_t b = ybits < 0x3F7FFFFFu ? ybits : 0x3F7FFFFFu;
  return b > 0x3F000000u ? (b << 8) | 0x80000000u : 0x80000000u;
}

// 1 / b from the seed's fraction y ~ 2^32 / (mantissa of b)
__host__ __device__ __forceinline__ uint64_t ircp64_seeded(uint64_t b, uint32_t y) {
  const uint64_t mb = mant64(b);
  // d = 1 - y b in units of 2^-62 (below 2^40)
  const uint64_t pl = (uint64_t)y * (uint32_t)mb, ph = (uint64_t)y * (uint32_t)(mb >> 32);
  const int64_t d = (int64_t)((1ull << 62) - ((ph << 10) + (pl >> 22)));
  const int32_t y31 = (int32_t)(y >> 1);
  // c ~ 2^105 / mb within 2^9; the exact residual 2^105 - c mb fits 63 bits
  uint64_t c = ((uint64_t)y << 21) + (uint64_t)(((int64_t)(int32_t)(d >> 10) * y31) >> 30);
  int64_t r = (int64_t)(0 - c * mb);
  const int32_t q =
      (int32_t)(((int64_t)(int32_t)(r >> 32) * y31 + (1ll << 50)) >> 51);
  c += (uint64_t)(int64_t)q;
  r -= (int64_t)q * (int64_t)mb;
  const int64_t h = (int64_t)mb;
  c += (uint64_t)(2 * r > h) - (uint64_t)(2 * r < -h);
  return pack64(2045 - (uint32_t)(b >> 52), c);
}

// sqrt(x) from the seed's fraction y ~ 2^32 / sqrt(v), x = v 4^k, v in [1, 4);
// sq receives the rounded square of the rounded root
__host__ __device__ __forceinline__ uint64_t isqrt64_seeded(uint64_t x, uint32_t y,
                                                            uint64_t& sq) {
  const uint32_t ex = (uint32_t)(x >> 52), even = ~ex & 1;
  const uint64_t m = mant64(x), M = m << (10 + even);  // v 2^62
  const int32_t y31 = (int32_t)(y >> 1);
  const uint32_t g = (uint32_t)(wide32((uint32_t)(M >> 32), y) >> 32);  // sqrt(v) 2^30
  const int64_t d = (int64_t)((M >> 2) - wide32(g, g));
  uint64_t c = ((uint64_t)g << 20) + (uint64_t)(((int64_t)(int32_t)(d >> 12) * y31) >> 30);
  // c ~ sqrt(v) 2^50 within 2^9; the exact residual v 2^100 - c^2 fits 62 bits
  int64_t r = (int64_t)((M << 38) - c * c);
  const int32_t q =
      (int32_t)(((int64_t)(int32_t)(r >> 32) * y31 + (1ll << 47)) >> 48);
  c <<= 2;
  r = (int64_t)((uint64_t)r << 4) - (int64_t)q * (int64_t)(2 * c + (uint64_t)(int64_t)q);
  c += (uint64_t)(int64_t)q;
  const int64_t h = (int64_t)c;
  if (r > h) {  // (c + 1)^2 = c^2 + 2 c + 1
    r -= 2 * h + 1;
    c++;
  } else if (r <= -h) {
    r += 2 * h - 1;
    c--;
  }
  const uint64_t root = pack64((ex + 1023) >> 1, c);
  // the square is m 2^(52 + even) - r, |r| < 2^53: m less r rounded to whole
  // units.  At the ends of the binade the unit may change: take the product.
  if (m - ((1ull << 52) + 2) < (1ull << 52) - 4) {
    const uint64_t t = m - (uint64_t)(r >> (52 + even));
    const uint64_t f = (uint64_t)r & ((1ull << (52 + even)) - 1);
    sq = pack64(ex, t - (uint64_t)(f + (t & 1) > (1ull << (51 + even))));
  } else {
    sq = imul64(root, root);
  }
  return root;
}

// a / b for a divisor known beforehand: y = divisor_fraction(b)
__host__ __device__ __forceinline__ uint64_t idiv64_const(uint64_t a, uint64_t b, uint64_t y) {
  const uint64_t ma = mant64(a), mb = mant64(b);
  uint64_t t, low;  // t = 2^63 a / b, at most 2 below
  mul128(ma << 11, y, t, low);
  const uint32_t s = (uint32_t)(t >> 63);
  uint64_t c = t >> (10 + s);
  const uint64_t r = (ma << (53 - s)) - c * mb;  // in [0, 2 mb)
  c += (uint64_t)(2 * r > mb) + (uint64_t)(2 * r > 3 * mb);
  return pack64((uint32_t)(a >> 52) - (uint32_t)(b >> 52) + 1022 + s, c);
}

// floor(2^116 / mantissa of b), at most 2^64 - 1
inline uint64_t divisor_fraction(uint64_t b) {
  const unsigned __int128 q = ((unsigned __int128)1 << 116) / mant64(b);
  return q >> 64 ? ~0ull : (uint64_t)q;
}

// x truncated to FP32 by moving the fields (a conversion instruction takes the
// FP64 pipe): tiny values to 0; NaN beyond FP32's range
__host__ __device__ __forceinline__ float trunc32(double x) {
#ifdef __CUDA_ARCH__
  const uint64_t u = (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  __builtin_memcpy(&u, &x, 8);
#endif
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
  const uint32_t e = (hi >> 20) & 0x7FFu;
  const uint32_t m = ((hi & 0xFFFFFu) << 3) | (lo >> 29);
  const uint32_t v = e >= 1151u  ? 0x7FC00000u
                     : e < 897u ? 0u
                                : (hi & 0x80000000u) | ((e - 896u) << 23) | m;
#ifdef __CUDA_ARCH__
  return __uint_as_float(v);
#else
  float f;
  __builtin_memcpy(&f, &v, 4);
  return f;
#endif
}

#ifdef __CUDACC__
__device__ __forceinline__ uint64_t ircp64(uint64_t b) {
  const uint32_t f = 0x3F800000u | (uint32_t)((b >> 29) & 0x7FFFFFu);
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
  return ircp64_seeded(b, seed_fraction(__float_as_uint(y)));
}

__device__ __forceinline__ uint64_t isqrt64(uint64_t x, uint64_t& sq) {
  const uint32_t odd = (uint32_t)(x >> 52) & 1;  // odd biased exponent: v in [1, 2)
  const uint32_t f = (odd ? 0x3F800000u : 0x40000000u) | (uint32_t)((x >> 29) & 0x7FFFFFu);
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
  return isqrt64_seeded(x, seed_fraction(__float_as_uint(y)), sq);
}

// ---- nearly rounded reciprocal, root and exponential for FP64 kernels whose
// results carry a tolerance (the bond order): one Newton step of third order
// from the same 22-bit seeds, three to five FP64 operations instead of the
// library's eight to ten.  Largest errors over 4 million arguments each, in units in
// the last place: 0.5000 (reciprocal, inverse root, root), 0.511 (exponential) ----

// 1 / b, b positive and normal with a normal reciprocal
__device__ __forceinline__ double rcp64(double b) {
  const uint64_t bb = (uint64_t)__double_as_longlong(b);
  const uint32_t f = 0x3F800000u | (uint32_t)((bb >> 29) & 0x7FFFFFu);
  float s;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(__uint_as_float(f)));
  const uint32_t m = seed_fraction(__float_as_uint(s)) << 1;  // below the leading one
  const double y = __hiloint2double(
      (int)(((2045u - (uint32_t)(bb >> 52)) << 20) | (m >> 12)), (int)(m << 20));
  const double e = fma(-b, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// 1 / sqrt(x), x positive and normal, or 0
__device__ __forceinline__ double rsqrt64(double x) {
  const uint64_t xb = (uint64_t)__double_as_longlong(x);
  const uint32_t ex = (uint32_t)(xb >> 52);
  if (ex == 0) return __longlong_as_double(0x7FF0000000000000ll);  // 0: infinity
  const uint32_t f = ((ex & 1) ? 0x3F800000u : 0x40000000u) | (uint32_t)((xb >> 29) & 0x7FFFFFu);
  float s;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(__uint_as_float(f)));
  const uint32_t m = seed_fraction(__float_as_uint(s)) << 1;
  // x = v 4^k with 1023 + k = (ex + 1023) >> 1
  const double y = __hiloint2double(
      (int)(((2045u - ((ex + 1023u) >> 1)) << 20) | (m >> 12)), (int)(m << 20));
  const double h = x * y, l = fma(x, y, -h);
  const double e = fma(-l, y, fma(-h, y, 1.0));
  return fma(y, e * fma(0.375, e, 0.5), y);
}

// sqrt(x) from ir = rsqrt64(x)
__device__ __forceinline__ double root64(double x, double ir) {
  const double r = x * ir;
  return fma(fma(-r, r, x), 0.5 * ir, r);
}

// 2^(k / 64), the nearest number and the rest
static __device__ const double2 kExp2Table[64] = {
    {0x1.0000000000000p+0, 0.0}, {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55}, {0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54}, {0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59},
    {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54}, {0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55}, {0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55},
    {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54}, {0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54}, {0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55},
    {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55}, {0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55}, {0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54},
    {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54}, {0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55}, {0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58},
    {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59}, {0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56}, {0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54},
    {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55}, {0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54}, {0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54},
    {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54}, {0x1.6623882552225p+0, -0x1.bb60987591c34p-54},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54}, {0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57},
    {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55}, {0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55}, {0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56},
    {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54}, {0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54}, {0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55},
    {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57}, {0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56}, {0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54},
    {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54}, {0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54}, {0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57},
    {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56}, {0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55}, {0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54},
    {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56}, {0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55}, {0x1.da9e603db3285p+0, 0x1.c2300696db532p-54},
    {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54}, {0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54}, {0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54},
    {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54}, {0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55}};

// exp(x) by the table-driven method of P. T. P. Tang (ACM TOMS 15, 1989): x =
// (64 q + k) ln 2 / 64 + r, exp(x) = 2^q 2^(k/64) (1 + r + r^2/2 + ... + r^6/720),
// |r| < 0.0055, ten FP64 operations.  |x| is held below 700: the bond order's
// exponents stay below 160 (distances up to its largest cutoff, 41 angstrom).
__device__ __forceinline__ double exp64(double x) {
  const float xt = trunc32(x);
  const bool far = !(fabsf(xt) <= 700.f);  // or not a number
  const bool nan = ((uint64_t)__double_as_longlong(x) << 1) > 0xFFE0000000000000ull;
  const float lim = nan ? 0.f : (__double2hiint(x) < 0 ? -700.f : 700.f);
  const float nf = rintf((far ? lim : xt) * 92.332482616893657f);
  const int n = (int)nf;
  // nf widened by moving the fields
  const uint32_t u = __float_as_uint(nf);
  const double nd = __hiloint2double(
      n == 0 ? 0 : (int)((u & 0x80000000u) | (((u >> 3) & 0x0FFFFFFFu) + (896u << 20))),
      (int)(u << 29));
  double r = fma(nd, -0x1.62e42fee00000p-7, x);
  r = fma(nd, -0x1.a39ef35793c76p-39, r);
  if (far) r = nan ? x : 0.0;
  const double p =
      fma(fma(fma(fma(1.0 / 720.0, r, 1.0 / 120.0), r, 1.0 / 24.0), r, 1.0 / 6.0), r, 0.5);
  const double q = fma(p, r * r, r);
  const double2 t = __ldg(&kExp2Table[n & 63]);
  const double v = t.x + fma(t.x, q, t.y);
  return __hiloint2double(__double2hiint(v) + ((n >> 6) << 20), __double2loint(v));
}
#endif

}  // namespace mdgb
