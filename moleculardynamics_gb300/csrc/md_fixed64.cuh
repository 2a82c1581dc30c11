// Angle terms of the bond order in 64-bit fixed point.
//
// GB300's FP64 pipe takes 64 cycles of a scheduler for a warp-wide operation; a
// 64-bit fixed-point product is four 32 x 32 -> 64 multiply-adds and about
// twelve simpler instructions.  The angle terms of a triplet are 75 FP64
// operations on quantities of known size (cosines, distances and their
// reciprocals), so they are evaluated here with 56 bits after the point,
// |v| < 64: a step of 1.4e-17, against FP64's 1.1e-16 for values about 1.
// The one quantity that runs over many sizes, the cutoff function (e^-4 per
// angstrom), carries a power of two beside its fixed-point number, as do the sums
// and the coefficients that it multiplies: a term of 1e-10 has as many bits as
// one of 1.  (Without it the force on an atom 4 angstrom from a bonded pair had an
// error of 8e-14 of its size, 7 angstrom away 6e-11; 3e-15 with it at either.  The
// reference's (1 - tanh) / 2 in FP64: 9e-15 and 2e-11.)
// The caller keeps distances within 0.5 .. 16 angstrom.
//
// Plain integer code but for the two seeds; compiled for the host as well.
#pragma once
#include <stdint.h>

#include <cuda_runtime.h>

#include "md_exact64.cuh"

namespace mdgb {

typedef long long q56;
constexpr q56 kQOne = 1ll << 56;

// a b, rounded; |a|, |b| and the product below 64.  Limbs of 31 bits keep
// every partial product a signed 32 x 32 one.
__host__ __device__ __forceinline__ q56 mulq(q56 a, q56 b) {
  const int32_t ah = (int32_t)(a >> 31), bh = (int32_t)(b >> 31);
  const int32_t al = (int32_t)a & 0x7FFFFFFF, bl = (int32_t)b & 0x7FFFFFFF;
  const int64_t mid =
      (int64_t)ah * bl + (int64_t)al * bh + (((int64_t)al * bl + (1ll << 55)) >> 31);
  return (((int64_t)ah * bh) << 6) + (mid >> 25);
}

// a0 b0 + a1 b1 + a2 b2 of unit vectors
__host__ __device__ __forceinline__ q56 dotq(q56 a0, q56 a1, q56 a2, q56 b0, q56 b1, q56 b2) {
  return mulq(a0, b0) + mulq(a1, b1) + mulq(a2, b2);
}

__host__ __device__ __forceinline__ q56 toq(double v) {
#ifdef __CUDA_ARCH__
  const uint64_t u = (uint64_t)__double_as_longlong(v);
#else
  uint64_t u;
  __builtin_memcpy(&u, &v, 8);
#endif
  const int sh = (int)((u >> 52) & 0x7FF) - 1019;  // mantissa 2^sh is v 2^56
  const uint64_t m = mant64(u);
  const uint64_t r = sh >= 0 ? m << (sh & 15) : (sh < -63 ? 0 : m >> -sh);
  return (u >> 63) ? -(q56)r : (q56)r;
}

// v 2^-n
__host__ __device__ __forceinline__ double fromq(q56 v, int n = 0) {
  const uint64_t a = v < 0 ? (uint64_t)-v : (uint64_t)v;
#ifdef __CUDA_ARCH__
  const int lz = __clzll((long long)a);
#else
  const int lz = a ? __builtin_clzll(a) : 64;
#endif
  const uint64_t top = a << (lz & 63);  // leading one at bit 63
  const uint64_t m = (top >> 11) + ((top >> 10) & 1);
  // v = m 2^(11 - lz - 56); m may have carried into 2^53
  const uint64_t u = a == 0 ? 0
                            : pack64(1023 + 7 - lz - n, m) |
                                  ((uint64_t)v & 0x8000000000000000ull);
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double d;
  __builtin_memcpy(&d, &u, 8);
  return d;
#endif
}

// y c 2^-31 for a correction c below 2^44 and y < 2^31, without losing c's low bits
__host__ __device__ __forceinline__ int64_t scaleq(int64_t c, int32_t y31) {
  return (((int64_t)(int32_t)(c >> 16) * y31) >> 15) +
         (((int64_t)(int32_t)(c & 0xFFFF) * y31) >> 31);
}

// 1 / den, den in [1, 2], y the seed's fraction
__host__ __device__ __forceinline__ q56 rcpq_seeded(q56 den, uint32_t y) {
  // e = 1 - den y, 56 bits after the point, below 2^34
  const int64_t p = (int64_t)(wide32((uint32_t)((uint64_t)den >> 32), y) +
                              (wide32((uint32_t)den, y) >> 32));
  const int64_t e = kQOne - p;
  const int32_t s = (int32_t)(e >> 17);
  const int64_t c = e + (((int64_t)s * s) >> 22);  // e + e^2
  return ((q56)y << 24) + scaleq(c, (int32_t)(y >> 1));
}

// r = sqrt(r2) and 1 / r from the bits of r2 in [0.25, 256), y the seed's fraction
__host__ __device__ __forceinline__ void rsqrtq_seeded(uint64_t r2, uint32_t y, q56& r, q56& ir) {
  const uint32_t ex = (uint32_t)(r2 >> 52), even = ~ex & 1;
  const uint64_t M = mant64(r2) << (10 + even);  // v 2^62, r2 = v 4^k
  const int k = (int)((ex + 1023) >> 1) - 1023;
  // d = 1 - v y^2 in units of 2^-62, below 2^42
  const uint64_t t = wide32((uint32_t)(M >> 32), y) + (wide32((uint32_t)M, y) >> 32);
  const uint64_t s = wide32((uint32_t)(t >> 32), y) + (wide32((uint32_t)t, y) >> 32);
  const int64_t d = (int64_t)((1ull << 62) - s);
  const int32_t e = (int32_t)(d >> 20);
  // y (1 + d / 2 + 3 d^2 / 8)
  const int64_t c = (d >> 1) + ((3 * ((int64_t)e * e)) >> 25);
  const uint64_t y63 = ((uint64_t)y << 31) + (uint64_t)(scaleq(c, (int32_t)(y >> 1)) << 1);
  ir = (q56)(y63 >> (7 + k));
  uint64_t hi, lo;
  mul128(M, y63, hi, lo);  // v y 2^61
  r = (q56)(hi >> (5 - k));
}

// 2^-(k / 128)
#ifdef __CUDA_ARCH__
static __device__ const
#else
static const
#endif
    long long kExpTableQ[129] = {
    0x100000000000000ll, 0xfe9e115c7b8f88ll, 0xfd3e0c0cf486c1ll, 0xfbdfed6ce5f09cll, 0xfa83b2db722a03ll, 0xf92959bb5dd4ball,
    0xf7d0df730ad13cll, 0xf67a416c733f84ll, 0xf5257d152486ccll, 0xf3d28fde3a641all, 0xf281773c59ffb1ll, 0xf13230a7ad0945ll,
    0xefe4b99bdcdaf6ll, 0xee990f980da302ll, 0xed4f301ed9942cll, 0xec0718b64c1cbell, 0xeac0c6e7dd2439ll, 0xe97c38406c4f8cll,
    0xe8396a503c4bdcll, 0xe6f85aaaee1fcell, 0xe5b906e77c8349ll, 0xe47b6ca0373da9ll, 0xe33f8972be8a5all, 0xe2055afffe83d3ll,
    0xe0ccdeec2a94e1ll, 0xdf9612deb8f044ll, 0xde60f4825e0e91ll, 0xdd2d818508324cll, 0xdbfbb797daf237ll, 0xdacb946f2ac9ccll,
    0xd99d15c278afd8ll, 0xd870394c6db32dll, 0xd744fccad69d6bll, 0xd61b5dfe9f9bcell, 0xd4f35aabcfedfall, 0xd3ccf099859ac3ll,
    0xd2a81d91f12ae4ll, 0xd184df6251699bll, 0xd06333daef2b26ll, 0xcf4318cf191919ll, 0xce248c151f8481ll, 0xcd078b86503dcell,
    0xcbec14fef2727cll, 0xcad2265e429077ll, 0xc9b9bd866e2f28ll, 0xc8a2d85c8ffe2cll, 0xc78d74c8abb9b1ll, 0xc67990b5aa245fll,
    0xc5672a115506dbll, 0xc4563ecc5334cbll, 0xc346ccda249764ll, 0xc238d2311e3d66ll, 0xc12c4cca667094ll, 0xc0213aa1f0d08ell,
    0xbf1799b67a7311ll, 0xbe0f6809860994ll, 0xbd08a39f580c37ll, 0xbc034a7ef2e9fbll, 0xbaff5ab2133e46ll, 0xb9fcd2452c0b9ell,
    0xb8fbaf4762fb9fll, 0xb7fbefca8ca41ell, 0xb6fd91e328d178ll, 0xb60093a85ed5f7ll, 0xb504f333f9de65ll, 0xb40aaea2654b98ll,
    0xb311c412a91125ll, 0xb21a31a66618fell, 0xb123f581d2ac26ll, 0xb02f0dcbb6e046ll, 0xaf3b78ad690a43ll, 0xae493452ca35b8ll,
    0xad583eea42a14bll, 0xac6896a4be3fe9ll, 0xab7a39b5a93ed3ll, 0xaa8d2652ec9076ll, 0xa9a15ab4ea7c0fll, 0xa8b6d5167b320ell,
    0xa7cd93b4e96535ll, 0xa6e594cfeee86bll, 0xa5fed6a9b15139ll, 0xa5195786be9ef3ll, 0xa43515ae09e681ll, 0xa3520f68e802bcll,
    0xa27043030c4968ll, 0xa18faeca8544b7ll, 0xa0b0510fb97150ll, 0x9fd228256400ddll, 0x9ef5326091a112ll, 0x9e196e189d4724ll,
    0x9d3ed9a72cffb7ll, 0x9c6573682ec32cll, 0x9b8d39b9d54e55ll, 0x9ab62afc94ff86ll, 0x99e0459320b7fall, 0x990b87e266c18all,
    0x9837f0518db8a9ll, 0x97657d49f17ab1ll, 0x96942d3720185all, 0x95c3fe86d6cc80ll, 0x94f4efa8fef709ll, 0x9426ff0fab1c05ll,
    0x935a2b2f13e6e9ll, 0x928e727d9531fall, 0x91c3d373ab11c3ll, 0x90fa4c8beee4b1ll, 0x9031dc431466b2ll, 0x8f6a8117e6c8e6ll,
    0x8ea4398b45cd54ll, 0x8ddf042022e69dll, 0x8d1adf5b7e5baall, 0x8c57c9c4646f4ell, 0x8b95c1e3ea8bd7ll, 0x8ad4c6452c7289ll,
    0x8a14d575496efell, 0x8955ee03618e60ll, 0x88980e8092da85ll, 0x87db357ff698d8ll, 0x871f61969e8d10ll, 0x8664915b923fball,
    0x85aac367cc487bll, 0x84f1f656379c1all, 0x843a28c3acde40ll, 0x8383594eefb6eell, 0x82cd8698ac2ba2ll, 0x8218af4373fc26ll,
    0x8164d1f3bc0307ll, 0x80b1ed4fd999abll, 0x80000000000000ll};

// exp(-a) = v 2^-n, a >= 0, v in (0.49, 1]: 2^-n 2^-(k / 128) e^-t, |t| <=
// ln 2 / 256, the last by its series to t^5 (the next term is 5e-19)
__host__ __device__ __forceinline__ q56 expnegq(q56 a, int& n) {
  // a / ln 2 (the second constant: 2^31 times what the first one rounds off, up to
  // 27 units for a = 58)
  const q56 w = mulq(a, 0x171547652b82fe1ll) +
                (((int64_t)(int32_t)(a >> 31) * 1002342399) >> 56);
  n = (int)(w >> 56);
  const q56 f = w & (kQOne - 1);
  const int k = (int)((f + (1ll << 48)) >> 49);
  const q56 t = mulq(f - ((q56)k << 49), 0xb17217f7d1cf7all);
  // h = 1/2 - t (1/6 - t (1/24 - t / 120)), 40 bits after the point
  const int32_t t39 = (int32_t)(t >> 17);  // |t| < 2^-8.5
  // 2^32 (1/6 - t (1/24 - t / 120))
  const int32_t u = 178956971 - (int32_t)(((int64_t)t39 * 35791394) >> 39);
  const int32_t p = 715827883 - (int32_t)(((int64_t)t39 * u) >> 39);
  const int64_t h = (1ll << 39) - (((int64_t)t39 * p) >> 31);
  const q56 e = kQOne - t + mulq(mulq(t, t), h << 16);
#ifdef __CUDA_ARCH__
  return mulq(__ldg(&kExpTableQ[k]), e);
#else
  return mulq(kExpTableQ[k], e);
#endif
}
__host__ __device__ __forceinline__ q56 expnegq(q56 a) {
  int n;
  const q56 v = expnegq(a, n);
  return n > 62 ? 0 : v >> n;
}

// the fractions of the two seeds, from an argument in [1, 2) and [1, 4) as FP32
// bits; correctly rounded on the host
__host__ __device__ __forceinline__ uint32_t rcp_seed(uint32_t f) {
  float s;
#ifdef __CUDA_ARCH__
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(__uint_as_float(f)));
  return seed_fraction(__float_as_uint(s));
#else
  __builtin_memcpy(&s, &f, 4);
  s = (float)(1.0 / (double)s);
  __builtin_memcpy(&f, &s, 4);
  return seed_fraction(f);
#endif
}
__host__ __device__ __forceinline__ uint32_t rsqrt_seed(uint32_t f) {
  float s;
#ifdef __CUDA_ARCH__
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(__uint_as_float(f)));
  return seed_fraction(__float_as_uint(s));
#else
  __builtin_memcpy(&s, &f, 4);
  s = (float)(1.0 / __builtin_sqrt((double)s));
  __builtin_memcpy(&f, &s, 4);
  return seed_fraction(f);
#endif
}

__host__ __device__ __forceinline__ q56 rcpq(q56 den) {
  return rcpq_seeded(den, rcp_seed(0x3F800000u + (uint32_t)((uint64_t)(den - kQOne) >> 33)));
}

__host__ __device__ __forceinline__ void rsqrtq(double x, q56& r, q56& ir) {
#ifdef __CUDA_ARCH__
  const uint64_t b = (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  __builtin_memcpy(&b, &x, 8);
#endif
  const uint32_t f = ((b >> 52) & 1 ? 0x3F800000u : 0x40000000u) | (uint32_t)((b >> 29) & 0x7FFFFFu);
  rsqrtq_seeded(b, rsqrt_seed(f), r, ir);
}

// the cutoff fc = 1 / (1 + e^x) = f 2^-n, x = 4 (r - R0), f in (0.24, 1], and
// h = 4 (1 - fc), with which its derivative is -h fc
__host__ __device__ __forceinline__ void cutoffq(q56 r, q56& f, int& n, q56& h) {
  const q56 x = (r - 0x14ccccc00000000ll) << 2;
  const q56 v = expnegq(x < 0 ? -x : x, n);
  const q56 s = n > 62 ? 0 : v >> n;
  const q56 d = rcpq(kQOne + s);
  if (x < 0) {
    f = d;
    h = (mulq(v << 2, d) + ((1ll << n) >> 1)) >> n;  // n at most 4
    n = 0;
  } else {
    f = mulq(v, d);
    h = d << 2;
  }
}

// the angular function K - C / (D + c^2) and its prefactor 2 C c / (D + c^2)^2
__host__ __device__ __forceinline__ void angularq(q56 c, q56& g, q56& gpre) {
  const q56 iq = rcpq((0x40aacd800000000ll + mulq(c, c)) >> 2) >> 2;
  const q56 h = 25 * iq;
  g = 0x72f7e0000000000ll - h;
  gpre = mulq(mulq(h, iq), c) << 1;
}

// two sums of terms that share a power of two: (x, y) 2^-n, n that of the
// largest term so far (smaller terms lose the bits below its last, as in FP64)
struct SumQ {
  q56 x = 0, y = 0;
  int n = 127;
};
__host__ __device__ __forceinline__ void addq(SumQ& s, q56 x, q56 y, int n) {
  const int d = n - s.n;
  const int down = d > 0 ? (d < 63 ? d : 63) : 0;  // of the term
  const int sum = d < 0 ? (d > -63 ? -d : 63) : 0;
  s.x = (s.x >> sum) + (x >> down);
  s.y = (s.y >> sum) + (y >> down);
  s.n = n < s.n ? n : s.n;
}

}  // namespace mdgb
