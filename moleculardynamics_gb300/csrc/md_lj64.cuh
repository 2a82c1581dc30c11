// The Lennard-Jones pair in FP64 with every rounding of the reference
// (cpu/common/LennardJones.h:12-30), in integer operations, for the kernels that
// sum it in row order (md_forces.cu, md_refshim.cu).
#pragma once
#include <cstring>

#include "md_exact64.cuh"
#include "md_neighbor.cuh"
#include "md_potential.cuh"

namespace mdgb {

// Per species-pair constants of the exact pair (LennardJones.h:12-30): sigma^2
// with its fraction for the division, 24 eps / sigma^2, and the energy terms.
struct LjPairConst {
  double sq[3], con[3], eps2[3], eshift[3];
  uint64_t yq[3];
};

// d d, rounded; the FP64 pipe near the ends of the exponent range (0 is 0)
__device__ __forceinline__ double sq64(double d) {
  const uint64_t b = (uint64_t)__double_as_longlong(d) & ~(1ull << 63);
  if ((uint32_t)(b >> 52) - 512u < 1022u) return __longlong_as_double((long long)imul64(b, b));
  return b == 0 ? 0.0 : xmul(d, d);
}

// the FP64 instructions, out of line (see lj_terms)
static __device__ __noinline__ double3 lj_terms_far(double r2, double ijx, double ijy, double ijz,
                                             double sq, double con) {
  // from zero sums the additions return the products themselves
  double3 t = make_double3(0.0, 0.0, 0.0);
  lj_pair_exact_c(t.x, t.y, t.z, __dsqrt_rn(r2), ijx, ijy, ijz, sq, con);
  return t;
}

// r_ij f_ij of a pair in (tx, ty, tz): LennardJones.h:12-30 with every rounding
// of the reference.  The root, the quotients and the power chain are integer
// operations (md_exact64.cuh); the last five operations stay on the FP64 pipe,
// which the integers leave idle otherwise (with those in integers too the
// 108,000-atom launch took 276 us, not 255).  Squared distances outside
// 2^-30 .. 2^30 take lj_pair_exact_c's instructions.
__device__ __forceinline__ void lj_terms(double r2, double ijx, double ijy, double ijz, double sq,
                                         uint64_t yq, double con, double& tx, double& ty,
                                         double& tz) {
  const uint64_t rb = (uint64_t)__double_as_longlong(r2);
  if ((uint32_t)(rb >> 52) - 993u < 60u) {
    uint64_t d2;  // the rounded square of the rounded root
    isqrt64(rb, d2);
    const uint64_t dist2 = idiv64_const(d2, (uint64_t)__double_as_longlong(sq), yq);
    const uint64_t dist4 = imul64(dist2, dist2);
    const uint64_t dist8 = imul64(dist4, dist4);
    const uint64_t dist14 = imul64(imul64(dist2, dist4), dist8);
    const uint64_t inv8 = ircp64(dist8), inv14 = ircp64(dist14);
    // 2 / dist14 is exact: one more in the exponent
    const double s = xsub(__longlong_as_double((long long)(inv14 + (1ull << 52))),
                          __longlong_as_double((long long)inv8));
    const double fij = xmul(s, con);
    tx = xmul(ijx, fij);
    ty = xmul(ijy, fij);
    tz = xmul(ijz, fij);
    return;
  }
  const double3 t = lj_terms_far(r2, ijx, ijy, ijz, sq, con);
  tx = t.x;
  ty = t.y;
  tz = t.z;
}

// (int)w of a species word (0, 1 or 2 as a double) without a conversion
// instruction, which takes the FP64 pipe
__device__ __forceinline__ int species64(double w) {
  const uint32_t hi = (uint32_t)__double2hiint(w);
  if (hi - 0x40000000u < 0x80000u) return 2;
  if (hi - 0x3FF00000u < 0x100000u) return 1;
  return (hi & 0x7FFFFFFFu) < 0x3FF00000u ? 0 : (int)w;
}

// x + img box, img in {-1, 0, 1} (the product is exact: no operation for it)
__device__ __forceinline__ double image64(double x, int img, double box) {
  return img == 0 ? x : xadd(x, img > 0 ? box : -box);
}

__device__ __forceinline__ bool below64(double r2, double rcutsq) {
  // r2 >= 0: the order of the bit patterns; a NaN counts as inside, as the
  // comparison r2 >= rcutsq is false for it
  const uint64_t a = (uint64_t)__double_as_longlong(r2);
  return a < (uint64_t)__double_as_longlong(rcutsq) || a > 0x7FF0000000000000ull;
}

inline LjPairConst lj_pair_const(const Species& sp, double rcutsq) {
  LjPairConst c;
  for (int t = 0; t < 3; t++) {
    const double sig = sp.sig[t], eps = sp.eps[t];
    c.sq[t] = sig * sig;
    c.con[t] = 24.0 * eps / c.sq[t];
    c.eps2[t] = 2.0 * eps;
    const double src2 = c.sq[t] / rcutsq, src6 = src2 * src2 * src2;
    const double src12 = src6 * src6;
    c.eshift[t] = c.eps2[t] * (src12 - src6);
    uint64_t b;
    memcpy(&b, &c.sq[t], sizeof(b));
    c.yq[t] = divisor_fraction(b);
  }
  return c;
}

}  // namespace mdgb
