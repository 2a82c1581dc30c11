// The Gear update of the plain FP64 form (cpu/common/Device.cpp:17-120), one
// lane per component with every rounding of the reference.  Lanes 0-2 of a
// group of at least four hold x, y, z of an atom, lane 3 its species; the
// component arrays are then read and written in consecutive doubles.  Used by
// the stand-alone Gear kernel and, after the force of the step, by the fused
// LJ kernel.
//
// 36 FP64 operations a component with the correct and the predict; a third of
// a warp's lanes would idle with a thread per atom holding 3 components in
// turn (90 operations one after another at 64 cycles each: 8.6 and 7.8 us a
// launch for 864 atoms, against 4 us here).
#pragma once
#include "md_exact64.cuh"
#include "md_gear.cuh"

namespace mdgb {

struct Gear64 {
  const md_double4* pos;
  md_double4* pos_next;    // may be pos itself where no other thread reads it
  double *vel, *acc, *b, *c;
  GearCoef k;
  double mass[3];          // by species
  uint64_t ymass[3];       // their division fractions
  double npos, energy_loss;
  int walls;
  int* wall_flag;          // set on a wall hit of this step
  int* trip;               // trip flag of the step the new positions are for
  const float4* pos_build; // skin reference positions (may be NULL)
  float trip2;
  int* status;
  int predict;             // the next step's predict follows
};

// f / m, rounded (m > 0); a force of zero, as on every atom of a perfect lattice,
// is its own quotient: on the FP64 pipe with the other rare exponents it made the
// first accelerations of 1,048,576 atoms take 117 us (18 now)
__device__ __forceinline__ double div_mass(double f, double m, uint64_t y) {
  const uint64_t fb = (uint64_t)__double_as_longlong(f);
  const uint64_t u = fb & ~(1ull << 63);
  if (u == 0) return f;
  if ((uint32_t)(u >> 52) - 512u < 1022u)
    return __longlong_as_double((long long)(
        idiv64_const(u, (uint64_t)__double_as_longlong(m), y) | (fb & (1ull << 63))));
  return xdiv(f, m);
}

enum { GEAR64_PREDICT = 0, GEAR64_CORRECT = 1, GEAR64_REDO = 2 };

// Component d (lanes d = 0..2 of each group, `base` the group's first lane) of
// atom i under force component f.  CORRECT: the correct with the reference's
// walls, then the predict if asked for; REDO: a = F/m where `hit` (the forces
// after a wall hit, Host.cpp:168-178), then the predict if asked for; PREDICT:
// the predict alone.  Warp-collective; `on` marks the lanes that hold an atom.
template <int MODE>
__device__ __forceinline__ void gear64_component(const Gear64& a, bool on, int i, int d, int base,
                                                 int type, double f, bool hit) {
  const GearCoef& k = a.k;
  const bool live = on && d < 3;
  const size_t o = 3 * (size_t)i + d;
  double r = 0, v = 0, ac = 0, b = 0, c = 0;
  if (live) {
    r = ((const double*)a.pos)[4 * (size_t)i + d];
    v = a.vel[o];
    ac = a.acc[o];
    b = a.b[o];
    c = a.c[o];
  }
  if (MODE != GEAR64_PREDICT) {
    const int sp = type == SP_N ? 0 : (type == SP_O ? 1 : 2);
    const double m = sp == 0 ? a.mass[0] : (sp == 1 ? a.mass[1] : a.mass[2]);
    const uint64_t y = sp == 0 ? a.ymass[0] : (sp == 1 ? a.ymass[1] : a.ymass[2]);
    if (MODE == GEAR64_CORRECT) {
      const double ai = div_mass(f, m, y);
      const double corr = xsub(ai, ac);
      r = xadd(r, xmul(k.cr, corr));
      v = xadd(v, xmul(k.cv, corr));
      ac = ai;
      b = xadd(b, xmul(k.cb, corr));
      c = xadd(c, xmul(k.cc, corr));
    } else if (hit) {
      ac = div_mass(f, m, y);
    }
  }
  if (MODE == GEAR64_CORRECT) {
    if (a.walls) {
      const double np = a.npos;
      const double ry = __shfl_sync(0xffffffffu, r, base + 1);
      bool wall = false;
      if (d == 0) {
        if (r > np && ry > 0) { wall = true; v = xmul(-v, a.energy_loss); r = np; }
        if (r > np && ry < 0) { wall = true; r = -np; }
        if (r < -np) { wall = true; v = -v; r = -np; }
      } else if (fabs(r) > np) {
        wall = true;
        v = -v;
        r = xmul(np, xdiv(r, fabs(r)));
      }
      if (live && wall) atomicOr(a.wall_flag, 1);
    }
    if (live && !(isfinite(r) && isfinite(v))) atomicOr(a.status, ST_NONFINITE);
  }
  const bool predict = MODE == GEAR64_PREDICT || a.predict;
  if (predict) {
    r = xadd(xadd(xadd(xadd(r, xmul(k.c1, v)), xmul(k.c2, ac)), xmul(k.c3, b)), xmul(k.c4, c));
    v = xadd(xadd(xadd(v, xmul(k.c1, ac)), xmul(k.c2, b)), xmul(k.c3, c));
    ac = xadd(xadd(ac, xmul(k.c1, b)), xmul(k.c2, c));
    b = xadd(b, xmul(k.c1, c));
  }
  if (live) {
    if (MODE != GEAR64_REDO || predict) {
      a.vel[o] = v;
      a.b[o] = b;
    }
    a.acc[o] = ac;
    if (MODE == GEAR64_CORRECT) a.c[o] = c;
  }
  if (MODE != GEAR64_REDO || predict) {
    if (on && d < 4)
      ((double*)a.pos_next)[4 * (size_t)i + d] =
          d < 3 ? r : ((const double*)a.pos)[4 * (size_t)i + 3];
    if (a.pos_build) {
      float t = 0.f;
      if (live) {
        t = narrow_rn(r) - ((const float*)a.pos_build)[4 * (size_t)i + d];
        t *= t;
      }
      const float s = __shfl_sync(0xffffffffu, t, base) + __shfl_sync(0xffffffffu, t, base + 1) +
                      __shfl_sync(0xffffffffu, t, base + 2);
      if (live && d == 0 && s > a.trip2) *a.trip = 1;
    }
  }
}

}  // namespace mdgb
