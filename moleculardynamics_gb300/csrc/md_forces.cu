// Force kernels: Lennard-Jones (cpu/common/LennardJones.h) and the bond-order
// many-body term (cpu/common/BondOrderFuncs.h).
//
// LJ, FP64 ("plain"): a few lanes per atom evaluate its compact row with the
// reference's roundings (integer operations in place of most of the narrow
// FP64 pipe's) and add the pairs in the reference's candidate order, so that
// forces are bit-identical to the reference on the same positions and list.
// LJ, FP32 (precision form): same rows; pair arithmetic in FP32 from the FP32
// position copy; pairs within 1e-5 of the cutoff are re-tested in FP64 so the
// pair set equals the FP64 one; per-atom sums are FP32 chunks of 16 pairs
// folded into a compensated (Kahan) FP32 pair (hi, lo), stored as FP64.
// Bond order: a short list per atom (candidates within rcut now), then
//   FP64: one block per atom i evaluates its bonds i-j with every third body m
//           once (BondOrderFuncs.h:12-143, 242-278) and leaves the force on
//           each m in a slot (:148-237), which m's warp collects (:339-393);
//   FP32: pass 1, one warp per atom i, one lane per pair (i, j), and pass 2,
//           one warp per atom k, one lane per i of k's short list, over the
//           bonds i-j whose j lies in k's candidate row.
#include <cmath>
#include <cstring>
#include <type_traits>

#include "md_exact64.cuh"
#include "md_fixed64.cuh"
#include "md_forces.h"
#include "md_gear64.cuh"
#include "md_lj64.cuh"
#include "md_neighbor.cuh"
#include "md_potential.cuh"
#include "md_tma.cuh"

namespace mdgb {

namespace {

// current FP32 position of atom j (the FP32 copy when there is one)
__device__ __forceinline__ float4 cur_pos(const md_double4* pos, const float4* posf, int j) {
  if (posf) return posf[j];
  const md_double4 p = pos[j];
  return make_float4((float)p.x, (float)p.y, (float)p.z, __int_as_float((int)p.w));
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum of NV doubles over the block, written to out[NV * blockIdx.x + k].
template <int NV>
__device__ __forceinline__ void block_partial(double (&v)[NV], double* out) {
  __shared__ double sm[NV][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; k++) {
    double x = warp_sum(v[k]);
    if (lane == 0) sm[k][warp] = x;
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < NV; k++) {
      double x = lane < nw ? sm[k][lane] : 0.0;
      x = warp_sum(x);
      if (lane == 0) out[NV * blockIdx.x + k] = x;
    }
  }
}

// ------------------------------------------------------------------ LJ FP64
// common/DebugCalculations.cpp:199-201 per ordered pair, restricted to the
// force's pairs; shifted by its value at the cutoff; the virial
__device__ __forceinline__ void lj64_energy(double r2, double ijx, double ijy, double ijz,
                                            double tx, double ty, double tz,
                                            const LjPairConst& c, int sel, double* ev) {
  const double sr2 = xdiv(c.sq[sel], r2);
  const double sr6 = xmul(xmul(sr2, sr2), sr2);
  const double e = xmul(c.eps2[sel], xsub(xmul(sr6, sr6), sr6));
  ev[0] += e;
  ev[1] += e - c.eshift[sel];
  ev[2] += 0.5 * (ijx * tx + ijy * ty + ijz * tz);
}

// One atom by one thread (a tripped skin: the full candidate row, the
// reference's row and order, and a fresh compact row at the current
// positions).
template <bool ENERGY>
__device__ __noinline__ void lj64_refresh(int i, const md_double4* __restrict__ pos,
                                          double* sums, int ld,
                                          uint32_t* __restrict__ list, int* __restrict__ len,
                                          const RowWalker& w, int* skin, int cap, float rv2,
                                          float4* __restrict__ pos_build, double rcutsq,
                                          const LjPairConst& c, double* ev) {
  const md_double4 pi = pos[i];
  const int ti = species64(pi.w);
  const double box = w.g.box;
  const float4 pc = cur_pos(pos, (const float4*)nullptr, i);
  double fx = 0.0, fy = 0.0, fz = 0.0;
  int kept = 0;
  walk_row(w, pos, i, [&](int m, int ix, int iy, int iz) {
    const md_double4 pj = pos[m];
    double xj = pj.x, yj = pj.y, zj = pj.z;
    if (w.g.periodic && (ix | iy | iz)) {
      xj = xadd(xj, (double)ix * box);
      yj = xadd(yj, (double)iy * box);
      zj = xadd(zj, (double)iz * box);
    }
    const double ijx = xsub(pi.x, xj), ijy = xsub(pi.y, yj), ijz = xsub(pi.z, zj);
    const double r2 = norm2_exact(ijx, ijy, ijz);
    const int tj = species64(pj.w);
    if (below64(r2, rcutsq) && (tj == SP_NG || ti == SP_NG)) {
      const int sel = lj_select(ti, tj);
      double tx, ty, tz;
      lj_terms(r2, ijx, ijy, ijz, c.sq[sel], c.yq[sel], c.con[sel], tx, ty, tz);
      fx = xadd(fx, tx);
      fy = xadd(fy, ty);
      fz = xadd(fz, tz);
      if (ENERGY) lj64_energy(r2, ijx, ijy, ijz, tx, ty, tz, c, sel, ev);
    }
    const float4 pm = cur_pos(pos, (const float4*)nullptr, m);
    const float dx = pc.x - (pm.x + (float)ix * w.g.box_f);
    const float dy = pc.y - (pm.y + (float)iy * w.g.box_f);
    const float dz = pc.z - (pm.z + (float)iz * w.g.box_f);
    if (dx * dx + dy * dy + dz * dz < rv2) {
      if (kept < cap) list[(size_t)kept * ld + i] = pack_entry(m, ix, iy, iz);
      kept++;
    }
  });
  if (kept > cap) atomicOr(&skin[3], 1);
  len[i] = kept < cap ? kept : cap;
  pos_build[i] = pc;
  sums[0] = fx;
  sums[1] = fy;
  sums[2] = fz;
}

constexpr int kLj64Cap = 96;  // screened entries of a group in shared memory

// G lanes of a warp per atom.  The row is read G entries at a time; an FP32
// screen (conservative: the cutoff widened by the truncation error of the
// coordinates) drops the entries beyond the cutoff, and the others queue in
// shared memory in row order.  Then each lane evaluates one queued pair, and
// three lanes add the G products of their component one after another, so the
// sums run in the reference's order and forces are bit-identical to it for
// every G.
// The FP64 pipe bounds it (14 operations per pair of one lane and 4 of three
// lanes for the sums, at 64 cycles each), then the latency of the integer
// chains: 64 registers (8 blocks per SM) took 255 us for 108,000 atoms, 72
// registers 259, 80 registers 267, 96 unbounded 280; one thread per atom with
// the FP64 instructions took 1010.
//
// FORCE: forces (and energies) alone.  STEP: the correct of the step follows
// for each atom in the lanes that hold its force (md_gear64.cuh), and where
// nothing else is due the predict of the next step; the new positions go to
// another buffer, as other blocks still read the present ones.  REDO: after a
// correct with a wall hit (*run_if) the forces and a = F/m again, and in any
// case the predict if asked for; the count of such steps and the flag of the
// next one are kept on the device, so a step with walls needs no host wait.
enum { LJ64_FORCE = 0, LJ64_STEP = 1, LJ64_REDO = 2 };
struct Lj64Args {
  const md_double4* pos;
  double* f3;
  int n, ld;
  uint32_t* list;
  int* len;
  RowWalker w;
  int* skin;
  SkinFlags sf;
  int cap;
  float rv2;
  float4* pos_build;
  double rcutsq;
  LjPairConst c;
  double* epart;
  const int* run_if;
  int* hits;       // REDO: steps with a wall hit
  int* flag_next;  // REDO: the wall flag of the next step
  int store;       // STEP: forces also to f3
  Gear64 g;
};

template <int G, int MODE, bool ENERGY>
__global__ void __launch_bounds__(128, 8) k_lj_fp64(const __grid_constant__ Lj64Args a) {
  constexpr int kAtoms = 32 / G;  // atoms per warp
  __shared__ uint32_t queue[128 / G][kLj64Cap];
  __shared__ double term[4][3][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gl = lane & (G - 1), group = lane / G;
  const int t = blockIdx.x * 128 + tid;
  grid_wait();
  grid_launch_dependents();
  const bool gate = !a.run_if || *a.run_if != 0;
  if (MODE == LJ64_REDO && t == 0) {
    if (gate) atomicAdd(a.hits, 1);
    *a.flag_next = 0;
  }
  if (!gate && !(MODE == LJ64_REDO && a.g.predict)) return;
  if (t == 0 && gate) a.skin[a.sf.clear] = 0;  // the flag of step t + 2 starts clear
  double ev[3] = {0.0, 0.0, 0.0};
  // The trip flag of the positions.  A correct without the predict (STEP)
  // leaves the trip of the corrected positions in the next step's flag: read
  // too by the launches that evaluate them.  One thread reads for the block:
  // REDO's own predict may set that flag meanwhile, and a block that sees it
  // walks full rows, which any block may.
  __shared__ int s_trip;
  if (tid == 0)
    s_trip = a.skin[a.sf.read] | a.skin[3] |
             (ENERGY || MODE == LJ64_REDO ? a.skin[(a.sf.read + 1) % 3] : 0);
  __syncthreads();
  const bool tripped = s_trip != 0;
  const int i = (blockIdx.x * 4 + warp) * kAtoms + group;
  const bool live = i < a.n;
  double acc = 0.0;  // lane gl < 3: component gl of the force
  int ti = SP_NG;
  if (!gate) {
    // the predict alone
  } else if (tripped) {
    // one thread per atom of the block
    double* sums = &term[0][0][0];
    const int first = blockIdx.x * 4 * kAtoms;
    if (tid < 4 * kAtoms && first + tid < a.n)
      lj64_refresh<ENERGY>(first + tid, a.pos, sums + 3 * tid, a.ld, a.list, a.len, a.w, a.skin,
                           a.cap, a.rv2, a.pos_build, a.rcutsq, a.c, ev);
    if (t == 0) atomicAdd(&a.skin[4], 1);
    __syncthreads();  // the whole block is here: it read the flag once (s_trip)
    if (live && gl < 3) acc = sums[3 * (warp * kAtoms + group) + gl];
    if (live) ti = species64(a.pos[i].w);
  } else {
    const LjPairConst& c = a.c;
    const md_double4* __restrict__ pos = a.pos;
    const uint32_t* __restrict__ list = a.list;
    const md_double4 pi = live ? pos[i] : md_double4{0, 0, 0, 0};
    ti = species64(pi.w);
    const double box = a.w.g.box;
    const float xf = trunc32(pi.x), yf = trunc32(pi.y), zf = trunc32(pi.z);
    // screen: each coordinate is off by less than 2^-23 of itself, and a pair
    // inside the cutoff has |x_j| <= |x_i| + rcut (+ the box, for an image)
    const float rc2 = (float)a.rcutsq * 1.000001f, rc = sqrtf(rc2), bf = a.w.g.box_f;
    const float off = (fmaxf(fabsf(xf), fmaxf(fabsf(yf), fabsf(zf))) + fabsf(bf) + rc) * 0x1p-20f;
    const float thr = rc2 + off * (8.0f * rc + 16.0f * off);
    uint32_t* q = queue[warp * kAtoms + group];
    const int L = live ? a.len[i] : 0;
    int k0 = 0;
    for (;;) {
      // screen until the queue could overflow or every row of the warp ends
      int cnt = 0;
      while (__any_sync(0xffffffffu, k0 < L && cnt + G <= kLj64Cap)) {
        const bool go = k0 < L && cnt + G <= kLj64Cap;
        const int k = k0 + gl;
        bool keep = false;
        uint32_t e = 0;
        if (go && k < L) {
          e = list[(size_t)k * a.ld + i];
          const md_double4 pj = pos[entry_index(e)];
          float dx = xf - trunc32(pj.x), dy = yf - trunc32(pj.y), dz = zf - trunc32(pj.z);
          if (e >> 26) {
            dx -= (float)entry_img(e, 0) * bf;
            dy -= (float)entry_img(e, 1) * bf;
            dz -= (float)entry_img(e, 2) * bf;
          }
          keep = !(dx * dx + dy * dy + dz * dz > thr);
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep) >> (group * G) &
                           (G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u);
        if (keep) q[cnt + __popc(m & ((1u << gl) - 1u))] = e;
        cnt += __popc(m);
        if (go) k0 += G;
      }
      __syncwarp();
      int most = cnt;
#pragma unroll
      for (int o = 16; o >= G; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
      for (int s0 = 0; s0 < most; s0 += G) {
        double tx = 0.0, ty = 0.0, tz = 0.0;
        bool in = s0 + gl < cnt;
        if (in) {
          const uint32_t e = q[s0 + gl];
          const md_double4 pj = pos[entry_index(e)];
          double xj = pj.x, yj = pj.y, zj = pj.z;
          if (e >> 26) {
            xj = image64(xj, entry_img(e, 0), box);
            yj = image64(yj, entry_img(e, 1), box);
            zj = image64(zj, entry_img(e, 2), box);
          }
          const double ijx = xsub(pi.x, xj), ijy = xsub(pi.y, yj), ijz = xsub(pi.z, zj);
          const double r2 = xadd(xadd(sq64(ijx), sq64(ijy)), sq64(ijz));
          const int tj = species64(pj.w);
          in = below64(r2, a.rcutsq) && (tj == SP_NG || ti == SP_NG);
          if (in) {
            const int sel = lj_select(ti, tj);
            const double sq = sel == 0 ? c.sq[0] : (sel == 1 ? c.sq[1] : c.sq[2]);
            const double con = sel == 0 ? c.con[0] : (sel == 1 ? c.con[1] : c.con[2]);
            const uint64_t yq = sel == 0 ? c.yq[0] : (sel == 1 ? c.yq[1] : c.yq[2]);
            lj_terms(r2, ijx, ijy, ijz, sq, yq, con, tx, ty, tz);
            if (ENERGY) lj64_energy(r2, ijx, ijy, ijz, tx, ty, tz, c, sel, ev);
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, in) >> (group * G);
        term[warp][0][lane] = tx;
        term[warp][1][lane] = ty;
        term[warp][2][lane] = tz;
        __syncwarp();
        if (gl < 3) {
          const double* tv = &term[warp][gl][group * G];
#pragma unroll
          for (int s = 0; s < G; s++)
            if ((m >> s) & 1u) acc = xadd(acc, tv[s]);
        }
        __syncwarp();
      }
      if (!__any_sync(0xffffffffu, k0 < L)) break;
    }
  }
  if (gate && (MODE != LJ64_STEP || a.store) && live && gl < 3) a.f3[3 * (size_t)i + gl] = acc;
  if (MODE == LJ64_STEP)
    gear64_component<GEAR64_CORRECT>(a.g, live, i, gl, group * G, ti, acc, false);
  if (MODE == LJ64_REDO)
    gear64_component<GEAR64_REDO>(a.g, live, i, gl, group * G, ti, acc, gate);
  if (ENERGY) block_partial<3>(ev, a.epart);
}

// ------------------------------------------------------------------ LJ FP32
__device__ __forceinline__ void kahan(float& hi, float& lo, float x) {
  float y = x - lo;
  float t = hi + y;
  lo = (t - hi) - y;
  hi = t;
}

// Is the FP32 pair (i, j) inside rcut?  Pairs within a relative 1e-5 band of
// the cutoff are decided in FP64 exactly as the FP64 path decides them.
__device__ __forceinline__ bool lj_inside(float r2, float rc_lo, float rc_hi,
                                          const md_double4* pos, int i, int j, bool img,
                                          int ix, int iy, int iz, const Grid& g,
                                          double rcutsq) {
  if (r2 >= rc_hi) return false;
  if (r2 <= rc_lo) return true;
  const md_double4 a = pos[i], b = pos[j];
  double xj = b.x, yj = b.y, zj = b.z;
  if (img) {
    xj = xadd(xj, (double)ix * g.box);
    yj = xadd(yj, (double)iy * g.box);
    zj = xadd(zj, (double)iz * g.box);
  }
  return norm2_exact(xsub(a.x, xj), xsub(a.y, yj), xsub(a.z, zj)) < rcutsq;
}

// One atom of the FP32 LJ force: the compact row, or (skin tripped) the full
// candidate row with a refresh of the compact row.  ev: E, E_shifted, W.
template <bool ENERGY>
__device__ __forceinline__ void lj32_atom(int i, const float4* __restrict__ posf,
                                          const md_double4* __restrict__ pos,
                                          double* __restrict__ f3, int ld,
                                          uint32_t* __restrict__ list, int* __restrict__ len,
                                          const RowWalker& w, bool tripped, int* skin, int cap,
                                          float rv2, float4* __restrict__ pos_build,
                                          double rcutsq, const Species& sp, double* ev) {
  const float4 pi = posf[i];
  const int ti = __float_as_int(pi.w);
  const float rc2 = (float)rcutsq;
  const float rc_lo = rc2 * (1.0f - 1e-5f), rc_hi = rc2 * (1.0f + 1e-5f);
  const float Lf = w.g.box_f, Llo = w.g.box_lo;
  float hx = 0.f, hy = 0.f, hz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
  float cx = 0.f, cy = 0.f, cz = 0.f;
  int inchunk = 0;
  auto visit = [&](int j, int ix, int iy, int iz, bool img) {
    const float4 pj = posf[j];
    float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
    if (img) {
      dx = (pi.x - fmaf((float)ix, Lf, pj.x)) - (float)ix * Llo;
      dy = (pi.y - fmaf((float)iy, Lf, pj.y)) - (float)iy * Llo;
      dz = (pi.z - fmaf((float)iz, Lf, pj.z)) - (float)iz * Llo;
    }
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (!lj_inside(r2, rc_lo, rc_hi, pos, i, j, img, ix, iy, iz, w.g, rcutsq)) return;
    const int tj = __float_as_int(pj.w);
    if (tj != SP_NG && ti != SP_NG) return;
    const int sel = lj_select(ti, tj);
    const float sig = sp.sig[sel], eps = sp.eps[sel];
    const float inv = 1.0f / r2;
    const float sr2 = sig * sig * inv;
    const float sr6 = sr2 * sr2 * sr2;
    const float fij = (24.0f * eps) * inv * sr6 * (2.0f * sr6 - 1.0f);
    cx = fmaf(dx, fij, cx);
    cy = fmaf(dy, fij, cy);
    cz = fmaf(dz, fij, cz);
    if (ENERGY) {
      const float src2 = sig * sig / rc2;
      const float src6 = src2 * src2 * src2;
      const float e = 2.0f * eps * (sr6 * sr6 - sr6);
      ev[0] += (double)e;
      ev[1] += (double)e - (double)(2.0f * eps * (src6 * src6 - src6));
      ev[2] += 0.5 * (double)(r2 * fij);
    }
    if (++inchunk == 16) {
      kahan(hx, lx, cx);
      kahan(hy, ly, cy);
      kahan(hz, lz, cz);
      cx = cy = cz = 0.f;
      inchunk = 0;
    }
  };
  if (!tripped) {
    const int L = len[i];
    for (int k = 0; k < L; k++) {
      const uint32_t e = list[(size_t)k * ld + i];
      visit(entry_index(e), entry_img(e, 0), entry_img(e, 1), entry_img(e, 2), (e >> 26) != 0);
    }
  } else {
    // skin exceeded: walk the full candidate row (the reference's row, same
    // order) and refresh this atom's compact row at the current positions
    const float4 pc = pi;
    int kept = 0;
    walk_row(w, pos, i, [&](int m, int ix, int iy, int iz) {
      visit(m, ix, iy, iz, w.g.periodic && (ix | iy | iz));
      const float4 pm = posf[m];
      const float dx = pc.x - (pm.x + (float)ix * w.g.box_f);
      const float dy = pc.y - (pm.y + (float)iy * w.g.box_f);
      const float dz = pc.z - (pm.z + (float)iz * w.g.box_f);
      if (dx * dx + dy * dy + dz * dz < rv2) {
        if (kept < cap) list[(size_t)kept * ld + i] = pack_entry(m, ix, iy, iz);
        kept++;
      }
    });
    if (kept > cap) atomicOr(&skin[3], 1);
    len[i] = kept < cap ? kept : cap;
    pos_build[i] = pc;
  }
  kahan(hx, lx, cx);
  kahan(hy, ly, cy);
  kahan(hz, lz, cz);
  f3[3 * i] = (double)hx - (double)lx;
  f3[3 * i + 1] = (double)hy - (double)ly;
  f3[3 * i + 2] = (double)hz - (double)lz;
}

// out-of-line copy of the tripped path for the TMA kernel (keeps its
// register allocation free of the rarely used full-row walk)
__device__ __noinline__ void lj32_atom_tripped(int i, const float4* posf, const md_double4* pos,
                                              double* f3, int ld, uint32_t* list, int* len,
                                              const RowWalker& w, int* skin, int cap, float rv2,
                                              float4* pos_build, double rcutsq,
                                              const Species& sp) {
  double ev[3];
  lj32_atom<false>(i, posf, pos, f3, ld, list, len, w, true, skin, cap, rv2, pos_build, rcutsq,
                   sp, ev);
}

template <bool ENERGY>
__global__ void __launch_bounds__(128)
    k_lj_fp32(const float4* __restrict__ posf, const md_double4* __restrict__ pos,
              double* __restrict__ f3, int n, int ld, uint32_t* __restrict__ list,
              int* __restrict__ len, RowWalker w, int* skin, SkinFlags sf, int cap, float rv2,
              float4* __restrict__ pos_build, double rcutsq, Species sp,
              double* __restrict__ epart, const int* __restrict__ run_if) {
  if (run_if && *run_if == 0) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double ev[3] = {0.0, 0.0, 0.0};
  const bool tripped = (skin[sf.read] | skin[3]) != 0;
  if (i < n)
    lj32_atom<ENERGY>(i, posf, pos, f3, ld, list, len, w, tripped, skin, cap, rv2, pos_build,
                      rcutsq, sp, ev);
  if (tripped && i == 0) atomicAdd(&skin[4], 1);
  if (i == 0) skin[sf.clear] = 0;  // the flag of step t + 2 starts clear
  if (ENERGY) block_partial<3>(ev, epart);
}

// The FP32 LJ force with the compact list streamed through shared memory by
// TMA: each block of 128 atoms walks its list in tiles of 16 slots x 128
// atoms (8 KB), double-buffered and synchronised with mbarriers, so that
// list traffic is bulk and in flight while the pairs of the previous tile
// are computed.  Positions are gathered through L1.  Each tile's FP32 sums
// are folded into a compensated (Kahan) FP32 pair.  ALL_NG: every atom is of
// the NG species (one parameter set, no type tests).
template <bool ALL_NG>
__global__ void __launch_bounds__(kListTileAtoms, 8)
    k_lj_tma(const __grid_constant__ CUtensorMap tmap, const float4* __restrict__ posf,
             const md_double4* __restrict__ pos, double* __restrict__ f3, int n, int ld,
             uint32_t* __restrict__ list, int* __restrict__ len, RowWalker w, int* skin,
             SkinFlags sf, int cap, float rv2, float4* __restrict__ pos_build, double rcutsq,
             Species sp, int* status, int wait_limit, const int* __restrict__ run_if) {
  if (run_if && *run_if == 0) return;  // the whole block
  __shared__ __align__(128) uint32_t tile[2][kListTileSlots][kListTileAtoms];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ int s_max[kListTileAtoms / 32];
  const int tid = threadIdx.x;
  const int i = blockIdx.x * kListTileAtoms + tid;
  const bool tripped = (skin[sf.read] | skin[3]) != 0;
  if (tripped) {
    if (i < n)
      lj32_atom_tripped(i, posf, pos, f3, ld, list, len, w, skin, cap, rv2, pos_build, rcutsq,
                        sp);
    if (i == 0) {
      atomicAdd(&skin[4], 1);
      skin[sf.clear] = 0;
    }
    return;
  }
  const int L = i < n ? len[i] : 0;
  int m = L;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((tid & 31) == 0) s_max[tid >> 5] = m;
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  int maxlen = s_max[0];
#pragma unroll
  for (int k = 1; k < kListTileAtoms / 32; k++) maxlen = max(maxlen, s_max[k]);
  const int T = (maxlen + kListTileSlots - 1) / kListTileSlots;
  constexpr uint32_t kTileBytes = kListTileSlots * kListTileAtoms * 4;
  const int x0 = blockIdx.x * kListTileAtoms;
  if (tid == 0) {
    for (int t = 0; t < 2 && t < T; t++) {
      mbar_expect_tx(&bar[t], kTileBytes);
      tma_load_2d(&tile[t][0][0], &tmap, x0, t * kListTileSlots, &bar[t]);
    }
  }
  const float4 pi = i < n ? posf[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const int ti = __float_as_int(pi.w);
  const float rc2 = (float)rcutsq;
  const float rc_lo = rc2 * (1.0f - 1e-5f), rc_hi = rc2 * (1.0f + 1e-5f);
  const float Lf = w.g.box_f, Llo = w.g.box_lo;
  // NG-NG parameters, and the two cross parameter sets for mixed systems
  const float s2_ng = sp.sig[2] * sp.sig[2], c_ng = 24.0f * sp.eps[2];
  const float s2_n = sp.sig[0] * sp.sig[0], c_n = 24.0f * sp.eps[0];
  const float s2_o = sp.sig[1] * sp.sig[1], c_o = 24.0f * sp.eps[1];
  float hx = 0.f, hy = 0.f, hz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
  bool ok = true;
  int failed_at = 0;
  for (int t = 0; t < T; t++) {
    const int b = t & 1;
    // the outcome is made block-uniform, so every thread leaves together
    if (!__syncthreads_and(mbar_wait(&bar[b], (uint32_t)((t >> 1) & 1), status, wait_limit))) {
      ok = false;
      failed_at = t;
      break;
    }
    const int kmax = min(kListTileSlots, L - t * kListTileSlots);
    float cx = 0.f, cy = 0.f, cz = 0.f;
    // every slot is evaluated by every lane (no divergence); slots past the
    // atom's row read the atom itself and contribute zero
#pragma unroll 4
    for (int kk = 0; kk < kListTileSlots; kk++) {
      const bool valid = kk < kmax;
      const uint32_t e = valid ? tile[b][kk][tid] : (uint32_t)(i < n ? i : 0);
      const int j = entry_index(e);
      const float4 pj = __ldg(&posf[j]);
      float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
      if (e >> 26) {  // periodic image (rare: boundary cells only)
        const float fx = (float)entry_img(e, 0), fy = (float)entry_img(e, 1),
                    fz = (float)entry_img(e, 2);
        dx = (pi.x - fmaf(fx, Lf, pj.x)) - fx * Llo;
        dy = (pi.y - fmaf(fy, Lf, pj.y)) - fy * Llo;
        dz = (pi.z - fmaf(fz, Lf, pj.z)) - fz * Llo;
      }
      const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      float s2 = s2_ng, c24 = c_ng;
      bool use = valid;
      if (!ALL_NG) {
        const int tj = __float_as_int(pj.w);
        use = use && (tj == SP_NG || ti == SP_NG);
        const int sel = lj_select(ti, tj);
        s2 = sel == SP_N ? s2_n : (sel == SP_O ? s2_o : s2_ng);
        c24 = sel == SP_N ? c_n : (sel == SP_O ? c_o : c_ng);
      }
      const float inv = rcp_approx(r2);
      const float sr2 = s2 * inv;
      const float sr6 = sr2 * sr2 * sr2;
      float fij = c24 * inv * sr6 * fmaf(2.0f, sr6, -1.0f);
      bool in = r2 <= rc_lo;
      if (use && !in && r2 < rc_hi)  // within 1e-5 of the cutoff: decide in FP64
        in = lj_inside(r2, rc_lo, rc_hi, pos, i, j, (e >> 26) != 0, entry_img(e, 0),
                       entry_img(e, 1), entry_img(e, 2), w.g, rcutsq);
      fij = (use && in) ? fij : 0.0f;
      cx = fmaf(dx, fij, cx);
      cy = fmaf(dy, fij, cy);
      cz = fmaf(dz, fij, cz);
    }
    kahan(hx, lx, cx);
    kahan(hy, ly, cy);
    kahan(hz, lz, cz);
    __syncthreads();  // everyone is done with buffer b
    if (tid == 0 && t + 2 < T) {
      fence_proxy_async();
      mbar_expect_tx(&bar[b], kTileBytes);
      tma_load_2d(&tile[b][0][0], &tmap, x0, (t + 2) * kListTileSlots, &bar[b]);
    }
  }
  if (!ok) {
    // tiles failed_at and failed_at + 1 may still be in flight: they land in
    // this block's shared memory before it leaves
    if (tid == 0)
      for (int t = failed_at; t < failed_at + 2 && t < T; t++)
        mbar_drain(&bar[t & 1], (uint32_t)((t >> 1) & 1), status);
    return;
  }
  if (i < n) {
    f3[3 * i] = (double)hx - (double)lx;
    f3[3 * i + 1] = (double)hy - (double)ly;
    f3[3 * i + 2] = (double)hz - (double)lz;
  }
  if (i == 0) skin[sf.clear] = 0;  // the flag of step t + 2 starts clear
}

// --------------------------------------------------------------- bond order
template <typename T>
struct PosT;
template <>
struct PosT<double> {
  static __device__ __forceinline__ void load(const md_double4* pos, const float4*, int j,
                                              double& x, double& y, double& z, int& t) {
    md_double4 p = pos[j];
    x = p.x;
    y = p.y;
    z = p.z;
    t = (int)p.w;
  }
  // image position: p + img * L, exactly as the oracle forms it
  static __device__ __forceinline__ void image(double& x, double& y, double& z, uint32_t e,
                                               const Grid& g) {
    if (e >> 26) image3(x, y, z, entry_img(e, 0), entry_img(e, 1), entry_img(e, 2), g);
  }
  static __device__ __forceinline__ void image3(double& x, double& y, double& z, int ix,
                                                int iy, int iz, const Grid& g) {
    x = xadd(x, (double)ix * g.box);
    y = xadd(y, (double)iy * g.box);
    z = xadd(z, (double)iz * g.box);
  }
};
template <>
struct PosT<float> {
  static __device__ __forceinline__ void load(const md_double4*, const float4* posf, int j,
                                              float& x, float& y, float& z, int& t) {
    float4 p = posf[j];
    x = p.x;
    y = p.y;
    z = p.z;
    t = __float_as_int(p.w);
  }
  static __device__ __forceinline__ void image(float& x, float& y, float& z, uint32_t e,
                                               const Grid& g) {
    if (e >> 26) image3(x, y, z, entry_img(e, 0), entry_img(e, 1), entry_img(e, 2), g);
  }
  static __device__ __forceinline__ void image3(float& x, float& y, float& z, int ix, int iy,
                                                int iz, const Grid& g) {
    x = fmaf((float)ix, g.box_f, x) + (float)ix * g.box_lo;
    y = fmaf((float)iy, g.box_f, y) + (float)iy * g.box_lo;
    z = fmaf((float)iz, g.box_f, z) + (float)iz * g.box_lo;
  }
};

// Short list: candidates within rcut at the current positions, row order.  A
// warp per atom, 32 candidates at a time (a ballot keeps the order).  FP64: a
// pair clear of the cutoff by more than the truncation of its FP32 copies
// needs no FP64 operation; the others, and in FP32 the pairs within 1e-5 of
// the cutoff, are decided in FP64.
template <typename T>
__global__ void __launch_bounds__(128)
    k_mb_short(const md_double4* __restrict__ pos, const float4* __restrict__ posf, int n,
               const uint32_t* __restrict__ list, size_t ri, size_t rk,
               const int* __restrict__ len, Grid g, double rcutsq, uint32_t* __restrict__ sl,
               size_t si, size_t ss, int* __restrict__ slen, const int* __restrict__ run_if) {
  grid_wait();
  grid_launch_dependents();
  if (run_if && *run_if == 0) return;  // the whole launch: a gated call with nothing to do
  constexpr bool k64 = sizeof(T) == 8;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= n) return;  // whole warp
  auto load = [&](int j) {
    if (!k64) return posf[j];
    const md_double4 p = pos[j];
    return make_float4(trunc32(p.x), trunc32(p.y), trunc32(p.z), 0.f);
  };
  const float4 pi = load(i);
  const float rc2 = (float)rcutsq;
  float band = 1e-5f * rc2;
  if (k64) {
    // each coordinate is off by less than 2^-23 of itself (k_lj_fp64's bound)
    const float rc = sqrtf(rc2) * 1.000001f;
    const float off =
        (fmaxf(fabsf(pi.x), fmaxf(fabsf(pi.y), fabsf(pi.z))) + fabsf(g.box_f) + rc) * 0x1p-20f;
    band += off * (8.0f * rc + 16.0f * off);
  }
  int cnt = 0;
  const int L = len[i];
  for (int k0 = 0; k0 < L; k0 += 32) {
    const int k = k0 + lane;
    bool keep = false;
    uint32_t e = 0;
    if (k < L) {
      e = list[(size_t)i * ri + (size_t)k * rk];
      const float4 pj = load(entry_index(e));
      float x = pj.x, y = pj.y, z = pj.z;
      PosT<float>::image(x, y, z, e, g);
      const float r2 = (pi.x - x) * (pi.x - x) + (pi.y - y) * (pi.y - y) + (pi.z - z) * (pi.z - z);
      keep = r2 < rc2;
      if (!(fabsf(r2 - rc2) >= band)) {  // near the cutoff, or not a number
        double a[3], b[3];
        int t0;
        PosT<double>::load(pos, posf, i, a[0], a[1], a[2], t0);
        PosT<double>::load(pos, posf, entry_index(e), b[0], b[1], b[2], t0);
        PosT<double>::image(b[0], b[1], b[2], e, g);
        keep = norm2_exact(xsub(a[0], b[0]), xsub(a[1], b[1]), xsub(a[2], b[2])) < rcutsq;
      }
    }
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    if (keep) sl[(size_t)i * si + (size_t)(cnt + __popc(mask & ((1u << lane) - 1u))) * ss] = e;
    cnt += __popc(mask);
  }
  if (lane == 0) slen[i] = cnt;
}

// common/arvdwfc.cpp:54-59, (1 - tanh x) / 2 as 1 / (1 + e^2x) and its
// derivative -ALFA (1 - tanh^2 x) / 2 = -2 ALFA fc (1 - fc)
__device__ __forceinline__ void mb_cutoff(double r, double& fc, double& dfc) {
  fc = rcp64(1.0 + exp64((double)(2.0f * MD_ALFA) * (r - (double)MD_R0)));
  const double t = (double)(2.0f * MD_ALFA) * fc;
  dfc = fma(t, fc, -t);
}

// the angular function and its derivative prefactor (angular in
// md_potential.cuh) from one reciprocal; MD_H is 0
__device__ __forceinline__ void mb_angular(double c, double& g, double& gpre) {
  static_assert(MD_H == 0.0f, "cos enters as H - cos");
  const double iq = rcp64(fma(c, c, (double)MD_D));
  const double h = (double)MD_C * iq;
  g = (double)(1.0f + MD_C / MD_D) - h;
  gpre = (h * iq) * (2.0 * c);
}

// Neighbours of the block's atom i (up to 32 of its short list), in shared
// memory: the vector r_i - r_s, the unit vector, the distance, its reciprocal
// and the cutoff; as the partner j of a bond the pair terms.
struct Nb {
  double d[3][32], u[3][32];
  q56 qu[3][32], qr[32], qir[32], qf[32], qh[32];  // fixed point (cutoffq's f and h)
  // bits 16 and up: cutoffq's n; bit 6: not a third body of i's bonds (NG), 7: not a bond (NG, or beyond
  // the pair cutoff), 8: its distance is outside the fixed point's range;
  // bits 0-2: in the cell below i's along x, y, z, 3-5: above
  int flag[32];
};
// pair terms: E, Va, Va', Vr' + Vdw', Vr + Vdw
struct NbPair {
  double E[32], va[32], dva[32], dv[32], v0[32];
};
constexpr int kNbNoThird = 64, kNbNoBond = 128, kNbFar = 256;

// squared distances that the fixed-point terms take (0.5 .. 8 angstrom; 16 between
// two neighbours)
__device__ __forceinline__ bool mb_in_range(double r2, double most) { return r2 >= 0.25 && r2 < most; }

// neighbour q by one thread
__device__ __forceinline__ void mb_stage(Nb& N, int q, uint32_t e, double xi, double yi, double zi,
                                         const md_double4* pos, const Grid& g, const int* cell3,
                                         int i) {
  const int j = entry_index(e);
  double x, y, z;
  int tj;
  PosT<double>::load(pos, nullptr, j, x, y, z, tj);
  PosT<double>::image(x, y, z, e, g);
  const double dx = xi - x, dy = yi - y, dz = zi - z;
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double ir = rsqrt64(r2);
  N.d[0][q] = dx, N.d[1][q] = dy, N.d[2][q] = dz;
  const double ux = dx * ir, uy = dy * ir, uz = dz * ir;
  N.u[0][q] = ux, N.u[1][q] = uy, N.u[2][q] = uz;
  int flag = tj == SP_NG ? kNbNoThird | kNbNoBond : 0;
  if (mb_in_range(r2, 64.0)) {
    q56 r, irq, f, h;
    int n;
    rsqrtq(r2, r, irq);
    N.qu[0][q] = toq(ux), N.qu[1][q] = toq(uy), N.qu[2][q] = toq(uz);
    N.qr[q] = r;
    N.qir[q] = irq;
    cutoffq(r, f, n, h);
    N.qf[q] = f;
    N.qh[q] = h;
    flag |= n << 16;
  } else {
    flag |= kNbFar;
  }
  if (r2 > (double)MD_CUTOFF_RIJSQ) flag |= kNbNoBond;
  if (cell3) {
    const int4 a = reinterpret_cast<const int4*>(cell3)[i],
               b = reinterpret_cast<const int4*>(cell3)[j];
    int s[3] = {b.x - a.x, b.y - a.y, b.z - a.z};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      if (g.periodic && s[d] > 1) s[d] -= g.cells;
      if (g.periodic && s[d] < -1) s[d] += g.cells;
      flag |= s[d] < 0 ? 1 << d : (s[d] > 0 ? 8 << d : 0);
    }
  }
  N.flag[q] = flag;
}

// its pair terms by a thread of another warp: common/arvdwfc.cpp:17-48 with the
// powers of one exponential
__device__ __forceinline__ void mb_stage_pair(NbPair& N, int q, uint32_t e, double xi, double yi,
                                              double zi, int ti, const md_double4* pos,
                                              const Grid& g) {
  double x, y, z;
  int tj;
  PosT<double>::load(pos, nullptr, entry_index(e), x, y, z, tj);
  PosT<double>::image(x, y, z, e, g);
  const double dx = xi - x, dy = yi - y, dz = zi - z;
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double r = root64(r2, rsqrt64(r2));
  const double de = get_de<double>(ti, tj), re = get_re<double>(ti, tj),
               beta = get_beta<double>(ti, tj);
  const double x1 = exp64(-beta * (r - re)), x2 = x1 * x1, x4 = x2 * x2;
  const double va = MD_S * de / (MD_S - 1.0f) * x1;
  const double vr = de / (MD_S - 1.0f) * x2 + 7.0e-8f * (x4 * x4 * x2);
  const double eplus = exp64(MD_ALFAV * (r - get_r0v<double>(ti, tj)));
  const double gmexp = MD_GM * rcp64(eplus);
  const double a = eplus + gmexp, b = MD_ALFAV * (eplus - gmexp), db = MD_ALFAVSQ * a;
  const double v = 1.0f + 50.0f * MD_GM + MD_GMSQ + 10.0f * (MD_GM - 1.0f) * b;
  const double ia = rcp64(a), ia2 = ia * ia;
  const double dvdw = -1.0e-4f * ((10.0f * (MD_GM - 1.0f) * db * a - 2.0f * b * v) * (ia2 * ia));
  N.E[q] = exp64((double)MD_LAMDA3 * (r - re));
  N.va[q] = va;
  N.dva[q] = beta * va;
  N.dv[q] = beta * 2.0f * vr + dvdw;
  N.v0[q] = vr + 1.0e-4f * v * ia2;
}

// What the angle terms of a bond i-j with the third body m give: the sums of
// the bond (x: sum of fc_im g_i, y: of its derivative along r_ij, both without
// the factor E; xj, yj the same for the angle at j) and the coefficients of
// the forces on m along u_im (a for the angle at i, b at j) and along
// r_j - r_m (p, q), each still without its bond's factor.
struct Angle {
  double x, y, xj, yj, a, b, p, q;
};
// in FP64, for distances outside the fixed point's range
__device__ __noinline__ Angle mb_angle_far(const Nb& J, int j, const Nb& M, int m) {
  const double vx = M.d[0][m] - J.d[0][j], vy = M.d[1][m] - J.d[1][j], vz = M.d[2][m] - J.d[2][j];
  const double r2 = vx * vx + vy * vy + vz * vz, irjm = rsqrt64(r2), rjm = root64(r2, irjm);
  const double rij2 = J.d[0][j] * J.d[0][j] + J.d[1][j] * J.d[1][j] + J.d[2][j] * J.d[2][j];
  const double rim2 = M.d[0][m] * M.d[0][m] + M.d[1][m] * M.d[1][m] + M.d[2][m] * M.d[2][m];
  const double irij = rsqrt64(rij2), rij = root64(rij2, irij);
  const double irim = rsqrt64(rim2), rim = root64(rim2, irim);
  double fi, dfi, fj, dfj, gi, pi, gj, pj;
  mb_cutoff(rim, fi, dfi);
  mb_cutoff(rjm, fj, dfj);
  // cosines of the angles at i (unit vectors) and at j (projection)
  const double ci = J.u[0][j] * M.u[0][m] + J.u[1][j] * M.u[1][m] + J.u[2][j] * M.u[2][m];
  const double cj = fma(-rim, ci, rij) * irjm;
  mb_angular(ci, gi, pi);
  mb_angular(cj, gj, pj);
  const double xi = fi * pi, xj = fj * pj;
  Angle A;
  A.x = fi * gi;
  A.y = xi * fma(-ci, irij, irim);
  A.xj = fj * gj;
  A.yj = xj * fma(-cj, irij, irjm);
  A.a = fma(xi, fma(-ci, irim, irij), dfi * gi);
  A.p = -xi * (irij * irim);
  A.b = -xj * (rim * irij) * irjm;
  A.q = fma(xj, fma(-cj, irjm, irij), dfj * gj) * irjm;
  return A;
}

// the same in fixed point; the sums stay there, (x, y) in si and (xj, yj) in sj.
// The cutoffs multiply last, so that each result keeps their power of two.
__device__ __forceinline__ void mb_angle_q(double r2, const Nb& J, int j, const Nb& M, int m,
                                           bool sums, SumQ& si, SumQ& sj, Angle& A) {
  const q56 rij = J.qr[j], irij = J.qir[j], rim = M.qr[m], irim = M.qir[m];
  const q56 fi = M.qf[m], hi = M.qh[m];
  const int ni = M.flag[m] >> 16;
  q56 rjm, irjm, fj, hj, gi, pi, gj, pj;
  int nj;
  rsqrtq(r2, rjm, irjm);
  cutoffq(rjm, fj, nj, hj);
  const q56 ci = dotq(J.qu[0][j], J.qu[1][j], J.qu[2][j], M.qu[0][m], M.qu[1][m], M.qu[2][m]);
  const q56 cj = mulq(rij - mulq(rim, ci), irjm);
  angularq(ci, gi, pi);
  angularq(cj, gj, pj);
  if (sums) {
    addq(si, mulq(fi, gi), mulq(fi, mulq(pi, irim - mulq(ci, irij))), ni);
    addq(sj, mulq(fj, gj), mulq(fj, mulq(pj, irjm - mulq(cj, irij))), nj);
  }
  A.a = fromq(mulq(fi, mulq(pi, irij - mulq(ci, irim)) - mulq(hi, gi)), ni);
  A.p = fromq(-mulq(fi, mulq(pi, mulq(irij, irim))), ni);
  A.b = fromq(-mulq(fj, mulq(mulq(pj, mulq(rim, irij)), irjm)), nj);
  A.q = fromq(mulq(fj, mulq(mulq(pj, irij - mulq(cj, irjm)) - mulq(hj, gj), irjm)), nj);
}

// columns of a warp's coefficient table: 34 keeps five blocks on an SM (36 would
// store without bank conflicts, but only four blocks fit)
constexpr int kMbPitch = 34;

// Sum of 4 values over the warp, each value to a quarter of the lanes: value
// ((lane >> 3) & 3) of every lane's v comes back in all lanes of that quarter
// (6 additions; 4 values by butterflies take 20).
__device__ __forceinline__ double quarter_sum(double v0, double v1, double v2, double v3,
                                              int lane) {
  const bool h = lane & 16, k = lane & 8;
  double a = h ? v2 : v0, b = h ? v3 : v1;
  a += __shfl_xor_sync(0xffffffffu, h ? v0 : v2, 16);
  b += __shfl_xor_sync(0xffffffffu, h ? v1 : v3, 16);
  double s = k ? b : a;
  s += __shfl_xor_sync(0xffffffffu, k ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// Bond-order forces of atom i, one block of four warps: BondOrderFuncs.h:12-143
// and 242-278 (the bonds i-j with the third bodies m of i) and, where the
// bonds' third bodies see j in their own candidate rows (the cells of the list
// build), :148-237 (the force on m), left in m's slot of i's short list for
// k_mb_gather.  A warp takes eight bonds at a time, four lanes to a bond, each
// every fourth m; the angle terms of a triplet are evaluated once: their sums
// give the bond, and the four force coefficients wait in shared memory until
// the bond's factors are known; then lane m adds over the eight bonds.  More
// than 32 neighbours take the triplets twice, in tiles of 32.
//
// The angle terms in FP64 (75 operations a triplet) kept the FP64 pipe 86% busy
// and everything else idle: 568 us for 4,096 atoms; in 64-bit fixed point
// (md_fixed64.cuh, 6 FP64 operations) 279 us, with the pair terms staged by a
// second warp and five blocks on an SM 265 us, and with the power of two that keeps
// small terms' bits, rounded products and exponentials to half a unit 293 us (FP64
// pipe 54%, issue 46%).
// SLOTS: with the engine's own rows; caller-supplied rows may lack symmetry,
// and k_mb_pass2 evaluates their third bodies.
template <bool ENERGY, bool SLOTS>
__global__ void __launch_bounds__(128, 5)
    k_mb_bonds(const md_double4* __restrict__ pos,
               double* __restrict__ f3, int n, const uint32_t* __restrict__ sl, int pitch,
               const int* __restrict__ slen, Grid g, const int* __restrict__ cell3, int ljexist,
               double* __restrict__ wi_s, double* __restrict__ wj_s, double* __restrict__ fslot,
               int slots, int* __restrict__ missing, double* __restrict__ epart,
               double* __restrict__ eatom, const int* __restrict__ run_if) {
  grid_wait();
  grid_launch_dependents();
  if (!ENERGY && run_if && *run_if == 0) return;
  __shared__ Nb NA, NB;
  __shared__ NbPair NP;
  __shared__ double table[4][4][8][kMbPitch];  // warp, coefficient, bond, m
  __shared__ double wsm[4][2][8];              // factors of the warp's bonds
  __shared__ double bsum[4][32];               // force of a bond, its energy
  const int i = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int jj = lane >> 2, quad = lane & 3;
  double xi, yi, zi;
  int ti;
  PosT<double>::load(pos, nullptr, i, xi, yi, zi, ti);
  const int S = slen[i];
  const uint32_t* row = sl + (size_t)i * pitch;
  double fx = 0, fy = 0, fz = 0;
  double energy = 0.0;
  int miss = 0;
  const bool once = S <= 32;
  for (int j0 = 0; j0 < S; j0 += 32) {
    __syncthreads();
    if (j0 + lane < S) {
      if (warp == 0) mb_stage(NA, lane, row[j0 + lane], xi, yi, zi, pos, g, cell3, i);
      if (warp == 1) mb_stage_pair(NP, lane, row[j0 + lane], xi, yi, zi, ti, pos, g);
    }
    __syncthreads();
    const int j = 8 * warp + jj;  // bond of this lane in the tile
    const bool bond = j0 + j < S && !(NA.flag[j & 31] & kNbNoBond);
    double x = 0, y = 0, xj = 0, yj = 0;
    SumQ si, sj;
    auto triplets = [&](const Nb& M, int m0, bool sums, bool store) {
      const int mn = min(32, S - m0);
      if (bond)
        for (int m = quad; m < mn; m += 4) {
          if (m0 + m == j0 + j) continue;
          const double vx = M.d[0][m] - NA.d[0][j], vy = M.d[1][m] - NA.d[1][j],
                       vz = M.d[2][m] - NA.d[2][j];
          const double r2 = vx * vx + vy * vy + vz * vz;
          const bool third = sums && !(M.flag[m] & kNbNoThird);
          Angle A;
          if (!((NA.flag[j] | M.flag[m]) & kNbFar) && mb_in_range(r2, 256.0)) {
            mb_angle_q(r2, NA, j, M, m, third, si, sj, A);
          } else {
            A = mb_angle_far(NA, j, M, m);
            if (third) {
              x += A.x;
              y += A.y;
              xj += A.xj;
              yj += A.yj;
            }
          }
          if (store) {
            table[warp][0][jj][m] = A.a;
            table[warp][1][jj][m] = A.b;
            table[warp][2][jj][m] = A.p;
            table[warp][3][jj][m] = A.q;
          }
        }
    };
    // the tile of third bodies at m0: the bonds' own tile or a second one
    auto tile = [&](int m0) -> const Nb& {
      if (m0 == j0) return NA;
      __syncthreads();
      if (tid < 32 && m0 + tid < S)
        mb_stage(NB, tid, row[m0 + tid], xi, yi, zi, pos, g, cell3, i);
      __syncthreads();
      return NB;
    };
    for (int m0 = 0; m0 < S; m0 += 32) {
      triplets(tile(m0), m0, true, once);
      // a lane's eight triplets of a tile stay below the fixed point's range
      x += fromq(si.x, si.n), y += fromq(si.y, si.n);
      xj += fromq(sj.x, sj.n), yj += fromq(sj.y, sj.n);
      si = sj = SumQ();
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
      xj += __shfl_xor_sync(0xffffffffu, xj, o);
      yj += __shfl_xor_sync(0xffffffffu, yj, o);
    }
    if (quad == 0 && j0 + j < S) {
      double wi = (double)NAN, wj = (double)NAN;
      if (bond) {
        const double E = NP.E[j], va = NP.va[j], lam = (double)MD_LAMDA3;
        const double bi = rcp64(fma(E, x, 1.0)), bj = rcp64(fma(E, xj, 1.0));
        const double pi = bi * bi * E, pj = bj * bj * E;  // E / (1 + xi)^2
        const double bo = 0.5 * (bi + bj);
        const double db = 0.5 * (pi * fma(lam, x, y) + pj * fma(lam, xj, yj));
        // what the third bodies need of this bond: va E / (4 (1 + xi)^2)
        wi = 0.25 * va * pi;
        wj = 0.25 * va * pj;
        const double f = NP.dv[j] - bo * NP.dva[j] - va * db;
        bsum[0][j] = f * NA.u[0][j];
        bsum[1][j] = f * NA.u[1][j];
        bsum[2][j] = f * NA.u[2][j];
        if (ENERGY) bsum[3][j] = 0.5 * (NP.v0[j] - bo * va);
      } else {
        bsum[0][j] = bsum[1][j] = bsum[2][j] = bsum[3][j] = 0.0;
      }
      wsm[warp][0][jj] = wi;
      wsm[warp][1][jj] = wj;
      wi_s[(size_t)i * pitch + j0 + j] = wi;
      wj_s[(size_t)i * pitch + j0 + j] = wj;
    }
    __syncwarp();
    for (int m0 = 0; m0 < S; m0 += 32) {
      const Nb& M = tile(m0);
      if (!once) triplets(M, m0, false, true);
      __syncwarp();
      // lane m: coefficients of this warp's bonds along u_im (c) and r_j - r_m
      double c = 0, cu = 0, s = 0, gx = 0, gy = 0, gz = 0;
      const int m = lane;
      if (m0 + m < S) {
        const int fm = M.flag[m];
        const int opposite = ((fm >> 3) & 7) | ((fm & 7) << 3);
#pragma unroll 1
        for (int b = 0; b < 8; b++) {
          const int jb = 8 * warp + b;
          if (j0 + jb >= S) break;
          if (m0 + m == j0 + jb) continue;
          // j and m on opposite sides of i's cell are no candidates of each other
          const bool seen = SLOTS && !(NA.flag[jb] & opposite);
          if (NA.flag[jb] & kNbNoBond) {
            // a third body beyond the slots counts its own (k_mb_gather)
            miss += seen && m0 + m < slots && NA.flag[jb] & kNbNoThird;
            continue;
          }
          const double wi = wsm[warp][0][b], wj = wsm[warp][1][b];
          const double ck = fma(wi, table[warp][0][b][m], wj * table[warp][1][b][m]);
          if (seen) {
            const double cv = fma(wi, table[warp][2][b][m], wj * table[warp][3][b][m]);
            c += ck;
            s += cv;
            gx = fma(-cv, NA.d[0][jb], gx);
            gy = fma(-cv, NA.d[1][jb], gy);
            gz = fma(-cv, NA.d[2][jb], gz);
          } else {
            cu += ck;
          }
        }
        // the warp's forces on m take the place of the coefficients that this
        // lane alone has read: x y z, c seen, c unseen
        table[warp][0][0][m] = fma(s, M.d[0][m], gx);
        table[warp][0][1][m] = fma(s, M.d[1][m], gy);
        table[warp][0][2][m] = fma(s, M.d[2][m], gz);
        table[warp][0][3][m] = c;
        table[warp][0][4][m] = cu;
      }
      __syncthreads();
      if (warp == 0 && m0 == j0 && j0 + lane < S) {
        fx += bsum[0][lane];
        fy += bsum[1][lane];
        fz += bsum[2][lane];
        if (ENERGY) energy += (double)bsum[3][lane];
      }
      if (warp == 0 && m0 + m < S) {
        double v[5];
#pragma unroll
        for (int d = 0; d < 5; d++)
          v[d] = (table[0][0][d][m] + table[1][0][d][m]) + (table[2][0][d][m] + table[3][0][d][m]);
        // the bond's own force: both ends of the angle's derivative along u_im
        if (!(M.flag[m] & kNbNoThird)) {
          const double w = -2.0 * (v[3] + v[4]);
          fx = fma(w, M.u[0][m], fx);
          fy = fma(w, M.u[1][m], fy);
          fz = fma(w, M.u[2][m], fz);
        }
        if (SLOTS && m0 + m < slots) {
          double* o = fslot + 3 * ((size_t)i * slots + m0 + m);
          const double ox = fma(v[3], M.u[0][m], v[0]), oy = fma(v[3], M.u[1][m], v[1]),
                  oz = fma(v[3], M.u[2][m], v[2]);
          o[0] = j0 ? o[0] + ox : ox;
          o[1] = j0 ? o[1] + oy : oy;
          o[2] = j0 ? o[2] + oz : oz;
        }
      }
      __syncthreads();
    }
  }
  if (SLOTS) {
    const int mw = __reduce_add_sync(0xffffffffu, miss);
    if (lane == 0 && mw) atomicAdd(missing, mw);
  }
  if (warp != 0) return;
  // the force on i, from warp 0's lanes
  const double q = quarter_sum(fx, fy, fz, energy, lane);
  const double v = __shfl_sync(0xffffffffu, q, (lane & 3) * 8);
  if (tid < 4) {
    if (tid < 3) {
      const size_t o = 3 * (size_t)i + tid;
      f3[o] = ljexist ? f3[o] + v : v;
    } else if (ENERGY) {
      // per-atom share: sum over j of 1/2 (Vr - b Va + Vdw) (the i-sum of
      // common/DebugCalculations.cpp:129-270 restricted to the force's pairs)
      if (eatom) eatom[i] = v;
      epart[2 * (size_t)i] = v;
    }
    if (ENERGY) {
      const double* p = (const double*)&pos[i];
      double w = tid < 3 ? p[tid] * v : 0.0;
      w += __shfl_xor_sync(0xfu, w, 1);
      w += __shfl_xor_sync(0xfu, w, 2);
      if (tid == 0) epart[2 * (size_t)i + 1] = w;
    }
  }
}

// the part of pass 2 for one pair (i, j) of the warp's atom k: i at (x, y, z)
// with its k-side terms, j = entry sl[q]; adds -F_k to (fx, fy, fz)
template <typename T>
struct Pass2I {
  T x, y, z, r, ir, fc, dfc, ux, uy, uz;
  int id;
};

// r and 1/r from r^2: one rsqrt in FP32; the square root and a quotient in FP64
template <typename T>
__device__ __forceinline__ void dist_recip(T r2, T& r, T& ir) {
  if constexpr (std::is_same<T, float>::value) {
    ir = rsqrtf(r2);
    r = r2 * ir;
  } else {
    r = md_sqrt(r2);
    ir = fdiv<T>(1.0, r);
  }
}

template <typename T>
__device__ __forceinline__ void pass2_pair(const Pass2I<T>& I, size_t q, int k, T xk, T yk, T zk,
                                           const md_double4* pos, const float4* posf,
                                           const uint32_t* sl, const Grid& g, const int* cell3,
                                           const int* ref_rows, int ref_nls, int ref_nlargest,
                                           T rc2, T cut_rijsq, const T* wi_s, const T* wj_s,
                                           T& fx, T& fy, T& fz, int& miss) {
  const int jp = entry_index(sl[q]);
  if (jp == k) return;
  int im[3] = {0, 0, 0};
  if (ref_rows) {
    // caller-supplied rows (no periodic box): is jp in row k?
    const int* row = ref_rows + (size_t)k * ref_nls;
    bool found = false;
    for (int q2 = 0; q2 < ref_nlargest && row[q2] != -1; q2++)
      if (row[q2] == jp) {
        found = true;
        break;
      }
    if (!found) return;
  } else if (!in_row(cell3, g, k, jp, im)) {
    return;
  }
  // j at its image in k's row, as BondOrderFuncs.h:367-369 sees it
  T xj, yj, zj;
  int tj;
  PosT<T>::load(pos, posf, jp, xj, yj, zj, tj);
  if (im[0] | im[1] | im[2]) PosT<T>::image3(xj, yj, zj, im[0], im[1], im[2], g);
  const T ijx = I.x - xj, ijy = I.y - yj, ijz = I.z - zj;
  const T r2ij = ijx * ijx + ijy * ijy + ijz * ijz;
  if (r2ij >= rc2 || r2ij > cut_rijsq) return;
  const T wi = wi_s[q], wj = wj_s[q];
  if (wi != wi || tj == SP_NG) {
    miss++;
    return;
  }
  T rij, irij, rjk, irjk;
  dist_recip<T>(r2ij, rij, irij);
  const T half_irij = (T)0.5 * irij;
  const T jkx = xj - xk, jky = yj - yk, jkz = zj - zk;
  dist_recip<T>(jkx * jkx + jky * jky + jkz * jkz, rjk, irjk);
  const T drjkx = -jkx * irjk, drjky = -jky * irjk, drjkz = -jkz * irjk;
  T fcj, dfcj;
  cutoff<T>(rjk, fcj, dfcj);
  T ck = 0, cj = 0;  // coefficients of d_ik and d_jk in -F_k
  if (I.fc > 0) {
    // d cos / d r_k = drik (1/rij - cos/rik) - drjk rjk / (rij rik)
    const T icos = (rij * rij + I.r * I.r - rjk * rjk) * half_irij * I.ir;
    T gth, gpre;
    angular1<T>(icos, gth, gpre);
    ck = wi * (I.dfc * gth + I.fc * gpre * (irij - icos * I.ir));
    cj = -wi * I.fc * gpre * rjk * irij * I.ir;
  }
  if (fcj > 0) {
    // d cos / d r_k = drjk (1/rij - cos/rjk) - drik rik / (rij rjk)
    const T jcos = (rij * rij + rjk * rjk - I.r * I.r) * half_irij * irjk;
    T gth, gpre;
    angular1<T>(jcos, gth, gpre);
    cj = fma(wj, dfcj * gth + fcj * gpre * (irij - jcos * irjk), cj);
    ck = fma(-wj * fcj * gpre, I.r * irij * irjk, ck);
  }
  fx -= fma(I.ux, ck, drjkx * cj);
  fy -= fma(I.uy, ck, drjky * cj);
  fz -= fma(I.uz, ck, drjkz * cj);
}

template <typename T>
__device__ __forceinline__ Pass2I<T> pass2_entry(uint32_t ei, T xk, T yk, T zk,
                                                 const md_double4* pos, const float4* posf,
                                                 const Grid& g) {
  Pass2I<T> I;
  I.id = entry_index(ei);
  int ti;
  PosT<T>::load(pos, posf, I.id, I.x, I.y, I.z, ti);
  PosT<T>::image(I.x, I.y, I.z, ei, g);
  const T ikx = xk - I.x, iky = yk - I.y, ikz = zk - I.z;
  dist_recip<T>(ikx * ikx + iky * iky + ikz * ikz, I.r, I.ir);
  cutoff<T>(I.r, I.fc, I.dfc);
  I.ux = ikx * I.ir;
  I.uy = iky * I.ir;
  I.uz = ikz * I.ir;
  return I;
}

// Pass 2 (BondOrderFuncs.h:148-237 bondOrder2 for every pair i-j with k as
// third body) for caller-supplied rows, which may name i in k's row and not k
// in i's: one warp per atom k, one entry i of k's short list per lane.  Per
// pair, k_mb_bonds left va E / (4 (1 + xi_ij)^2) and va E / (4 (1 + xi_ji)^2)
// in the slot (NaN where it evaluated none: counted as missing, no force).
__global__ void __launch_bounds__(128)
    k_mb_pass2(const md_double4* __restrict__ pos, double* __restrict__ f3, int n,
               const uint32_t* __restrict__ sl, int pitch, const int* __restrict__ slen, Grid g,
               const int* __restrict__ ref_rows, int ref_nls, int ref_nlargest, double rcutsq,
               const double* __restrict__ wi_s, const double* __restrict__ wj_s,
               int* __restrict__ missing) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = blockIdx.x * 4 + warp;
  if (k >= n) return;
  const md_double4 pk = pos[k];
  const int Sk = slen[k];
  double fx = 0, fy = 0, fz = 0;
  int miss = 0;
  for (int s = lane; s < Sk; s += 32) {
    const Pass2I<double> I = pass2_entry<double>(sl[(size_t)k * pitch + s], pk.x, pk.y, pk.z, pos,
                                                 nullptr, g);
    const int Si = slen[I.id];
    for (int sj = 0; sj < Si; sj++)
      pass2_pair<double>(I, (size_t)I.id * pitch + sj, k, pk.x, pk.y, pk.z, pos, nullptr, sl, g,
                         nullptr, ref_rows, ref_nls, ref_nlargest, rcutsq,
                         (double)MD_CUTOFF_RIJSQ, wi_s, wj_s, fx, fy, fz, miss);
  }
  const double v = quarter_sum(fx, fy, fz, 0.0, lane);
  if ((lane & 7) == 0 && lane < 24) f3[3 * (size_t)k + (lane >> 3)] += v;
  const int m = __reduce_add_sync(0xffffffffu, miss);
  if (lane == 0 && m) atomicAdd(missing, m);
}

// The forces on k as the third body of its neighbours' bonds (BondOrderFuncs.h:
// 339-393): one warp per atom k, a neighbour i per lane, which finds k in i's
// short list and takes the force k_mb_bonds left there.  Rows of the engine are
// symmetric up to the last bit of a distance at the cutoff and the reference's
// cells at the edge of its box; where k is missing in i's list (or beyond the
// slots), the lane evaluates i's bonds itself.
template <bool ENERGY>
__global__ void __launch_bounds__(128)
    k_mb_gather(const md_double4* __restrict__ pos, const float4* __restrict__ posf,
                double* __restrict__ f3, int n, const uint32_t* __restrict__ sl, int pitch,
                const int* __restrict__ slen, Grid g, const int* __restrict__ cell3,
                double rcutsq, const double* __restrict__ wi_s, const double* __restrict__ wj_s,
                const double* __restrict__ fslot, int slots, int* __restrict__ missing,
                double* __restrict__ epart, const int* __restrict__ run_if) {
  grid_wait();
  grid_launch_dependents();
  if (!ENERGY && run_if && *run_if == 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = blockIdx.x * 4 + warp;
  if (k >= n) return;
  const int Sk = slen[k];
  double fx = 0, fy = 0, fz = 0;
  int miss = 0;
  for (int s = lane; s < Sk; s += 32) {
    const uint32_t e = sl[(size_t)k * pitch + s];
    const int i = entry_index(e);
    const int Si = slen[i], lim = min(Si, slots);
    const uint4* row = reinterpret_cast<const uint4*>(sl + (size_t)i * pitch);
    int q = -1;
    for (int q0 = 0; q0 < lim && q < 0; q0 += 4) {  // pitch is a multiple of 4
      const uint4 w = row[q0 >> 2];
      if (entry_index(w.w) == k) q = q0 + 3;
      if (entry_index(w.z) == k) q = q0 + 2;
      if (entry_index(w.y) == k) q = q0 + 1;
      if (entry_index(w.x) == k) q = q0;
    }
    if (q >= 0 && q < lim) {
      const double* o = fslot + 3 * ((size_t)i * slots + q);
      fx += o[0];
      fy += o[1];
      fz += o[2];
    } else {
      double xk, yk, zk;
      int tk;
      PosT<double>::load(pos, posf, k, xk, yk, zk, tk);
      const Pass2I<double> I = pass2_entry<double>(e, xk, yk, zk, pos, posf, g);
      for (int sj = 0; sj < Si; sj++)
        pass2_pair<double>(I, (size_t)i * pitch + sj, k, xk, yk, zk, pos, posf, sl, g, cell3, nullptr,
                      0, 0, rcutsq, (double)MD_CUTOFF_RIJSQ, wi_s, wj_s, fx, fy, fz, miss);
    }
  }
  const double v = quarter_sum(fx, fy, fz, 0.0, lane);
  const int c = lane >> 3;
  if ((lane & 7) == 0 && c < 3) f3[3 * (size_t)k + c] += v;
  const int m = __reduce_add_sync(0xffffffffu, miss);
  if (lane == 0 && m) atomicAdd(missing, m);
  if (ENERGY) {
    double w = c < 3 ? ((const double*)&pos[k])[c] * v : 0.0;
    w += __shfl_xor_sync(0xffffffffu, w, 8);
    w += __shfl_xor_sync(0xffffffffu, w, 16);
    if (lane == 0) epart[k] = w;
  }
}

// ---- the precision form: pass 1 and pass 2 ----
// The order and the roundings of these FP32 sums are part of the form's results:
// the bond order jumps by 1e-3 of a force where a pair passes the cutoff, so two
// runs that differ in the last FP32 bit part once a pair crosses it a step earlier
// in one of them.  k_mb_bonds in FP32 took 228 us per evaluation of 32,768 atoms
// against 420 here, but after 50 steps at 900 K its velocities differed from the
// present ones by up to 1e-2 of their size for 45% of the seeds, by 1e-6 for the
// others; so the passes and their bits stay.

// Third bodies m of the warp's atom i (pass 1): what depends on i and m
// only, computed once per warp instead of once per pair i-j.
constexpr int kThirdMax = 64;
struct ThirdSm {
  float x[kThirdMax], y[kThirdMax], z[kThirdMax];  // position at its image
  float r[kThirdMax], ir[kThirdMax], fc[kThirdMax], dfc[kThirdMax];  // r_im, 1 / r_im
  float ux[kThirdMax], uy[kThirdMax], uz[kThirdMax];                // (r_i - r_m) / r_im
  int id[kThirdMax];                                            // atom, -1 for an NG atom
};

// 64 registers without spills, 8 blocks per SM instead of 7
template <bool ENERGY>
__global__ void __launch_bounds__(128, 8)
    k_mb_pass1_32(const md_double4* __restrict__ pos, const float4* __restrict__ posf,
               double* __restrict__ f3, int n, const uint32_t* __restrict__ sl,
               const int* __restrict__ slen, Grid g, int ljexist, float* __restrict__ xsi_s,
               float* __restrict__ xsj_s, double* __restrict__ epart,
               double* __restrict__ eatom, const int* __restrict__ run_if) {
  grid_wait();
  grid_launch_dependents();
  if (!ENERGY && run_if && *run_if == 0) return;
  const int warps = blockDim.x >> 5;
  const int i = blockIdx.x * warps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  using T = float;
  double ev[2] = {0.0, 0.0};
  __shared__ ThirdSm third_sm[4];
  ThirdSm& TS = third_sm[(threadIdx.x >> 5) & 3];
  if (i < n) {
    T xi, yi, zi;
    int ti;
    PosT<T>::load(pos, posf, i, xi, yi, zi, ti);
    const int S = slen[i];
    T fx = 0, fy = 0, fz = 0;
    const T cut_rijsq = (T)MD_CUTOFF_RIJSQ;
    const T nanv = (T)NAN;
    const bool staged = S <= kThirdMax && blockDim.x <= 128;  // warp-uniform
    if (staged) {
      for (int m = lane; m < S; m += 32) {
        const uint32_t em = sl[(size_t)m * n + i];
        const int mp = entry_index(em);
        T xm, ym, zm;
        int tm;
        PosT<T>::load(pos, posf, mp, xm, ym, zm, tm);
        PosT<T>::image(xm, ym, zm, em, g);
        TS.id[m] = tm == SP_NG ? -1 : mp;
        TS.x[m] = xm;
        TS.y[m] = ym;
        TS.z[m] = zm;
        const float imx = xi - xm, imy = yi - ym, imz = zi - zm;
        const float r2 = imx * imx + imy * imy + imz * imz;
        const float irim = rsqrtf(r2), rim = r2 * irim;
        float fci, dfci;
        cutoff<float>(rim, fci, dfci);
        TS.r[m] = rim;
        TS.ir[m] = irim;
        TS.fc[m] = fci;
        TS.dfc[m] = dfci;
        TS.ux[m] = imx * irim;
        TS.uy[m] = imy * irim;
        TS.uz[m] = imz * irim;
      }
      __syncwarp();
    }
    for (int s = lane; s < S; s += 32) {
      const uint32_t e = sl[(size_t)s * n + i];
      const int j = entry_index(e);
      T xj, yj, zj;
      int tj;
      PosT<T>::load(pos, posf, j, xj, yj, zj, tj);
      PosT<T>::image(xj, yj, zj, e, g);
      const size_t slot = (size_t)s * n + i;
      const T ijx = xi - xj, ijy = yi - yj, ijz = zi - zj;
      T rij = ijx * ijx + ijy * ijy + ijz * ijz;
      if (tj == SP_NG || rij > cut_rijsq) {
        xsi_s[slot] = nanv;
        xsj_s[slot] = nanv;
        continue;
      }
      rij = md_sqrt(rij);
      // BondOrderFuncs.h:242-278 bondForces
      T va = 0, dva = 0, vr = 0, dvr = 0, vdw, dvdw, bo = 0;
      T dbx = 0, dby = 0, dbz = 0;
      T fcut, dfcut;
      cutoff<T>(fdiv<T>(rij, 10), fcut, dfcut);
      T xs_i = nanv, xs_j = nanv;
      if (fcut > 0) {
        const T de = get_de<T>(ti, tj), re = get_re<T>(ti, tj), beta = get_beta<T>(ti, tj);
        attractive<T>(va, dva, rij, de, beta, re);
        repulsive<T>(vr, dvr, rij, de, beta, re);
        // BondOrderFuncs.h:12-143 bondOrder1
        const T drijx = fdiv<T>(ijx, rij), drijy = fdiv<T>(ijy, rij), drijz = fdiv<T>(ijz, rij);
        const T E = md_exp((T)MD_LAMDA3 * (rij - re));
        const T inv_rij = fdiv<T>(1.0f, rij), half_inv_rij = 0.5f * inv_rij;
        T xsi = 0, xsj = 0;
        T dxsix = 0, dxsiy = 0, dxsiz = 0, dxsjx = 0, dxsjy = 0, dxsjz = 0;
        for (int m = 0; m < S; m++) {
          T xm, ym, zm, rim, inv_rim, fci, dfci, drimx, drimy, drimz;
          if (staged) {
            const int mp = TS.id[m];
            if (mp < 0 || mp == j) continue;
            xm = TS.x[m];
            ym = TS.y[m];
            zm = TS.z[m];
            rim = TS.r[m];
            inv_rim = TS.ir[m];
            fci = TS.fc[m];
            dfci = TS.dfc[m];
            drimx = TS.ux[m];
            drimy = TS.uy[m];
            drimz = TS.uz[m];
          } else {
            const uint32_t em = sl[(size_t)m * n + i];
            const int mp = entry_index(em);
            int tm;
            PosT<T>::load(pos, posf, mp, xm, ym, zm, tm);
            if (tm == SP_NG || mp == j) continue;
            PosT<T>::image(xm, ym, zm, em, g);
            const T imx = xi - xm, imy = yi - ym, imz = zi - zm;
            rim = md_sqrt(imx * imx + imy * imy + imz * imz);
            cutoff<T>(rim, fci, dfci);
            drimx = fdiv<T>(imx, rim);
            drimy = fdiv<T>(imy, rim);
            drimz = fdiv<T>(imz, rim);
            inv_rim = fdiv<T>(1.0f, rim);
          }
          const T jmx = xj - xm, jmy = yj - ym, jmz = zj - zm;
          T rjm, inv_rjm = 0;
          {  // the distance and its reciprocal from one rsqrt
            const float r2 = (float)(jmx * jmx + jmy * jmy + jmz * jmz);
            const float ir = rsqrtf(r2);
            inv_rjm = ir;
            rjm = r2 * ir;
          }
          T fcj, dfcj;
          cutoff<T>(rjm, fcj, dfcj);
          if (fci > 0) {
            // d cos / d r_i = drij (1/rim - cos/rij) + drim (1/rij - cos/rim): the
            // reference's quotient per component (BondOrderFuncs.h) in two scalars
            const T num2 = rij * rij + rim * rim - rjm * rjm;
            const T icos = num2 * half_inv_rij * inv_rim;
            T gth, gpre;
            angular1<T>(icos, gth, gpre);
            xsi += fci * gth * E;
            const T fE = fci * E;
            const T cm = dfci * gth * E + fE * gpre * (inv_rij - icos * inv_rim);
            const T cj = fE * (gpre * (inv_rim - icos * inv_rij) + gth * (T)MD_LAMDA3);
            dxsix = fma(drimx, cm, fma(drijx, cj, dxsix));
            dxsiy = fma(drimy, cm, fma(drijy, cj, dxsiy));
            dxsiz = fma(drimz, cm, fma(drijz, cj, dxsiz));
          }
          if (fcj > 0) {
            // d cos / d r_i = drij (1/rjm - cos/rij) - drim rim / (rij rjm)
            const T num2 = rij * rij + rjm * rjm - rim * rim;
            const T jcos = num2 * half_inv_rij * inv_rjm;
            T gth, gpre;
            angular1<T>(jcos, gth, gpre);
            xsj += fcj * gth * E;
            const T fE = fcj * E;
            const T cj = fE * (gpre * (inv_rjm - jcos * inv_rij) + (T)MD_LAMDA3 * gth);
            const T cm = -fE * gpre * rim * inv_rij * inv_rjm;
            dxsjx = fma(drijx, cj, fma(drimx, cm, dxsjx));
            dxsjy = fma(drijy, cj, fma(drimy, cm, dxsjy));
            dxsjz = fma(drijz, cj, fma(drimz, cm, dxsjz));
          }
        }
        xs_i = xsi;
        xs_j = xsj;
        const T bij = fdiv<T>(1.0f, 1.0f + xsi), pbi = fdiv<T>(1.0f, (1.0f + xsi) * (1.0f + xsi));
        const T bji = fdiv<T>(1.0f, 1.0f + xsj), pbj = fdiv<T>(1.0f, (1.0f + xsj) * (1.0f + xsj));
        bo = 0.5f * (bij + bji);
        dbx = 0.5f * (pbi * dxsix + pbj * dxsjx);
        dby = 0.5f * (pbi * dxsiy + pbj * dxsjy);
        dbz = 0.5f * (pbi * dxsiz + pbj * dxsjz);
        // what pass 2 needs of this pair: va E / (4 (1 + xi)^2) for either
        // end (its force is -factor x the derivative of the angle terms)
        xs_i = (T)0.25 * va * E * pbi;
        xs_j = (T)0.25 * va * E * pbj;
      }
      xsi_s[slot] = xs_i;
      xsj_s[slot] = xs_j;
      vander_waals<T>(vdw, dvdw, rij, get_r0v<T>(ti, tj));
      const T fij = dvr - bo * dva + dvdw;
      fx += fdiv<T>(fij * ijx, rij) - dbx * va;
      fy += fdiv<T>(fij * ijy, rij) - dby * va;
      fz += fdiv<T>(fij * ijz, rij) - dbz * va;
      if (ENERGY) ev[0] += (double)(0.5f * ((vr - bo * va) + vdw));
    }
    double sx = warp_sum((double)fx), sy = warp_sum((double)fy), sz = warp_sum((double)fz);
    if (ENERGY && eatom) {
      // per-atom share: sum over j of 1/2 (Vr - b Va + Vdw) (the i-sum of
      // common/DebugCalculations.cpp:129-270 restricted to the force's pairs)
      const double ei = warp_sum(ev[0]);
      if (lane == 0) eatom[i] = ei;
    }
    if (lane == 0) {
      if (ljexist) {
        f3[3 * i] += sx;
        f3[3 * i + 1] += sy;
        f3[3 * i + 2] += sz;
      } else {
        f3[3 * i] = sx;
        f3[3 * i + 1] = sy;
        f3[3 * i + 2] = sz;
      }
      if (ENERGY) {
        const md_double4 p = pos[i];
        ev[1] = p.x * sx + p.y * sy + p.z * sz;
      }
    }
  }
  if (ENERGY) block_partial<2>(ev, epart);
}

// Pass 2 of the precision form: one warp per atom k, one entry i of k's short
// list per lane, over i's bonds i-j; 40 registers, 12 blocks per SM instead of
// 10.  (Spreading the bonds of k over all 32 lanes was measured slower, 348
// against 249 us on 32,768 atoms: lanes of one i read 32 different lines of the
// slot arrays, where lanes of neighbouring i, stored side by side, share
// sectors.)  ref_rows is NULL here; it stays an argument because without the
// branch the compiler fuses other products into FMAs, which moves the last bit.
template <bool ENERGY>
__global__ void __launch_bounds__(128, 12)
    k_mb_pass2_32(const md_double4* __restrict__ pos, const float4* __restrict__ posf,
               double* __restrict__ f3, int n, const uint32_t* __restrict__ sl,
               const int* __restrict__ slen, Grid g, const int* __restrict__ cell3,
               const int* __restrict__ ref_rows, int ref_nls, int ref_nlargest, double rcutsq,
               const float* __restrict__ wi_s, const float* __restrict__ wj_s,
               int* __restrict__ missing, double* __restrict__ epart,
               const int* __restrict__ run_if) {
  grid_wait();
  grid_launch_dependents();
  if (!ENERGY && run_if && *run_if == 0) return;
  using T = float;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = blockIdx.x * 4 + warp;
  double ev[1] = {0.0};
  if (k < n) {
    T xk, yk, zk;
    int tk;
    PosT<T>::load(pos, posf, k, xk, yk, zk, tk);
    const int Sk = slen[k];
    const T rc2 = (T)rcutsq, cut_rijsq = (T)MD_CUTOFF_RIJSQ;
    T fx = 0, fy = 0, fz = 0;
    int miss = 0;
    for (int s = lane; s < Sk; s += 32) {
      const Pass2I<T> I = pass2_entry<T>(sl[(size_t)s * n + k], xk, yk, zk, pos, posf, g);
      const int Si = slen[I.id];
      for (int sj = 0; sj < Si; sj++)
        pass2_pair<T>(I, (size_t)sj * n + I.id, k, xk, yk, zk, pos, posf, sl, g, cell3,
                      ref_rows, ref_nls, ref_nlargest, rc2, cut_rijsq, wi_s, wj_s, fx, fy, fz,
                      miss);
    }
    const double sx = warp_sum((double)fx), sy = warp_sum((double)fy), sz = warp_sum((double)fz);
    const int m = __reduce_add_sync(0xffffffffu, miss);
    if (lane == 0) {
      f3[3 * k] += sx;
      f3[3 * k + 1] += sy;
      f3[3 * k + 2] += sz;
      if (m) atomicAdd(missing, m);
      if (ENERGY) {
        const md_double4 p = pos[k];
        ev[0] = p.x * sx + p.y * sy + p.z * sz;
      }
    }
  }
  if (ENERGY) block_partial<1>(ev, epart);
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

// Lanes per atom of the FP64 LJ kernel.  More lanes shorten an atom's chain of
// pairs, but its ordered sums keep three of them and its last batch leaves the
// others idle, so the lines lie where more warps stop helping: at 5 (32 lanes),
// 8.5 (16) and 21 warps (8) an SM.  Measured, ms per 100 steps in a periodic box
// (640, 1,700, 2,432 atoms: within walls) with 32 / 16 / 8 / 4 lanes:
//    640 atoms  2.39 2.54 3.29 4.91     2,432  4.12 3.53 3.55 5.05
//    864        2.46 2.37 3.17 4.91     2,916  4.17 3.77 3.75 5.04
//  1,372        3.08 2.95 3.29 4.94     6,912  7.97 5.67 4.65 6.02
//  1,700        4.55 4.30 4.62 6.31    13,500  13.9 9.59 6.95 6.83
// (a thread per atom with the FP64 instructions: 20.5 at 864 to 8,000 atoms).
static int lj64_lanes(int n) {
  return n <= 5 * kSms ? 32 : (n <= 17 * kSms ? 16 : (n <= 85 * kSms ? 8 : 4));
}

template <int G>
static void launch_lj64_g(const Lj64Args& k, int mode, bool energy, cudaStream_t st) {
  const int B = nblk((long long)k.n * G, 128);
  // Blocks that wait early keep their places, and a grid of about one wave then
  // lies unevenly on the SMs: 100 steps of 8,000 atoms within walls took 6.2 ms
  // with early launches and 5.1 without; at 172 atoms they save a sixth.
  if (mode == LJ64_STEP)
    launch_dependent(B <= 2 * kSms, k_lj_fp64<G, LJ64_STEP, false>, B, 128, st, k);
  else if (mode == LJ64_REDO)
    launch_dependent(B <= 2 * kSms, k_lj_fp64<G, LJ64_REDO, false>, B, 128, st, k);
  else if (energy)
    launch_dependent(B <= 2 * kSms, k_lj_fp64<G, LJ64_FORCE, true>, B, 128, st, k);
  else
    launch_dependent(B <= 2 * kSms, k_lj_fp64<G, LJ64_FORCE, false>, B, 128, st, k);
}

static void launch_lj64(const ForceArgs& a, int mode, bool energy, cudaStream_t st) {
  Lj64Args k{};
  k.pos = a.pos;
  k.f3 = a.f3;
  k.n = a.n;
  k.ld = a.ld;
  k.list = a.list;
  k.len = a.len;
  k.w = a.walker;
  k.skin = a.skin;
  k.sf = a.sf;
  k.cap = a.cap;
  k.rv2 = a.rv2;
  k.pos_build = a.pos_build;
  k.rcutsq = a.rcutsq;
  k.c = lj_pair_const(a.sp, a.rcutsq);
  k.epart = energy ? a.epart : nullptr;
  k.run_if = energy ? nullptr : a.run_if;
  if (mode != LJ64_FORCE) {
    k.g = *a.gear64;
    k.hits = a.hits;
    k.flag_next = a.flag_next;
    k.store = a.f3 != nullptr;
  }
  switch (lj64_lanes(a.n)) {
    case 32: launch_lj64_g<32>(k, mode, energy, st); break;
    case 16: launch_lj64_g<16>(k, mode, energy, st); break;
    case 8: launch_lj64_g<8>(k, mode, energy, st); break;
    default: launch_lj64_g<4>(k, mode, energy, st);
  }
}

void launch_lj_step64(const ForceArgs& a, cudaStream_t st) {
  if (a.n > 0) launch_lj64(a, LJ64_STEP, false, st);
}

void launch_lj_redo64(const ForceArgs& a, cudaStream_t st) {
  if (a.n > 0) launch_lj64(a, LJ64_REDO, false, st);
}

void launch_lj(const ForceArgs& a, bool fp32, bool energy, cudaStream_t st) {
  const int T = 128;
  const int B = nblk(a.n, T);
  if (B == 0) return;
  if (!fp32) {
    launch_lj64(a, LJ64_FORCE, energy, st);
  } else if (!energy && a.tmap) {
    const int TB = nblk(a.n, kListTileAtoms);
    if (a.all_ng)
      k_lj_tma<true><<<TB, kListTileAtoms, 0, st>>>(*a.tmap, a.posf, a.pos, a.f3, a.n, a.ld,
                                                    a.list, a.len, a.walker, a.skin, a.sf,
                                                    a.cap, a.rv2, a.pos_build, a.rcutsq, a.sp,
                                                    a.status, a.wait_limit, a.run_if);
    else
      k_lj_tma<false><<<TB, kListTileAtoms, 0, st>>>(*a.tmap, a.posf, a.pos, a.f3, a.n, a.ld,
                                                     a.list, a.len, a.walker, a.skin, a.sf,
                                                     a.cap, a.rv2, a.pos_build, a.rcutsq, a.sp,
                                                     a.status, a.wait_limit, a.run_if);
  } else {
    if (energy)
      k_lj_fp32<true><<<B, T, 0, st>>>(a.posf, a.pos, a.f3, a.n, a.ld, a.list, a.len, a.walker,
                                       a.skin, a.sf, a.cap, a.rv2, a.pos_build, a.rcutsq,
                                       a.sp, a.epart, nullptr);
    else
      k_lj_fp32<false><<<B, T, 0, st>>>(a.posf, a.pos, a.f3, a.n, a.ld, a.list, a.len, a.walker,
                                        a.skin, a.sf, a.cap, a.rv2, a.pos_build, a.rcutsq,
                                        a.sp, a.epart, a.run_if);
  }
}

int lj_blocks(int n, bool fp32) {
  return fp32 ? nblk(n, 128) : nblk((long long)n * lj64_lanes(n), 128);
}
int mb_blocks(int n, bool fp32) { return fp32 ? nblk(n, 4) : n; }

template <bool ENERGY>
static void launch_mb64(const MbArgs& a, cudaStream_t st) {
  const int* gate = ENERGY ? nullptr : a.run_if;
  double *wi = (double*)a.xsi, *wj = (double*)a.xsj, *fs = (double*)a.fslot;
  double *e1 = ENERGY ? a.epart1 : nullptr, *e2 = ENERGY ? a.epart2 : nullptr;
  double* ea = ENERGY ? a.eatom : nullptr;
  const int B = nblk(a.n, 4);
  launch_dependent(a.early, k_mb_short<double>, B, 128, st, a.pos, a.posf, a.n, a.list, a.ri, a.rk,
                   a.len, a.grid, a.rcutsq, a.sl, (size_t)a.pitch, 1, a.slen, gate);
  if (!a.ref_rows) {
    launch_dependent(a.early, k_mb_bonds<ENERGY, true>, a.n, 128, st, a.pos, a.f3, a.n, a.sl, a.pitch,
                     a.slen, a.grid, a.cell3, a.ljexist, wi, wj, fs, a.slots, a.missing, e1, ea, gate);
    launch_dependent(a.early, k_mb_gather<ENERGY>, B, 128, st, a.pos, a.posf, a.f3, a.n, a.sl,
                     a.pitch, a.slen, a.grid, a.cell3, a.rcutsq, wi, wj, fs, a.slots, a.missing, e2, gate);
  } else if constexpr (!ENERGY) {
    launch_dependent(a.early, k_mb_bonds<false, false>, a.n, 128, st, a.pos, a.f3, a.n, a.sl, a.pitch,
                     a.slen, a.grid, nullptr, a.ljexist, wi, wj, nullptr, 0, a.missing, nullptr, nullptr,
                     gate);
    k_mb_pass2<<<B, 128, 0, st>>>(a.pos, a.f3, a.n, a.sl, a.pitch, a.slen, a.grid, a.ref_rows,
                                  a.ref_nls, a.ref_nlargest, a.rcutsq, wi, wj, a.missing);
  }
}

template <bool ENERGY>
static void launch_mb32(const MbArgs& a, cudaStream_t st) {
  const int* gate = ENERGY ? nullptr : a.run_if;
  float *wi = (float*)a.xsi, *wj = (float*)a.xsj;
  const int B = nblk(a.n, 4);
  // Blocks that wait early keep their places, and a grid of up to a wave (8 blocks
  // an SM) then lies unevenly on the SMs: us per step in a periodic box with early
  // launches and without 1,000 atoms 76.9 and 74.4, 2,744 101.8 and 80.2, 4,096 105.8
  // and 90.1; below and beyond 512 71.0 and 72.3, 5,832 110.5 and 112.7, 32,768 406.6
  // and 410.5.  Gated launches, which mostly return at once, start early at any size
  // (walls: 1,728 atoms 88.0 and 94.7); energy launches for a block per SM at most
  // (records of 64 atoms 100.8 and 105.2, of 2,744 163.2 and 141.9, of 32,768 the same).
  const bool early = a.early && (ENERGY ? B <= kSms : gate || B <= kSms || B > 8 * kSms);
  launch_dependent(early, k_mb_short<float>, B, 128, st, a.pos, a.posf, a.n, a.list, a.ri, a.rk,
                   a.len, a.grid, a.rcutsq, a.sl, 1, (size_t)a.n, a.slen, gate);
  launch_dependent(early, k_mb_pass1_32<ENERGY>, B, 128, st, a.pos, a.posf, a.f3, a.n, a.sl, a.slen,
                   a.grid, a.ljexist, wi, wj, ENERGY ? a.epart1 : nullptr, ENERGY ? a.eatom : nullptr,
                   gate);
  launch_dependent(early, k_mb_pass2_32<ENERGY>, B, 128, st, a.pos, a.posf, a.f3, a.n, a.sl, a.slen,
                   a.grid, a.cell3, a.ref_rows, a.ref_nls, a.ref_nlargest, a.rcutsq, wi, wj, a.missing,
                   ENERGY ? a.epart2 : nullptr, gate);
}

void launch_mb(const MbArgs& a, bool fp32, bool energy, cudaStream_t st) {
  if (a.n <= 0) return;
  if (fp32)
    energy ? launch_mb32<true>(a, st) : launch_mb32<false>(a, st);
  else
    energy ? launch_mb64<true>(a, st) : launch_mb64<false>(a, st);
}

}  // namespace mdgb
