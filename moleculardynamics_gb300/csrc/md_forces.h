// Launch interface of the force kernels (md_forces.cu).
#pragma once
#include "md_internal.h"

namespace mdgb {

struct Gear64;

// Trip flags of a row list by step: the force launches of step t read [t % 3],
// the update to the positions of step t + 1 sets [(t + 1) % 3] and the force
// launch of step t clears [(t + 2) % 3], so that one kernel can do all three.
struct SkinFlags {
  int read, clear;
};
inline SkinFlags skin_flags(int step) { return {step % 3, (step + 2) % 3}; }

struct ForceArgs {
  const md_double4* pos;
  const float4* posf;   // FP32 copy (precision form)
  double* f3;
  int n;
  uint32_t* list;       // compact rows (rewritten per atom after a skin trip)
  int* len;
  int ld;               // list[k * ld + i]
  const CUtensorMap* tmap;  // TMA descriptor of the list (NULL: no TMA kernel)
  int all_ng;           // every atom is of the NG species
  int* status;
  RowWalker walker;     // full rows, walked when the skin is tripped
  int* skin;            // NeighborList::skin
  SkinFlags sf;
  int cap;              // compact row capacity
  float rv2;            // compact filter radius squared
  float4* pos_build;    // skin reference positions
  double rcutsq;
  Species sp;
  double* epart;        // 3 doubles per block when energy is requested
  int wait_limit = 1 << 20;  // polls of a bounded mbarrier wait (0: give up at once)
  const int* run_if = nullptr;  // force launches only: return at once unless *run_if != 0
  // the FP64 kernel with the Gear update (launch_lj_step64, launch_lj_redo64)
  const Gear64* gear64 = nullptr;
  int *hits = nullptr, *flag_next = nullptr;  // redo: steps with a wall hit; next step's flag
};

struct MbArgs {
  const md_double4* pos;
  const float4* posf;
  double* f3;
  int n;                // many-body atoms [0, n)
  const uint32_t* list; // full candidate rows, list[i * ri + k * rk]
  const int* len;
  size_t ri, rk;
  Grid grid;
  const int* cell3;     // build-time cells of the many-body list
  const int* ref_rows;  // or: rows in the reference layout (membership by scan)
  int ref_nls;
  int ref_nlargest;
  double rcutsq;
  int ljexist;          // accumulate onto F (BondOrderFuncs.h:325-336)
  uint32_t* sl;         // short lists (scratch, n * pitch): FP64 sl[i * pitch + s], FP32
                        // sl[s * n + i]; xsi, xsj alike
  int pitch;            // slots per atom; a multiple of 4 unless ref_rows is set
  int* slen;
  void* xsi;            // per (i, slot), T: the bond's factor va E / (4 (1 + xi_ij)^2)
  void* xsj;            // and va E / (4 (1 + xi_ji)^2), NaN where there is no bond
  void* fslot = nullptr;  // FP64: forces on third bodies, 3 for each of an atom's first
  int slots = 0;          // `slots` slots (not needed with ref_rows)
  int* missing;
  bool early = false;   // launches may start early (streams of this library only)
  const int* run_if = nullptr;  // force launches only: return at once unless *run_if != 0
  double* epart1;       // energy launches: 2 doubles per entry of mb_blocks (bonds)
  double* epart2;       // and 1 (third bodies)
  double* eatom = nullptr;  // energy launches: per-atom energy (sum over j of half the pair)
};

void launch_lj(const ForceArgs& a, bool fp32, bool energy, cudaStream_t st);
// FP64: forces and correct (then predict, gear64->predict) in one kernel;
// f3 NULL: the forces are not stored.  redo: after a correct with walls, the
// forces and a = F/m again if *run_if, then the predict.
void launch_lj_step64(const ForceArgs& a, cudaStream_t st);
void launch_lj_redo64(const ForceArgs& a, cudaStream_t st);
void launch_mb(const MbArgs& a, bool fp32, bool energy, cudaStream_t st);
int lj_blocks(int n, bool fp32);  // blocks of an energy launch of launch_lj
int mb_blocks(int n, bool fp32);  // entries of an energy launch in epart1, epart2
// Force slots for each of n atoms with short lists of up to `pitch`: 64 (usual
// lattices use 28), fewer where those would take more than a quarter of the free
// memory.  Third bodies beyond them are evaluated by k_mb_gather, so any number will
// do; with 64 of them an atom takes 1.5 KB more.
inline int mb_slot_count(long long n, int pitch, unsigned long long free_bytes) {
  int slots = pitch < 64 ? pitch : 64;
  while (slots && 3ull * sizeof(double) * (unsigned long long)slots * (unsigned long long)n >
                      free_bytes / 4)
    slots /= 2;
  return slots;
}

}  // namespace mdgb
