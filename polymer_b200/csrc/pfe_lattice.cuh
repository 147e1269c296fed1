// Lattice/helix path state shared by the interpreter (pfe_lattice.cu) and the
// straight-line kernels (pfe_lattice_sl.cu).
#pragma once

#include "pfe_common.cuh"
#include "pfe_context.cuh"

namespace pfe {

struct LatGeom {
  int c1[3], c2[3];
  int n1[3];
  double period[3];
  double helix;
};

__device__ __forceinline__ int cell1_index(const LatGeom& g, int qx, int qy, int qz) {
  return (qx + g.c1[0]) + g.n1[0] * ((qy + g.c1[1]) + g.n1[1] * (qz + g.c1[2]));
}

struct LatticeRun {
  PairArrays pairs;
  const unsigned char* swp;
  const int* prim;
  const double* boys;  // table rows (boys_tab)
  const double* down;  // the table of boys_down
  const double* pp;    // P_P (npgs,npgs,cells1)
  const double* pph;   // P_P_HELIX or null
  double* cp;          // C_P (npgs,npgs,cells1)
  double* xp;
  const int4* chunks;
  const int* nchunks;
  const int4* tickets;
  const int* qcell;
  LatGeom g;
  int npgs;
  // mixed precision: ket images Q3 outside the CUTOFF1 box (the far cells) run
  // the recursion in FP32, the rest in FP64; n32 counts the FP32 quartets
  int far32;
  unsigned long long* n32;
  int* queue;          // the class's chunk counters, zero at launch
  const int* tidx;     // primitive -> contracted function (-1: a ghost)
  // set where P_P or P_P_HELIX has a non-zero element of a ghost; null where the
  // interpreter runs a class in any case
  const int* ghost;
};

// Work-queue counters per lattice class: one per register pass of the straight-line
// kernels, or one for k_lat_wide and one for the interpreter after it.
constexpr int kLatQueueSlots = 8;
// The straight-line kernel of evaluated class (e1|e2) (e1 >= e2, swap: the chunk's bra
// class is e2) on `grid` blocks of 128 threads, in one launch or a launch per register
// pass, or null for the classes that run one quartet per warp.
using LatSlFn = void (*)(const LatticeRun&, int grid, cudaStream_t);
LatSlFn lattice_sl_launcher(int e1, int e2, bool sw);
// The warp-per-quartet kernel of a class with d shells for bases whose d shells are all
// pure (pfe_lattice_wide.cu), on the class's top-level-d table; nx: kept integrals.
struct OpTableDev;
using LatWideFn = int (*)(const LatticeRun&, const OpTableDev&, int nx, int nchunks, int num_sms, cudaStream_t);
LatWideFn lattice_wide_launcher(int e1, int e2, bool sw);
void lattice_ghost_check(const double* p, long long n, int npgs, const int* tidx, int* flag, int num_sms,
                         cudaStream_t s);
// launches (register passes) of a straight-line class, 0 where the class has none
int lattice_sl_passes(int e1, int e2, bool sw);
// the launchers of classes with d shells in register passes (pfe_lattice_sl2.cu, pfe_lattice_sl3.cu)
LatSlFn lattice_sl_launcher_d(int e1, int e2, bool sw);
LatSlFn lattice_sl_launcher_2110(bool sw);

}  // namespace pfe
