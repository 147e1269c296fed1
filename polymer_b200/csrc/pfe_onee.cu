// One-electron integrals on the device: S_P and T_P (OVERLAP_KINETIC(0),
// src/ponee.f90:1-160) and N_P (NUCLEAR_ATTRACTION(0), src/ponee.f90:418-603)
// over primitive shells, per lattice cell, with the helical image of the second
// centre.  These are set-up inputs of the Fock build (S_P feeds its pair
// prefactors), computed once per geometry.  One thread per (shell pair, cell);
// the Obara-Saika recursions are those of the reference, the Boys function is
// the same tabulated evaluation as the two-electron kernels.

#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "pfe_common.cuh"
#include "pfe_context.cuh"

namespace pfe {

// storage index of a Cartesian power triple of total <= 2 (10 slots)
__device__ __forceinline__ int cidx(int a, int b, int c) {
  // order: 000 001 002 010 011 020 100 101 110 200
  const int s = a * 100 + b * 10 + c;
  switch (s) {
    case 0: return 0;
    case 1: return 1;
    case 2: return 2;
    case 10: return 3;
    case 11: return 4;
    case 20: return 5;
    case 100: return 6;
    case 101: return 7;
    case 110: return 8;
    default: return 9;  // 200
  }
}

struct OneeDev {
  int npgs, npshell, natom;
  const int* p_shell;  // Fortran P_SHELL(npshell,0:4,0:4,0:4), 1-based
  const int* ang;
  const double *x, *y, *z, *zt;
  const int* iatom;
  const double *ax, *ay, *az;
  int cel1[3], cel2[3];
  double period[3], helix;
  const double* boys;  // row-major [T][m]
};

__device__ __forceinline__ int psh(const OneeDev& a, int s, int i1, int i2, int i3) {
  return a.p_shell[s + a.npshell * (i1 + NPOW * (i2 + NPOW * i3))] - 1;
}

__global__ void k_overlap_kinetic(OneeDev a, double* __restrict__ s_p, double* __restrict__ t_p) {
  const int n1x = 2 * a.cel1[0] + 1, n1y = 2 * a.cel1[1] + 1, n1z = 2 * a.cel1[2] + 1;
  const long long total = (long long)a.npshell * a.npshell * n1x * n1y * n1z;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int I = (int)(t % a.npshell), J = (int)((t / a.npshell) % a.npshell);
  const long long cell = t / ((long long)a.npshell * a.npshell);
  const int kx = (int)(cell % n1x) - a.cel1[0];
  const int ky = (int)((cell / n1x) % n1y) - a.cel1[1];
  const int kz = (int)(cell / ((long long)n1x * n1y)) - a.cel1[2];
  const double qx = kx * a.period[0], qy = ky * a.period[1], qz = kz * a.period[2];
  const double ang = kx * a.helix, cs = cos(ang), sn = sin(ang);
  const int ii = psh(a, I, 0, 0, 0), jj = psh(a, J, 0, 0, 0);
  const double Ax = a.x[ii], Ay = a.y[ii], Az = a.z[ii];
  const double Bx = a.x[jj] + qx, By = a.y[jj] * cs - a.z[jj] * sn + qy, Bz = a.y[jj] * sn + a.z[jj] * cs + qz;
  const double r = (Ax - Bx) * (Ax - Bx) + (Ay - By) * (Ay - By) + (Az - Bz) * (Az - Bz);
  const double z1 = a.zt[ii] + a.zt[jj], z2 = sqrt(z1 * z1 * z1), gzi = a.zt[ii] * a.zt[jj] / z1;
  const double pisub = sqrt(REF_PI * REF_PI * REF_PI);
  double S1[10][10], T1[10][10];
  S1[0][0] = pisub / z2 * exp(-gzi * r);
  T1[0][0] = gzi * (3.0 - 2.0 * gzi * r) * S1[0][0];
  const double Px = (Ax * a.zt[ii] + Bx * a.zt[jj]) / z1, Py = (Ay * a.zt[ii] + By * a.zt[jj]) / z1,
               Pz = (Az * a.zt[ii] + Bz * a.zt[jj]) / z1;
  const double PA[3] = {Px - Ax, Py - Ay, Pz - Az}, PB[3] = {Px - Bx, Py - By, Pz - Bz};
  const int LI = a.ang[I], LJ = a.ang[J];
  for (int i1 = 0; i1 <= LI; ++i1)
    for (int i2 = 0; i2 <= LI - i1; ++i2)
      for (int i3 = 0; i3 <= LI - i1 - i2; ++i3)
        for (int j1 = 0; j1 <= LJ; ++j1)
          for (int j2 = 0; j2 <= LJ - j1; ++j2)
            for (int j3 = 0; j3 <= LJ - j1 - j2; ++j3) {
              if (i1 + i2 + i3 + j1 + j2 + j3 == 0) continue;
              int A[3] = {i1, i2, i3}, B[3] = {j1, j2, j3};
              int ax = -1;
              bool onA = false;
              for (int k = 0; k < 3 && ax < 0; ++k) if (A[k] >= 1) { ax = k; onA = true; }
              for (int k = 0; k < 3 && ax < 0; ++k) if (B[k] >= 1) { ax = k; onA = false; }
              const int ci = cidx(i1, i2, i3), cj = cidx(j1, j2, j3);
              if (onA) {
                int A1[3] = {i1, i2, i3};
                A1[ax]--;
                const int c1 = cidx(A1[0], A1[1], A1[2]);
                double s = PA[ax] * S1[c1][cj];
                double sm2 = 0.0, tm2 = 0.0, sb = 0.0, tb = 0.0;
                if (A[ax] >= 2) {
                  int A2[3] = {A1[0], A1[1], A1[2]};
                  A2[ax]--;
                  const int c2 = cidx(A2[0], A2[1], A2[2]);
                  sm2 = S1[c2][cj];
                  tm2 = T1[c2][cj];
                  s += 0.5 * (double)(A[ax] - 1) / z1 * sm2;
                }
                if (B[ax] >= 1) {
                  int B2[3] = {j1, j2, j3};
                  B2[ax]--;
                  const int cb = cidx(B2[0], B2[1], B2[2]);
                  sb = S1[c1][cb];
                  tb = T1[c1][cb];
                  s += 0.5 * (double)B[ax] / z1 * sb;
                }
                S1[ci][cj] = s;
                double tv = 2.0 * gzi * s + PA[ax] * T1[c1][cj];
                if (A[ax] >= 2) tv += 0.5 * (double)(A[ax] - 1) / z1 * tm2 - (double)(A[ax] - 1) * gzi / a.zt[ii] * sm2;
                if (B[ax] >= 1) tv += 0.5 * (double)B[ax] / z1 * tb;
                T1[ci][cj] = tv;
              } else {
                int B1[3] = {j1, j2, j3};
                B1[ax]--;
                const int c1 = cidx(B1[0], B1[1], B1[2]);
                double s = PB[ax] * S1[ci][c1];
                double sm2 = 0.0, tm2 = 0.0;
                if (B[ax] >= 2) {
                  int B2[3] = {B1[0], B1[1], B1[2]};
                  B2[ax]--;
                  const int c2 = cidx(B2[0], B2[1], B2[2]);
                  sm2 = S1[ci][c2];
                  tm2 = T1[ci][c2];
                  s += 0.5 * (double)(B[ax] - 1) / z1 * sm2;
                }
                S1[ci][cj] = s;
                double tv = 2.0 * gzi * s + PB[ax] * T1[ci][c1];
                if (B[ax] >= 2) tv += 0.5 * (double)(B[ax] - 1) / z1 * tm2 - (double)(B[ax] - 1) * gzi / a.zt[jj] * sm2;
                T1[ci][cj] = tv;
              }
            }
  const size_t pp = (size_t)a.npgs * a.npgs;
  for (int i1 = 0; i1 <= LI; ++i1)
    for (int i2 = 0; i2 <= LI - i1; ++i2)
      for (int i3 = 0; i3 <= LI - i1 - i2; ++i3)
        for (int j1 = 0; j1 <= LJ; ++j1)
          for (int j2 = 0; j2 <= LJ - j1; ++j2)
            for (int j3 = 0; j3 <= LJ - j1 - j2; ++j3) {
              const size_t o = (size_t)psh(a, I, i1, i2, i3) + (size_t)a.npgs * psh(a, J, j1, j2, j3) + pp * cell;
              s_p[o] = S1[cidx(i1, i2, i3)][cidx(j1, j2, j3)];
              t_p[o] = T1[cidx(i1, i2, i3)][cidx(j1, j2, j3)];
            }
}

// Cartesian powers of total <= L ordered by total: the index space of the vertical
// recursion, and where each row of it comes from (one power removed on axis `ax`,
// two removed on that axis or -1, and the factor of the latter); up: one power added on
// an axis, or -1.
template <int L>
struct CartTable {
  static constexpr int N = (L + 1) * (L + 2) * (L + 3) / 6;
  int p[N][3], tot[N], ax[N], one[N], two[N], fac[N], up[N][3];
  static constexpr int at(int x, int y, int z) {
    const int t = x + y + z;
    int n = t * (t + 1) * (t + 2) / 6;   // rows of smaller total
    for (int i = 0; i <= t; ++i)
      for (int j = 0; j <= t - i; ++j) {
        if (i == x && j == y) return n;
        ++n;
      }
    return -1;
  }
  constexpr CartTable() : p(), tot(), ax(), one(), two(), fac(), up() {
    int n = 0;
    for (int t = 0; t <= L; ++t)
      for (int x = 0; x <= t; ++x)
        for (int y = 0; y <= t - x; ++y, ++n) {
          p[n][0] = x; p[n][1] = y; p[n][2] = t - x - y;
          tot[n] = t;
          const int k = x > 0 ? 0 : (y > 0 ? 1 : 2);
          ax[n] = k;
          int e[3] = {p[n][0], p[n][1], p[n][2]};
          e[k] -= 1;
          one[n] = t > 0 ? at(e[0], e[1], e[2]) : -1;
          fac[n] = t > 0 ? e[k] : 0;
          e[k] -= 1;
          two[n] = (t > 0 && e[k] >= 0) ? at(e[0], e[1], e[2]) : -1;
          for (int i = 0; i < 3; ++i)
            up[n][i] = t < L ? at(x + (i == 0), y + (i == 1), t - x - y + (i == 2)) : -1;
        }
  }
};

// f(0), f(1), ... f(N - 1) with the index a compile-time constant (the table entries of
// the two d classes are not folded by loop unrolling, and the recursion's array would
// land in local memory).
template <int N, int I = 0, typename F>
__device__ __forceinline__ void each_index(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    each_index<N, I + 1>(f);
  }
}

// Nuclear attraction of one class of shell pairs, LA >= LB, one pair and cell per
// thread: the shells with LA in listA, those with LB in listB.  The first shell of a
// pair (at cell 0) has LA, or LB with SWAP; the recursion always runs on the centre
// of the LA shell.  What bounds it is FP64 work in registers: only [e|0] with
// |e| <= LA + LB is built per nucleus, summed over the nuclei, and the horizontal
// recursion to (a|b), which does not depend on the nucleus, runs once per pair.  The
// earlier kernel (every class in one kernel, the full two-centre recursion per
// nucleus in dynamically indexed local memory) took 3.47 ms on C10H22 6-31G**.
template <int LA, int LB, bool SWAP>
__global__ void __launch_bounds__(128) k_nuclear(OneeDev a, const int* __restrict__ listA, int na,
                                                 const int* __restrict__ listB, int nb, double* __restrict__ n_p) {
  constexpr int LT = LA + LB;
  constexpr int NE = CartTable<LT>::N;
  const int n1x = 2 * a.cel1[0] + 1, n1y = 2 * a.cel1[1] + 1, n1z = 2 * a.cel1[2] + 1;
  const long long total = (long long)na * nb * n1x * n1y * n1z;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int SA = listA[t % na], SB = listB[(t / na) % nb];
  const long long cell = t / ((long long)na * nb);
  const int k1x = (int)(cell % n1x) - a.cel1[0];
  const int k1y = (int)((cell / n1x) % n1y) - a.cel1[1];
  const int k1z = (int)(cell / ((long long)n1x * n1y)) - a.cel1[2];
  const double ang = k1x * a.helix, cs = cos(ang), sn = sin(ang);
  const int ia = psh(a, SA, 0, 0, 0), ib = psh(a, SB, 0, 0, 0);
  // centres of the two shells: the pair's second one is the image in the cell
  auto centre = [&](int i, bool image, double* c) {
    const double x = a.x[i], y = a.y[i], z = a.z[i];
    c[0] = image ? x + k1x * a.period[0] : x;
    c[1] = image ? y * cs - z * sn + k1y * a.period[1] : y;
    c[2] = image ? y * sn + z * cs + k1z * a.period[2] : z;
  };
  double A[3], B[3], P[3], PA[3], AB[3];
  centre(ia, SWAP, A);
  centre(ib, !SWAP, B);
  const double za = a.zt[ia], zb = a.zt[ib], comz = za + zb;
  double r = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    P[k] = (A[k] * za + B[k] * zb) / comz;
    PA[k] = P[k] - A[k];
    AB[k] = A[k] - B[k];
    r += AB[k] * AB[k];
  }
  const double sab = sqrt(REF_PI * REF_PI * REF_PI) / sqrt(comz * comz * comz) * exp(-za * zb / comz * r);
  const double e1 = 2.0 / sqrt(REF_PI) * sqrt(comz) * sab;
  const double h = 0.5 / comz;
  double S[NE];
#pragma unroll
  for (int e = 0; e < NE; ++e) S[e] = 0.0;
  for (int k2x = -a.cel2[0]; k2x <= a.cel2[0]; ++k2x) {
    const double ang2 = k2x * a.helix, cs2 = cos(ang2), sn2 = sin(ang2);
    for (int k2y = -a.cel2[1]; k2y <= a.cel2[1]; ++k2y)
      for (int k2z = -a.cel2[2]; k2z <= a.cel2[2]; ++k2z)
        for (int k = 0; k < a.natom; ++k) {
          const double y = a.ay[k], z = a.az[k];
          const double PC[3] = {P[0] - (a.ax[k] + k2x * a.period[0]), P[1] - (y * cs2 - z * sn2 + k2y * a.period[1]),
                                P[2] - (y * sn2 + z * cs2 + k2z * a.period[2])};
          double F[LT + 1];
          boys_tab<LT>(comz * (PC[0] * PC[0] + PC[1] * PC[1] + PC[2] * PC[2]), -(double)a.iatom[k] * e1, a.boys, F);
          // V[e][m] for |e| + m <= LT
          double V[NE][LT + 1];
#pragma unroll
          for (int m = 0; m <= LT; ++m) V[0][m] = F[m];
          each_index<NE - 1>([&](auto i) {
            constexpr int e = decltype(i)::value + 1;
            constexpr CartTable<LT> E{};
            constexpr int ax = E.ax[e], one = E.one[e], two = E.two[e], fac = E.fac[e], top = LT - E.tot[e];
#pragma unroll
            for (int m = 0; m <= top; ++m) {
              double v = PA[ax] * V[one][m] - PC[ax] * V[one][m + 1];
              if constexpr (two >= 0) v += (double)fac * h * (V[two][m] - V[two][m + 1]);
              V[e][m] = v;
            }
          });
#pragma unroll
          for (int e = 0; e < NE; ++e) S[e] += V[e][0];
        }
  }
  // (a|b) from [e|0]: (a|b + 1i) = (a + 1i|b) + AB_i (a|b)
  const size_t pp = (size_t)a.npgs * a.npgs;
  each_index<CartTable<LA>::N * CartTable<LB>::N>([&](auto i) {
    constexpr int ea = decltype(i)::value / CartTable<LB>::N, eb = decltype(i)::value % CartTable<LB>::N;
    constexpr CartTable<LT> E{};
    double v;
    if constexpr (E.tot[eb] == 0) {
      v = S[ea];
    } else if constexpr (E.tot[eb] == 1) {
      constexpr int x = E.ax[eb];
      v = S[E.up[ea][x]] + AB[x] * S[ea];
    } else {
      constexpr int x = E.ax[eb], y = E.ax[E.one[eb]];
      v = (S[E.up[E.up[ea][x]][y]] + AB[y] * S[E.up[ea][x]]) + AB[x] * (S[E.up[ea][y]] + AB[y] * S[ea]);
    }
    const int pra = psh(a, SA, E.p[ea][0], E.p[ea][1], E.p[ea][2]), prb = psh(a, SB, E.p[eb][0], E.p[eb][1], E.p[eb][2]);
    n_p[(size_t)(SWAP ? prb : pra) + (size_t)a.npgs * (SWAP ? pra : prb) + pp * cell] = v;
  });
}

// Every class of shell pairs; lists: the shells ordered by L (start[L] .. start[L + 1]).
static void launch_nuclear(const OneeDev& d, const int* list, const int* start, long long cells, double* n_p) {
  auto run = [&](auto kern, int la, int lb) {
    const int na = start[la + 1] - start[la], nb = start[lb + 1] - start[lb];
    const long long total = (long long)na * nb * cells;
    if (total > 0)
      kern<<<(unsigned)((total + 127) / 128), 128>>>(d, list + start[la], na, list + start[lb], nb, n_p);
      note_launch();
  };
  run(k_nuclear<2, 2, false>, 2, 2);
  run(k_nuclear<2, 1, false>, 2, 1);
  run(k_nuclear<2, 1, true>, 2, 1);
  run(k_nuclear<2, 0, false>, 2, 0);
  run(k_nuclear<2, 0, true>, 2, 0);
  run(k_nuclear<1, 1, false>, 1, 1);
  run(k_nuclear<1, 0, false>, 1, 0);
  run(k_nuclear<1, 0, true>, 1, 0);
  run(k_nuclear<0, 0, false>, 0, 0);
}

// Host-side checks shared by the one-electron entry points, made before any
// device work: the kernels index S_P/T_P/N_P by P_SHELL of every component a
// shell reaches (i1+i2+i3 <= P_SHELL_ANG) and by the shell head P_SHELL(s,0,0,0),
// so each of those entries must name a primitive 1..NPGS.  `need_atoms`: the
// allocating entry point uploads the atom list and the Boys table as well.
static int onee_validate(const pfe_onee_args* a, bool need_atoms) {
  if (!a || a->npgs <= 0 || a->npshell <= 0 || (need_atoms && a->natom <= 0)) {
    set_error("invalid one-electron arguments");
    return PFE_EINVAL;
  }
  if (!a->p_shell || !a->p_shell_ang || !a->pgsx || !a->pgsy || !a->pgsz || !a->zt ||
      (need_atoms && (!a->iatom || !a->atomx || !a->atomy || !a->atomz || !a->igamma))) {
    set_error("a required one-electron array pointer is null");
    return PFE_EINVAL;
  }
  for (int k = 0; k < 3; ++k)
    if (a->cel1[k] < 0 || a->cel2[k] < 0) { set_error("negative cutoff"); return PFE_EINVAL; }
  for (int s = 0; s < a->npshell; ++s) {
    const int L = a->p_shell_ang[s];
    if (L < 0 || L > LMAX_SUPPORTED) {
      set_error("P_SHELL_ANG outside the one-electron kernels (s, p, d)");
      return L < 0 ? PFE_EINVAL : PFE_EUNSUPPORTED;
    }
    for (int i1 = 0; i1 <= L; ++i1)
      for (int i2 = 0; i2 <= L - i1; ++i2)
        for (int i3 = 0; i3 <= L - i1 - i2; ++i3) {
          const int p = a->p_shell[(size_t)s + (size_t)a->npshell * (i1 + NPOW * (i2 + NPOW * i3))];
          if (p < 1 || p > a->npgs) {
            char msg[160];
            std::snprintf(msg, sizeof msg, "P_SHELL(%d,%d,%d,%d) = %d is not a primitive 1..NPGS (%d)", s + 1, i1, i2,
                          i3, p, a->npgs);
            set_error(msg);
            return PFE_EINVAL;
          }
        }
  }
  return PFE_OK;
}

// Device scratch of the allocating entry points, per device: the inputs, packed, and the
// results.  Up to kScratchKept bytes stay from call to call (the thirteen allocations and
// copies of a call were most of its time); larger calls allocate and free their own.
struct OneeScratch {
  std::mutex mu;   // held for the whole call
  char* p = nullptr;
  size_t n = 0;
  std::vector<char> host;              // the packed inputs
  std::shared_ptr<BoysTables> boys;    // of the last IGAMMA
};
static OneeScratch g_onee[64];
constexpr size_t kScratchKept = (size_t)64 << 20;

static size_t round256(size_t b) { return (b + 255) & ~size_t(255); }

static int onee_run(const pfe_onee_args* a, double* s_p, double* t_p, double* n_p) {
  if (const int v = onee_validate(a, true)) return v;
  int dev = 0;
  PFE_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) { set_error("device index out of range"); return PFE_EINVAL; }
  OneeScratch& sc = g_onee[dev];
  std::lock_guard<std::mutex> lock(sc.mu);
  int rc = acquire_boys(dev, a->igamma, nullptr, &sc.boys);
  if (rc != PFE_OK) return rc;
  const size_t psz = (size_t)a->npshell * NPOW * NPOW * NPOW;
  const int n1 = (2 * a->cel1[0] + 1) * (2 * a->cel1[1] + 1) * (2 * a->cel1[2] + 1);
  const size_t out_bytes = sizeof(double) * (size_t)a->npgs * a->npgs * n1;
  std::vector<int> list;   // the shells ordered by L
  int start[4] = {0, 0, 0, 0};
  for (int L = 0; L <= LMAX_SUPPORTED; ++L) {
    for (int sh = 0; sh < a->npshell; ++sh)
      if (a->p_shell_ang[sh] == L) list.push_back(sh);
    start[L + 1] = (int)list.size();
  }
  // the inputs, packed, and their places
  struct Part {
    const void* h;
    size_t bytes, at;
  };
  const size_t pg = sizeof(double) * a->npgs, at = sizeof(double) * a->natom;
  Part part[] = {{a->p_shell, sizeof(int) * psz, 0}, {a->p_shell_ang, sizeof(int) * a->npshell, 0},
                 {a->pgsx, pg, 0}, {a->pgsy, pg, 0}, {a->pgsz, pg, 0}, {a->zt, pg, 0},
                 {a->iatom, sizeof(int) * a->natom, 0}, {a->atomx, at, 0}, {a->atomy, at, 0}, {a->atomz, at, 0},
                 {list.data(), sizeof(int) * list.size(), 0}};
  size_t in_bytes = 0;
  for (Part& p : part) {
    p.at = in_bytes;
    in_bytes += round256(p.bytes);
  }
  const int nout = n_p ? 1 : 2;
  const size_t need = in_bytes + nout * round256(out_bytes);
  char* own = nullptr;   // freed on every way out
  struct Guard {
    char*& p;
    ~Guard() { cudaFree(p); }
  } guard{own};
  char* base = nullptr;
  if (need > kScratchKept) {
    PFE_CUDA(cudaMalloc((void**)&own, need));
    base = own;
  } else {
    if (need > sc.n) {
      cudaFree(sc.p);
      sc.p = nullptr;
      sc.n = 0;
      PFE_CUDA(cudaMalloc((void**)&sc.p, need));
      sc.n = need;
    }
    base = sc.p;
  }
  sc.host.resize(in_bytes);
  for (const Part& p : part) memcpy(sc.host.data() + p.at, p.h, p.bytes);
  PFE_CUDA(cudaMemcpy(base, sc.host.data(), in_bytes, cudaMemcpyHostToDevice));
  auto i32 = [&](int k) { return reinterpret_cast<const int*>(base + part[k].at); };
  auto f64 = [&](int k) { return reinterpret_cast<const double*>(base + part[k].at); };
  OneeDev d{};
  d.npgs = a->npgs; d.npshell = a->npshell; d.natom = a->natom;
  d.p_shell = i32(0); d.ang = i32(1); d.x = f64(2); d.y = f64(3); d.z = f64(4); d.zt = f64(5);
  d.iatom = i32(6); d.ax = f64(7); d.ay = f64(8); d.az = f64(9); d.boys = sc.boys->rows;
  for (int k = 0; k < 3; ++k) { d.cel1[k] = a->cel1[k]; d.cel2[k] = a->cel2[k]; d.period[k] = a->period[k]; }
  d.helix = a->helix;
  double* out0 = reinterpret_cast<double*>(base + in_bytes);
  double* out1 = reinterpret_cast<double*>(base + in_bytes + round256(out_bytes));
  // elements of primitives that no shell component reaches stay zero
  PFE_CUDA(cudaMemsetAsync(out0, 0, nout * round256(out_bytes), nullptr));
  if (n_p) {
    launch_nuclear(d, i32(10), start, n1, out0);
    PFE_CUDA(launch_status());
  } else {
    const long long total = (long long)a->npshell * a->npshell * n1;
    k_overlap_kinetic<<<(unsigned)((total + 127) / 128), 128>>>(d, out0, out1);
    PFE_CUDA(cudaGetLastError());
  }
  if (n_p) {
    PFE_CUDA(cudaMemcpy(n_p, out0, out_bytes, cudaMemcpyDeviceToHost));
  } else {
    if (s_p) PFE_CUDA(cudaMemcpy(s_p, out0, out_bytes, cudaMemcpyDeviceToHost));
    if (t_p) PFE_CUDA(cudaMemcpy(t_p, out1, out_bytes, cudaMemcpyDeviceToHost));
    if (!s_p && !t_p) PFE_CUDA(cudaDeviceSynchronize());
  }
  return PFE_OK;
}

// ---------------------------------------------------------------- fixed-scratch variant
//
// pfe_overlap_kinetic_noalloc runs k_overlap_kinetic with all of its device
// data (the shell map, centres, exponents and the S_P/T_P results) staged in
// one statically sized device array of this file instead of cudaMalloc'd
// buffers, for callers that may not allocate device memory once they are
// running (a pre-reserved memory budget, a custom allocator that owns the
// device, a process that must not grow its footprint).  Limit: everything must
// fit in kNoAllocScratchBytes (16 MiB), i.e. 2*npgs^2*cells + the inputs; a
// C20H42 6-31G** molecule (976 primitives) fits, larger inputs are refused.

constexpr size_t kNoAllocScratchBytes = size_t(16) << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

static std::mutex g_noalloc_mu;          // held for the whole call: calls share the one buffer
static void* g_noalloc_ptr[64] = {nullptr};

// Device address of the scratch on the current device.  The first call on a
// device does the set-up (loads the module there, looks up the symbol).
static int noalloc_scratch(void** out) {
  int dev = 0;
  PFE_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) { set_error("device index out of range"); return PFE_EINVAL; }
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      set_error(std::string("cudaGetSymbolAddress of the fixed scratch failed: ") + cudaGetErrorString(e));
      return PFE_ECUDA;
    }
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return PFE_OK;
}

static int onee_noalloc(const pfe_onee_args* a, double* s_p, double* t_p) {
  if (!s_p || !t_p) { set_error("invalid one-electron arguments"); return PFE_EINVAL; }
  if (const int v = onee_validate(a, false)) return v;
  const long long n1 = (long long)(2 * a->cel1[0] + 1) * (2 * a->cel1[1] + 1) * (2 * a->cel1[2] + 1);
  const size_t out_n = (size_t)a->npgs * a->npgs * n1;
  const size_t psz = (size_t)a->npshell * NPOW * NPOW * NPOW;
  // scratch layout: S_P | T_P | x | y | z | zt | P_SHELL | P_SHELL_ANG
  const size_t b_out = round256(sizeof(double) * out_n), b_pg = round256(sizeof(double) * a->npgs);
  const size_t b_ps = round256(sizeof(int) * psz), b_ang = round256(sizeof(int) * a->npshell);
  const size_t need = 2 * b_out + 4 * b_pg + b_ps + b_ang;
  if (need > kNoAllocScratchBytes) {
    char msg[256];
    std::snprintf(msg, sizeof msg,
                  "pfe_overlap_kinetic_noalloc: needs %zu bytes of device scratch, the fixed buffer holds %zu "
                  "(npgs %d, %lld cells); use pfe_overlap_kinetic",
                  need, kNoAllocScratchBytes, a->npgs, n1);
    set_error(msg);
    return PFE_EINVAL;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  void* base = nullptr;
  int rc = noalloc_scratch(&base);
  if (rc != PFE_OK) return rc;
  unsigned char* p = static_cast<unsigned char*>(base);
  double* ds = reinterpret_cast<double*>(p);
  double* dt = reinterpret_cast<double*>(p + b_out);
  double* dx = reinterpret_cast<double*>(p + 2 * b_out);
  double* dy = reinterpret_cast<double*>(p + 2 * b_out + b_pg);
  double* dz = reinterpret_cast<double*>(p + 2 * b_out + 2 * b_pg);
  double* dzt = reinterpret_cast<double*>(p + 2 * b_out + 3 * b_pg);
  int* dps = reinterpret_cast<int*>(p + 2 * b_out + 4 * b_pg);
  int* dang = reinterpret_cast<int*>(p + 2 * b_out + 4 * b_pg + b_ps);
  PFE_CUDA(cudaMemcpy(dx, a->pgsx, sizeof(double) * a->npgs, cudaMemcpyHostToDevice));
  PFE_CUDA(cudaMemcpy(dy, a->pgsy, sizeof(double) * a->npgs, cudaMemcpyHostToDevice));
  PFE_CUDA(cudaMemcpy(dz, a->pgsz, sizeof(double) * a->npgs, cudaMemcpyHostToDevice));
  PFE_CUDA(cudaMemcpy(dzt, a->zt, sizeof(double) * a->npgs, cudaMemcpyHostToDevice));
  PFE_CUDA(cudaMemcpy(dps, a->p_shell, sizeof(int) * psz, cudaMemcpyHostToDevice));
  PFE_CUDA(cudaMemcpy(dang, a->p_shell_ang, sizeof(int) * a->npshell, cudaMemcpyHostToDevice));
  // S_P/T_P entries of primitives that no shell component reaches stay zero,
  // as with the allocating entry point: clear both results first
  PFE_CUDA(cudaMemset(ds, 0, sizeof(double) * out_n));
  PFE_CUDA(cudaMemset(dt, 0, sizeof(double) * out_n));
  OneeDev d{};
  d.npgs = a->npgs; d.npshell = a->npshell; d.natom = a->natom;
  d.p_shell = dps; d.ang = dang; d.x = dx; d.y = dy; d.z = dz; d.zt = dzt;
  for (int k = 0; k < 3; ++k) { d.cel1[k] = a->cel1[k]; d.cel2[k] = a->cel2[k]; d.period[k] = a->period[k]; }
  d.helix = a->helix;
  const long long total = (long long)a->npshell * a->npshell * n1;
  k_overlap_kinetic<<<(unsigned)((total + 127) / 128), 128>>>(d, ds, dt);
  PFE_CUDA(cudaGetLastError());
  PFE_CUDA(cudaMemcpy(s_p, ds, sizeof(double) * out_n, cudaMemcpyDeviceToHost));
  PFE_CUDA(cudaMemcpy(t_p, dt, sizeof(double) * out_n, cudaMemcpyDeviceToHost));
  return PFE_OK;
}

}  // namespace pfe

extern "C" {
int32_t pfe_overlap_kinetic(const pfe_onee_args* a, double* s_p, double* t_p) { return pfe::onee_run(a, s_p, t_p, nullptr); }
int32_t pfe_nuclear_attraction(const pfe_onee_args* a, double* n_p) { return pfe::onee_run(a, nullptr, nullptr, n_p); }
int32_t pfe_overlap_kinetic_noalloc(const pfe_onee_args* a, double* s_p, double* t_p) { return pfe::onee_noalloc(a, s_p, t_p); }
}
