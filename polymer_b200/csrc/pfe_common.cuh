// Shared device helpers of libpolymer_fock: constants, error plumbing, the
// tabulated Boys function and the cumulative-shell component counts.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string>

#include "../../include/polymer_fock.h"
#include "generated/eri_classes.cuh"

namespace pfe {

// The reference's own constant (src/pmodules.f90:7), used wherever it enters
// normalisation/prefactors so that integrals agree with it to the last digits.
constexpr double REF_PI = 3.14159265358979;
constexpr int LMAX_SUPPORTED = 2;   // cumulative s, sp, spd shells (what the workloads use)
constexpr int NPOW = 5;             // P_SHELL power extent 0..BASIS_LMAX+1
constexpr int MAXCOMP = 10;         // components of a cumulative d shell
constexpr int NIG_T = 1701;         // IGAMMA rows (T = 0..85 step 0.05)
constexpr int NIG_M = 28;           // IGAMMA orders 0..27

__host__ __device__ constexpr int ncum(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }

void set_error(const std::string& msg);

// Dynamic shared memory a kernel whose blocks' size depends on the molecule is allowed: all a
// block can have.  The limit belongs to the kernel on its device, not to a context, so one
// context's set-up must not lower it below what another's launches need.
constexpr int kMostSmem = 227 * 1024;

// Launches that return no status (launchers behind function pointers): a launch refused by
// the runtime shows in cudaGetLastError only until the next call that succeeds (CUDA 12.9),
// so every launch is followed by note_launch(), and whoever called them by
// PFE_CUDA(launch_status()).  Each thread has its own.
inline thread_local cudaError_t t_launch = cudaSuccess;   // the first failure not yet reported
inline void note(cudaError_t e) {
  if (e != cudaSuccess && t_launch == cudaSuccess) t_launch = e;
}
inline void note_launch() { note(cudaGetLastError()); }
inline cudaError_t launch_status() {
  note_launch();
  const cudaError_t e = t_launch;
  t_launch = cudaSuccess;
  return e;
}

#define PFE_CUDA(call)                                                                   \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess) {                                                             \
      ::pfe::t_launch = cudaSuccess;                                                     \
      ::pfe::set_error(std::string(#call) + ": " + cudaGetErrorString(e_));             \
      return (e_ == cudaErrorMemoryAllocation) ? PFE_ENOMEM : PFE_ECUDA;               \
    }                                                                                    \
  } while (0)

// Switch points of the asymptotic Boys form, TF(0:21) (src/pmodules.f90:156-159).
static __constant__ const double c_TF[22] = {33, 37, 41, 43, 46, 49, 51, 54, 56, 58, 61,
                                             63, 66, 68, 70, 72, 74, 76, 78, 80, 82, 84};

// Doubles of one IGAMMA row a Boys evaluation of orders 0..L reads (L+7 rounded
// up to even: whole 16-byte loads; rows are 28 doubles, so this stays inside one).
template <int L>
struct BoysRow {
  static constexpr int NV = (L + 8) / 2;
  static constexpr int N = 2 * NV;
};

// Gather the IGAMMA row nearest T (row-major [T][m], 16-byte aligned rows); the
// index is clamped to the table so a row can be fetched before knowing whether
// the Taylor branch will read it.
template <int L>
__device__ __forceinline__ void boys_row(double T, const double* __restrict__ tab, double* __restrict__ gv) {
  int ts = (int)floor(T * 20.0 + 0.5);
  ts = ts < NIG_T - 1 ? ts : NIG_T - 1;
  const double2* g2 = reinterpret_cast<const double2*>(tab + ts * NIG_M);
#pragma unroll
  for (int k = 0; k < BoysRow<L>::NV; ++k) {
    const double2 v = __ldg(g2 + k);
    gv[2 * k] = v.x;
    gv[2 * k + 1] = v.y;
  }
}

// F_m(T)*pref for m = 0..L exactly as the reference evaluates it
// (src/pfourindexdirect.f90:543-553): below TF(m) a 6-term Taylor series about
// the nearest tabulated point of IGAMMA (its row gv, from boys_row), above it
// the asymptotic form.  The asymptotic power T^(-m-1/2) is formed as
// rsqrt(T)*(1/T)^m instead of exp((-m-1/2) log T): same function, rounding
// differs in the last bit.
template <int L>
__device__ __forceinline__ void boys_eval(double T, double pref, const double* __restrict__ gv,
                                          double* __restrict__ F) {
  if (T < c_TF[L]) {
    const int ts = (int)floor(T * 20.0 + 0.5);  // NINT for T >= 0
    const double h = 0.05 * (double)ts - T;
#pragma unroll
    for (int m = 0; m <= L; ++m) {
      if (T < c_TF[m]) {
        F[m] = ((((((gv[m + 6] * h * 0.166666666666667 + gv[m + 5]) * h * 0.2 + gv[m + 4]) * h * 0.25 +
                   gv[m + 3]) * h * 0.333333333333333 + gv[m + 2]) * h * 0.5 + gv[m + 1]) * h + gv[m]) * pref;
      } else {
        // asymptotic prefactor F1(m) = (2m-1)!!/2^m * sqrt(PI)/2 (src/pfourindexdirect.f90:75-81)
        double v = pref * PFE_F1_0 * rsqrt(T);
        const double it = 1.0 / T;
        for (int k = 1; k <= m; ++k) v *= it * (0.5 * (double)(2 * k - 1));
        F[m] = v;
      }
    }
  } else {
    const double it = 1.0 / T;
    double v = pref * PFE_F1_0 * rsqrt(T);
    F[0] = v;
#pragma unroll
    for (int m = 1; m <= L; ++m) {
      v *= it * (0.5 * (double)(2 * m - 1));
      F[m] = v;
    }
  }
}

// Both steps; the row is read only on the Taylor branch.
template <int L>
__device__ __forceinline__ void boys_tab(double T, double pref, const double* __restrict__ tab,
                                         double* __restrict__ F) {
  double gv[BoysRow<L>::N];
  if (T < c_TF[L]) boys_row<L>(T, tab, gv);
  boys_eval<L>(T, pref, gv, F);
}

// The table of boys_down: for every top order L = 0 .. kDownMax and every grid point
// T0 = t/20 eight doubles (64 bytes, so a row is two sectors of one line):
// F_{L+k}(T0)/k! for k = 0..6, and e^-T0.
constexpr int kDownMax = 8;
constexpr int kDownCols = 8;
__host__ __device__ constexpr size_t down_row(int L, int t) { return ((size_t)L * NIG_T + t) * kDownCols; }

// The rows of boys_down that top order L reads (T below TF(L)), as four arrays of 16-byte
// pieces in shared memory: a gather there costs the conflicts of eight lanes over eight
// bank groups (about 11 wavefronts), in global memory a wavefront per lane.
constexpr int kTF[3] = {33, 37, 41};   // TF(0:2)
template <int L>
struct DownSmem {
  static constexpr bool use = L <= 2;
  static constexpr int ROWS = use ? 20 * kTF[L < 3 ? L : 0] + 1 : 0;
  static constexpr size_t BYTES = sizeof(double) * kDownCols * (size_t)ROWS;
};

template <int L>
__device__ __forceinline__ void down_stage(const double* __restrict__ down, double2* __restrict__ s) {
  constexpr int N = DownSmem<L>::ROWS;
  const double2* g = reinterpret_cast<const double2*>(down + down_row(L, 0));
  for (int i = threadIdx.x; i < 4 * N; i += blockDim.x) s[(i & 3) * N + (i >> 2)] = __ldg(g + i);
}

// F_m(T)*pref for m = 0..L (L <= kDownMax): below TF(L) the top order alone from the
// reference's 6-term series about the nearest grid point, e^-T from its tabulated value and
// the series of e^(T0-T) (|T0-T| <= 0.025: 8 terms leave 4e-18), and the lower orders by
// downward recursion F_m = (2T F_{m+1} + e^-T)/(2m+1), which is stable; above TF(L) the
// asymptotic form of boys_eval.  Against boys_tab, which expands every order: four 16-byte
// gathers per lane from rows of one line instead of up to eight from rows 224 bytes apart
// (the part of the table that a class reads shrinks from 190 to 55 KB at L = 3, inside the
// L1), and 15 + 2L multiply-adds instead of 7(L + 1).  The two agree to rounding.
// SMEM: `staged` holds the rows (down_stage), else they are read from `down`.
template <int L, bool SMEM = false>
__device__ __forceinline__ void boys_down(double T, double pref, const double* __restrict__ down,
                                          double* __restrict__ F, const double2* staged = nullptr) {
  static_assert(L <= kDownMax, "boys_down: orders 0..8");
  if (T < c_TF[L]) {
    const int ts = (int)floor(T * 20.0 + 0.5);   // NINT for T >= 0; <= 20 TF(L) < NIG_T
    const double h = 0.05 * (double)ts - T;
    double2 a, b, c, d;
    if constexpr (SMEM) {
      constexpr int N = DownSmem<L>::ROWS;
      a = staged[ts]; b = staged[N + ts]; c = staged[2 * N + ts]; d = staged[3 * N + ts];
    } else {
      const double2* r = reinterpret_cast<const double2*>(down + down_row(L, ts));
      a = __ldg(r); b = __ldg(r + 1); c = __ldg(r + 2); d = __ldg(r + 3);
    }
    const double f = fma(fma(fma(fma(fma(fma(d.x, h, c.y), h, c.x), h, b.y), h, b.x), h, a.y), h, a.x);
    const double x = fma(fma(fma(fma(fma(fma(fma(1.0 / 5040.0, h, 1.0 / 720.0), h, 1.0 / 120.0), h, 1.0 / 24.0), h,
                                     1.0 / 6.0), h, 0.5), h, 1.0), h, 1.0);
    const double e = pref * d.y * x, t2 = T + T;
    F[L] = pref * f;
#pragma unroll
    for (int m = L - 1; m >= 0; --m) F[m] = fma(t2, F[m + 1], e) * (1.0 / (double)(2 * m + 1));
  } else {
    const double it = 1.0 / T;
    double v = pref * PFE_F1_0 * rsqrt(T);
    F[0] = v;
#pragma unroll
    for (int m = 1; m <= L; ++m) {
      v *= it * (0.5 * (double)(2 * m - 1));
      F[m] = v;
    }
  }
}

}  // namespace pfe
