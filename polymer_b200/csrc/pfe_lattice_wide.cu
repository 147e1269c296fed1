// Lattice/helix quartets of the classes with d shells: one quartet per warp on the
// op table that keeps the d shells' top level only, digesting the components that
// have a contracted function.
//
// The interpreter of every class (pfe_lattice.cu:k_lattice) evaluates and digests all
// components of the cumulative shells: (dd|dp) is 6552 operations and 4000 integrals, of
// which 3079 and at most 864 matter when every d shell of the basis is pure (its s and p
// components are ghosts without a contracted function).  A ghost's rows of C_P and X_P
// are dropped by the contraction CC . CC^T; its density is zero whenever P_P is a
// decontracted density.  That is checked on the device (k_ghost_check): where it does not
// hold these kernels return at once and the interpreters, which otherwise return at once,
// do the whole class.  Besides, every lane evaluates the Boys values and the geometry
// itself, tickets are single (bra, ket) pairs instead of 32 kets, and the output slots are
// listed once per ticket for all image cells.
// Measured (B200), helical polyethylene 6-31G**, CUTOFF1/2 = 1/2, both orders of the
// classes, against the interpreter of every component: (22|21) 7.8 -> 0.28 ms, (22|11) 3.4
// -> 0.35, (21|11) 4.1 -> 1.9, (22|22) 1.8 -> 0.21; the build 39.8 -> 14.5 ms.

#include <algorithm>

#include "pfe_common.cuh"
#include "pfe_context.cuh"
#include "pfe_interp.cuh"
#include "pfe_lattice.cuh"

namespace pfe {

namespace {

template <int N1, int N2, int M1, int M2>
struct LatWide {
  static constexpr int GEO = (int)((sizeof(OpGeom) + 7) / 8);
  static constexpr int MAXJ = N1 > N2 ? N1 : N2, MAXK = M1 > M2 ? M1 : M2;
  static constexpr int INTS = 2 * (N1 + N2 + M1 + M2) + 4;
  // doubles of one warp: slots | D(k,l) | D(k,j) | geometry | ints | output slots
  static __host__ __device__ int doubles(int nslots, int nx) {
    return nslots + M1 * M2 + MAXK * MAXJ + GEO + (INTS + 1) / 2 + (nx + 1) / 2;
  }
};

// Components of shell s that have a contracted function (lanes of one warp): their
// indices and primitives; returns the count.
template <int N>
__device__ __forceinline__ int kept_prims(const int* __restrict__ prim, const int* __restrict__ tidx, int s, int* k,
                                          int* pr, int lane) {
  const int p = lane < N ? prim[s * MAXCOMP + lane] : -1;
  const bool keep = p >= 0 && tidx[p] >= 0;
  const unsigned int m = __ballot_sync(0xffffffffu, keep);
  if (keep) {
    const int i = __popc(m & ((1u << lane) - 1));
    k[i] = lane;
    pr[i] = p;
  }
  return __popc(m);
}

// (LA LB|LC LD) is the evaluated class; SWAP: the chunk's bra pair is its ket pair.
template <int LA, int LB, int LC, int LD, bool SWAP>
__global__ void __launch_bounds__(128) k_lat_wide(LatticeRun R, OpTableDev tab, int per_warp) {
  constexpr int N1 = SWAP ? ncum(LC) : ncum(LA), N2 = SWAP ? ncum(LD) : ncum(LB);   // the chunk's bra
  constexpr int M1 = SWAP ? ncum(LA) : ncum(LC), M2 = SWAP ? ncum(LB) : ncum(LD);   // its kets
  constexpr int LT = LA + LB + LC + LD;
  using W = LatWide<N1, N2, M1, M2>;
  if (*R.ghost) return;   // some ghost has a density: the interpreter's launch does the class
  extern __shared__ double smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double* v = smem + (size_t)wid * per_warp;
  double* DJ = v + tab.nslots;
  double* DK = DJ + M1 * M2;
  OpGeom& geo = *reinterpret_cast<OpGeom*>(DK + W::MAXK * W::MAXJ);
  int* ka = reinterpret_cast<int*>(DK + W::MAXK * W::MAXJ + W::GEO);
  int* kb = ka + N1;
  int* kc = kb + N2;
  int* kd = kc + M1;
  int* pa = kd + M2;
  int* pb = pa + N1;
  int* pc = pb + N2;
  int* pd = pc + M1;
  int* xs = ka + W::INTS + (W::INTS & 1);
  const PairArrays pr = R.pairs;
  const int npgs = R.npgs;
  const size_t pp2 = (size_t)npgs * npgs;
  const LatGeom& g = R.g;
  const double c2pi = 2.0 / sqrt(REF_PI);
  const int h3 = g.c2[0] + g.c1[0];
  const bool helix = R.pph != nullptr;
  const long long ntickets = 32ll * *R.nchunks;
  if (lane == 0) v[0] = 0.0;
  for (;;) {
    int tk = 0;
    if (lane == 0) tk = atomicAdd(R.queue, 1);
    tk = __shfl_sync(0xffffffffu, tk, 0);
    if (tk >= ntickets) break;
    const int4 ch = R.chunks[tk >> 5];
    const int p = ch.x, q = ch.y + (tk & 31);
    if (q >= ch.z) continue;   // warp-uniform
    const int4 tkt = R.tickets[ch.w];
    const int q1[3] = {R.qcell[3 * tkt.x], R.qcell[3 * tkt.x + 1], R.qcell[3 * tkt.x + 2]};
    const int q2[3] = {R.qcell[3 * tkt.y], R.qcell[3 * tkt.y + 1], R.qcell[3 * tkt.y + 2]};
    const bool swb = R.swp[p] != 0, swk = R.swp[q] != 0;
    __syncwarp();   // the previous ticket is done with the lists
    const int na = kept_prims<N1>(R.prim, R.tidx, pr.si[p], ka, pa, lane);
    const int nb = kept_prims<N2>(R.prim, R.tidx, pr.sj[p], kb, pb, lane);
    const int nc = kept_prims<M1>(R.prim, R.tidx, pr.si[q], kc, pc, lane);
    const int nd = kept_prims<M2>(R.prim, R.tidx, pr.sj[q], kd, pd, lane);
    __syncwarp();
    const int nab = na * nb, ncd = nc * nd;
    for (int i = lane; i < nab * ncd; i += 32) {
      const int ab = i / ncd, cd = i - ab * ncd;
      const int a = ka[ab / nb], b = kb[ab % nb], c = kc[cd / nd], d = kd[cd % nd];
      xs[i] = tab.out[SWAP ? ((c * M2 + d) * N1 + a) * N2 + b : ((a * N2 + b) * M1 + c) * M2 + d];
    }
    const double zb = pr.zeta[p], ze = pr.zeta[q], zz = zb + ze, rzz = 1.0 / zz, rho = zb * ze * rzz;
    const double pref = c2pi * pr.S[p] * pr.S[q] * sqrt(rho);
    const double Pb[3] = {pr.P[0][p], pr.P[1][p], pr.P[2][p]};
    const double Qb[3] = {pr.P[0][q], pr.P[1][q], pr.P[2][q]};
    // the digestion's orders: i, j of the bra and k, l of the ket (first centre first
    // unless swapped), with the strides of an integral's index ((a nb + b) nc + c) nd + d
    const int nI = swb ? nb : na, nJ = swb ? na : nb, nK = swk ? nd : nc, nL = swk ? nc : nd;
    const int sI = swb ? ncd : nb * ncd, sJ = swb ? nb * ncd : ncd, sK = swk ? 1 : nd, sL = swk ? nd : 1;
    const int *pi = swb ? pb : pa, *pj = swb ? pa : pb, *pk = swk ? pd : pc, *pl = swk ? pc : pd;
    double jacc[4] = {0.0, 0.0, 0.0, 0.0};   // J of bra component pair lane + 32 r, over the cells
    for (int q3z = -g.c2[2]; q3z <= g.c2[2]; ++q3z)
    for (int q3y = -g.c2[1]; q3y <= g.c2[1]; ++q3y)
    for (int q3x = -g.c2[0]; q3x <= g.c2[0]; ++q3x) {
      const int q3[3] = {q3x, q3y, q3z};
      bool lcel = true;
#pragma unroll
      for (int k = 0; k < 3; ++k)
        lcel = lcel && (q3[k] + q2[k] >= -g.c1[k]) && (q3[k] + q2[k] <= g.c1[k]) && (q1[k] - q3[k] >= -g.c1[k]) &&
               (q1[k] - q3[k] <= g.c1[k]);
      const double ang = q3x * g.helix, cs = cos(ang), sn = sin(ang);
      // screw image of the ket pair: rotate about x, then translate
      const double Q[3] = {Qb[0] + q3x * g.period[0], Qb[1] * cs - Qb[2] * sn + q3y * g.period[1],
                           Qb[1] * sn + Qb[2] * cs + q3z * g.period[2]};
      const double T = rho * ((Pb[0] - Q[0]) * (Pb[0] - Q[0]) + (Pb[1] - Q[1]) * (Pb[1] - Q[1]) +
                              (Pb[2] - Q[2]) * (Pb[2] - Q[2]));
      double F[LT + 1];
      boys_down<LT>(T, pref, R.down, F);
      __syncwarp();   // the previous cell's digestion has read the slots and blocks
#pragma unroll
      for (int m = 0; m <= LT; ++m)
        if (lane == m) v[1 + m] = F[m];
      if (lane == LT + 1) {
        const double QCb[3] = {pr.PA[0][q], pr.PA[1][q], pr.PA[2][q]};
        const double CDb[3] = {pr.AB[0][q], pr.AB[1][q], pr.AB[2][q]};
        const double QC[3] = {QCb[0], QCb[1] * cs - QCb[2] * sn, QCb[1] * sn + QCb[2] * cs};
        const double CD[3] = {CDb[0], CDb[1] * cs - CDb[2] * sn, CDb[1] * sn + CDb[2] * cs};
        double PA[3], AB[3], WP[3], WQ[3];
        for (int k = 0; k < 3; ++k) {
          const double Wk = (zb * Pb[k] + ze * Q[k]) * rzz;
          PA[k] = pr.PA[k][p];
          AB[k] = pr.AB[k][p];
          WP[k] = Wk - Pb[k];
          WQ[k] = Wk - Q[k];
        }
        if (!SWAP) set_geom(geo, PA, WP, QC, WQ, AB, CD, 0.5 / zb, 0.5 / ze, 0.5 * rzz, ze * rzz, zb * rzz);
        else set_geom(geo, QC, WQ, PA, WP, CD, AB, 0.5 / ze, 0.5 / zb, 0.5 * rzz, zb * rzz, ze * rzz);
      }
      const double* __restrict__ dj =
          helix ? R.pph + pp2 * ((size_t)(q3x + g.c2[0]) + (size_t)(2 * g.c2[0] + 1) * (q3x + q2[0] + h3))
                : R.pp + pp2 * cell1_index(g, q2[0], q2[1], q2[2]);
      for (int t = lane; t < ncd; t += 32) {   // D(k,l) by ket component pair (c, d)
        const int c = t / nd, d = t - c * nd;
        DJ[t] = __ldg(dj + (swk ? pd[d] : pc[c]) + (size_t)npgs * (swk ? pc[c] : pd[d]));
      }
      if (lcel) {
        const double* __restrict__ dk =
            helix ? R.pph + pp2 * ((size_t)(q3x + g.c2[0]) + (size_t)(2 * g.c2[0] + 1) * (q1[0] + h3))
                  : R.pp + pp2 * cell1_index(g, q1[0] - q3x, q1[1] - q3y, q1[2] - q3z);
        for (int t = lane; t < nK * nJ; t += 32) {
          const int k = t / nJ, j = t - k * nJ;
          DK[t] = __ldg(dk + pk[k] + (size_t)npgs * pj[j]);
        }
      }
      __syncwarp();
      for (int l = 0; l < tab.nlevels; ++l) {
        run_level(tab.ops, tab.levels[l], tab.levels[l + 1], v, geo, lane, 32, EvalD{});
        __syncwarp();
      }
      // J: C(i,j,Q1) += sum_kl D(k,l) (ij|kl)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int t = lane + 32 * r;
        if (t < nab) {
          double acc = 0.0;
          for (int cd = 0; cd < ncd; ++cd) acc = fma(DJ[cd], v[xs[t * ncd + cd]], acc);
          jacc[r] += acc;
        }
      }
      // K: X(i,l,Q3+Q2) += sum_jk D(k,j) (ij|kl)
      if (lcel) {
        double* __restrict__ xp = R.xp + pp2 * cell1_index(g, q3x + q2[0], q3y + q2[1], q3z + q2[2]);
        for (int t = lane; t < nI * nL; t += 32) {
          const int l = t / nI, i = t - l * nI;
          const int* __restrict__ x0 = xs + i * sI + l * sL;
          double acc = 0.0;
          for (int k = 0; k < nK; ++k)
            for (int j = 0; j < nJ; ++j) acc = fma(DK[k * nJ + j], v[x0[j * sJ + k * sK]], acc);
          if (acc != 0.0) atomicAdd(xp + pi[i] + (size_t)npgs * pl[l], acc);
        }
      }
    }
    double* __restrict__ cp = R.cp + pp2 * cell1_index(g, q1[0], q1[1], q1[2]);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int t = lane + 32 * r;
      if (t < nab && jacc[r] != 0.0) {
        const int a = t / nb, b = t - a * nb;
        atomicAdd(cp + (swb ? pb[b] : pa[a]) + (size_t)npgs * (swb ? pa[a] : pb[b]), jacc[r]);
      }
    }
  }
}

template <int LA, int LB, int LC, int LD, bool SWAP>
int launch_wide(const LatticeRun& r, const OpTableDev& t, int nx, int nchunks, int num_sms, cudaStream_t s) {
  using W = LatWide<SWAP ? ncum(LC) : ncum(LA), SWAP ? ncum(LD) : ncum(LB), SWAP ? ncum(LA) : ncum(LC),
                    SWAP ? ncum(LB) : ncum(LD)>;
  const int per_warp = W::doubles(t.nslots, nx);
  const size_t one = sizeof(double) * (size_t)per_warp, cap = 160 * 1024;   // the rest of the SM's memory is L1: op records
  if (one > 200 * 1024) { set_error("lattice op table exceeds shared memory"); return PFE_EUNSUPPORTED; }
  const int wpb = (int)std::max<size_t>(1, std::min<size_t>(4, cap / 4 / one));
  const size_t smem = one * wpb;
  auto kern = k_lat_wide<LA, LB, LC, LD, SWAP>;
  PFE_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem));
  const int per_sm = std::max(1, std::min(16, (int)(cap / smem)));
  const long long work = (32ll * nchunks + wpb - 1) / wpb;
  const int grid = (int)std::max<long long>(1, std::min<long long>(work, (long long)num_sms * per_sm));
  kern<<<grid, 32 * wpb, smem, s>>>(r, t, per_warp);
  PFE_CUDA(cudaGetLastError());
  return PFE_OK;
}

__global__ void k_ghost_check(const double* __restrict__ p, long long n, int npgs, const int* __restrict__ tidx,
                              int* __restrict__ flag) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t % npgs), j = (int)((t / npgs) % npgs);
    if ((tidx[i] < 0 || tidx[j] < 0) && p[t] != 0.0) *flag = 1;   // NaN counts as non-zero
  }
}

}  // namespace

void lattice_ghost_check(const double* p, long long n, int npgs, const int* tidx, int* flag, int num_sms,
                         cudaStream_t s) {
  k_ghost_check<<<(unsigned)std::min<long long>((n + 255) / 256, 16ll * num_sms), 256, 0, s>>>(p, n, npgs, tidx, flag);
  note_launch();
}

// evaluated class (e1 >= e2) and swap flag -> launcher, or null for the classes without a
// d shell or with straight-line code
LatWideFn lattice_wide_launcher(int e1, int e2, bool sw) {
#define L2(A, B, C, D) (sw ? &launch_wide<A, B, C, D, true> : &launch_wide<A, B, C, D, false>)
  switch (e1 * 8 + e2) {
    case 34: return L2(2, 1, 1, 1);
    case 35: return L2(2, 1, 2, 0);
    case 36: return L2(2, 1, 2, 1);
    case 40: return L2(2, 2, 0, 0);
    case 41: return L2(2, 2, 1, 0);
    case 42: return L2(2, 2, 1, 1);
    case 43: return L2(2, 2, 2, 0);
    case 44: return L2(2, 2, 2, 1);
    case 45: return L2(2, 2, 2, 2);
    default: return nullptr;
  }
#undef L2
}

}  // namespace pfe
