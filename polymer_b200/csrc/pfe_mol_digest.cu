// Digestion of the straight-line molecular classes: X(abcd) of every group quartet,
// stored by the register passes (k_gq) as one 256-byte row per integral and chunk,
// contracted with the density into J' and K' once.
//
// What bounds it: the L1's wavefronts.  A lane's targets lie at addresses of its own
// (its ket's shells), so a scattered load or atomic of a warp costs 32 wavefronts;
// digested inside every register pass that was 55 % of the C20H42 build ((21|11): 56
// gathers and 56 atomics per lane in each of 9 passes).  Here
//   * the density and the accumulators are block panels: the matrix of a shell pair is
//     contiguous, so the warp copies the blocks of its 32 quartets cooperatively, lanes
//     along the elements (one or two lines per block instead of one per element), into
//     shared memory rows of 33 doubles, from where each lane reads its own column;
//   * K' and J'(cd) leave the same way: columns to shared memory, then atomics with the
//     lanes along the elements of a block;
//   * the bra is the warp's, so J'(ab) is summed over the lanes first.
// The multiply-adds (six per integral) run per lane from registers.
// Measured, C20H42 6-31G** (B200): (21|11) 2.9 ms inside its nine passes, 0.7 ms here;
// (11|10) 2.4 and 0.9 ms; all classes 17 and 6.9 ms.  A tile's integrals are read once, at
// a quarter of the DRAM rate: the kernel waits on loads with 16 warps per SM.

#include <algorithm>

#include "pfe_common.cuh"
#include "pfe_context.cuh"
#include "pfe_mol_kernels.cuh"

namespace pfe {

namespace {

// Kept components of the class's shells: KEPT is the lower_kept bits of L = 1 and 2.
template <int LA, int LB, int LC, int LD, int KEPT>
struct DigestShape {
  static constexpr int NA = kept_n(LA, KEPT), NB = kept_n(LB, KEPT), NC = kept_n(LC, KEPT), ND = kept_n(LD, KEPT);
  static constexpr int R_AC = 0, R_AD = NA * NC, R_BC = R_AD + NA * ND, R_BD = R_BC + NB * NC, R_CD = R_BD + NB * ND;
  static constexpr int ROWS = R_CD + NC * ND;
  static constexpr int PER_WARP = ROWS * 33 + NA * NB;   // doubles: the rows, then the bra's density block
  static constexpr int WARPS = PER_WARP * 8 * 4 <= 100 * 1024 ? 4 : (PER_WARP * 8 * 2 <= 100 * 1024 ? 2 : 1);
  // Resident blocks the register allocation aims at.  The kernel waits on loads (a chain of
  // six dependent ones to reach the blocks, then X from HBM), so warps count for more than
  // registers beyond the accumulators: (11|10) at 158 registers issued in 18.6 % of the
  // cycles on 10 warps per SM.
  static constexpr int ACC = NB * (NC + ND) + NC * ND;
  static constexpr int TARGET = ACC <= 12 ? 24 : (ACC <= 28 ? 20 : (ACC <= 52 ? 12 : 8));   // warps per SM
  static constexpr int BY_SMEM = (220 * 1024) / (PER_WARP * 8 * WARPS + 1024);
  static constexpr int BLOCKS = TARGET / WARPS < BY_SMEM ? TARGET / WARPS : BY_SMEM;
};

// The warp's copy of 32 blocks of M doubles into rows [0, M) of s, lane l's block in
// column l: block of lane l at m + scale * (lane l's row).
template <int M>
__device__ __forceinline__ void load_blocks(const double* __restrict__ m, int row, long long scale,
                                            double* __restrict__ s, int lane) {
#pragma unroll(M < 8 ? M : 8)
  for (int i = 0; i < M; ++i) {
    const int f = i * 32 + lane, l = f / M, e = f - l * M;
    s[e * 33 + l] = __ldg(m + scale * __shfl_sync(0xffffffffu, row, l) + e);
  }
}

// The reverse with atomics, for the first `cnt` lanes' blocks, scaled by w.
template <int M>
__device__ __forceinline__ void add_blocks(double* __restrict__ m, int row, long long scale,
                                           const double* __restrict__ s, int cnt, double w, int lane) {
#pragma unroll(M < 8 ? M : 8)
  for (int i = 0; i < M; ++i) {
    const int f = i * 32 + lane, l = f / M, e = f - l * M;
    double* to = m + scale * __shfl_sync(0xffffffffu, row, l) + e;
    const double v = s[e * 33 + l];
    if (l < cnt && v != 0.0) atomicAdd(to, w * v);
  }
}

// Sums over the warp of four values at once (12 shuffles instead of 40): lane 8 k gets
// that of v[k].
__device__ __forceinline__ double warp_sum4(const double (&v)[4], int lane) {
  const bool hi = lane & 16, odd = lane & 8;
  double a = hi ? v[2] : v[0], b = hi ? v[3] : v[1];
  a += __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
  b += __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 16);
  double r = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}

template <int LA, int LB, int LC, int LD, int KEPT>
__global__ void __launch_bounds__(32 * DigestShape<LA, LB, LC, LD, KEPT>::WARPS,
                                  DigestShape<LA, LB, LC, LD, KEPT>::BLOCKS) k_digest(const __grid_constant__ MolLaunch lq) {
  using S = DigestShape<LA, LB, LC, LD, KEPT>;
  constexpr int NA = S::NA, NB = S::NB, NC = S::NC, ND = S::ND, NCD = NC * ND;
  extern __shared__ double smem[];
  const int lane = threadIdx.x & 31;
  double* __restrict__ sm = smem + (size_t)(threadIdx.x >> 5) * S::PER_WARP;
  double* __restrict__ col = sm + lane;   // this lane's column
  double* __restrict__ dab = sm + S::ROWS * 33;
  const int nchunks = *lq.nchunks;
  const int step = gridDim.x * S::WARPS;
  for (int t = blockIdx.x * S::WARPS + (threadIdx.x >> 5); t < lq.tn; t += step) {
    const int c = (lq.t0 + t) * lq.numprocs + lq.myid;
    if (c >= nchunks) break;
    if (!lq.xlive[t]) continue;
    __syncwarp();                      // every lane has read the flag
    if (lane == 0) lq.xlive[t] = 0;    // clean for the next tile or build
    const Chunk ch = lq.chunks[c];
    const PairRec* __restrict__ rec = lq.rec;
    const int *bk_list = lq.bk_list, *gr_start = lq.gr_start, *poff = lq.poff, *ptgt = lq.ptgt;
    const double* __restrict__ pd = lq.pd;
    double *pj = lq.pj, *pk = lq.pk;
    int np = lq.np;
    if (lq.insts) {
      const MolLaunch* q = lq.insts + ch.inst;
      rec = q->rec; bk_list = q->bk_list; gr_start = q->gr_start; poff = q->poff; ptgt = q->ptgt;
      pd = q->pd; pj = q->pj; pk = q->pk; np = q->np;
    }
    const int cnt = ch.end - ch.first;
    const int H = bk_list[ch.first + (lane < cnt ? lane : 0)];
    const int2 ij = __ldg(reinterpret_cast<const int2*>(&rec[gr_start[ch.G]].si));
    const int2 kl = __ldg(reinterpret_cast<const int2*>(&rec[gr_start[H]].si));
    const int pA = poff[ij.x], pB = poff[ij.y], pC = poff[kl.x], pD = poff[kl.y];
    // block (X, Y) of a panel matrix begins at pX * np + pY * nX
    const double* __restrict__ dA = pd + (long long)pA * np;
    const double* __restrict__ dB = pd + (long long)pB * np;
    load_blocks<NA * NC>(dA, pC, NA, sm + S::R_AC * 33, lane);
    load_blocks<NA * ND>(dA, pD, NA, sm + S::R_AD * 33, lane);
    load_blocks<NB * NC>(dB, pC, NB, sm + S::R_BC * 33, lane);
    load_blocks<NB * ND>(dB, pD, NB, sm + S::R_BD * 33, lane);
    {
      const long long o = (long long)pC * np + (long long)pD * NC;
      const int lo = (int)o, hi = (int)(o >> 32);
#pragma unroll(NCD < 8 ? NCD : 8)
      for (int i = 0; i < NCD; ++i) {
        const int f = i * 32 + lane, l = f / NCD, e = f - l * NCD;
        const long long ol = ((long long)__shfl_sync(0xffffffffu, hi, l) << 32) |
                             (unsigned int)__shfl_sync(0xffffffffu, lo, l);
        sm[(S::R_CD + e) * 33 + l] = __ldg(pd + ol + e);
      }
    }
    for (int i = lane; i < NA * NB; i += 32) dab[i] = __ldg(dA + (long long)pB * NA + i);
    // components without a target have no stored integrals
    const unsigned int live_a = __ballot_sync(0xffffffffu, lane < NA && ptgt[pA + (lane < NA ? lane : 0)] >= 0);
    const unsigned int live_b = __ballot_sync(0xffffffffu, lane < NB && ptgt[pB + (lane < NB ? lane : 0)] >= 0);
    __syncwarp();
    const double* __restrict__ xb = lq.xbuf + (size_t)t * ((size_t)NA * NB * NCD * 32) + lane;
    double kbc[NB * NC], kbd[NB * ND], jcd[NCD];
#pragma unroll
    for (int i = 0; i < NB * NC; ++i) kbc[i] = 0.0;
#pragma unroll
    for (int i = 0; i < NB * ND; ++i) kbd[i] = 0.0;
#pragma unroll
    for (int i = 0; i < NCD; ++i) jcd[i] = 0.0;
#pragma unroll 1
    for (int a = 0; a < NA; ++a) {
      double dac[NC], dad[ND], kac[NC], kad[ND];
#pragma unroll
      for (int x = 0; x < NC; ++x) { dac[x] = col[(S::R_AC + x * NA + a) * 33]; kac[x] = 0.0; }
#pragma unroll
      for (int x = 0; x < ND; ++x) { dad[x] = col[(S::R_AD + x * NA + a) * 33]; kad[x] = 0.0; }
      if ((live_a >> a) & 1) {
        double jab[(NB + 3) / 4 * 4];
#pragma unroll
        for (int b = 0; b < (NB + 3) / 4 * 4; ++b) jab[b] = 0.0;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          if (!((live_b >> b) & 1)) continue;   // warp-uniform
          const double pab = dab[b * NA + a];
          double x[NCD];
#pragma unroll
          for (int cd = 0; cd < NCD; ++cd) x[cd] = __ldcs(xb + ((a * NB + b) * NCD + cd) * 32);
#pragma unroll
          for (int cc = 0; cc < NC; ++cc) {
            const double dbc = col[(S::R_BC + cc * NB + b) * 33];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              const double v = x[cc * ND + d];
              jab[b] = fma(col[(S::R_CD + d * NC + cc) * 33], v, jab[b]);
              jcd[cc * ND + d] = fma(pab, v, jcd[cc * ND + d]);
              kad[d] = fma(dbc, v, kad[d]);
              kac[cc] = fma(col[(S::R_BD + d * NB + b) * 33], v, kac[cc]);
              kbd[b * ND + d] = fma(dac[cc], v, kbd[b * ND + d]);
              kbc[b * NC + cc] = fma(dad[d], v, kbc[b * NC + cc]);
            }
          }
        }
        double* __restrict__ jA = pj + (long long)pA * np + (long long)pB * NA;
        if constexpr (NB == 1) {
          const double v = warp_sum(jab[0]);
          if (lane == 0 && v != 0.0) atomicAdd(jA + a, 0.25 * v);
        } else {
#pragma unroll
          for (int b0 = 0; b0 < NB; b0 += 4) {
            const double v4[4] = {jab[b0], jab[b0 + 1], jab[b0 + 2], jab[b0 + 3]};
            const double v = warp_sum4(v4, lane);
            const int b = b0 + (lane >> 3);
            if ((lane & 7) == 0 && b < NB && v != 0.0) atomicAdd(jA + b * NA + a, 0.25 * v);
          }
        }
      }
#pragma unroll
      for (int x = 0; x < NC; ++x) col[(S::R_AC + x * NA + a) * 33] = kac[x];
#pragma unroll
      for (int x = 0; x < ND; ++x) col[(S::R_AD + x * NA + a) * 33] = kad[x];
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int x = 0; x < NC; ++x) col[(S::R_BC + x * NB + b) * 33] = kbc[b * NC + x];
#pragma unroll
      for (int x = 0; x < ND; ++x) col[(S::R_BD + x * NB + b) * 33] = kbd[b * ND + x];
    }
#pragma unroll
    for (int cc = 0; cc < NC; ++cc)
#pragma unroll
      for (int d = 0; d < ND; ++d) col[(S::R_CD + d * NC + cc) * 33] = jcd[cc * ND + d];
    __syncwarp();
    double* __restrict__ kA = pk + (long long)pA * np;
    double* __restrict__ kB = pk + (long long)pB * np;
    add_blocks<NA * NC>(kA, pC, NA, sm + S::R_AC * 33, cnt, 0.125, lane);
    add_blocks<NA * ND>(kA, pD, NA, sm + S::R_AD * 33, cnt, 0.125, lane);
    add_blocks<NB * NC>(kB, pC, NB, sm + S::R_BC * 33, cnt, 0.125, lane);
    add_blocks<NB * ND>(kB, pD, NB, sm + S::R_BD * 33, cnt, 0.125, lane);
    {
      const long long o = (long long)pC * np + (long long)pD * NC;
      const int lo = (int)o, hi = (int)(o >> 32);
#pragma unroll(NCD < 8 ? NCD : 8)
      for (int i = 0; i < NCD; ++i) {
        const int f = i * 32 + lane, l = f / NCD, e = f - l * NCD;
        const long long ol = ((long long)__shfl_sync(0xffffffffu, hi, l) << 32) |
                             (unsigned int)__shfl_sync(0xffffffffu, lo, l);
        const double v = sm[(S::R_CD + e) * 33 + l];
        if (l < cnt && v != 0.0) atomicAdd(pj + ol + e, 0.25 * v);
      }
    }
    __syncwarp();   // the rows are refilled for the next chunk
  }
}

template <int LA, int LB, int LC, int LD, int KEPT>
void run(const MolLaunch& ql, int num_sms, cudaStream_t s) {
  using S = DigestShape<LA, LB, LC, LD, KEPT>;
  constexpr int bytes = S::PER_WARP * S::WARPS * 8;
  auto kern = k_digest<LA, LB, LC, LD, KEPT>;
  note(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  const int grid = std::min((ql.tn + S::WARPS - 1) / S::WARPS, num_sms * S::BLOCKS);
  kern<<<std::max(grid, 1), 32 * S::WARPS, bytes, s>>>(ql);
  note_launch();
}

// the kept bits that matter to a class: those of the angular momenta it has
template <int LA, int LB, int LC, int LD>
void pick(const MolLaunch& ql, int num_sms, cudaStream_t s) {
  constexpr bool p = LA == 1 || LB == 1 || LC == 1 || LD == 1, d = LA == 2 || LB == 2 || LC == 2 || LD == 2;
  const int bits = ql.lower_kept_bits & ((p ? 2 : 0) | (d ? 4 : 0));
  if (bits == 0) return run<LA, LB, LC, LD, 0>(ql, num_sms, s);
  if constexpr (p) {
    if (bits == 2) return run<LA, LB, LC, LD, 2>(ql, num_sms, s);
  }
  if constexpr (d) {
    if (bits == 4) return run<LA, LB, LC, LD, 4>(ql, num_sms, s);
  }
  if constexpr (p && d) return run<LA, LB, LC, LD, 6>(ql, num_sms, s);
}

}  // namespace

void launch_digest(int cb, int ck, const MolLaunch& ql, int num_sms, cudaStream_t s) {
  switch (cb * 8 + ck) {
#define D(CB, CK, A, B, C, E) case CB * 8 + CK: return pick<A, B, C, E>(ql, num_sms, s);
    D(1, 0, 1, 0, 0, 0) D(1, 1, 1, 0, 1, 0)
    D(2, 0, 1, 1, 0, 0) D(2, 1, 1, 1, 1, 0) D(2, 2, 1, 1, 1, 1)
    D(3, 0, 2, 0, 0, 0) D(3, 1, 2, 0, 1, 0) D(3, 2, 2, 0, 1, 1) D(3, 3, 2, 0, 2, 0)
    D(4, 0, 2, 1, 0, 0) D(4, 1, 2, 1, 1, 0) D(4, 2, 2, 1, 1, 1) D(4, 3, 2, 1, 2, 0) D(4, 4, 2, 1, 2, 1)
    D(5, 0, 2, 2, 0, 0) D(5, 1, 2, 2, 1, 0) D(5, 2, 2, 2, 1, 1) D(5, 3, 2, 2, 2, 0)
#undef D
    default: return;
  }
}

}  // namespace pfe
