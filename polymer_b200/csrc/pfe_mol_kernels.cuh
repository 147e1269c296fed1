// Molecular quartet kernels shared by the FP64 and mixed-precision
// instantiations (pfe_mol.cu, pfe_mol_mixed.cu): the launch block, density
// bounds, the precision switch of the recursion, the digestion helpers and the
// straight-line group-quartet kernel with its pass launchers.
#pragma once

#include <algorithm>

#include "pfe_common.cuh"
#include "pfe_context.cuh"
#include "generated/eri_classes.cuh"

namespace pfe {

// One shell pair as the quartet kernels read it, 128 bytes (seven 16-byte
// loads): P[3], PA[3], AB[3], zeta, S, Schwarz bound, (si, sj), 1/(2 zeta),
// padding.
struct __align__(16) PairRec {
  double P[3], PA[3], AB[3];
  double zeta, S, schwarz;
  int si, sj;
  double oz;
  double pad[2];
};
static_assert(sizeof(PairRec) == 128, "PairRec layout");

struct PairView {
  double P[3], PA[3], AB[3], zeta, S, oz, bound;
  int si, sj;
};

// the record of pair t with its Schwarz bound (the quartet loops load the whole
// record before screening on the bound: one load latency per pair, not two)
__device__ __forceinline__ PairView pair_view(const double2* __restrict__ r, int stride) {
  const double2 a = __ldg(r), b = __ldg(r + stride), c = __ldg(r + 2 * stride), d = __ldg(r + 3 * stride),
                e = __ldg(r + 4 * stride), f = __ldg(r + 5 * stride), g = __ldg(r + 6 * stride);
  PairView v;
  v.P[0] = a.x; v.P[1] = a.y; v.P[2] = b.x;
  v.PA[0] = b.y; v.PA[1] = c.x; v.PA[2] = c.y;
  v.AB[0] = d.x; v.AB[1] = d.y; v.AB[2] = e.x;
  v.zeta = e.y; v.S = f.x; v.bound = f.y;
  v.si = __double2loint(g.x); v.sj = __double2hiint(g.x);
  v.oz = g.y;
  return v;
}

__device__ __forceinline__ PairView load_pair(const PairRec* __restrict__ rec, int t) {
  return pair_view(reinterpret_cast<const double2*>(rec + t), 1);
}

// Ket records by tile: the records of 32 consecutive ket groups of a bucket, interleaved
// by lane, so that a warp whose lanes each read their own group's pair qi touches 28
// lines instead of 224.  Piece k of pair qi of lane l of a tile lies at
// ((base + qi) * kTileRec + k) * 32 + l.
constexpr int kTileRec = 7;   // 16-byte pieces of a record
__device__ __forceinline__ PairView load_tile(const double2* __restrict__ tile, int at, int lane) {
  return pair_view(tile + (size_t)at * (kTileRec * 32) + lane, 32);
}

__device__ __forceinline__ double pair_bound(const PairRec* __restrict__ rec, int t) {
  return __ldg(&rec[t].schwarz);
}

struct MolLaunch {
  PairArrays pairs;
  const PairRec* rec;     // the sorted pairs as records
  const int* prim;        // shell components -> primitive
  const int* stidx;       // shell x component -> target row (-1: none)
  const double* scoef;    // shell x component -> coefficient
  const double* boys;     // table rows (boys_tab)
  const double* down;     // the table of boys_down
  const double* dt;       // density in target space (nt x nt, column-major)
  double* jt;             // J' targets (nt x nt)
  double* kt;             // K' targets
  const int* gr_start;    // group -> first pair
  const int* gr_n;        // group -> number of pairs
  const double* gr_max;   // group -> largest bound
  const int* bk_list;     // ket groups by (class, bucket, group)
  const double2* tile;    // their records by tile (load_tile)
  const int* tile_at;     // list position of a tile's first group -> base of the tile
  const int* blk;         // shell -> contracted block
  const int* tblk;        // target -> contracted block (-1: none)
  const double* bmax;     // block-pair maxima of |P_T| (density screening / mixed precision)
  int nblk;
  double dtol;            // skip quartets with bound * max|P| < dtol (0: the reference's screen only)
  double mcut;            // FP32 recursion where bound * max|P| < mcut (0: FP64 only)
  unsigned long long* n32;  // quartets run in FP32
  const Chunk* chunks;    // costliest first
  const int* nchunks;
  int* queue;             // chunk counters (one per pass), zero at launch: warps take chunks in order
  double inttol;
  int nt;
  int myid, numprocs;
  const MolLaunch* insts;   // batches: the launch record of every instance (Chunk::inst), else null
  int own_boys;             // batches: the instances' Boys tables differ (set up with different IGAMMA)
  int lower_kept_bits;      // bit L: some shell of top L has a coefficient on a lower component
  // block panels (pfe_context): the density and the J', K' accumulators of the
  // digestion kernels, and the panel row where a shell's block begins
  const double* pd;
  double* pj;
  double* pk;
  const int* poff;
  const int* ptgt;        // panel row -> target (-1: none)
  int np;                 // panel rows
  int num_sms;
  // one tile of a straight-line class: tickets [t0, t0 + tn) of this rank's chunks; X of
  // ticket t0 + t at xbuf + t * (kept integrals) * 32, xlive[t] set when it holds any quartet
  int t0, tn;
  unsigned long long live;   // register passes launched (live_passes)
  double* xbuf;
  unsigned char* xlive;
};

// The launch record of a set-up molecular context for target-space density d_dt.
MolLaunch molecular_launch(pfe_context* ctx, const double* d_dt);

// max|P_T| over the six density blocks a group quartet's digestion reads
__device__ __forceinline__ double quartet_pmax(const MolLaunch& ql, int I, int J, int K, int L) {
  const int bI = ql.blk[I], bJ = ql.blk[J], bK = ql.blk[K], bL = ql.blk[L], nb = ql.nblk;
  const double* bm = ql.bmax;
  return fmax(fmax(fmax(bm[bI * nb + bJ], bm[bK * nb + bL]), fmax(bm[bI * nb + bK], bm[bI * nb + bL])),
              fmax(bm[bJ * nb + bK], bm[bJ * nb + bL]));
}

// Screening threshold on Schwarz(ij)*Schwarz(kl) of a group quartet: the
// reference's INTTOL, raised to dtol/max|P| under density screening.
__device__ __forceinline__ double quartet_threshold(const MolLaunch& ql, double pmax) {
  if (ql.dtol <= 0.0) return ql.inttol;
  return pmax > 0.0 ? fmax(ql.inttol, ql.dtol / pmax) : INFINITY;
}

// Primitive-quartet integrals in FP64, or in FP32 from Boys values and geometry
// computed in FP64 (the recursion is linear in F: it runs on F/pref, and the
// outputs are scaled by pref in FP64, so FP32 sees values of order one).
template <typename R, int LA, int LB, int LC, int LD>
__device__ __forceinline__ void eri_prec(const double* F, double pref, const EriGeom<double>& g, double* out) {
  constexpr int NI = ncum(LA) * ncum(LB) * ncum(LC) * ncum(LD);
  constexpr int LT = LA + LB + LC + LD;
  if constexpr (sizeof(R) == sizeof(double)) {
    eri_dispatch<LA, LB, LC, LD>(F, g, out);
  } else {
    float Ff[LT + 1];
#pragma unroll
    for (int m = 0; m <= LT; ++m) Ff[m] = (float)F[m];
    EriGeom<float> gf;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      gf.PA[k] = (float)g.PA[k]; gf.WP[k] = (float)g.WP[k]; gf.QC[k] = (float)g.QC[k];
      gf.WQ[k] = (float)g.WQ[k]; gf.AB[k] = (float)g.AB[k]; gf.CD[k] = (float)g.CD[k];
    }
    gf.oz = (float)g.oz; gf.oe = (float)g.oe; gf.oze = (float)g.oze; gf.roz = (float)g.roz; gf.roe = (float)g.roe;
    float of[NI];
    eri_dispatch<LA, LB, LC, LD>(Ff, gf, of);
#pragma unroll
    for (int i = 0; i < NI; ++i) out[i] = pref * (double)of[i];
  }
}

// ------------------------------------------------------------------ digestion helpers

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void add_target(double* __restrict__ M, int nt, int r, int c, double v) {
  if (r >= 0 && c >= 0 && v != 0.0) atomicAdd(M + r + (size_t)nt * c, v);
}

__device__ __forceinline__ double dt_at(const double* __restrict__ D, int nt, int i, int j) {
  return (i >= 0 && j >= 0) ? __ldg(D + i + (size_t)nt * j) : 0.0;
}

// ------------------------------------------------------------------ straight-line classes

// One group quartet per lane: the warp shares the bra group, each lane owns one
// ket group of the chunk.  X(abcd) of the lane's group quartet stays in
// registers; the bra's primitive pairs are walked in step by the whole warp.
// Classes with more integrals than registers hold X in NPASS launches, pass
// PASS keeping the bra components ab in [AB0, AB1) (the recursion is repeated
// per pass; the outputs a pass does not keep are dead code in it).  X then goes to
// memory and is digested once per group quartet by the class's digestion kernel
// (pfe_mol_digest.cu).
// Angular momentum of component i of a cumulative shell, in the reference's
// component order (x power outer, z power inner: s, z, zz, y, yz, yy, x, xz, xy, xx).
__host__ __device__ constexpr int comp_tot(int L, int i) {
  return L == 0 ? 0 : (L == 1 ? (i == 0 ? 0 : 1) : (i == 0 ? 0 : (i == 1 || i == 3 || i == 6) ? 1 : 2));
}

// Position of component i among its shell's components ordered by |i| (stable): the
// order of the panel rows and of the stored integrals.
__host__ __device__ constexpr int comp_rank(int L, int i) {
  int r = 0;
  for (int k = 0; k < ncum(L); ++k)
    if (comp_tot(L, k) < comp_tot(L, i) || (comp_tot(L, k) == comp_tot(L, i) && k < i)) ++r;
  return r;
}

// Components a shell of top L keeps: all of them where some shell of that L has a
// coefficient below its top level (bit L of the lower_kept bits), else the top level,
// which comes last in the order.
__host__ __device__ constexpr int kept_first(int L, int bits) { return (L == 0 || ((bits >> L) & 1)) ? 0 : ncum(L - 1); }
__host__ __device__ constexpr int kept_n(int L, int bits) { return ncum(L) - kept_first(L, bits); }

// Bra component pairs ab = a*NB + b ordered by (|a|, |b|): the passes of a
// class then keep the lower (for pure shells coefficient-free) components
// together, and such passes skip their chunks.
__host__ __device__ constexpr void ab_order_fill(int LA, int LB, int* ab, int* pos) {
  const int NB = ncum(LB), N = ncum(LA) * NB;
  for (int i = 0; i < N; ++i) ab[i] = i;
  for (int i = 1; i < N; ++i)   // stable insertion sort by (|a|, |b|)
    for (int j = i; j > 0; --j) {
      const int x = ab[j - 1], y = ab[j];
      const int kx = comp_tot(LA, x / NB) * 8 + comp_tot(LB, x % NB);
      const int ky = comp_tot(LA, y / NB) * 8 + comp_tot(LB, y % NB);
      if (kx <= ky) break;
      ab[j - 1] = y;
      ab[j] = x;
    }
  for (int i = 0; i < N; ++i) pos[ab[i]] = i;
}

template <int LA, int LB>
struct AbOrder {
  static constexpr int NA = ncum(LA), NB = ncum(LB), N = NA * NB;
  int ab[N];    // k-th pair
  int pos[N];   // position of pair ab
  __host__ __device__ constexpr AbOrder() : ab(), pos() { ab_order_fill(LA, LB, ab, pos); }
};

// Bra component pairs below the top level (|a| < LA or |b| < LB): in AbOrder
// they come first.
__host__ __device__ constexpr int lower_pairs(int LA, int LB) {
  int c = 0;
  for (int a = 0; a < ncum(LA); ++a)
    for (int b = 0; b < ncum(LB); ++b)
      if (comp_tot(LA, a) < LA || comp_tot(LB, b) < LB) ++c;
  return c;
}

// The bra component pairs [ab0, ab1) (positions in AbOrder) register pass `pass`
// of `npass` keeps.  Two-pass (d s| classes split at the level boundary: the
// lower components of the d shell first, the top-level ones second, so that a
// pure d shell (lower components coefficient-free) skips the first pass entirely.
__host__ __device__ constexpr void pass_range(int LA, int LB, int LC, int LD, int npass, int pass, int& ab0, int& ab1) {
  const int NAB = ncum(LA) * ncum(LB), NCD = ncum(LC) * ncum(LD);
  const int abp = (NAB + npass - 1) / npass;
  const int nlow = lower_pairs(LA, LB);
  const bool lsplit = npass == 2 && LA == 2 && LB == 0 && nlow * NCD <= 40 && (NAB - nlow) * NCD <= 40;
  ab0 = lsplit ? (pass == 0 ? 0 : nlow) : pass * abp;
  ab1 = lsplit ? (pass == 0 ? nlow : NAB) : ((ab0 + abp < NAB) ? ab0 + abp : NAB);
}

// The angular momenta a class has, as lower_kept bits: KEPT of its general variant, which
// keeps every component.
__host__ __device__ constexpr int class_bits(int LA, int LB, int LC, int LD) {
  return ((LA == 1 || LB == 1 || LC == 1 || LD == 1) ? 2 : 0) | ((LA == 2 || LB == 2 || LC == 2 || LD == 2) ? 4 : 0);
}

// The variant of a class's passes for a molecule's lower_kept bits: where the d shells (or,
// without d shells in the class, the p shells) are pure, one that holds only the kept
// components of all four shells in X, so that more integrals fit a pass and the recursion
// runs less often ((21|21) of 6-31G**: 12 passes of 48 kept integrals for 24 of 40 with the
// ket's ghosts among them); else the general one.
__host__ __device__ constexpr int pass_variant(int LA, int LB, int LC, int LD, int bits) {
  const int mask = class_bits(LA, LB, LC, LD), r = bits & mask;
  return (mask & 4) ? ((r & 4) ? mask : r) : r;
}

// Register passes of a variant: kPassIntegrals kept integrals each.
constexpr int kPassIntegrals = 48;
__host__ __device__ constexpr int kept_pairs_per_pass(int LC, int LD, int KEPT) {
  return kPassIntegrals / (kept_n(LC, KEPT) * kept_n(LD, KEPT)) > 0
             ? kPassIntegrals / (kept_n(LC, KEPT) * kept_n(LD, KEPT)) : 1;
}
__host__ __device__ constexpr int variant_passes(int LA, int LB, int LC, int LD, int KEPT, int npass_general) {
  if (KEPT == class_bits(LA, LB, LC, LD)) return npass_general;
  const int per = kept_pairs_per_pass(LC, LD, KEPT);
  return (kept_n(LA, KEPT) * kept_n(LB, KEPT) + per - 1) / per;
}

// The register passes of a class's general variant that keep a bra component pair that can carry a
// coefficient (bit p of the mask): a component below its shell's top level has none
// unless bit L of lower_kept_bits is set (the kernel skips such chunks anyway; a pass
// that keeps none of them is not launched at all).
inline unsigned long long live_passes(int LA, int LB, int LC, int LD, int npass, int lower_kept_bits) {
  int ab[MAXCOMP * MAXCOMP] = {}, pos[MAXCOMP * MAXCOMP] = {};
  ab_order_fill(LA, LB, ab, pos);
  const int NB = ncum(LB);
  unsigned long long live = 0;
  for (int p = 0; p < npass; ++p) {
    int ab0 = 0, ab1 = 0;
    pass_range(LA, LB, LC, LD, npass, p, ab0, ab1);
    for (int k = ab0; k < ab1; ++k) {
      const int a = ab[k] / NB, b = ab[k] % NB;
      const bool ka = comp_tot(LA, a) == LA || ((lower_kept_bits >> LA) & 1);
      const bool kb = comp_tot(LB, b) == LB || ((lower_kept_bits >> LB) & 1);
      if (ka && kb) live |= 1ull << p;
    }
  }
  return npass == 1 ? 1ull : live;
}

// Resident blocks of 128 threads the register allocation aims at.  The kernels wait on
// loads more than on the FP64 pipe, so a block more is worth some spilling as long as the
// recursion's temporaries are few: measured per class on C20H42 and the water batch,
// (11|10) 2.89 -> 2.45 ms, (20|10) 1.03 -> 0.87, (11|11) 2.11 -> 1.93 and (21|00) 0.48 -> 0.44
// at three blocks (168 registers) against two; four cost (11|10) and (21|10) 15 %.  Above a
// total of 4 the 255 registers of two blocks are better ((21|11), (21|20), (22|11): 5-10 %).
// (10|00) gains 5 % at five blocks, (10|10) and (11|00) lose 10-20 % there.  The classes up
// to a total of 2 hold the same warps in two blocks, each with its copy of the Boys rows in
// shared memory, on a grid of resident blocks.
// OWN: a batch whose instances were set up with different IGAMMA, for which no one copy is
// right, reads each instance's rows from global memory.
template <int LA, int LB, int LC, int LD, bool OWN = false>
struct GqOccupancy {
  static constexpr int LT = LA + LB + LC + LD;
  static constexpr bool staged = DownSmem<LT>::use && !OWN;
  static constexpr int threads = staged ? (LT <= 1 ? 320 : 256) : 128;
  static constexpr int blocks = staged ? 2 : (LT <= 4 ? 3 : 1);
};

template <int LA, int LB, int LC, int LD, int KEPT, int NPASS, int PASS, bool MIXED, bool BATCH, bool OWN>
__device__ __forceinline__ void gq_pass(const MolLaunch& lq, const double2* s_boys) {
  constexpr int NA = ncum(LA), NB = ncum(LB), NC = ncum(LC), ND = ncum(LD);
  constexpr int NI = NA * NB * NC * ND;
  constexpr int NCD = NC * ND;
  constexpr int LT = LA + LB + LC + LD;
  constexpr bool GENERAL = KEPT == class_bits(LA, LB, LC, LD);
  constexpr AbOrder<LA, LB> ORD{};
  // the kept bra component pairs are the last of AbOrder (both shells' top levels, or the
  // d shell's with all of the other's)
  constexpr int NKP = kept_n(LA, KEPT) * kept_n(LB, KEPT), KP0 = NA * NB - NKP;
  constexpr int FC = kept_first(LC, KEPT), FD = kept_first(LD, KEPT);
  constexpr int NDK = kept_n(LD, KEPT), NCDK = kept_n(LC, KEPT) * NDK;
  // the pass keeps the kept pairs [AB0, AB1); X(k, cd) is that of pair AB0 + k
  constexpr int AB0 = [] {
    int a = PASS * kept_pairs_per_pass(LC, LD, KEPT), b = 0;
    if (GENERAL) pass_range(LA, LB, LC, LD, NPASS, PASS, a, b);
    return a;
  }();
  constexpr int AB1 = [] {
    int a = 0, b = (PASS + 1) * kept_pairs_per_pass(LC, LD, KEPT);
    if (GENERAL) pass_range(LA, LB, LC, LD, NPASS, PASS, a, b);
    return b < NKP ? b : NKP;
  }();
  constexpr int XN = (AB1 - AB0) * NCDK;
  static_assert(AB0 < NKP, "every pass keeps at least one bra component pair");
  // pair k's component pair, and the kept position of ket component pair (cc, d), or -1
  auto ab_of = [&](int k) { return ORD.ab[KP0 + k]; };
  auto cd_at = [&](int cc, int d) {
    const int rc = comp_rank(LC, cc) - FC, rd = comp_rank(LD, d) - FD;
    return (rc < 0 || rd < 0) ? -1 : rc * NDK + rd;
  };
  const int lane = threadIdx.x & 31;
  const int nchunks = *lq.nchunks;
  const double c2pi = 2.0 / sqrt(REF_PI);
  // the warp takes the next chunk of this rank's share (every numprocs-th,
  // starting at myid) from the pass's work queue: chunks are sorted costliest
  // first, so the launch ends with the cheap ones
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(lq.queue + PASS, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    const int c = (lq.t0 + t) * lq.numprocs + lq.myid;
    if (t >= lq.tn || c >= nchunks) break;
    const Chunk ch = lq.chunks[c];
    // this chunk's instance: batches read its launch record from global memory
    const MolLaunch& ql = [&]() -> const MolLaunch& {
      if constexpr (BATCH) return lq.insts[ch.inst];
      else return lq;
    }();
    // the tables the loops read, held in registers (ql may live in global memory)
    const PairRec* __restrict__ rec = ql.rec;
    const double* __restrict__ scoef = ql.scoef;
    const double* __restrict__ down = ql.down;
    const int* __restrict__ stidx = ql.stidx;
    const double mcut = ql.mcut;
    const int nt = ql.nt;
    const int G = ch.G;
    const int g0 = ql.gr_start[G];
    const int2 ijg = __ldg(reinterpret_cast<const int2*>(&rec[g0].si));
    if constexpr (NPASS > 1) {
      // a pass whose bra components all lack a coefficient (the lower components of a
      // pure d or p shell) contributes nothing: skip the chunk (warp-uniform)
      bool live = false;
#pragma unroll
      for (int k = AB0; k < AB1; ++k)
        live = live || (stidx[ijg.x * MAXCOMP + ab_of(k) / NB] >= 0 && stidx[ijg.y * MAXCOMP + ab_of(k) % NB] >= 0);
      if (!live) continue;
    }
    const int li = ch.first + lane;
    const bool act = li < ch.end;
    const int H = ql.bk_list[act ? li : ch.first];
    const int h0 = ql.gr_start[H], hn = act ? min(ql.gr_n[H], ch.q1) : 0;
    const bool dens = ql.dtol > 0.0 || ql.mcut > 0.0;
    const int2 klh = __ldg(reinterpret_cast<const int2*>(&rec[h0].si));
    const double pmax = dens ? quartet_pmax(ql, ijg.x, ijg.y, klh.x, klh.y) : 0.0;
    const double thr = quartet_threshold(ql, pmax);
    unsigned n32 = 0;
    bool any = false;   // this lane evaluated a quartet
    double X[XN];
#pragma unroll
    for (int i = 0; i < XN; ++i) X[i] = 0.0;
    const double gmax = pair_bound(rec, g0 + ch.p0);   // the largest of this piece (bounds descend)
    // Each lane walks its own ket group's pairs (outer loop, one gather of the ket
    // record per pair); the warp walks the bra group's pairs in step (inner loop:
    // every lane reads the same bra record, one L1 wavefront per load).  Both
    // lists are sorted by Schwarz bound, so the screens end the loops.
    const double2* __restrict__ tile = ql.tile;
    const int tile0 = ql.tile_at[ch.first];
    for (int qi = ch.q0;; ++qi) {
      const bool lv = qi < hn;
      if (!__any_sync(0xffffffffu, lv)) break;   // past the tile's longest group
      const int q = h0 + qi;
      const PairView kq = load_tile(tile, tile0 + qi, lane);
      const double sq = lv ? kq.bound : 0.0;
      const bool qok = lv && sq * gmax >= thr;
      if (!__any_sync(0xffffffffu, qok)) break;
      const double ze = kq.zeta;
      const double Qx = kq.P[0], Qy = kq.P[1], Qz = kq.P[2];
      const double Sq = kq.S;
      const int K = kq.si, L = kq.sj;
      const double wKL = (K != L) ? 2.0 : 1.0;
      // ket coefficients: products held when small, factors otherwise
      constexpr bool HOLD = NCDK <= 16;
      double ccd[HOLD ? NCDK : 1];
      double sK[NC], sL[ND];
#pragma unroll
      for (int cc = 0; cc < NC; ++cc) sK[cc] = scoef[K * MAXCOMP + cc];
#pragma unroll
      for (int d = 0; d < ND; ++d) sL[d] = scoef[L * MAXCOMP + d];
      if constexpr (HOLD) {
#pragma unroll
        for (int cc = 0; cc < NC; ++cc)
#pragma unroll
          for (int d = 0; d < ND; ++d)
            if (cd_at(cc, d) >= 0) ccd[cd_at(cc, d)] = wKL * sK[cc] * sL[d];
      }
      for (int p = g0 + ch.p0; p < g0 + ch.p1; ++p) {
        const PairView bp = load_pair(rec, p);
        const double sp = bp.bound;
        const bool pass = qok && sp * sq >= thr;
        if (!__any_sync(0xffffffffu, pass)) break;   // later bra pairs fail for every lane
        // a group paired with itself: each unordered pair of pairs once (p >= q)
        if (!pass || (G == H && p < q)) continue;
        const int I = bp.si, J = bp.sj;
        const double zb = bp.zeta;
        const double Px = bp.P[0], Py = bp.P[1], Pz = bp.P[2];
        const double zz = zb + ze;
        // one reciprocal per primitive quartet; 1/(2 zeta) of either pair comes with its record
        const double rzz = 1.0 / zz;
        const double rho = zb * ze * rzz;
        const double dx = Px - Qx, dy = Py - Qy, dz = Pz - Qz;
        const double T = rho * (dx * dx + dy * dy + dz * dz);
        const double pref = c2pi * bp.S * Sq * sqrt(rho);
        // FP32 only when every lane running this step qualifies
        bool f32 = false;
        if constexpr (MIXED && LT > 0) f32 = __all_sync(__activemask(), sp * sq * pmax < mcut);
        n32 += f32 ? 1u : 0u;
        double F[LT + 1];
        boys_down<LT, GqOccupancy<LA, LB, LC, LD, OWN>::staged>(T, f32 ? 1.0 : pref, down, F, s_boys);
        double out[NI];
        if constexpr (LT == 0) {
          out[0] = F[0];
        } else {
          EriGeom<double> g;
          const double Wx = (zb * Px + ze * Qx) * rzz, Wy = (zb * Py + ze * Qy) * rzz, Wz = (zb * Pz + ze * Qz) * rzz;
          g.PA[0] = bp.PA[0]; g.PA[1] = bp.PA[1]; g.PA[2] = bp.PA[2];
          g.QC[0] = kq.PA[0]; g.QC[1] = kq.PA[1]; g.QC[2] = kq.PA[2];
          g.AB[0] = bp.AB[0]; g.AB[1] = bp.AB[1]; g.AB[2] = bp.AB[2];
          g.CD[0] = kq.AB[0]; g.CD[1] = kq.AB[1]; g.CD[2] = kq.AB[2];
          g.WP[0] = Wx - Px; g.WP[1] = Wy - Py; g.WP[2] = Wz - Pz;
          g.WQ[0] = Wx - Qx; g.WQ[1] = Wy - Qy; g.WQ[2] = Wz - Qz;
          g.oz = bp.oz; g.oe = kq.oz; g.oze = 0.5 * rzz; g.roz = ze * rzz; g.roe = zb * rzz;
          if constexpr (MIXED) {
            if (f32) eri_prec<float, LA, LB, LC, LD>(F, pref, g, out);
            else eri_prec<double, LA, LB, LC, LD>(F, pref, g, out);
          } else {
            eri_prec<double, LA, LB, LC, LD>(F, pref, g, out);
          }
        }
        any = true;
        const double w = ((I != J) ? 2.0 : 1.0) * ((p != q) ? 2.0 : 1.0);
#pragma unroll
        for (int k = AB0; k < AB1; ++k) {
          const double ca = w * scoef[I * MAXCOMP + ab_of(k) / NB] * scoef[J * MAXCOMP + ab_of(k) % NB];
#pragma unroll
          for (int cc = 0; cc < NC; ++cc) {
            double cb;
            if constexpr (HOLD) cb = ca;
            else cb = ca * (wKL * sK[cc]);
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              const int j = cd_at(cc, d);
              if (j < 0) continue;
              const double c4 = HOLD ? cb * ccd[HOLD ? j : 0] : cb * sL[d];
              const int x = (k - AB0) * NCDK + j;
              X[x] = fma(c4, out[ab_of(k) * NCD + cc * ND + d], X[x]);
            }
          }
        }
      }
    }
    if (MIXED && PASS == 0) {
      unsigned long long n = n32;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
      if (lane == 0 && n) atomicAdd(ql.n32, n);
    }
    if (!__any_sync(0xffffffffu, any)) continue;   // nothing passed the screens in this chunk
    if constexpr (LT == 0) {
      // one integral per lane: digested here against the target-space density
      const double* __restrict__ D = ql.dt;
      const int ta = stidx[ijg.x * MAXCOMP], tb = stidx[ijg.y * MAXCOMP];
      const int tc = stidx[klh.x * MAXCOMP], td = stidx[klh.y * MAXCOMP];
      const double v = warp_sum(dt_at(D, nt, tc, td) * X[0]);   // the bra is the warp's
      if (lane == 0) add_target(ql.jt, nt, ta, tb, 0.25 * v);
      if (act && any) {
        add_target(ql.jt, nt, tc, td, 0.25 * dt_at(D, nt, ta, tb) * X[0]);
        add_target(ql.kt, nt, ta, td, 0.125 * dt_at(D, nt, tb, tc) * X[0]);
        add_target(ql.kt, nt, ta, tc, 0.125 * dt_at(D, nt, tb, td) * X[0]);
        add_target(ql.kt, nt, tb, td, 0.125 * dt_at(D, nt, ta, tc) * X[0]);
        add_target(ql.kt, nt, tb, tc, 0.125 * dt_at(D, nt, ta, td) * X[0]);
      }
    } else {
      // this pass's part of X to the digestion kernel: the kept components, one
      // coalesced 256-byte row per integral
      const int bits = GENERAL ? lq.lower_kept_bits : KEPT;
      const int fa = kept_first(LA, bits), fb = kept_first(LB, bits), fc = kept_first(LC, bits),
                fd = kept_first(LD, bits);
      const int nb = NB - fb, nc = NC - fc, nd = ND - fd;
      double* __restrict__ xb = lq.xbuf + (size_t)t * ((size_t)(NA - fa) * nb * nc * nd * 32) + lane;
#pragma unroll
      for (int k = AB0; k < AB1; ++k) {
        const int ra = comp_rank(LA, ab_of(k) / NB) - fa, rb = comp_rank(LB, ab_of(k) % NB) - fb;
        if (ra < 0 || rb < 0) continue;
#pragma unroll
        for (int cc = 0; cc < NC; ++cc)
#pragma unroll
          for (int d = 0; d < ND; ++d) {
            const int rc = comp_rank(LC, cc) - fc, rd = comp_rank(LD, d) - fd;
            if (rc < 0 || rd < 0 || cd_at(cc, d) < 0) continue;
            xb[(((ra * nb + rb) * nc + rc) * nd + rd) * 32] = X[(k - AB0) * NCDK + cd_at(cc, d)];
          }
      }
      if (lane == 0) lq.xlive[t] = 1;
    }
  }
}

// Digestion of the stored X of a class's tile (pfe_mol_digest.cu), after its passes.
void launch_digest(int cb, int ck, const MolLaunch& ql, int num_sms, cudaStream_t s);

// ------------------------------------------------------------------ launch tables

// Register passes per kernel: the live ones of a group run side by side in one launch
// (blockIdx.y), so that their tails overlap and a small molecule's build is not
// launch-bound.
constexpr int kPassGroup = 8;

template <int LA, int LB, int LC, int LD, int KEPT, int NPASS, int P0, int PN, bool MIXED, bool BATCH, bool OWN>
__device__ __forceinline__ void gq_select(const MolLaunch& lq, int p, const double2* s_boys) {
  if constexpr (PN == 1) {
    gq_pass<LA, LB, LC, LD, KEPT, NPASS, P0, MIXED, BATCH, OWN>(lq, s_boys);
  } else {
    if (p == P0) gq_pass<LA, LB, LC, LD, KEPT, NPASS, P0, MIXED, BATCH, OWN>(lq, s_boys);
    else gq_select<LA, LB, LC, LD, KEPT, NPASS, P0 + 1, PN - 1, MIXED, BATCH, OWN>(lq, p, s_boys);
  }
}

// Passes P0 .. P0 + PN - 1; blockIdx.y is the position among the live ones (bits of live).
template <int LA, int LB, int LC, int LD, int KEPT, int NPASS, int P0, int PN, bool MIXED, bool BATCH, bool OWN>
__global__ void __launch_bounds__(GqOccupancy<LA, LB, LC, LD, OWN>::threads, GqOccupancy<LA, LB, LC, LD, OWN>::blocks)
    k_gq(const __grid_constant__ MolLaunch lq, unsigned int live) {
  extern __shared__ double2 s_boys[];
  if constexpr (GqOccupancy<LA, LB, LC, LD, OWN>::staged) {   // once per resident block
    down_stage<LA + LB + LC + LD>(lq.down, s_boys);
    __syncthreads();
  }
  unsigned int m = live;
  for (int y = blockIdx.y; y > 0; --y) m &= m - 1;
  gq_select<LA, LB, LC, LD, KEPT, NPASS, P0, PN, MIXED, BATCH, OWN>(lq, P0 + __ffs(m) - 1, s_boys);
}

using LaunchFn = void (*)(const MolLaunch&, int grid, cudaStream_t);

template <int LA, int LB, int LC, int LD, int KEPT, int NPASS, int P0, bool MIXED, bool BATCH, bool OWN = false>
void launch_groups(const MolLaunch& ql, unsigned long long live, int grid, cudaStream_t s) {
  constexpr int PN = NPASS - P0 < kPassGroup ? NPASS - P0 : kPassGroup;
  using O = GqOccupancy<LA, LB, LC, LD, OWN>;
  if constexpr (BATCH && O::staged) {
    if (ql.own_boys) return launch_groups<LA, LB, LC, LD, KEPT, NPASS, P0, MIXED, BATCH, true>(ql, live, grid, s);
  }
  const unsigned int m = (unsigned int)(live >> P0) & ((1u << PN) - 1);
  if (m) {
    auto kern = k_gq<LA, LB, LC, LD, KEPT, NPASS, P0, PN, MIXED, BATCH, OWN>;
    constexpr size_t bytes = O::staged ? DownSmem<O::LT>::BYTES : 0;
    // `grid` counts blocks of four warps
    int g = grid;
    if constexpr (O::staged) {
      note(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
      g = std::max(1, std::min((grid * 128 + O::threads - 1) / O::threads, O::blocks * ql.num_sms));
    }
    kern<<<dim3(g, __builtin_popcount(m)), O::threads, bytes, s>>>(ql, m);
    note_launch();
  }
  if constexpr (P0 + PN < NPASS)
    launch_groups<LA, LB, LC, LD, KEPT, NPASS, P0 + PN, MIXED, BATCH, OWN>(ql, live, grid, s);
}

// A variant that holds the kept components only (KEPT: 0 or 2); those of the large
// classes are instantiated in units of their own (pfe_mol_kept*.cu).
template <int LA, int LB, int LC, int LD, int KEPT, bool MIXED, bool BATCH>
void launch_kept(const MolLaunch& ql, int grid, cudaStream_t s) {
  launch_groups<LA, LB, LC, LD, KEPT, variant_passes(LA, LB, LC, LD, KEPT, 0), 0, MIXED, BATCH>(ql, ql.live, grid, s);
}
#define PFE_KEPT(A, B, C, D, WORD)                                                            \
  WORD template void launch_kept<A, B, C, D, 0, false, false>(const MolLaunch&, int, cudaStream_t); \
  WORD template void launch_kept<A, B, C, D, 0, false, true>(const MolLaunch&, int, cudaStream_t);  \
  WORD template void launch_kept<A, B, C, D, 2, false, false>(const MolLaunch&, int, cudaStream_t); \
  WORD template void launch_kept<A, B, C, D, 2, false, true>(const MolLaunch&, int, cudaStream_t);
#ifndef PFE_KEPT_UNIT
PFE_KEPT(2, 1, 1, 1, extern)
PFE_KEPT(2, 1, 2, 0, extern)
PFE_KEPT(2, 1, 2, 1, extern)
PFE_KEPT(2, 2, 1, 0, extern)
PFE_KEPT(2, 2, 1, 1, extern)
PFE_KEPT(2, 2, 2, 0, extern)
#endif

template <int LA, int LB, int LC, int LD, int NPASS, bool MIXED, bool BATCH = false>
void launch_q(const MolLaunch& ql, int grid, cudaStream_t s) {
  static_assert(NPASS <= 64, "a bit per pass");
  constexpr int ALL = class_bits(LA, LB, LC, LD);
  const int kept = pass_variant(LA, LB, LC, LD, ql.lower_kept_bits);
  if constexpr (ALL != 0) {
    if (kept == 0) return launch_kept<LA, LB, LC, LD, 0, MIXED, BATCH>(ql, grid, s);
  }
  if constexpr (ALL == 6) {
    if (kept == 2) return launch_kept<LA, LB, LC, LD, 2, MIXED, BATCH>(ql, grid, s);
  }
  launch_groups<LA, LB, LC, LD, ALL, NPASS, 0, MIXED, BATCH>(ql, ql.live, grid, s);
}

// Kernels launch_q launches for a class (groups with a live pass).
inline int pass_groups(int npass, unsigned long long live) {
  int n = 0;
  for (int p0 = 0; p0 < npass; p0 += kPassGroup) n += ((live >> p0) & ((1ull << kPassGroup) - 1)) ? 1 : 0;
  return n;
}

// Register passes per straight-line class's general variant; must match the table below.
static inline int straight_npass(int cb, int ck) {
  static const int np[6][6] = {{1, 0, 0, 0, 0, 0}, {1, 1, 0, 0, 0, 0}, {1, 2, 8, 0, 0, 0},
                               {2, 2, 5, 3, 0, 0}, {1, 4, 14, 10, 40, 0}, {3, 10, 50, 25, 0, 0}};
  return np[cb][ck];
}

// straight-line classes and their passes (X of at most 40 integrals per pass)
template <bool MIXED, bool BATCH = false>
static LaunchFn straight_launcher_t(int cb, int ck) {
#define Q(A, B, C, D, P) &launch_q<A, B, C, D, P, MIXED, BATCH>
  static const LaunchFn table[6][6] = {
      {Q(0, 0, 0, 0, 1), nullptr, nullptr, nullptr, nullptr, nullptr},
      {Q(1, 0, 0, 0, 1), Q(1, 0, 1, 0, 1), nullptr, nullptr, nullptr, nullptr},
      {Q(1, 1, 0, 0, 1), Q(1, 1, 1, 0, 2), Q(1, 1, 1, 1, 8), nullptr, nullptr, nullptr},
      {Q(2, 0, 0, 0, 2), Q(2, 0, 1, 0, 2), Q(2, 0, 1, 1, 5), Q(2, 0, 2, 0, 3), nullptr, nullptr},
      {Q(2, 1, 0, 0, 1), Q(2, 1, 1, 0, 4), nullptr, nullptr, nullptr, nullptr},
      {Q(2, 2, 0, 0, 3), nullptr, nullptr, nullptr, nullptr, nullptr}};
#undef Q
  return table[cb][ck];
}

// The large classes' FP64 passes, one translation unit each (pfe_mol_big*.cu)
// so that they compile in parallel; `batch`: the instantiations for batches.
LaunchFn straight_launcher_big(int cb, int ck, bool batch = false);

}  // namespace pfe
