// Two-electron part of the nuclear gradient of a molecule: the work of
// FOURINDEX_ERI_GRADIENT (src/pfourindexgradient.f90:1-1478, molecular branch).
//
// For a fixed density P (target space: contracted functions, or primitives
// under a general contraction) the two-electron energy is
//   E2 = 1/2 sum (ij|kl) P_ij P_kl  -  HFX/4 sum (ij|kl) P_ik P_jl
// and its derivative with respect to the centre A of primitive i follows from
// d/dA_x phi_a = 2 zeta_a phi_{a+1x} - a_x phi_{a-1x} (the reference's
// FN = 2 ZT(II) ERI(UP1) - 2 DOWN1_C ERI(DOWN1), :1353-1361); the derivative
// with respect to B is minus the sum of the other three (translational
// invariance, as the reference forms its J-atom force, :1396-1398).  The
// J part and the K part are returned apart (the caller weighs K by HFX):
//   grad_J = 1/2 sum' w P_ab P_cd d(ab|cd)
//   grad_K = -1/8 sum' w (P_ac P_bd + P_ad P_bc) d(ab|cd)
// over the unique primitive quartets with their 8-fold degeneracy w and the
// contraction coefficients of each component, the quartets and screening of
// the Fock build (the same chunk lists).
//
// The derivative integrals come from three op tables per class, each with one
// centre raised by one (A, C, D: opg_<class>_a/c/d, generated next to the
// Fock tables), evaluated one primitive quartet per team with the slots in shared
// memory.  A team is a warp where the tables are small enough for several per SM
// (most quartets are of classes with few operations, whose levels a block spends on
// barriers), else a block of 256 threads; it takes one group quartet at a time,
// contracts the derivatives against the density blocks and adds twelve numbers (three
// per centre) to the atoms' gradients.

#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "pfe_common.cuh"
#include "pfe_context.cuh"
#include "pfe_interp.cuh"
#include "pfe_mol_kernels.cuh"
#include "generated/eri_grad_tables.cuh"

namespace pfe {

namespace {

// Index maps of a cumulative shell's components under x/y/z raising and
// lowering: comps(L) in the reference's order (x power outer, z inner), the
// raised/lowered component's index in comps(L+1) (-1: none), and the power.
struct GradMaps {
  signed char up[3][10][3], dn[3][10][3], pw[3][10][3];
};

constexpr int comp_index(int L, int px, int py, int pz) {
  int n = 0;
  for (int i1 = 0; i1 <= L; ++i1)
    for (int i2 = 0; i2 <= L - i1; ++i2)
      for (int i3 = 0; i3 <= L - i1 - i2; ++i3) {
        if (i1 == px && i2 == py && i3 == pz) return n;
        ++n;
      }
  return -1;
}

constexpr GradMaps make_maps() {
  GradMaps m{};
  for (int L = 0; L < 3; ++L) {
    int n = 0;
    for (int i1 = 0; i1 <= L; ++i1)
      for (int i2 = 0; i2 <= L - i1; ++i2)
        for (int i3 = 0; i3 <= L - i1 - i2; ++i3, ++n) {
          const int p[3] = {i1, i2, i3};
          for (int x = 0; x < 3; ++x) {
            int u[3] = {p[0], p[1], p[2]}, d[3] = {p[0], p[1], p[2]};
            u[x] += 1;
            d[x] -= 1;
            m.up[L][n][x] = (signed char)comp_index(L + 1, u[0], u[1], u[2]);
            m.dn[L][n][x] = (signed char)(d[x] < 0 ? -1 : comp_index(L + 1, d[0], d[1], d[2]));
            m.pw[L][n][x] = (signed char)p[x];
          }
        }
  }
  return m;
}

__constant__ GradMaps c_gmap = make_maps();

struct GradTables {
  OpTableDev t[3];   // raised centre A, C, D
};

struct GradOut {
  double* gj;          // (natom, 3) column-major: dE_J/dx of atom a at a + natom*x
  double* gk;
  int natom;
  const int* satom;    // shell -> atom (0-based)
  const double* szeta; // shell -> exponent
};

template <int NA, int NB, int NC, int ND>
struct GLayout {
  static constexpr int OAB = 0, OCD = NA * NB, OAC = OCD + NC * ND, OAD = OAC + NA * NC, OBC = OAD + NA * ND,
                       OBD = OBC + NB * NC, NP = OBD + NB * ND;
};

// doubles of one team: slots | density blocks | cab | ccd | geometry | ints
template <int NA, int NB, int NC, int ND>
struct GTeam {
  static constexpr int GEO = (int)((sizeof(OpGeom) + 7) / 8);
  static constexpr int INTS = 2 * (NA + NB + NC + ND) + 4;
  static constexpr int NP = GLayout<NA, NB, NC, ND>::NP + NA * NB + NC * ND + GEO + (INTS + 1) / 2;
};

// The components of shell s that carry a target row, and their rows.
template <int L>
__device__ __forceinline__ int grad_kept(const int* __restrict__ stidx, int s, int* k, int* t) {
  int n = 0;
  for (int x = 0; x < ncum(L); ++x) {
    const int r = stidx[s * MAXCOMP + x];
    if (r >= 0) { k[n] = x; t[n] = r; ++n; }
  }
  return n;
}

template <int LA, int LB, int LC, int LD, bool BLOCK>
__global__ void __launch_bounds__(256) k_grad(MolLaunch ql, GradTables tabs, GradOut go, int vmax, int per_team) {
  constexpr int NA = ncum(LA), NB = ncum(LB), NC = ncum(LC), ND = ncum(LD);
  constexpr int NC1 = ncum(LC + 1), ND1 = ncum(LD + 1);
  constexpr int LT = LA + LB + LC + LD + 1;   // the raised classes' total angular momentum
  using GL = GLayout<NA, NB, NC, ND>;
  using GT = GTeam<NA, NB, NC, ND>;
  extern __shared__ double smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int tid = BLOCK ? threadIdx.x : lane, team = BLOCK ? (int)blockDim.x : 32;
  const int teams = BLOCK ? (int)gridDim.x : (int)(gridDim.x * (blockDim.x >> 5));
  const int me = BLOCK ? (int)blockIdx.x : (int)(blockIdx.x * (blockDim.x >> 5)) + wid;
  auto sync = [&]() { if constexpr (BLOCK) __syncthreads(); else __syncwarp(); };
  double* v = smem + (BLOCK ? 0 : (size_t)wid * per_team);
  double* P = v + vmax;
  double* cab = P + GL::NP;
  double* ccd = cab + NA * NB;
  OpGeom& geo = *reinterpret_cast<OpGeom*>(ccd + NC * ND);
  int* kA = reinterpret_cast<int*>(ccd + NC * ND + GT::GEO);
  int* kB = kA + NA;
  int* kC = kB + NB;
  int* kD = kC + NC;
  int* tA = kD + ND;
  int* tB = tA + NA;
  int* tC = tB + NB;
  int* tD = tC + NC;
  int* cnt = tD + ND;
  __shared__ double red[BLOCK ? 8 : 1][18];
  const double c2pi = 2.0 / sqrt(REF_PI);
  const double* __restrict__ D = ql.dt;
  const double* __restrict__ scoef = ql.scoef;
  const PairRec* __restrict__ rec = ql.rec;
  const int nt = ql.nt;
  const double thr = ql.inttol;
  const long long ntickets = 32ll * *ql.nchunks;   // one ket group of a chunk each
  for (long long tk = me; tk < ntickets; tk += teams) {
    const Chunk ch = ql.chunks[tk >> 5];
    const int k = ch.first + (int)(tk & 31);
    if (k >= ch.end) continue;   // team-uniform, as every decision below
    const int G = ch.G, H = ql.bk_list[k];
    const int g0 = ql.gr_start[G], h0 = ql.gr_start[H], hn = ql.gr_n[H];
    const double hmax = ql.gr_max[H];
    if (pair_bound(rec, g0 + ch.p0) * hmax < thr) continue;
    const int2 ij0 = __ldg(reinterpret_cast<const int2*>(&rec[g0].si));
    const int2 kl0 = __ldg(reinterpret_cast<const int2*>(&rec[h0].si));
    sync();   // the previous ticket is done with the lists and blocks
    if (tid == 0) cnt[0] = grad_kept<LA>(ql.stidx, ij0.x, kA, tA);
    if (tid == 1) cnt[1] = grad_kept<LB>(ql.stidx, ij0.y, kB, tB);
    if (tid == 2) cnt[2] = grad_kept<LC>(ql.stidx, kl0.x, kC, tC);
    if (tid == 3) cnt[3] = grad_kept<LD>(ql.stidx, kl0.y, kD, tD);
    sync();
    const int na = cnt[0], nb = cnt[1], nc = cnt[2], nd = cnt[3];
    const int nab = na * nb, ncd = nc * nd, nx = nab * ncd;
    for (int t = tid; t < nab; t += team) P[GL::OAB + t] = dt_at(D, nt, tA[t / nb], tB[t % nb]);
    for (int t = tid; t < ncd; t += team) P[GL::OCD + t] = dt_at(D, nt, tC[t / nd], tD[t % nd]);
    for (int t = tid; t < na * nc; t += team) P[GL::OAC + t] = dt_at(D, nt, tA[t / nc], tC[t % nc]);
    for (int t = tid; t < na * nd; t += team) P[GL::OAD + t] = dt_at(D, nt, tA[t / nd], tD[t % nd]);
    for (int t = tid; t < nb * nc; t += team) P[GL::OBC + t] = dt_at(D, nt, tB[t / nc], tC[t % nc]);
    for (int t = tid; t < nb * nd; t += team) P[GL::OBD + t] = dt_at(D, nt, tB[t / nd], tD[t % nd]);
    // this group quartet's gradient per centre (A, C, D) and axis, J and K, summed by thread
    double gj[3][3] = {}, gk[3][3] = {};
    for (int p = g0 + ch.p0; p < g0 + ch.p1; ++p) {
      const PairView bp = load_pair(rec, p);
      const double sp = bp.bound;
      if (sp * hmax < thr) break;
      const int qe = min((G == H) ? p + 1 : h0 + hn, h0 + min(hn, ch.q1));
      for (int q = h0 + ch.q0; q < qe; ++q) {
        const PairView kq = load_pair(rec, q);
        if (sp * kq.bound < thr) break;
        const double zb = bp.zeta, ze = kq.zeta, zz = zb + ze, rzz = 1.0 / zz, rho = zb * ze * rzz;
        sync();   // the previous quartet's slots and coefficients have been read
        if (!BLOCK || wid == 0) {   // every lane of a warp evaluates the Boys values itself
          const double dx = bp.P[0] - kq.P[0], dy = bp.P[1] - kq.P[1], dz = bp.P[2] - kq.P[2];
          const double T = rho * (dx * dx + dy * dy + dz * dz);
          double F[LT + 1];
          boys_tab<LT>(T, c2pi * bp.S * kq.S * sqrt(rho), ql.boys, F);
#pragma unroll
          for (int m = 0; m <= LT; ++m)
            if (lane == m) v[1 + m] = F[m];
          if (lane == LT + 1) {
            v[0] = 0.0;
            double WP[3], WQ[3];
            for (int x = 0; x < 3; ++x) {
              const double W = (zb * bp.P[x] + ze * kq.P[x]) * rzz;
              WP[x] = W - bp.P[x];
              WQ[x] = W - kq.P[x];
            }
            set_geom(geo, bp.PA, WP, kq.PA, WQ, bp.AB, kq.AB, bp.oz, kq.oz, 0.5 * rzz, ze * rzz, zb * rzz);
          }
        }
        const double w = ((bp.si != bp.sj) ? 2.0 : 1.0) * ((kq.si != kq.sj) ? 2.0 : 1.0) * ((p != q) ? 2.0 : 1.0);
        for (int t = tid; t < nab; t += team)
          cab[t] = scoef[bp.si * MAXCOMP + kA[t / nb]] * scoef[bp.sj * MAXCOMP + kB[t % nb]];
        for (int t = tid; t < ncd; t += team)
          ccd[t] = w * scoef[kq.si * MAXCOMP + kC[t / nd]] * scoef[kq.sj * MAXCOMP + kD[t % nd]];
#pragma unroll
        for (int cen = 0; cen < 3; ++cen) {
          const OpTableDev& tb = tabs.t[cen];
          sync();
          for (int l = 0; l < tb.nlevels; ++l) {
            run_level(tb.ops, tb.levels[l], tb.levels[l + 1], v, geo, tid, team, EvalD{});
            sync();
          }
          const double z2 = 2.0 * go.szeta[cen == 0 ? bp.si : (cen == 1 ? kq.si : kq.sj)];
          for (int i = tid; i < nx; i += team) {
            const int ab = i / ncd, cd = i - ab * ncd;
            const int ia = ab / nb, ib = ab - ia * nb, ic = cd / nd, id = cd - ic * nd;
            const int a = kA[ia], b = kB[ib], cc = kC[ic], d = kD[id];
            const double co = cab[ab] * ccd[cd];
            const double wj = co * P[GL::OAB + ab] * P[GL::OCD + cd];
            const double wk = co * (P[GL::OAC + ia * nc + ic] * P[GL::OBD + ib * nd + id] +
                                    P[GL::OAD + ia * nd + id] * P[GL::OBC + ib * nc + ic]);
#pragma unroll
            for (int x = 0; x < 3; ++x) {
              int up, dn, pw, iu, idn;
              if (cen == 0) {
                up = c_gmap.up[LA][a][x]; dn = c_gmap.dn[LA][a][x]; pw = c_gmap.pw[LA][a][x];
                iu = ((up * NB + b) * NC + cc) * ND + d;
                idn = dn < 0 ? -1 : ((dn * NB + b) * NC + cc) * ND + d;
              } else if (cen == 1) {
                up = c_gmap.up[LC][cc][x]; dn = c_gmap.dn[LC][cc][x]; pw = c_gmap.pw[LC][cc][x];
                iu = ((a * NB + b) * NC1 + up) * ND + d;
                idn = dn < 0 ? -1 : ((a * NB + b) * NC1 + dn) * ND + d;
              } else {
                up = c_gmap.up[LD][d][x]; dn = c_gmap.dn[LD][d][x]; pw = c_gmap.pw[LD][d][x];
                iu = ((a * NB + b) * NC + cc) * ND1 + up;
                idn = dn < 0 ? -1 : ((a * NB + b) * NC + cc) * ND1 + dn;
              }
              double der = z2 * v[tb.out[iu]];
              if (idn >= 0) der -= (double)pw * v[tb.out[idn]];
              gj[cen][x] = fma(wj, der, gj[cen][x]);
              gk[cen][x] = fma(wk, der, gk[cen][x]);
            }
          }
        }
      }
    }
    // the team's sums, then one thread adds them to the atoms
#pragma unroll
    for (int cen = 0; cen < 3; ++cen)
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        gj[cen][x] = warp_sum(gj[cen][x]);
        gk[cen][x] = warp_sum(gk[cen][x]);
      }
    if constexpr (BLOCK) {
      sync();
      if (lane == 0)
        for (int i = 0; i < 9; ++i) { red[wid][i] = gj[i / 3][i % 3]; red[wid][9 + i] = gk[i / 3][i % 3]; }
      sync();
      if (tid == 0)
        for (int wv = 1; wv < (int)(blockDim.x >> 5); ++wv)
          for (int i = 0; i < 9; ++i) { gj[i / 3][i % 3] += red[wv][i]; gk[i / 3][i % 3] += red[wv][9 + i]; }
    }
    if (tid == 0) {
      // centre atoms: A, C, D from the group quartet's shells, B by translational invariance
      const int at[3] = {go.satom[ij0.x], go.satom[kl0.x], go.satom[kl0.y]}, atB = go.satom[ij0.y];
      for (int x = 0; x < 3; ++x) {
        double sj = 0.0, sk = 0.0;
        for (int cen = 0; cen < 3; ++cen) {
          const double vj = 0.5 * gj[cen][x], vk = -0.125 * gk[cen][x];
          sj += vj;
          sk += vk;
          if (vj != 0.0) atomicAdd(go.gj + at[cen] + (size_t)go.natom * x, vj);
          if (vk != 0.0) atomicAdd(go.gk + at[cen] + (size_t)go.natom * x, vk);
        }
        if (sj != 0.0) atomicAdd(go.gj + atB + (size_t)go.natom * x, -sj);
        if (sk != 0.0) atomicAdd(go.gk + atB + (size_t)go.natom * x, -sk);
      }
    }
  }
}

using GradFn = void (*)(const MolLaunch&, const GradTables&, const GradOut&, int vmax, int per_team, int grid, int threads,
                        size_t smem, cudaStream_t);

template <int LA, int LB, int LC, int LD, bool BLOCK>
void launch_grad(const MolLaunch& ql, const GradTables& t, const GradOut& go, int vmax, int per_team, int grid,
                 int threads, size_t smem, cudaStream_t s) {
  k_grad<LA, LB, LC, LD, BLOCK><<<grid, threads, smem, s>>>(ql, t, go, vmax, per_team);
  note_launch();
}

template <int LA, int LB, int LC, int LD, bool BLOCK>
cudaError_t allow_grad(size_t smem) {
  return cudaFuncSetAttribute(k_grad<LA, LB, LC, LD, BLOCK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

struct GradClass {
  GradFn warp, block;
  cudaError_t (*allow_warp)(size_t);
  cudaError_t (*allow_block)(size_t);
  const OpTableHost* tab[3];
  int np;   // doubles of a team besides the slots
};

GradClass grad_class(int cb, int ck) {
#define GC(A, B, C, D)                                                                                      \
  GradClass{&launch_grad<A, B, C, D, false>, &launch_grad<A, B, C, D, true>,                                \
            &allow_grad<A, B, C, D, false>, &allow_grad<A, B, C, D, true>,                                  \
            {&opg_##A##B##C##D##_a, &opg_##A##B##C##D##_c, &opg_##A##B##C##D##_d},                          \
            GTeam<ncum(A), ncum(B), ncum(C), ncum(D)>::NP}
  switch (cb * 8 + ck) {
    case 0: return GC(0, 0, 0, 0);
    case 8: return GC(1, 0, 0, 0);
    case 9: return GC(1, 0, 1, 0);
    case 16: return GC(1, 1, 0, 0);
    case 17: return GC(1, 1, 1, 0);
    case 18: return GC(1, 1, 1, 1);
    case 24: return GC(2, 0, 0, 0);
    case 25: return GC(2, 0, 1, 0);
    case 26: return GC(2, 0, 1, 1);
    case 27: return GC(2, 0, 2, 0);
    case 32: return GC(2, 1, 0, 0);
    case 33: return GC(2, 1, 1, 0);
    case 34: return GC(2, 1, 1, 1);
    case 35: return GC(2, 1, 2, 0);
    case 36: return GC(2, 1, 2, 1);
    case 40: return GC(2, 2, 0, 0);
    case 41: return GC(2, 2, 1, 0);
    case 42: return GC(2, 2, 1, 1);
    case 43: return GC(2, 2, 2, 0);
    case 44: return GC(2, 2, 2, 1);
    case 45: return GC(2, 2, 2, 2);
    default: return GradClass{nullptr, nullptr, nullptr, nullptr, {nullptr, nullptr, nullptr}, 0};
  }
#undef GC
}

}  // namespace

// dE_J/dR and dE_K/dR (natom x 3 each, column-major) of the molecule set up in
// ctx for the target-space density d_dt, into device arrays d_gj, d_gk
// (overwritten).  satom: shell -> atom on the device.
int molecular_gradient(pfe_context* ctx, const double* d_dt, const int* d_satom, int natom, double* d_gj,
                       double* d_gk, cudaStream_t s) {
  // what can fail comes first: the tables' uploads, the launch shapes and the attributes
  struct Launch {
    GradFn fn;
    GradTables t;
    const ClassLaunch* cl;
    int vmax, per_team, grid, threads, side;
    size_t smem;
  };
  Launch launch[64];
  int n = 0;
  for (int i = ctx->nlaunch - 1; i >= 0; --i) {   // the classes of the longest quartets first
    const ClassLaunch& cl = ctx->launches[i];
    const GradClass gc = grad_class(cl.cb, cl.ck);
    if (!gc.warp) { set_error("no gradient kernel for a quartet class"); return PFE_EUNSUPPORTED; }
    Launch& g = launch[n++];
    g = Launch{};
    for (int k = 0; k < 3; ++k) {
      const int rc = upload_optable(ctx, gc.tab[k], &g.t.t[k]);
      if (rc != PFE_OK) return rc;
      g.vmax = std::max(g.vmax, gc.tab[k]->nslots);
    }
    // a warp per quartet where at least kWarpTeams fit an SM's shared memory, else a block
    constexpr int kWarpTeams = 8;
    g.per_team = g.vmax + gc.np;
    const size_t one = sizeof(double) * (size_t)g.per_team, sm = 220 * 1024;
    const bool warp = one * kWarpTeams <= sm;
    const long long tickets = 32ll * cl.nchunks_host;
    int teams = 1;   // per block
    if (warp) teams = (int)std::min<size_t>(8, std::max<size_t>(1, sm / 4 / one));
    g.smem = one * teams;
    if (g.smem > 227 * 1024) { set_error("gradient op table exceeds shared memory"); return PFE_EUNSUPPORTED; }
    PFE_CUDA((warp ? gc.allow_warp : gc.allow_block)(g.smem));
    g.threads = warp ? 32 * teams : 256;
    const int per_sm = std::max(1, std::min(2048 / g.threads, (int)((228 * 1024) / (g.smem + 2048))));
    g.grid = (int)std::max<long long>(
        1, std::min<long long>((tickets + teams - 1) / teams, (long long)ctx->num_sms * std::min(per_sm, 8)));
    g.fn = warp ? gc.warp : gc.block;
    g.cl = &cl;
    g.side = i % pfe_context::kSide;
  }
  {
    const int rc = ensure_side(ctx);
    if (rc != PFE_OK) return rc;
  }
  PFE_CUDA(cudaMemsetAsync(d_gj, 0, sizeof(double) * 3 * (size_t)natom, s));
  PFE_CUDA(cudaMemsetAsync(d_gk, 0, sizeof(double) * 3 * (size_t)natom, s));
  MolLaunch ql = molecular_launch(ctx, d_dt);
  GradOut go{d_gj, d_gk, natom, d_satom, ctx->shells.zeta};
  // the classes side by side on the context's streams: their launches end on few teams
  SideFork sides(ctx, s);
  PFE_CUDA(sides.fork((1u << pfe_context::kSide) - 1));
  for (int i = 0; i < n; ++i) {
    const Launch& g = launch[i];
    ql.chunks = g.cl->chunks;
    ql.nchunks = g.cl->d_nchunks;
    g.fn(ql, g.t, go, g.vmax, g.per_team, g.grid, g.threads, g.smem, ctx->side[g.side]);
  }
  PFE_CUDA(launch_status());
  PFE_CUDA(sides.join());
  return PFE_OK;
}

}  // namespace pfe
