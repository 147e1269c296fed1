// Device-side state of one Fock-build context (struct pfe_context of the C ABI).
#pragma once

#include <algorithm>
#include <atomic>

#include <cublas_v2.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <memory>
#include <unordered_map>
#include <vector>

#include "pfe_common.cuh"

namespace pfe {

// Allocation-failure injection for tests of the error paths: the n-th device
// allocation a context or batch asks for from now on fails as out of memory
// (pfe_debug_fail_allocation); negative: never.  Nothing reaches the GPU: the
// allocation is simply not attempted.
inline std::atomic<long long> g_fail_alloc_after{-1};

inline cudaError_t injected_alloc_failure() {
  long long v = g_fail_alloc_after.load();
  while (v >= 0)
    if (g_fail_alloc_after.compare_exchange_weak(v, v - 1)) return v == 0 ? cudaErrorMemoryAllocation : cudaSuccess;
  return cudaSuccess;
}


// The Boys tables of one IGAMMA on one device, shared by every context set up with the
// same values (a batch holds hundreds) and freed with the last of them.
struct BoysTables {
  int device = 0;
  std::vector<double> igamma;   // as given, column-major
  double* rows = nullptr;       // [T][m]
  double* down = nullptr;       // the table of boys_down
  ~BoysTables() {
    cudaFree(rows);
    cudaFree(down);
  }
};
int acquire_boys(int device, const double* igamma, cudaStream_t s, std::shared_ptr<BoysTables>* out);

// Device memory of a context or batch.  Requests of up to kSmall bytes are cut from
// blocks that are kept from one set-up to the next (a set-up makes over a hundred, and
// cudaMalloc and cudaFree were most of a small molecule's: 1.1 of 2.6 ms); larger ones,
// and small ones that no block has room for, are allocations of their own, but for one
// buffer of up to kKept bytes (`kept`) that also stays.  A piece that free_now gives back
// is cut again for the requests that follow, so scratch does not add up: the work on it
// must be ordered before theirs (a set-up's work is all on one stream; other callers wait
// first).  Kept at most: 13.5 MiB of blocks (512 KiB, 1 MiB, then 2 MiB each; one water
// molecule takes the first two) and the 64 MiB buffer; all of it is freed with the owner.
// A block's memory may still be read by a build in flight when the next set-up begins, so
// release_all waits for the device, as cudaFree does.
struct DeviceMemory {
  static constexpr size_t kSmall = 256 << 10, kFirst = 512 << 10, kBlock = 2 << 20, kKept = 64 << 20;
  static constexpr int kBlocks = 8;
  struct Block {
    char* p;
    size_t n;
  };
  std::vector<void*> owned;    // allocations of their own
  std::vector<Block> blocks;
  size_t block = 0, offset = 0;             // the next uncut byte: blocks[block].p + offset
  std::unordered_map<void*, size_t> cut;    // pieces in use
  std::multimap<size_t, char*> spare;       // pieces to cut from first, by size
  void* kept = nullptr;
  size_t kept_bytes = 0;
  DeviceMemory() = default;
  DeviceMemory(const DeviceMemory&) = delete;
  DeviceMemory& operator=(const DeviceMemory&) = delete;
  ~DeviceMemory() {
    for (const Block& b : blocks) cudaFree(b.p);
    cudaFree(kept);
  }

  cudaError_t alloc(void** p, size_t bytes) {
    if (cudaError_t f = injected_alloc_failure()) return f;
    const size_t n = (std::max<size_t>(bytes, 1) + 255) & ~size_t(255);
    if (n <= kSmall) {
      const auto it = spare.lower_bound(n);
      if (it != spare.end()) {
        char* q = it->second;
        const size_t left = it->first - n;
        spare.erase(it);
        if (left > 0) spare.emplace(left, q + n);
        cut[q] = n;
        *p = q;
        return cudaSuccess;
      }
      if (block < blocks.size() && offset + n > blocks[block].n) {
        if (offset < blocks[block].n) spare.emplace(blocks[block].n - offset, blocks[block].p + offset);
        ++block;
        offset = 0;
      }
      if (block == blocks.size() && blocks.size() < (size_t)kBlocks) {
        Block b{nullptr, std::min(kBlock, kFirst << blocks.size())};
        const cudaError_t e = cudaMalloc((void**)&b.p, b.n);
        if (e != cudaSuccess) return e;
        blocks.push_back(b);
      }
      if (block < blocks.size()) {
        *p = blocks[block].p + offset;
        offset += n;
        cut[*p] = n;
        return cudaSuccess;
      }
    }
    const cudaError_t e = cudaMalloc(p, n);
    if (e == cudaSuccess) owned.push_back(*p);
    return e;
  }
  // The one buffer that outlasts set-ups: as large as the largest asked for, up to kKept.
  cudaError_t alloc_kept(void** p, size_t bytes) {
    if (bytes > kKept) return alloc(p, bytes);
    if (cudaError_t f = injected_alloc_failure()) return f;
    if (bytes > kept_bytes) {
      cudaFree(kept);
      kept = nullptr;
      kept_bytes = 0;
      const cudaError_t e = cudaMalloc(&kept, bytes);
      if (e != cudaSuccess) return e;
      kept_bytes = bytes;
    }
    *p = kept;
    return cudaSuccess;
  }
  void free_now(void* p) {
    if (!p) return;
    const auto it = cut.find(p);
    if (it != cut.end()) {
      spare.emplace(it->second, (char*)p);
      cut.erase(it);
      return;
    }
    for (size_t i = 0; i < owned.size(); ++i)
      if (owned[i] == p) {
        owned.erase(owned.begin() + i);
        cudaFree(p);
        return;
      }
  }
  void release_all() {
    if (block > 0 || offset > 0 || kept) cudaDeviceSynchronize();
    for (void* p : owned) cudaFree(p);
    owned.clear();
    cut.clear();
    spare.clear();
    block = offset = 0;
  }
};

// Primitive-shell table, struct of arrays (n shells).
struct DevShells {
  int n;
  double *x, *y, *z, *zeta;
  int* L;
  int* prim;  // n * MAXCOMP, 0-based primitive of each cumulative component (-1 ghost/absent)
};

// Shell-pair records, struct of arrays; sorted by class and bound after setup.
struct PairArrays {
  double* P[3];
  double* PA[3];
  double* AB[3];
  double* zeta;
  double* S;        // S_P of the two s components (the reference's OV / C1 factor)
  double* schwarz;  // the reference's IJIJ/KLKL bound
  int* si;
  int* sj;
  unsigned char* cls;
  unsigned long long* key;
  int* gid;         // contracted block pair (molecules)
  double* gmax;     // largest bound in the pair's block-pair group (molecules)
};

// A piece of work of the molecular quartet kernels: bra group G against the ket
// groups [first, end) of the bucketed list, of which the bra pairs [p0, p1) and
// the ket pairs [q0, q1) (positions in their groups; q1 beyond a ket group's end
// means its end).  A group quartet cut into several pieces is digested piece by
// piece: J and K are linear in its integrals.
struct __align__(16) Chunk {
  int G, first, end, inst;   // inst: the instance of a batch (0 otherwise)
  int p0, p1, q0, q1;
};
constexpr int kAllPairs = 1 << 30;   // q1 of a chunk that takes the ket groups whole
constexpr int kClassPairs = 21;      // (bra class, ket class) pairs, bra class >= ket class

// One launch of the quartet kernel: a (bra class, ket class) pair and its chunks.
struct ClassLaunch {
  int cb, ck;
  int nchunks_host;
  int* d_nchunks;
  Chunk* chunks;             // costliest first
  double quartets;
  // execution variant: 0 = straight-line thread per quartet, 1 = warp per
  // quartet on the op table, 2 = block per quartet on the op table, 3 = warp
  // per quartet on the op table with per-lane Boys/geometry and only the
  // outputs that carry a coefficient (pfe_mol_wide.cu)
  int variant;
  bool has_straight, has_table;
  const unsigned short* ops;
  const int* levels;
  const unsigned short* out;
  int nlevels, nout, nslots;
  const unsigned short* ops_p;   // pure-bra table (see OpTableDev), or null
  const int* levels_p;
  const unsigned short* out_p;
  int nlevels_p;
  const unsigned short* ops_p2;  // pure bra and pure ket table, or null
  const int* levels_p2;
  const unsigned short* out_p2;
  int nlevels_p2;
  int wpb, per_warp;         // warps per block and doubles per warp (variant 1)
  size_t smem_big, smem_warp;
  float tuned_ms[4];         // autotuner timings per variant (0 = not run)
  // straight-line variant: X of up to xcap chunks (a tile) at xbuf, and a flag per chunk
  double* xbuf;
  unsigned char* xlive;
  int xcap;
  double* xg;                // block variant: per-block X scratch in global memory, or null
  int nslots_p, nslots_p2;   // slots of the pure-bra and bra-and-ket tables (0: none)
  // variant 3 (warp per primitive quartet, kept outputs only): per-warp shared
  // memory in doubles, of which wide_vmax op-table slots and wide_xmax outputs
  bool has_wide;
  int wide_wpb, wide_per_warp, wide_vmax, wide_xmax;
  size_t smem_wide;
  int* queue;                // device work queue: one chunk counter per launch (pass), zeroed before each
  int npass;                 // register passes of the straight-line variant (general; see pass_variant)
  unsigned long long live;   // the passes launched: those with a component that has a coefficient
  int launches_live;         // kernel launches of a tile: pass groups with a component that has a coefficient, digestion
  int gmul = 32;             // straight-line variant: persistent grid of up to gmul blocks per SM
};

// Kernel launches of one class of a build (launch_class): those of its tiles, or one.
// (An instance of a batch has no launches of its own: no chunks, no memory for a tile.)
inline int class_launches(const ClassLaunch& cl, int numprocs) {
  if (cl.has_table && !(cl.variant == 0 && cl.has_straight)) return 1;
  const int work = (cl.nchunks_host + numprocs - 1) / numprocs;
  if (work <= 0) return 0;
  return (cl.cb > 0 ? (work + cl.xcap - 1) / std::max(1, cl.xcap) : 1) * cl.launches_live;
}

}  // namespace pfe

// The opaque handle of the C ABI.
struct pfe_context : pfe::DeviceMemory {
  // block panels of the digestion (molecules; pfe_mol.cu): the kept components of every
  // contracted block are consecutive panel rows, and the matrices of a block pair are
  // contiguous: element (p, q) at row_base[p] + q * row_n[p], where a block of n rows
  // from row p0 has row_base[p] = p0 * np + (p - p0) and row_n[p] = n
  std::vector<int> h_blk, h_blk_L, h_blk_t;   // shell -> block; block -> L, -> target per component (MAXCOMP)
  int np = 0;
  int* d_poff = nullptr;        // shell -> first panel row of its block
  int* d_ptgt = nullptr;        // panel row -> target (-1: none)
  long long* d_prow = nullptr;  // row_base
  int* d_prown = nullptr;       // row_n
  int* d_pinv = nullptr;        // target -> its panel rows: d_pinv[t] .. d_pinv[t + 1] of d_pinv_row
  int* d_pinv_row = nullptr;
  double *d_pd = nullptr, *d_pj = nullptr, *d_pk = nullptr;
  int device = 0;
  int num_sms = 148;
  cudaStream_t stream = nullptr;
  // class launches beside those on the caller's stream (launch_classes), forked
  // and joined with the events; made at set-up (ensure_side)
  static constexpr int kSide = 7;
  cudaStream_t side[kSide] = {};
  cudaEvent_t ev_fork = nullptr, ev_join[kSide] = {};
  bool concurrent = false;   // every class has a buffer of its own for its stored integrals
  cublasHandle_t blas = nullptr;
  bool ready = false;
  uint64_t key = 0;
  bool molecular = true;
  int npgs = 0, ncgs = 0, npshell = 0, ncell1 = 1;
  int cel1[3] = {0, 0, 0}, cel2[3] = {0, 0, 0}, rc1[3] = {0, 0, 0};
  double period[3] = {0, 0, 0};
  double helix = 0.0;
  double inttol = 0.0;
  int myid = 0, numprocs = 1;
  int precision = 0;
  double mixed_cutoff = 0.0;

  // device data
  pfe::DevShells shells{};
  double* d_sss = nullptr;   // S_P(head I, head J, cell) for shell heads, [cell][J][I]
  std::shared_ptr<pfe::BoysTables> boys;
  double* d_boys = nullptr;  // boys->rows
  double* d_maxc = nullptr;  // max_i |CC(i, p)| per primitive
  double* d_cc = nullptr;    // CC (ncgs x npgs, column-major)
  double* d_c2h = nullptr;
  double* d_jp = nullptr;
  double* d_kp = nullptr;
  // digestion targets: contracted functions when every primitive feeds at most
  // one contracted row of CC (the reference's READ3 bases), else primitives
  bool contracted = false;
  int nt = 0;                // target dimension (ncgs or npgs)
  int* d_tidx = nullptr;     // primitive -> target row, -1 when it has no coefficient
  double* d_tcoef = nullptr; // primitive -> coefficient (CC entry, or 1)
  double* d_scoef = nullptr; // shell x component -> coefficient of its primitive (tcoef)
  int* d_stidx = nullptr;    // shell x component -> target row of its primitive (tidx)
  int* d_blk = nullptr;      // shell -> contracted block id
  // per angular momentum L of a shell: the most components with a target row
  // one shell of that L has, and whether some shell of that L has a target on
  // a component below L (a cumulative sp/spd shell, not a pure p/d one)
  int kept_max[3] = {1, 4, 10};
  bool lower_kept[3] = {false, true, true};
  int nblk = 0;
  bool force_primitive = false;  // set before set-up: primitive targets even when CC allows contracted ones
  int* d_rep = nullptr;      // target -> representative primitive (largest |coefficient|)
  double* d_repc = nullptr;  // its coefficient
  double* d_pt = nullptr;    // density in target space (nt x nt): P_C read off P_P, or P_P
  unsigned int* d_flag = nullptr;  // set when P_P is not the decontraction of a contracted density
  // groups: runs of pairs of one contracted block pair (molecules)
  void* d_prec = nullptr;    // the sorted pairs as 128-byte records (PairRec)
  int ngroups = 0;
  int* d_gr_start = nullptr;
  int* d_gr_n = nullptr;
  double* d_gr_max = nullptr;
  int* d_bk_list = nullptr;  // group ids ordered by (class, size bucket, group)
  double2* d_tile = nullptr; // their pair records by tile of 32 list entries (load_tile)
  int* d_tile_at = nullptr;  // list position of a tile's first group -> base of the tile
  // density-dependent screening of molecular builds (no counterpart in the reference, which
  // screens by the Schwarz bounds alone): skip quartets with bound * max|P| < dtol, and run
  // the recursion in FP32 where bound * max|P| < mcut; max|P| per pair of contracted blocks
  double dtol = 0.0, mcut = 0.0;
  int* d_tblk = nullptr;     // target -> block (-1: none)
  double* d_bmax = nullptr;  // nblk x nblk block maxima of |P_T| of the last build
  unsigned long long* d_n32 = nullptr;  // quartets of the last build run in FP32
  double* d_w1 = nullptr;
  double* d_w2 = nullptr;
  pfe::PairArrays pairs{};
  long long npairs = 0;
  int class_off[8] = {0}, class_n[8] = {0};
  pfe::ClassLaunch launches[64];
  int nlaunch = 0;
  int* d_queue = nullptr;    // 64 chunk counters per class launch (the work queues of launches[])
  double census_quartets = 0.0, census_flops = 0.0, census_ref = 0.0, census_fp32 = 0.0;
  // the chunks of every class pair before they are cut into pieces and sorted
  // (molecular set-up; a batch joins those of its instances): per chunk its class
  // pair, its screened quartets and its length in steps, per class pair the sum of the lengths
  bool in_batch = false;     // set before set-up: the batch finishes the chunk lists
  int nraw = 0;
  pfe::Chunk* d_raw = nullptr;
  unsigned int* d_raw_steps = nullptr;
  unsigned int* d_raw_cost = nullptr;
  unsigned char* d_raw_pair = nullptr;
  double pair_steps[pfe::kClassPairs] = {};

  // host-path staging (pfe_fourindex_eri)
  double* d_pp = nullptr;
  double* d_pph = nullptr;
  double* d_out_c = nullptr;
  double* d_out_x = nullptr;
  size_t pp_bytes = 0, pph_bytes = 0, out_bytes = 0;

  // lattice path state lives in pfe_lattice.cu
  void* lattice = nullptr;

  // per-launch timing (pfe_context_profile)
  bool profile = false;
  bool tuned = false;
  cudaEvent_t ev[130] = {};
  int nev = 0;
  int ev_cls[64] = {0};
  int ev_variant[64] = {0};
  float ev_tuned[64][4] = {};
  double ev_quartets[64] = {0}, ev_flops[64] = {0};
  int ev_gmul[64] = {0};
  int nprof = 0;

  std::vector<void*> pending;  // scratch freed at the end of setup

  void free_later(void* p) { pending.push_back(p); }
  void free_pending() {
    for (void* p : pending) free_now(p);
    pending.clear();
  }
  void release_all() {
    pfe::DeviceMemory::release_all();
    pending.clear();
  }
};

// Many molecules whose Fock builds run together (struct pfe_batch of the C ABI):
// every instance has its own context (set-up, pairs, chunks); the batch joins
// their chunk lists per quartet class, each chunk tagged with its instance, so
// one launch per class (and pass) covers every instance.
struct pfe_batch : pfe::DeviceMemory {
  int device = 0;
  std::vector<pfe_context*> inst;
  std::vector<long long> off;       // packed offsets (doubles) of the ncgs x ncgs matrices, n+1
  pfe::ClassLaunch launches[64];    // joined chunk lists; ops/tables of the first instance with the class
  int nlaunch = 0;
  int* d_queue = nullptr;           // the joined launches' work queues (64 counters each)
  long long* d_off = nullptr;       // off[] on the device (the batched symmetrisation)
  bool all_contracted = false;      // every instance digests in contracted space
  bool concurrent = false;          // every class has a buffer of its own for its stored integrals
  void* d_insts = nullptr;          // the instances' launch records (MolLaunch) on the device
  void* h_insts = nullptr;          // ... and their pinned host copy, uploaded by every build (so a
                                    // captured graph re-reads it at each replay)
  cudaEvent_t ev_insts = nullptr;   // the last upload of h_insts
  bool ev_pending = false;
  const double* insts_for = nullptr;  // density the records point at (null: rewrite them)
  bool mixed = false;               // FP32-capable kernels (sticky once any instance asked for them)
  bool ready = false;               // set by a pfe_batch_setup that succeeded
  void release_all() {
    pfe::DeviceMemory::release_all();
    if (h_insts) cudaFreeHost(h_insts);
    h_insts = nullptr;
    if (ev_insts) cudaEventDestroy(ev_insts);
    ev_insts = nullptr;
    ev_pending = false;
    d_insts = nullptr;
    insts_for = nullptr;
    nlaunch = 0;   // the launches pointed into the memory freed above
    ready = false;
  }
};

namespace pfe {
// The context's cuBLAS handle, created on first use: molecules with contracted
// targets never call cuBLAS, and a batch holds hundreds of contexts.
inline bool ensure_blas(pfe_context* ctx) {
  if (ctx->blas) return true;
  if (cublasCreate(&ctx->blas) != CUBLAS_STATUS_SUCCESS) {
    ctx->blas = nullptr;
    return false;
  }
  return true;
}
int ensure_side(pfe_context* ctx);
void debug_integral_memory(long long tile, long long together);

// Work of a build on the context's side streams (bit k of `used`: side[k]), forked from
// stream s and joined back to it on every way out: after an error too, later work on s
// waits for what was launched, and a stream capture ends with no stream unjoined.
class SideFork {
 public:
  SideFork(pfe_context* cx, cudaStream_t s) : cx_(cx), s_(s) {}
  ~SideFork() { join(); }
  cudaError_t fork(unsigned int used) {
    if (!used) return cudaSuccess;
    cudaError_t e = cudaEventRecord(cx_->ev_fork, s_);
    for (int k = 0; k < pfe_context::kSide && e == cudaSuccess; ++k) {
      if (!((used >> k) & 1)) continue;
      e = cudaStreamWaitEvent(cx_->side[k], cx_->ev_fork, 0);
      if (e == cudaSuccess) forked_ |= 1u << k;
    }
    return e;
  }
  cudaError_t join() {
    cudaError_t first = cudaSuccess;
    for (int k = 0; k < pfe_context::kSide; ++k) {
      if (!((forked_ >> k) & 1)) continue;
      cudaError_t e = cudaEventRecord(cx_->ev_join[k], cx_->side[k]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(s_, cx_->ev_join[k], 0);
      if (first == cudaSuccess) first = e;
    }
    forked_ = 0;
    return first;
  }

 private:
  pfe_context* cx_;
  cudaStream_t s_;
  unsigned int forked_ = 0;
};
int batch_setup(pfe_batch* b);
int batch_fock_pc(pfe_batch* b, const double* d_pc, double* d_cc, double* d_xc, cudaStream_t s);
int batch_refresh(pfe_batch* b, const double* d_pc);
int batch_autotune(pfe_batch* b, const double* d_pc, cudaStream_t s);
int alloc_pairs(pfe_context* ctx, PairArrays* pa, long long n);
void free_pairs(pfe_context* ctx, PairArrays* pa);
void launch_symmetrize(const double* a, double* out, int n, int ncell, cudaStream_t s);
void launch_select_class(const unsigned char* cls, int want, int* list, int* count, long long n, cudaStream_t s);
int upload_constants(int device);
int molecular_setup(pfe_context* ctx, const pfe_args* a);
int molecular_fock(pfe_context* ctx, const double* d_pp, double* d_cc, double* d_xc, cudaStream_t s);
int contract_outputs(pfe_context* ctx, const double* jp, const double* kp, double* d_cc, double* d_xc,
                     bool symmetrize, int ncell, cudaStream_t s);
int autotune(pfe_context* ctx, const double* d_pp, cudaStream_t s);
int molecular_density_ok(pfe_context* ctx, cudaStream_t s, bool* ok);
int molecular_fock_pc(pfe_context* ctx, const double* d_pc, double* d_cc, double* d_xc, cudaStream_t s);
struct OpTableDev;
const struct OpTableHost* host_optable(int cb, int ck);
const struct OpTableHost* host_optable_pure(int cb, int ck);
const struct OpTableHost* host_optable_pure2(int cb, int ck);
const struct OpTableHost* host_optable_topd(int cb, int ck);
int upload_optable(pfe_context* ctx, const struct OpTableHost* h, OpTableDev* d);
double class_flops(int cb, int ck);
int lattice_setup(pfe_context* ctx, const pfe_args* a);
int lattice_fock(pfe_context* ctx, const double* d_pp, const double* d_pph, double* d_cc, double* d_xc,
                 cudaStream_t s);
void lattice_release(pfe_context* ctx);
void lattice_force_interpreter(pfe_context* ctx, bool on);
int lattice_launches(pfe_context* ctx);
int molecular_gradient_pp(pfe_context* ctx, const double* d_pp, const int* d_satom, int natom, double* d_gj,
                          double* d_gk, cudaStream_t s);
const char* last_error_cstr();
int measure_fp64_peak(int device, double* tflops);
}  // namespace pfe
