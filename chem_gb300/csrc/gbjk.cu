// libgbjk: context, device memory and the C-ABI of the DF J/K engine.
//
// The context owns the resident 3-center tensor (panel layout), the metric
// factors, per-nocc workspaces and the launch plans (tile lists) of every
// contraction.  One compute call issues a fixed sequence of launches on the
// context's stream:
//   J:  gather P rows -> row dots (g partials) -> reduce -> h = V^-1 g
//       -> column sums J = B^T h -> block filter
//   K:  gather C rows -> half transform H = B C (grouped GEMM over panels)
//       -> fit (L^-1 or V^-1, batched over mu) -> K = -Hfit^T Hfit (split-K)
//       -> reduce -> block filter
// The split-precision path (kernels_split.cuh) replaces the three GEMMs.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <unordered_map>
#include <vector>

#include "common.cuh"
#include "gbjk.h"
#include "aok_host.cuh"
#include "eri3c_gpu.cuh"
#include "asymk_host.cuh"
#include "kernels_fp64.cuh"
#include "mp2_host.cuh"
#include "scf_host.cuh"
#include "split_host.cuh"

using namespace gbjk;

// SMs the mixed-path exchange GEMM leaves to the concurrent J column sums
// unless gbjk_set_overlap says otherwise: 0, the exchange takes every SM and
// the J blocks fill the registers and shared memory its CTAs leave free
constexpr int kDefaultOverlapSms = 0;
// ... as long as J's tensor copy is smaller than this.  Builds through the host
// call, beside against in order, by the size of the copy: 27 MB (five waters)
// 129 / 147 us, 56 MB 158 / 178, 125 MB 260 / 269, 227 MB (C10H22) 375 / 386,
// 358 MB 581 / 579, 433 MB 681 / 674, 516 MB 808 / 790, 702 MB 1121 / 1120,
// 1159 MB (C20H42) 1913 / 1889.
constexpr size_t kOverlapJBytes = size_t(384) << 20;

// Auxiliary functions of an engine at most: a metric of 5 GB.  (The FP64 J sums once
// kept a vector of naux in shared memory; larger ones have never been run.)
constexpr int kMaxNaux = 25600;

// The engines' host copies of their error flags, one int each: a page-locked page
// that stays for the process, its slots taken and given back under a lock.  (A
// page-locked allocation per engine took 300 us of its life, as long as all else
// of a small one.)  More engines than slots take pageable ints; those of a page
// whose lock was lost (a device reset) are no more than that.
class FlagPool {
  static constexpr int kSlots = 1024;
  std::mutex m_;
  int* page_ = nullptr;
  std::vector<int*> free_;

 public:
  int* take() {
    std::lock_guard<std::mutex> l(m_);
    if (!page_ && (page_ = (int*)std::aligned_alloc(4096, kSlots * sizeof(int)))) {
      if (cudaHostRegister(page_, kSlots * sizeof(int), cudaHostRegisterPortable) != cudaSuccess)
        cudaGetLastError();  // works pageable
      for (int i = kSlots; i-- > 0;) free_.push_back(page_ + i);
    }
    if (free_.empty()) return (int*)std::malloc(sizeof(int));
    int* p = free_.back();
    free_.pop_back();
    return p;
  }
  void give(int* p) {
    std::lock_guard<std::mutex> l(m_);
    if (page_ && p >= page_ && p < page_ + kSlots)
      free_.push_back(p);
    else
      std::free(p);
  }
};
FlagPool& flag_pool() {
  static FlagPool* p = new FlagPool;  // never destroyed: engines may outlive statics
  return *p;
}

enum Phase {
  PH_GATHER = 0,
  PH_J_ROWDOT,
  PH_J_REDUCE,
  PH_J_METRIC,
  PH_J_COLSUM,
  PH_HT,
  PH_FIT,
  PH_KGEMM,
  PH_KREDUCE,
  PH_FILTER,
  PH_SPLIT,
  PH_COUNT
};
static const char* kPhaseNames[PH_COUNT] = {
    "gather", "j_rowdot", "j_reduce", "j_metric", "j_colsum", "half_transform",
    "fit",    "k_gemm",   "k_reduce", "filter",   "split_operands"};

struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
};

// One Fock build recorded as a CUDA graph, valid while the engine epoch it
// was captured at is current.
struct CapturedBuild {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int64_t launches = 0;
  uint64_t epoch = 0;
  void reset() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    exec = nullptr;
    graph = nullptr;
    launches = 0;
  }
};

struct gbjk_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  // Mixed-path J column sums run on `side`, forked after the half transform
  // and joined before the build ends, while the exchange GEMM runs on
  // `stream` on all SMs but overlap_sms of them (0: on all, the J blocks
  // co-resident; -1: no second stream, the phases in order).
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  int* h_err = nullptr;  // page-locked copy of the split path's error flag (flag_pool)
  int overlap_sms = kDefaultOverlapSms;
  // FP64 K of a pre-fitted tensor in auxiliary batches (gbjk_set_aux_batch):
  // per batch b the half transform of rows [b*xb, b*xb + xbc) (one group per
  // AO function mu; groups b*nbf .. b*nbf+nbf-1) and its split-K exchange,
  // accumulated into K in batch order.  Index 0 of the per-size arrays is a
  // full batch, 1 the shorter last one.
  struct Fp64Batch {
    int nocc = -1, xb = 0, nbatch = 0, xlast = 0;
    int ks[2] = {1, 1};
    long long kc[2] = {0, 0};
    int ht_t0[2] = {0, 0}, ht_nt[2] = {0, 0}, k_t0[2] = {0, 0}, k_nt[2] = {0, 0};
    bool elem_ht[2] = {false, false}, narrow[2] = {false, false}, elem_k[2] = {false, false};
    int tn[2] = {64, 64};
    GemmGroup* d_groups = nullptr;
    GemmTile* d_tiles = nullptr;
    double* d_H = nullptr;
    double* d_Kpart = nullptr;
  } fb;
  // FP64 DF-MO / DF-LMO K with the occupied orbitals in batches
  // (gbjk_set_occ_batch, megalochem's occ_nbatches): per batch the half
  // transform of its columns, the fit and the split-K exchange, accumulated
  // into K in batch order.  Per batch gs groups: nblk panels, nbf L^-1 fits,
  // nbf V^-1 fits, the DF-MO and the DF-LMO exchange.  Index 0 of the
  // per-size arrays is a full batch, 1 the shorter last one.
  int occ_req = 0;
  struct Fp64OccBatch {
    int nocc = -1, ob = 0, nbatch = 0, olast = 0, gs = 0;
    int ks[2] = {1, 1};
    long long kc[2] = {0, 0};
    bool elem_ht[2] = {false, false}, narrow[2] = {false, false}, elem_k[2] = {false, false};
    int tn[2] = {64, 64};
    int ht_t0[2] = {0, 0}, ht_nt[2] = {0, 0}, fit_t0[2] = {0, 0}, fit_nt[2] = {0, 0},
        fitv_t0[2] = {0, 0}, mo_t0[2] = {0, 0}, mo_nt[2] = {0, 0}, lmo_t0[2] = {0, 0},
        lmo_nt[2] = {0, 0};
    GemmGroup* d_groups = nullptr;
    GemmTile* d_tiles = nullptr;
    double *d_H = nullptr, *d_H2 = nullptr, *d_Kpart = nullptr;
  } ob;
  // launch configuration: requested (0 = built-in rule) and in effect
  gbjk_tunables tune{};
  gbjk_tunables tune_eff{};
  long long kchunk = 0;  // FP64 exchange k per part
  std::string err;
  int64_t launches = 0;
  size_t dev_bytes = 0;
  std::unordered_map<void*, size_t> alloc_bytes;
  // layout (host)
  int nbf = 0, naux = 0, nblk = 0;
  double eps = 0.0;
  std::vector<int> bsize, boff, panelK, cmoff, colmap, blk_of;
  std::vector<long long> panel_off, pg_off;
  long long nnz = 0, pg_total = 0;
  int ncols_total = 0, maxK = 0;
  // layout (device)
  int *d_blk_of = nullptr, *d_boff = nullptr, *d_panelK = nullptr, *d_cmoff = nullptr,
      *d_colmap = nullptr;
  long long *d_panel_off = nullptr, *d_pg_off = nullptr;
  // resident data
  double* d_B = nullptr;
  double *d_Linv = nullptr, *d_Vinv = nullptr;
  bool have_B = false, have_metric = false;
  bool fitted = false;  // the uploaded tensor already is L^-1 B (no metric)
  // J workspace
  double *d_P = nullptr, *d_Pg = nullptr, *d_part = nullptr, *d_g = nullptr, *d_h = nullptr,
         *d_y = nullptr, *d_J = nullptr;
  int jmode = GBJK_J_VINV;
  // K workspace (per nocc)
  int ws_nocc = -1;
  int wc_nocc = -1;
  int ksplit = 1;
  bool narrow = false;  // half transform and fit on 64 x 16 tiles
  int ht_tn = 64;        // tile width of the half transform and fit
  bool elem_ht = false, elem_k = false;  // one thread per output (tiny problems)
  double *d_C = nullptr, *d_Cg = nullptr, *d_H = nullptr, *d_H2 = nullptr, *d_Kpart = nullptr,
         *d_K = nullptr;
  GemmGroup* d_groups = nullptr;
  GemmTile* d_tiles = nullptr;
  int n_ht_groups = 0, n_fit_groups = 0;
  int ht_tile0 = 0, ht_ntiles = 0, fit_tile0 = 0, fit_ntiles = 0, fitV_tile0 = 0, syrk_tile0 = 0,
      syrk_ntiles = 0, lmo_tile0 = 0, lmo_ntiles = 0;
  int fitL_group0 = 0, fitV_group0 = 0, syrk_group = 0, lmo_group = 0;
  // precision
  int precision = GBJK_FP64;
  int nslices = 0;
  SplitState split;
  // SOS-AO-MP2 Laplace batch (ll_full Z builder) on the prefitted tensor
  Mp2State mp2;
  // DF-AO exchange (fitted coefficients, dense intermediates)
  AoKState aok;
  // non-symmetric DF-LMO exchange (left and right coefficients)
  AsymKState asymk;
  // SCF iteration on the device (graphs around the Fock build)
  ScfState scf;
  // profiling
  bool profile = false;
  cudaEvent_t ev[PH_COUNT][2] = {};
  double ph_ms[PH_COUNT] = {};
  int64_t ph_launch[PH_COUNT] = {};
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> pending;
  std::vector<cudaEvent_t> ev_pool;
  // captured Fock builds: the caller's (device pointers) and the host-buffer
  // call's own (context buffers, keyed by its arguments' shape)
  CapturedBuild user_graph, host_graph;
  int host_kmethod = -1, host_nocc = -1;
  bool host_j = false, host_k = false, host_uncapturable = false;
  // bumped by every free or replacement of a buffer and by every setting
  // that changes the launch sequence; a captured build older than it is stale
  uint64_t epoch = 0;
};

namespace {

gbjk_status fail(gbjk_ctx* c, gbjk_status s, const std::string& msg) {
  if (c) c->err = msg;
  return s;
}

#define CK(call)                                                                         \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess)                                                               \
      return fail(ctx, e_ == cudaErrorMemoryAllocation ? GBJK_OOM : GBJK_CUDA_ERROR,     \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                   \
  } while (0)

#define CKL(phase)                                                                       \
  do {                                                                                   \
    ctx->launches++;                                                                     \
    cudaError_t e_ = cudaGetLastError();                                                 \
    if (e_ != cudaSuccess)                                                               \
      return fail(ctx, GBJK_CUDA_ERROR,                                                  \
                  std::string("launch ") + kPhaseNames[phase] + ": " + cudaGetErrorString(e_)); \
  } while (0)

template <class T>
gbjk_status dalloc(gbjk_ctx* ctx, T** p, size_t count) {
  if (*p) return GBJK_OK;
  if (count == 0) count = 1;
  cudaError_t e = cudaMalloc((void**)p, count * sizeof(T));
  if (e != cudaSuccess) {
    *p = nullptr;
    cudaGetLastError();
    return fail(ctx, GBJK_OOM,
                "cudaMalloc of " + std::to_string(count * sizeof(T)) + " bytes failed: " +
                    cudaGetErrorString(e));
  }
  ctx->alloc_bytes[(void*)*p] = count * sizeof(T);
  ctx->dev_bytes += count * sizeof(T);
  return GBJK_OK;
}

template <class T>
void dfree(gbjk_ctx* ctx, T** p) {
  if (*p) {
    ctx->epoch++;
    cudaFree(*p);
    auto it = ctx->alloc_bytes.find((void*)*p);
    if (it != ctx->alloc_bytes.end()) {
      ctx->dev_bytes -= it->second;
      ctx->alloc_bytes.erase(it);
    }
    *p = nullptr;
  }
}

cudaEvent_t get_event(gbjk_ctx* ctx) {
  if (!ctx->ev_pool.empty()) {
    cudaEvent_t e = ctx->ev_pool.back();
    ctx->ev_pool.pop_back();
    return e;
  }
  cudaEvent_t e;
  cudaEventCreate(&e);
  return e;
}

struct PhaseScope {
  gbjk_ctx* ctx;
  int ph;
  cudaEvent_t a = nullptr, b = nullptr;
  PhaseScope(gbjk_ctx* c, int p) : ctx(c), ph(p) {
    if (ctx->profile) {
      a = get_event(ctx);
      b = get_event(ctx);
      cudaEventRecord(a, ctx->stream);
    }
  }
  ~PhaseScope() {
    if (ctx->profile) {
      cudaEventRecord(b, ctx->stream);
      ctx->pending.push_back({ph, {a, b}});
    }
    ctx->ph_launch[ph]++;
  }
};

void resolve_profile(gbjk_ctx* ctx) {
  for (auto& pe : ctx->pending) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, pe.second.first, pe.second.second) == cudaSuccess)
      ctx->ph_ms[pe.first] += ms;
    ctx->ev_pool.push_back(pe.second.first);
    ctx->ev_pool.push_back(pe.second.second);
  }
  ctx->pending.clear();
}

int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }
// Tiles of tm rows x tn columns: 64 x 64, 64 x 16 (narrow kernel) or
// 16 x 16 (one thread per output).
void add_tiles(std::vector<GemmTile>& tiles, int group, int M, int N, int k0, int k1,
               long long coff, bool upper_only, int tn = 64, int tm = 64) {
  for (int mt = 0; mt < cdiv(M, tm); ++mt)
    for (int nt = 0; nt < cdiv(N, tn); ++nt) {
      if (upper_only && nt < mt) continue;
      tiles.push_back({group, mt, nt, k0, k1, coff});
    }
}

// Occupied counts up to this many use 64 x 16 tiles in the FP64 half
// transform and fit (a 64 x 64 tile would be mostly padding); where these have at
// most kElemOutputs outputs they run on 16 x 16 tiles, one thread per output, as
// the exchange does at every size.
constexpr int kNarrowN = 16;
constexpr long long kElemOutputs = 1 << 20;

// FP64 launch choices for a problem (the built-in rules where req asks for
// none): tile width of the half transform and fit (1 = one thread per
// output), exchange tile (1 or 64) and the exchange's k parts.
struct Fp64Plan {
  bool elem_ht, narrow, elem_k;
  int ht_tn, ks;
  long long kc;
};
gbjk_status fp64_plan(int nbf, int naux, int nocc, const gbjk_tunables& req, Fp64Plan* pl) {
  if (nbf <= 0 || naux <= 0 || nocc <= 0) return GBJK_INVALID_ARG;
  const int t = req.fp64_ht_tn;
  if (t != 0 && t != 1 && t != 16 && t != 32 && t != 64) return GBJK_INVALID_ARG;
  if (req.fp64_k_tile != 0 && req.fp64_k_tile != 1 && req.fp64_k_tile != 64)
    return GBJK_INVALID_ARG;
  if (req.fp64_kchunk < 0) return GBJK_INVALID_ARG;
  if (t == 0) {
    pl->elem_ht = (long long)nbf * naux * nocc <= kElemOutputs;
    pl->narrow = !pl->elem_ht && nocc <= kNarrowN;
    // the kernel computes whole patches of TN/4 columns, so the width that
    // pads nocc least wins; narrower tiles load A more often and have to save
    // 5 % of the columns (C8H18 fit, nocc 33: 11.8 ms at 36 columns of 64 x 16
    // tiles, 13.5 at 40 of 64 x 32, 15.3 at 48 of 64 x 64)
    const auto pad = [&](int w) { return cdiv(nocc, w) * w; };
    if (!pl->elem_ht && 100 * pad(4) <= 95 * std::min(pad(8), pad(16))) pl->narrow = true;
    const bool mid = !pl->elem_ht && !pl->narrow && pad(8) < pad(16);
    pl->ht_tn = pl->elem_ht || pl->narrow ? 16 : (mid ? 32 : 64);
  } else {
    pl->elem_ht = t == 1;
    pl->narrow = t == 16;
    pl->ht_tn = t == 1 ? 16 : t;
  }
  const long long kdim = (long long)naux * nocc;
  int ks = 1;
  long long kc = kdim;
  gbjk_k_split_plan(nbf, naux, nocc, &ks, &kc);
  if (req.fp64_kchunk > 0) {
    kc = std::min((req.fp64_kchunk + 15) / 16 * 16, (kdim + 15) / 16 * 16);
    ks = (int)((kdim + kc - 1) / kc);
  }
  pl->ks = ks;
  pl->kc = kc;
  // the exchange in 16 x 16 tiles: they follow the diagonal and the matrix
  // edge closest, and their staged operands keep the FP64 pipe as busy as 64 x
  // 64 tiles do (exchange of C20H42: 39.6 ms against 48.1; nbf 800, naux 2400,
  // nocc 120: 152.6 against 193.6; water, nbf 24: 10 us against 31)
  pl->elem_k = req.fp64_k_tile != 64;
  return GBJK_OK;
}

// Coefficient workspaces shared by both paths.
gbjk_status ensure_c_workspace(gbjk_ctx* ctx, int nocc) {
  if (ctx->wc_nocc == nocc) return GBJK_OK;
  dfree(ctx, &ctx->d_C);
  dfree(ctx, &ctx->d_Cg);
  ctx->wc_nocc = -1;
  gbjk_status s;
  if ((s = dalloc(ctx, &ctx->d_C, (size_t)ctx->nbf * nocc))) return s;
  if ((s = dalloc(ctx, &ctx->d_Cg, (size_t)ctx->ncols_total * nocc))) return s;
  ctx->wc_nocc = nocc;
  return GBJK_OK;
}

// (Re)build the FP64-path K workspaces and launch plans for a given nocc.
gbjk_status ensure_k_workspace(gbjk_ctx* ctx, int nocc) {
  if (ctx->ws_nocc == nocc) return GBJK_OK;
  const size_t nbf = ctx->nbf, naux = ctx->naux;
  const size_t hsz = nbf * naux * nocc;
  dfree(ctx, &ctx->d_H);
  dfree(ctx, &ctx->d_H2);
  dfree(ctx, &ctx->d_Kpart);
  dfree(ctx, &ctx->d_groups);
  dfree(ctx, &ctx->d_tiles);
  ctx->ws_nocc = -1;
  gbjk_status s;
  if ((s = ensure_c_workspace(ctx, nocc))) return s;
  if ((s = dalloc(ctx, &ctx->d_H, hsz))) return s;
  if ((s = dalloc(ctx, &ctx->d_H2, hsz))) return s;
  // split-K of the exchange GEMM and tile shapes: requested or by rule
  const long long kdim = (long long)naux * nocc;
  Fp64Plan pl;
  if ((s = fp64_plan(ctx->nbf, ctx->naux, nocc, ctx->tune, &pl)))
    return fail(ctx, s, "invalid FP64 tunables");
  const int ks = pl.ks;
  const long long kchunk64 = pl.kc;
  ctx->ksplit = ks;
  ctx->kchunk = kchunk64;
  if ((s = dalloc(ctx, &ctx->d_Kpart, (size_t)ks * nbf * nbf))) return s;
  const bool elem_ht = pl.elem_ht, elem_k = pl.elem_k, narrow = pl.narrow;
  ctx->narrow = narrow;
  ctx->ht_tn = pl.ht_tn;
  ctx->elem_ht = elem_ht;
  ctx->elem_k = elem_k;
  ctx->tune_eff.fp64_ht_tn = elem_ht ? 1 : pl.ht_tn;
  ctx->tune_eff.fp64_k_tile = elem_k ? 1 : 64;
  ctx->tune_eff.fp64_kchunk = kchunk64;
  const int ht_tm = elem_ht ? 16 : 64, ht_tn = ctx->ht_tn;
  const int k_t = elem_k ? 16 : 64;

  std::vector<GemmGroup> groups;
  std::vector<GemmTile> tiles;
  // half transform: one group per panel
  ctx->ht_tile0 = 0;
  for (int I = 0; I < ctx->nblk; ++I) {
    GemmGroup g;
    g.A = ctx->d_B + ctx->panel_off[I];
    g.B = ctx->d_Cg + (long long)ctx->cmoff[I] * nocc;
    g.C = ctx->d_H + (long long)ctx->boff[I] * naux * nocc;
    g.M = ctx->bsize[I] * (int)naux;
    g.N = nocc;
    g.K = ctx->panelK[I];
    g.lda = ctx->panelK[I];
    g.ldb = nocc;
    g.ldc = nocc;
    g.flags = 0;
    if (g.K == 0) continue;
    add_tiles(tiles, (int)groups.size(), g.M, g.N, 0, g.K, 0, false, ht_tn, ht_tm);
    groups.push_back(g);
  }
  ctx->ht_ntiles = (int)tiles.size();
  // fit with L^-1 (lower) : per mu, H2[mu] = Linv H[mu]
  ctx->fit_tile0 = (int)tiles.size();
  ctx->fitL_group0 = (int)groups.size();
  for (size_t mu = 0; mu < nbf; ++mu) {
    GemmGroup g;
    g.A = ctx->d_Linv;
    g.B = ctx->d_H + mu * naux * nocc;
    g.C = ctx->d_H2 + mu * naux * nocc;
    g.M = (int)naux;
    g.N = nocc;
    g.K = (int)naux;
    g.lda = (int)naux;
    g.ldb = nocc;
    g.ldc = nocc;
    g.flags = kLowerA;
    add_tiles(tiles, (int)groups.size(), g.M, g.N, 0, g.K, 0, false, ht_tn, ht_tm);
    groups.push_back(g);
  }
  ctx->fit_ntiles = (int)tiles.size() - ctx->fit_tile0;
  // A row tile of L^-1 costs what its last row is; of a few blocks per SM the
  // last should be the short ones.  (Larger problems have many blocks per SM,
  // and read H in its own order.)
  if (elem_ht)
    std::stable_sort(tiles.begin() + ctx->fit_tile0, tiles.end(),
                     [](const GemmTile& x, const GemmTile& y) { return x.mt > y.mt; });
  // fit with V^-1 (full) for DF-LMO: same shapes, groups pointing at V^-1
  ctx->fitV_group0 = (int)groups.size();
  for (size_t mu = 0; mu < nbf; ++mu) {
    GemmGroup g = groups[ctx->fitL_group0 + mu];
    g.A = ctx->d_Vinv;
    g.flags = 0;
    groups.push_back(g);
  }
  ctx->fitV_tile0 = (int)tiles.size();
  for (int t = 0; t < ctx->fit_ntiles; ++t) {
    GemmTile tt = tiles[ctx->fit_tile0 + t];
    tt.group += ctx->fitV_group0 - ctx->fitL_group0;
    tiles.push_back(tt);
  }
  // exchange GEMM (DF-MO): K = -H2^T H2, upper tiles, split-K
  const int kchunk = (int)kchunk64;
  {
    GemmGroup g;
    g.A = ctx->fitted ? ctx->d_H : ctx->d_H2;  // fitted tensor: H already carries L^-1
    g.B = g.A;
    g.C = ctx->d_Kpart;
    g.M = (int)nbf;
    g.N = (int)nbf;
    g.K = (int)kdim;
    g.lda = (int)kdim;
    g.ldb = (int)kdim;
    g.ldc = (int)nbf;
    g.flags = kTransB | kUpperC;
    ctx->syrk_group = (int)groups.size();
    groups.push_back(g);
    ctx->syrk_tile0 = (int)tiles.size();
    for (int k = 0; k < ks; ++k) {
      const int k0 = k * kchunk, k1 = (int)std::min<long long>(kdim, (long long)(k + 1) * kchunk);
      add_tiles(tiles, ctx->syrk_group, g.M, g.N, k0, std::max(k0, k1), (long long)k * nbf * nbf,
                true, k_t, k_t);
    }
    ctx->syrk_ntiles = (int)tiles.size() - ctx->syrk_tile0;
  }
  // exchange GEMM (DF-LMO): K_nm = -sum H[m] Hfit[n]  -> rows n from H2 (Hfit), cols m from H
  {
    GemmGroup g;
    g.A = ctx->d_H2;
    g.B = ctx->d_H;
    g.C = ctx->d_Kpart;
    g.M = (int)nbf;
    g.N = (int)nbf;
    g.K = (int)kdim;
    g.lda = (int)kdim;
    g.ldb = (int)kdim;
    g.ldc = (int)nbf;
    g.flags = kTransB;
    ctx->lmo_group = (int)groups.size();
    groups.push_back(g);
    ctx->lmo_tile0 = (int)tiles.size();
    for (int k = 0; k < ks; ++k) {
      const int k0 = k * kchunk, k1 = (int)std::min<long long>(kdim, (long long)(k + 1) * kchunk);
      add_tiles(tiles, ctx->lmo_group, g.M, g.N, k0, std::max(k0, k1), (long long)k * nbf * nbf,
                false, k_t, k_t);
    }
    ctx->lmo_ntiles = (int)tiles.size() - ctx->lmo_tile0;
  }
  if ((s = dalloc(ctx, &ctx->d_groups, groups.size()))) return s;
  if ((s = dalloc(ctx, &ctx->d_tiles, tiles.size()))) return s;
  CK(cudaMemcpy(ctx->d_groups, groups.data(), groups.size() * sizeof(GemmGroup),
                cudaMemcpyHostToDevice));
  CK(cudaMemcpy(ctx->d_tiles, tiles.data(), tiles.size() * sizeof(GemmTile),
                cudaMemcpyHostToDevice));
  ctx->ws_nocc = nocc;
  return GBJK_OK;
}

// Batched FP64 exchange of a pre-fitted tensor: plans and buffers per nocc.
gbjk_status ensure_k_batched(gbjk_ctx* ctx, int nocc) {
  auto& fb = ctx->fb;
  if (fb.nocc == nocc) return GBJK_OK;
  dfree(ctx, &fb.d_groups);
  dfree(ctx, &fb.d_tiles);
  dfree(ctx, &fb.d_H);
  dfree(ctx, &fb.d_Kpart);
  fb.nocc = -1;
  gbjk_status s;
  if ((s = ensure_c_workspace(ctx, nocc))) return s;
  const int nbf = ctx->nbf, naux = ctx->naux;
  fb.xb = std::min(naux, std::max(32, ctx->split.xb_req & ~31));
  fb.nbatch = cdiv(naux, fb.xb);
  fb.xlast = naux - (fb.nbatch - 1) * fb.xb;
  const int sizes[2] = {fb.xb, fb.xlast};
  std::vector<GemmGroup> groups;
  std::vector<GemmTile> tiles;
  // half-transform groups, batch after batch: H_b[mu][y][i] = sum_k
  // B_I[m][Y0 + y][k] Cg_I[k][i] (rows of one AO function)
  for (int b = 0; b < fb.nbatch; ++b) {
    const int Y0 = b * fb.xb, xbc = std::min(fb.xb, naux - Y0);
    for (int I = 0; I < ctx->nblk; ++I)
      for (int m = 0; m < ctx->bsize[I]; ++m) {
        GemmGroup g;
        const int K = ctx->panelK[I];
        g.A = ctx->d_B + ctx->panel_off[I] + ((long long)m * naux + Y0) * K;
        g.B = ctx->d_Cg + (long long)ctx->cmoff[I] * nocc;
        g.C = nullptr;  // set below once d_H exists
        g.M = xbc;
        g.N = nocc;
        g.K = K;
        g.lda = K;
        g.ldb = nocc;
        g.ldc = nocc;
        g.flags = 0;
        groups.push_back(g);
      }
  }
  const int ng_ht = (int)groups.size();
  long long kpart_max = 1;
  for (int v = 0; v < 2; ++v) {
    const int xbc = sizes[v];
    Fp64Plan pl;
    if ((s = fp64_plan(nbf, xbc, nocc, ctx->tune, &pl))) return fail(ctx, s, "invalid FP64 tunables");
    fb.elem_ht[v] = pl.elem_ht;
    fb.narrow[v] = pl.narrow;
    fb.tn[v] = pl.ht_tn;
    fb.elem_k[v] = pl.elem_k;
    fb.ks[v] = pl.ks;
    fb.kc[v] = pl.kc;
    kpart_max = std::max<long long>(kpart_max, pl.ks);
    const int tm = pl.elem_ht ? 16 : 64;
    // half-transform tiles of one batch of this size (groups 0..nbf-1
    // relative to the batch's first group)
    fb.ht_t0[v] = (int)tiles.size();
    for (int mu = 0; mu < nbf; ++mu) {
      const int I = ctx->blk_of[mu];
      if (ctx->panelK[I] == 0) continue;
      add_tiles(tiles, mu, xbc, nocc, 0, ctx->panelK[I], 0, false, pl.ht_tn, tm);
    }
    fb.ht_nt[v] = (int)tiles.size() - fb.ht_t0[v];
    // exchange of one batch: K_part = H_b H_b^T, upper tiles, split-K
    GemmGroup g;
    g.A = nullptr;
    g.B = nullptr;
    g.C = nullptr;
    g.M = nbf;
    g.N = nbf;
    g.K = xbc * nocc;
    g.lda = xbc * nocc;
    g.ldb = xbc * nocc;
    g.ldc = nbf;
    g.flags = kTransB | kUpperC;
    groups.push_back(g);  // group ng_ht + v
    const long long kd = (long long)xbc * nocc;
    const int kt = pl.elem_k ? 16 : 64;
    fb.k_t0[v] = (int)tiles.size();
    for (int k = 0; k < pl.ks; ++k) {
      const int k0 = (int)(k * pl.kc), k1 = (int)std::min<long long>(kd, (k + 1) * pl.kc);
      add_tiles(tiles, 0, nbf, nbf, k0, std::max(k0, k1), (long long)k * nbf * nbf, true, kt, kt);
    }
    fb.k_nt[v] = (int)tiles.size() - fb.k_t0[v];
  }
  if ((s = dalloc(ctx, &fb.d_H, (size_t)nbf * fb.xb * nocc))) return s;
  if ((s = dalloc(ctx, &fb.d_Kpart, (size_t)kpart_max * nbf * nbf))) return s;
  for (int b = 0; b < fb.nbatch; ++b) {
    const int xbc = std::min(fb.xb, naux - b * fb.xb);
    for (int mu = 0; mu < nbf; ++mu)
      groups[(size_t)b * nbf + mu].C = fb.d_H + (long long)mu * xbc * nocc;
  }
  for (int v = 0; v < 2; ++v) {
    groups[ng_ht + v].A = fb.d_H;
    groups[ng_ht + v].B = fb.d_H;
    groups[ng_ht + v].C = fb.d_Kpart;
  }
  if ((s = dalloc(ctx, &fb.d_groups, groups.size()))) return s;
  if ((s = dalloc(ctx, &fb.d_tiles, tiles.size()))) return s;
  CK(cudaMemcpy(fb.d_groups, groups.data(), groups.size() * sizeof(GemmGroup),
                cudaMemcpyHostToDevice));
  CK(cudaMemcpy(fb.d_tiles, tiles.data(), tiles.size() * sizeof(GemmTile),
                cudaMemcpyHostToDevice));
  ctx->tune_eff.fp64_ht_tn = fb.elem_ht[0] ? 1 : fb.tn[0];
  ctx->tune_eff.fp64_k_tile = fb.elem_k[0] ? 1 : 64;
  ctx->tune_eff.fp64_kchunk = fb.kc[0];
  fb.nocc = nocc;
  return GBJK_OK;
}

gbjk_status filter(gbjk_ctx* ctx, double* M);

// One grouped FP64 GEMM launch with the tile shape of a plan.
void launch_fp64(cudaStream_t st, const GemmGroup* g, const GemmTile* t, int nt, bool elem,
                 bool narrow, int tn, bool transB) {
  if (nt == 0) return;
  if (elem && transB)
    k_gemm_fp64_elem<true><<<nt, 256, 0, st>>>(g, t, 1.0);
  else if (elem)
    k_gemm_fp64_elem<false><<<nt, 256, 0, st>>>(g, t, 1.0);
  else if (transB)
    k_gemm_fp64<true><<<nt, 256, 0, st>>>(g, t, 1.0);
  else if (narrow)
    k_gemm_fp64<false, false, 16><<<nt, 64, 0, st>>>(g, t, 1.0);
  else if (tn == 32)
    k_gemm_fp64<false, false, 32><<<nt, 128, 0, st>>>(g, t, 1.0);
  else
    k_gemm_fp64<false><<<nt, 256, 0, st>>>(g, t, 1.0);
}

// Occupied-batched FP64 exchange (DF-MO and DF-LMO): plans and buffers.
gbjk_status ensure_k_occ_batched(gbjk_ctx* ctx, int nocc) {
  auto& ob = ctx->ob;
  if (ob.nocc == nocc) return GBJK_OK;
  dfree(ctx, &ob.d_groups);
  dfree(ctx, &ob.d_tiles);
  dfree(ctx, &ob.d_H);
  dfree(ctx, &ob.d_H2);
  dfree(ctx, &ob.d_Kpart);
  ob.nocc = -1;
  gbjk_status s;
  if ((s = ensure_c_workspace(ctx, nocc))) return s;
  const int nbf = ctx->nbf, naux = ctx->naux, nblk = ctx->nblk;
  ob.ob = std::min(nocc, ctx->occ_req);
  ob.nbatch = cdiv(nocc, ob.ob);
  ob.olast = nocc - (ob.nbatch - 1) * ob.ob;
  ob.gs = nblk + 2 * nbf + 2;
  const int sizes[2] = {ob.ob, ob.olast};
  std::vector<GemmGroup> groups((size_t)ob.nbatch * ob.gs);
  std::vector<GemmTile> tiles;
  long long kmax = 1;
  for (int v = 0; v < 2; ++v) {
    const int obc = sizes[v];
    Fp64Plan pl;
    if ((s = fp64_plan(nbf, naux, obc, ctx->tune, &pl))) return fail(ctx, s, "invalid FP64 tunables");
    ob.elem_ht[v] = pl.elem_ht;
    ob.narrow[v] = pl.narrow;
    ob.tn[v] = pl.ht_tn;
    ob.elem_k[v] = pl.elem_k;
    ob.ks[v] = pl.ks;
    ob.kc[v] = pl.kc;
    kmax = std::max<long long>(kmax, pl.ks);
    const int tm = pl.elem_ht ? 16 : 64, kt = pl.elem_k ? 16 : 64;
    ob.ht_t0[v] = (int)tiles.size();
    for (int I = 0; I < nblk; ++I)
      if (ctx->panelK[I])
        add_tiles(tiles, I, ctx->bsize[I] * naux, obc, 0, ctx->panelK[I], 0, false, pl.ht_tn, tm);
    ob.ht_nt[v] = (int)tiles.size() - ob.ht_t0[v];
    ob.fit_t0[v] = (int)tiles.size();
    for (int mu = 0; mu < nbf; ++mu)
      add_tiles(tiles, nblk + mu, naux, obc, 0, naux, 0, false, pl.ht_tn, tm);
    ob.fit_nt[v] = (int)tiles.size() - ob.fit_t0[v];
    ob.fitv_t0[v] = (int)tiles.size();
    for (int t = 0; t < ob.fit_nt[v]; ++t) {
      GemmTile tt = tiles[ob.fit_t0[v] + t];
      tt.group += nbf;
      tiles.push_back(tt);
    }
    const long long kd = (long long)naux * obc;
    for (int lmo = 0; lmo < 2; ++lmo) {
      (lmo ? ob.lmo_t0[v] : ob.mo_t0[v]) = (int)tiles.size();
      for (int k = 0; k < pl.ks; ++k) {
        const int k0 = (int)(k * pl.kc), k1 = (int)std::min<long long>(kd, (k + 1) * pl.kc);
        add_tiles(tiles, nblk + 2 * nbf + lmo, nbf, nbf, k0, std::max(k0, k1),
                  (long long)k * nbf * nbf, !lmo, kt, kt);
      }
      (lmo ? ob.lmo_nt[v] : ob.mo_nt[v]) = (int)tiles.size() - (lmo ? ob.lmo_t0[v] : ob.mo_t0[v]);
    }
  }
  const size_t hsz = (size_t)nbf * naux * ob.ob;
  if ((s = dalloc(ctx, &ob.d_H, hsz)) || (s = dalloc(ctx, &ob.d_H2, hsz)) ||
      (s = dalloc(ctx, &ob.d_Kpart, (size_t)kmax * nbf * nbf)))
    return s;
  for (int b = 0; b < ob.nbatch; ++b) {
    const int i0 = b * ob.ob, obc = std::min(ob.ob, nocc - i0);
    GemmGroup* g = groups.data() + (size_t)b * ob.gs;
    for (int I = 0; I < nblk; ++I) {
      const int K = ctx->panelK[I];
      g[I] = {ctx->d_B + ctx->panel_off[I], ctx->d_Cg + (long long)ctx->cmoff[I] * nocc + i0,
              ob.d_H + (long long)ctx->boff[I] * naux * obc, ctx->bsize[I] * naux, obc, K,
              std::max(K, 1), nocc, obc, 0};
    }
    for (int mu = 0; mu < nbf; ++mu) {
      const long long off = (long long)mu * naux * obc;
      g[nblk + mu] = {ctx->d_Linv, ob.d_H + off, ob.d_H2 + off, naux, obc, naux, naux, obc, obc,
                      kLowerA};
      g[nblk + nbf + mu] = {ctx->d_Vinv, ob.d_H + off, ob.d_H2 + off, naux, obc, naux, naux, obc,
                            obc, 0};
    }
    const int kd = naux * obc;
    g[nblk + 2 * nbf] = {ob.d_H2, ob.d_H2, ob.d_Kpart, nbf, nbf, kd, kd, kd, nbf,
                         kTransB | kUpperC};
    // DF-LMO: K_nm = -sum Hfit[n] H[m]
    g[nblk + 2 * nbf + 1] = {ob.d_H2, ob.d_H, ob.d_Kpart, nbf, nbf, kd, kd, kd, nbf, kTransB};
  }
  if ((s = dalloc(ctx, &ob.d_groups, groups.size()))) return s;
  if ((s = dalloc(ctx, &ob.d_tiles, tiles.size()))) return s;
  CK(cudaMemcpy(ob.d_groups, groups.data(), groups.size() * sizeof(GemmGroup),
                cudaMemcpyHostToDevice));
  CK(cudaMemcpy(ob.d_tiles, tiles.data(), tiles.size() * sizeof(GemmTile),
                cudaMemcpyHostToDevice));
  ctx->tune_eff.fp64_ht_tn = ob.elem_ht[0] ? 1 : ob.tn[0];
  ctx->tune_eff.fp64_k_tile = ob.elem_k[0] ? 1 : 64;
  ctx->tune_eff.fp64_kchunk = ob.kc[0];
  ob.nocc = nocc;
  return GBJK_OK;
}

// (plans and buffers: ensure_k_occ_batched)
gbjk_status run_k_occ_batched(gbjk_ctx* ctx, int kmethod, const double* dC, int nocc,
                              double* dK) {
  auto& ob = ctx->ob;
  const int nbf = ctx->nbf, nblk = ctx->nblk;
  const bool mo = kmethod == GBJK_K_DFMO;
  {
    PhaseScope ps(ctx, PH_GATHER);
    const long long total = (long long)ctx->ncols_total * nocc;
    k_gather_cols<<<cdiv(total, 256), 256, 0, ctx->stream>>>(dC, nocc, ctx->d_colmap,
                                                             ctx->ncols_total, ctx->d_Cg);
    CKL(PH_GATHER);
  }
  for (int b = 0; b < ob.nbatch; ++b) {
    const int v = (b == ob.nbatch - 1 && ob.olast != ob.ob) ? 1 : 0;
    const GemmGroup* g = ob.d_groups + (size_t)b * ob.gs;
    {
      PhaseScope ps(ctx, PH_HT);
      launch_fp64(ctx->stream, g, ob.d_tiles + ob.ht_t0[v], ob.ht_nt[v], ob.elem_ht[v],
                  ob.narrow[v], ob.tn[v], false);
      CKL(PH_HT);
    }
    {
      PhaseScope ps(ctx, PH_FIT);
      launch_fp64(ctx->stream, g, ob.d_tiles + (mo ? ob.fit_t0[v] : ob.fitv_t0[v]), ob.fit_nt[v],
                  ob.elem_ht[v], ob.narrow[v], ob.tn[v], false);
      CKL(PH_FIT);
    }
    {
      PhaseScope ps(ctx, PH_KGEMM);
      launch_fp64(ctx->stream, g, ob.d_tiles + (mo ? ob.mo_t0[v] : ob.lmo_t0[v]),
                  mo ? ob.mo_nt[v] : ob.lmo_nt[v], ob.elem_k[v], false, 64, true);
      CKL(PH_KGEMM);
    }
    {
      PhaseScope ps(ctx, PH_KREDUCE);
      const long long n2 = (long long)nbf * nbf;
      k_splitk_reduce_acc<<<cdiv(n2, 256), 256, 0, ctx->stream>>>(
          ob.d_Kpart, ob.ks[v], nbf, -1.0, mo ? 1 : 0, b > 0 ? 1 : 0, dK);
      CKL(PH_KREDUCE);
    }
  }
  (void)nblk;
  return filter(ctx, dK);
}

// (plans and buffers: ensure_k_batched)
gbjk_status run_k_batched(gbjk_ctx* ctx, const double* dC, int nocc, double* dK) {
  auto& fb = ctx->fb;
  const int nbf = ctx->nbf;
  {
    PhaseScope ps(ctx, PH_GATHER);
    const long long total = (long long)ctx->ncols_total * nocc;
    k_gather_cols<<<cdiv(total, 256), 256, 0, ctx->stream>>>(dC, nocc, ctx->d_colmap,
                                                             ctx->ncols_total, ctx->d_Cg);
    CKL(PH_GATHER);
  }
  const int ng_ht = fb.nbatch * nbf;
  for (int b = 0; b < fb.nbatch; ++b) {
    const int v = (b == fb.nbatch - 1 && fb.xlast != fb.xb) ? 1 : 0;
    const GemmGroup* g = fb.d_groups + (size_t)b * nbf;
    const GemmTile* t = fb.d_tiles + fb.ht_t0[v];
    const int nt = fb.ht_nt[v];
    if (nt) {
      PhaseScope ps(ctx, PH_HT);
      if (fb.elem_ht[v])
        k_gemm_fp64_elem<false><<<nt, 256, 0, ctx->stream>>>(g, t, 1.0);
      else if (fb.narrow[v])
        k_gemm_fp64<false, false, 16><<<nt, 64, 0, ctx->stream>>>(g, t, 1.0);
      else if (fb.tn[v] == 32)
        k_gemm_fp64<false, false, 32><<<nt, 128, 0, ctx->stream>>>(g, t, 1.0);
      else
        k_gemm_fp64<false><<<nt, 256, 0, ctx->stream>>>(g, t, 1.0);
      CKL(PH_HT);
    }
    {
      PhaseScope ps(ctx, PH_KGEMM);
      const GemmGroup* gk = fb.d_groups + ng_ht + v;
      const GemmTile* tk = fb.d_tiles + fb.k_t0[v];
      if (fb.elem_k[v])
        k_gemm_fp64_elem<true><<<fb.k_nt[v], 256, 0, ctx->stream>>>(gk, tk, 1.0);
      else
        k_gemm_fp64<true><<<fb.k_nt[v], 256, 0, ctx->stream>>>(gk, tk, 1.0);
      CKL(PH_KGEMM);
    }
    {
      PhaseScope ps(ctx, PH_KREDUCE);
      const long long n2 = (long long)nbf * nbf;
      k_splitk_reduce_acc<<<cdiv(n2, 256), 256, 0, ctx->stream>>>(fb.d_Kpart, fb.ks[v], nbf,
                                                                  -1.0, 1, b > 0 ? 1 : 0, dK);
      CKL(PH_KREDUCE);
    }
  }
  return filter(ctx, dK);
}

gbjk_status ensure_j_workspace(gbjk_ctx* ctx) {
  gbjk_status s;
  const size_t nbf = ctx->nbf, naux = ctx->naux;
  if ((s = dalloc(ctx, &ctx->d_P, nbf * nbf))) return s;
  if ((s = dalloc(ctx, &ctx->d_Pg, (size_t)ctx->pg_total))) return s;
  if ((s = dalloc(ctx, &ctx->d_part, nbf * naux))) return s;
  if ((s = dalloc(ctx, &ctx->d_g, naux))) return s;
  if ((s = dalloc(ctx, &ctx->d_h, naux))) return s;
  if ((s = dalloc(ctx, &ctx->d_y, naux))) return s;
  if ((s = dalloc(ctx, &ctx->d_J, nbf * nbf))) return s;
  if ((s = dalloc(ctx, &ctx->d_K, nbf * nbf))) return s;
  return GBJK_OK;
}

gbjk_status launch_gemm(gbjk_ctx* ctx, int tile0, int ntiles, bool transB, double alpha,
                        int phase, bool narrow = false, bool elem = false, int tn = 64) {
  if (ntiles == 0) return GBJK_OK;
  PhaseScope ps(ctx, phase);
  const GemmGroup* g = ctx->d_groups;
  const GemmTile* t = ctx->d_tiles + tile0;
  if (elem && transB)
    k_gemm_fp64_elem<true><<<ntiles, 256, 0, ctx->stream>>>(g, t, alpha);
  else if (elem)
    k_gemm_fp64_elem<false><<<ntiles, 256, 0, ctx->stream>>>(g, t, alpha);
  else if (narrow)
    k_gemm_fp64<false, false, 16><<<ntiles, 64, 0, ctx->stream>>>(g, t, alpha);
  else if (!transB && tn == 32)
    k_gemm_fp64<false, false, 32><<<ntiles, 128, 0, ctx->stream>>>(g, t, alpha);
  else if (transB)
    k_gemm_fp64<true><<<ntiles, 256, 0, ctx->stream>>>(g, t, alpha);
  else
    k_gemm_fp64<false><<<ntiles, 256, 0, ctx->stream>>>(g, t, alpha);
  CKL(phase);
  return GBJK_OK;
}

gbjk_status filter(gbjk_ctx* ctx, double* M, cudaStream_t st) {
  if (ctx->eps <= 0) return GBJK_OK;
  PhaseScope ps(ctx, PH_FILTER);
  k_block_filter<<<cdiv((long long)ctx->nblk * ctx->nblk, 8), 256, 0, st>>>(
      M, ctx->nbf, ctx->d_boff, ctx->nblk, ctx->eps);
  CKL(PH_FILTER);
  return GBJK_OK;
}

gbjk_status filter(gbjk_ctx* ctx, double* M) { return filter(ctx, M, ctx->stream); }

// FP64 J on `st` (the context's stream, or its side stream beside K)
gbjk_status run_j(gbjk_ctx* ctx, const double* dP, double* dJ, cudaStream_t st) {
  const int nbf = ctx->nbf, naux = ctx->naux;
  // blocks of screened (I, J) pairs are never written by the column sums
  CK(cudaMemsetAsync(dJ, 0, (size_t)nbf * nbf * sizeof(double), st));
  {
    PhaseScope ps(ctx, PH_GATHER);
    k_gather_panel_rows<<<dim3(cdiv(ctx->maxK, 128), nbf), 128, 0, st>>>(
        dP, nbf, ctx->d_blk_of, ctx->d_boff, ctx->d_panelK, ctx->d_pg_off, ctx->d_cmoff,
        ctx->d_colmap, ctx->d_Pg);
    CKL(PH_GATHER);
  }
  {
    PhaseScope ps(ctx, PH_J_ROWDOT);
    const long long rows = (long long)nbf * naux;
    k_j_rowdot<<<cdiv(rows * 32, 256), 256, 0, st>>>(
        ctx->d_B, ctx->d_panel_off, ctx->d_blk_of, ctx->d_boff, ctx->d_panelK, ctx->d_pg_off,
        ctx->d_Pg, nbf, naux, ctx->d_part);
    CKL(PH_J_ROWDOT);
  }
  {
    PhaseScope ps(ctx, PH_J_REDUCE);
    k_reduce_rows<<<cdiv(naux, 32), 32, 0, st>>>(ctx->d_part, nbf, naux, ctx->d_g);
    CKL(PH_J_REDUCE);
  }
  const double* hvec = ctx->d_h;
  if (ctx->fitted) {
    hvec = ctx->d_g;  // the tensor carries the metric: h = g
  } else {
    PhaseScope ps(ctx, PH_J_METRIC);
    if (ctx->jmode == GBJK_J_CHOLESKY) {
      // h = L^-T (L^-1 g): no explicit V^-1
      k_gemv<<<cdiv((long long)naux * 32, 256), 256, 0, st>>>(ctx->d_Linv, ctx->d_g,
                                                                         naux, ctx->d_y);
      CKL(PH_J_METRIC);
      k_gemv_lower_t<<<cdiv(naux, 32), 32, 0, st>>>(ctx->d_Linv, ctx->d_y, naux,
                                                               ctx->d_h);
    } else {
      k_gemv<<<cdiv((long long)naux * 32, 256), 256, 0, st>>>(ctx->d_Vinv, ctx->d_g,
                                                                         naux, ctx->d_h);
    }
    CKL(PH_J_METRIC);
  }
  {
    PhaseScope ps(ctx, PH_J_COLSUM);
    k_j_colsum<<<dim3(cdiv(ctx->maxK, 32), nbf), 128, 0, st>>>(
        ctx->d_B, ctx->d_panel_off, ctx->d_blk_of, ctx->d_boff, ctx->d_panelK, ctx->d_cmoff,
        ctx->d_colmap, hvec, nbf, naux, dJ);
    CKL(PH_J_COLSUM);
  }
  return filter(ctx, dJ, st);
}

gbjk_status run_k(gbjk_ctx* ctx, int kmethod, const double* dC, int nocc, double* dK) {
  gbjk_status s;
  if ((s = ensure_k_workspace(ctx, nocc))) return s;
  const int nbf = ctx->nbf;
  {
    PhaseScope ps(ctx, PH_GATHER);
    const long long total = (long long)ctx->ncols_total * nocc;
    k_gather_cols<<<cdiv(total, 256), 256, 0, ctx->stream>>>(dC, nocc, ctx->d_colmap,
                                                             ctx->ncols_total, ctx->d_Cg);
    CKL(PH_GATHER);
  }
  if ((s = launch_gemm(ctx, ctx->ht_tile0, ctx->ht_ntiles, false, 1.0, PH_HT, ctx->narrow,
                       ctx->elem_ht, ctx->ht_tn)))
    return s;
  const bool mo = kmethod == GBJK_K_DFMO || ctx->fitted;
  if (!ctx->fitted &&
      (s = launch_gemm(ctx, mo ? ctx->fit_tile0 : ctx->fitV_tile0, ctx->fit_ntiles, false, 1.0,
                       PH_FIT, ctx->narrow, ctx->elem_ht, ctx->ht_tn)))
    return s;
  if ((s = launch_gemm(ctx, mo ? ctx->syrk_tile0 : ctx->lmo_tile0,
                       mo ? ctx->syrk_ntiles : ctx->lmo_ntiles, true, 1.0, PH_KGEMM, false,
                       ctx->elem_k)))
    return s;
  {
    PhaseScope ps(ctx, PH_KREDUCE);
    const long long n2 = (long long)nbf * nbf;
    k_splitk_reduce<<<cdiv(n2, 256), 256, 0, ctx->stream>>>(ctx->d_Kpart, ctx->ksplit, nbf, -1.0,
                                                            mo ? 1 : 0, dK);
    CKL(PH_KREDUCE);
  }
  return filter(ctx, dK);
}

}  // namespace

extern "C" {

gbjk_status gbjk_k_split_plan(int nbf, int naux, int nocc, int* ksplit, long long* kchunk) {
  if (nbf <= 0 || naux <= 0 || nocc <= 0 || !ksplit || !kchunk) return GBJK_INVALID_ARG;
  const long long kdim = (long long)naux * nocc;
  const int nt = (nbf + 63) / 64;
  const int ntile_upper = nt * (nt + 1) / 2;
  int ks = std::max(1, std::min<int>(64, 4 * 152 / std::max(1, ntile_upper)));
  // at least 64 k per part; tiny problems split further so that the few
  // output tiles still spread over many SMs (the FP64 pipe is the bound)
  while (ks > 1 && kdim / ks < 64) --ks;
  long long kc = ((kdim + ks - 1) / ks + 15) / 16 * 16;
  ks = (int)((kdim + kc - 1) / kc);
  *ksplit = ks;
  *kchunk = kc;
  return GBJK_OK;
}

gbjk_status gbjk_create(gbjk_ctx** out, const gbjk_desc* d) {
  if (!out || !d) return GBJK_INVALID_ARG;
  *out = nullptr;
  if (d->nbf <= 0 || d->naux <= 0 || d->nblk <= 0 || !d->blk_size || !d->panel_K || !d->colmap)
    return GBJK_INVALID_ARG;
  if (d->naux > kMaxNaux) return GBJK_INVALID_ARG;
  auto* ctx = new (std::nothrow) gbjk_ctx;
  if (!ctx) return GBJK_OOM;
  ctx->device = d->device;
  ctx->nbf = d->nbf;
  ctx->naux = d->naux;
  ctx->nblk = d->nblk;
  ctx->eps = d->filter_eps;
  ctx->bsize.assign(d->blk_size, d->blk_size + d->nblk);
  ctx->panelK.assign(d->panel_K, d->panel_K + d->nblk);
  ctx->boff.assign(d->nblk + 1, 0);
  ctx->cmoff.assign(d->nblk + 1, 0);
  ctx->panel_off.assign(d->nblk, 0);
  ctx->pg_off.assign(d->nblk, 0);
  long long po = 0, pg = 0;
  for (int I = 0; I < d->nblk; ++I) {
    if (d->blk_size[I] <= 0 || d->panel_K[I] < 0 || d->panel_K[I] > d->nbf) {
      delete ctx;
      return GBJK_INVALID_ARG;
    }
    ctx->boff[I + 1] = ctx->boff[I] + d->blk_size[I];
    ctx->cmoff[I + 1] = ctx->cmoff[I] + d->panel_K[I];
    ctx->panel_off[I] = po;
    ctx->pg_off[I] = pg;
    po += (long long)d->blk_size[I] * d->naux * d->panel_K[I];
    pg += (long long)d->blk_size[I] * d->panel_K[I];
    ctx->maxK = std::max(ctx->maxK, d->panel_K[I]);
  }
  if (ctx->boff[d->nblk] != d->nbf) {
    delete ctx;
    return GBJK_INVALID_ARG;
  }
  ctx->nnz = po;
  ctx->pg_total = pg;
  ctx->ncols_total = ctx->cmoff[d->nblk];
  ctx->colmap.assign(d->colmap, d->colmap + ctx->ncols_total);
  for (int c : ctx->colmap)
    if (c < 0 || c >= d->nbf) {
      delete ctx;
      return GBJK_INVALID_ARG;
    }
  ctx->blk_of.resize(d->nbf);
  for (int I = 0; I < d->nblk; ++I)
    for (int m = ctx->boff[I]; m < ctx->boff[I + 1]; ++m) ctx->blk_of[m] = I;

  if (cudaSetDevice(ctx->device) != cudaSuccess) {
    delete ctx;
    return GBJK_CUDA_ERROR;
  }
  if (cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete ctx;
    return GBJK_CUDA_ERROR;
  }
  if (cudaStreamCreateWithFlags(&ctx->side, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&ctx->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&ctx->ev_join, cudaEventDisableTiming) != cudaSuccess) {
    gbjk_destroy(ctx);
    return GBJK_CUDA_ERROR;
  }
  if (!(ctx->h_err = flag_pool().take())) {
    gbjk_destroy(ctx);
    return GBJK_OOM;
  }
  gbjk_status s;
  auto up = [&](auto** dptr, const auto& vec) -> gbjk_status {
    gbjk_status st = dalloc(ctx, dptr, vec.size());
    if (st) return st;
    if (cudaMemcpy(*dptr, vec.data(), vec.size() * sizeof(vec[0]), cudaMemcpyHostToDevice) !=
        cudaSuccess)
      return fail(ctx, GBJK_CUDA_ERROR, "layout upload failed");
    return GBJK_OK;
  };
  if ((s = up(&ctx->d_blk_of, ctx->blk_of)) || (s = up(&ctx->d_boff, ctx->boff)) ||
      (s = up(&ctx->d_panelK, ctx->panelK)) || (s = up(&ctx->d_cmoff, ctx->cmoff)) ||
      (s = up(&ctx->d_colmap, ctx->colmap)) || (s = up(&ctx->d_panel_off, ctx->panel_off)) ||
      (s = up(&ctx->d_pg_off, ctx->pg_off))) {
    gbjk_destroy(ctx);
    return s;
  }
  ctx->split.init(ctx->nbf, ctx->naux, ctx->nblk, ctx->bsize, ctx->boff, ctx->panelK, ctx->cmoff,
                  ctx->panel_off, ctx->colmap, ctx->blk_of);
  ctx->split.set_dev_layout(ctx->d_panel_off, ctx->d_blk_of, ctx->d_boff, ctx->d_panelK,
                            ctx->d_colmap);
  *out = ctx;
  return GBJK_OK;
}

void gbjk_destroy(gbjk_ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  if (ctx->side) cudaStreamSynchronize(ctx->side);
  ctx->mp2.release();
  ctx->aok.release();
  ctx->asymk.release();
  ctx->scf.release();
  ctx->split.release();
  void* ptrs[] = {ctx->d_blk_of, ctx->d_boff,  ctx->d_panelK, ctx->d_cmoff, ctx->d_colmap,
                  ctx->d_panel_off, ctx->d_pg_off, ctx->d_B, ctx->d_Linv, ctx->d_Vinv,
                  ctx->d_P, ctx->d_Pg, ctx->d_part, ctx->d_g, ctx->d_h, ctx->d_y, ctx->d_J,
                  ctx->d_C, ctx->d_Cg, ctx->d_H, ctx->d_H2, ctx->d_Kpart, ctx->d_K,
                  ctx->d_groups, ctx->d_tiles};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  for (void* p : {(void*)ctx->fb.d_groups, (void*)ctx->fb.d_tiles, (void*)ctx->fb.d_H,
                  (void*)ctx->fb.d_Kpart, (void*)ctx->ob.d_groups, (void*)ctx->ob.d_tiles,
                  (void*)ctx->ob.d_H, (void*)ctx->ob.d_H2, (void*)ctx->ob.d_Kpart})
    if (p) cudaFree(p);
  for (auto& pe : ctx->pending) {
    cudaEventDestroy(pe.second.first);
    cudaEventDestroy(pe.second.second);
  }
  for (auto e : ctx->ev_pool) cudaEventDestroy(e);
  ctx->user_graph.reset();
  ctx->host_graph.reset();
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  if (ctx->side) cudaStreamDestroy(ctx->side);
  if (ctx->ev_fork) cudaEventDestroy(ctx->ev_fork);
  if (ctx->ev_join) cudaEventDestroy(ctx->ev_join);
  if (ctx->h_err) flag_pool().give(ctx->h_err);
  delete ctx;
}

const char* gbjk_last_error(const gbjk_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

gbjk_status gbjk_upload_b(gbjk_ctx* ctx, const double* B) {
  if (!ctx || !B) return fail(ctx, GBJK_INVALID_ARG, "gbjk_upload_b: null argument");
  CK(cudaSetDevice(ctx->device));
  gbjk_status s;
  if ((s = dalloc(ctx, &ctx->d_B, (size_t)ctx->nnz))) return s;
  CK(cudaMemcpy(ctx->d_B, B, (size_t)ctx->nnz * sizeof(double), cudaMemcpyHostToDevice));
  ctx->have_B = true;
  ctx->ws_nocc = -1;  // plans hold d_B
  ctx->mp2.release();
  ctx->aok.release();
  ctx->asymk.release();
  ctx->split.invalidate_b();
  ctx->fb.nocc = -1;  // batched FP64 plans point into the tensor
  ctx->ob.nocc = -1;
  return GBJK_OK;
}

gbjk_status gbjk_upload_metric(gbjk_ctx* ctx, const double* Linv, const double* Vinv) {
  if (!ctx || !Linv || !Vinv) return fail(ctx, GBJK_INVALID_ARG, "gbjk_upload_metric: null argument");
  CK(cudaSetDevice(ctx->device));
  const size_t n2 = (size_t)ctx->naux * ctx->naux;
  gbjk_status s;
  if ((s = dalloc(ctx, &ctx->d_Linv, n2)) || (s = dalloc(ctx, &ctx->d_Vinv, n2))) return s;
  CK(cudaMemcpy(ctx->d_Linv, Linv, n2 * sizeof(double), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(ctx->d_Vinv, Vinv, n2 * sizeof(double), cudaMemcpyHostToDevice));
  ctx->have_metric = true;
  ctx->ws_nocc = -1;
  ctx->mp2.release();
  ctx->aok.release();
  ctx->asymk.release();
  ctx->split.invalidate_b();
  ctx->fb.nocc = -1;  // batched FP64 plans point into the tensor
  ctx->ob.nocc = -1;
  return GBJK_OK;
}

gbjk_status gbjk_set_precision(gbjk_ctx* ctx, int precision, int nslices) {
  if (!ctx) return GBJK_INVALID_ARG;
  if (precision != GBJK_FP64 && precision != GBJK_SPLIT_BF16)
    return fail(ctx, GBJK_INVALID_ARG, "unknown precision");
  if (nslices < 0 || nslices > kMaxSlices)
    return fail(ctx, GBJK_INVALID_ARG, "nslices out of range");
  ctx->epoch++;
  ctx->precision = precision;
  ctx->nslices = nslices;
  return GBJK_OK;
}

gbjk_status gbjk_set_fitted(gbjk_ctx* ctx, int fitted) {
  if (!ctx) return GBJK_INVALID_ARG;
  ctx->epoch++;
  ctx->fitted = fitted != 0;
  ctx->split.fitted = ctx->fitted;
  ctx->mp2.release();
  ctx->aok.release();
  ctx->asymk.release();
  ctx->split.invalidate_b();
  ctx->fb.nocc = -1;  // batched FP64 plans point into the tensor
  ctx->ob.nocc = -1;
  ctx->ws_nocc = -1;  // exchange plan reads H or the fitted H
  return GBJK_OK;
}

gbjk_status gbjk_set_aux_batch(gbjk_ctx* ctx, int rows) {
  if (!ctx || rows < 0) return GBJK_INVALID_ARG;
  ctx->epoch++;
  ctx->split.xb_req = rows;
  ctx->mp2.release();
  ctx->aok.release();
  ctx->asymk.release();
  ctx->split.invalidate_b();
  ctx->fb.nocc = -1;  // batched FP64 plans point into the tensor
  ctx->ob.nocc = -1;
  return GBJK_OK;
}

gbjk_status gbjk_upload_b_synthetic(gbjk_ctx* ctx, unsigned long long seed, double decay) {
  if (!ctx || !(decay > 0)) return fail(ctx, GBJK_INVALID_ARG, "gbjk_upload_b_synthetic: decay");
  CK(cudaSetDevice(ctx->device));
  gbjk_status s;
  if ((s = dalloc(ctx, &ctx->d_B, (size_t)ctx->nnz))) return s;
  {
    PhaseScope ps(ctx, PH_GATHER);
    k_synthetic_panels<<<dim3(cdiv(ctx->maxK, 128), ctx->naux, ctx->nbf), 128, 0, ctx->stream>>>(
        ctx->d_B, ctx->d_panel_off, ctx->d_blk_of, ctx->d_boff, ctx->d_panelK, ctx->d_cmoff,
        ctx->d_colmap, ctx->nbf, ctx->naux, seed, (float)decay);
    CKL(PH_GATHER);
  }
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->have_B = true;
  ctx->ws_nocc = -1;
  ctx->mp2.release();
  ctx->aok.release();
  ctx->asymk.release();
  ctx->split.invalidate_b();
  ctx->fb.nocc = -1;  // batched FP64 plans point into the tensor
  ctx->ob.nocc = -1;
  return GBJK_OK;
}

gbjk_status gbjk_upload_b_eri3c(gbjk_ctx* ctx, const gbjk_shells* ao, const gbjk_shells* aux,
                                const double* sph, const int* blk_shell_off, int nablk,
                                const int* ablk_shell_off, int npairs, const int* pair_I,
                                const int* pair_J, const unsigned char* keep, const int* col_IJ,
                                const int* col_JI) {
  if (!ctx || !ao || !aux || !sph || !blk_shell_off || !ablk_shell_off || !pair_I || !pair_J ||
      !keep || !col_IJ || !col_JI || npairs <= 0 || nablk <= 0)
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_upload_b_eri3c: null argument");
  for (int s = 0; s < ao->nshell; ++s)
    if (ao->l[s] < 0 || ao->l[s] > kEriMaxLao)
      return fail(ctx, GBJK_INVALID_ARG, "gbjk_upload_b_eri3c: AO shells above d are not supported");
  for (int s = 0; s < aux->nshell; ++s) {
    if (aux->l[s] < 0 || aux->l[s] > kEriMaxLaux)
      return fail(ctx, GBJK_INVALID_ARG,
                  "gbjk_upload_b_eri3c: auxiliary shells above f are not supported");
    if (aux->nprim[s] < 1 || aux->nprim[s] > kEriRnChunk)
      return fail(ctx, GBJK_INVALID_ARG,
                  "gbjk_upload_b_eri3c: auxiliary contraction length out of range");
  }
  for (int s = 0; s < ao->nshell; ++s)
    if (ao->nprim[s] < 1)
      return fail(ctx, GBJK_INVALID_ARG, "gbjk_upload_b_eri3c: empty AO contraction");
  CK(cudaSetDevice(ctx->device));
  // host-side tables: shells, primitives, work items (AO shell pairs)
  auto shells = [](const gbjk_shells* b, std::vector<EriShell>& out) {
    out.resize(b->nshell);
    int p0 = 0;
    for (int s = 0; s < b->nshell; ++s) {
      out[s].l = b->l[s];
      out[s].nprim = b->nprim[s];
      out[s].prim0 = p0;
      out[s].bf_off = b->bf_off[s];
      out[s].blk = 0;
      for (int d = 0; d < 3; ++d) out[s].A[d] = b->centers[3 * s + d];
      p0 += b->nprim[s];
    }
    return p0;
  };
  std::vector<EriShell> hao, hax;
  const int npa = shells(ao, hao), npx = shells(aux, hax);
  for (int A = 0; A < nablk; ++A)
    for (int c = ablk_shell_off[A]; c < ablk_shell_off[A + 1]; ++c) hax[c].blk = A;
  // Work items, s-s shell pairs (their own kernel) and the others.  A pair of
  // contracted shells costs a thousand times one of single primitives, and
  // blocks in the order of the pairs left the SMs idle for a third (s-s) and half
  // (others) of the time; so a pair is cut along its auxiliary blocks into
  // items of at most an eighth of an SM's share of the launch (half of one of its
  // four blocks'; a quarter, a sixteenth and so on measure the same), the largest
  // first.  Items of s-s pairs also hold auxiliary shells of one momentum and run
  // in its order: four code paths at once did not fit the instruction cache.
  // (Six waters / jkfit: s-s 4.0 -> 2.6 ms, 3.1 before the order; others 8.0 -> 3.7.)
  std::vector<EriItem> items, rest;
  size_t bra_max[2] = {0, 0}, pair_max = 0;
  // costs of a primitive pair with auxiliary block A: s-s pairs by the block's s,
  // p, d, f shells, then every (la, lb) with all of them
  constexpr int kSs = kEriMaxLaux + 1, kCosts = kSs + (kEriMaxLao + 1) * (kEriMaxLao + 1);
  std::vector<double> unit((size_t)kCosts * nablk, 0.0);
  for (int la = 0; la <= kEriMaxLao; ++la)
    for (int lb = 0; lb <= kEriMaxLao; ++lb) {
      double cost[kEriMaxLaux + 1];
      for (int lc = 0; lc <= kEriMaxLaux; ++lc) cost[lc] = eri_cost(la, lb, lc);
      for (int A = 0; A < nablk; ++A)
        for (int c = ablk_shell_off[A]; c < ablk_shell_off[A + 1]; ++c) {
          const int k = la + lb == 0 ? hax[c].l : kSs + la * (kEriMaxLao + 1) + lb;
          unit[(size_t)k * nablk + A] += hax[c].nprim * cost[hax[c].l];
        }
    }
  struct Pair {
    double cost;
    int kind;  // row of unit
    EriItem it;
  };
  std::vector<Pair> cand[2];
  double total[2] = {0.0, 0.0};
  int nsm = 1;
  CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device));
  for (int p = 0; p < npairs; ++p) {
    const int I = pair_I[p], J = pair_J[p];
    if (I < 0 || J < I || J >= ctx->nblk)
      return fail(ctx, GBJK_INVALID_ARG, "gbjk_upload_b_eri3c: bad block pair");
    double kept[kCosts] = {};
    for (int A = 0; A < nablk; ++A)
      if (keep[(size_t)p * nablk + A])
        for (int k = 0; k < kCosts; ++k) kept[k] += unit[(size_t)k * nablk + A];
    for (int a = blk_shell_off[I]; a < blk_shell_off[I + 1]; ++a)
      for (int b = blk_shell_off[J]; b < blk_shell_off[J + 1]; ++b) {
        if (I == J && b < a) continue;
        const int la = hao[a].l, lb = hao[b].l;
        const int ss = la + lb == 0 ? 0 : 1;
        const int npp = hao[a].nprim * hao[b].nprim;
        const int k0 = ss ? kSs + la * (kEriMaxLao + 1) + lb : 0, k1 = ss ? k0 + 1 : kSs;
        for (int k = k0; k < k1; ++k) {
          const double cost = npp * kept[k];
          cand[ss].push_back({cost, k, {p, a, b, 0, nablk, ss ? ~0 : 1 << k}});
          total[ss] += cost;
        }
        size_t bra = (size_t)npp * eri_pair_size(la, lb);
        pair_max = std::max(pair_max, bra);
        if (ss) bra += (size_t)eri_sph_chunk(la, lb, npp) * eri_sph_size(la, lb);
        bra_max[ss] = std::max(bra_max[ss], bra);
      }
  }
  for (int ss = 0; ss < 2; ++ss) {
    const double most = total[ss] / (8.0 * nsm);
    std::vector<Pair> cut;
    for (const Pair& c : cand[ss]) {
      if (c.cost <= most) {
        if (c.cost > 0) cut.push_back(c);
        continue;
      }
      const double* u = &unit[(size_t)c.kind * nablk];
      const double per = c.cost / std::ceil(c.cost / most) * (1 - 1e-9);
      Pair n{0.0, c.kind, c.it};
      for (int A = 0; A < nablk; ++A) {
        if (!keep[(size_t)c.it.p * nablk + A]) continue;
        n.cost += hao[c.it.a].nprim * hao[c.it.b].nprim * u[A];
        if (n.cost < per) continue;
        n.it.A1 = A + 1;
        cut.push_back(n);
        n = {0.0, c.kind, c.it};
        n.it.A0 = A + 1;
      }
      if (n.cost > 0) cut.push_back(n);
    }
    std::stable_sort(cut.begin(), cut.end(), [ss](const Pair& x, const Pair& y) {
      return ss == 0 && x.kind != y.kind ? x.kind > y.kind : x.cost > y.cost;
    });
    for (const Pair& c : cut) (ss == 0 ? items : rest).push_back(c.it);
  }
  const size_t n_ss = items.size();
  items.insert(items.end(), rest.begin(), rest.end());
  size_t smem_k[2];
  for (int k = 0; k < 2; ++k)
    smem_k[k] = (bra_max[k] + (size_t)kEriWarps * kEriWarpDoubles) * sizeof(double);
  // the pairs' tables and the warps' buffers within 200 KB, the others' matrices
  // (24 KB at most) on top
  if ((pair_max + (size_t)kEriWarps * kEriWarpDoubles) * sizeof(double) > 200 * 1024)
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_upload_b_eri3c: contraction too long for the kernel");
  gbjk_status s;
  if ((s = dalloc(ctx, &ctx->d_B, (size_t)ctx->nnz))) return s;
  CK(cudaMemsetAsync(ctx->d_B, 0, (size_t)ctx->nnz * sizeof(double), ctx->stream));
  // device copies (temporary)
  std::vector<void*> tmp;
  auto up = [&](const void* src, size_t bytes, void** dst) -> cudaError_t {
    cudaError_t e = cudaMalloc(dst, std::max<size_t>(bytes, 1));
    if (e != cudaSuccess) return e;
    tmp.push_back(*dst);
    return cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice);
  };
  void *d_items, *d_ao, *d_ax, *d_aoa, *d_aoc, *d_axa, *d_axc, *d_pI, *d_pJ, *d_keep, *d_aoff,
      *d_cij, *d_cji;
  cudaError_t e = cudaSuccess;
  if (!e) e = up(items.data(), items.size() * sizeof(EriItem), &d_items);
  if (!e) e = up(hao.data(), hao.size() * sizeof(EriShell), &d_ao);
  if (!e) e = up(hax.data(), hax.size() * sizeof(EriShell), &d_ax);
  if (!e) e = up(ao->alpha, (size_t)npa * 8, &d_aoa);
  if (!e) e = up(ao->coef, (size_t)npa * 8, &d_aoc);
  if (!e) e = up(aux->alpha, (size_t)npx * 8, &d_axa);
  if (!e) e = up(aux->coef, (size_t)npx * 8, &d_axc);
  if (!e) e = up(pair_I, (size_t)npairs * 4, &d_pI);
  if (!e) e = up(pair_J, (size_t)npairs * 4, &d_pJ);
  if (!e) e = up(keep, (size_t)npairs * nablk, &d_keep);
  if (!e) e = up(ablk_shell_off, (size_t)(nablk + 1) * 4, &d_aoff);
  if (!e) e = up(col_IJ, (size_t)npairs * 4, &d_cij);
  if (!e) e = up(col_JI, (size_t)npairs * 4, &d_cji);
  if (!e) e = cudaMemcpyToSymbol(c_eri_sph, sph, sizeof(double) * (1 + 9 + 30 + 70));
  if (!e) {
    // compact Hermite index -> (t, u, v), in the order of eri_idx
    int tuv[kEriNR], n = 0;
    for (int sum = 0; sum <= kEriMaxL; ++sum)
      for (int r = 0; r <= sum; ++r)
        for (int v = 0; v <= r; ++v) tuv[n++] = (sum - r) | ((r - v) << 8) | (v << 16);
    e = cudaMemcpyToSymbol(c_eri_tuv, tuv, sizeof(tuv));
  }
  if (!e) {
    double rodd[kEriMaxL + 1];
    for (int j = 0; j <= kEriMaxL; ++j) rodd[j] = 1.0 / (2 * j + 1);
    e = cudaMemcpyToSymbol(c_eri_rodd, rodd, sizeof(rodd));
  }
  void *d_boys = nullptr, *d_ket = nullptr;
  if (!e) {
    std::vector<double> boys(kEriBoysTable);
    eri_boys_table(boys.data());
    e = up(boys.data(), boys.size() * sizeof(double), &d_boys);
  }
  if (!e) {
    e = cudaMalloc(&d_ket, (size_t)npx * kEriKetSize * sizeof(double));
    if (!e) tmp.push_back(d_ket);
  }
  if (!e)
    e = cudaFuncSetAttribute(k_eri3c<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_k[0]);
  if (!e)
    e = cudaFuncSetAttribute(k_eri3c<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_k[1]);
  if (!e && !items.empty()) {
    {
      PhaseScope ps(ctx, PH_GATHER);
      k_eri_ket<<<cdiv(npx, 4), 128, 0, ctx->stream>>>((const EriShell*)d_ax, (int)hax.size(),
                                                        (const double*)d_axa, npx, (double*)d_ket);
      ctx->launches++;
      // [0, n_ss): s-s pairs, [n_ss, end): the others; grid slices of 2^30
      const size_t seg[3] = {0, n_ss, items.size()};
      for (int k = 0; k < 2; ++k)
        for (size_t i0 = seg[k]; i0 < seg[k + 1]; i0 += (1u << 30)) {
          const int n = (int)std::min<size_t>(1u << 30, seg[k + 1] - i0);
          auto kern = k == 0 ? k_eri3c<true> : k_eri3c<false>;
          kern<<<n, 32 * kEriWarps, smem_k[k], ctx->stream>>>(
              (const EriItem*)d_items + i0, (const EriShell*)d_ao, (const EriShell*)d_ax,
              (const double*)d_aoa, (const double*)d_aoc, (const double*)d_axa,
              (const double*)d_axc, (const double*)d_ket, (const double*)d_boys, (const int*)d_pI,
              (const int*)d_pJ,
              (const unsigned char*)d_keep, nablk, (const int*)d_aoff, ctx->d_boff,
              ctx->d_panel_off, ctx->d_panelK, (const int*)d_cij, (const int*)d_cji, ctx->naux,
              ctx->d_B);
          ctx->launches++;
        }
    }
    e = cudaGetLastError();
    if (!e) e = cudaStreamSynchronize(ctx->stream);
  }
  for (void* p : tmp) cudaFree(p);
  if (e != cudaSuccess)
    return fail(ctx, GBJK_CUDA_ERROR, std::string("gbjk_upload_b_eri3c: ") + cudaGetErrorString(e));
  ctx->have_B = true;
  ctx->ws_nocc = -1;
  ctx->mp2.release();
  ctx->aok.release();
  ctx->asymk.release();
  ctx->split.invalidate_b();
  ctx->fb.nocc = -1;  // batched FP64 plans point into the tensor
  ctx->ob.nocc = -1;
  return GBJK_OK;
}

gbjk_status gbjk_download_b(gbjk_ctx* ctx, double* B) {
  if (!ctx || !B || !ctx->have_B) return fail(ctx, GBJK_INVALID_ARG, "gbjk_download_b");
  CK(cudaSetDevice(ctx->device));
  CK(cudaMemcpy(B, ctx->d_B, (size_t)ctx->nnz * sizeof(double), cudaMemcpyDeviceToHost));
  return GBJK_OK;
}

gbjk_status gbjk_download_fitted(gbjk_ctx* ctx, double* B) {
  if (!ctx || !B) return fail(ctx, GBJK_INVALID_ARG, "gbjk_download_fitted");
  if (!ctx->split.b_ready)
    return fail(ctx, GBJK_NOT_READY, "gbjk_download_fitted: no mixed-precision build yet");
  CK(cudaSetDevice(ctx->device));
  CK(cudaStreamSynchronize(ctx->stream));
  CK(cudaMemcpy(B, ctx->split.Bfit, (size_t)ctx->nnz * sizeof(double), cudaMemcpyDeviceToHost));
  return GBJK_OK;
}

gbjk_status gbjk_test_split_stall(gbjk_ctx* ctx, int item, double wait_ms) {
  if (!ctx) return GBJK_INVALID_ARG;
  if (item >= 0 && !(wait_ms >= 1.0 && wait_ms <= 2000.0))
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_test_split_stall: 1 <= wait_ms <= 2000");
  ctx->split.stop_item = item < 0 ? -1 : item;
  ctx->split.spin_ns = item < 0 ? kSpinNs : (unsigned long long)(wait_ms * 1e6);
  ctx->epoch++;  // kernel arguments of a captured build change
  return GBJK_OK;
}

gbjk_status gbjk_test_prefit_room(gbjk_ctx* ctx, long long bytes) {
  if (!ctx) return GBJK_INVALID_ARG;
  ctx->split.prefit_room = bytes < 0 ? ~size_t(0) : (size_t)bytes;
  return GBJK_OK;
}

gbjk_status gbjk_set_occ_batch(gbjk_ctx* ctx, int cols) {
  if (!ctx || cols < 0) return GBJK_INVALID_ARG;
  if (cols != ctx->occ_req) ctx->epoch++;
  ctx->occ_req = cols;
  ctx->ob.nocc = -1;
  return GBJK_OK;
}

gbjk_status gbjk_set_overlap(gbjk_ctx* ctx, int sms) {
  if (!ctx) return GBJK_INVALID_ARG;
  if (sms < -1 || sms > 128) return fail(ctx, GBJK_INVALID_ARG, "gbjk_set_overlap: -1 <= sms <= 128");
  if (sms != ctx->overlap_sms) ctx->epoch++;  // the launch sequence changes
  ctx->overlap_sms = sms;
  ctx->tune.overlap_sms = sms;
  return GBJK_OK;
}

gbjk_status gbjk_set_split_fuse(gbjk_ctx* ctx, int on) {
  if (!ctx) return GBJK_INVALID_ARG;
  if (on != 0 && on != 1) return fail(ctx, GBJK_INVALID_ARG, "gbjk_set_split_fuse: 0 or 1");
  if ((on != 0) != ctx->split.hfuse) {
    ctx->epoch++;  // the launch sequence and the per-build buffers change
    ctx->split.hfuse = on != 0;
    ctx->split.release_build();
  }
  return GBJK_OK;
}
int gbjk_get_split_fuse(const gbjk_ctx* ctx) { return ctx ? (ctx->split.fuses() ? 1 : 0) : -1; }

// --- launch configuration and autotuning -----------------------------------
static gbjk_status check_ready(gbjk_ctx* ctx);
// relative time a candidate must save to replace the incumbent in gbjk_autotune
constexpr double kTuneMargin = 0.005;

gbjk_status gbjk_tune_plan(int nbf, int naux, int nocc, const gbjk_tunables* req,
                           gbjk_tunables* eff, int* ksplit) {
  gbjk_tunables r{};
  if (req) r = *req;
  Fp64Plan pl;
  gbjk_status s = fp64_plan(nbf, naux, nocc, r, &pl);
  if (s) return s;
  if (eff) {
    *eff = r;
    eff->fp64_ht_tn = pl.elem_ht ? 1 : pl.ht_tn;
    eff->fp64_k_tile = pl.elem_k ? 1 : 64;
    eff->fp64_kchunk = pl.kc;
  }
  if (ksplit) *ksplit = pl.ks;
  return GBJK_OK;
}

gbjk_status gbjk_set_tunables(gbjk_ctx* ctx, const gbjk_tunables* t) {
  if (!ctx || !t) return GBJK_INVALID_ARG;
  if (t->split_ksplit < 0 || t->overlap_sms < -1 || t->overlap_sms > 128)
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_set_tunables: split_ksplit or overlap_sms out of range");
  Fp64Plan pl;
  if (fp64_plan(ctx->nbf, ctx->naux, 1, *t, &pl))
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_set_tunables: invalid FP64 choice");
  const gbjk_tunables o = ctx->tune;
  if (o.fp64_ht_tn != t->fp64_ht_tn || o.fp64_k_tile != t->fp64_k_tile ||
      o.fp64_kchunk != t->fp64_kchunk)
    ctx->ws_nocc = -1;  // FP64 plans and workspaces are rebuilt at the next build
  if (o.fp64_ht_tn != t->fp64_ht_tn || o.fp64_k_tile != t->fp64_k_tile ||
      o.fp64_kchunk != t->fp64_kchunk) {
    ctx->fb.nocc = -1;
    ctx->ob.nocc = -1;
  }
  if (o.split_ksplit != t->split_ksplit) {
    ctx->split.ks_req = t->split_ksplit;
    ctx->split.release_build();
  }
  ctx->overlap_sms = t->overlap_sms;
  ctx->tune = *t;
  ctx->epoch++;
  return GBJK_OK;
}

gbjk_status gbjk_get_tunables(const gbjk_ctx* ctx, gbjk_tunables* t) {
  if (!ctx || !t) return GBJK_INVALID_ARG;
  *t = ctx->tune_eff;
  t->split_ksplit = ctx->split.ks_eff;
  t->overlap_sms = ctx->overlap_sms;
  return GBJK_OK;
}

gbjk_status gbjk_tune_signature(const gbjk_ctx* ctx, int kmethod, int nocc, char* sig,
                                size_t len) {
  if (!ctx || !sig || !len) return GBJK_INVALID_ARG;
  cudaDeviceProp prop{};
  std::string dev = "unknown";
  int nsm = 0;
  if (cudaGetDeviceProperties(&prop, ctx->device) == cudaSuccess) {
    dev = prop.name;
    nsm = prop.multiProcessorCount;
  }
  for (char& c : dev)
    if (c == ' ' || c == '|') c = '_';
  long long ksum = 0;
  for (int k : ctx->panelK) ksum += k;
  std::snprintf(sig, len,
                "gbjk1|%s|sm%d|prec%d|k%d|j%d|fit%d|xb%d|hf%d|nbf%d|naux%d|nocc%d|nblk%d|nnz%lld|"
                "kp%lld",
                dev.c_str(), nsm, ctx->precision, kmethod, ctx->jmode, ctx->fitted ? 1 : 0,
                ctx->split.xb_req, ctx->split.hfuse ? 1 : 0, ctx->nbf, ctx->naux, nocc, ctx->nblk,
                ctx->nnz, ksum);
  return GBJK_OK;
}

gbjk_status gbjk_tune_cache_lookup(const char* path, const char* sig, gbjk_tunables* t) {
  if (!path || !sig || !t) return GBJK_INVALID_ARG;
  FILE* f = std::fopen(path, "r");
  if (!f) return GBJK_NOT_READY;
  char line[1024], key[768];
  bool found = false;
  gbjk_tunables v{};
  while (std::fgets(line, sizeof line, f)) {
    gbjk_tunables x{};
    if (std::sscanf(line, "%767s %d %d %lld %d %d", key, &x.fp64_ht_tn, &x.fp64_k_tile,
                    &x.fp64_kchunk, &x.split_ksplit, &x.overlap_sms) == 6 &&
        std::strcmp(key, sig) == 0) {
      v = x;  // the last line of a signature wins
      found = true;
    }
  }
  std::fclose(f);
  if (!found) return GBJK_NOT_READY;
  *t = v;
  return GBJK_OK;
}

gbjk_status gbjk_tune_cache_store(const char* path, const char* sig, const gbjk_tunables* t) {
  if (!path || !sig || !t || std::strlen(sig) >= 768 || std::strchr(sig, ' ') ||
      std::strchr(sig, '\n'))
    return GBJK_INVALID_ARG;
  FILE* f = std::fopen(path, "a");
  if (!f) return GBJK_INVALID_ARG;
  std::fprintf(f, "%s %d %d %lld %d %d\n", sig, t->fp64_ht_tn, t->fp64_k_tile, t->fp64_kchunk,
               t->split_ksplit, t->overlap_sms);
  const bool ok = std::fclose(f) == 0;
  return ok ? GBJK_OK : GBJK_INVALID_ARG;
}

static gbjk_status capture_build(gbjk_ctx* ctx, CapturedBuild& cb, int kmethod, const double* dP,
                                 const double* dC, int nocc, double* dJ, double* dK);

namespace {
std::string tunables_json(const gbjk_tunables& t) {
  char b[256];
  std::snprintf(b, sizeof b,
                "{\"fp64_ht_tn\": %d, \"fp64_k_tile\": %d, \"fp64_kchunk\": %lld, "
                "\"split_ksplit\": %d, \"overlap_sms\": %d}",
                t.fp64_ht_tn, t.fp64_k_tile, t.fp64_kchunk, t.split_ksplit, t.overlap_sms);
  return b;
}

// Mean time of `reps` builds on the context's own buffers; < 0 on failure.
// Each is timed as the engine runs it (every caller path replays a captured
// graph): one ordinary build prepares plans and buffers, the build is
// captured, replayed once untimed, then `reps` replays are timed with CUDA
// events on the context's stream.  (Timing direct launches instead biased
// the choice of the J overlap: the in-order build measured faster there
// and slower as a graph.)
double time_builds(gbjk_ctx* ctx, int kmethod, int nocc, int reps, gbjk_status* st) {
  *st = gbjk_compute_jk_dev(ctx, kmethod, ctx->d_P, ctx->d_C, nocc, ctx->d_J, ctx->d_K);
  if (*st || (*st = gbjk_synchronize(ctx))) return -1.0;
  CapturedBuild cb;
  *st = capture_build(ctx, cb, kmethod, ctx->d_P, ctx->d_C, nocc, ctx->d_J, ctx->d_K);
  if (*st) return -1.0;
  if (cudaGraphLaunch(cb.exec, ctx->stream) != cudaSuccess ||
      (*st = gbjk_synchronize(ctx)) != GBJK_OK) {
    if (!*st) *st = fail(ctx, GBJK_CUDA_ERROR, "autotune: graph launch failed");
    cb.reset();
    return -1.0;
  }
  cudaEvent_t a = get_event(ctx), b = get_event(ctx);
  cudaEventRecord(a, ctx->stream);
  for (int r = 0; r < reps && !*st; ++r)
    if (cudaGraphLaunch(cb.exec, ctx->stream) != cudaSuccess)
      *st = fail(ctx, GBJK_CUDA_ERROR, "autotune: graph launch failed");
  cudaEventRecord(b, ctx->stream);
  if (!*st) *st = gbjk_synchronize(ctx);
  float ms = -1.f;
  if (!*st) cudaEventElapsedTime(&ms, a, b);
  ctx->ev_pool.push_back(a);
  ctx->ev_pool.push_back(b);
  cb.reset();
  return *st ? -1.0 : (double)ms / std::max(1, reps);
}
}  // namespace

gbjk_status gbjk_autotune(gbjk_ctx* ctx, int kmethod, const double* P, const double* C, int nocc,
                          int reps, const char* cache_path, char* report, size_t report_len) {
  gbjk_status s;
  if ((s = check_ready(ctx))) return s;
  if (!P || !C || nocc <= 0 || reps < 0)
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_autotune: density, coefficients and nocc needed");
  if (kmethod != GBJK_K_DFMO && kmethod != GBJK_K_DFLMO)
    return fail(ctx, GBJK_INVALID_ARG, "Invalid kmethod");
  auto put = [&](const std::string& r) {
    if (report && report_len) std::snprintf(report, report_len, "%s", r.c_str());
  };
  char sig[768];
  gbjk_tune_signature(ctx, kmethod, nocc, sig, sizeof sig);
  gbjk_tunables cached{};
  if (cache_path && gbjk_tune_cache_lookup(cache_path, sig, &cached) == GBJK_OK) {
    if ((s = gbjk_set_tunables(ctx, &cached))) return s;
    put(std::string("{\"signature\": \"") + sig + "\", \"source\": \"cache\", \"chosen\": " +
        tunables_json(cached) + "}");
    return GBJK_OK;
  }
  if (reps == 0) return fail(ctx, GBJK_NOT_READY, "gbjk_autotune: signature not in the cache");
  if ((s = ensure_j_workspace(ctx)) || (s = ensure_c_workspace(ctx, nocc))) return s;
  const size_t n2 = (size_t)ctx->nbf * ctx->nbf;
  CK(cudaMemcpyAsync(ctx->d_P, P, n2 * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaMemcpyAsync(ctx->d_C, C, (size_t)ctx->nbf * nocc * sizeof(double),
                     cudaMemcpyHostToDevice, ctx->stream));
  const bool prof = ctx->profile;
  ctx->profile = false;
  ctx->split.profile = false;
  // the choices of the other precision stay; this precision's start from
  // the built-in rules
  const bool fp64 = ctx->precision == GBJK_FP64;
  gbjk_tunables cur = ctx->tune;
  if (fp64) {
    cur.fp64_ht_tn = cur.fp64_k_tile = 0;
    cur.fp64_kchunk = 0;
  } else {
    cur.split_ksplit = cur.overlap_sms = 0;
  }
  if ((s = gbjk_set_tunables(ctx, &cur))) return s;
  std::string cands;
  int ncand = 0;
  auto measure = [&](const gbjk_tunables& t, double* ms) -> gbjk_status {
    gbjk_status st = gbjk_set_tunables(ctx, &t);
    if (st) return st;
    *ms = time_builds(ctx, kmethod, nocc, reps, &st);
    if (st) return st;
    gbjk_tunables eff{};
    gbjk_get_tunables(ctx, &eff);
    char b[64];
    std::snprintf(b, sizeof b, ", \"ms\": %.5f}", *ms);
    cands += (ncand++ ? ", " : "") + std::string("{\"requested\": ") + tunables_json(t) +
             ", \"effective\": " + tunables_json(eff) + b;
    return GBJK_OK;
  };
  double best = 0.0;
  s = measure(cur, &best);
  gbjk_tunables base{};
  gbjk_get_tunables(ctx, &base);  // what the rules chose
  const long long big = 2 * kElemOutputs;  // one thread per output beyond: far too slow
  // one dimension at a time, each starting from the best so far
  std::vector<std::vector<gbjk_tunables>> dims;
  if (fp64) {
    std::vector<gbjk_tunables> d1, d2, d3;
    for (int tn : {1, 16, 32, 64}) {
      if (tn == 1 && (long long)ctx->nbf * ctx->naux * nocc > big) continue;
      gbjk_tunables t{};
      t.fp64_ht_tn = tn;
      d1.push_back(t);
    }
    for (int kt : {1, 64}) {
      gbjk_tunables t{};
      t.fp64_k_tile = kt;
      d2.push_back(t);
    }
    for (long long mul : {1LL, 2LL, 4LL}) {  // chunk x 1/2, 1, 2
      gbjk_tunables t{};
      t.fp64_kchunk = std::max(16LL, base.fp64_kchunk * mul / 2);
      d3.push_back(t);
    }
    dims = {d1, d2, d3};
  } else {
    std::vector<gbjk_tunables> d1, d2;
    for (int mul : {1, 2, 4}) {  // parts x 1/2, 1, 2
      gbjk_tunables t{};
      t.split_ksplit = std::max(1, base.split_ksplit * mul / 2);
      d1.push_back(t);
    }
    for (int o : {0, -1, 8}) {
      gbjk_tunables t{};
      t.overlap_sms = o;
      d2.push_back(t);
    }
    dims = {d1, d2};
  }
  for (size_t d = 0; d < dims.size() && !s; ++d) {
    gbjk_tunables pick = cur;
    for (const gbjk_tunables& c : dims[d]) {
      gbjk_tunables t = cur;
      if (fp64) {
        if (d == 0) t.fp64_ht_tn = c.fp64_ht_tn;
        if (d == 1) t.fp64_k_tile = c.fp64_k_tile;
        if (d == 2) t.fp64_kchunk = c.fp64_kchunk;
      } else {
        if (d == 0) t.split_ksplit = c.split_ksplit;
        if (d == 1) t.overlap_sms = c.overlap_sms;
      }
      double ms = 0.0;
      if ((s = measure(t, &ms))) break;
      // a candidate replaces the incumbent only when clearly faster: the
      // candidates of one dimension often lie within 1 % of each other,
      // about the spread of repeated timings
      if (ms < best * (1.0 - kTuneMargin)) {
        best = ms;
        pick = t;
      }
    }
    cur = pick;
  }
  ctx->profile = prof;
  ctx->split.profile = prof;
  if (s) return s;
  if ((s = gbjk_set_tunables(ctx, &cur))) return s;
  if (cache_path && gbjk_tune_cache_store(cache_path, sig, &cur) != GBJK_OK)
    return fail(ctx, GBJK_INVALID_ARG, std::string("gbjk_autotune: cannot write ") + cache_path);
  char b[64];
  std::snprintf(b, sizeof b, ", \"best_ms\": %.5f", best);
  put(std::string("{\"signature\": \"") + sig + "\", \"source\": \"timed\", \"reps\": " +
      std::to_string(reps) + ", \"chosen\": " + tunables_json(cur) + b +
      ", \"candidates\": [" + cands + "]}");
  return GBJK_OK;
}

int gbjk_get_overlap(const gbjk_ctx* ctx) { return ctx ? ctx->overlap_sms : -1; }

gbjk_status gbjk_set_jmode(gbjk_ctx* ctx, int jmode) {
  if (!ctx) return GBJK_INVALID_ARG;
  if (jmode != GBJK_J_VINV && jmode != GBJK_J_CHOLESKY)
    return fail(ctx, GBJK_INVALID_ARG, "unknown J mode");
  ctx->epoch++;
  ctx->jmode = jmode;
  return GBJK_OK;
}

static gbjk_status check_ready(gbjk_ctx* ctx) {
  if (!ctx) return GBJK_INVALID_ARG;
  if (!ctx->have_B || (!ctx->have_metric && !ctx->fitted))
    return fail(ctx, GBJK_NOT_READY, "3-center tensor and metric must be uploaded first");
  if (cudaSetDevice(ctx->device) != cudaSuccess)
    return fail(ctx, GBJK_CUDA_ERROR, "cudaSetDevice failed");
  return GBJK_OK;
}

// FP64 exchange of a pre-fitted tensor with an auxiliary batch size set
static bool fp64_batched(const gbjk_ctx* ctx) {
  return ctx->fitted && ctx->split.xb_req > 0 && ctx->split.xb_req < ctx->naux;
}
// FP64 exchange of an unfitted tensor in occupied batches
static bool fp64_occ_batched(const gbjk_ctx* ctx, int nocc) {
  return !ctx->fitted && ctx->occ_req > 0 && ctx->occ_req < nocc;
}

static gbjk_status prepare_split(gbjk_ctx* ctx, int nocc) {
  if (ctx->precision != GBJK_SPLIT_BF16) return GBJK_OK;
  return ctx->split.prepare(ctx->stream, ctx->d_B, ctx->d_Linv, nocc, &ctx->launches, &ctx->err);
}

// Work forked to the side stream: whatever way the build returns, the context's
// stream waits for it, so that the caller's next use of J, P or the J buffers on
// that stream (or after a synchronisation with it) follows.
struct SideFork {
  gbjk_ctx* ctx;
  bool on = false;
  explicit SideFork(gbjk_ctx* c) : ctx(c) {}
  // the side stream goes on from `from` (recorded on the context's stream)
  cudaError_t fork(cudaEvent_t from) {
    const cudaError_t e = cudaStreamWaitEvent(ctx->side, from, 0);
    on = on || e == cudaSuccess;
    return e;
  }
  cudaError_t join() {
    on = false;
    const cudaError_t e = cudaEventRecord(ctx->ev_join, ctx->side);
    return e != cudaSuccess ? e : cudaStreamWaitEvent(ctx->stream, ctx->ev_join, 0);
  }
  ~SideFork() {
    if (on && join() != cudaSuccess) cudaGetLastError();  // the build's own error stands
  }
};

// Mixed-precision J + K.  The density rows of every panel ride along as
// extra B-operand rows of the split half transform, whose epilogue emits
// the partials of dt = L^-1 g; J = (L^-1 B)^T dt is one pass over the compact
// copy of the prefitted tensor (6 bytes an element, the upper block triangle where
// it is symmetric), in FP32 pairs.  Without dJ the density rows are zero.
static gbjk_status run_jk_split(gbjk_ctx* ctx, const double* dP, const double* dC, int nocc,
                                double* dJ, double* dK) {
  const int nbf = ctx->nbf, naux = ctx->naux;
  gbjk_status s;
  // J = (L^-1 B)^T dt needs only the half transform's density partials: with
  // overlap on (and no per-phase timing, whose events sit on one stream) it
  // runs on the side stream beside the exchange.  Where J alone fills the
  // GPU's memory bandwidth the two only delay each other, and the phases run in
  // order (kOverlapJBytes).
  const bool fused = dJ && ctx->split.fused_j();
  const bool overlap = fused && !ctx->profile &&
                       (ctx->overlap_sms > 0 ||
                        (ctx->overlap_sms == 0 && ctx->split.j_bytes() < kOverlapJBytes));
  ctx->split.ev_ht = overlap ? ctx->ev_fork : nullptr;
  ctx->split.k_grid = overlap ? ctx->overlap_sms : 0;
  s = ctx->split.run_k(ctx->stream, dC, dJ ? dP : nullptr, dK, &ctx->launches, &ctx->err);
  ctx->split.ev_ht = nullptr;
  ctx->split.k_grid = 0;
  if (s) return s;
  SideFork side(ctx);
  if (fused) {
    cudaStream_t js = overlap ? ctx->side : ctx->stream;
    if (overlap) CK(side.fork(ctx->ev_fork));
    CK(cudaMemsetAsync(dJ, 0, (size_t)nbf * nbf * sizeof(double), js));
    {
      PhaseScope ps(ctx, PH_J_REDUCE);
      k_reduce_rows16<<<cdiv(naux, 32), 512, 0, js>>>(ctx->split.d_dpart, nbf, naux,
                                                      ctx->split.d_dt);
      CKL(PH_J_REDUCE);
    }
    {
      PhaseScope ps(ctx, PH_J_COLSUM);
      ctx->split.run_j_cols(js, ctx->split.d_dt, dJ, &ctx->launches);
      ctx->launches--;  // CKL counts one
      CKL(PH_J_COLSUM);
    }
    if (ctx->eps > 0) {
      PhaseScope ps(ctx, PH_FILTER);
      k_block_filter<<<cdiv((long long)ctx->nblk * ctx->nblk, 8), 256, 0, js>>>(
          dJ, ctx->nbf, ctx->d_boff, ctx->nblk, ctx->eps);
      CKL(PH_FILTER);
    }
  }
  if ((s = filter(ctx, dK))) return s;
  if (overlap) CK(side.join());
  if (!dJ || fused) return GBJK_OK;
  return run_j(ctx, dP, dJ, ctx->stream);  // auxiliary-batched: FP64 J
}

gbjk_status gbjk_compute_jk_dev(gbjk_ctx* ctx, int kmethod, const double* dP, const double* dC,
                                int nocc, double* dJ, double* dK) {
  gbjk_status s;
  if ((s = check_ready(ctx))) return s;
  if (kmethod != GBJK_K_DFMO && kmethod != GBJK_K_DFLMO)
    return fail(ctx, GBJK_INVALID_ARG, "Invalid kmethod");
  if ((dK && (!dC || nocc <= 0)) || (dJ && !dP))
    return fail(ctx, GBJK_INVALID_ARG, "missing density or coefficients");
  if ((s = ensure_j_workspace(ctx))) return s;
  if (dK) {
    if (ctx->precision == GBJK_SPLIT_BF16) {
      if ((s = prepare_split(ctx, nocc))) return s;
      return run_jk_split(ctx, dP, dC, nocc, dJ, dK);
    }
    // every plan and buffer before J starts beside K
    s = fp64_batched(ctx)             ? ensure_k_batched(ctx, nocc)
        : fp64_occ_batched(ctx, nocc) ? ensure_k_occ_batched(ctx, nocc)
                                      : ensure_k_workspace(ctx, nocc);
    if (s) return s;
  }
  // J and K share nothing but the tensor: J runs on the side stream beside K
  // unless phases are asked for in order or timed (water: a dozen launches of a
  // few microseconds in two lines instead of one, 95 -> 70 us per call)
  const bool beside = dJ && dK && ctx->overlap_sms >= 0 && !ctx->profile;
  cudaStream_t js = beside ? ctx->side : ctx->stream;
  SideFork side(ctx);
  if (beside) {
    CK(cudaEventRecord(ctx->ev_fork, ctx->stream));
    CK(side.fork(ctx->ev_fork));
  }
  if (dJ && (s = run_j(ctx, dP, dJ, js))) return s;
  if (dK) {
    s = fp64_batched(ctx)               ? run_k_batched(ctx, dC, nocc, dK)
        : fp64_occ_batched(ctx, nocc)   ? run_k_occ_batched(ctx, kmethod, dC, nocc, dK)
                                        : run_k(ctx, kmethod, dC, nocc, dK);
    if (s) return s;
  }
  if (beside) CK(side.join());
  return GBJK_OK;
}

static uint64_t build_epoch(const gbjk_ctx* ctx) { return ctx->epoch + ctx->split.frees; }

// Record one device-pointer Fock build (plans and buffers already prepared
// by an ordinary build) as a CUDA graph on the context's stream.
static gbjk_status capture_build(gbjk_ctx* ctx, CapturedBuild& cb, int kmethod, const double* dP,
                                 const double* dC, int nocc, double* dJ, double* dK) {
  cb.reset();
  const uint64_t ep = build_epoch(ctx);
  const bool prof = ctx->profile;
  ctx->profile = false;
  ctx->split.profile = false;
  cudaError_t e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) {
    ctx->profile = prof;
    ctx->split.profile = prof;
    return fail(ctx, GBJK_CUDA_ERROR, std::string("graph capture: ") + cudaGetErrorString(e));
  }
  const int64_t l0 = ctx->launches;
  gbjk_status s = gbjk_compute_jk_dev(ctx, kmethod, dP, dC, nocc, dJ, dK);
  const int64_t n = ctx->launches - l0;
  ctx->launches = l0;
  cudaGraph_t g = nullptr;
  e = cudaStreamEndCapture(ctx->stream, &g);
  ctx->profile = prof;
  ctx->split.profile = prof;
  if (s || e != cudaSuccess || build_epoch(ctx) != ep) {
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    if (s) return s;
    return fail(ctx, GBJK_CUDA_ERROR,
                e != cudaSuccess ? std::string("graph capture: ") + cudaGetErrorString(e)
                                 : std::string("graph capture: the build replaced engine buffers"));
  }
  cudaGraphExec_t x = nullptr;
  e = cudaGraphInstantiate(&x, g, 0);
  if (e != cudaSuccess) {
    cudaGraphDestroy(g);
    cudaGetLastError();
    return fail(ctx, GBJK_CUDA_ERROR, std::string("graph instantiate: ") + cudaGetErrorString(e));
  }
  cb.graph = g;
  cb.exec = x;
  cb.launches = n;
  cb.epoch = ep;
  return GBJK_OK;
}

gbjk_status gbjk_capture_graph(gbjk_ctx* ctx, int kmethod, const double* dP, const double* dC,
                               int nocc, double* dJ, double* dK) {
  gbjk_status s;
  if (!ctx) return GBJK_INVALID_ARG;
  // one ordinary build prepares every plan, buffer and kernel attribute so
  // that the captured sequence contains launches and memsets only
  if ((s = gbjk_compute_jk_dev(ctx, kmethod, dP, dC, nocc, dJ, dK))) return s;
  if ((s = gbjk_synchronize(ctx))) return s;
  return capture_build(ctx, ctx->user_graph, kmethod, dP, dC, nocc, dJ, dK);
}

gbjk_status gbjk_launch_graph(gbjk_ctx* ctx) {
  if (!ctx) return GBJK_INVALID_ARG;
  CapturedBuild& cb = ctx->user_graph;
  if (!cb.exec) return fail(ctx, GBJK_NOT_READY, "no captured build");
  if (cb.epoch != build_epoch(ctx)) {
    cb.reset();
    return fail(ctx, GBJK_NOT_READY,
                "engine buffers or settings changed since the build was captured; capture again");
  }
  CK(cudaGraphLaunch(cb.exec, ctx->stream));
  ctx->launches += cb.launches;
  return GBJK_OK;
}

gbjk_status gbjk_synchronize(gbjk_ctx* ctx) {
  if (!ctx) return GBJK_INVALID_ARG;
  // the flag of a timed-out wait comes back with the results: reading it after
  // the synchronisation was a second round trip
  const bool flag = ctx->precision == GBJK_SPLIT_BF16 && ctx->split.d_err;
  *ctx->h_err = 0;
  if (flag)
    CK(cudaMemcpyAsync(ctx->h_err, ctx->split.d_err, sizeof(int), cudaMemcpyDeviceToHost,
                       ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  resolve_profile(ctx);
  if (flag) {
    const int code = *ctx->h_err;
    if (code != 0)
      return fail(ctx, GBJK_TIMEOUT,
                  "split GEMM: a pipeline wait timed out (code " + std::to_string(code) + ")");
  }
  return GBJK_OK;
}

void* gbjk_stream(gbjk_ctx* ctx) { return ctx ? (void*)ctx->stream : nullptr; }

gbjk_status gbjk_compute_jk(gbjk_ctx* ctx, int kmethod, const double* P, const double* Cocc,
                            int nocc, double* J, double* K) {
  gbjk_status s;
  if ((s = check_ready(ctx))) return s;
  if ((s = ensure_j_workspace(ctx))) return s;
  const size_t n2 = (size_t)ctx->nbf * ctx->nbf;
  if (K) {
    if (!Cocc || nocc <= 0) return fail(ctx, GBJK_INVALID_ARG, "missing coefficients");
    if ((s = ensure_c_workspace(ctx, nocc))) return s;
    CK(cudaMemcpyAsync(ctx->d_C, Cocc, (size_t)ctx->nbf * nocc * sizeof(double),
                       cudaMemcpyHostToDevice, ctx->stream));
  }
  if (J) {
    if (!P) return fail(ctx, GBJK_INVALID_ARG, "missing density");
    CK(cudaMemcpyAsync(ctx->d_P, P, n2 * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  }
  const int key_nocc = K ? nocc : 0;
  const bool same_shape = ctx->host_kmethod == kmethod && ctx->host_nocc == key_nocc &&
                          ctx->host_j == (J != nullptr) && ctx->host_k == (K != nullptr) &&
                          ctx->host_graph.epoch == build_epoch(ctx);
  const bool replay = !ctx->profile && same_shape && ctx->host_graph.exec;
  if (replay) {
    CK(cudaGraphLaunch(ctx->host_graph.exec, ctx->stream));
    ctx->launches += ctx->host_graph.launches;
  } else if ((s = gbjk_compute_jk_dev(ctx, kmethod, J ? ctx->d_P : nullptr, K ? ctx->d_C : nullptr,
                                      nocc, J ? ctx->d_J : nullptr, K ? ctx->d_K : nullptr))) {
    return s;
  }
  if (J) CK(cudaMemcpyAsync(J, ctx->d_J, n2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  if (K) CK(cudaMemcpyAsync(K, ctx->d_K, n2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  if ((s = gbjk_synchronize(ctx))) return s;
  if (!replay && !ctx->profile && !(same_shape && ctx->host_uncapturable)) {
    // record this shape for the next call; a build that cannot be captured
    // keeps its direct launches
    ctx->host_kmethod = kmethod;
    ctx->host_nocc = key_nocc;
    ctx->host_j = J != nullptr;
    ctx->host_k = K != nullptr;
    const std::string err = ctx->err;
    ctx->host_uncapturable =
        capture_build(ctx, ctx->host_graph, kmethod, J ? ctx->d_P : nullptr,
                      K ? ctx->d_C : nullptr, nocc, J ? ctx->d_J : nullptr,
                      K ? ctx->d_K : nullptr) != GBJK_OK;
    if (ctx->host_uncapturable) {
      ctx->host_graph.epoch = build_epoch(ctx);
      ctx->err = err;
    }
  }
  return GBJK_OK;
}

void* gbjk_host_alloc(size_t bytes) {
  void* p = nullptr;
  if (cudaHostAlloc(&p, bytes ? bytes : 1, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return p;
}

void gbjk_host_free(void* p) {
  if (p) cudaFreeHost(p);
}

gbjk_status gbjk_compute_j(gbjk_ctx* ctx, const double* P, double* J) {
  if (!P || !J) return fail(ctx, GBJK_INVALID_ARG, "gbjk_compute_j: null argument");
  return gbjk_compute_jk(ctx, GBJK_K_DFMO, P, nullptr, 0, J, nullptr);
}

gbjk_status gbjk_compute_k(gbjk_ctx* ctx, int kmethod, const double* Cocc, int nocc, double* K) {
  if (!Cocc || !K) return fail(ctx, GBJK_INVALID_ARG, "gbjk_compute_k: null argument");
  return gbjk_compute_jk(ctx, kmethod, nullptr, Cocc, nocc, nullptr, K);
}

size_t gbjk_device_bytes(const gbjk_ctx* ctx) {
  return ctx ? ctx->dev_bytes + ctx->split.bytes + ctx->mp2.bytes + ctx->aok.bytes + ctx->scf.bytes +
                   ctx->asymk.bytes
             : 0;
}
int64_t gbjk_kernel_launches(const gbjk_ctx* ctx) { return ctx ? ctx->launches : 0; }

gbjk_status gbjk_profile(gbjk_ctx* ctx, int enable) {
  if (!ctx) return GBJK_INVALID_ARG;
  cudaStreamSynchronize(ctx->stream);
  resolve_profile(ctx);
  ctx->profile = enable != 0;
  ctx->split.profile = enable != 0;
  ctx->mp2.profile = enable != 0;
  ctx->mp2.reset_profile();
  for (int i = 0; i < PH_COUNT; ++i) {
    ctx->ph_ms[i] = 0;
    ctx->ph_launch[i] = 0;
  }
  ctx->split.reset_profile();
  return GBJK_OK;
}

int gbjk_profile_read(const gbjk_ctx* ctx, int idx, const char** name, double* ms,
                      int64_t* launches) {
  if (!ctx || idx < 0) return 0;
  if (idx < PH_COUNT) {
    if (name) *name = kPhaseNames[idx];
    if (ms) *ms = ctx->ph_ms[idx];
    if (launches) *launches = ctx->ph_launch[idx];
    return 1;
  }
  gbjk_ctx* c = const_cast<gbjk_ctx*>(ctx);
  if (c->split.profile_read(idx - PH_COUNT, name, ms, launches)) return 1;
  return c->mp2.profile_read(idx - PH_COUNT - 4, name, ms, launches);
}

// --- DF-AO exchange -------------------------------------------------------------

static AoKState::Layout aok_layout(gbjk_ctx* ctx) {
  AoKState::Layout L;
  L.nbf = ctx->nbf;
  L.naux = ctx->naux;
  L.nblk = ctx->nblk;
  L.ncols_total = ctx->ncols_total;
  L.maxK = ctx->maxK;
  L.bsize = &ctx->bsize;
  L.boff = &ctx->boff;
  L.panelK = &ctx->panelK;
  L.cmoff = &ctx->cmoff;
  L.panel_off = &ctx->panel_off;
  L.d_blk_of = ctx->d_blk_of;
  L.d_boff = ctx->d_boff;
  L.d_panelK = ctx->d_panelK;
  L.d_cmoff = ctx->d_cmoff;
  L.d_colmap = ctx->d_colmap;
  L.d_panel_off = ctx->d_panel_off;
  return L;
}

gbjk_status gbjk_compute_k_ao_dev(gbjk_ctx* ctx, const double* dP, double* dK) {
  gbjk_status s;
  if ((s = check_ready(ctx))) return s;
  if (!dP || !dK) return fail(ctx, GBJK_INVALID_ARG, "gbjk_compute_k_ao_dev: null argument");
  const AoKState::Layout L = aok_layout(ctx);
  if (ctx->precision == GBJK_SPLIT_BF16 && !ctx->split.b_ready &&
      (s = ctx->split.prepare_b(ctx->stream, ctx->d_B, ctx->d_Linv, &ctx->launches, &ctx->err)))
    return s;
  if (ctx->precision == GBJK_SPLIT_BF16 && (s = ctx->split.clear_error(ctx->stream)))
    return fail(ctx, s, "split path: memset failed");
  if ((s = ctx->aok.prepare(ctx->stream, ctx->precision, L, ctx->d_B,
                            ctx->fitted ? nullptr : ctx->d_Vinv, ctx->split, &ctx->launches,
                            &ctx->err)))
    return s;
  {
    PhaseScope ps(ctx, PH_KGEMM);
    if ((s = ctx->aok.run(ctx->stream, L, dP, dK, ctx->split, &ctx->launches, &ctx->err)))
      return s;
  }
  return filter(ctx, dK);
}

gbjk_status gbjk_compute_k_ao(gbjk_ctx* ctx, const double* P, double* K) {
  gbjk_status s;
  if ((s = check_ready(ctx))) return s;
  if (!P || !K) return fail(ctx, GBJK_INVALID_ARG, "gbjk_compute_k_ao: null argument");
  if ((s = ensure_j_workspace(ctx))) return s;
  const size_t n2 = (size_t)ctx->nbf * ctx->nbf;
  CK(cudaMemcpyAsync(ctx->d_P, P, n2 * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  if ((s = gbjk_compute_k_ao_dev(ctx, ctx->d_P, ctx->d_K))) return s;
  CK(cudaMemcpyAsync(K, ctx->d_K, n2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  return gbjk_synchronize(ctx);
}

// --- non-symmetric DF-LMO exchange -----------------------------------------

gbjk_status gbjk_compute_k_lmo_asym(gbjk_ctx* ctx, const double* U, const double* Vt, int nocc,
                                    double* K) {
  gbjk_status s;
  if ((s = check_ready(ctx))) return s;
  if (!U || !Vt || !K || nocc <= 0)
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_compute_k_lmo_asym: null argument or nocc <= 0");
  if (ctx->precision == GBJK_FP64 && ctx->fitted)
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_compute_k_lmo_asym: FP64 path needs the metric");
  if ((s = ensure_j_workspace(ctx))) return s;
  if (ctx->precision == GBJK_SPLIT_BF16 && !ctx->split.b_ready &&
      (s = ctx->split.prepare_b(ctx->stream, ctx->d_B, ctx->d_Linv, &ctx->launches, &ctx->err)))
    return s;
  AsymKState& a = ctx->asymk;
  if (!a.ready || a.precision != ctx->precision || a.nocc != nocc) {
    AsymKState::Layout L{ctx->nbf, ctx->naux, ctx->nblk, ctx->ncols_total, &ctx->bsize,
                         &ctx->boff, &ctx->panelK, &ctx->cmoff, &ctx->panel_off};
    if ((s = a.plan(ctx->precision, nocc, L, ctx->d_B, ctx->d_Vinv, ctx->split, &ctx->err)))
      return s;
  }
  const int nbf = ctx->nbf;
  CK(cudaMemcpyAsync(a.d_U, U, (size_t)nbf * nocc * 8, cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaMemcpyAsync(a.d_V, Vt, (size_t)nbf * nocc * 8, cudaMemcpyHostToDevice, ctx->stream));
  if (ctx->precision == GBJK_SPLIT_BF16 && (s = ctx->split.clear_error(ctx->stream)))
    return fail(ctx, s, "split path: memset failed");
  {
    PhaseScope ps(ctx, PH_KGEMM);
    if ((s = a.run(ctx->stream, nbf, ctx->naux, ctx->nblk, ctx->ncols_total, ctx->d_colmap,
                   ctx->d_K, ctx->split, &ctx->launches, &ctx->err)))
      return s;
  }
  if ((s = filter(ctx, ctx->d_K))) return s;
  CK(cudaMemcpyAsync(K, ctx->d_K, (size_t)nbf * nbf * 8, cudaMemcpyDeviceToHost, ctx->stream));
  return gbjk_synchronize(ctx);
}

// --- SCF iteration on the device -------------------------------------------

gbjk_status gbjk_scf_begin(gbjk_ctx* ctx, const double* H, const double* S, const double* X,
                           int nocc, int max_diis) {
  gbjk_status s;
  if ((s = check_ready(ctx))) return s;
  if (!H || !S || !X || nocc <= 0 || nocc > ctx->nbf || max_diis < 1 || max_diis > kScfMaxDiis)
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_scf_begin: H, S, X, 0 < nocc <= nbf, 1 <= max_diis <= 16");
  return (s = ctx->scf.begin(ctx->stream, ctx->nbf, nocc, max_diis, H, S, X, &ctx->err))
             ? fail(ctx, s, ctx->err)
             : GBJK_OK;
}

gbjk_status gbjk_scf_build(gbjk_ctx* ctx, int kmethod, const double* Cocc, int slot, double* out) {
  gbjk_status s;
  if ((s = check_ready(ctx))) return s;
  ScfState& sc = ctx->scf;
  if (!sc.ready) return fail(ctx, GBJK_NOT_READY, "gbjk_scf_build: call gbjk_scf_begin first");
  if (!Cocc || !out || slot < 0 || slot >= sc.nslots)
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_scf_build: coefficients, output and 0 <= slot < max_diis");
  if (kmethod != GBJK_K_DFMO && kmethod != GBJK_K_DFLMO)
    return fail(ctx, GBJK_INVALID_ARG, "Invalid kmethod");
  CK(cudaMemcpyAsync(sc.dC, Cocc, (size_t)sc.nbf * sc.nocc * sizeof(double),
                     cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaMemcpyAsync(sc.dslot, &slot, sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
  const bool stale = !sc.gA || sc.epA != build_epoch(ctx) || sc.kmethodA != kmethod;
  if (!stale && !ctx->profile) {
    CK(cudaGraphLaunch(sc.gA, ctx->stream));
    ctx->launches += sc.launchesA;
  } else {
    // direct launches (they prepare every plan and buffer of the build) ...
    ctx->launches += sc.launch_pre(ctx->stream);
    CK(cudaGetLastError());
    if ((s = gbjk_compute_jk_dev(ctx, kmethod, sc.dPt, sc.dC, sc.nocc, sc.dJ, sc.dK))) return s;
    ctx->launches += sc.launch_post(ctx->stream);
    CK(cudaGetLastError());
  }
  CK(cudaMemcpyAsync(out, sc.dscal, (size_t)(2 + sc.nslots) * sizeof(double),
                     cudaMemcpyDeviceToHost, ctx->stream));
  if ((s = gbjk_synchronize(ctx))) return s;
  if (stale && !ctx->profile) {
    // ... then the same sequence is recorded for the next iterations
    if (sc.gA) cudaGraphExecDestroy(sc.gA);
    if (sc.grA) cudaGraphDestroy(sc.grA);
    sc.gA = nullptr;
    sc.grA = nullptr;
    const uint64_t ep = build_epoch(ctx);
    if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      const int64_t l0 = ctx->launches;
      int64_t n = sc.launch_pre(ctx->stream);
      gbjk_status cs = gbjk_compute_jk_dev(ctx, kmethod, sc.dPt, sc.dC, sc.nocc, sc.dJ, sc.dK);
      n += sc.launch_post(ctx->stream) + (ctx->launches - l0);
      ctx->launches = l0;
      cudaGraph_t g = nullptr;
      const cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
      if (!cs && e == cudaSuccess && build_epoch(ctx) == ep &&
          cudaGraphInstantiate(&sc.gA, g, 0) == cudaSuccess) {
        sc.grA = g;
        sc.epA = ep;
        sc.kmethodA = kmethod;
        sc.launchesA = n;
      } else if (g) {
        cudaGraphDestroy(g);
      }
    }
    cudaGetLastError();  // a build that cannot be captured keeps direct launches
  }
  return GBJK_OK;
}

gbjk_status gbjk_scf_extrapolate(gbjk_ctx* ctx, const double* coef, double* Fo) {
  if (!ctx) return GBJK_INVALID_ARG;
  ScfState& sc = ctx->scf;
  if (!sc.ready) return fail(ctx, GBJK_NOT_READY, "gbjk_scf_extrapolate: call gbjk_scf_begin first");
  if (!coef || !Fo) return fail(ctx, GBJK_INVALID_ARG, "gbjk_scf_extrapolate: null argument");
  CK(cudaSetDevice(ctx->device));
  CK(cudaMemcpyAsync(sc.dcoef, coef, (size_t)sc.nslots * sizeof(double), cudaMemcpyHostToDevice,
                     ctx->stream));
  if (!sc.gB) {
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    sc.launchesB = sc.launch_extrapolate(ctx->stream);
    CK(cudaStreamEndCapture(ctx->stream, &g));
    CK(cudaGraphInstantiate(&sc.gB, g, 0));
    sc.grB = g;
  }
  CK(cudaGraphLaunch(sc.gB, ctx->stream));
  ctx->launches += sc.launchesB;
  CK(cudaMemcpyAsync(Fo, sc.dFo, (size_t)sc.nbf * sc.nbf * sizeof(double),
                     cudaMemcpyDeviceToHost, ctx->stream));
  return gbjk_synchronize(ctx);
}

gbjk_status gbjk_scf_read(gbjk_ctx* ctx, int slot, double* F, double* J, double* K) {
  if (!ctx) return GBJK_INVALID_ARG;
  ScfState& sc = ctx->scf;
  if (!sc.ready) return fail(ctx, GBJK_NOT_READY, "gbjk_scf_read: call gbjk_scf_begin first");
  if (slot < 0 || slot >= sc.nslots) return fail(ctx, GBJK_INVALID_ARG, "gbjk_scf_read: slot");
  CK(cudaSetDevice(ctx->device));
  const size_t n2 = (size_t)sc.nbf * sc.nbf;
  if (F)
    CK(cudaMemcpyAsync(F, sc.dFring + (size_t)slot * n2, n2 * 8, cudaMemcpyDeviceToHost,
                       ctx->stream));
  if (J) CK(cudaMemcpyAsync(J, sc.dJ, n2 * 8, cudaMemcpyDeviceToHost, ctx->stream));
  if (K) CK(cudaMemcpyAsync(K, sc.dK, n2 * 8, cudaMemcpyDeviceToHost, ctx->stream));
  return gbjk_synchronize(ctx);
}

gbjk_status gbjk_scf_end(gbjk_ctx* ctx) {
  if (!ctx) return GBJK_INVALID_ARG;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  ctx->scf.release();
  return GBJK_OK;
}

// --- SOS-AO-MP2 Laplace batch -----------------------------------------------

gbjk_status gbjk_mp2_set_factors(gbjk_ctx* ctx, int npts, const int* rank_o,
                                 const double* const* Lo, const int* rank_v,
                                 const double* const* Lv) {
  gbjk_status s;
  if ((s = check_ready(ctx))) return s;
  if (npts < 1 || !rank_o || !Lo || !rank_v || !Lv)
    return fail(ctx, GBJK_INVALID_ARG, "gbjk_mp2_set_factors: null argument or npts < 1");
  for (int t = 0; t < npts; ++t) {
    if (!Lo[t] || !Lv[t])
      return fail(ctx, GBJK_INVALID_ARG, "gbjk_mp2_set_factors: null factor");
    if (rank_o[t] < 1 || rank_o[t] > ctx->nbf || rank_v[t] < 1 || rank_v[t] > ctx->nbf)
      return fail(ctx, GBJK_INVALID_ARG, "gbjk_mp2_set_factors: rank out of range [1, nbf]");
  }
  Mp2State& m = ctx->mp2;
  if (ctx->precision == GBJK_FP64) {
    if ((s = m.prefit_fp64(ctx->stream, ctx->d_B, ctx->d_Linv, ctx->nnz, ctx->split,
                           &ctx->launches, &ctx->err)))
      return s;
  } else if (!ctx->split.b_ready &&
             (s = ctx->split.prepare_b(ctx->stream, ctx->d_B, ctx->d_Linv, &ctx->launches,
                                       &ctx->err))) {
    return s;
  }
  bool same = m.ready && m.precision == ctx->precision && m.npts == npts;
  for (int t = 0; same && t < npts; ++t) same = m.ro[t] == rank_o[t] && m.rv[t] == rank_v[t];
  if (!same && (s = m.plan(ctx->stream, ctx->precision, npts, rank_o, rank_v, ctx->nbf, ctx->naux,
                           ctx->nblk, ctx->ncols_total, ctx->bsize, ctx->boff, ctx->panelK,
                           ctx->cmoff, ctx->panel_off, ctx->d_B, ctx->split, &ctx->err)))
    return s;
  return m.upload(ctx->stream, ctx->nbf, Lo, Lv, &ctx->err);
}

gbjk_status gbjk_mp2_compute_dev(gbjk_ctx* ctx) {
  gbjk_status s;
  if ((s = check_ready(ctx))) return s;
  if (!ctx->mp2.ready || ctx->mp2.precision != ctx->precision)
    return fail(ctx, GBJK_NOT_READY, "gbjk_mp2_compute_dev: set the factors first (after any precision change)");
  if ((s = ctx->split.clear_error(ctx->stream))) return fail(ctx, s, "split path: memset failed");
  return ctx->mp2.run(ctx->stream, ctx->nbf, ctx->naux, ctx->nblk, ctx->ncols_total,
                      ctx->d_colmap, ctx->split, &ctx->launches, &ctx->err);
}

gbjk_status gbjk_mp2_read(gbjk_ctx* ctx, double* energies, double* Z) {
  if (!ctx) return GBJK_INVALID_ARG;
  if (!ctx->mp2.have_result) return fail(ctx, GBJK_NOT_READY, "gbjk_mp2_read: nothing computed");
  CK(cudaSetDevice(ctx->device));
  const int npts = ctx->mp2.npts;
  // the flag of a timed-out wait and the energies come in one round trip
  double* h_E = ctx->mp2.h_E;
  *ctx->h_err = 0;
  if (ctx->mp2.precision == GBJK_SPLIT_BF16 && ctx->split.d_err)
    CK(cudaMemcpyAsync(ctx->h_err, ctx->split.d_err, sizeof(int), cudaMemcpyDeviceToHost,
                       ctx->stream));
  if (h_E)
    CK(cudaMemcpyAsync(h_E, ctx->mp2.d_E, npts * sizeof(double), cudaMemcpyDeviceToHost,
                       ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  if (const int code = *ctx->h_err)
    return fail(ctx, GBJK_TIMEOUT,
                "split GEMM: a pipeline wait timed out (code " + std::to_string(code) + ")");
  if (energies && h_E)
    std::copy(h_E, h_E + npts, energies);
  else if (energies)
    CK(cudaMemcpy(energies, ctx->mp2.d_E, (size_t)npts * sizeof(double), cudaMemcpyDeviceToHost));
  if (Z)
    CK(cudaMemcpy(Z, ctx->mp2.d_Z, (size_t)npts * ctx->naux * ctx->naux * sizeof(double),
                  cudaMemcpyDeviceToHost));
  return GBJK_OK;
}

gbjk_status gbjk_mp2_laplace(gbjk_ctx* ctx, int npts, const int* rank_o, const double* const* Lo,
                             const int* rank_v, const double* const* Lv, double* energies,
                             double* Z) {
  gbjk_status s;
  if ((s = gbjk_mp2_set_factors(ctx, npts, rank_o, Lo, rank_v, Lv))) return s;
  if ((s = gbjk_mp2_compute_dev(ctx))) return s;
  return gbjk_mp2_read(ctx, energies, Z);
}

gbjk_status gbjk_mp2_release(gbjk_ctx* ctx) {
  if (!ctx) return GBJK_INVALID_ARG;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  ctx->mp2.release();
  return GBJK_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// DF-J without device allocation.
//
// Some callers cannot call cudaMalloc: code running inside a host framework
// that owns all device memory through its own pool, or code that must not
// allocate while a CUDA graph is being captured.  gbjk_compute_j_noalloc
// runs the same J kernels as the context path, with every scratch buffer
// (launch metadata, gathered density rows, per-row partial sums, g and h)
// carved out of one file-scope device array of kNoallocScratchBytes.  The
// module holds that array on every GPU that loads the library, until exit.
// ---------------------------------------------------------------------------
namespace {

constexpr size_t kNoallocScratchBytes = 16u << 20;  // 16 MiB
constexpr int kNoallocMaxDevices = 64;
// Atom blocks per call: the block sizes and panel widths travel inside the
// kernel arguments (8 KB), so a call copies nothing from host memory and
// issues only launches and memsets.
constexpr int kNoallocMaxBlocks = 1024;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocScratchBytes];

// Device address of g_noalloc_scratch per device, looked up once per device.
void* g_noalloc_ptr[kNoallocMaxDevices] = {};
std::mutex g_noalloc_mu;

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

struct NoallocLayout {
  int nblk;
  int bsize[kNoallocMaxBlocks];
  int panelK[kNoallocMaxBlocks];
};

// Prefix sums of the layout inside the scratch array (one block).
__global__ void k_noalloc_layout(int nbf, int naux, const NoallocLayout lay, int* bsize,
                                 int* panelK, int* boff, int* cmoff, long long* panel_off,
                                 long long* pg_off, int* blk_of) {
  const int nblk = lay.nblk;
  for (int I = threadIdx.x; I < nblk; I += blockDim.x) {
    bsize[I] = lay.bsize[I];
    panelK[I] = lay.panelK[I];
  }
  if (threadIdx.x == 0) {
    int b = 0, c = 0;
    long long po = 0, pg = 0;
    for (int I = 0; I < nblk; ++I) {
      boff[I] = b;
      cmoff[I] = c;
      panel_off[I] = po;
      pg_off[I] = pg;
      b += lay.bsize[I];
      c += lay.panelK[I];
      po += (long long)lay.bsize[I] * naux * lay.panelK[I];
      pg += (long long)lay.bsize[I] * lay.panelK[I];
    }
    boff[nblk] = b;
    cmoff[nblk] = c;
  }
  __syncthreads();
  for (int I = 0; I < nblk; ++I)
    for (int m = threadIdx.x; m < lay.bsize[I]; m += blockDim.x) blk_of[boff[I] + m] = I;
}

}  // namespace

extern "C" gbjk_status gbjk_compute_j_noalloc(const gbjk_desc* d, const int* d_colmap,
                                              const double* d_B, const double* d_Vinv,
                                              const double* d_Ptot, double* d_J, void* stream,
                                              char* errbuf, size_t errlen) {
  auto err = [&](gbjk_status s, const std::string& m) {
    if (errbuf && errlen) {
      std::snprintf(errbuf, errlen, "%s", m.c_str());
    }
    return s;
  };
  if (!d || !d->blk_size || !d->panel_K || !d_colmap || !d_B || !d_Vinv || !d_Ptot || !d_J)
    return err(GBJK_INVALID_ARG, "gbjk_compute_j_noalloc: null argument");
  const int nbf = d->nbf, naux = d->naux, nblk = d->nblk;
  if (nbf <= 0 || naux <= 0 || nblk <= 0)
    return err(GBJK_INVALID_ARG, "gbjk_compute_j_noalloc: sizes must be positive");
  if (nblk > kNoallocMaxBlocks)
    return err(GBJK_INVALID_ARG, "gbjk_compute_j_noalloc: more than " +
                                     std::to_string(kNoallocMaxBlocks) + " atom blocks");
  if (nbf > 65535)  // grid.y of the gather and column-sum launches
    return err(GBJK_INVALID_ARG, "gbjk_compute_j_noalloc: nbf > 65535 not supported");
  long long bsum = 0, pg_total = 0;
  int maxK = 0;
  for (int I = 0; I < nblk; ++I) {
    if (d->blk_size[I] <= 0 || d->panel_K[I] < 0 || d->panel_K[I] > nbf)
      return err(GBJK_INVALID_ARG, "gbjk_compute_j_noalloc: bad block size or panel width");
    bsum += d->blk_size[I];
    pg_total += (long long)d->blk_size[I] * d->panel_K[I];
    maxK = std::max(maxK, d->panel_K[I]);
  }
  if (bsum != nbf) return err(GBJK_INVALID_ARG, "gbjk_compute_j_noalloc: block sizes != nbf");
  if ((size_t)naux * sizeof(double) > 48 * 1024)
    return err(GBJK_INVALID_ARG, "gbjk_compute_j_noalloc: naux > 6144 not supported");
  // scratch layout
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off = align256(off + bytes);
    return o;
  };
  const size_t o_bsize = take(sizeof(int) * nblk), o_panelK = take(sizeof(int) * nblk);
  const size_t o_boff = take(sizeof(int) * (nblk + 1)), o_cmoff = take(sizeof(int) * (nblk + 1));
  const size_t o_poff = take(sizeof(long long) * nblk), o_pgoff = take(sizeof(long long) * nblk);
  const size_t o_blkof = take(sizeof(int) * nbf);
  const size_t o_pg = take(sizeof(double) * (size_t)pg_total);
  const size_t o_part = take(sizeof(double) * (size_t)nbf * naux);
  const size_t o_g = take(sizeof(double) * naux), o_h = take(sizeof(double) * naux);
  if (off > kNoallocScratchBytes)
    return err(GBJK_INVALID_ARG, "gbjk_compute_j_noalloc: problem needs " + std::to_string(off) +
                                     " scratch bytes, limit is " +
                                     std::to_string(kNoallocScratchBytes) +
                                     " (nbf*naux + sum b_I*K_I + 2*naux doubles + layout)");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoallocMaxDevices)
    return err(GBJK_CUDA_ERROR, "gbjk_compute_j_noalloc: no current device");
  unsigned char* base;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess || !p)
        return err(GBJK_CUDA_ERROR, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
      g_noalloc_ptr[dev] = p;
    }
    base = (unsigned char*)g_noalloc_ptr[dev];
  }
  cudaStream_t st = (cudaStream_t)stream;
  int* bsize = (int*)(base + o_bsize);
  int* panelK = (int*)(base + o_panelK);
  int* boff = (int*)(base + o_boff);
  int* cmoff = (int*)(base + o_cmoff);
  long long* poff = (long long*)(base + o_poff);
  long long* pgoff = (long long*)(base + o_pgoff);
  int* blk_of = (int*)(base + o_blkof);
  double* Pg = (double*)(base + o_pg);
  double* part = (double*)(base + o_part);
  double* g = (double*)(base + o_g);
  double* h = (double*)(base + o_h);
  auto ck = [&](cudaError_t e, const char* what) {
    return e == cudaSuccess ? GBJK_OK
                            : err(GBJK_CUDA_ERROR, std::string(what) + ": " + cudaGetErrorString(e));
  };
  gbjk_status s;
  NoallocLayout lay;
  lay.nblk = nblk;
  for (int I = 0; I < nblk; ++I) {
    lay.bsize[I] = d->blk_size[I];
    lay.panelK[I] = d->panel_K[I];
  }
  k_noalloc_layout<<<1, 256, 0, st>>>(nbf, naux, lay, bsize, panelK, boff, cmoff, poff, pgoff,
                                      blk_of);
  if ((s = ck(cudaGetLastError(), "layout kernel"))) return s;
  if ((s = ck(cudaMemsetAsync(d_J, 0, sizeof(double) * (size_t)nbf * nbf, st), "clear J")))
    return s;
  k_gather_panel_rows<<<dim3(cdiv(std::max(maxK, 1), 128), nbf), 128, 0, st>>>(
      d_Ptot, nbf, blk_of, boff, panelK, pgoff, cmoff, d_colmap, Pg);
  k_j_rowdot<<<cdiv((long long)nbf * naux * 32, 256), 256, 0, st>>>(d_B, poff, blk_of, boff,
                                                                     panelK, pgoff, Pg, nbf, naux,
                                                                     part);
  k_reduce_rows<<<cdiv(naux, 32), 32, 0, st>>>(part, nbf, naux, g);
  k_gemv<<<cdiv((long long)naux * 32, 256), 256, 0, st>>>(d_Vinv, g, naux, h);
  k_j_colsum<<<dim3(cdiv(std::max(maxK, 1), 32), nbf), 128, 0, st>>>(
      d_B, poff, blk_of, boff, panelK, cmoff, d_colmap, h, nbf, naux, d_J);
  if (d->filter_eps > 0)
    k_block_filter<<<cdiv((long long)nblk * nblk, 8), 256, 0, st>>>(d_J, nbf, boff, nblk,
                                                                    d->filter_eps);
  return ck(cudaGetLastError(), "J kernels");
}
