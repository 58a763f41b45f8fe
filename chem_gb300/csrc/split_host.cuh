// Host side of the split-precision K path: operand preparation and launch
// plans.
//
// Once per tensor upload:
//   Bfit = L^-1 B (prefit_gemm.cuh, to FP64 accuracy on the tensor cores), its
//   row exponents and slice images (the A operands of the half transform).
// Per nocc: buffers and the two work lists (half transform, exchange).
// Per build (stream-ordered, no host sync):
//   rows of C and P -> digits (B operand of every panel) -> split GEMM
//   Hfit = Bfit C (the product's integers, row exponents by atomicMax) -> H
//   digits -> split GEMM Kpart = Hfit Hfit^T (upper tiles, split-K) -> ordered
//   reduce K = -sum Kpart.
// With hfuse the half-transform epilogue cuts the digits of Hfit itself
// (one exponent per AO function and group of 32 auxiliary indices) and the
// exchange is the segmented variant that applies those exponents.
// The A operand rows (m, y) of panel I sit at m * pad32(batch) + y, so that
// every 32-row block is one AO function and one auxiliary group.
// With the fit folded into the tensor, DF-MO and DF-LMO compute the same
// K = -(L^-1 B C)^T (L^-1 B C).
#pragma once
#include <algorithm>
#include <string>
#include <utility>
#include <vector>

#include "kernels_fp64.cuh"
#include "prefit_gemm.cuh"
#include "split_gemm.cuh"

namespace gbjk {

struct SplitState {
  size_t bytes = 0;
  uint64_t frees = 0;  // buffers freed so far (a captured build using them is stale)
  int nbf = 0, naux = 0, nblk = 0;
  std::vector<int> bsize, boff, panelK, cmoff;
  std::vector<long long> panel_off;
  bool b_ready = false;
  int nocc = -1;
  // A operands and the prefitted tensor L^-1 B (FP64).  With `fitted` the
  // uploaded tensor already is L^-1 B and Bfit aliases it.
  bool fitted = false;
  bool bfit_owned = false;
  double* Bfit = nullptr;
  // compact copy of Bfit for the mixed-path J (k_encode_f32i16: FP32 hi and
  // a 16-bit remainder per element, 6 bytes), unbatched only; of a symmetric
  // tensor the upper block triangle alone (prepare_j)
  float* d_Bhi = nullptr;
  uint16_t* d_Blo = nullptr;
  JPanel* d_jp = nullptr;
  int2 *d_jblk = nullptr, *d_jmap = nullptr;
  double* d_jpart = nullptr;
  int n_jblk = 0, jchunk = 0, jnchunk = 0;
  long long jcols = 0;
  std::vector<int> colmap, blk_of;
  // the context's device copies of the panel layout (not owned)
  const long long* dd_panel_off = nullptr;
  const int *dd_blk_of = nullptr, *dd_boff = nullptr, *dd_panelK = nullptr, *dd_colmap = nullptr;
  uint16_t* d_Aslices = nullptr;
  // auxiliary batching: xb auxiliary rows per batch (nbatch > 1 streams the
  // half transform and the exchange batch by batch; A digits per batch)
  int xb_req = 0, xb = 0, nbatch = 1;
  // A-row pitch of the full batch: pad32(xb) (pad32(naux) unbatched)
  int apitch = 0;
  // fused digit cut of H in the half transform (requested; in effect for
  // the per-nocc buffers).  Off by default: on GB300 the fused half
  // transform and segmented exchange together take longer than the H round
  // trip and digit pass they replace.
  bool hfuse = false, hfuse_eff = false;  // asked for; what the current plan does
  // what the builds do, as far as a plan has decided it
  bool fuses() const { return hfuse && (nocc < 0 || hfuse_eff); }
  SplitJob* d_bjobs = nullptr;  // A-digit jobs, nbatch * nbf (one per (batch, mu))
  std::vector<long long> a_off, eA_off;
  std::vector<int> a_nrb, nkt;
  int* d_eA = nullptr;
  // per build
  uint16_t* d_Cslices = nullptr;
  std::vector<long long> c_off;
  int c_nrb = 0;
  int* d_eC = nullptr;
  long long* d_H = nullptr;  // integers of the half transform (SplitItem::iout)
  uint16_t* d_Hslices = nullptr;
  int h_nrb = 0, h_nkt = 0, hld = 0;
  int* d_eH = nullptr;
  int* d_eHs = nullptr;  // fused: exponents [mu][auxiliary group], es_ld per row
  int es_ld = 0;
  double* d_Kpart = nullptr;
  double* d_dpart = nullptr;  // J partials [mu][Y] from the density columns
  double* d_dt = nullptr;     // L^-1 g
  int ksplit = 1;
  int maxb = 0;
  SplitItem* d_items = nullptr;
  int ht_nitems = 0, k_nitems = 0;
  PrepJob* d_jobs = nullptr;  // [0,nblk): C rows, [nblk,2nblk): P rows
  std::vector<SplitIntJob> hjobs;  // digits of H, one per distinct batch size
  long long* d_eoff = nullptr;     // their exponent offsets per AO function
  int c_groups = 0;  // most 8-row groups of a job
  int* d_err = nullptr;
  int nsm = 148;
  bool profile = false;
  // set by the caller for one build: event recorded right after the half
  // transform (the fork point of the J column sums), and the number of SMs
  // the exchange GEMM leaves free (0: all SMs)
  cudaEvent_t ev_ht = nullptr;
  int k_grid = 0;
  // requested exchange k parts (0 = choose_ksplit) and the number in effect
  int ks_req = 0, ks_eff = 0;
  // test hook (gbjk_test_split_stall): the producer stops at this work item
  // of every split GEMM launch (-1: never), and the waits' time limit
  int stop_item = -1;
  size_t prefit_room = ~size_t(0);  // most bytes of temporary digits in the prefit
  unsigned long long spin_ns = kSpinNs;
  double ms[4] = {0, 0, 0, 0};
  int64_t nl[4] = {0, 0, 0, 0};
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> pending;

  void set_dev_layout(const long long* po, const int* blk_of, const int* bo, const int* pk,
                      const int* cm) {
    dd_colmap = cm;
    dd_panel_off = po;
    dd_blk_of = blk_of;
    dd_boff = bo;
    dd_panelK = pk;
  }
  void init(int nbf_, int naux_, int nblk_, const std::vector<int>& bs,
            const std::vector<int>& bo, const std::vector<int>& pk, const std::vector<int>& cmo,
            const std::vector<long long>& po, const std::vector<int>& cm,
            const std::vector<int>& blko) {
    nbf = nbf_;
    naux = naux_;
    nblk = nblk_;
    bsize = bs;
    boff = bo;
    panelK = pk;
    cmoff = cmo;
    panel_off = po;
    colmap = cm;
    blk_of = blko;
  }
  template <class T>
  cudaError_t alloc(T** p, size_t n) {
    const size_t b = std::max<size_t>(n, 1) * sizeof(T);
    cudaError_t e = cudaMalloc((void**)p, b);
    if (e == cudaSuccess)
      bytes += b;
    else
      cudaGetLastError();
    return e;
  }
  template <class T>
  void free_(T** p) {
    if (*p) {
      cudaFree(*p);
      frees++;
    }
    *p = nullptr;
  }
  void release_build() {
    free_(&d_Cslices);
    free_(&d_eC);
    free_(&d_H);
    free_(&d_Hslices);
    free_(&d_eH);
    free_(&d_eHs);
    free_(&d_Kpart);
    free_(&d_dpart);
    free_(&d_dt);
    free_(&d_items);
    free_(&d_jobs);
    free_(&d_eoff);
    plans.clear();
    nocc = -1;
  }
  void release() {
    release_build();
    if (bfit_owned) free_(&Bfit);
    Bfit = nullptr;
    bfit_owned = false;
    free_(&d_Bhi);
    free_(&d_Blo);
    free_(&d_jp);
    free_(&d_jblk);
    free_(&d_jmap);
    free_(&d_jpart);
    free_(&d_Aslices);
    free_(&d_bjobs);
    free_(&d_eA);
    free_(&d_err);
    for (auto& pe : pending) {
      cudaEventDestroy(pe.second.first);
      cudaEventDestroy(pe.second.second);
    }
    pending.clear();
    b_ready = false;
    bytes = 0;
  }
  void invalidate_b() { release(); }
  void reset_profile() {
    resolve();
    for (int i = 0; i < 4; ++i) {
      ms[i] = 0;
      nl[i] = 0;
    }
  }
  void resolve() {
    for (auto& pe : pending) {
      float t = 0.f;
      if (cudaEventElapsedTime(&t, pe.second.first, pe.second.second) == cudaSuccess)
        ms[pe.first] += t;
      cudaEventDestroy(pe.second.first);
      cudaEventDestroy(pe.second.second);
    }
    pending.clear();
  }
  int profile_read(int idx, const char** name, double* out_ms, int64_t* launches) {
    static const char* names[4] = {"split_gemm_ht", "split_gemm_k", "split_digits", "prefit"};
    if (idx < 0 || idx >= 4) return 0;
    resolve();
    if (name) *name = names[idx];
    if (out_ms) *out_ms = ms[idx];
    if (launches) *launches = nl[idx];
    return 1;
  }
  struct Scope {
    SplitState* s;
    int ph;
    cudaStream_t st;
    cudaEvent_t a = nullptr, b = nullptr;
    Scope(SplitState* s_, int p, cudaStream_t st_) : s(s_), ph(p), st(st_) {
      if (s->profile) {
        cudaEventCreate(&a);
        cudaEventCreate(&b);
        cudaEventRecord(a, st);
      }
      s->nl[ph]++;
    }
    ~Scope() {
      if (s->profile) {
        cudaEventRecord(b, st);
        s->pending.push_back({ph, {a, b}});
      }
    }
  };

  static int cdiv_(long long a, long long b) { return (int)((a + b - 1) / b); }
  // most 8-row groups of a job: the grid of k_prep_rows
  static int prep_groups(const std::vector<PrepJob>& jobs) {
    int g = 1;
    for (const PrepJob& j : jobs)
      if (j.nrows) g = std::max(g, (j.row0 + j.nrows + 7) / 8 - j.row0 / 8);
    return g;
  }
  // digits of operands left as integers by a split GEMM
  template <bool kFull>
  static void launch_ints(cudaStream_t st, const SplitIntJob* jobs, int n, int64_t* launches) {
    for (int j0 = 0; j0 < n; j0 += kMaxIntJobs) {
      const int m = std::min(kMaxIntJobs, n - j0);
      SplitIntJobs p;
      long long warps = 0;
      for (int j = 0; j < m; ++j) {
        p.j[j] = jobs[j0 + j];
        warps = std::max(warps, (long long)cdiv_(p.j[j].nrows, 8) * p.j[j].nkt);
      }
      k_split_ints<kFull><<<dim3(cdiv_(warps, 8), m), 256, 0, st>>>(p);
      (*launches)++;
    }
  }
  // H rows hold the half transform in groups of 32 auxiliary indices (the
  // column-pair-outermost layout of SplitItem::perm_rs), so a batch of xbc
  // auxiliary rows spans pad32(xbc) * hld columns of H
  static int pad32(int x) { return (x + 31) & ~31; }

  bool attr_v[8] = {};
  template <bool kH, bool kS, int kOut>
  gbjk_status launch_gemm_v(cudaStream_t st, SplitItem* items, int n, int64_t* launches,
                            std::string* err, int leave_sms) {
    if (n == 0) return GBJK_OK;
    const int v = kH ? 5 : (kS ? 6 : kOut);
    if (!attr_v[v]) {
      if (cudaFuncSetAttribute(k_split_gemm<kH, kS, kOut>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess) {
        *err = "cannot reserve shared memory for the split GEMM";
        return GBJK_CUDA_ERROR;
      }
      int dev = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
      attr_v[v] = true;
    }
    const int grid = std::min(n, std::max(1, nsm - leave_sms));
    k_split_gemm<kH, kS, kOut>
        <<<grid, kThreads, kSmemBytes, st>>>(items, n, d_err, stop_item, spin_ns);
    (*launches)++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      *err = std::string("split GEMM launch: ") + cudaGetErrorString(e);
      return GBJK_CUDA_ERROR;
    }
    return GBJK_OK;
  }
  template <int kOut = kOutF64>
  gbjk_status launch_gemm(cudaStream_t st, SplitItem* items, int n, int64_t* launches,
                          std::string* err, int leave_sms = 0) {
    return launch_gemm_v<false, false, kOut>(st, items, n, launches, err, leave_sms);
  }

  // --- once per tensor: Bfit = L^-1 B ----------------------------------------
  // On the FP64 pipe, each element the in-order fma chain of the oracle's
  // prefit (the FP64 MP2 batch needs that order).
  gbjk_status prefit_fp64(cudaStream_t st, const double* d_B, const double* d_Linv, double* d_Bfit,
                          int64_t* launches, std::string* err) {
    std::vector<GemmGroup> groups;
    std::vector<GemmTile> tiles;
    for (int I = 0; I < nblk; ++I) {
      const int K = panelK[I];
      if (K == 0) continue;
      for (int m = 0; m < bsize[I]; ++m) {
        GemmGroup g;
        const long long off = panel_off[I] + (long long)m * naux * K;
        g.A = d_Linv;
        g.B = d_B + off;
        g.C = d_Bfit + off;
        g.M = naux;
        g.N = K;
        g.K = naux;
        g.lda = naux;
        g.ldb = K;
        g.ldc = K;
        g.flags = kLowerA;
        for (int mt = 0; mt < cdiv_(naux, 64); ++mt)
          for (int nt = 0; nt < cdiv_(K, 64); ++nt)
            tiles.push_back({(int)groups.size(), mt, nt, 0, naux, 0});
        groups.push_back(g);
      }
    }
    GemmGroup* dg = nullptr;
    GemmTile* dt = nullptr;
    if (cudaMalloc((void**)&dg, std::max<size_t>(1, groups.size()) * sizeof(GemmGroup)) !=
            cudaSuccess ||
        cudaMalloc((void**)&dt, std::max<size_t>(1, tiles.size()) * sizeof(GemmTile)) !=
            cudaSuccess) {
      cudaGetLastError();
      cudaFree(dg);
      *err = "out of memory for the prefit plan";
      return GBJK_OOM;
    }
    cudaMemcpy(dg, groups.data(), groups.size() * sizeof(GemmGroup), cudaMemcpyHostToDevice);
    cudaMemcpy(dt, tiles.data(), tiles.size() * sizeof(GemmTile), cudaMemcpyHostToDevice);
    {
      Scope sc(this, 3, st);
      // the grid limit is 2^31-1 blocks; launch in slices of 1M tiles
      for (size_t t0 = 0; t0 < tiles.size(); t0 += (1u << 20)) {
        const int n = (int)std::min<size_t>(1u << 20, tiles.size() - t0);
        k_gemm_fp64<false><<<n, 256, 0, st>>>(dg, dt + t0, 1.0);
        (*launches)++;
      }
    }
    const cudaError_t e = cudaStreamSynchronize(st);
    cudaFree(dg);
    cudaFree(dt);
    if (e != cudaSuccess) {
      *err = std::string("prefit: ") + cudaGetErrorString(e);
      return GBJK_CUDA_ERROR;
    }
    return GBJK_OK;
  }

  // On the tensor cores (prefit_gemm.cuh).  ws: device memory that may be
  // overwritten, for the digits of as many tensor columns as it holds (at
  // most 1 GB of them at a time); a temporary buffer where it holds too few to
  // occupy the SMs.  The digits of L^-1 (16 naux^2 bytes) have a buffer of their
  // own, of fewer 48-row tiles at a time where there is no room for all; one
  // tile of each, in ws, is the least.  The parts change no result: every output
  // is one exact sum.
  gbjk_status prefit(cudaStream_t st, const double* d_B, const double* d_Linv, double* d_Bfit,
                     void* ws, size_t ws_bytes, int64_t* launches, std::string* err) {
    std::vector<PfTile> tiles;
    for (int I = 0; I < nblk; ++I) {
      const int ncol = bsize[I] * panelK[I];
      for (int c0 = 0; c0 < ncol; c0 += kPfM)
        tiles.push_back({d_B + panel_off[I], d_Bfit + panel_off[I], panelK[I], c0, ncol});
    }
    if (tiles.empty()) return GBJK_OK;
    const int nkt_all = cdiv_(naux, kPfK), nxt = cdiv_(naux, kPfN);
    const size_t abytes = (size_t)nkt_all * kPfBytesA, bbytes = (size_t)nkt_all * kPfBytesB;
    const size_t most = std::min(tiles.size(), std::max<size_t>(1, (size_t(1) << 30) / abytes));
    const size_t ny = (size_t)nkt_all * kPfK;
    // balance of Y, exponents of the X rows and of the tensor columns; the tiles
    const size_t nint = (ny + (size_t)nxt * kPfN + most * kPfM + 63) & ~size_t(63);
    int* de = nullptr;
    void *own = nullptr, *db = nullptr;
    auto done = [&]() {
      cudaFree(own);
      cudaFree(db);
      cudaFree(de);
    };
    size_t room = prefit_room;
    // a buffer of n units, n the first of want, want / 2, .. that there is memory
    // for, and more than `least`; 0 if none
    auto grab = [&](void** p, size_t unit, size_t want, size_t least) {
      for (size_t n = want; n > least; n /= 2) {
        if (unit * n > room) continue;
        if (cudaMalloc(p, unit * n) == cudaSuccess) {
          room -= unit * n;
          return n;
        }
        cudaGetLastError();
      }
      *p = nullptr;
      return size_t(0);
    };
    const bool ok = cudaMalloc((void**)&de, nint * sizeof(int) + tiles.size() * sizeof(PfTile)) ==
                    cudaSuccess;
    size_t nx = 0, per = 0;  // X tiles and tensor tiles at a time
    if (ok) {
      nx = grab(&db, bbytes, nxt, 0);
      uint8_t* w = (uint8_t*)ws;
      uint16_t* bd = (uint16_t*)db;
      if (nx == 0 && ws_bytes >= bbytes) {
        nx = 1;
        bd = (uint16_t*)w;
        w += bbytes;
        ws_bytes -= bbytes;
      }
      per = std::min(most, ws_bytes / abytes);
      if (per < most && per * nx < 1024)
        if (const size_t n = grab(&own, abytes, most, per)) {
          per = n;
          w = (uint8_t*)own;
        }
      if (nx && per)
        return prefit_parts(st, d_Linv, tiles, (PfTile*)(de + nint), de, bd, (int)nx,
                            (uint16_t*)w, per, launches, err, done);
    }
    cudaGetLastError();
    done();
    *err = "split path: out of memory for the prefit's operand digits";
    return GBJK_OOM;
  }
  // ... with digit buffers bd and ad for nx tiles of L^-1 and `per` tiles of the
  // tensor; done() frees what prefit() allocated
  template <class Done>
  gbjk_status prefit_parts(cudaStream_t st, const double* d_Linv,
                           const std::vector<PfTile>& tiles, PfTile* dt, int* de, uint16_t* bd,
                           int nx, uint16_t* ad, size_t per, int64_t* launches, std::string* err,
                           Done done) {
    const int nkt_all = cdiv_(naux, kPfK), nxt = cdiv_(naux, kPfN);
    const size_t bbytes = (size_t)nkt_all * kPfBytesB, ny = (size_t)nkt_all * kPfK;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    int *bal = de, *eb = de + ny, *ea = eb + (size_t)nxt * kPfN;
    cudaError_t e = cudaFuncSetAttribute(
        k_prefit_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, kPfSmem);
    if (!e)
      e = cudaMemcpyAsync(dt, tiles.data(), tiles.size() * sizeof(PfTile), cudaMemcpyHostToDevice,
                          st);
    if (!e) {
      Scope sc(this, 3, st);
      k_pf_balance<<<nkt_all, dim3(32, 32), 0, st>>>(d_Linv, naux, bal);
      (*launches)++;
      for (int x0 = 0; x0 < nxt && !e; x0 += nx) {
        const int m = std::min(nx, nxt - x0), row0 = x0 * kPfN;
        e = cudaMemsetAsync(bd, 0, (size_t)m * bbytes, st);
        k_pf_metric<<<cdiv_(std::min(naux - row0, m * kPfN), 8), 256, 0, st>>>(
            d_Linv, bal, naux, row0, nkt_all, eb, bd);
        (*launches)++;
        for (size_t t0 = 0; t0 < tiles.size(); t0 += per) {
          const int n = (int)std::min(per, tiles.size() - t0);
          k_pf_colexp<<<n, dim3(128, 4), 0, st>>>(dt + t0, bal, naux, ea);
          k_pf_coldigits<<<dim3(n, 2 * nkt_all), 256, 0, st>>>(dt + t0, ea, bal, naux, nkt_all, ad);
          k_prefit_gemm<<<std::min(n * m, nsm), kThreads, kPfSmem, st>>>(
              dt + t0, n * m, m, x0, naux, nkt_all, ad, ea, bd, eb, d_err, kSpinNs);
          *launches += 3;
        }
      }
      if (!e) e = cudaGetLastError();
    }
    // on an error too: nothing in flight uses the buffers any more
    const cudaError_t es = cudaStreamSynchronize(st);
    done();
    if (e || es) {
      *err = std::string("prefit: ") + cudaGetErrorString(e ? e : es);
      return GBJK_CUDA_ERROR;
    }
    if (const int code = read_error()) {
      *err = "prefit: a pipeline wait timed out (code " + std::to_string(code) + ")";
      return GBJK_TIMEOUT;
    }
    return GBJK_OK;
  }

  // --- once per tensor: the compact copy the mixed-path J reads ------------
  // Block pairs (I, J), I < J, whose columns lie side by side in both panels,
  // and k0[I], the first column of a block J >= I.  False if a panel's columns
  // are not whole blocks in ascending order or a pair is kept on one side only.
  bool symmetric_pattern(std::vector<SymPair>* pairs, std::vector<int>* k0) const {
    std::vector<std::vector<std::pair<int, int>>> cols(nblk);  // (J, first column)
    for (int I = 0; I < nblk; ++I) {
      (*k0)[I] = panelK[I];
      const int* cm = colmap.data() + cmoff[I];
      for (int k = 0; k < panelK[I];) {
        const int J = blk_of[cm[k]];
        if (cm[k] != boff[J] || k + bsize[J] > panelK[I]) return false;
        for (int n = 1; n < bsize[J]; ++n)
          if (cm[k + n] != boff[J] + n) return false;
        if (!cols[I].empty() && cols[I].back().first >= J) return false;
        if (J >= I) (*k0)[I] = std::min((*k0)[I], k);
        cols[I].push_back({J, k});
        k += bsize[J];
      }
    }
    size_t lower = 0;
    for (int I = 0; I < nblk; ++I)
      for (const auto& c : cols[I]) {
        const int J = c.first;
        if (J < I) lower++;
        if (J <= I) continue;
        auto it = std::lower_bound(cols[J].begin(), cols[J].end(), std::make_pair(I, -1));
        if (it == cols[J].end() || it->first != I) return false;
        pairs->push_back({panel_off[I], panel_off[J], panelK[I], panelK[J], c.second, it->second,
                          bsize[I], bsize[J]});
      }
    return lower == pairs->size();
  }

  gbjk_status prepare_j(cudaStream_t st, int64_t* launches, std::string* err) {
    auto oom = [&]() {
      *err = "split path: out of memory for the compact J tensor";
      return GBJK_OOM;
    };
    // J is symmetric where the tensor is: a tensor that holds the same bits
    // in both copies of every off-diagonal block pair (as the integral engines
    // write it) is read in its upper block triangle only, and J mirrored
    std::vector<SymPair> pairs;
    std::vector<int> k0(nblk, 0);
    bool sym = symmetric_pattern(&pairs, &k0);
    if (sym && !pairs.empty()) {
      SymPair* dp = nullptr;
      int* df = nullptr;
      int h = 0;
      if (alloc(&dp, pairs.size()) != cudaSuccess || alloc(&df, 1) != cudaSuccess) {
        free_(&dp);
        return oom();
      }
      cudaMemcpy(dp, pairs.data(), pairs.size() * sizeof(SymPair), cudaMemcpyHostToDevice);
      cudaMemsetAsync(df, 0, sizeof(int), st);
      {
        Scope sc(this, 3, st);
        k_check_symmetric<<<dim3((unsigned)pairs.size(), cdiv_(naux, 64)), 128, 0, st>>>(
            Bfit, dp, naux, df);
        (*launches)++;
      }
      cudaMemcpyAsync(&h, df, sizeof(int), cudaMemcpyDeviceToHost, st);
      const cudaError_t e = cudaStreamSynchronize(st);
      bytes -= pairs.size() * sizeof(SymPair) + sizeof(int);
      free_(&dp);
      free_(&df);
      if (e != cudaSuccess) {
        *err = std::string("split path preparation: ") + cudaGetErrorString(e);
        return GBJK_CUDA_ERROR;
      }
      sym = h == 0;
    }
    if (!sym) std::fill(k0.begin(), k0.end(), 0);
    std::vector<JPanel> jp(nblk);
    std::vector<int2> blk, map;
    long long ncomp = 0;
    for (int I = 0; I < nblk; ++I) {
      const int ks = panelK[I] - k0[I], ncol = bsize[I] * ks, cp = (ncol + 7) & ~7;
      jp[I] = {ncomp, (long long)map.size(), cp, ncol, k0[I]};
      for (int c0 = 0; c0 < ncol; c0 += 128) blk.push_back(make_int2(I, c0));
      for (int c = 0; c < cp; ++c) {
        if (c >= ncol) {
          map.push_back(make_int2(-1, 0));
          continue;
        }
        const int m = c / ks, nu = colmap[cmoff[I] + k0[I] + c % ks];
        map.push_back(make_int2(boff[I] + m, sym && blk_of[nu] != I ? ~nu : nu));
      }
      ncomp += (long long)naux * cp;
    }
    jcols = (long long)map.size();
    n_jblk = (int)blk.size();
    // rows per block: 128, or fewer while the blocks would not fill the SMs
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    jchunk = 128;
    while (jchunk > 32 && (long long)n_jblk * cdiv_(naux, jchunk) < 16LL * nsm) jchunk /= 2;
    jnchunk = cdiv_(naux, jchunk);
    if (alloc(&d_Bhi, (size_t)ncomp) != cudaSuccess || alloc(&d_Blo, (size_t)ncomp) != cudaSuccess ||
        alloc(&d_jp, jp.size()) != cudaSuccess || alloc(&d_jblk, blk.size()) != cudaSuccess ||
        alloc(&d_jmap, map.size()) != cudaSuccess ||
        alloc(&d_jpart, (size_t)jnchunk * jcols) != cudaSuccess ||
        cudaMemcpy(d_jp, jp.data(), jp.size() * sizeof(JPanel), cudaMemcpyHostToDevice) ||
        cudaMemcpy(d_jblk, blk.data(), blk.size() * sizeof(int2), cudaMemcpyHostToDevice) ||
        cudaMemcpy(d_jmap, map.data(), map.size() * sizeof(int2), cudaMemcpyHostToDevice))
      return oom();
    Scope sc(this, 3, st);
    k_encode_f32i16<<<dim3(naux, nblk), 128, 0, st>>>(Bfit, dd_panel_off, d_jp, dd_panelK, naux,
                                                      d_Bhi, d_Blo);
    (*launches)++;
    return GBJK_OK;
  }

  // J = (L^-1 B)^T d from the compact copy into dJ (screened blocks untouched)
  void run_j_cols(cudaStream_t st, const double* d, double* dJ, int64_t* launches) {
    if (n_jblk == 0) return;
    k_j_colsum_f32i16<<<dim3(n_jblk, jnchunk), 32, jchunk * sizeof(float2), st>>>(
        d_Bhi, d_Blo, d_jp, d_jblk, d, naux, jchunk, jcols, d_jpart);
    k_j_colsum_chunks<<<cdiv_(jcols, 128), 128, 0, st>>>(d_jpart, jnchunk, jcols, nbf, d_jmap, dJ);
    *launches += 2;
  }
  size_t j_bytes() const { return (size_t)naux * jcols * 6; }

  // --- once per tensor: prefit and A-operand digits -----------------------
  gbjk_status prepare_b(cudaStream_t st, const double* d_B, const double* d_Linv,
                        int64_t* launches, std::string* err) {
    const gbjk_status s = prepare_tensor(st, d_B, d_Linv, launches, err);
    if (s) release();  // nothing half prepared stays behind
    return s;
  }
  gbjk_status prepare_tensor(cudaStream_t st, const double* d_B, const double* d_Linv,
                             int64_t* launches, std::string* err) {
    const long long nnz = panel_off.back() + (long long)bsize.back() * naux * panelK.back();
    if (alloc(&d_err, 1) != cudaSuccess || cudaMemsetAsync(d_err, 0, sizeof(int), st) != cudaSuccess) {
      *err = "split path: cannot allocate the error flag";
      return GBJK_OOM;
    }
    // batches of a multiple of 32 auxiliary rows, so that only the last
    // (shorter) batch has unused slots in its last 32-index group of H
    xb = (xb_req > 0 && xb_req < naux) ? std::max(32, xb_req & ~31) : naux;
    if (xb > naux) xb = naux;
    nbatch = (naux + xb - 1) / xb;
    apitch = pad32(xb);
    // A operands: rows (m, y) of panel I, y < xb (all auxiliary rows when
    // not batched), at m * pad32(batch) + y; columns k
    a_off.assign(nblk, 0);
    eA_off.assign(nblk, 0);
    a_nrb.assign(nblk, 0);
    nkt.assign(nblk, 0);
    long long atot = 0, etot = 0;
    for (int I = 0; I < nblk; ++I) {
      const long long rows = (long long)bsize[I] * apitch;
      a_nrb[I] = cdiv_(rows, kTileM) * (kTileM / 32);
      nkt[I] = std::max(1, cdiv_(panelK[I], kTileK));
      a_off[I] = atot;
      eA_off[I] = etot;
      atot += (long long)a_nrb[I] * nkt[I] * kSlices * kImage;
      etot += (long long)a_nrb[I] * 32;
    }
    double* d_Bfit = nullptr;
    if (fitted) {
      d_Bfit = const_cast<double*>(d_B);
      bfit_owned = false;
    } else if (alloc(&d_Bfit, (size_t)nnz) != cudaSuccess) {
      *err = "split path: out of memory for the prefitted tensor";
      return GBJK_OOM;
    } else {
      bfit_owned = true;
    }
    Bfit = d_Bfit;
    if (alloc(&d_Aslices, (size_t)atot) != cudaSuccess ||
        alloc(&d_eA, (size_t)etot) != cudaSuccess) {
      *err = "split path: out of memory for the operand digits";
      return GBJK_OOM;
    }
    if (!fitted) {
      // the buffer of the operand digits holds the prefit's until it is needed
      gbjk_status ps = prefit(st, d_B, d_Linv, d_Bfit, d_Aslices, (size_t)atot * 2, launches, err);
      if (ps) return ps;
    }
    if (cudaMemsetAsync(d_Aslices, 0, (size_t)atot * 2, st) != cudaSuccess ||
        cudaMemsetAsync(d_eA, 0, (size_t)etot * 4, st) != cudaSuccess) {
      *err = "split path: memset failed";
      return GBJK_CUDA_ERROR;
    }
    if (nbatch == 1) {
      gbjk_status js = prepare_j(st, launches, err);
      if (js) return js;
    }
    if (nbatch == 1) {
      // one job per AO function: its naux rows (m, y) at m * apitch + y
      std::vector<SplitJob> jobs(nbf);
      for (int I = 0; I < nblk; ++I)
        for (int m = 0; m < bsize[I]; ++m) {
          SplitJob& j = jobs[boff[I] + m];
          j.src = d_Bfit + panel_off[I] + (long long)m * naux * panelK[I];
          j.rs = panelK[I];
          j.cs = 1;
          j.row0 = m * apitch;
          j.nrows = naux;
          j.ncols = panelK[I];
          j.e = d_eA + eA_off[I];
          j.nrb = a_nrb[I];
          j.nkt = nkt[I];
          j.dst = d_Aslices + a_off[I];
        }
      SplitJob* dj = nullptr;
      if (alloc(&dj, jobs.size()) != cudaSuccess) {
        *err = "split path: out of memory";
        return GBJK_OOM;
      }
      cudaMemcpy(dj, jobs.data(), jobs.size() * sizeof(SplitJob), cudaMemcpyHostToDevice);
      {
        Scope sc(this, 2, st);
        k_split_rows<<<dim3(cdiv_(naux / 8 + 2, 8), nbf), 256, 0, st>>>(dj);
        (*launches)++;
      }
      cudaStreamSynchronize(st);
      cudaFree(dj);
    } else {
      // one job per (batch, AO function): rows (m, y) of its panel
      std::vector<SplitJob> jobs((size_t)nbatch * nbf);
      for (int b = 0; b < nbatch; ++b) {
        const int Y0 = b * xb, xbc = std::min(xb, naux - Y0);
        for (int I = 0; I < nblk; ++I)
          for (int m = 0; m < bsize[I]; ++m) {
            SplitJob& j = jobs[(size_t)b * nbf + boff[I] + m];
            j.src = d_Bfit + panel_off[I] + ((long long)m * naux + Y0) * panelK[I];
            j.rs = panelK[I];
            j.cs = 1;
            j.row0 = m * pad32(xbc);
            j.nrows = xbc;
            j.ncols = panelK[I];
            j.e = d_eA + eA_off[I];
            j.nrb = a_nrb[I];
            j.nkt = nkt[I];
            j.dst = d_Aslices + a_off[I];
          }
      }
      if (alloc(&d_bjobs, jobs.size()) != cudaSuccess) {
        *err = "split path: out of memory for the batch jobs";
        return GBJK_OOM;
      }
      cudaMemcpy(d_bjobs, jobs.data(), jobs.size() * sizeof(SplitJob), cudaMemcpyHostToDevice);
    }
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
      *err = std::string("split path preparation: ") + cudaGetErrorString(e);
      return GBJK_CUDA_ERROR;
    }
    b_ready = true;
    return GBJK_OK;
  }

  // --- per nocc: buffers and work lists ------------------------------------
  // One plan per distinct auxiliary batch size (the last batch may be
  // shorter): item ranges of the half transform and of the exchange.
  struct BatchPlan {
    int xbc, ht0, nht, k0, nk, ksplit, hjob;
  };
  std::vector<BatchPlan> plans;

  // parts of the exchange's k range: requested, or by the wave model below;
  // never fewer than an item's int64 headroom allows (<= 8192 k per item)
  int exchange_ksplit(int nkt_total, int ntile) const {
    if (ks_req > 0) return std::max(cdiv_(nkt_total, 256), std::min(ks_req, nkt_total));
    return choose_ksplit(nkt_total, ntile);
  }
  int choose_ksplit(int nkt_total, int ntile) const {
    const int ks_min = cdiv_(nkt_total, 256);  // int64 headroom: <= 8192 k per item
    double best = 1e300;
    int pick = ks_min;
    for (int ks = ks_min; ks <= std::max(ks_min, 4 * nsm); ++ks) {
      const int per = cdiv_(nkt_total, ks);
      if (per < 8 && ks > ks_min) break;
      const long long waves = ((long long)ntile * ks + nsm - 1) / nsm;
      const double t = (double)waves * (per + 2.0);  // +2: per-item overhead in k-tiles
      if (t < best) {
        best = t;
        pick = ks;
      }
    }
    return pick;
  }

  gbjk_status prepare_nocc(cudaStream_t st, int nocc_, std::string* err) {
    release_build();
    const bool jfused = nbatch == 1;  // density rows ride along only unbatched
    maxb = 0;
    for (int I = 0; I < nblk; ++I) maxb = std::max(maxb, bsize[I]);
    // B operand rows of panel I: nocc orbitals, then b_I density rows
    const int ntn = cdiv_(nocc_ + (jfused ? maxb : 0), kTileN);
    c_nrb = ntn * (kTileN / 32);
    c_off.assign(nblk, 0);
    long long ctot = 0;
    for (int I = 0; I < nblk; ++I) {
      c_off[I] = ctot;
      ctot += (long long)c_nrb * nkt[I] * kSlices * kImage;
    }
    hld = nocc_ + (nocc_ & 1);  // even row stride: 16-byte aligned pairs
    // one exponent per (AO function, auxiliary group) needs all of a row's
    // columns in one tile: with more, the tiles' exponents would overwrite each
    // other
    hfuse_eff = hfuse && ntn == 1;
    const bool fuse = hfuse_eff;
    es_ld = apitch / 32;  // auxiliary groups of a full batch
    const long long hk = (long long)pad32(xb) * hld;
    // exchange k-tiles of a batch: fused, one per (auxiliary group, orbital);
    // unfused, the H row of pad32(xbc) * hld values in 32-value tiles
    auto xk_nkt = [&](int xbc) {
      return fuse ? (pad32(xbc) / 32) * nocc_ : cdiv_((long long)pad32(xbc) * hld, kTileK);
    };
    h_nkt = xk_nkt(xb);
    h_nrb = std::max(cdiv_(nbf, kTileM) * (kTileM / 32), cdiv_(nbf, kTileN) * (kTileN / 32));
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // exchange output tiles: a staircase over the upper triangle, the
    // column tiles of row tile r0 starting at column r0 (32-row operand
    // blocks allow any multiple of 32); every (m, c >= m) lies in the row
    // tile of m.  nbf 490: 15 tiles of 128 x 96 instead of 17 on the grid.
    std::vector<std::pair<int, int>> ktiles;
    for (int r0 = 0; r0 < nbf; r0 += kTileM)
      for (int c0 = r0; c0 < nbf; c0 += kTileN) ktiles.push_back({r0, c0});
    const int ntile = (int)ktiles.size();
    for (const auto& t : ktiles) h_nrb = std::max(h_nrb, cdiv_(t.second + kTileN, 32));
    std::vector<int> sizes = {xb};
    const int xlast = naux - (nbatch - 1) * xb;
    if (xlast != xb) sizes.push_back(xlast);
    ksplit = 1;
    for (int xbc : sizes) ksplit = std::max(ksplit, exchange_ksplit(xk_nkt(xbc), ntile));
    const size_t nH = fuse ? 1 : (size_t)nbf * hk;
    const size_t nEs = fuse ? (size_t)h_nrb * 32 * es_ld : 1;
    if (alloc(&d_Cslices, (size_t)ctot) != cudaSuccess ||
        alloc(&d_eC, (size_t)nblk * c_nrb * 32) != cudaSuccess ||
        alloc(&d_H, nH) != cudaSuccess ||
        alloc(&d_eoff, 2 * sizes.size() * nbf) != cudaSuccess ||
        alloc(&d_Hslices, (size_t)h_nrb * h_nkt * kSlices * kImage) != cudaSuccess ||
        alloc(&d_eH, (size_t)h_nrb * 32) != cudaSuccess ||
        alloc(&d_eHs, nEs) != cudaSuccess ||
        alloc(&d_Kpart, (size_t)ksplit * nbf * nbf) != cudaSuccess ||
        alloc(&d_dpart, jfused ? (size_t)nbf * naux : 1) != cudaSuccess ||
        alloc(&d_dt, (size_t)naux) != cudaSuccess ||
        cudaMemsetAsync(d_Cslices, 0, (size_t)ctot * 2, st) != cudaSuccess ||
        cudaMemsetAsync(d_eC, 0, (size_t)nblk * c_nrb * 32 * 4, st) != cudaSuccess ||
        cudaMemsetAsync(d_H, 0, nH * 8, st) != cudaSuccess ||
        cudaMemsetAsync(d_Hslices, 0, (size_t)h_nrb * h_nkt * kSlices * kImage * 2, st) !=
            cudaSuccess) {
      release_build();
      *err = "split path: out of memory for the per-build buffers";
      return GBJK_OOM;
    }
    // group exponents of rows that no half transform writes (beyond nbf,
    // panels without columns) stay "all zero"
    k_fill_int<<<(int)std::min<size_t>(cdiv_((long long)nEs, 256), 4 * nsm), 256, 0, st>>>(
        d_eHs, (long long)nEs, -2000);
    std::vector<SplitItem> items;
    std::vector<PrepJob> jobs(2 * nblk);
    hjobs.clear();
    std::vector<long long> eoff(2 * sizes.size() * nbf);
    plans.clear();
    for (size_t pi = 0; pi < sizes.size(); ++pi) {
      const int xbc = sizes[pi];
      BatchPlan pl;
      pl.xbc = xbc;
      // half transform: Hfit rows (m, y) of panel I, columns i (+ density);
      // A rows at m * pad32(xbc) + y
      pl.ht0 = (int)items.size();
      for (int I = 0; I < nblk; ++I) {
        const long long rows = (long long)bsize[I] * pad32(xbc);
        const int ncolI = nocc_ + (jfused ? bsize[I] : 0);
        for (int mt = 0; mt < cdiv_(rows, kTileM); ++mt)
          for (int nt = 0; nt < cdiv_(ncolI, kTileN); ++nt) {
            SplitItem w;
            w.a = d_Aslices + a_off[I];
            w.a_nrb = a_nrb[I];
            w.a_rb0 = mt * (kTileM / 32);
            w.b = d_Cslices + c_off[I];
            w.b_nrb = c_nrb;
            w.b_rb0 = nt * (kTileN / 32);
            w.kt0 = 0;
            w.nkt = nkt[I];
            w.ea = d_eA + eA_off[I] + (long long)mt * kTileM;
            w.eb = d_eC + (long long)I * c_nrb * 32 + (long long)nt * kTileN;
            w.apitch = pad32(xbc);
            w.arow0 = mt * kTileM;
            w.ay_valid = xbc;
            if (fuse) {
              // digits of H rows boff[I] + m, k-tile (y / 32) * nocc + i
              w.out = nullptr;
              w.ldr = 0;
              w.hdig = d_Hslices;
              w.h_nrb = h_nrb;
              w.hrow0 = boff[I];
              w.eseg = d_eHs;
              w.es_ld = es_ld;
              w.seg_nkt = nocc_;
            } else {
              // column-pair-outermost layout: each epilogue store is one
              // contiguous 512-byte run (SplitItem::perm_rs)
              w.out = nullptr;
              w.iout = d_H + (long long)boff[I] * pad32(xbc) * hld;
              w.ldr = hld;
              w.perm_rs = (long long)pad32(xbc) * hld;
              w.perm_div = xbc;
            }
            w.m_valid = (int)std::min<long long>(kTileM, rows - (long long)mt * kTileM);
            w.n_valid = std::min(kTileN, ncolI - nt * kTileN);
            // row (m, y) of panel I belongs to H row mu = boff[I] + m
            w.emax = d_eH + boff[I];
            w.emax_row0 = mt * kTileM;
            w.emax_div = xbc;
            // density column m' = col - nocc: g-partial of row (m, Y) if m' == m
            w.out2 = jfused ? d_dpart + (long long)boff[I] * naux : nullptr;
            w.c0 = nt * kTileN;
            w.ncol1 = nocc_;
            items.push_back(w);
          }
      }
      pl.nht = (int)items.size() - pl.ht0;
      // exchange: upper tiles, split over k
      const int nk_b = xk_nkt(xbc);
      const int ksb = exchange_ksplit(nk_b, ntile);
      const int kt_per = cdiv_(nk_b, ksb);
      pl.ksplit = cdiv_(nk_b, kt_per);
      pl.k0 = (int)items.size();
      for (int ks = 0; ks < pl.ksplit; ++ks) {
        const int kt0 = ks * kt_per;
        const int n_kt = std::min(kt_per, nk_b - kt0);
        for (const auto& t : ktiles) {
            const int r0 = t.first, c0 = t.second;
            SplitItem w;
            w.a = d_Hslices;
            w.a_nrb = h_nrb;
            w.a_rb0 = r0 / 32;
            w.b = d_Hslices;
            w.b_nrb = h_nrb;
            w.b_rb0 = c0 / 32;
            w.kt0 = kt0;
            w.nkt = n_kt;
            w.ea = d_eH + r0;
            w.eb = d_eH + c0;
            w.out = d_Kpart + (long long)ks * nbf * nbf + (long long)r0 * nbf + c0;
            w.ldr = nbf;
            w.m_valid = std::min(kTileM, nbf - r0);
            w.n_valid = std::min(kTileN, nbf - c0);
            w.emax = nullptr;
            w.emax_row0 = 0;
            w.emax_div = 1;
            w.out2 = nullptr;
            w.c0 = 0;
            w.ncol1 = 1 << 30;
            if (fuse) {
              // segment g = auxiliary group: nocc k-tiles with the
              // exponents of (row, g)
              w.seg_nkt = nocc_;
              w.esa = d_eHs + (long long)r0 * es_ld;
              w.esb = d_eHs + (long long)c0 * es_ld;
              w.es_ld = es_ld;
            }
            items.push_back(w);
          }
      }
      pl.nk = (int)items.size() - pl.k0;
      // digits of the half-transformed batch (row exponents from the
      // epilogue, element exponents from the two operands of the transform)
      SplitIntJob hj;
      hj.src = d_H;
      hj.rs = (long long)pad32(xbc) * hld;
      hj.ncols = hj.rs;
      hj.gs = 32LL * hld;
      hj.nrows = nbf;
      hj.ny = pad32(xbc);
      hj.ld = hld;
      hj.e = d_eH;
      hj.ea = d_eA;
      hj.ea_off = d_eoff + 2 * pi * nbf;
      hj.eb = d_eC;
      hj.eb_off = d_eoff + (2 * pi + 1) * nbf;
      hj.nrb = h_nrb;
      hj.nkt = nk_b;
      hj.dst = d_Hslices;
      for (int I = 0; I < nblk; ++I)
        for (int m = 0; m < bsize[I]; ++m) {
          eoff[2 * pi * nbf + boff[I] + m] = eA_off[I] + (long long)m * pad32(xbc);
          eoff[(2 * pi + 1) * nbf + boff[I] + m] = (long long)I * c_nrb * 32;
        }
      pl.hjob = (int)hjobs.size();
      hjobs.push_back(hj);
      plans.push_back(pl);
    }
    ht_nitems = plans[0].nht;
    ks_eff = plans[0].ksplit;
    k_nitems = plans[0].nk;
    for (int I = 0; I < nblk; ++I) {
      // rows of C: element (i, k) = C[colmap[k]][i]; then the density rows of the
      // panel's functions: P[boff + m][colmap[k]] (none when batched)
      PrepJob j;
      j.which = 0;
      j.off = 0;
      j.rs = 1;
      j.cs = nocc_;
      j.cm = dd_colmap + cmoff[I];
      j.ncols = panelK[I];
      j.row0 = 0;
      j.nrows = nocc_;
      j.e = d_eC + (long long)I * c_nrb * 32;
      j.nrb = c_nrb;
      j.nkt = nkt[I];
      j.dst = d_Cslices + c_off[I];
      jobs[I] = j;
      j.which = 1;
      j.off = (long long)boff[I] * nbf;
      j.rs = nbf;
      j.cs = 1;
      j.row0 = nocc_;
      j.nrows = jfused ? bsize[I] : 0;
      jobs[nblk + I] = j;
    }
    c_groups = prep_groups(jobs);
    if (alloc(&d_items, items.size()) != cudaSuccess || alloc(&d_jobs, jobs.size()) != cudaSuccess) {
      release_build();
      *err = "split path: out of memory for the work lists";
      return GBJK_OOM;
    }
    cudaMemcpy(d_items, items.data(), items.size() * sizeof(SplitItem), cudaMemcpyHostToDevice);
    cudaMemcpy(d_eoff, eoff.data(), eoff.size() * sizeof(long long), cudaMemcpyHostToDevice);
    cudaMemcpy(d_jobs, jobs.data(), jobs.size() * sizeof(PrepJob), cudaMemcpyHostToDevice);
    nocc = nocc_;
    return GBJK_OK;
  }

  gbjk_status prepare(cudaStream_t st, const double* d_B, const double* d_Linv, int nocc_,
                      int64_t* launches, std::string* err) {
    gbjk_status s;
    if (!b_ready && (s = prepare_b(st, d_B, d_Linv, launches, err))) return s;
    if (nocc != nocc_ && (s = prepare_nocc(st, nocc_, err))) return s;
    return GBJK_OK;
  }

  bool fused_j() const { return nbatch == 1; }

  // --- per build ------------------------------------------------------------
  // dC: nbf x nocc; dP: nbf x nbf, or null (no density partials)
  gbjk_status run_k(cudaStream_t st, const double* dC, const double* dP, double* dK,
                    int64_t* launches, std::string* err) {
    gbjk_status s;
    // the flag a timed-out wait sets is per build: cleared at its start
    if (cudaMemsetAsync(d_err, 0, sizeof(int), st) != cudaSuccess) {
      *err = "split path: memset failed";
      return GBJK_CUDA_ERROR;
    }
    {
      Scope sc(this, 2, st);
      k_prep_rows<<<dim3(c_groups, 2 * nblk), 256, 0, st>>>(d_jobs, dC, dP);
      (*launches)++;
    }
    for (int b = 0; b < nbatch; ++b) {
      const BatchPlan& pl = plans[(b == nbatch - 1 && plans.size() > 1) ? 1 : 0];
      if (nbatch > 1) {
        Scope sc(this, 2, st);
        const SplitJob* bj = d_bjobs + (size_t)b * nbf;
        k_split_rows<<<dim3(cdiv_(pl.xbc / 8 + 2, 8), nbf), 256, 0, st>>>(bj);
        (*launches)++;
      }
      if (nbatch > 1 && !hfuse_eff && pad32(pl.xbc) != pl.xbc) {
        // the last batch's H layout reuses slots the full batches wrote:
        // clear its unused auxiliary slots
        Scope sc(this, 2, st);
        const long long per = (long long)nbf * (hld / 2) * (32 - (pl.xbc & 31));
        k_zero_hpad<<<(int)std::min<long long>(cdiv_(per, 256), 4LL * nsm), 256, 0, st>>>(
            d_H, nbf, (long long)pad32(pl.xbc) * hld, (long long)(pl.xbc & ~31) * hld,
            pl.xbc & 31, hld / 2);
        (*launches)++;
      }
      {
        Scope sc(this, 0, st);
        // H row exponents are atomically maximised by the half-transform epilogue
        if (cudaMemsetAsync(d_eH, kNoExpByte, (size_t)h_nrb * 32 * sizeof(int), st) !=
            cudaSuccess) {
          *err = "split path: memset failed";
          return GBJK_CUDA_ERROR;
        }
        if (hfuse_eff)
          s = launch_gemm_v<true, false, kOutF64>(st, d_items + pl.ht0, pl.nht, launches, err, 0);
        else
          s = launch_gemm<kOutInt>(st, d_items + pl.ht0, pl.nht, launches, err);
        if (s) return s;
      }
      if (ev_ht && nbatch == 1 && cudaEventRecord(ev_ht, st) != cudaSuccess) {
        *err = "split path: event record failed";
        return GBJK_CUDA_ERROR;
      }
      if (!hfuse_eff) {
        Scope sc(this, 2, st);
        launch_ints<true>(st, &hjobs[pl.hjob], 1, launches);
      }
      {
        Scope sc(this, 1, st);
        if (hfuse_eff)
          s = launch_gemm_v<false, true, kOutF64>(st, d_items + pl.k0, pl.nk, launches, err, k_grid);
        else
          s = launch_gemm(st, d_items + pl.k0, pl.nk, launches, err, k_grid);
        if (s) return s;
      }
      k_splitk_reduce_acc<<<cdiv_((long long)nbf * nbf, 256), 256, 0, st>>>(
          d_Kpart, pl.ksplit, nbf, -1.0, 1, b > 0 ? 1 : 0, dK);
      (*launches)++;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      *err = std::string("split path launch: ") + cudaGetErrorString(e);
      return GBJK_CUDA_ERROR;
    }
    return GBJK_OK;
  }

  // clear the timed-out-wait flag at the start of a computation (stream order)
  gbjk_status clear_error(cudaStream_t st) {
    if (d_err && cudaMemsetAsync(d_err, 0, sizeof(int), st) != cudaSuccess) return GBJK_CUDA_ERROR;
    return GBJK_OK;
  }
  // error code recorded by a timed-out wait inside the split GEMM (0 = none)
  int read_error() {
    int h = 0;
    if (d_err) cudaMemcpy(&h, d_err, sizeof(int), cudaMemcpyDeviceToHost);
    return h;
  }
};

}  // namespace gbjk
