// The prefit Bfit = L^-1 B of the mixed path on the tensor cores, to FP64
// accuracy.
//
// FP64 operands become 63-bit integers: a row's elements relative to the
// row's exponent e (|x| < 2^e), X = rint(|x| 2^(63-e)), in eight balanced
// base-256 digits, exact in BF16 (the top one in [0, 128]).  Before that the
// contracted index is balanced: column Y of L^-1 is divided, row Y of B
// multiplied, by a power of two that takes the column's largest element to 1
// (k_pf_balance), so that the scale of an auxiliary function does not matter.  The product keeps
// the 36 digit pairs (s, t) with s + t <= 7; all eight diagonals d = s + t are
// summed exactly: a digit product is at most 2^14, so 128 k of at most eight
// pairs stay within 2^24, exact in the FP32 accumulators.  Every 128 k the
// epilogue adds them, as integers, to two int64 per output,
//   HI = sum_{d<4} r_d 256^(3-d),  LO = sum_{d>=4} r_d 256^(7-d),
// and a result is (HI 2^32 + LO) 2^(eA+eB-70), rounded once.  What is lost is
// the operands' rounding at 2^-63 of their rows' largest elements and the
// dropped pairs: for a result (X, c) about 2^-56 max_Y |L^-1[X][Y]| max_Y
// |B[Y][c]| of the balanced operands.  An in-order FP64 sum loses 2^-53 of its
// partial sums.  Over a column c the first is the smaller by far, but a
// single result whose terms are all far below the column's is further off here;
// those who read the tensor take sums over X, where it drowns.
//
// This is the set-up cost of every new molecule: naux nnz(B) / 2 products, on
// GB300's FP64 pipe (6e11 fma/s) 162 ms for C12H26 and 740 ms for C20H42.
//
// Operand A (M = 128): tensor columns (m, k) of a panel, contracted over Y;
// operand B (N = 48): rows X of L^-1, so that TMEM lanes are tensor columns and
// a warp's results of one X are 256 contiguous bytes.  Tiles of both are stored
// as [k-tile][digit][8-row group][k/8][row][8] in one run each, so a pipeline
// stage is two bulk copies (64 KB + 24 KB).  Adjacent digits of B and adjacent
// diagonals let one MMA of N = 48 n cover n pairs: 11 MMAs per 16 k.  A lower
// triangular L^-1 ends the k range of an X tile at its last row.  One CTA per
// SM: producer warp, MMA warp, twelve epilogue warps (three column thirds per
// TMEM lane quadrant); two stages; waits bounded as in split_gemm.cuh.
#pragma once
#include <stdint.h>

#include "common.cuh"
#include "split_gemm.cuh"

namespace gbjk {

constexpr int kPfDigits = 8, kPfM = 128, kPfN = 48, kPfK = 32;
constexpr int kPfChunk = 4;  // k-tiles per exact chunk (128 k)
constexpr int kPfStages = 2;
constexpr int kPfBytesA = kPfDigits * kPfM * kPfK * 2, kPfBytesB = kPfDigits * kPfN * kPfK * 2;
constexpr int kPfSmem = kPfStages * (kPfBytesA + kPfBytesB) + 1024;
constexpr int kPfCols = kPfN / 3;  // output columns per epilogue thread
// exponent of a row without a nonzero element; those of balanced rows reach
// from -9213 to 2048
constexpr int kPfNone = -1000000;

// 128 tensor columns: c = c0 .. c0 + 127 of the panel's ncol = b_I K_I columns
// (m, k), element Y at src[(m * naux + Y) * K + k], results likewise in dst.
struct PfTile {
  const double* src;
  double* dst;
  int K, c0, ncol;
};

// The eight digits of eight elements x 2^b of one row (k run), 16 bytes per
// digit.
__device__ __forceinline__ void store_digits8x8(const double (&x)[8], const int (&b)[8], int e,
                                                uint16_t* p, int sstride) {
  unsigned long long T[8];
  uint32_t sgn[4] = {0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x[j]);
    const int E = (int)((u >> 52) & 0x7FF);
    const unsigned long long m = (u & ((1ull << 52) - 1)) | (1ull << 52);
    // X = m 2^-sh, sh >= -10 since |x 2^b| < 2^e
    const int sh = e + 1012 - E - b[j];
    unsigned long long X = sh <= 0 ? m << min(-sh, 10) : (shr_u64(m, sh - 1) + 1) >> 1;
    if (E == 0 || e == kPfNone) X = 0;
    T[j] = X + 0x0080808080808080ull;
    if (u >> 63) sgn[j >> 1] |= (j & 1) ? 0x80000000u : 0x8000u;
  }
#pragma unroll
  for (int s = 0; s < kPfDigits; ++s) {
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float f[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const unsigned long long t = T[2 * j + h];
        const uint32_t w = s < 4 ? (uint32_t)(t >> 32) : (uint32_t)t;
        const float d = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 | (3 - (s & 3))));
        f[h] = s == 0 ? d - 8388608.0f : d - 8388736.0f;
      }
      o[j] = __byte_perm(__float_as_uint(f[0]), __float_as_uint(f[1]), 0x7632) ^ sgn[j];
    }
    *reinterpret_cast<uint4*>(p + s * sstride) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// b[Y]: the exponent of the largest element of column Y of L^-1; a function taken
// 2^s times as large lowers it by s, which leaves every digit as it is.  No
// element of the balanced L^-1 is above 1, and in every column some are: the
// error of a result (X, c) is bounded by the largest product |L^-1[X'][Y] B[Y][c]|
// of its column c, whatever the other columns' scales are.  (Balancing against
// the tensor's rows too halves the error of fitting bases, but takes a pass
// over the tensor, and the largest columns then spoil the others.)  A column of
// zeros takes its row of the tensor out of the sums.  A block walks 32 columns of
// the lower triangle, 32 rows at a time: 11 us for C12H26.
// grid ceil(naux / 32), block (32, 32).
__global__ void __launch_bounds__(1024)
    k_pf_balance(const double* __restrict__ L, int naux, int* __restrict__ b) {
  __shared__ unsigned int sm[32][33];
  const int Y = blockIdx.x * 32 + threadIdx.x;
  unsigned int mx = 0;
  if (Y < naux)
#pragma unroll 4
    for (int X = blockIdx.x * 32 + threadIdx.y; X < naux; X += 32)
      if (X >= Y)
        mx = max(mx, (unsigned int)(__double_as_longlong(L[(long long)X * naux + Y]) >> 52) & 0x7FF);
  sm[threadIdx.x][threadIdx.y] = mx;
  __syncthreads();
  // warp y holds column 32 blockIdx.x + y
  mx = __reduce_max_sync(0xffffffffu, sm[threadIdx.y][threadIdx.x]);
  if (threadIdx.x == 0) b[blockIdx.x * 32 + threadIdx.y] = mx ? (int)mx - 1023 : -8192;
}

// Exponents of a tile's 128 tensor columns (max over Y); grid ntiles, block
// (128, 4).
__global__ void __launch_bounds__(512)
    k_pf_colexp(const PfTile* __restrict__ tiles, const int* __restrict__ b, int naux,
                int* __restrict__ e) {
  __shared__ int sm[4][128];
  const PfTile t = tiles[blockIdx.x];
  const int c = t.c0 + threadIdx.x, lane = threadIdx.x & 31;
  int mx = kPfNone;
  {
    const int cc = min(c, t.ncol - 1);
    const int m = cc / t.K, k = cc - m * t.K;
    const double* p = t.src + (long long)m * naux * t.K + k;
    // Bound by the latency of its loads: sixteen high words on their way, then
    // the balances of their Y, which the lanes brought and pass on (six waters 62
    // us; 148 with a load each beside the element's and eight on their way).
    for (int Y0 = threadIdx.y; Y0 < naux; Y0 += 64) {
      const int Yl = min(Y0 + 4 * (lane & 15), naux - 1);
      const int bl = __ldg(b + Yl);
      unsigned int h[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int Y = Y0 + 4 * j;
        h[j] = Y < naux ? __ldg(reinterpret_cast<const unsigned int*>(p + (long long)Y * t.K) + 1)
                        : 0u;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int E = (int)(h[j] >> 20) & 0x7FF;
        const int eb = __shfl_sync(0xffffffffu, bl, j) + E - 1022;
        mx = max(mx, E ? eb : kPfNone);
      }
    }
  }
  sm[threadIdx.y][threadIdx.x] = mx;
  __syncthreads();
  if (threadIdx.y == 0) {
    mx = max(max(sm[0][threadIdx.x], sm[1][threadIdx.x]),
             max(sm[2][threadIdx.x], sm[3][threadIdx.x]));
    e[blockIdx.x * kPfM + threadIdx.x] = mx;
  }
}

// Digits of the tensor columns.  One warp per (8-column group, k-tile): lane
// (rr, kc) handles column 8 g + rr, Y = 32 kt + 8 kc .. + 7.  grid (ntiles,
// ceil(16 nkt / 8)), block 256.
__global__ void __launch_bounds__(256)
    k_pf_coldigits(const PfTile* __restrict__ tiles, const int* __restrict__ e,
                   const int* __restrict__ b, int naux, int nkt, uint16_t* __restrict__ dst) {
  const int wid = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int g = wid & 15, kt = wid >> 4;
  if (kt >= nkt) return;
  const PfTile t = tiles[blockIdx.x];
  const int r = 8 * g + (lane & 7), kc = lane >> 3;
  const int c = t.c0 + r;
  const int Y0 = kt * kPfK + kc * 8;
  double x[8];
  int bal[8];
  const int m = c / t.K, k = c - m * t.K;
  const double* p = t.src + ((long long)m * naux + Y0) * t.K + k;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    x[j] = c < t.ncol && Y0 + j < naux ? __ldg(p + (long long)j * t.K) : 0.0;
    bal[j] = __ldg(b + Y0 + j);
  }
  uint16_t* o = dst + ((long long)blockIdx.x * nkt + kt) * (kPfBytesA / 2) + g * 256 + kc * 64 +
                (lane & 7) * 8;
  store_digits8x8(x, bal, e[blockIdx.x * kPfM + r], o, kPfM * kPfK);
}

// Exponents and digits of the rows of L^-1 from row0 on (a multiple of 48;
// entries right of the diagonal are taken as zero).  grid ceil(rows / 8), block
// 256: the block's eight warps find the exponents of its eight rows, then share
// their k-tiles.  Row X goes to tile (X - row0) / 48; rows of the last tile beyond
// naux stay as they are (zero).
__global__ void __launch_bounds__(256)
    k_pf_metric(const double* __restrict__ L, const int* __restrict__ b, int naux, int row0,
                int nkt, int* __restrict__ e, uint16_t* __restrict__ dst) {
  __shared__ int se[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  {
    const int X = row0 + blockIdx.x * 8 + warp;
    int mx = kPfNone;
    if (X < naux)
      for (int Y = lane; Y <= X; Y += 32) {
        const int E = (int)(__double_as_longlong(L[(long long)X * naux + Y]) >> 52) & 0x7FF;
        const int eb = E - __ldg(b + Y) - 1022;
        mx = max(mx, E ? eb : kPfNone);
      }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) {
      se[warp] = mx;
      if (X < naux) e[X] = mx;
    }
  }
  __syncthreads();
  const int rr = lane & 7, kc = lane >> 3;
  const int X = row0 + blockIdx.x * 8 + rr;
  const int xt = (blockIdx.x * 8) / kPfN, g = blockIdx.x - xt * (kPfN / 8);
  for (int kt = warp; kt < nkt; kt += 8) {
    const int Y0 = kt * kPfK + kc * 8;
    double x[8];
    int bal[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      x[j] = X < naux && Y0 + j <= X ? L[(long long)X * naux + Y0 + j] : 0.0;
      bal[j] = -__ldg(b + Y0 + j);
    }
    store_digits8x8(x, bal, se[rr],
                    dst + ((long long)xt * nkt + kt) * (kPfBytesB / 2) + g * 256 + kc * 64 + rr * 8,
                    kPfN * kPfK);
  }
}

// v 2^e for a finite v: the exponent field where the result stays normal
__device__ __forceinline__ double scale_exp2(double v, int e) {
  const long long b = __double_as_longlong(v);
  const int E = (int)((b >> 52) & 0x7FF);
  if (E == 0) return v;  // only zero: a nonzero v is an integer
  const int ex = E + e;
  return ex > 0 && ex < 2047 ? __longlong_as_double(b + ((long long)e << 52)) : ldexp(v, e);
}

// Work item it of a launch over nxt X tiles: tensor tile it / nxt, X tile rotated by
// the tile so that every CTA meets all k lengths whatever the grid size.
__device__ __forceinline__ void pf_item(int it, int nxt, int* tile, int* xt) {
  *tile = it / nxt;
  *xt = nxt - 1 - (it + *tile) % nxt;
}
__device__ __forceinline__ int pf_nkt(int xt, int naux) {
  return (min(naux, (xt + 1) * kPfN) + kPfK - 1) / kPfK;
}

// X tiles xt0 .. xt0 + nxt - 1, whose digits bdig holds.
__global__ void __launch_bounds__(kThreads, 1)
    k_prefit_gemm(const PfTile* __restrict__ tiles, int nitems, int nxt, int xt0, int naux, int nkt_all,
                  const uint16_t* __restrict__ adig, const int* __restrict__ ea,
                  const uint16_t* __restrict__ bdig, const int* __restrict__ eb,
                  int* __restrict__ err, unsigned long long spin_ns) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sA = smem;
  unsigned char* sB = smem + kPfStages * kPfBytesA;
  __shared__ uint64_t full_bar[kPfStages], empty_bar[kPfStages];
  __shared__ uint64_t acc_full, acc_empty, mma_drain;
  __shared__ uint32_t tmem_base_sh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kPfStages; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init(&acc_empty, kEpiWarps);
    mbar_init(&mma_drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_sh)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_sh;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      uint32_t last_par[kPfStages];
      bool issued[kPfStages];
#pragma unroll
      for (int i = 0; i < kPfStages; ++i) issued[i] = false;
      for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
        int tile, xt;
        pf_item(it, nxt, &tile, &xt);
        const int nkt = pf_nkt(xt0 + xt, naux);
        const unsigned char* ga = (const unsigned char*)adig + (long long)tile * nkt_all * kPfBytesA;
        const unsigned char* gb = (const unsigned char*)bdig + (long long)xt * nkt_all * kPfBytesB;
        for (int k = 0; k < nkt; ++k) {
          ok = mbar_wait(&empty_bar[stage], phase ^ 1, err, 11, spin_ns);
          if (!ok) break;
          mbar_arrive_expect_tx(&full_bar[stage], kPfBytesA + kPfBytesB);
          bulk_g2s(sA + stage * kPfBytesA, ga + (long long)k * kPfBytesA, kPfBytesA,
                   &full_bar[stage]);
          bulk_g2s(sB + stage * kPfBytesB, gb + (long long)k * kPfBytesB, kPfBytesB,
                   &full_bar[stage]);
          last_par[stage] = phase;
          issued[stage] = true;
          if (++stage == kPfStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      // every copy this CTA issued lands before it can exit
      for (int i = 0; i < kPfStages; ++i)
        if (issued[i]) mbar_wait_own(&full_bar[i], last_par[i], spin_ns);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
        int tile, xt;
        pf_item(it, nxt, &tile, &xt);
        const int nkt = pf_nkt(xt0 + xt, naux);
        for (int k = 0; k < nkt; ++k) {
          const bool chunk_start = (k % kPfChunk) == 0;
          const bool chunk_end = ((k + 1) % kPfChunk) == 0 || k + 1 == nkt;
          ok = mbar_wait(&full_bar[stage], phase, err, 12, spin_ns);
          if (!ok) break;
          if (chunk_start) {
            ok = mbar_wait(&acc_empty, acc_phase ^ 1, err, 13, spin_ns);
            acc_phase ^= 1;
            if (!ok) {
              mma_commit(&empty_bar[stage]);
              break;
            }
          }
          tc_fence_after();
          const uint64_t adesc = smem_desc(smem_u32(sA + stage * kPfBytesA));
          const uint64_t bdesc = smem_desc(smem_u32(sB + stage * kPfBytesB));
          // descriptor start addresses advance in 16-byte units; the second
          // K = 16 step is two core matrices (256 B) on
          constexpr uint32_t kSliceA = kPfM * kPfK * 2 / 16, kSliceB = kPfN * kPfK * 2 / 16;
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int s = 0; s < kPfDigits; ++s)
#pragma unroll
              for (int t0 = 0; t0 < kPfDigits - s; t0 += 5) {
                const int n = min(5, kPfDigits - s - t0);
                mma_bf16(tmem + (uint32_t)((s + t0) * kPfN),
                         adesc + (uint64_t)(s * kSliceA + j * 16),
                         bdesc + (uint64_t)(t0 * kSliceB + j * 16), instr_desc(kPfM, kPfN * n),
                         chunk_start && s == 0 && j == 0 ? 0u : 1u);
              }
          mma_commit(&empty_bar[stage]);
          if (chunk_end) mma_commit(&acc_full);
          if (++stage == kPfStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      // every MMA completes before TMEM is freed and the CTA exits
      mma_commit(&mma_drain);
      mbar_wait_own(&mma_drain, 0, spin_ns);
    }
  } else {
    const int q = warp & 3, third = (warp - 2) >> 2;
    const int row = q * 32 + lane;
    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(third * kPfCols);
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
      int tile, xt;
      pf_item(it, nxt, &tile, &xt);
      const int nchunk = (pf_nkt(xt0 + xt, naux) + kPfChunk - 1) / kPfChunk;
      const PfTile& t = tiles[tile];
      const int er = ea[tile * kPfM + row];
      const int X0 = (xt0 + xt) * kPfN + third * kPfCols;
      long long HI[kPfCols], LO[kPfCols];
#pragma unroll
      for (int c = 0; c < kPfCols; ++c) HI[c] = LO[c] = 0;
      for (int ch = 0; ch < nchunk; ++ch) {
        ok = mbar_wait(&acc_full, acc_phase, err, 14, spin_ns);
        acc_phase ^= 1;
        if (!ok) break;
        tc_fence_after();
        uint32_t a[16], b[16];
        int t01[kPfCols];
        tmem_ld16(taddr, a);
        tmem_ld16(taddr + kPfN, b);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < kPfCols; ++c)  // |r0| <= 2^21
          t01[c] = (__float2int_rn(__uint_as_float(a[c])) << 8) +
                   __float2int_rn(__uint_as_float(b[c]));
        tmem_ld16(taddr + 2 * kPfN, a);
        tmem_ld16(taddr + 3 * kPfN, b);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < kPfCols; ++c)  // |r2| <= 3 * 2^21
          HI[c] += ((long long)t01[c] << 16) +
                   ((__float2int_rn(__uint_as_float(a[c])) << 8) +
                    __float2int_rn(__uint_as_float(b[c])));
        tmem_ld16(taddr + 4 * kPfN, a);
        tmem_ld16(taddr + 5 * kPfN, b);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < kPfCols; ++c)
          LO[c] += (long long)__float2int_rn(__uint_as_float(a[c])) * 16777216 +
                   (long long)__float2int_rn(__uint_as_float(b[c])) * 65536;
        tmem_ld16(taddr + 6 * kPfN, a);
        tmem_ld16(taddr + 7 * kPfN, b);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty);
#pragma unroll
        for (int c = 0; c < kPfCols; ++c)
          LO[c] += (long long)__float2int_rn(__uint_as_float(a[c])) * 256 +
                   __float2int_rn(__uint_as_float(b[c]));
      }
      if (!ok) break;
      const int col = t.c0 + row;
      if (col < t.ncol) {
        const int K = t.K, m = col / K, k = col - m * K;
        double* o = t.dst + ((long long)m * naux + X0) * K + k;
#pragma unroll
        for (int c = 0; c < kPfCols; ++c) {
          if (X0 + c >= naux) break;
          const int ec = __ldg(eb + X0 + c);
          const double v = fma((double)HI[c], 4294967296.0, (double)LO[c]);
          o[(long long)c * K] = er == kPfNone || ec == kPfNone ? 0.0 : scale_exp2(v, er + ec - 70);
        }
      }
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols)
                 : "memory");
  }
}

}  // namespace gbjk
