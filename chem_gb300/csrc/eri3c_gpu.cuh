// 3-center Coulomb integrals (X|mu nu) on the device, written straight into
// the atom-block panel layout of the resident tensor.
//
// The host engine (chem_gb300/csrc/ints, standing in for the libcint calls
// of megalochem's ints::aoloader, src/ints/integrals.cpp:250-370) computes
// the same tensor; this kernel follows its McMurchie-Davidson scheme and
// conventions (normalised contractions exported by gbints_basis_shells,
// real spherical harmonics from gbints_sph_coeffs, the primitive cut 1e-16)
// so that the two agree to rounding:
//   for a primitive pair (a_i, b_j): Hermite coefficients E^{ab}_{tuv}
//   (Helgaker, Jorgensen, Olsen eq. 9.5.6-9.5.7), for every auxiliary
//   primitive c_k the Hermite Coulomb integrals R_{tuv}(alpha, P - C)
//   (eq. 9.9.18-9.9.20, Boys function from a table of Taylor expansions and
//   downward recursion, or erf and upward recursion for large arguments),
//   contracted with the single-centre expansion of c and its spherical
//   transform into W[tuv][mc], then with E^{ab} folded with both spherical
//   transforms into the results.
// Work: a block takes an AO shell pair (a in block I, b in block J, a <= b
// when I == J) of a kept block pair and a range of auxiliary blocks; its 4
// warps take the kept auxiliary shells of the range in turn (k_eri3c).  The R
// table of a primitive triple lives in the warp's shared memory.  Supported:
// AO shells up to d and auxiliary shells up to f (la + lb + lc <= 7); the host
// checks.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <cstring>

namespace gbjk {

constexpr int kEriMaxLao = 2, kEriMaxLaux = 3;
constexpr int kEriMaxL = 2 * kEriMaxLao + kEriMaxLaux;                           // 7
constexpr int kEriNR = (kEriMaxL + 1) * (kEriMaxL + 2) * (kEriMaxL + 3) / 6;     // 120
constexpr int kEriLb = 2 * kEriMaxLao;                                           // 4
constexpr int kEriNW = (kEriLb + 1) * (kEriLb + 2) * (kEriLb + 3) / 6;           // 35
constexpr int kEriMaxSph = 7;
constexpr int kEriWarps = 4;
// Boys values (-2 alpha)^n F_n(T), n <= L, of up to kEriRnChunk (bra
// primitive pair, auxiliary primitive) combinations, computed across the
// lanes of a warp before the combinations are processed one by one
constexpr int kEriRnChunk = 64;
// ket matrix M[mc][j] of an auxiliary primitive: j over the Hermite
// indices of t + u + v <= l_aux (at most 20), mc over its spherical components
constexpr int kEriNKet = (kEriMaxLaux + 1) * (kEriMaxLaux + 2) * (kEriMaxLaux + 3) / 6;  // 20
constexpr int kEriList = 512;  // kept auxiliary shells listed at a time
constexpr int kEriWarpDoubles = 2 * kEriNR + kEriNW * kEriMaxSph +
                                kEriRnChunk * (kEriMaxL + 1) +
                                kEriMaxSph * kEriNKet;  // R x2, W, rn, M
// cartesian -> spherical tables for l = 0..3, at offsets 0, 1, 10, 40
__constant__ double c_eri_sph[1 + 9 + 30 + 70];
// (t, u, v) of the compact Hermite index e (t + u + v <= 7): t | u << 8 | v << 16
__constant__ int c_eri_tuv[kEriNR];
// 1 / (2 j + 1) for the Boys recursion (no FP64 division there)
__constant__ double c_eri_rodd[kEriMaxL + 1];

struct EriShell {
  int l, nprim, prim0, bf_off, blk;  // blk: auxiliary block (auxiliary shells)
  double A[3];
};
// AO shells a, b of block pair p with the auxiliary blocks [A0, A1), of their
// shells those with a momentum in the mask ls
struct EriItem {
  int p, a, b, A0, A1, ls;
};

__device__ __forceinline__ int eri_tet(int n) { return n * (n + 1) * (n + 2) / 6; }
// compact index of (t, u, v) among all t + u + v <= L (independent of L)
__device__ __forceinline__ int eri_idx(int t, int u, int v) {
  const int s = t + u + v, r = u + v;
  return eri_tet(s) + r * (r + 1) / 2 + v;
}
__device__ __forceinline__ int eri_sph_off(int l) { return l == 0 ? 0 : l == 1 ? 1 : l == 2 ? 10 : 40; }
__device__ __forceinline__ void eri_cart(int l, int c, int* ex) {
  int idx = 0;
  for (int ix = l; ix >= 0; --ix)
    for (int iy = l - ix; iy >= 0; --iy) {
      if (idx == c) {
        ex[0] = ix;
        ex[1] = iy;
        ex[2] = l - ix - iy;
        return;
      }
      ++idx;
    }
}

// Boys function F_0..F_n at T.  Below T = kEriBoysTmax F_n comes from its
// Taylor expansion about the nearest grid point (eight terms, |dT| <= 1/32, the
// next one below 3e-17 of F), e^-T likewise, and the lower orders by downward
// recursion; above, erf and upward recursion, as in the host engine.  FP64
// instructions are what bounds this kernel, and the series this replaces took
// two to three hundred of them per argument.
constexpr double kEriBoysTmax = 33.0;
constexpr int kEriBoysStep = 16;  // grid points per unit of T
constexpr int kEriBoysRows = (int)kEriBoysTmax * kEriBoysStep + 2;
// table row of order n at T0 = i / 16: F_{n+k}(T0) / k!, k = 0..7, at
// tab[(n * kEriBoysRows + i) * 8]; e^-T0 at tab[kEriBoysExp + i]
constexpr int kEriBoysExp = (kEriMaxL + 1) * kEriBoysRows * 8;
constexpr int kEriBoysTable = kEriBoysExp + kEriBoysRows;

// Host: the table, by the ascending series of F_15 and downward recursion.
inline void eri_boys_table(double* tab) {
  for (int i = 0; i < kEriBoysRows; ++i) {
    const double T = (double)i / kEriBoysStep, eT = std::exp(-T);
    double F[kEriMaxL + 8];
    const int top = kEriMaxL + 7;
    double term = 1.0 / (2 * top + 1), sum = term;
    for (int k = 1; k < 400 && term > 1e-18 * sum; ++k) {
      term *= 2.0 * T / (2 * (top + k) + 1);
      sum += term;
    }
    F[top] = eT * sum;
    for (int m = top - 1; m >= 0; --m) F[m] = (2.0 * T * F[m + 1] + eT) / (2 * m + 1);
    for (int n = 0; n <= kEriMaxL; ++n) {
      double fac = 1.0;
      for (int k = 0; k < 8; ++k) {
        if (k) fac *= k;
        tab[((size_t)n * kEriBoysRows + i) * 8 + k] = F[n + k] / fac;
      }
    }
    tab[kEriBoysExp + i] = eT;
  }
}

// T as the table takes it: an argument below zero, which only a negative exponent
// gives, counts as zero; NaN stays.  (On the bits: an FP64 compare would cost as
// much as a product.)
__host__ __device__ __forceinline__ double eri_boys_arg(double T) {
#ifdef __CUDA_ARCH__
  const uint32_t hi = (uint32_t)__double2hiint(T);
#else
  uint64_t u;
  std::memcpy(&u, &T, 8);
  const uint32_t hi = (uint32_t)(u >> 32);
#endif
  return hi - 0x80000000u <= 0x7FF00000u ? 0.0 : T;
}
// Its table row, for 0 <= T <= kEriBoysTmax or NaN (row 0)
__host__ __device__ __forceinline__ int eri_boys_row(double T) {
  return (int)((float)T * (float)kEriBoysStep + 0.5f);
}

__device__ __forceinline__ void eri_boys(const double* __restrict__ tab, int nmax, double T,
                                         double* F) {
  T = eri_boys_arg(T);
  if (T > kEriBoysTmax) {
    const double eT = exp(-T);
    F[0] = 0.5 * sqrt(3.14159265358979323846 / T) * erf(sqrt(T));
    const double inv2T = 0.5 / T;
    for (int m = 0; m < nmax; ++m) F[m + 1] = ((2 * m + 1) * F[m] - eT) * inv2T;
    return;
  }
  const int i = eri_boys_row(T);
  const double x = (double)i * (1.0 / kEriBoysStep) - T;
  const double2* c = reinterpret_cast<const double2*>(tab + ((long long)nmax * kEriBoysRows + i) * 8);
  const double2 c0 = __ldg(c), c1 = __ldg(c + 1), c2 = __ldg(c + 2), c3 = __ldg(c + 3);
  double f = fma(c3.y, x, c3.x);
  f = fma(f, x, c2.y);
  f = fma(f, x, c2.x);
  f = fma(f, x, c1.y);
  f = fma(f, x, c1.x);
  f = fma(f, x, c0.y);
  f = fma(f, x, c0.x);
  F[nmax] = f;
  if (nmax == 0) return;
  double e = fma(x, 1.0 / 5040, 1.0 / 720);
  e = fma(e, x, 1.0 / 120);
  e = fma(e, x, 1.0 / 24);
  e = fma(e, x, 1.0 / 6);
  e = fma(e, x, 0.5);
  e = fma(e, x, 1.0);
  e = fma(e, x, 1.0);
  const double eT = e * __ldg(tab + kEriBoysExp + i);
  const double twoT = 2.0 * T;
  for (int m = nmax - 1; m >= 0; --m) F[m] = fma(twoT, F[m + 1], eT) * c_eri_rodd[m];
}

// Ket matrix of an auxiliary primitive of exponent qq and angular momentum
// lc, computed across the lanes of a warp into M (row stride kEriNKet):
//   M[mc][j] = (-1)^(t+u+v) sum_cc sph[mc][cc] Ec[cx][t] Ec[cy][u] Ec[cz][v],
// (t, u, v) the Hermite index j, (cx, cy, cz) the cartesian exponents of cc,
// Ec the single-centre Hermite expansion.  The contraction with the R table
// is then W[tuv][mc] = pref sum_j M[mc][j] R[(t, u, v) + j].
__device__ void eri_ket_matrix(int lc, double qq, int lane, double* M) {
  double Ec[kEriMaxLaux + 1][kEriMaxLaux + 2];
  for (int i = 0; i <= kEriMaxLaux; ++i)
    for (int t = 0; t <= kEriMaxLaux + 1; ++t) Ec[i][t] = 0.0;
  Ec[0][0] = 1.0;
  const double oo2q = 0.5 / qq;
  for (int i = 0; i < lc; ++i)
    for (int t = 0; t <= i + 1; ++t) {
      double v = (t + 1) * Ec[i][t + 1];
      if (t > 0) v += oo2q * Ec[i][t - 1];
      Ec[i + 1][t] = v;
    }
  const int ncc = (lc + 1) * (lc + 2) / 2, nsc = 2 * lc + 1, nr = eri_tet(lc + 1);
  const double* sc = c_eri_sph + eri_sph_off(lc);
  for (int en = lane; en < nsc * nr; en += 32) {
    const int mc = en / nr, j = en % nr;
    const int tuv = c_eri_tuv[j];
    const int t = tuv & 255, u = (tuv >> 8) & 255, v = tuv >> 16;
    double m = 0.0;
    for (int cc = 0; cc < ncc; ++cc) {
      int ex[3];
      eri_cart(lc, cc, ex);
      if (t > ex[0] || u > ex[1] || v > ex[2]) continue;
      m += sc[mc * ncc + cc] * (Ec[ex[0]][t] * Ec[ex[1]][u] * Ec[ex[2]][v]);
    }
    M[mc * kEriNKet + j] = ((t + u + v) & 1) ? -m : m;
  }
}

// The ket matrices of every auxiliary primitive, kEriKetSize doubles each: once
// per tensor (every AO shell pair used to rebuild them).  grid ceil(nprim / 4),
// block 128.
constexpr int kEriKetSize = kEriMaxSph * kEriNKet;
__global__ void k_eri_ket(const EriShell* __restrict__ ax, int nshell,
                          const double* __restrict__ ax_alpha, int nprim, double* __restrict__ M) {
  const int k = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k >= nprim) return;
  int lo = 0, hi = nshell - 1;  // the shell of primitive k
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (ax[mid].prim0 <= k)
      lo = mid;
    else
      hi = mid - 1;
  }
  eri_ket_matrix(ax[lo].l, ax_alpha[k], lane, M + (long long)k * kEriKetSize);
}
// A primitive's ket matrix into the warp's shared memory.
__device__ __forceinline__ void eri_load_ket(const double* __restrict__ Mg, int nsc, int lane,
                                             double* M) {
  for (int i = lane; i < nsc * kEriNKet; i += 32) M[i] = __ldg(Mg + i);
}

// E[axis][i][j][t] of one primitive pair, i <= la, j <= lb, t <= i + j, in
// a flat array with strides ((lb+1)*(la+lb+1), (la+lb+1), 1) per axis.
__device__ void eri_hermite_pair(int la, int lb, double p, const double* PA, const double* PB,
                                 double kab, double* E) {
  const int nt = la + lb + 1, sj = nt, si = (lb + 1) * nt, sax = (la + 1) * si;
  const double oo2p = 0.5 / p;
  for (int d = 0; d < 3; ++d) {
    double* e = E + d * sax;
    for (int i = 0; i < sax; ++i) e[i] = 0.0;
    e[0] = d == 0 ? kab : 1.0;
    for (int i = 0; i < la; ++i)
      for (int t = 0; t <= i + 1; ++t) {
        double v = PA[d] * e[i * si + t] + (t + 1 < nt ? (t + 1) * e[i * si + t + 1] : 0.0);
        if (t > 0) v += oo2p * e[i * si + t - 1];
        e[(i + 1) * si + t] = v;
      }
    for (int i = 0; i <= la; ++i)
      for (int j = 0; j < lb; ++j)
        for (int t = 0; t <= i + j + 1; ++t) {
          double v = PB[d] * e[i * si + j * sj + t] +
                     (t + 1 < nt ? (t + 1) * e[i * si + j * sj + t + 1] : 0.0);
          if (t > 0) v += oo2p * e[i * si + j * sj + t - 1];
          e[i * si + (j + 1) * sj + t] = v;
        }
  }
}

// Compile-time forms of eri_idx's inverse and of the cartesian order.
__host__ __device__ constexpr int eri_tuv_of(int e) {
  int n = 0;
  for (int sum = 0; sum <= kEriMaxL; ++sum)
    for (int r = 0; r <= sum; ++r)
      for (int v = 0; v <= r; ++v) {
        if (n == e) return (sum - r) | ((r - v) << 8) | (v << 16);
        ++n;
      }
  return 0;
}
__host__ __device__ constexpr int eri_cart_of(int l, int c) {
  int idx = 0;
  for (int ix = l; ix >= 0; --ix)
    for (int iy = l - ix; iy >= 0; --iy) {
      if (idx == c) return ix | (iy << 8) | ((l - ix - iy) << 16);
      ++idx;
    }
  return 0;
}
__host__ __device__ constexpr int eri_idx_c(int t, int u, int v) {
  return (t + u + v) * (t + u + v + 1) * (t + u + v + 2) / 6 + (u + v) * (u + v + 1) / 2 + v;
}

// An s-s AO shell pair against one auxiliary shell of angular momentum LC:
// the lanes take the bra primitive pairs (the work of an s-s pair is all in
// its primitives), each with its R table in registers; per auxiliary
// primitive the warp first builds the ket matrix M (shared memory), then
// W[mc] = pref sum_j M[mc][j] R[j].  The partial sums of the spherical
// auxiliary components end in acc of every lane (butterfly sum).  Same
// terms as the general path, summed in another order.
template <int LC>
__device__ void eri_ss_aux(const double* pp, int psz, int npp, const EriShell& c,
                           const double* __restrict__ ax_alpha,
                           const double* __restrict__ ax_coef, const double* __restrict__ Mg,
                           const double* __restrict__ tab, int lane, double* M, double* acc) {
  constexpr int NSC = 2 * LC + 1;
  constexpr int NR = (LC + 1) * (LC + 2) * (LC + 3) / 6;
  double part[NSC];
#pragma unroll
  for (int m = 0; m < NSC; ++m) part[m] = 0.0;
  for (int k = 0; k < c.nprim; ++k) {
    const double qq = ax_alpha[c.prim0 + k];
    const double cq = ax_coef[c.prim0 + k] / qq;
    __syncwarp();  // the previous primitive's M is no longer read
    eri_load_ket(Mg + (long long)(c.prim0 + k) * kEriKetSize, NSC, lane, M);
    __syncwarp();
    for (int q = lane; q < npp; q += 32) {
      const double* o = pp + q * psz;
      if (o[5] == 0.0) continue;
      const double p = o[0];
      // alpha = p q / (p + q), pref = 2 pi^{5/2} / (p q sqrt(p + q)) (o[4] holds
      // the bra's part)
      const double rs = rsqrt(p + qq);
      const double alpha = p * qq * (rs * rs);
      const double pref = o[4] * cq * rs;
      const double X = o[1] - c.A[0], Y = o[2] - c.A[1], Z = o[3] - c.A[2];
      double F[LC + 1];
      eri_boys(tab, LC, alpha * (X * X + Y * Y + Z * Z), F);
      double rn[LC + 1];
      double fac = 1.0;
#pragma unroll
      for (int n = 0; n <= LC; ++n) {
        rn[n] = fac * F[n];
        fac *= -2.0 * alpha;
      }
      // R^n_{tuv} level by level, n = LC .. 0
      double R[NR], Ro[NR];
      R[0] = rn[LC];
#pragma unroll
      for (int n = LC - 1; n >= 0; --n) {
#pragma unroll
        for (int e = 0; e < NR; ++e) Ro[e] = R[e];
#pragma unroll
        for (int e = 0; e < NR; ++e) {
          const int tuv = eri_tuv_of(e);
          const int t = tuv & 255, u = (tuv >> 8) & 255, v = tuv >> 16;
          if (t + u + v > LC - n) continue;
          double val;
          if (t > 0) {
            val = X * Ro[eri_idx_c(t - 1, u, v)];
            if (t > 1) val += (t - 1) * Ro[eri_idx_c(t - 2, u, v)];
          } else if (u > 0) {
            val = Y * Ro[eri_idx_c(t, u - 1, v)];
            if (u > 1) val += (u - 1) * Ro[eri_idx_c(t, u - 2, v)];
          } else if (v > 0) {
            val = Z * Ro[eri_idx_c(t, u, v - 1)];
            if (v > 1) val += (v - 1) * Ro[eri_idx_c(t, u, v - 2)];
          } else {
            val = rn[n];
          }
          R[e] = val;
        }
      }
      const double cf = o[6] * o[7] * o[8] * pref;  // E^{00} of the three axes
#pragma unroll
      for (int mc = 0; mc < NSC; ++mc) {
        double w = 0.0;
#pragma unroll
        for (int jj = 0; jj < NR; ++jj) w += M[mc * kEriNKet + jj] * R[jj];
        part[mc] += cf * w;
      }
    }
  }
#pragma unroll
  for (int mc = 0; mc < NSC; ++mc) {
    double v = part[mc];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    acc[mc] = v;
  }
}

// How lane e of an R level forms R^n[e] from level n + 1: coordinate (axis)
// times entry i1 plus fac times entry i2; packed i1 | i2 << 8 | axis << 16 |
// fac << 20 (e = 0 is the Boys value itself).
__device__ __forceinline__ int eri_r_step(int e) {
  const int tuv = c_eri_tuv[e];
  const int t = tuv & 255, u = (tuv >> 8) & 255, v = tuv >> 16;
  const int axis = t > 0 ? 0 : (u > 0 ? 1 : 2);
  const int n = axis == 0 ? t : (axis == 1 ? u : v);
  if (n == 0) return 0;
  const int i1 = eri_idx(t - (axis == 0), u - (axis == 1), v - (axis == 2));
  const int i2 = n > 1 ? eri_idx(t - 2 * (axis == 0), u - 2 * (axis == 1), v - 2 * (axis == 2)) : 0;
  return i1 | (i2 << 8) | (axis << 16) | ((n - 1) << 20);
}

// doubles of one bra primitive pair: p, P[3], coefficient, keep flag, E
__host__ __device__ constexpr int eri_pair_size(int la, int lb) {
  return 6 + 3 * (la + 1) * (lb + 1) * (la + lb + 1);
}
// FP64 warp instructions of a primitive pair of angular momentum Lb with a
// primitive of an auxiliary shell of lc, about: Boys values, R levels, W, and
// the results' share; what the work items are balanced by
inline double eri_cost(int la, int lb, int lc) {
  auto tet = [](int n) { return n * (n + 1) * (n + 2) / 6; };
  auto warps = [](int n) { return (n + 31) / 32; };
  const int L = la + lb + lc, nsc = 2 * lc + 1;
  double c = 4.0 + L;
  for (int l = 1; l <= L; ++l) c += 2 * warps(tet(l + 1));
  c += warps(tet(la + lb + 1) * nsc) * tet(lc + 1);
  c += warps((2 * la + 1) * (2 * lb + 1) * nsc) * tet(la + lb + 1);
  return c;
}
// doubles of its Hermite -> spherical (a, b) matrix (not for s-s pairs)
__host__ __device__ constexpr int eri_sph_size(int la, int lb) {
  return (2 * la + 1) * (2 * lb + 1) * ((la + lb + 1) * (la + lb + 2) * (la + lb + 3) / 6);
}
// primitive pairs whose matrices are held at a time (about 24 KB)
__host__ __device__ constexpr int eri_sph_chunk(int la, int lb, int npp) {
  const int fit = 3072 / eri_sph_size(la, lb);
  const int n = fit < 1 ? 1 : fit;
  return n < npp ? n : npp;
}

// One block per AO shell pair (a, b) and range of auxiliary blocks; its warps
// take the kept shells of the range in turn.  What bounds it is the FP64 pipe, where a warp instruction costs 16
// clocks however few lanes take part, so every phase spreads over the lanes:
//   Boys values   lanes over the (shell, primitive pair, primitive)
//                 combinations of up to 64 at once, several shells together
//   R levels      one entry per lane, one fma and one product each
//   W[e][mc]      lanes over (Hermite index e, spherical component mc)
//   (a, b)        lanes over (spherical pair, mc), against a matrix per
//                 primitive pair that folds E and both spherical transforms
// SS: the launch holds only s-s shell pairs (lanes over primitive pairs),
// else only the other pairs; two kernels with half the code each keep the
// instruction working set of a block small.  Six waters / jkfit: s-s 13.1 -> 4.2
// ms, the others 34.4 -> 8.4 ms against lanes over e and over cartesian pairs,
// and 2.6 and 3.7 ms with the work in even items.
template <bool SS>
__global__ void __launch_bounds__(32 * kEriWarps, 4)
    k_eri3c(const EriItem* __restrict__ items, const EriShell* __restrict__ ao,
            const EriShell* __restrict__ ax, const double* __restrict__ ao_alpha,
            const double* __restrict__ ao_coef, const double* __restrict__ ax_alpha,
            const double* __restrict__ ax_coef, const double* __restrict__ ket,
            const double* __restrict__ boys, const int* __restrict__ pair_I,
            const int* __restrict__ pair_J, const unsigned char* __restrict__ keep, int nablk,
            const int* __restrict__ ablk_shell_off, const int* __restrict__ blk_bf_off,
            const long long* __restrict__ panel_off, const int* __restrict__ panel_K,
            const int* __restrict__ col_IJ, const int* __restrict__ col_JI, int naux,
            double* __restrict__ B) {
  extern __shared__ double sm[];
  __shared__ unsigned char plus[kEriNW * kEriNKet];  // index of e + j (Hermite indices)
  __shared__ int list[kEriList];                     // kept auxiliary shells
  __shared__ int nlist, next_s;
  __shared__ double small[kEriMaxL];  // 0, 1, .. (a conversion is an FP64 instruction too)
  const EriItem it = items[blockIdx.x];
  const EriShell a = ao[it.a], b = ao[it.b];
  const int la = a.l, lb = b.l, Lb = la + lb;
  const int nsa = 2 * la + 1, nsb = 2 * lb + 1, nab = nsa * nsb;
  const int npp = a.nprim * b.nprim;
  const int psz = eri_pair_size(la, lb);
  const int nW = eri_tet(Lb + 1);  // bra Hermite indices
  const int qcs = SS ? npp : eri_sph_chunk(la, lb, npp);
  double* pp = sm;  // npp * psz
  double* Es = sm + npp * psz;
  double* wbase = Es + (SS ? 0 : qcs * nab * nW) + (threadIdx.x >> 5) * kEriWarpDoubles;
  double* R0 = wbase;
  double* R1 = wbase + kEriNR;
  double* W = wbase + 2 * kEriNR;
  double* rnq = W + kEriNW * kEriMaxSph;            // kEriRnChunk x (kEriMaxL + 1)
  double* Mk = rnq + kEriRnChunk * (kEriMaxL + 1);  // kEriMaxSph x kEriNKet
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  if (threadIdx.x < kEriMaxL) small[threadIdx.x] = threadIdx.x;
  // bra primitive pairs
  double ab2 = 0.0;
  for (int d = 0; d < 3; ++d) ab2 += (a.A[d] - b.A[d]) * (a.A[d] - b.A[d]);
  for (int q = threadIdx.x; q < npp; q += blockDim.x) {
    const int ia = q / b.nprim, ib = q % b.nprim;
    const double al = ao_alpha[a.prim0 + ia], be = ao_alpha[b.prim0 + ib];
    const double p = al + be;
    double P[3], PA[3], PB[3];
    for (int d = 0; d < 3; ++d) {
      P[d] = (al * a.A[d] + be * b.A[d]) / p;
      PA[d] = P[d] - a.A[d];
      PB[d] = P[d] - b.A[d];
    }
    const double kab = exp(-al * be / p * ab2);
    const double coef = ao_coef[a.prim0 + ia] * ao_coef[b.prim0 + ib];
    double* o = pp + q * psz;
    o[0] = p;
    o[1] = P[0];
    o[2] = P[1];
    o[3] = P[2];
    o[4] = 2.0 * 17.493418327624862 * coef / p;  // 2 pi^{5/2}
    if (SS) o[4] *= c_eri_sph[0] * c_eri_sph[0];  // both s functions' normalisation
    o[5] = fabs(coef * kab) < 1e-16 ? 0.0 : 1.0;
    eri_hermite_pair(la, lb, p, PA, PB, kab, o + 6);
  }
  if (!SS)
    for (int i = threadIdx.x; i < nW * kEriNKet; i += blockDim.x) {
      const int x = c_eri_tuv[i / kEriNKet], y = c_eri_tuv[i % kEriNKet];
      const int t = (x & 255) + (y & 255), u = ((x >> 8) & 255) + ((y >> 8) & 255),
                v = (x >> 16) + (y >> 16);
      plus[i] = t + u + v <= kEriMaxL ? (unsigned char)eri_idx(t, u, v) : 0;
    }
  __syncthreads();

  const int I = pair_I[it.p], J = pair_J[it.p];
  const int I0 = blk_bf_off[I], J0 = blk_bf_off[J];
  const int KI = panel_K[I], KJ = panel_K[J];
  double* const PI = B + panel_off[I];
  double* const PJ = B + panel_off[J];
  // one result (ma, mb, mc) of auxiliary shell c into the panels; add: the
  // part of a later chunk of primitive pairs (the same thread wrote the first)
  auto store = [&](int ma, int mb, int X, double v, bool add) {
    const int mu = a.bf_off + ma - I0, nu = b.bf_off + mb - J0;
    double* o1 = PI + ((long long)mu * naux + X) * KI + col_IJ[it.p] + nu;
    double* o2 = I != J ? PJ + ((long long)nu * naux + X) * KJ + col_JI[it.p] + mu
                        : (it.a != it.b ? PI + ((long long)nu * naux + X) * KI + col_IJ[it.p] + mu
                                        : nullptr);
    if (add) v += *o1;
    *o1 = v;
    if (o2) *o2 = v;
  };
  int rstep[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) rstep[i] = !SS && lane + 32 * i < kEriNR ? eri_r_step(lane + 32 * i) : 0;

  for (int qs0 = 0; qs0 < npp; qs0 += qcs) {
    const int qs1 = min(npp, qs0 + qcs);
    if constexpr (!SS) {
      // Es[q][ab][e] = sum_{ca, cb} sph_a sph_b E^x_t E^y_u E^z_v
      __syncthreads();
      const int nca = (la + 1) * (la + 2) / 2, ncb = (lb + 1) * (lb + 2) / 2;
      const int Eax = (la + 1) * (lb + 1) * (Lb + 1), Esi = (lb + 1) * (Lb + 1), Esj = Lb + 1;
      const double* sa = c_eri_sph + eri_sph_off(la);
      const double* sb = c_eri_sph + eri_sph_off(lb);
      for (int i = threadIdx.x; i < (qs1 - qs0) * nab * nW; i += blockDim.x) {
        const int e = i % nW, ab = (i / nW) % nab, q = qs0 + i / (nW * nab);
        const int ma = ab / nsb, mb = ab % nsb;
        const int tuv = c_eri_tuv[e];
        const int t = tuv & 255, u = (tuv >> 8) & 255, v = tuv >> 16;
        const double* E = pp + q * psz + 6;
        double sum = 0.0;
        for (int ca = 0; ca < nca; ++ca) {
          const double fa = sa[ma * nca + ca];
          if (fa == 0.0) continue;
          int ea[3];
          eri_cart(la, ca, ea);
          for (int cb = 0; cb < ncb; ++cb) {
            const double fb = sb[mb * ncb + cb];
            if (fb == 0.0) continue;
            int eb[3];
            eri_cart(lb, cb, eb);
            if (t > ea[0] + eb[0] || u > ea[1] + eb[1] || v > ea[2] + eb[2]) continue;
            sum += (fa * fb) * (E[ea[0] * Esi + eb[0] * Esj + t] *
                                E[Eax + ea[1] * Esi + eb[1] * Esj + u] *
                                E[2 * Eax + ea[2] * Esi + eb[2] * Esj + v]);
          }
        }
        Es[i] = sum;
      }
      __syncthreads();
    }
    // kept auxiliary shells, kEriList of them at a time
    const int s_end = ablk_shell_off[it.A1];
    if (threadIdx.x == 0) next_s = ablk_shell_off[it.A0];
    for (;;) {
      __syncthreads();
      if (warp == 0) {
        int n = 0, s = next_s;
        for (; s < s_end && n + 32 <= kEriList; s += 32) {
          bool in = s + lane < s_end;
          if (in) {
            const EriShell& c = ax[s + lane];
            in = (it.ls >> c.l & 1) && keep[(long long)it.p * nablk + c.blk];
          }
          const unsigned int m = __ballot_sync(0xffffffffu, in);
          if (in) list[n + __popc(m & ((1u << lane) - 1))] = s + lane;
          n += __popc(m);
        }
        if (lane == 0) {
          nlist = n;
          next_s = s;
        }
      }
      __syncthreads();
      if (nlist == 0 && next_s >= s_end) break;
      if constexpr (SS) {
        for (int i = warp; i < nlist; i += kEriWarps) {
          const EriShell c = ax[list[i]];
          double acc[kEriMaxSph];
          if (c.l == 0)
            eri_ss_aux<0>(pp, psz, npp, c, ax_alpha, ax_coef, ket, boys, lane, Mk, acc);
          else if (c.l == 1)
            eri_ss_aux<1>(pp, psz, npp, c, ax_alpha, ax_coef, ket, boys, lane, Mk, acc);
          else if (c.l == 2)
            eri_ss_aux<2>(pp, psz, npp, c, ax_alpha, ax_coef, ket, boys, lane, Mk, acc);
          else
            eri_ss_aux<3>(pp, psz, npp, c, ax_alpha, ax_coef, ket, boys, lane, Mk, acc);
          // every lane has the sums
          double v = acc[0];
#pragma unroll
          for (int m = 1; m < kEriMaxSph; ++m) v = lane == m && m < 2 * c.l + 1 ? acc[m] : v;
          if (lane < 2 * c.l + 1) store(0, 0, c.bf_off + lane, v, false);
        }
      } else {
        const double* Esq = Es - (long long)qs0 * nab * nW;
        for (int i0 = warp; i0 < nlist;) {
          // a batch of shells with the same contraction whose combinations fit
          // the Boys buffer (one shell, in pieces, if it has too many)
          const int nck = ax[list[i0]].nprim;
          const int per = (qs1 - qs0) * nck;  // combinations of a shell
          int nb = 1;
          while (nb < 32 && i0 + nb * kEriWarps < nlist && (nb + 1) * per <= kEriRnChunk &&
                 ax[list[i0 + nb * kEriWarps]].nprim == nck)
            ++nb;
          const int qch = max(1, min(qs1 - qs0, kEriRnChunk / nck));
          double acc[6];  // results (ab, mc): lane + 32 i
          for (int q0 = qs0; q0 < qs1; q0 += qch) {
            const int q1 = min(qs1, q0 + qch), nqk = (q1 - q0) * nck;
            __syncwarp();  // the Boys buffer is no longer read
            for (int jq = lane; jq < nb * nqk; jq += 32) {
              const int sh = jq / nqk, r0 = jq - sh * nqk;
              const int q = q0 + r0 / nck, k = r0 % nck;
              const double* o = pp + q * psz;
              if (o[5] == 0.0) continue;
              const EriShell& c = ax[list[i0 + sh * kEriWarps]];
              const int L = Lb + c.l;
              const double p = o[0], qq = ax_alpha[c.prim0 + k];
              const double rs = rsqrt(p + qq);
              const double alpha = p * qq * (rs * rs);
              const double X = o[1] - c.A[0], Y = o[2] - c.A[1], Z = o[3] - c.A[2];
              double F[kEriMaxL + 1];
              eri_boys(boys, L, alpha * (X * X + Y * Y + Z * Z), F);
              double fac = o[4] * (ax_coef[c.prim0 + k] / qq) * rs;  // the prefactor rides along
              double* r = rnq + jq * (kEriMaxL + 1);
              for (int n = 0; n <= L; ++n) {
                r[n] = fac * F[n];
                fac *= -2.0 * alpha;
              }
            }
            __syncwarp();
            for (int sh = 0; sh < nb; ++sh) {
              const EriShell c = ax[list[i0 + sh * kEriWarps]];
              const int lc = c.l, nsc = 2 * lc + 1, L = Lb + lc, nr = eri_tet(lc + 1);
              const int nw = nW * nsc, no = nab * nsc;
              // this lane's W entries (e, mc) and results (ab, mc)
              int wid[8], oid[6];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int id = lane + 32 * i, e = id / nsc;
                wid[i] = id < nw ? (e * kEriNKet) | ((id - e * nsc) * kEriNKet) << 16 : 0;
              }
#pragma unroll
              for (int i = 0; i < 6; ++i) {
                const int id = lane + 32 * i, ab = id / nsc;
                oid[i] = id < no ? (ab * nW) | (id - ab * nsc) << 16 : 0;
              }
              if (q0 == qs0)
#pragma unroll
                for (int i = 0; i < 6; ++i) acc[i] = 0.0;
              if (nck == 1) {
                eri_load_ket(ket + (long long)c.prim0 * kEriKetSize, nsc, lane, Mk);
                __syncwarp();
              }
              for (int q = q0; q < q1; ++q) {
                const double* o = pp + q * psz;
                if (o[5] == 0.0) continue;
                const double X = o[1] - c.A[0], Y = o[2] - c.A[1], Z = o[3] - c.A[2];
                double w[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) w[i] = 0.0;
                for (int k = 0; k < nck; ++k) {
                  const double* rn = rnq + (sh * nqk + (q - q0) * nck + k) * (kEriMaxL + 1);
                  // R^n_{tuv}, levels n = L .. 0; level 0 ends in cur
                  double* cur = (L & 1) ? R1 : R0;
                  double* old = (L & 1) ? R0 : R1;
                  if (lane == 0) cur[0] = rn[L];
                  if (nck > 1)
                    eri_load_ket(ket + (long long)(c.prim0 + k) * kEriKetSize, nsc, lane, Mk);
                  __syncwarp();
                  for (int n = L - 1; n >= 0; --n) {
                    double* t_ = cur;
                    cur = old;
                    old = t_;
                    const int cnt = eri_tet(L - n + 1);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                      const int e = lane + 32 * i;
                      if (32 * i >= cnt) break;
                      if (e < cnt) {
                        const int st = rstep[i];
                        const int ax_ = (st >> 16) & 3;
                        const double x = ax_ == 0 ? X : (ax_ == 1 ? Y : Z);
                        const double val =
                            fma(small[st >> 20], old[(st >> 8) & 255], x * old[st & 255]);
                        cur[e] = e == 0 ? rn[n] : val;
                      }
                    }
                    __syncwarp();
                  }
                  // W[e][mc] += sum_j M[mc][j] R[e + j]
                  for (int jj = 0; jj < nr; ++jj)
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                      if (32 * i >= nw) break;
                      w[i] = fma(Mk[(wid[i] >> 16) + jj], cur[plus[(wid[i] & 0xFFFF) + jj]], w[i]);
                    }
                  __syncwarp();  // R and M are rewritten by the next primitive
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
                  if (lane + 32 * i < nw) W[lane + 32 * i] = w[i];
                __syncwarp();
                const double* Eq = Esq + (long long)q * nab * nW;
                for (int e = 0; e < nW; ++e)
#pragma unroll
                  for (int i = 0; i < 6; ++i) {
                    if (32 * i >= no) break;
                    acc[i] = fma(Eq[(oid[i] & 0xFFFF) + e], W[e * nsc + (oid[i] >> 16)], acc[i]);
                  }
                __syncwarp();
              }
              if (q1 == qs1) {
#pragma unroll
                for (int i = 0; i < 6; ++i) {
                  const int id = lane + 32 * i;
                  if (id >= no) break;
                  const int ab = id / nsc, ma = ab / nsb;
                  store(ma, ab - ma * nsb, c.bf_off + id - ab * nsc, acc[i], qs0 > 0);
                }
              }
            }
          }
          i0 += nb * kEriWarps;
        }
      }
    }
  }
}

}  // namespace gbjk
