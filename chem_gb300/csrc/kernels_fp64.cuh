// FP64 kernels of the DF J/K build (the plain path).
//
// The 3-center tensor lives in atom-block panels (see gbjk.h):
//   panel I = [b_I][naux][K_I] FP64 at B + panel_off[I].
// Every kernel is deterministic: each output element is produced by exactly
// one thread (or one warp) with a fixed summation order, and cross-block
// sums go through partial buffers reduced in a fixed order.
#pragma once
#include "common.cuh"

namespace gbjk {

// Ordered sum of the split-K partials of one output, eight loads in flight
// (one at a time, small matrices spend the whole launch on load latency).
__device__ __forceinline__ double splitk_sum(const double* __restrict__ p, int nsplit,
                                             long long stride) {
  double s = 0.0;
  int k = 0;
  for (; k + 8 <= nsplit; k += 8) {
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = p[(long long)(k + j) * stride];
#pragma unroll
    for (int j = 0; j < 8; ++j) s += v[j];
  }
  for (; k < nsplit; ++k) s += p[(long long)k * stride];
  return s;
}

// Pg[pg_off[I] + m*K_I + k] = P[(boff[I]+m)*ld + colmap[cmoff[I]+k]]
// grid: (ceil(maxK/128), nbf); block 128.
__global__ void k_gather_panel_rows(const double* __restrict__ P, int ld,
                                    const int* __restrict__ blk_of, const int* __restrict__ boff,
                                    const int* __restrict__ panel_K,
                                    const long long* __restrict__ pg_off,
                                    const int* __restrict__ cmoff, const int* __restrict__ colmap,
                                    double* __restrict__ Pg) {
  const int mu = blockIdx.y;
  const int I = blk_of[mu];
  const int m = mu - boff[I];
  const int KI = panel_K[I];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= KI) return;
  Pg[pg_off[I] + (long long)m * KI + k] = P[(long long)mu * ld + colmap[cmoff[I] + k]];
}

// Cg[r*n + i] = C[colmap[r]*n + i] for all panel columns r.
__global__ void k_gather_cols(const double* __restrict__ Cm, int n, const int* __restrict__ colmap,
                              int nrows, double* __restrict__ Cg) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)nrows * n;
  if (idx >= total) return;
  const int r = (int)(idx / n), i = (int)(idx % n);
  Cg[idx] = Cm[(long long)colmap[r] * n + i];
}

// Cg[r*n + i] = Ct[i*ld + colmap[r]]: the same from the transposed matrix.
__global__ void k_gather_cols_t(const double* __restrict__ Ct, int n, int ld,
                                const int* __restrict__ colmap, int nrows,
                                double* __restrict__ Cg) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)nrows * n) return;
  const int r = (int)(idx / n), i = (int)(idx % n);
  Cg[idx] = Ct[(long long)i * ld + colmap[r]];
}

// part[mu][X] = sum_k B_I[m][X][k] * Pg_I[m][k]; one warp per (mu, X) row.
__global__ void k_j_rowdot(const double* __restrict__ B, const long long* __restrict__ panel_off,
                           const int* __restrict__ blk_of, const int* __restrict__ boff,
                           const int* __restrict__ panel_K, const long long* __restrict__ pg_off,
                           const double* __restrict__ Pg, int nbf, int naux,
                           double* __restrict__ part) {
  const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= (long long)nbf * naux) return;
  const int mu = (int)(row / naux), X = (int)(row % naux);
  const int I = blk_of[mu];
  const int m = mu - boff[I];
  const int KI = panel_K[I];
  const double* br = B + panel_off[I] + ((long long)m * naux + X) * KI;
  const double* pr = Pg + pg_off[I] + (long long)m * KI;
  double s = 0.0;
  for (int k = lane; k < KI; k += 32) s = fma(br[k], pr[k], s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) part[(long long)mu * naux + X] = s;
}

// g[X] = sum_{mu} part[mu][X], in increasing mu.  One thread per X, so the
// sum is a serial chain; what bounds it is the latency of its loads, hence
// sixteen of them in flight and one-warp blocks that spread over the SMs.
__global__ void k_reduce_rows(const double* __restrict__ part, int nrows, int ncols,
                              double* __restrict__ g) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x;
  if (X >= ncols) return;
  const double* p = part + X;
  double s = 0.0;
  int r = 0;
  for (; r + 16 <= nrows; r += 16) {
    double v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = p[(long long)(r + j) * ncols];
#pragma unroll
    for (int j = 0; j < 16; ++j) s += v[j];
  }
  for (; r < nrows; ++r) s += p[(long long)r * ncols];
  g[X] = s;
}

// g[X] = sum_{mu} part[mu][X] for the mixed path: warp w of a block sums
// the rows w, w + 16, ... in order (four loads in flight), then the sixteen
// partial sums are added in warp order.  A fixed order, coalesced row reads,
// and sixteen times the parallelism of one thread per column.
__global__ void __launch_bounds__(512)
    k_reduce_rows16(const double* __restrict__ part, int nrows, int ncols,
                    double* __restrict__ g) {
  __shared__ double ps[16][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int X = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (X < ncols) {
    int r = w;
    for (; r + 48 < nrows; r += 64) {
      const double a0 = part[(long long)r * ncols + X];
      const double a1 = part[(long long)(r + 16) * ncols + X];
      const double a2 = part[(long long)(r + 32) * ncols + X];
      const double a3 = part[(long long)(r + 48) * ncols + X];
      s += a0;
      s += a1;
      s += a2;
      s += a3;
    }
    for (; r < nrows; r += 16) s += part[(long long)r * ncols + X];
  }
  ps[w][lane] = s;
  __syncthreads();
  if (w == 0 && X < ncols) {
    double t = ps[0][lane];
    for (int i = 1; i < 16; ++i) t += ps[i][lane];
    g[X] = t;
  }
}

// y = M x, M n x n row-major; one warp per row.
__global__ void k_gemv(const double* __restrict__ M, const double* __restrict__ x, int n,
                       double* __restrict__ y) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  const double* mr = M + (long long)row * n;
  double s = 0.0;
  for (int k = lane; k < n; k += 32) s = fma(mr[k], x[k], s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) y[row] = s;
}

// y = L^T x for lower-triangular L (n x n row-major): y[X] = sum_{Y >= X}
// L[Y][X] x[Y], one thread per X, in increasing Y.  A serial chain of up to n
// fmas per thread, so its loads are what can be hidden: a warp walks the rows
// from its first X on, sixteen rows' coalesced loads before their fmas, and a
// thread skips the rows above its own.
__global__ void k_gemv_lower_t(const double* __restrict__ L, const double* __restrict__ x, int n,
                               double* __restrict__ y) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x;
  const int Xc = min(X, n - 1);
  double s = 0.0;
  int Y = X & ~31;
  for (; Y + 16 <= n; Y += 16) {
    double v[16], w[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      v[j] = L[(long long)(Y + j) * n + Xc];
      w[j] = x[Y + j];
    }
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (Y + j >= X) s = fma(v[j], w[j], s);
  }
  for (; Y < n; ++Y)
    if (Y >= X) s = fma(L[(long long)Y * n + Xc], x[Y], s);
  if (X < n) y[X] = s;
}

// J[mu][colmap[k]] = sum_X B_I[m][X][k] h[X]; grid (ceil(maxK/32), nbf),
// block 128.  Each output is (s0 + s1) + (s2 + s3), s_a the in-order sum over
// X = a mod 4 below 4 floor(naux / 4) and the last naux mod 4 terms in s0.
// Warp a of a block forms s_a of 32 columns: four times the loads in flight
// of one thread per output, which is what bounds small tensors.
__global__ void __launch_bounds__(128)
    k_j_colsum(const double* __restrict__ B, const long long* __restrict__ panel_off,
               const int* __restrict__ blk_of, const int* __restrict__ boff,
               const int* __restrict__ panel_K, const int* __restrict__ cmoff,
               const int* __restrict__ colmap, const double* __restrict__ h, int nbf, int naux,
               double* __restrict__ J) {
  __shared__ double ps[4][32];
  const int mu = blockIdx.y;
  const int I = blk_of[mu];
  const int m = mu - boff[I];
  const int KI = panel_K[I];
  if (blockIdx.x * 32 >= KI) return;
  const int lane = threadIdx.x & 31, a = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (k < KI) {
    const double* b = B + panel_off[I] + (long long)m * naux * KI + k;
    const int n4 = naux & ~3;
    int X = a;
    for (; X + 28 < n4; X += 32) {
      double v[8], w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[j] = __ldg(b + (long long)(X + 4 * j) * KI);
        w[j] = __ldg(h + X + 4 * j);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) s = fma(v[j], w[j], s);
    }
    {
      // up to seven more, loaded together
      double v[8], w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const bool in = X + 4 * j < n4;
        v[j] = in ? __ldg(b + (long long)(X + 4 * j) * KI) : 0.0;
        w[j] = in ? __ldg(h + X + 4 * j) : 0.0;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (X + 4 * j < n4) s = fma(v[j], w[j], s);
    }
    if (a == 0)
      for (int Xt = n4; Xt < naux; ++Xt) s = fma(b[(long long)Xt * KI], h[Xt], s);
  }
  ps[a][lane] = s;
  __syncthreads();
  if (a == 0 && k < KI)
    J[(long long)mu * nbf + colmap[cmoff[I] + k]] =
        (ps[0][lane] + ps[1][lane]) + (ps[2][lane] + ps[3][lane]);
}

// x as hi + lo, two FP32 values built from the FP64 bit pattern with
// integer operations (no FP64 instruction): hi = the top 24 significand bits
// (truncated), lo = the remaining 29 bits rounded to FP32.  |x| < 2^-126
// gives (0, 0) and a lo below FP32's normal range gives lo = 0; both are
// below 2^-100 relative to the O(1) sums they enter.
__device__ __forceinline__ void f64_split_f32(double x, float& hi, float& lo) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const int E = (int)((u >> 52) & 0x7FF);
  const unsigned int sgn = (unsigned int)(u >> 32) & 0x80000000u;
  const int ef = E - 896;  // FP32 biased exponent of hi (E - 1023 + 127)
  if (ef < 1 || ef > 254) {
    hi = 0.f;
    lo = 0.f;
    return;
  }
  hi = __uint_as_float(sgn | ((unsigned int)ef << 23) | (unsigned int)((u >> 29) & 0x7FFFFF));
  // lo = m29 * 2^(E - 1075): the scale 2^(E-1075) as an FP32 bit pattern
  const int es = E - 1075 + 127;
  if (es < 1) {
    lo = 0.f;
    return;
  }
  const float m29 = (float)(unsigned int)(u & 0x1FFFFFFFu);
  lo = __uint_as_float(sgn | ((unsigned int)es << 23)) * m29;
}

// Compact copy of the prefitted tensor for the mixed-path J: element x as
// hi = its sign, exponent and top 24 significand bits (FP32; 0 outside the
// FP32 normal range) and lo = the next 29 bits rounded to 16
// (lo16 = min(rint(m29 / 2^13), 65535)), so x = hi + lo16 2^(E-1062) to
// about 40 significant bits in 6 bytes.  The copy holds the columns [k0, K_I)
// of each panel: all of them, or, for a tensor whose two copies of every
// off-diagonal block pair agree bit for bit, those of the blocks J >= I.
// Panel I is [naux][cp]: row X holds the ncol = b_I (K_I - k0) values (m, k)
// side by side, padded with zeros to a multiple of 8, in two planes (hi FP32,
// lo16), so that four consecutive values are one 16-byte and one 8-byte load
// and a warp's 128 values lie in one row whatever the block sizes are.
struct JPanel {
  long long off;   // first element in the two planes
  long long gcol;  // first column among all panels' columns
  int cp, ncol;    // row stride, columns
  int k0;          // first panel column
};
// grid (naux, nblk), block 128.
__global__ void k_encode_f32i16(const double* __restrict__ B, const long long* __restrict__ panel_off,
                                const JPanel* __restrict__ jp, const int* __restrict__ panel_K,
                                int naux, float* __restrict__ hi, uint16_t* __restrict__ lo) {
  const int X = blockIdx.x, I = blockIdx.y;
  const JPanel p = jp[I];
  const int KI = panel_K[I], ks = KI - p.k0;
  const double* src = B + panel_off[I] + (long long)X * KI + p.k0;
  const long long d = p.off + (long long)X * p.cp;
  for (int c = threadIdx.x; c < p.cp; c += blockDim.x) {
    float h = 0.f;
    unsigned int l = 0;
    if (c < p.ncol) {
      const int m = c / ks, k = c - m * ks;
      const unsigned long long u =
          (unsigned long long)__double_as_longlong(src[(long long)m * naux * KI + k]);
      const int E = (int)((u >> 52) & 0x7FF);
      const unsigned int sgn = (unsigned int)(u >> 32) & 0x80000000u;
      const int ef = E - 896;
      if (ef >= 1 && ef <= 254) {
        h = __uint_as_float(sgn | ((unsigned int)ef << 23) | (unsigned int)((u >> 29) & 0x7FFFFF));
        l = min(((unsigned int)(u & 0x1FFFFFFFu) + 4096u) >> 13, 65535u);
      }
    }
    hi[d + c] = h;
    lo[d + c] = (uint16_t)l;
  }
}

// Whether the two copies of every off-diagonal block pair (I, J), I < J, hold
// the same bits: (m, X, kIJ + n) of panel I and (n, X, kJI + m) of panel J.
// A difference sets *flag.  grid (npairs, ceil(naux / 64)), block 128.
struct SymPair {
  long long offI, offJ;
  int KI, KJ, kIJ, kJI, bI, bJ;
};
__global__ void k_check_symmetric(const double* __restrict__ B, const SymPair* __restrict__ pairs,
                                  int naux, int* __restrict__ flag) {
  const SymPair p = pairs[blockIdx.x];
  const int x0 = blockIdx.y * 64, x1 = min(naux, x0 + 64);
  const int nn = p.bI * p.bJ;
  bool differ = false;
  for (int e = threadIdx.x; e < nn; e += blockDim.x) {
    const int m = e / p.bJ, n = e - m * p.bJ;
    const double* a = B + p.offI + (long long)m * naux * p.KI + p.kIJ + n;
    const double* b = B + p.offJ + (long long)n * naux * p.KJ + p.kJI + m;
    for (int X = x0; X < x1; ++X)
      differ |= __double_as_longlong(a[(long long)X * p.KI]) !=
                __double_as_longlong(b[(long long)X * p.KJ]);
  }
  if (differ) *flag = 1;
}

// The pair (hi, lo) of a compact element as FP32 values: lo = lo16 *
// 2^(ef - 39 - 127) with hi's sign (0 when that scale leaves the normal range).
__device__ __forceinline__ float f32i16_lo(float hi, unsigned int lo16) {
  const unsigned int b = __float_as_uint(hi);
  const int es = (int)((b >> 23) & 0xFF) - 39;
  const float sc = __uint_as_float((b & 0x80000000u) | ((unsigned int)max(es, 0) << 23));
  return es >= 1 ? sc * (float)lo16 : 0.f;
}

// Mixed-path J columns: J_c = sum_X B[X][c] h[X] over the columns c of the
// compact copy (6 bytes per element), with the products and the sum in
// FP32 pairs (hi/lo operands, exact product error by fma, TwoSum
// accumulation), so no FP64 arithmetic runs in the loop and the pass is
// bound by HBM rather than by GB300's FP64 rate.  The auxiliary range is cut
// into chunks of xchunk rows (blockIdx.y); chunk z writes its partial column
// sums to part[z * ncols + column] and k_j_colsum_chunks adds the chunks in
// order.  Block x takes the 128 columns from blk[x].y of panel blk[x].x, lane
// t the columns 4 t .. 4 t + 3.  C20H42: 0.188 ms, 6.0 TB/s, for the upper
// triangle (0.437 ms over the whole tensor in rows of one AO function).
// grid (nblkcol, nchunk), block 32, dynamic smem xchunk float2.
__global__ void __launch_bounds__(32)
    k_j_colsum_f32i16(const float* __restrict__ Bhi, const uint16_t* __restrict__ Blo,
                      const JPanel* __restrict__ jp, const int2* __restrict__ blk,
                      const double* __restrict__ h, int naux, int xchunk, long long ncols,
                      double* __restrict__ part) {
  extern __shared__ float2 h2[];
  const int x0 = blockIdx.y * xchunk;
  const int nx = min(xchunk, naux - x0);
  for (int x = threadIdx.x; x < nx; x += blockDim.x) {
    float a, b;
    f64_split_f32(h[x0 + x], a, b);
    h2[x] = make_float2(a, b);
  }
  __syncthreads();
  const int2 bk = blk[blockIdx.x];
  const JPanel p = jp[bk.x];
  const int k0 = bk.y + 4 * threadIdx.x;
  if (k0 >= p.cp) return;
  const long long off = p.off + (long long)x0 * p.cp + k0;
  const float4* bh = reinterpret_cast<const float4*>(Bhi + off);
  const uint2* bl = reinterpret_cast<const uint2*>(Blo + off);
  const int st4 = p.cp / 4;  // row stride in float4 / uint2 units
  float sh[4] = {0.f, 0.f, 0.f, 0.f}, sl[4] = {0.f, 0.f, 0.f, 0.f}, se[4] = {0.f, 0.f, 0.f, 0.f};
  auto acc = [](float b_h, float b_l, float2 hh, float& s_h, float& s_l, float& s_e) {
    const float p = __fmul_rn(b_h, hh.x);
    float e = fmaf(b_h, hh.x, -p);
    e = fmaf(b_h, hh.y, e);
    e = fmaf(b_l, hh.x, e);
    const float t = __fadd_rn(s_h, p);
    const float z = __fsub_rn(t, s_h);
    s_l = __fadd_rn(s_l, __fadd_rn(__fsub_rn(s_h, __fsub_rn(t, z)), __fsub_rn(p, z)));
    s_h = t;
    s_e = __fadd_rn(s_e, e);
  };
  auto row = [&](const float4 v, const uint2 w, float2 hh) {
    acc(v.x, f32i16_lo(v.x, w.x & 0xFFFFu), hh, sh[0], sl[0], se[0]);
    acc(v.y, f32i16_lo(v.y, w.x >> 16), hh, sh[1], sl[1], se[1]);
    acc(v.z, f32i16_lo(v.z, w.y & 0xFFFFu), hh, sh[2], sl[2], se[2]);
    acc(v.w, f32i16_lo(v.w, w.y >> 16), hh, sh[3], sl[3], se[3]);
  };
  // software-pipelined: the next eight rows (192 bytes per thread) are
  // loaded before the current eight are summed, so sixteen rows are in
  // flight (a plain unrolled loop of eight kept only a few: 0.55 ms against
  // 0.45 ms on n-C20H42)
  int X = 0;
  if (nx >= 8) {
    float4 v[8];
    uint2 w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = __ldg(bh + (long long)j * st4);
      w[j] = __ldg(bl + (long long)j * st4);
    }
    for (; X + 15 < nx; X += 8) {
      float4 vn[8];
      uint2 wn[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        vn[j] = __ldg(bh + (long long)(X + 8 + j) * st4);
        wn[j] = __ldg(bl + (long long)(X + 8 + j) * st4);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) row(v[j], w[j], h2[X + j]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[j] = vn[j];
        w[j] = wn[j];
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) row(v[j], w[j], h2[X + j]);
    X += 8;
  }
  for (; X < nx; ++X) row(__ldg(bh + (long long)X * st4), __ldg(bl + (long long)X * st4), h2[X]);
  double v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = (double)sh[j] + ((double)sl[j] + (double)se[j]);
  double2* out = reinterpret_cast<double2*>(part + (long long)blockIdx.y * ncols + p.gcol + k0);
  out[0] = make_double2(v[0], v[1]);
  out[1] = make_double2(v[2], v[3]);
}

// J[mu][nu] = sum over chunks (in order) of part[z][c], (mu, nu) = map[c];
// nu < 0: nu = ~nu and the column stands for (nu, mu) too.  mu < 0: padding.
__global__ void k_j_colsum_chunks(const double* __restrict__ part, int nchunk, long long ncols,
                                  int nbf, const int2* __restrict__ map, double* __restrict__ J) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncols) return;
  const int2 mn = map[c];
  if (mn.x < 0) return;
  const double s = splitk_sum(part + c, nchunk, ncols);
  const int nu = mn.y < 0 ? ~mn.y : mn.y;
  J[(long long)mn.x * nbf + nu] = s;
  if (mn.y < 0) J[(long long)nu * nbf + mn.x] = s;
}

// Dense expansion of the panel array: D[mu][X][colmap(k)] = P_I[m][X][k]
// (mu = boff[I] + m); entries outside the kept pattern are not written.
// grid (ceil(maxK/128), naux, nbf).
__global__ void k_expand_panels(const double* __restrict__ P, const long long* __restrict__ panel_off,
                                const int* __restrict__ blk_of, const int* __restrict__ boff,
                                const int* __restrict__ panel_K, const int* __restrict__ cmoff,
                                const int* __restrict__ colmap, int nbf, int naux,
                                double* __restrict__ D) {
  const int mu = blockIdx.z, X = blockIdx.y;
  const int I = blk_of[mu];
  const int KI = panel_K[I];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= KI) return;
  const int m = mu - boff[I];
  D[((long long)mu * naux + X) * nbf + colmap[cmoff[I] + k]] =
      P[panel_off[I] + ((long long)m * naux + X) * KI + k];
}

// The same expansion in the column-pair-outermost order of a split half
// transform (rows of rs values, ld columns): D[mu * rs + (X / 32) * 32 ld +
// (c / 2) * 64 + (X % 32) * 2 + c % 2], c = colmap(k).
__global__ void k_expand_panels_perm(const double* __restrict__ P,
                                     const long long* __restrict__ panel_off,
                                     const int* __restrict__ blk_of, const int* __restrict__ boff,
                                     const int* __restrict__ panel_K,
                                     const int* __restrict__ cmoff, const int* __restrict__ colmap,
                                     int naux, int ld, long long rs, double* __restrict__ D) {
  const int mu = blockIdx.z, X = blockIdx.y;
  const int I = blk_of[mu];
  const int KI = panel_K[I];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= KI) return;
  const int m = mu - boff[I], c = colmap[cmoff[I] + k];
  D[(long long)mu * rs + (long long)(X >> 5) * 32 * ld + (long long)(c >> 1) * 64 + (X & 31) * 2 +
    (c & 1)] = P[panel_off[I] + ((long long)m * naux + X) * KI + k];
}

// Grouped FP64 GEMM over a tile list; 64 x TN tiles (TN = 64, 32 or 16),
// 16 * TN / 4 threads, 4x4 outputs per thread.  Every output is one in-order
// fma chain over its k range, whatever the tile shape.
// TRANSA: A is stored K x M row-major, op(A)(m, k) = A[k * lda + m].
// Bound by the FP64 pipe (about two fmas per clock and SM), so fmas of
// outputs nobody reads are what it can save: thread (ty, tx) holds rows
// ty + 16 r and columns tx + TN/4 c, and the 16 x TN/4 patches (r, c) that
// lie outside the matrix, below the diagonal of an upper-triangle tile
// (kUpperC) or beyond the diagonal of a lower-triangular A are skipped.
template <bool TRANSB, bool TRANSA = false, int TN = 64>
__global__ void __launch_bounds__(TN * 4)
    k_gemm_fp64(const GemmGroup* __restrict__ groups, const GemmTile* __restrict__ tiles,
                double alpha) {
  static_assert(TN == 64 || TN == 32 || TN == 16, "tile width");
  constexpr int NT = TN * 4;   // threads
  constexpr int CW = TN / 4;   // thread columns
  __shared__ double As[16][65];
  __shared__ double Bs[16][TN + 1];
  const GemmTile t = tiles[blockIdx.x];
  const GemmGroup g = groups[t.group];
  const int tid = threadIdx.x;
  const int tx = tid % CW, ty = tid / CW;
  const int m0 = t.mt * 64, n0 = t.nt * TN;
  int kend = t.k1;
  if ((g.flags & kLowerA) && kend > m0 + 64) kend = m0 + 64;  // A[m][k] = 0 for k > m
  // active patches: bit 4 r + c
  unsigned int act = 0;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const bool in = m0 + 16 * r < g.M && n0 + CW * c < g.N;
      const bool below = (g.flags & kUpperC) && m0 + 16 * r > n0 + CW * c + CW - 1;
      if (in && !below) act |= 1u << (4 * r + c);
    }
  double acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.0;
  for (int k0 = t.k0; k0 < kend; k0 += 16) {
#pragma unroll
    for (int r = 0; r < 1024 / NT; ++r) {
      const int idx = tid + NT * r;
      if (TRANSA) {
        const int kk = idx >> 6, row = idx & 63;
        const int gm = m0 + row, gk = k0 + kk;
        As[kk][row] = (gm < g.M && gk < kend) ? g.A[(long long)gk * g.lda + gm] : 0.0;
      } else {
        const int row = idx >> 4, kk = idx & 15;
        const int gm = m0 + row, gk = k0 + kk;
        As[kk][row] = (gm < g.M && gk < kend) ? g.A[(long long)gm * g.lda + gk] : 0.0;
      }
    }
#pragma unroll
    for (int r = 0; r < (16 * TN) / NT; ++r) {
      const int idx = tid + NT * r;
      if (TRANSB) {
        const int col = idx >> 4, kk = idx & 15;
        const int gn = n0 + col, gk = k0 + kk;
        Bs[kk][col] = (gn < g.N && gk < kend) ? g.B[(long long)gn * g.ldb + gk] : 0.0;
      } else {
        const int kk = idx / TN, col = idx % TN;
        const int gn = n0 + col, gk = k0 + kk;
        Bs[kk][col] = (gn < g.N && gk < kend) ? g.B[(long long)gk * g.ldb + gn] : 0.0;
      }
    }
    __syncthreads();
    // a lower-triangular A has no terms for the rows that end before k0
    const unsigned int on =
        (g.flags & kLowerA) && k0 >= m0 + 16 ? act & (0xFFFFu << (4 * ((k0 - m0) >> 4))) : act;
    if (on == 0xFFFFu) {
#pragma unroll
      for (int kk = 0; kk < 16; ++kk) {
        double a[4], b[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) a[r] = As[kk][ty + 16 * r];
#pragma unroll
        for (int c = 0; c < 4; ++c) b[c] = Bs[kk][tx + CW * c];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
      }
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (!((on >> (4 * r + c)) & 1)) continue;
          double s = acc[r][c];
#pragma unroll
          for (int kk = 0; kk < 16; ++kk) s = fma(As[kk][ty + 16 * r], Bs[kk][tx + CW * c], s);
          acc[r][c] = s;
        }
    }
    __syncthreads();
  }
  double* C = g.C + t.coff;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int gm = m0 + ty + 16 * r;
    if (gm >= g.M) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int gn = n0 + tx + CW * c;
      if (gn >= g.N || !((act >> (4 * r + c)) & 1)) continue;
      double v = alpha * acc[r][c];
      if (g.flags & kAccum) v += C[(long long)gm * g.ldc + gn];
      C[(long long)gm * g.ldc + gn] = v;
    }
  }
}

// 16 x 16 tiles, one thread per output, each output the in-order fma chain over
// the tile's k range.  A lower-triangular A stops at k = m: the terms beyond
// are exact zeros, so every nonzero result equals the tiled kernel's bit for
// bit.  For the exchange and the SCF's square products, whose tiles follow the
// diagonal and the edge closest (FP64 pipe), and for half transforms and fits so
// small that 64-row tiles would be mostly padding and the few tiles would leave
// most SMs' FP64 units idle.  The latter are bound by latency: 64 k of both operands are staged in shared memory at a
// time, the next 64 in registers meanwhile, so the chain waits for memory
// once per tile and not once per eight k.  The threads take the outputs that
// the matrix has, in row order: an FP64 instruction of a warp costs 16 clocks
// however few lanes it has, and five columns are three warps' work and not eight
// (the half transform of one water molecule 6.8 -> 5.2 us; its fit 18.3 -> 9.1,
// with the long tiles first).
template <bool TRANSB>
__global__ void __launch_bounds__(256)
    k_gemm_fp64_elem(const GemmGroup* __restrict__ groups, const GemmTile* __restrict__ tiles,
                     double alpha) {
  constexpr int KC = 64;
  __shared__ double As[16][KC + 1];
  __shared__ double Bs[KC][17];
  const GemmTile t = tiles[blockIdx.x];
  const GemmGroup g = groups[t.group];
  const int tid = threadIdx.x;
  const int m0 = t.mt * 16, n0 = t.nt * 16;
  const int nc = min(16, g.N - n0);
  const bool used = tid < nc * min(16, g.M - m0);
  const int ty = used ? tid / nc : 0, tx = used ? tid - ty * nc : 0;
  const int gm = m0 + ty, gn = n0 + tx;
  int kblk = t.k1;  // end of the tile's k range, and of this row's
  if ((g.flags & kLowerA) && kblk > m0 + 16) kblk = m0 + 16;
  const int kend = !used ? t.k0 : (g.flags & kLowerA) ? min(kblk, gm + 1) : kblk;
  double ra[4], rb[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int idx = tid + 256 * j;
      const int row = idx >> 6, ka = k0 + (idx & 63);
      ra[j] = (m0 + row < g.M && ka < kblk) ? g.A[(long long)(m0 + row) * g.lda + ka] : 0.0;
      if (TRANSB) {
        rb[j] = (n0 + row < g.N && ka < kblk) ? g.B[(long long)(n0 + row) * g.ldb + ka] : 0.0;
      } else {
        const int kb = k0 + (idx >> 4), col = n0 + (idx & 15);
        rb[j] = (col < g.N && kb < kblk) ? g.B[(long long)kb * g.ldb + col] : 0.0;
      }
    }
  };
  double acc = 0.0;
  fetch(t.k0);
  for (int k0 = t.k0; k0 < kblk; k0 += KC) {
    __syncthreads();  // the previous chunk's readers are done
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int idx = tid + 256 * j;
      As[idx >> 6][idx & 63] = ra[j];
      if (TRANSB)
        Bs[idx & 63][idx >> 6] = rb[j];
      else
        Bs[idx >> 4][idx & 15] = rb[j];
    }
    __syncthreads();
    if (k0 + KC < kblk) fetch(k0 + KC);
    const int n = min(KC, kend - k0);
    int k = 0;
    for (; k + 8 <= n; k += 8)
#pragma unroll
      for (int u = 0; u < 8; ++u) acc = fma(As[ty][k + u], Bs[k + u][tx], acc);
    for (; k < n; ++k) acc = fma(As[ty][k], Bs[k][tx], acc);
  }
  if (!used) return;
  double* C = g.C + t.coff + (long long)gm * g.ldc + gn;
  double v = alpha * acc;
  if (g.flags & kAccum) v += *C;
  *C = v;
}

// out[m][n] = alpha * sum_s part[s][m][n] over the upper triangle (n >= m)
// when symmetric (mirrored to the lower one), else everywhere.
__global__ void k_splitk_reduce(const double* __restrict__ part, int nsplit, int n,
                                double alpha, int symmetric, double* __restrict__ out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n * n) return;
  const int m = (int)(idx / n), c = (int)(idx % n);
  if (symmetric && c < m) return;
  double s = splitk_sum(part + idx, nsplit, (long long)n * n);
  s *= alpha;
  out[idx] = s;
  if (symmetric && c != m) out[(long long)c * n + m] = s;
}

// Zero atom blocks (I, J) of the n x n matrix M with Frobenius norm < eps.  One
// warp to a block, which is a few hundred bytes: the time is one trip to L2, and
// a block of 128 threads with a shared-memory sum waited eight times at its
// barriers (20 us for 490 functions in 62 blocks, now 10).  Squares go to 128
// partial sums (element e to e mod 128), added pairwise.
// grid ceil(nblk^2 / 8), block 256.
__global__ void __launch_bounds__(256)
    k_block_filter(double* __restrict__ M, int n, const int* __restrict__ boff, int nblk,
                   double eps) {
  const int w = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (w >= nblk * nblk) return;
  const int I = w / nblk, J = w % nblk;
  const int r0 = boff[I], nr = boff[I + 1] - r0;
  const int c0 = boff[J], nc = boff[J + 1] - c0;
  double* m = M + (long long)r0 * n + c0;
  double s[4] = {};
  for (int e0 = lane; e0 < nr * nc; e0 += 128) {
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = e0 + 32 * q;
      v[q] = e < nr * nc ? m[(long long)(e / nc) * n + e % nc] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] = fma(v[q], v[q], s[q]);
  }
  double t = (s[0] + s[2]) + (s[1] + s[3]);
#pragma unroll
  for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (sqrt(t) < eps)
    for (int e = lane; e < nr * nc; e += 32) m[(long long)(e / nc) * n + e % nc] = 0.0;
}

}  // namespace gbjk

namespace gbjk {

// Seeded synthetic 3-center tensor in the panel layout (the synthetic DF-K
// workload): element (Y, mu, nu) = N(0,1)[seed, min(mu,nu), max(mu,nu), Y] *
// exp(-0.5 |I - J| / decay), I and J the atom blocks of mu and nu, so the
// tensor is symmetric in (mu, nu).  Normal deviates come from a splitmix64
// hash of the indices through Box-Muller.  grid (ceil(maxK/128), naux, nbf).
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

__global__ void k_synthetic_panels(double* __restrict__ B, const long long* __restrict__ panel_off,
                                   const int* __restrict__ blk_of, const int* __restrict__ boff,
                                   const int* __restrict__ panel_K, const int* __restrict__ cmoff,
                                   const int* __restrict__ colmap, int nbf, int naux,
                                   unsigned long long seed, float decay) {
  const int mu = blockIdx.z;
  const int Y = blockIdx.y;
  const int I = blk_of[mu];
  const int m = mu - boff[I];
  const int KI = panel_K[I];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= KI) return;
  const int nu = colmap[cmoff[I] + k];
  const int J = blk_of[nu];
  const unsigned long long a = (unsigned long long)min(mu, nu), b = (unsigned long long)max(mu, nu);
  const unsigned long long h = splitmix64(seed ^ splitmix64((a * (unsigned long long)nbf + b) *
                                                               (unsigned long long)naux + Y));
  const float u1 = ((float)(h >> 40) + 0.5f) * (1.0f / 16777216.0f);
  const float u2 = (float)((h >> 16) & 0xFFFFFF) * (1.0f / 16777216.0f);
  const float g = sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
  const float w = expf(-0.5f * fabsf((float)(I - J)) / decay);
  B[panel_off[I] + ((long long)m * naux + Y) * KI + k] = (double)(g * w);
}

// out = alpha * sum_s part[s] (+ out when accumulate), upper triangle
// mirrored when symmetric; order: existing value, then splits in order.
__global__ void k_splitk_reduce_acc(const double* __restrict__ part, int nsplit, int n,
                                    double alpha, int symmetric, int accumulate,
                                    double* __restrict__ out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n * n) return;
  const int m = (int)(idx / n), c = (int)(idx % n);
  if (symmetric && c < m) return;
  double s = splitk_sum(part + idx, nsplit, (long long)n * n);
  s *= alpha;
  if (accumulate) s += out[idx];
  out[idx] = s;
  if (symmetric && c != m) out[(long long)c * n + m] = s;
}

}  // namespace gbjk
