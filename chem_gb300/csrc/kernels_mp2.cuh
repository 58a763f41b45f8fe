// Kernels of the SOS-AO-MP2 Laplace batch (ll_full Z builder) that are not
// GEMMs: coefficient gathers, operand exponents, the split-K reduction of Z
// and the energy sums.  Every point t of the batch uses the same padded
// strides (hld occupied columns, vld virtual columns), so grid.y = t and a
// fixed per-point stride address all of them.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gbjk {

// Cg_t[r][i] = Lo_t[colmap[r]][i]: panel-column copies of every point's
// occupied factor.  grid (ceil(nrows*ld / 256), npts).
__global__ void k_mp2_gather(const double* __restrict__ Lo, long long lo_stride, int ld,
                             const int* __restrict__ colmap, int nrows,
                             double* __restrict__ Cg, long long cg_stride) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)nrows * ld) return;
  const int r = (int)(idx / ld), i = (int)(idx % ld);
  const int t = blockIdx.y;
  Cg[t * cg_stride + idx] = Lo[t * lo_stride + (long long)colmap[r] * ld + i];
}

// Z_t[X][Y] = Z_t[Y][X] = sum_s part[s][t][X][Y] (s in order) for X <= Y.
// grid (ceil(n*n / 256), npts).
__global__ void k_mp2_z_reduce(const double* __restrict__ part, int nsplit, int npts, int n,
                               double* __restrict__ Z) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nn = (long long)n * n;
  if (idx >= nn) return;
  const int t = blockIdx.y;
  const int X = (int)(idx / n), Y = (int)(idx % n);
  if (Y < X) return;
  double s = 0.0;
  for (int k = 0; k < nsplit; ++k) s += part[((long long)k * npts + t) * nn + idx];
  Z[t * nn + idx] = s;
  Z[t * nn + (long long)Y * n + X] = s;
}

// Z_t[Y][X] = Z_t[X][Y] for X < Y.  grid (ceil(n*n / 256), npts).
__global__ void k_mp2_z_mirror(double* __restrict__ Z, int n) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nn = (long long)n * n;
  if (idx >= nn) return;
  const int X = (int)(idx / n), Y = (int)(idx % n);
  if (Y <= X) return;
  double* z = Z + blockIdx.y * nn;
  z[(long long)Y * n + X] = z[idx];
}

// rsq[t][X] = sum_Y Z_t[X][Y]^2: one warp per row, lane l sums Y = l, l+32,
// ... with fma, then an xor butterfly.  grid (ceil(n*32 / 256), npts).
__global__ void k_mp2_rowsq(const double* __restrict__ Z, int n, double* __restrict__ rsq) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= n) return;
  const int t = blockIdx.y;
  const double* z = Z + (long long)t * n * n + w * n;
  double s = 0.0;
  for (int Y = lane; Y < n; Y += 32) s = fma(z[Y], z[Y], s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) rsq[(long long)t * n + w] = s;
}

// The same sum as strided partials of 256 threads added pairwise, for the split
// path, whose energies follow no summation order of an FP64 chain (40 us for 700
// rows in order, 4.5 so).  grid npts, block 256.
__global__ void __launch_bounds__(256)
    k_mp2_energy_tree(const double* __restrict__ rsq, int n, double* __restrict__ e) {
  __shared__ double red[8];
  const int t = blockIdx.x, tid = threadIdx.x;
  double s = 0.0;
  for (int X = tid; X < n; X += 256) s += rsq[(long long)t * n + X];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((tid & 31) == 0) red[tid >> 5] = s;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < 8; ++w) s += red[w];
    e[t] = s;
  }
}

// FP64 path: e[t] = sum_X rsq[t][X] in X order: a serial chain of n additions, bound by
// their latency once thirty-two loads are in flight (one warp per point
// passes them on by shuffles).  grid npts, block 32.
__global__ void k_mp2_energy(const double* __restrict__ rsq, int n, int npts,
                             double* __restrict__ e) {
  const int t = blockIdx.x, lane = threadIdx.x;
  const double* p = rsq + (long long)t * n;
  double s = 0.0;
  double next = lane < n ? p[lane] : 0.0;
  for (int X0 = 0; X0 < n; X0 += 32) {
    const double v = next;
    if (X0 + 32 + lane < n) next = p[X0 + 32 + lane];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const double x = __shfl_sync(0xffffffffu, v, j);
      if (X0 + j < n) s += x;
    }
  }
  if (lane == 0) e[t] = s;
}

}  // namespace gbjk
