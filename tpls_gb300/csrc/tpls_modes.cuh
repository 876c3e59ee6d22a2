// tpls_modes.cuh -- the coarsest multigrid level without a dense inverse
// (FP64), a fixed number of damped z-line Jacobi sweeps from zero, by modes.
//
// A sweep is e' = (1 - w) e + w D^{-1} (b + cx (e[i-1] + e[i+1]) + cy (e[j-1] +
// e[j+1])) with D the z-line matrix of column (i, j): its x and y terms differ
// between columns only by the x class (first, interior, last).  The cosine
// modes of z diagonalise D and the Fourier modes of periodic y the y coupling,
// so in (y, z) modes every sweep is a three-term recurrence along x,
//   e'_i = a_i e_i + q_i (e_{i-1} + e_{i+1}) + g_i,
// with a_i = 1 - w + 2 w cy cos(theta) / d_i, q_i = w cx / d_i, g_i = w b_i /
// d_i, d_i = cx nx_i + 2 cy + cz lambda: all sweeps run in a warp's registers
// between two transforms, instead of one launch each with a Thomas solve of
// one warp per 32 columns (9.4 us per sweep at 37x19x23, 23 us at 25x25x75,
// forty per V-cycle).  The result is the sweeps' own up to rounding.
#pragma once
#include "tpls_common.cuh"

namespace tpls {

constexpr int MODE_PPL = 8;  // x points per lane, at most: lines of up to 256 points
// Warps per block: two, so that the few hundred warps of a small level spread
// over all SMs: a warp's FP64 instruction holds its scheduler's FP64 unit for
// about 80 cycles (40 ns), so a small level takes as long as the busiest of
// the 608 schedulers has FP64 instructions.  The transforms therefore take one
// output per warp and column group (M, P, J = 1) while there are fewer warps
// than twice that, and several, which share the loads, beyond.
constexpr int MODE_W = 2, MODE_WARPS = 2 * 608;

// out[m][c] = sum_k Q[m][k] in[k][c], Q[m][n-1-k] = (-1)^m Q[m][k] (cosine
// modes), columns c consecutive.  A warp takes 32 columns and M modes of one
// parity, and folds the input's two halves: n/2 products per mode.
template <int MODE_M>
__global__ void __launch_bounds__(32 * MODE_W)
    k_modes_z(int n, int ncol, const double *__restrict__ Q, const double *__restrict__ in, double *__restrict__ out) {
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), g = blockIdx.y * MODE_W + (threadIdx.x >> 5);
  const int par = g & 1, m0 = (g >> 1) * (2 * MODE_M) + par;  // modes m0, m0 + 2, ...
  if (c >= ncol || m0 >= n) return;
  const int half = n / 2;
  double acc[MODE_M] = {};
  const double *q[MODE_M];
#pragma unroll
  for (int r = 0; r < MODE_M; r++) q[r] = Q + (size_t)min(m0 + 2 * r, n - 1) * n;
#pragma unroll 4
  for (int k = 0; k < half; k++) {
    const double a = in[c + (size_t)ncol * k], b = in[c + (size_t)ncol * (n - 1 - k)];
    const double v = par ? a - b : a + b;
#pragma unroll
    for (int r = 0; r < MODE_M; r++) acc[r] = fma(q[r][k], v, acc[r]);
  }
  if ((n & 1) && !par) {  // the middle point (odd modes vanish there)
    const double v = in[c + (size_t)ncol * half];
#pragma unroll
    for (int r = 0; r < MODE_M; r++) acc[r] = fma(q[r][half], v, acc[r]);
  }
#pragma unroll
  for (int r = 0; r < MODE_M; r++)
    if (m0 + 2 * r < n) out[c + (size_t)ncol * (m0 + 2 * r)] = acc[r];
}

// out[k][c] = sum_m Q[m][k] in[m][c]: even and odd modes summed apart give
// the points k and n-1-k together; a warp takes P (1 or 2) such pairs.
template <int P>
__global__ void __launch_bounds__(32 * MODE_W)
    k_points_z(int n, int ncol, const double *__restrict__ Q, const double *__restrict__ in, double *__restrict__ out) {
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), k0 = P * (blockIdx.y * MODE_W + (threadIdx.x >> 5));
  const int half = (n + 1) / 2;  // the middle point pairs with itself
  if (c >= ncol || k0 >= half) return;
  const int k1 = min(k0 + P - 1, half - 1);
  double e0 = 0.0, o0 = 0.0, e1 = 0.0, o1 = 0.0;
#pragma unroll 4
  for (int m = 0; m + 1 < n; m += 2) {
    const double a = in[c + (size_t)ncol * m], b = in[c + (size_t)ncol * (m + 1)];
    const double *q = Q + (size_t)m * n;
    e0 = fma(q[k0], a, e0);
    o0 = fma(q[n + k0], b, o0);
    if constexpr (P == 2) {
      e1 = fma(q[k1], a, e1);
      o1 = fma(q[n + k1], b, o1);
    }
  }
  if (n & 1) {
    const double a = in[c + (size_t)ncol * (n - 1)];
    e0 = fma(Q[(size_t)(n - 1) * n + k0], a, e0);
    if constexpr (P == 2) e1 = fma(Q[(size_t)(n - 1) * n + k1], a, e1);
  }
  out[c + (size_t)ncol * k0] = e0 + o0;
  out[c + (size_t)ncol * (n - 1 - k0)] = e0 - o0;
  if (k1 > k0) {
    out[c + (size_t)ncol * k1] = e1 + o1;
    out[c + (size_t)ncol * (n - 1 - k1)] = e1 - o1;
  }
}

struct ModeSweeps {
  int nx, ny, nz, sweeps;
  double cx, cy, cz, w;
};

// y modes of the z-transformed right-hand side and all sweeps of their x
// lines: a warp per line, PPL consecutive x points per lane.
template <int PPL>
__global__ void __launch_bounds__(32 * MODE_W)
    k_mode_lines(ModeSweeps M, const double *__restrict__ Qy, const double *__restrict__ ly,
                 const double *__restrict__ lz, const double *__restrict__ t, double *__restrict__ out) {
  const int lane = threadIdx.x & 31, my = blockIdx.x * MODE_W + (threadIdx.x >> 5), mz = blockIdx.y;
  const int nx = M.nx, ny = M.ny;
  if (my >= ny) return;
  const double *tp = t + (size_t)nx * ny * mz;
  const double *qy = Qy + (size_t)my * ny;
  double e[PPL], al[PPL], be[PPL], ga[PPL];
#pragma unroll
  for (int p = 0; p < PPL; p++) ga[p] = 0.0;
#pragma unroll 4
  for (int j = 0; j < ny; j++) {
    const double q = qy[j];
#pragma unroll
    for (int p = 0; p < PPL; p++) {
      const int i = lane * PPL + p;
      if (i < nx) ga[p] = fma(q, tp[i + (size_t)nx * j], ga[p]);
    }
  }
  const double cc = M.cy * (2.0 - ly[my]);  // 2 cy cos(theta)
#pragma unroll
  for (int p = 0; p < PPL; p++) {
    const int i = lane * PPL + p;
    const double nb = (nx == 1) ? 0.0 : ((i == 0 || i == nx - 1) ? 1.0 : 2.0);
    const double wd = M.w / (M.cx * nb + 2.0 * M.cy + M.cz * lz[mz]);
    const bool in = i < nx;
    al[p] = in ? (1.0 - M.w) + wd * cc : 0.0;
    be[p] = in ? wd * M.cx : 0.0;
    ga[p] *= in ? wd : 0.0;
    e[p] = ga[p];  // the first sweep, from zero
  }
  for (int s = 1; s < M.sweeps; s++) {
    double l = __shfl_up_sync(0xffffffffu, e[PPL - 1], 1), r = __shfl_down_sync(0xffffffffu, e[0], 1);
    if (lane == 0) l = 0.0;  // lanes past the line hold zeros
    if (lane == 31) r = 0.0;
    double prev = l;
#pragma unroll
    for (int p = 0; p < PPL; p++) {
      const double own = e[p], next = (p + 1 < PPL) ? e[p + 1 < PPL ? p + 1 : p] : r;
      e[p] = fma(be[p], prev + next, fma(al[p], own, ga[p]));
      prev = own;
    }
  }
  double *op = out + (size_t)nx * (my + (size_t)ny * mz);
#pragma unroll
  for (int p = 0; p < PPL; p++) {
    const int i = lane * PPL + p;
    if (i < nx) op[i] = e[p];
  }
}

// out[mz][j][i] = sum_my Qy[my][j] in[mz][my][i]; a warp takes 32 points of a
// line and J rows j.
template <int J>
__global__ void __launch_bounds__(32 * MODE_W)
    k_points_y(int nx, int ny, const double *__restrict__ Qy, const double *__restrict__ in,
               double *__restrict__ out) {
  const int i = blockIdx.x * 32 + (threadIdx.x & 31), j0 = J * (blockIdx.y * MODE_W + (threadIdx.x >> 5));
  if (i >= nx || j0 >= ny) return;
  const double *p = in + (size_t)nx * ny * blockIdx.z + i;
  double acc[J] = {};
  int j[J];
#pragma unroll
  for (int r = 0; r < J; r++) j[r] = min(j0 + r, ny - 1);
#pragma unroll 4
  for (int m = 0; m < ny; m++) {
    const double v = p[(size_t)nx * m];
    const double *q = Qy + (size_t)m * ny;
#pragma unroll
    for (int r = 0; r < J; r++) acc[r] = fma(q[j[r]], v, acc[r]);
  }
  double *o = out + (size_t)nx * ny * blockIdx.z + i;
#pragma unroll
  for (int r = 0; r < J; r++)
    if (j0 + r < ny) o[(size_t)nx * (j0 + r)] = acc[r];
}

}  // namespace tpls
