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

// The recurrence's factors at point i of line (y eigenvalue l, z eigenvalue h).
struct ModePoint {
  double al, be, ga;  // e' = al e + be (e_{i-1} + e_{i+1}) + ga b
};
__device__ __forceinline__ ModePoint mode_point(const ModeSweeps &M, double l, double h, int i) {
  const double nb = (M.nx == 1) ? 0.0 : ((i == 0 || i == M.nx - 1) ? 1.0 : 2.0);
  const double wd = M.w / (M.cx * nb + 2.0 * M.cy + M.cz * h);
  ModePoint q = {0.0, 0.0, 0.0};
  if (i < M.nx) q = {(1.0 - M.w) + wd * (M.cy * (2.0 - l)), wd * M.cx, wd};  // cy (2 - l) = 2 cy cos(theta)
  return q;
}

// All sweeps of a line of up to 32 PPL points in a warp's registers, PPL
// consecutive points per lane, from zero: e = ga b in the first, e in place.
template <int PPL>
__device__ __forceinline__ void line_sweeps(const ModeSweeps &M, const ModePoint (&q)[PPL], double (&e)[PPL], int lane) {
  double g[PPL];
#pragma unroll
  for (int p = 0; p < PPL; p++) e[p] = g[p] = q[p].ga * e[p];
  for (int s = 1; s < M.sweeps; s++) {
    double l = __shfl_up_sync(0xffffffffu, e[PPL - 1], 1), r = __shfl_down_sync(0xffffffffu, e[0], 1);
    if (lane == 0) l = 0.0;  // lanes past the line hold zeros
    if (lane == 31) r = 0.0;
    double prev = l;
#pragma unroll
    for (int p = 0; p < PPL; p++) {
      const double own = e[p], next = (p + 1 < PPL) ? e[p + 1 < PPL ? p + 1 : p] : r;
      e[p] = fma(q[p].be, prev + next, fma(q[p].al, own, g[p]));
      prev = own;
    }
  }
}

// Lines of up to 64 points: the sweeps of a line are one matrix of its (y, z)
// mode, applied instead of swept through: nx products per point for 120
// operations in a chain of forty dependent pairs (19.4 us at 37x19x23, 22.5 at
// 25x25x75; by matrices 9.4 and 9.7).  The factors are symmetric about the
// line's middle, so are its sweeps: the even part (b_j + b_j', j' = nx-1-j) and
// the odd part (b_j - b_j') of the right-hand side give those of the result,
// two matrices of half the order.  D[class][mz][j][i] = (even, odd), i
// consecutive, half = (nx+1)/2 of each; the sine and cosine modes of y share
// theirs (class = (my+1)/2).  Up to 64 points because half a line then fits a
// warp.  No limit on their size beyond modes_pay's on the level (81 MB at
// 63x69x141, a seventh of the context): building them is repaid within two steps
// at every size.  Without / with them, creation and one step: 63x35x75 (22 MB)
// 2.4 / 3.4 and 3.33 / 2.79 ms; 47x45x121 (26 MB) 2.6 / 4.1 and 7.60 / 5.99 ms;
// 31x69x121 (17 MB) 2.6 / 3.5 and 6.79 / 5.74 ms; 63x69x141 2.7 / 6.1 and 18.2 /
// 15.3 ms.
constexpr int DENSE_NX = 64;
__host__ __device__ inline int mode_classes(int ny) { return ny / 2 + 1; }
inline size_t dense_values(int nx, int ny, int nz) {
  const size_t half = (nx + 1) / 2;
  return 2 * half * half * (size_t)mode_classes(ny) * nz;
}
inline bool dense_pays(int nx) { return nx <= DENSE_NX; }

// A column j of the matrices: the sweeps of the unit pair at j and nx-1-j, on
// half the line (its other half is plus or minus the mirror image), a point
// per lane; both parities per warp where they fit.
__global__ void __launch_bounds__(32 * MODE_W)
    k_dense_build(ModeSweeps M, const double *__restrict__ ly, const double *__restrict__ lz, double *__restrict__ D) {
  const int lane = threadIdx.x & 31, nx = M.nx, half = (nx + 1) / 2, width = half <= 16 ? 16 : 32;
  const int col = (blockIdx.x * MODE_W + (threadIdx.x >> 5)) * (32 / width) + lane / width;
  const int j = col >> 1, odd = col & 1, jm = nx - 1 - j, i = lane & (width - 1);
  const int mz = blockIdx.y, cl = blockIdx.z;
  const ModePoint q = mode_point(M, ly[cl == 0 ? 0 : 2 * cl - 1], lz[mz], i);
  double g = 0.0;
  if (i == j) g = (j == jm) ? (odd ? 0.0 : 1.0) : 0.5;
  g *= q.ga;
  double e = g;
  const bool end = i == half - 1, own = !(nx & 1);  // beyond the half line: the mirror image of its end, or of its neighbour
  for (int s = 1; s < M.sweeps; s++) {
    double l = __shfl_up_sync(0xffffffffu, e, 1, width), r = __shfl_down_sync(0xffffffffu, e, 1, width);
    if (end) r = own ? e : l;
    if (end && odd) r = -r;
    if (i == 0) l = 0.0;
    if (end && nx == 1) r = 0.0;
    e = fma(q.be, l + r, fma(q.al, e, g));
    if (end && odd && !own) e = 0.0;  // the middle point of an odd part
  }
  if (j < half && i < half) D[2 * ((size_t)half * (j + half * ((size_t)mz + (size_t)M.nz * cl)) + i) + odd] = e;
}

// y modes of the z-transformed right-hand side and the matrix of their line: a
// warp per line.  PAIR: points i and nx-1-i and both parts on lane i.  Else (up
// to 32 points) a point per lane for the modes, then the even part on lanes
// 0-15 and the odd on 16-31: half the FP64 instructions.
template <bool PAIR>
__global__ void __launch_bounds__(32 * MODE_W)
    k_mode_dense(int nx, int ny, int nz, const double *__restrict__ Qy, const double *__restrict__ D,
                 const double *__restrict__ t, double *__restrict__ out) {
  const int lane = threadIdx.x & 31, my = blockIdx.x * MODE_W + (threadIdx.x >> 5), mz = blockIdx.y;
  if (my >= ny) return;
  const int half = (nx + 1) / 2, i = min(PAIR ? lane : lane & 15, half - 1), im = nx - 1 - i;
  const double *qy = Qy + (size_t)my * ny;
  const double *d = D + 2 * ((size_t)half * half * (mz + (size_t)nz * ((my + 1) / 2)) + i);
  double *op = out + (size_t)nx * (my + (size_t)ny * mz);
  const double *tp = t + (size_t)nx * ny * mz;
  double e, o;
  if constexpr (PAIR) {
    double a[2] = {0.0, 0.0}, b[2] = {0.0, 0.0};
    int j = 0;
#pragma unroll 4
    for (; j + 1 < ny; j += 2) {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        a[r] = fma(qy[j + r], tp[i + (size_t)nx * (j + r)], a[r]);
        b[r] = fma(qy[j + r], tp[im + (size_t)nx * (j + r)], b[r]);
      }
    }
    if (j < ny) {
      a[0] = fma(qy[j], tp[i + (size_t)nx * j], a[0]);
      b[0] = fma(qy[j], tp[im + (size_t)nx * j], b[0]);
    }
    const double x = a[0] + a[1], y = b[0] + b[1];
    const double ev = (i == im) ? x : x + y, od = x - y;  // the middle point is its own mirror
    double se[2] = {0.0, 0.0}, so[2] = {0.0, 0.0};
#pragma unroll 4
    for (j = 0; j + 1 < half; j += 2) {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const double2 m = __ldg(reinterpret_cast<const double2 *>(d + 2 * (size_t)half * (j + r)));
        se[r] = fma(m.x, __shfl_sync(0xffffffffu, ev, j + r), se[r]);
        so[r] = fma(m.y, __shfl_sync(0xffffffffu, od, j + r), so[r]);
      }
    }
    if (j < half) {
      const double2 m = __ldg(reinterpret_cast<const double2 *>(d + 2 * (size_t)half * j));
      se[0] = fma(m.x, __shfl_sync(0xffffffffu, ev, j), se[0]);
      so[0] = fma(m.y, __shfl_sync(0xffffffffu, od, j), so[0]);
    }
    e = se[0] + se[1];
    o = so[0] + so[1];
  } else {
    const int odd = lane >> 4;
    double mm[16];  // the lane's row of its part, in flight during the modes
#pragma unroll
    for (int j = 0; j < 16; j++) mm[j] = __ldg(d + 2 * (size_t)half * min(j, half - 1) + odd);
    const int xl = min(lane, nx - 1);
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    int j = 0;
#pragma unroll 4
    for (; j + 3 < ny; j += 4) {
#pragma unroll
      for (int r = 0; r < 4; r++) a[r] = fma(qy[j + r], tp[xl + (size_t)nx * (j + r)], a[r]);
    }
    for (; j < ny; j++) a[0] = fma(qy[j], tp[xl + (size_t)nx * j], a[0]);
    const double x = (a[0] + a[1]) + (a[2] + a[3]);
    const double xi = __shfl_sync(0xffffffffu, x, i), xm = __shfl_sync(0xffffffffu, x, im);
    const double v = odd ? xi - xm : (i == im ? xi : xi + xm);
    double s[2] = {0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const double u = __shfl_sync(0xffffffffu, v, 16 * odd + q);
      if (q < half) s[q & 1] = fma(mm[q], u, s[q & 1]);
    }
    e = s[0] + s[1];
    o = __shfl_down_sync(0xffffffffu, e, 16);
  }
  if (lane < half) {
    op[i] = e + o;
    op[im] = e - o;
  }
}

// y modes of the z-transformed right-hand side and all sweeps of their x
// lines, of more than DENSE_NX points: a warp per line, PPL consecutive x
// points per lane.
template <int PPL>
__global__ void __launch_bounds__(32 * MODE_W)
    k_mode_lines(ModeSweeps M, const double *__restrict__ Qy, const double *__restrict__ ly,
                 const double *__restrict__ lz, const double *__restrict__ t, double *__restrict__ out) {
  const int lane = threadIdx.x & 31, my = blockIdx.x * MODE_W + (threadIdx.x >> 5), mz = blockIdx.y;
  const int nx = M.nx, ny = M.ny;
  if (my >= ny) return;
  const double *tp = t + (size_t)nx * ny * mz;
  const double *qy = Qy + (size_t)my * ny;
  double e[PPL];
#pragma unroll
  for (int p = 0; p < PPL; p++) e[p] = 0.0;
#pragma unroll 4
  for (int j = 0; j < ny; j++) {
    const double q = qy[j];
#pragma unroll
    for (int p = 0; p < PPL; p++) {
      const int i = lane * PPL + p;
      if (i < nx) e[p] = fma(q, tp[i + (size_t)nx * j], e[p]);
    }
  }
  ModePoint q[PPL];
#pragma unroll
  for (int p = 0; p < PPL; p++) q[p] = mode_point(M, ly[my], lz[mz], lane * PPL + p);
  line_sweeps<PPL>(M, q, e, lane);
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
