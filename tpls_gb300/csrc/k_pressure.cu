// k_pressure.cu -- pressure Poisson solve (replaces the PETSc KSPSolve of
// main_ns_hybrid.F90:896-913 with the callbacks of pressure_solver.F90:
// 205-486).
//
// The system PETSc is handed has unknowns on x = 0..nx+1, z = 0..nz+1 and
// periodic y.  Its ghost rows are 2-point rows (zero-flux, or the inlet
// flux (dx/dt)(u_inlet-u3(0))/dy at x = 0), so they are eliminated exactly:
// the interior operator becomes the symmetric 7-point operator with
// Neumann conditions in x and z and periodic y,
//   A p = cx(2p - p[x-1] - p[x+1]) + cy(2p - p[y-1] - p[y+1])
//       + cz(2p - p[z-1] - p[z+1]),  missing x/z neighbours -> p itself,
// with cx = 1/dy^2, cy = 1/dx^2, cz = 1/dz^2 exactly as compute_matrix
// assigns them (PETSc's first index is physical y).  It is singular with
// the constant null space (pressure_solver.F90:436-439): the right-hand
// side is projected to zero mean and the solution keeps the interior mean
// of the initial guess p_old.
//
// Solver: CG preconditioned by one symmetric multigrid V-cycle.
//   levels: cell-centred coarsening of every dimension that is even and
//           >= 4 (y >= 4), down to <= 512 cells or no coarsenable dimension;
//   smoother: red-black Gauss-Seidel (red, black before the coarse correction,
//           black, red after it) on near-isotropic levels of even y extent,
//           damped z-line Jacobi (precomputed Thomas factors) on the others;
//           levels that halve in all axes, or (FP64) in x and y, run the
//           kernels of tpls_mg.cuh;
//   transfer: trilinear prolongation P, restriction R = P^T / 2^d;
//   coarse operator: rediscretisation; coarsest grid: dense FP64
//           pseudo-inverse built from the separable eigen-decomposition up to
//           512 cells, else forty smoothing sweeps (FP64: by modes,
//           tpls_modes.cuh).
// All reductions are deterministic (per-block partials summed in a fixed
// order), so a solve's iterates do not depend on timing.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#include "tpls_mg.cuh"
#include "tpls_modes.cuh"
#include "tpls_pair.cuh"
#include "tpls_pressure.h"

namespace tpls {

constexpr int PB = 256;  // threads per block for 1-D pressure kernels

// Level vectors are stored in the level type of the solver (double, or
// float for the FP32 preconditioner of the FP32-mixed form); void pointers
// here, typed at each launch.
struct PLevel {
  int nx, ny, nz, n;
  int cxs, cys, czs;     // this level was coarsened in x/y/z from the finer one
  double cx, cy, cz;
  void *b = nullptr, *e = nullptr, *e2 = nullptr, *r = nullptr, *t = nullptr;
  void *thomas = nullptr;  // [3 classes][nz][2] = (cprime, inv_den)
  int halved = 0;  // red-black level whose three axes are coarsened below it: the k_mg_* kernels
  int planar = 0;  // FP64 red-black level of which x and y are coarsened, z (odd) is not: the same passes by planes
  int point = 0;  // near-isotropic level: red-black Gauss-Seidel instead of z-lines
  double invd[3][3];  // point smoother: 1/diagonal by x class (first, interior, last) and z class
};

struct PoissonSolver {
  int nx, ny, nz, N;
  std::vector<PLevel> lv;
  double *cinv = nullptr;  // coarsest pseudo-inverse (nc x nc), or null
  int coarse_sweeps = 0;
  double *modes = nullptr;  // coarsest level by modes: Qz, Qy, lambda_z, lambda_y
  double *dense = nullptr;  // and the matrices of its lines (dense_values), where dense_pays
  double *x = nullptr, *r = nullptr, *p = nullptr, *q = nullptr, *bvec = nullptr;
  void *z = nullptr;           // preconditioned residual, in the level type
  float *r32 = nullptr;        // FP32 levels: r rounded once, for the V-cycle
  double *bin = nullptr;     // inlet ghost-row data (ny*nz)
  double *part = nullptr;    // reduction partials (3 * rblk)
  unsigned *counter = nullptr;  // last-block ticket of the reductions
  double *s = nullptr;       // device scalars
  double *s_host = nullptr;  // pinned mirror
  int rblk;                  // blocks of the grid-stride reduction kernels
  double omega = 0.8;
  int fp32 = 0;              // multigrid levels in FP32 (CG stays FP64)
  cudaStream_t side = nullptr;  // capture stream of the WHILE body
};

// device scalars of the CG iteration
// S_IT: iterations of the current solve; S_REASON: its KSP-style reason (0
// while iterating); S_WORST: lowest reason since the last stats read;
// S_ITS_TOTAL: iterations since the solver was created.
enum {
  S_SUMB = 0, S_SUMX0, S_BB, S_RR, S_RZ, S_ZMEAN, S_BETA, S_ALPHA, S_SUMX,
  S_TARGET, S_IT, S_REASON, S_WORST, S_ITS_TOTAL, S_COUNT
};

// Convergence test of pressure_solver.F90's KSP settings on the device, by
// the last block of a reduction: NaN, ||r|| <= rtol ||b||, or maxits.  With a
// graph, the WHILE node's condition is set here, so a captured solve needs
// no host round trip.
struct CgCtl {
  int maxits;
  int use_cond;
  cudaGraphConditionalHandle cond;
};

__device__ __forceinline__ void cg_decide(double *s, double rr2, int it, const CgCtl &ctl, bool init) {
  const double rr = sqrt(rr2);
  int rsn = 0;
  if (!(rr == rr)) rsn = TPLS_KSP_DIVERGED_NAN;
  else if (rr <= s[S_TARGET] || (init && s[S_BB] == 0.0)) rsn = TPLS_KSP_CONVERGED_RTOL;
  else if (!init && it >= ctl.maxits) rsn = TPLS_KSP_DIVERGED_ITS;
  s[S_IT] = (double)it;
  s[S_REASON] = (double)rsn;
  if (rsn != 0) {
    if ((double)rsn < s[S_WORST]) s[S_WORST] = (double)rsn;
    s[S_ITS_TOTAL] += (double)it;
  }
  if (ctl.use_cond) cudaGraphSetConditional(ctl.cond, rsn == 0 ? 1u : 0u);
}

static inline int nblocks(int n) { return (n + PB - 1) / PB; }

// ---------------------------------------------------------------------------
// Reductions: a fixed grid of rblk blocks, each thread accumulating a fixed
// strided subset, one partial per block, and the last block to finish (by
// an atomic ticket) summing the partials in a fixed order.  The result does
// not depend on scheduling.  Returns true in the last block, with the sums
// in tot[] of thread 0.
// A block's sums are the trees of its eight warps added in warp order.  The
// trees run in shared memory, a level of all warps and sums at a time, so a
// sum takes 17 FP64 warp instructions instead of the 48 of a shuffle tree in
// every warp (most of them on idle lanes), in the same order: 1216 blocks of
// three sums had spent 11 us on them, of a kernel of 33 us at 192x96x112.
template <int NQ>
__device__ __forceinline__ void block_sums(const double (&v)[NQ], double (&out)[NQ]) {  // in thread 0
  __shared__ double sh[NQ][PB];
  const int t = threadIdx.x;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NQ; q++) sh[q][t] = v[q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    __syncthreads();
    for (int m = t; m < NQ * (PB / 32) * o; m += PB) {
      const int q = m / (PB / 32 * o), w = m / o % (PB / 32), l = m % o;
      sh[q][32 * w + l] += sh[q][32 * w + l + o];
    }
  }
  __syncthreads();
  if (t == 0) {
    for (int q = 0; q < NQ; q++) {
      double a = 0.0;
      for (int w = 0; w < PB / 32; w++) a += sh[q][32 * w];
      out[q] = a;
    }
  }
}
template <int NQ>
__device__ __forceinline__ bool reduce_last(double (&v)[NQ], double *part, unsigned *counter,
                                            double (&tot)[NQ]) {
  __shared__ bool last;
  const int nblk = gridDim.x;
  double a[NQ];
  block_sums<NQ>(v, a);
  if (threadIdx.x == 0) {
    for (int q = 0; q < NQ; q++) part[(size_t)q * nblk + blockIdx.x] = a[q];
    __threadfence();
    last = (atomicAdd(counter, 1u) == (unsigned)(nblk - 1));
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  for (int q = 0; q < NQ; q++) {
    v[q] = 0.0;
    for (int b = threadIdx.x; b < nblk; b += PB) v[q] += __ldcg(part + (size_t)q * nblk + b);
  }
  block_sums<NQ>(v, tot);
  if (threadIdx.x == 0) *counter = 0u;
  return true;
}

template <typename R, typename TE>
__device__ __forceinline__ R applyA(const TE *__restrict__ e, int i, int j, int k, int nx, int ny, int nz,
                                    R cx, R cy, R cz) {
  const int c = i + nx * (j + ny * k);
  const R v = (R)e[c];
  const R xm = (i > 0) ? (R)e[c - 1] : v, xp = (i < nx - 1) ? (R)e[c + 1] : v;
  const R ym = (R)e[c + nx * ((j > 0) ? -1 : ny - 1)];
  const R yp = (R)e[c + nx * ((j < ny - 1) ? 1 : 1 - ny)];
  const R zm = (k > 0) ? (R)e[c - nx * ny] : v, zp = (k < nz - 1) ? (R)e[c + nx * ny] : v;
  // (2cx + 2cy + 2cz) v - cx (xm + xp) - cy (ym + yp) - cz (zm + zp): seven
  // FP64 operations (the FP64 pipe bounds these kernels on GB300)
  const R d = (R)2 * (cx + cy + cz);
  R a = d * v;
  a = fma(-cx, xm + xp, a);
  a = fma(-cy, ym + yp, a);
  return fma(-cz, zm + zp, a);
}

#define GRID_STRIDE(c, N) for (int c = blockIdx.x * PB + threadIdx.x; c < (N); c += gridDim.x * PB)
// rows (j, k) of the compact nx*ny*nz grid handed to warps in a fixed
// order, lanes striding over i; row = j + ny k, c = i + nx row
#define ROW_LOOP(nx, ny, nz)                                                                          \
  for (int row = blockIdx.x * (PB / 32) + (int)(threadIdx.x >> 5); row < (ny) * (nz);                \
       row += gridDim.x * (PB / 32))                                                                 \
    for (int j = row % (ny), k = row / (ny), i = (int)(threadIdx.x & 31); i < (nx); i += 32)

// b (compact interior) = -RHS_p + inlet contribution; x0 = p_old interior;
// sums of b and x0.
template <typename TU>
__global__ void __launch_bounds__(PB)
    k_build_b(Geo g, double dxdt_over_dy, double rdy, const double *__restrict__ rhs_p,
              const TU *__restrict__ u3, const double *__restrict__ uin,
              const double *__restrict__ pold, double *__restrict__ b, double *__restrict__ x0,
              double *__restrict__ bin, double *part, unsigned *counter, double *s) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  double v[2] = {0.0, 0.0};
  ROW_LOOP(nx, ny, nz) {
    const int c = i + nx * row;
    const int pc = TPLS_IDX(g, i + 1, j + 1, k + 1);
    double bb = -rhs_p[pc];
    if (i == 0) {
      // pressure_solver.F90:280-286: b(i,0,k) = (dx/dt)(u_inlet(k-1)-u3(0,i,k-1))/dy
      const int ju = (j == 0) ? ny : j;  // u row (j+1)-1; row 0 is the copy of row ny
      const double bi = dxdt_over_dy * (uin[k] - (double)u3[TPLS_IDX(g, 0, ju, k)]);
      bin[j + ny * k] = bi;
      bb += bi * rdy;
    }
    b[c] = bb;
    const double p0 = pold[pc];
    x0[c] = p0;
    v[0] += bb;
    v[1] += p0;
  }
  double tot[2];
  if (reduce_last<2>(v, part, counter, tot) && threadIdx.x == 0) {
    s[S_SUMB] = tot[0];
    s[S_SUMX0] = tot[1];
  }
}

// b -= mean(b); r = b - A x; ||b||^2, ||r||^2
__global__ void __launch_bounds__(PB)
    k_init_r(int nx, int ny, int nz, double cx, double cy, double cz, double invN, double rtol, CgCtl ctl,
             double *s, double *__restrict__ b, const double *__restrict__ x, double *__restrict__ r,
             float *__restrict__ r32, double *part, unsigned *counter) {
  const double mb = s[S_SUMB] * invN;
  double v[2] = {0.0, 0.0};
  ROW_LOOP(nx, ny, nz) {
    const int c = i + nx * row;
    const double bb = b[c] - mb;
    b[c] = bb;
    const double rr = bb - applyA<double, double>(x, i, j, k, nx, ny, nz, cx, cy, cz);
    r[c] = rr;
    if (r32) r32[c] = float_bits(rr);
    v[0] += bb * bb;
    v[1] += rr * rr;
  }
  double tot[2];
  if (reduce_last<2>(v, part, counter, tot) && threadIdx.x == 0) {
    s[S_BB] = tot[0];
    s[S_RR] = tot[1];
    s[S_TARGET] = rtol * sqrt(tot[0]);
    cg_decide(s, tot[1], 0, ctl, true);
  }
}

// FP64 levels: the mean of z is not removed.  A maps a constant to zero and r
// has zero sum, so neither r.z nor the iterates' differences see it, and the
// write-back sets the solution's mean; it cost three FP64 operations per
// point and iteration of the 16 outside the V-cycle.  (An FP32 level's z
// answers a last-bit change of r by FP32 roundings, which later steps of the
// FP32-mixed form amplify to its own accuracy of 1e-7: its CG keeps the
// order of every sum.)
__device__ __forceinline__ void cg_beta(double *s, double rz) {
  s[S_BETA] = (s[S_IT] == 0.0) ? 0.0 : rz / s[S_RZ];
  s[S_RZ] = rz;
}

// r.z -> beta (levels whose last smoothing sweep does not form it)
__global__ void __launch_bounds__(PB)
    k_rdot(int N, const double *__restrict__ r, const double *__restrict__ z, double *part, unsigned *counter,
           double *s) {
  double v[1] = {0.0};
  GRID_STRIDE(c, N) v[0] = fma(r[c], z[c], v[0]);
  double tot[1];
  if (reduce_last<1>(v, part, counter, tot) && threadIdx.x == 0) cg_beta(s, tot[0]);
}

// FP32 levels: sum z, sum r, r.z -> mean(z), rz_new = r.(z - mean z),
// beta = rz_new/rz
__global__ void __launch_bounds__(PB)
    k_zdot(int N, double invN, const double *__restrict__ r, const float *__restrict__ z, double *part,
           unsigned *counter, double *s) {
  double v[3] = {0.0, 0.0, 0.0};
  GRID_STRIDE(c, N) {
    const double zz = widen_bits(z[c]), rr = r[c];
    v[0] += zz;
    v[1] += rr;
    v[2] += rr * zz;
  }
  double tot[3];
  if (reduce_last<3>(v, part, counter, tot) && threadIdx.x == 0) {
    const double zm = tot[0] * invN;
    s[S_ZMEAN] = zm;
    cg_beta(s, tot[2] - zm * tot[1]);
  }
}

// The last red half-sweep of the finest level and r.z of its result (b is r).
__global__ void __launch_bounds__(PB)
    k_mg_half_dot(const __grid_constant__ MgLev<double> L, const double *__restrict__ b, double *e, int kz,
                  double *part, unsigned *counter, double *s) {
  const MgBlk B = mg_block(L, kz);
  double v[1] = {0.0};
  if (B.in) {
    const int nx = L.nx, plane = nx * L.ny;
    const int jm = (B.j > 0) ? -nx : plane - nx, jp = (B.j < L.ny - 1) ? nx : nx - plane;
    int c = 2 * B.i2 + nx * B.j + plane * B.k0;
    const double2 zero = {0.0, 0.0};
    double2 pm = (B.k0 > 0) ? *reinterpret_cast<const double2 *>(e + c - plane) : zero;
    double2 p0 = *reinterpret_cast<const double2 *>(e + c);
    for (int k = B.k0; k < B.k1; k++, c += plane) {
      const double2 pp = (k < L.nz - 1) ? *reinterpret_cast<const double2 *>(e + c + plane) : zero;
      const double2 bb = *reinterpret_cast<const double2 *>(b + c);
      const int odd = (B.j + k) & 1;
      const double z = mg_relax(L, B, e, odd ? bb.y : bb.x, odd, c, jm, jp, k, pm, p0, pp);
      e[c + odd] = z;
      v[0] = fma(odd ? bb.y : bb.x, z, fma(odd ? bb.x : bb.y, odd ? p0.x : p0.y, v[0]));
      pm = p0;
      p0 = pp;
    }
  }
  double tot[1];
  if (reduce_last<1>(v, part, counter, tot) && threadIdx.x == 0) cg_beta(s, tot[0]);
}

// k_mg_up of the finest level (FP64, b is r), with r.z of its result.
template <int CX, int CY, int CZ>
__global__ void __launch_bounds__(PB)
    k_mg_up_dot(const __grid_constant__ MgLev<double> L, const double *__restrict__ b, const double *__restrict__ ec,
                double *__restrict__ e, double *part, unsigned *counter, double *s) {
  using T = MgTile<CX, CY, CZ>;
  __shared__ double se[T::EN];
  __shared__ double ss[T::SN];
  __shared__ double sb[T::EN];
  const int gx = (L.nx / 2 + CX - 1) / CX, gy = (L.ny / 2 + CY - 1) / CY;
  const int x0 = (blockIdx.x % gx) * T::FX, y0 = (blockIdx.x / gx % gy) * T::FY, z0 = blockIdx.x / (gx * gy) * T::FZ;
  mg_up_tile<double, CX, CY, CZ>(L, b, ec, se, ss, sb, x0, y0, z0);
  double v[1] = {0.0};
  for (int q = threadIdx.x; q < T::FX * T::FY * T::FZ; q += PB) {
    const int lx = q % T::FX, ly = q / T::FX % T::FY, lz = q / (T::FX * T::FY);
    if (x0 + lx < L.nx && y0 + ly < L.ny && z0 + lz < L.nz) {
      const size_t c = x0 + lx + L.nx * (y0 + ly + (size_t)L.ny * (z0 + lz));
      const int o = lx + 2 + T::EX * (ly + 2 + T::EY * (lz + 2));
      const double z = se[o];
      e[c] = z;
      v[0] = fma(sb[o], z, v[0]);
    }
  }
  double tot[1];
  if (reduce_last<1>(v, part, counter, tot) && threadIdx.x == 0) cg_beta(s, tot[0]);
}

// p = z + beta p, z without its mean on FP32 levels (the first iteration's
// beta is 0 and p not read)
template <typename R>
__global__ void __launch_bounds__(PB)
    k_pupdate(int N, const double *__restrict__ s, const R *__restrict__ z, double *__restrict__ p) {
  const double beta = s[S_BETA];
  const bool first = (__double_as_longlong(beta) == 0);
  const int c = blockIdx.x * PB + threadIdx.x;
  if (c >= N) return;
  double zz;
  if constexpr (sizeof(R) == sizeof(float)) zz = widen_bits(z[c]) - s[S_ZMEAN];
  else zz = z[c];
  p[c] = first ? zz : fma(beta, p[c], zz);
}

// q = A p; p.q -> alpha = rz / p.q.  FLAT: points in order over all lanes
// (rows of a length that 32 does not divide, and numbers of rows that the
// blocks do not, left lanes and SMs idle: 19.9 us at 100x50x75, 14.5 so); the FP32 form keeps its rows, whose
// sums' order it must not change.
template <bool FLAT>
__global__ void __launch_bounds__(PB)
    k_apply_dot(int nx, int ny, int nz, double cx, double cy, double cz, const double *__restrict__ p,
                double *__restrict__ q, double *part, unsigned *counter, double *s) {
  double v[1] = {0.0};
  auto point = [&](int i, int j, int k, int c) {
    const double a = applyA<double, double>(p, i, j, k, nx, ny, nz, cx, cy, cz);
    q[c] = a;
    v[0] += p[c] * a;
  };
  if constexpr (FLAT) {
#pragma unroll 2
    GRID_STRIDE(c, nx * ny * nz) {
      const int row = c / nx, k = row / ny;
      point(c - nx * row, row - ny * k, k, c);
    }
  } else {
    ROW_LOOP(nx, ny, nz) point(i, j, k, i + nx * row);
  }
  double tot[1];
  if (reduce_last<1>(v, part, counter, tot) && threadIdx.x == 0) s[S_ALPHA] = s[S_RZ] / tot[0];
}

// x += alpha p; r -= alpha q; ||r||^2
__global__ void __launch_bounds__(PB)
    k_axpy(int N, CgCtl ctl, double *s, const double *__restrict__ p, const double *__restrict__ q,
           double *__restrict__ x, double *__restrict__ r, float *__restrict__ r32, double *part,
           unsigned *counter) {
  const double alpha = s[S_ALPHA];
  double v[1] = {0.0};
  GRID_STRIDE(c, N) {
    x[c] += alpha * p[c];
    const double rr = r[c] - alpha * q[c];
    r[c] = rr;
    if (r32) r32[c] = float_bits(rr);
    v[0] += rr * rr;
  }
  double tot[1];
  if (reduce_last<1>(v, part, counter, tot) && threadIdx.x == 0) {
    s[S_RR] = tot[0];
    cg_decide(s, tot[0], (int)s[S_IT] + 1, ctl, false);
  }
}

__global__ void __launch_bounds__(PB)
    k_sumx(int N, const double *__restrict__ x, double *part, unsigned *counter, double *s) {
  double v[1] = {0.0};
  GRID_STRIDE(c, N) v[0] += x[c];
  double tot[1];
  if (reduce_last<1>(v, part, counter, tot) && threadIdx.x == 0) s[S_SUMX] = tot[0];
}

// write the solution back into the full p-grid array with every ghost
// value rebuilt from its 2-point row, and the constant fixed.
__global__ void k_writeback(Geo g, double dy, double invN, const double *__restrict__ s,
                            const double *__restrict__ x, const double *__restrict__ bin,
                            double *__restrict__ pres) {
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 4 + threadIdx.y, k = blockIdx.z;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  if (i > nx + 1 || j > ny + 1) return;
  const double shift = (s[S_SUMX0] - s[S_SUMX]) * invN;
  const int jj = wrapy(j, ny) - 1;
  const int kk = (k == 0) ? 0 : ((k == nz + 1) ? nz - 1 : k - 1);  // z ghost planes copy
  double v;
  if (i == 0) {
    v = x[nx * (jj + ny * kk)] + shift + dy * bin[jj + ny * kk];
  } else {
    const int ii = (i == nx + 1) ? nx - 1 : i - 1;
    v = x[ii + nx * (jj + ny * kk)] + shift;
  }
  pres[TPLS_IDX(g, i, j, k)] = v;
}

// ---------------------------------------------------------------------------
// multigrid kernels of the levels k_mg_* (tpls_mg.cuh) do not cover: axes
// that do not halve, anisotropic couplings, odd y extents.  R is the type of
// the level (double, or float for the FP32 preconditioner, whose finest
// right-hand side is the CG residual rounded once per iteration).
template <typename R>
struct LevArgs {
  int nx, ny, nz;
  R cx, cy, cz;
};

// one damped z-line Jacobi sweep: eo = (1-w) ei + w Dline^{-1}(b - N ei);
// zero_init: ei == 0.
constexpr int LJB = 64;  // threads per block of the line smoother (one column each)

// TS: values per level of the factor table (k_line_jacobi3's carries four).
template <typename R, int TS>
__global__ void __launch_bounds__(LJB)
    k_line_jacobi(LevArgs<R> L, R omega, R one_m_omega, int zero_init, const R *__restrict__ thomas,
                  const R *__restrict__ b, const R *__restrict__ ei, R *__restrict__ t, R *__restrict__ eo) {
  const int col = blockIdx.x * LJB + threadIdx.x;
  const int nx = L.nx, ny = L.ny, nz = L.nz;
  if (col >= nx * ny) return;
  const int i = col % nx, j = col / nx;
  const int cls = (nx == 1) ? 1 : ((i == 0) ? 0 : ((i == nx - 1) ? 2 : 1));
  const R *th = thomas + (size_t)cls * nz * TS;
  const int plane = nx * ny;
  const int jm = (j > 0) ? -nx : nx * (ny - 1), jp = (j < ny - 1) ? nx : -nx * (ny - 1);
  R y = (R)0;
  for (int k = 0; k < nz; k++) {
    const int c = col + plane * k;
    R rhs = b[c];
    if (!zero_init) {
      R nb = L.cy * (ei[c + jm] + ei[c + jp]);
      if (i > 0) nb += L.cx * ei[c - 1];
      if (i < nx - 1) nb += L.cx * ei[c + 1];
      rhs += nb;
    }
    y = (rhs + L.cz * y) * th[TS * k + 1];
    t[c] = y;
  }
  R xn = (R)0;
  for (int k = nz - 1; k >= 0; k--) {
    const int c = col + plane * k;
    xn = t[c] - ((k < nz - 1) ? th[TS * k] * xn : (R)0);
    eo[c] = zero_init ? omega * xn : one_m_omega * ei[c] + omega * xn;
  }
}

// The same sweep for 32 columns per block in three phases: all threads
// assemble the line right-hand sides into shared memory, one warp runs the
// Thomas forward/backward substitution in shared memory, all threads write
// the damped result.  Dynamic shared memory: nz * 32 values of float.
// 1024 threads: a level has few blocks (20 at 25x25x75), and with 256 each
// thread assembled and wrote its ten levels one load after another (875 launches
// of a solve's V-cycles at 100x50x75 8.4 -> 7.1 ms, at 145x70x99 21.7 -> 18.3).
constexpr int LJ2_T = 1024;

__global__ void __launch_bounds__(LJ2_T)
    k_line_jacobi2(LevArgs<float> L, float omega, float one_m_omega, int zero_init, const float *__restrict__ thomas,
                   const float *__restrict__ b, const float *__restrict__ ei, float *__restrict__ eo) {
  extern __shared__ __align__(16) unsigned char lj2_raw[];
  float *buf = reinterpret_cast<float *>(lj2_raw);  // [nz][32]
  const int nx = L.nx, ny = L.ny, nz = L.nz, ncol = nx * ny, plane = nx * ny;
  const int col0 = blockIdx.x * 32;
  // every thread keeps one column (LJ2_T is a multiple of 32)
  const int mycol = col0 + (threadIdx.x & 31);
  const int ci = mycol % nx, cj = mycol / nx;
  const int jm = (cj > 0) ? -nx : nx * (ny - 1), jp = (cj < ny - 1) ? nx : -nx * (ny - 1);
  for (int t = threadIdx.x; t < nz * 32; t += LJ2_T) {
    const int k = t >> 5;
    float rhs = 0.0f;
    if (mycol < ncol) {
      const int c = mycol + plane * k;
      rhs = b[c];
      if (!zero_init) {
        float nb = L.cy * (ei[c + jm] + ei[c + jp]);
        if (ci > 0) nb += L.cx * ei[c - 1];
        if (ci < nx - 1) nb += L.cx * ei[c + 1];
        rhs += nb;
      }
    }
    buf[t] = rhs;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int col = col0 + threadIdx.x;
    if (col < ncol) {
      const int i = col % nx;
      const int cls = (nx == 1) ? 1 : ((i == 0) ? 0 : ((i == nx - 1) ? 2 : 1));
      const float *th = thomas + (size_t)cls * nz * 2;
      float y = 0.0f;
      for (int k = 0; k < nz; k++) {
        y = (buf[k * 32 + threadIdx.x] + L.cz * y) * th[2 * k + 1];
        buf[k * 32 + threadIdx.x] = y;
      }
      float xn = y;
      for (int k = nz - 2; k >= 0; k--) {
        xn = buf[k * 32 + threadIdx.x] - th[2 * k] * xn;
        buf[k * 32 + threadIdx.x] = xn;
      }
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nz * 32; t += LJ2_T) {
    const int k = t >> 5, col = col0 + (t & 31);
    if (col < ncol) {
      const int c = col + plane * k;
      eo[c] = zero_init ? omega * buf[t] : one_m_omega * ei[c] + omega * buf[t];
    }
  }
}

// FP64: the same sweep with the two substitutions in parallel.  Both are
// recurrences v_k = a_k + m_k v_{k-1} whose multipliers m do not depend on the
// data, so a warp takes 32 columns of one of LJ_W runs of levels, solves it
// from zero, and the value entering the run times the (precomputed) product
// of its multipliers is added once the runs below have been folded: chains of
// nz/8 + 8 dependent FP64 operations instead of nz of two each (23 us at
// 50x25x75 with one warp per block in the substitutions; 75 levels).
// th: per class and level c', 1/den, the forward and the backward product
// from the start of the level's run.
constexpr int LJ_W = 8;
static inline __host__ __device__ int lj_run(int nz) { return (nz + LJ_W - 1) / LJ_W; }

__global__ void __launch_bounds__(32 * LJ_W)
    k_line_jacobi3(LevArgs<double> L, double omega, double one_m_omega, int zero_init,
                   const double *__restrict__ thomas, const double *__restrict__ b, const double *__restrict__ ei,
                   double *__restrict__ eo) {
  extern __shared__ __align__(16) unsigned char lj3_raw[];
  double *buf = reinterpret_cast<double *>(lj3_raw);  // [nz][32]
  __shared__ double se[LJ_W][32], sp[LJ_W][32];       // a run's end from zero, and its product
  const int nx = L.nx, ny = L.ny, nz = L.nz, ncol = nx * ny, plane = nx * ny;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int col = min(blockIdx.x * 32 + lane, ncol - 1);  // past the end: the last column again, not stored
  const bool own = blockIdx.x * 32 + lane < ncol;
  const int i = col % nx, j = col / nx;
  const int jm = (j > 0) ? -nx : nx * (ny - 1), jp = (j < ny - 1) ? nx : -nx * (ny - 1);
  const int cls = (nx == 1) ? 1 : ((i == 0) ? 0 : ((i == nx - 1) ? 2 : 1));
  const double *th = thomas + (size_t)cls * nz * 4;
  const int run = lj_run(nz), k0 = min(w * run, nz), k1 = min(k0 + run, nz);
  double y = 0.0;
  for (int k = k0; k < k1; k++) {
    const int c = col + plane * k;
    double rhs = b[c];
    if (!zero_init) {
      double nb = L.cy * (ei[c + jm] + ei[c + jp]);
      if (i > 0) nb = fma(L.cx, ei[c - 1], nb);
      if (i < nx - 1) nb = fma(L.cx, ei[c + 1], nb);
      rhs += nb;
    }
    y = fma(L.cz, y, rhs) * th[4 * k + 1];
    buf[k * 32 + lane] = y;
  }
  se[w][lane] = y;
  sp[w][lane] = k1 > k0 ? th[4 * (k1 - 1) + 2] : 1.0;
  __syncthreads();
  double in = 0.0;  // y entering this run
  for (int v = 0; v < w; v++) in = fma(sp[v][lane], in, se[v][lane]);
  __syncthreads();
  double x = 0.0;  // from the top of the run down, zero above it
  for (int k = k1 - 1; k >= k0; k--) {
    const double yk = fma(th[4 * k + 2], in, buf[k * 32 + lane]);
    x = (k < nz - 1) ? fma(-th[4 * k], x, yk) : yk;
    buf[k * 32 + lane] = x;
  }
  se[w][lane] = x;
  sp[w][lane] = k1 > k0 ? th[4 * k0 + 3] : 1.0;
  __syncthreads();
  in = 0.0;
  for (int v = LJ_W - 1; v > w; v--) in = fma(sp[v][lane], in, se[v][lane]);
  for (int k = k0; k < k1; k++) {
    const int c = col + plane * k;
    const double v = omega * fma(th[4 * k + 3], in, buf[k * 32 + lane]);
    if (own) eo[c] = zero_init ? v : fma(one_m_omega, ei[c], v);
  }
}

// point kernels of the V-cycle run on 3-D grids of 32x8 blocks (x, y) and
// one z plane per grid z index
constexpr int MG_BX = 32, MG_BY = 8;
static inline dim3 mg_grid(int nx, int ny, int nz) {
  return dim3((nx + MG_BX - 1) / MG_BX, (ny + MG_BY - 1) / MG_BY, nz);
}

// Red-black Gauss-Seidel half-sweep for near-isotropic levels (where
// z-lines buy nothing): points with (i + j + k) % 2 == colour get
// e = (b + sum of neighbour couplings) / diagonal; with `copy`, the other
// colour is copied from ein to eout so that eout holds the whole iterate.
// One thread per x pair.  zero_init: ein is zero (first half-sweep from a
// zero start).
template <typename R>
struct InvD {
  R v[3][3];
};

template <typename R>
__global__ void k_rbgs(LevArgs<R> L, InvD<R> inv, int colour, int zero_init, int copy, const R *__restrict__ b,
                       const R *ein, R *eout) {
  const int nx = L.nx, ny = L.ny, nz = L.nz;
  const int i2 = blockIdx.x * MG_BX + threadIdx.x, j = blockIdx.y * MG_BY + threadIdx.y, k = blockIdx.z;
  if (2 * i2 >= nx || j >= ny) return;
  const int plane = nx * ny;
  const int jm = (j > 0) ? -nx : nx * (ny - 1), jp = (j < ny - 1) ? nx : -nx * (ny - 1);
  const int zc = (nz == 1) ? 1 : ((k == 0) ? 0 : ((k == nz - 1) ? 2 : 1));
  for (int q = 0; q < 2; q++) {
    const int i = 2 * i2 + q;
    if (i >= nx) break;
    const int c = i + nx * j + plane * k;
    if (((i + j + k) & 1) == colour) {
      R acc = b[c];
      if (!zero_init) {
        R sx = (R)0, sz = (R)0;
        if (i > 0) sx += ein[c - 1];
        if (i < nx - 1) sx += ein[c + 1];
        if (k > 0) sz += ein[c - plane];
        if (k < nz - 1) sz += ein[c + plane];
        acc = fma(L.cx, sx, acc);
        acc = fma(L.cy, ein[c + jm] + ein[c + jp], acc);
        acc = fma(L.cz, sz, acc);
      }
      const int xc = (nx == 1) ? 1 : ((i == 0) ? 0 : ((i == nx - 1) ? 2 : 1));
      eout[c] = acc * inv.v[xc][zc];
    } else if (copy) {
      eout[c] = ein[c];
    }
  }
}

template <typename R>
__global__ void k_residual(LevArgs<R> L, const R *__restrict__ b, const R *__restrict__ e, R *__restrict__ r) {
  const int nx = L.nx, ny = L.ny, nz = L.nz;
  const int i = blockIdx.x * MG_BX + threadIdx.x, j = blockIdx.y * MG_BY + threadIdx.y, k = blockIdx.z;
  if (i >= nx || j >= ny) return;
  const int c = i + nx * (j + ny * k);
  r[c] = b[c] - applyA<R, R>(e, i, j, k, nx, ny, nz, L.cx, L.cy, L.cz);
}

// 1-D restriction stencil: fine indices and weights contributing to coarse c
template <typename R>
__device__ __forceinline__ int rstencil(int c, int nc, int coarsened, int periodic, int *f, R *w) {
  if (!coarsened) {
    f[0] = c;
    w[0] = (R)1;
    return 1;
  }
  const int nf = 2 * nc;
  int m = 0;
  f[m] = 2 * c;
  w[m++] = (!periodic && c == 0) ? (R)1 : (R)0.75;
  f[m] = 2 * c + 1;
  w[m++] = (!periodic && c == nc - 1) ? (R)1 : (R)0.75;
  if (c > 0) { f[m] = 2 * c - 1; w[m++] = (R)0.25; }
  else if (periodic) { f[m] = nf - 1; w[m++] = (R)0.25; }
  if (c < nc - 1) { f[m] = 2 * c + 2; w[m++] = (R)0.25; }
  else if (periodic) { f[m] = 0; w[m++] = (R)0.25; }
  return m;
}

// 1-D prolongation: coarse indices and weights for fine f
template <typename R>
__device__ __forceinline__ int pstencil(int f, int nc, int coarsened, int periodic, int *c, R *w) {
  if (!coarsened) {
    c[0] = f;
    w[0] = (R)1;
    return 1;
  }
  const int c0 = f >> 1;
  int c1 = (f & 1) ? c0 + 1 : c0 - 1;
  if (c1 < 0 || c1 >= nc) {
    if (!periodic) {
      c[0] = c0;
      w[0] = (R)1;
      return 1;
    }
    c1 = (c1 < 0) ? c1 + nc : c1 - nc;
  }
  c[0] = c0;
  w[0] = (R)0.75;
  c[1] = c1;
  w[1] = (R)0.25;
  return 2;
}

// Separable transfers: P = Px (x) Py (x) Pz and R = P^T / 2^d applied one
// axis at a time through intermediate grids, 2 (P) or 4 (R) multiply-adds
// per output point instead of the 8 (P) or 64 (R) of the direct 3-D
// stencils.  (nx, ny, nz) are the output dimensions; the input has the same
// dimensions except `nin` along axis `ax`.
template <typename R>
__global__ void k_prolong_axis(int ax, int periodic, int nx, int ny, int nz, int nin, const R *__restrict__ in,
                               R *__restrict__ out, int add) {
  const int i = blockIdx.x * MG_BX + threadIdx.x, j = blockIdx.y * MG_BY + threadIdx.y, k = blockIdx.z;
  if (i >= nx || j >= ny) return;
  const int f = (ax == 0) ? i : ((ax == 1) ? j : k);
  int cc[2];
  R w[2];
  const int m = pstencil<R>(f, nin, 1, periodic, cc, w);
  const int inx = (ax == 0) ? nin : nx, iny = (ax == 1) ? nin : ny;
  R acc = (R)0;
  for (int q = 0; q < m; q++) {
    const int ii = (ax == 0) ? cc[q] : i, jj = (ax == 1) ? cc[q] : j, kk = (ax == 2) ? cc[q] : k;
    acc = fma(w[q], in[ii + inx * (jj + iny * kk)], acc);
  }
  const int o = i + nx * (j + ny * k);
  out[o] = add ? out[o] + acc : acc;
}

template <typename R>
__global__ void k_restrict_axis(int ax, int periodic, int nx, int ny, int nz, int nin, R scale,
                                const R *__restrict__ in, R *__restrict__ out) {
  const int i = blockIdx.x * MG_BX + threadIdx.x, j = blockIdx.y * MG_BY + threadIdx.y, k = blockIdx.z;
  if (i >= nx || j >= ny) return;
  const int cidx = (ax == 0) ? i : ((ax == 1) ? j : k);
  const int nco = (ax == 0) ? nx : ((ax == 1) ? ny : nz);
  int ff[4];
  R w[4];
  const int m = rstencil<R>(cidx, nco, 1, periodic, ff, w);
  const int inx = (ax == 0) ? nin : nx, iny = (ax == 1) ? nin : ny;
  R acc = (R)0;
  for (int q = 0; q < m; q++) {
    const int ii = (ax == 0) ? ff[q] : i, jj = (ax == 1) ? ff[q] : j, kk = (ax == 2) ? ff[q] : k;
    acc = fma(w[q], in[ii + inx * (jj + iny * kk)], acc);
  }
  out[i + nx * (j + ny * k)] = acc * scale;
}

// coarsest grid: e = Cinv b (the pseudo-inverse and the products stay FP64
// in both forms).  One warp per row, eight rows per block, lanes along the
// row: 4.6 us at 192 unknowns, where one block with a thread per row took 27.8
// us (144 us at 504: every lane on its own row of a 2 MB matrix, one SM's FP64
// pipe, and a chain of 504 dependent FMAs).
constexpr int CSB = 8;
template <typename T>
__global__ void __launch_bounds__(CSB * 32)
    k_coarse_solve(int n, const double *__restrict__ cinv, const T *__restrict__ b, T *__restrict__ e) {
  const int a = blockIdx.x * CSB + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (a >= n) return;
  const double *row = cinv + (size_t)a * n;
  double acc = 0.0;
#pragma unroll 4
  for (int q = lane; q < n; q += 32) {
    if constexpr (sizeof(T) == sizeof(float)) acc = fma(row[q], widen_bits(b[q]), acc);
    else acc = fma(row[q], b[q], acc);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (lane == 0) e[a] = (T)acc;
}

// ---------------------------------------------------------------------------
// host side

static void neumann_basis(int n, std::vector<double> &Q, std::vector<double> &lam) {
  Q.assign((size_t)n * n, 0.0);
  lam.assign(n, 0.0);
  for (int k = 0; k < n; k++) {
    const double c = (k == 0) ? sqrt(1.0 / n) : sqrt(2.0 / n);
    for (int i = 0; i < n; i++) Q[(size_t)k * n + i] = c * cos(M_PI * k * (i + 0.5) / n);
    const double s = sin(M_PI * k / (2.0 * n));
    lam[k] = 4.0 * s * s;
  }
}
static void periodic_basis(int n, std::vector<double> &Q, std::vector<double> &lam) {
  Q.assign((size_t)n * n, 0.0);
  lam.assign(n, 0.0);
  int idx = 0;
  for (int i = 0; i < n; i++) Q[i] = sqrt(1.0 / n);
  lam[idx++] = 0.0;
  for (int m = 1; 2 * m < n; m++) {
    const double s = sin(M_PI * m / n);
    for (int i = 0; i < n; i++) Q[(size_t)idx * n + i] = sqrt(2.0 / n) * cos(2.0 * M_PI * m * i / n);
    lam[idx++] = 4.0 * s * s;
    for (int i = 0; i < n; i++) Q[(size_t)idx * n + i] = sqrt(2.0 / n) * sin(2.0 * M_PI * m * i / n);
    lam[idx++] = 4.0 * s * s;
  }
  if (n % 2 == 0) {
    for (int i = 0; i < n; i++) Q[(size_t)idx * n + i] = (i % 2 == 0) ? sqrt(1.0 / n) : -sqrt(1.0 / n);
    lam[idx++] = 4.0;
  }
}

// dense pseudo-inverse of the separable level operator
static std::vector<double> coarse_pinv(const PLevel &L) {
  std::vector<double> Qx, Qy, Qz, lx, ly, lz;
  neumann_basis(L.nx, Qx, lx);
  periodic_basis(L.ny, Qy, ly);
  neumann_basis(L.nz, Qz, lz);
  const int n = L.n;
  std::vector<double> M((size_t)n * n, 0.0);
  for (int mz = 0; mz < L.nz; mz++)
    for (int my = 0; my < L.ny; my++)
      for (int mx = 0; mx < L.nx; mx++) {
        const double lam = L.cx * lx[mx] + L.cy * ly[my] + L.cz * lz[mz];
        if (mx == 0 && my == 0 && mz == 0) continue;
        const double il = 1.0 / lam;
        std::vector<double> v(n);
        for (int k = 0; k < L.nz; k++)
          for (int j = 0; j < L.ny; j++)
            for (int i = 0; i < L.nx; i++)
              v[i + L.nx * (j + L.ny * k)] =
                  Qx[(size_t)mx * L.nx + i] * Qy[(size_t)my * L.ny + j] * Qz[(size_t)mz * L.nz + k];
        for (int a = 0; a < n; a++) {
          const double va = v[a] * il;
          double *row = &M[(size_t)a * n];
          for (int b = 0; b < n; b++) row[b] += va * v[b];
        }
      }
  return M;
}

// Thomas factors of the z-line matrix per x-class (first, interior, last)
static std::vector<double> thomas_factors(const PLevel &L) {
  std::vector<double> th((size_t)3 * L.nz * 2);
  for (int cls = 0; cls < 3; cls++) {
    double nbx = 2.0;
    if (L.nx == 1) nbx = 0.0;
    else if (cls != 1) nbx = 1.0;
    const double dxy = L.cx * nbx + 2.0 * L.cy;
    double cprev = 0.0;
    for (int k = 0; k < L.nz; k++) {
      double nbz = 2.0;
      if (L.nz == 1) nbz = 0.0;
      else if (k == 0 || k == L.nz - 1) nbz = 1.0;
      const double d = dxy + L.cz * nbz;
      const double den = (k == 0) ? d : d + L.cz * cprev;  // d - a*c'_{k-1}, a = -cz
      const double cp = -L.cz / den;
      th[((size_t)cls * L.nz + k) * 2 + 0] = cp;
      th[((size_t)cls * L.nz + k) * 2 + 1] = 1.0 / den;
      cprev = cp;
    }
  }
  return th;
}
// with the run products of k_line_jacobi3: forward multipliers cz/den (the
// substitution is y_k = (rhs + cz y_{k-1})/den), backward -c'
static std::vector<double> thomas_runs(const PLevel &L) {
  const std::vector<double> th = thomas_factors(L);
  std::vector<double> r((size_t)3 * L.nz * 4);
  const int run = lj_run(L.nz);
  for (int cls = 0; cls < 3; cls++) {
    const double *t = &th[(size_t)cls * L.nz * 2];
    double *o = &r[(size_t)cls * L.nz * 4];
    for (int k0 = 0; k0 < L.nz; k0 += run) {
      const int k1 = k0 + run < L.nz ? k0 + run : L.nz;
      double p = 1.0;
      for (int k = k0; k < k1; k++) {
        p *= L.cz * t[2 * k + 1];
        o[4 * k] = t[2 * k];
        o[4 * k + 1] = t[2 * k + 1];
        o[4 * k + 2] = p;
      }
      p = 1.0;
      for (int k = k1 - 1; k >= k0; k--) {
        p *= k < L.nz - 1 ? -t[2 * k] : 0.0;  // nothing above the last level
        o[4 * k + 3] = p;
      }
    }
  }
  return r;
}

// Sweeps on a coarsest level without a dense inverse, and whether they run by
// modes (FP64): the transforms take about nz + 2 ny operations per point and
// the x recurrences 3 per sweep, against about 9.5 per sweep for the line
// solves, whose serial part (nz dependent pairs of FP64 operations) is what
// they wait for until a level has millions of points.
constexpr int COARSE_SWEEPS = 40;
static bool modes_pay(int nx, int ny, int nz) {
  return nx <= 32 * MODE_PPL && nz + 2 * ny + 3 * COARSE_SWEEPS <= 400;
}

#define PCK(x)                        \
  do {                                \
    cudaError_t e_ = (x);             \
    if (e_ != cudaSuccess) return e_; \
  } while (0)

static cudaError_t lj2_attr() {
  return cudaFuncSetAttribute(k_line_jacobi2, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
}

static size_t mg_dot_blocks(const PLevel &L);

static ModeSweeps mode_sweeps(const PoissonSolver *S, const PLevel &L) {
  return {L.nx, L.ny, L.nz, S->coarse_sweeps, L.cx, L.cy, L.cz, S->omega};
}

cudaError_t poisson_create(const Geo &g, double cx, double cy, double cz, int fp32,
                           PoissonSolver **out) {
  PoissonSolver *S = new PoissonSolver();
  S->fp32 = fp32 ? 1 : 0;
  S->nx = g.nx;
  S->ny = g.ny;
  S->nz = g.nz;
  S->N = g.nx * g.ny * g.nz;
  PLevel L0;
  L0.nx = g.nx;
  L0.ny = g.ny;
  L0.nz = g.nz;
  L0.n = S->N;
  L0.cxs = L0.cys = L0.czs = 0;
  L0.cx = cx;
  L0.cy = cy;
  L0.cz = cz;
  S->lv.push_back(L0);
  while (true) {
    const PLevel &f = S->lv.back();
    if (f.n <= 512) break;
    PLevel c;
    c.cxs = (f.nx % 2 == 0 && f.nx >= 4);
    c.cys = (f.ny % 2 == 0 && f.ny >= 4);
    c.czs = (f.nz % 2 == 0 && f.nz >= 4);
    if (!c.cxs && !c.cys && !c.czs) break;
    c.nx = c.cxs ? f.nx / 2 : f.nx;
    c.ny = c.cys ? f.ny / 2 : f.ny;
    c.nz = c.czs ? f.nz / 2 : f.nz;
    c.n = c.nx * c.ny * c.nz;
    c.cx = c.cxs ? f.cx / 4.0 : f.cx;
    c.cy = c.cys ? f.cy / 4.0 : f.cy;
    c.cz = c.czs ? f.cz / 4.0 : f.cz;
    S->lv.push_back(c);
  }
  if (S->lv.size() == 1 && S->lv[0].n <= 512) S->fp32 = 0;  // one dense FP64 solve: nothing to run in FP32
  const size_t esz = S->fp32 ? sizeof(float) : sizeof(double);
  for (size_t l = 0; l < S->lv.size(); l++) {
    PLevel &L = S->lv[l];
    {
      const double cmax = fmax(fmax(L.cx, L.cy), L.cz), cmin = fmin(fmin(L.cx, L.cy), L.cz);
      // red-black needs an even periodic y extent (j = 0 and ny - 1 are
      // neighbours); otherwise, or when z couplings dominate, z-lines
      L.point = (cmax <= 2.0 * cmin && L.ny % 2 == 0) ? 1 : 0;
      for (int a = 0; a < 3; a++)
        for (int q = 0; q < 3; q++) {
          const double nbx = (L.nx == 1) ? 0.0 : ((a == 1) ? 2.0 : 1.0);
          const double nbz = (L.nz == 1) ? 0.0 : ((q == 1) ? 2.0 : 1.0);
          L.invd[a][q] = 1.0 / (L.cx * nbx + 2.0 * L.cy + L.cz * nbz);
        }
      if (l + 1 < S->lv.size()) {
        const PLevel &c = S->lv[l + 1];
        L.halved = L.point && c.cxs && c.cys && c.czs;
        L.planar = L.point && c.cxs && c.cys && !c.czs && !S->fp32;
      }
    }
    const size_t bytes = esz * (size_t)L.n;
    if (l > 0) PCK(cudaMalloc(&L.b, bytes));
    if (l > 0) PCK(cudaMalloc(&L.e, bytes));
    if (!L.halved && !L.planar) {
      PCK(cudaMalloc(&L.e2, bytes));
      PCK(cudaMalloc(&L.r, bytes));
      PCK(cudaMalloc(&L.t, bytes));
    }
    if (S->fp32) {
      std::vector<double> th = thomas_factors(L);
      std::vector<float> thf(th.begin(), th.end());
      PCK(cudaMalloc(&L.thomas, thf.size() * sizeof(float)));
      PCK(cudaMemcpy(L.thomas, thf.data(), thf.size() * sizeof(float), cudaMemcpyHostToDevice));
    } else {
      std::vector<double> th = thomas_runs(L);
      PCK(cudaMalloc(&L.thomas, th.size() * sizeof(double)));
      PCK(cudaMemcpy(L.thomas, th.data(), th.size() * sizeof(double), cudaMemcpyHostToDevice));
    }
  }
  if (S->fp32) {
    PCK(lj2_attr());
  } else {
    PCK(cudaFuncSetAttribute(k_line_jacobi3, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  }
  const PLevel &C = S->lv.back();
  if (C.n <= 512) {
    std::vector<double> M = coarse_pinv(C);
    PCK(cudaMalloc(&S->cinv, M.size() * sizeof(double)));
    PCK(cudaMemcpy(S->cinv, M.data(), M.size() * sizeof(double), cudaMemcpyHostToDevice));
  } else {
    S->coarse_sweeps = COARSE_SWEEPS;
    if (!S->fp32 && modes_pay(C.nx, C.ny, C.nz)) {
      std::vector<double> Qz, Qy, lz, ly;
      neumann_basis(C.nz, Qz, lz);
      periodic_basis(C.ny, Qy, ly);
      Qz.insert(Qz.end(), Qy.begin(), Qy.end());
      Qz.insert(Qz.end(), lz.begin(), lz.end());
      Qz.insert(Qz.end(), ly.begin(), ly.end());
      PCK(cudaMalloc(&S->modes, Qz.size() * sizeof(double)));
      PCK(cudaMemcpy(S->modes, Qz.data(), Qz.size() * sizeof(double), cudaMemcpyHostToDevice));
      if (dense_pays(C.nx)) {
        const ModeSweeps M = mode_sweeps(S, C);
        const double *lzd = S->modes + (size_t)C.nz * C.nz + (size_t)C.ny * C.ny;
        PCK(cudaMalloc(&S->dense, sizeof(double) * dense_values(C.nx, C.ny, C.nz)));
        const int half = (C.nx + 1) / 2, warps = half <= 16 ? half : 2 * half;  // both parities per warp, or one
        k_dense_build<<<dim3((warps + MODE_W - 1) / MODE_W, C.nz, mode_classes(C.ny)), 32 * MODE_W>>>(
            M, lzd + C.nz, lzd, S->dense);
        PCK(cudaGetLastError());
        PCK(cudaStreamSynchronize(cudaStreamLegacy));  // before any stream of the context reads them
      }
    }
  }
  const size_t nb = sizeof(double) * (size_t)S->N;
  PCK(cudaMalloc(&S->x, nb));
  PCK(cudaMalloc(&S->r, nb));
  PCK(cudaMalloc(&S->z, S->fp32 ? nb / 2 : nb));
  if (S->fp32) PCK(cudaMalloc((void **)&S->r32, nb / 2));
  PCK(cudaMalloc(&S->p, nb));
  PCK(cudaMalloc(&S->q, nb));
  PCK(cudaMalloc(&S->bvec, nb));
  PCK(cudaMalloc(&S->bin, sizeof(double) * (size_t)g.ny * g.nz));
  // Blocks of the reductions: 8 per SM on 152 SMs, which hide the loads of a
  // large grid (7 iterations at 256x128x192: 5110 us, 5210 with 4 per SM); FP64,
  // below 2M points, 4, half the blocks' own sums (15 iterations at 100x50x75:
  // 3665 us with 8, 3510 with 4; 6 at 128x64x96: 1490, 1450).  (The FP32 form
  // keeps one order of its sums for every size.)
  const int rb = (!S->fp32 && S->N < 2000000) ? 608 : 1216;
  S->rblk = nblocks(S->N) < rb ? nblocks(S->N) : rb;
  {
    size_t np = (size_t)S->rblk * 3;  // reductions of up to three sums, or one partial per block of k_mg_half_dot
    if (S->lv[0].halved || S->lv[0].planar) {
      const size_t nb = S->fp32 ? 0 : mg_dot_blocks(S->lv[0]);
      if (nb > np) np = nb;
    }
    PCK(cudaMalloc(&S->part, sizeof(double) * np));
  }
  PCK(cudaMalloc(&S->counter, sizeof(unsigned)));
  PCK(cudaMemset(S->counter, 0, sizeof(unsigned)));
  PCK(cudaMalloc(&S->s, sizeof(double) * S_COUNT));
  PCK(cudaMemset(S->s, 0, sizeof(double) * S_COUNT));
  PCK(cudaMallocHost(&S->s_host, sizeof(double) * S_COUNT));
  *out = S;
  return cudaSuccess;
}

void poisson_destroy(PoissonSolver *S) {
  if (!S) return;
  for (PLevel &L : S->lv) {
    cudaFree(L.b);
    cudaFree(L.e);
    cudaFree(L.e2);
    cudaFree(L.r);
    cudaFree(L.t);
    cudaFree(L.thomas);
  }
  cudaFree(S->cinv);
  cudaFree(S->modes);
  cudaFree(S->dense);
  cudaFree(S->x);
  cudaFree(S->r);
  cudaFree(S->z);
  cudaFree(S->r32);
  cudaFree(S->p);
  cudaFree(S->q);
  cudaFree(S->bvec);
  cudaFree(S->bin);
  cudaFree(S->part);
  cudaFree(S->counter);
  cudaFree(S->s);
  cudaFreeHost(S->s_host);
  if (S->side) cudaStreamDestroy(S->side);
  delete S;
}

int poisson_levels(const PoissonSolver *S) { return (int)S->lv.size(); }

size_t poisson_footprint(const Geo &g, int fp32, size_t (*rnd)(size_t)) {
  // the level sizes poisson_create builds, without allocating
  const size_t esz = fp32 ? sizeof(float) : sizeof(double);
  size_t tot = 0;
  int nx = g.nx, ny = g.ny, nz = g.nz, l = 0;
  while (true) {
    const size_t n = (size_t)nx * ny * nz;
    tot += (l > 0 ? 5 : 4) * rnd(esz * n) + rnd(esz * 3 * nz * (fp32 ? 2 : 4));
    if (n <= 512) {
      tot += rnd(sizeof(double) * n * n);
      break;
    }
    const int cx = (nx % 2 == 0 && nx >= 4), cy = (ny % 2 == 0 && ny >= 4), cz = (nz % 2 == 0 && nz >= 4);
    if (!cx && !cy && !cz) {
      if (!fp32 && modes_pay(nx, ny, nz)) {
        tot += rnd(sizeof(double) * ((size_t)nz * nz + (size_t)ny * ny + nz + ny));
        if (dense_pays(nx)) tot += rnd(sizeof(double) * dense_values(nx, ny, nz));
      }
      break;
    }
    nx = cx ? nx / 2 : nx;
    ny = cy ? ny / 2 : ny;
    nz = cz ? nz / 2 : nz;
    l++;
  }
  const size_t N = (size_t)g.nx * g.ny * g.nz;
  tot += 6 * rnd(sizeof(double) * N) + rnd(sizeof(double) * (size_t)g.ny * g.nz);
  // reduction partials: three sums of 1216 blocks, or one of every block that forms r.z, at most one per 16 x 4 x 4
  // points while there are few and one per 32 x 8 x 4 beyond
  const size_t blk = (size_t)(g.nx / 32 + 1) * (g.ny / 8 + 1) * (g.nz / 4 + 1);
  tot += rnd(sizeof(double) * (blk > 8 * 1216 ? blk : 8 * 1216)) + rnd(sizeof(unsigned)) + rnd(sizeof(double) * S_COUNT);
  return tot;
}

template <typename R>
static LevArgs<R> largs(const PLevel &L) {
  LevArgs<R> a;
  a.nx = L.nx;
  a.ny = L.ny;
  a.nz = L.nz;
  a.cx = (R)L.cx;
  a.cy = (R)L.cy;
  a.cz = (R)L.cz;
  return a;
}

static void line_sweep(const PLevel &L, double w, double w1, int zero_init, const double *b, const double *ei,
                       double *eo, cudaStream_t st) {
  const LevArgs<double> A = largs<double>(L);
  const double *th = static_cast<const double *>(L.thomas);
  const size_t smem = sizeof(double) * 32 * (size_t)L.nz;
  if (smem <= 200 * 1024)
    k_line_jacobi3<<<(L.nx * L.ny + 31) / 32, 32 * LJ_W, smem, st>>>(A, w, w1, zero_init, th, b, ei, eo);
  else
    k_line_jacobi<double, 4><<<(L.nx * L.ny + LJB - 1) / LJB, LJB, 0, st>>>(A, w, w1, zero_init, th, b, ei,
                                                                           static_cast<double *>(L.t), eo);
}
static void line_sweep(const PLevel &L, float w, float w1, int zero_init, const float *b, const float *ei, float *eo,
                       cudaStream_t st) {
  const LevArgs<float> A = largs<float>(L);
  const float *th = static_cast<const float *>(L.thomas);
  const size_t smem = sizeof(float) * 32 * (size_t)L.nz;
  if (smem <= 200 * 1024)
    k_line_jacobi2<<<(L.nx * L.ny + 31) / 32, LJ2_T, smem, st>>>(A, w, w1, zero_init, th, b, ei, eo);
  else
    k_line_jacobi<float, 2><<<(L.nx * L.ny + LJB - 1) / LJB, LJB, 0, st>>>(A, w, w1, zero_init, th, b, ei,
                                                                          static_cast<float *>(L.t), eo);
}

// The coarsest level's sweeps by modes: b -> e; t and u are scratch of the
// level's size.
template <int PPL>
static void mode_lines(const ModeSweeps &M, const double *Qy, const double *ly, const double *lz, const double *t,
                       double *u, cudaStream_t st) {
  k_mode_lines<PPL><<<dim3((M.ny + MODE_W - 1) / MODE_W, M.nz), 32 * MODE_W, 0, st>>>(M, Qy, ly, lz, t, u);
}
static cudaError_t coarse_modes(const PoissonSolver *S, const PLevel &L, const double *b, double *t, double *u,
                                double *e, cudaStream_t st, long *nl) {
  const ModeSweeps M = mode_sweeps(S, L);
  const double *Qz = S->modes, *Qy = Qz + (size_t)L.nz * L.nz, *lz = Qy + (size_t)L.ny * L.ny, *ly = lz + L.nz;
  const int ncol = L.nx * L.ny, gc = (ncol + 31) / 32;
  constexpr int T = 32 * MODE_W;
  auto blocks = [](int warps) { return (warps + MODE_W - 1) / MODE_W; };
  const int m4 = 2 * ((L.nz + 7) / 8), m1 = 2 * ((L.nz + 1) / 2);  // groups of four modes of one parity, of one
  if (gc * m4 >= MODE_WARPS) k_modes_z<4><<<dim3(gc, blocks(m4)), T, 0, st>>>(L.nz, ncol, Qz, b, t);
  else k_modes_z<1><<<dim3(gc, blocks(m1)), T, 0, st>>>(L.nz, ncol, Qz, b, t);
  const dim3 lines((L.ny + MODE_W - 1) / MODE_W, L.nz);
  if (S->dense && L.nx <= 32) k_mode_dense<false><<<lines, T, 0, st>>>(L.nx, L.ny, L.nz, Qy, S->dense, t, u);
  else if (S->dense) k_mode_dense<true><<<lines, T, 0, st>>>(L.nx, L.ny, L.nz, Qy, S->dense, t, u);
  else if (L.nx <= 128) mode_lines<4>(M, Qy, ly, lz, t, u, st);
  else mode_lines<MODE_PPL>(M, Qy, ly, lz, t, u, st);
  const int gi = (L.nx + 31) / 32, r4 = (L.ny + 3) / 4;
  if (gi * r4 * L.nz >= MODE_WARPS) k_points_y<4><<<dim3(gi, blocks(r4), L.nz), T, 0, st>>>(L.nx, L.ny, Qy, u, t);
  else k_points_y<1><<<dim3(gi, blocks(L.ny), L.nz), T, 0, st>>>(L.nx, L.ny, Qy, u, t);
  const int p1 = (L.nz + 1) / 2, p2 = (p1 + 1) / 2;  // pairs of points
  if (gc * p2 >= MODE_WARPS) k_points_z<2><<<dim3(gc, blocks(p2)), T, 0, st>>>(L.nz, ncol, Qz, t, e);
  else k_points_z<1><<<dim3(gc, blocks(p1)), T, 0, st>>>(L.nz, ncol, Qz, t, e);
  *nl += 4;
  return cudaGetLastError();
}
static cudaError_t coarse_modes(const PoissonSolver *, const PLevel &, const float *, float *, float *, float *,
                                cudaStream_t, long *) {
  return cudaErrorInvalidValue;  // FP32 levels keep the sweeps
}

// R = P^T / 2^d over the coarsened axes in the order x, y, z; the
// intermediate grids live in the fine level's scratch t (n values: the
// first intermediate uses its first n/2, the second the next n/4).
template <typename R>
static cudaError_t restrict_chain(const PLevel &F, const PLevel &C, const R *rf, R *t, R *bc, cudaStream_t st,
                                  long *nl) {
  int d[3] = {F.nx, F.ny, F.nz};
  const int cd[3] = {C.nx, C.ny, C.nz};
  const int cs[3] = {C.cxs, C.cys, C.czs};
  int last = -1, nax = 0;
  for (int a = 0; a < 3; a++)
    if (cs[a]) last = a, nax++;
  const R scale = (R)(1.0 / (double)(1 << nax));
  const R *src = rf;
  R *bufs[2] = {t, t + (size_t)F.n / 2};
  int b = 0;
  for (int a = 0; a < 3; a++) {
    if (!cs[a]) continue;
    const int nin = d[a];
    d[a] = cd[a];
    R *dst = (a == last) ? bc : bufs[b++];
    k_restrict_axis<R><<<mg_grid(d[0], d[1], d[2]), dim3(MG_BX, MG_BY), 0, st>>>(
        a, a == 1, d[0], d[1], d[2], nin, (a == last) ? scale : (R)1, src, dst);
    (*nl)++;
    src = dst;
  }
  return cudaGetLastError();
}

// ef += P ec over the coarsened axes in the order z, y, x.
template <typename R>
static cudaError_t prolong_chain(const PLevel &F, const PLevel &C, const R *ec, R *t, R *ef, cudaStream_t st,
                                 long *nl) {
  int d[3] = {C.nx, C.ny, C.nz};
  const int fd[3] = {F.nx, F.ny, F.nz};
  const int cs[3] = {C.cxs, C.cys, C.czs};
  int last = -1;
  for (int a = 2; a >= 0; a--)
    if (cs[a]) last = a;
  const R *src = ec;
  R *bufs[2] = {t + (size_t)F.n / 2, t};  // the smaller intermediate first
  int b = 0;
  for (int a = 2; a >= 0; a--) {
    if (!cs[a]) continue;
    const int nin = d[a];
    d[a] = fd[a];
    const bool fin = (a == last);
    R *dst = fin ? ef : bufs[b++];
    k_prolong_axis<R><<<mg_grid(d[0], d[1], d[2]), dim3(MG_BX, MG_BY), 0, st>>>(a, a == 1, d[0], d[1], d[2], nin,
                                                                                src, dst, fin ? 1 : 0);
    (*nl)++;
    src = dst;
  }
  return cudaGetLastError();
}

template <typename R>
static InvD<R> invd_of(const PLevel &L) {
  InvD<R> v;
  for (int a = 0; a < 3; a++)
    for (int q = 0; q < 3; q++) v.v[a][q] = (R)L.invd[a][q];
  return v;
}

template <typename R>
static MgLev<R> mglev(const PLevel &L) {
  MgLev<R> m;
  m.nx = L.nx;
  m.ny = L.ny;
  m.nz = L.nz;
  m.cx = (R)L.cx;
  m.cy = (R)L.cy;
  m.cz = (R)L.cz;
  for (int a = 0; a < 3; a++)
    for (int q = 0; q < 3; q++) {
      m.inv[a][q] = (R)L.invd[a][q];
      m.tx[a][q] = (R)(L.cx * L.invd[a][q]);
      m.ty[a][q] = (R)(L.cy * L.invd[a][q]);
      m.tz[a][q] = (R)(L.cz * L.invd[a][q]);
    }
  return m;
}

// Levels a thread of the k_mg_* pair kernels marches: 8 where the level
// still gives 8 blocks of 256 threads per SM (152), fewer below, so that the
// coarse levels, which are short of blocks, spread over the SMs.  Even.
static int mg_columns(const PLevel &L) {
  return ((L.nx / 2 + MGP_X - 1) / MGP_X) * ((L.ny + MGP_Y - 1) / MGP_Y);
}
static int mg_kz(const PLevel &L) {
  int kz = 8;
  while (kz > 2 && mg_columns(L) * ((L.nz + kz - 1) / kz) < 8 * 152) kz /= 2;
  return kz;
}
static int mg_blocks(const PLevel &L, int kz) { return mg_columns(L) * ((L.nz + kz - 1) / kz); }

// Which form a halved level takes: levels of more points run the five passes
// (fewest operations), smaller ones the two tile launches.
constexpr int MG_SPLIT64 = 200000, MG_SPLIT32 = 300000;
template <typename R>
static bool mg_split(const PLevel &L) {
  return L.n > (sizeof(R) == sizeof(double) ? MG_SPLIT64 : MG_SPLIT32);
}
static int mg_tiles(const PLevel &L, int cx, int cy, int cz) {
  return ((L.nx / 2 + cx - 1) / cx) * ((L.ny / 2 + cy - 1) / cy) * ((L.nz / 2 + cz - 1) / cz);
}
// blocks of the launch that forms r.z on the finest level (FP64)
static size_t mg_dot_blocks(const PLevel &L) {
  return (L.planar || mg_split<double>(L)) ? mg_blocks(L, mg_kz(L)) : mg_tiles(L, 8, 2, 2);
}

// pre-smoothing from a zero start into e2: z-line Jacobi, or red then black
template <typename R>
static void pre_smooth(const PLevel &L, R w, R w1, const R *b, R *e2, cudaStream_t st, long *nl) {
  if (!L.point) {
    line_sweep(L, w, w1, 1, b, nullptr, e2, st);
    (*nl)++;
    return;
  }
  const LevArgs<R> A = largs<R>(L);
  const dim3 grd = mg_grid((L.nx + 1) / 2, L.ny, L.nz);
  k_rbgs<R><<<grd, dim3(MG_BX, MG_BY), 0, st>>>(A, invd_of<R>(L), 0, 1, 0, b, e2, e2);
  k_rbgs<R><<<grd, dim3(MG_BX, MG_BY), 0, st>>>(A, invd_of<R>(L), 1, 0, 0, b, e2, e2);
  *nl += 2;
}

// post-smoothing of e2 into res: z-line Jacobi, or black (in place) then red
// (with the black values copied), the adjoint order of the pre-smoothing
template <typename R>
static void post_smooth(const PLevel &L, R w, R w1, const R *b, R *e2, R *res, cudaStream_t st, long *nl) {
  if (!L.point) {
    line_sweep(L, w, w1, 0, b, e2, res, st);
    (*nl)++;
    return;
  }
  const LevArgs<R> A = largs<R>(L);
  const dim3 grd = mg_grid((L.nx + 1) / 2, L.ny, L.nz);
  k_rbgs<R><<<grd, dim3(MG_BX, MG_BY), 0, st>>>(A, invd_of<R>(L), 1, 0, 0, b, e2, e2);
  k_rbgs<R><<<grd, dim3(MG_BX, MG_BY), 0, st>>>(A, invd_of<R>(L), 0, 0, 1, b, e2, res);
  *nl += 2;
}

// Coarse levels per block of k_mg_restrict: up to 8 while every SM keeps four
// blocks (each block also forms the residual of two fine levels of its
// neighbours).
static void mg_restrict_grid(const PLevel &L, int ncz, int *czb, int *blocks) {
  const int gxy = ((L.nx + MGR_FX - 1) / MGR_FX) * ((L.ny + MGR_FY - 1) / MGR_FY);
  *czb = 8;
  while (*czb > 1 && gxy * ((ncz + *czb - 1) / *czb) < 4 * 152) *czb /= 2;
  *blocks = gxy * ((ncz + *czb - 1) / *czb);
}

// b -> the coarse right-hand side bc (ncz levels); the five-pass form keeps
// the pre-smoothed iterate in e.
template <typename R>
static cudaError_t mg_down_level(const MgLev<R> &M, const PLevel &L, int ncz, const R *b, R *e, R *bc,
                                 cudaStream_t st, long *nl) {
  if (mg_split<R>(L)) {
    const int kz = mg_kz(L);
    int czb, nb;
    mg_restrict_grid(L, ncz, &czb, &nb);
    if constexpr (sizeof(R) == sizeof(double)) k_mg_black<<<mg_blocks(L, kz), 256, 0, st>>>(M, b, e, kz);
    else k_mg_pre<<<mg_blocks(L, kz), 256, 0, st>>>(M, b, e, kz);
    k_mg_restrict<R, true><<<nb, 256, 0, st>>>(M, b, e, bc, czb);
    *nl += 2;
  } else {
    k_mg_down<R, 8, 2, 2><<<mg_tiles(L, 8, 2, 2), 256, 0, st>>>(M, b, bc);
    *nl += 1;
  }
  return cudaGetLastError();
}

// The five passes of a level whose z axis is not coarsened (FP64), in place of
// ten launches of the general ones: 34 us instead of 70 at 100x50x75.
static cudaError_t mg_down_planar(const PLevel &L, const double *b, double *e, double *bc, cudaStream_t st, long *nl) {
  const MgLev<double> M = mglev<double>(L);
  const int kz = mg_kz(L);
  int czb, nb;
  mg_restrict_grid(L, L.nz, &czb, &nb);
  k_mg_black<<<mg_blocks(L, kz), 256, 0, st>>>(M, b, e, kz);
  k_mg_restrict<double, false><<<nb, 256, 0, st>>>(M, b, e, bc, czb);
  *nl += 2;
  return cudaGetLastError();
}
static cudaError_t mg_up_planar(PoissonSolver *S, const PLevel &L, bool finest, const double *b, const double *ec,
                                double *e, cudaStream_t st, long *nl) {
  const MgLev<double> M = mglev<double>(L);
  const int kz = mg_kz(L), nb = mg_blocks(L, kz);
  k_mg_prolong<false><<<nb, 256, 0, st>>>(M, b, ec, e, kz);
  k_mg_half<<<nb, 256, 0, st>>>(M, 1, b, e, kz);
  if (finest) k_mg_half_dot<<<nb, PB, 0, st>>>(M, b, e, kz, S->part, S->counter, S->s);
  else k_mg_half<<<nb, 256, 0, st>>>(M, 0, b, e, kz);
  *nl += 3;
  return cudaGetLastError();
}
// (FP32 levels of that kind keep the general passes.)
static cudaError_t mg_down_planar(const PLevel &, const float *, float *, float *, cudaStream_t, long *) {
  return cudaErrorInvalidValue;
}
static cudaError_t mg_up_planar(PoissonSolver *, const PLevel &, bool, const float *, const float *, float *,
                                cudaStream_t, long *) {
  return cudaErrorInvalidValue;
}

// b and the coarse correction ec -> e; FP64: on the finest level r.z too.
static cudaError_t mg_up_level(PoissonSolver *S, const MgLev<double> &M, const PLevel &L, bool finest,
                               const double *b, const double *ec, double *e, cudaStream_t st, long *nl) {
  if (mg_split<double>(L)) {
    const int kz = mg_kz(L), nb = mg_blocks(L, kz);
    k_mg_prolong<true><<<nb, 256, 0, st>>>(M, b, ec, e, kz);
    k_mg_half<<<nb, 256, 0, st>>>(M, 1, b, e, kz);
    if (finest) k_mg_half_dot<<<nb, PB, 0, st>>>(M, b, e, kz, S->part, S->counter, S->s);
    else k_mg_half<<<nb, 256, 0, st>>>(M, 0, b, e, kz);
    *nl += 3;
  } else {
    const int nb = mg_tiles(L, 8, 2, 2);
    if (finest) k_mg_up_dot<8, 2, 2><<<nb, PB, 0, st>>>(M, b, ec, e, S->part, S->counter, S->s);
    else k_mg_up<double, 8, 2, 2><<<nb, 256, 0, st>>>(M, b, ec, e);
    *nl += 1;
  }
  return cudaGetLastError();
}
static cudaError_t mg_up_level(PoissonSolver *, const MgLev<float> &M, const PLevel &L, bool, const float *b,
                               const float *ec, float *e, cudaStream_t st, long *nl) {
  if (mg_split<float>(L)) {
    const int kz = mg_kz(L), nb = mg_blocks(L, kz);
    k_mg_prolong32<<<nb, 256, 0, st>>>(M, b, ec, e, kz);
    k_mg_half<<<nb, 256, 0, st>>>(M, 1, b, e, kz);
    k_mg_half<<<nb, 256, 0, st>>>(M, 0, b, e, kz);
    *nl += 3;
  } else {
    k_mg_up<float, 8, 2, 2><<<mg_tiles(L, 8, 2, 2), 256, 0, st>>>(M, b, ec, e);
    *nl += 1;
  }
  return cudaGetLastError();
}

// r.z and beta of the preconditioned residual out.
static cudaError_t mg_dot(PoissonSolver *S, const double *out, cudaStream_t st, long *nl) {
  if (S->lv.size() > 1 && (S->lv[0].halved || S->lv[0].planar)) return cudaSuccess;  // formed on the way up
  k_rdot<<<S->rblk, PB, 0, st>>>(S->N, S->r, out, S->part, S->counter, S->s);
  (*nl)++;
  return cudaGetLastError();
}
static cudaError_t mg_dot(PoissonSolver *S, const float *out, cudaStream_t st, long *nl) {
  k_zdot<<<S->rblk, PB, 0, st>>>(S->N, 1.0 / (double)S->N, S->r, out, S->part, S->counter, S->s);
  (*nl)++;
  return cudaGetLastError();
}

// one symmetric V-cycle: out = M b0, and r.z into the CG scalars.  A level
// whose axes are all coarsened, or all but z, runs the k_mg_* kernels in place
// in its result array (L.halved, L.planar); the others pre-smooth into their scratch e2 (one
// damped line-Jacobi sweep from zero, or red-black), restrict the residual,
// add the prolonged coarse correction into e2 and post-smooth into the
// result (out on the finest level, e elsewhere).  R: level type.
template <typename R>
static cudaError_t vcycle(PoissonSolver *S, const R *b0, R *out, cudaStream_t st, long *nl) {
  const int nlev = (int)S->lv.size();
  const R w = (R)S->omega, w1 = (R)(1.0 - S->omega);
  auto lvp = [](void *p) { return static_cast<R *>(p); };
  for (int l = 0; l < nlev; l++) {
    PLevel &L = S->lv[l];
    const R *b = (l == 0) ? b0 : lvp(L.b);
    R *res = (l == 0) ? out : lvp(L.e);
    if (l == nlev - 1) {
      if (S->cinv) {
        k_coarse_solve<R><<<(L.n + CSB - 1) / CSB, CSB * 32, 0, st>>>(L.n, S->cinv, b, res);
        (*nl)++;
      } else if (S->modes) {
        PCK(coarse_modes(S, L, b, lvp(L.r), lvp(L.e2), res, st, nl));
      } else {  // no dense inverse: damped line-Jacobi sweeps
        R *cur = lvp(L.e2), *oth = res;
        line_sweep(L, w, w1, 1, b, nullptr, cur, st);
        (*nl)++;
        for (int sw = 1; sw < S->coarse_sweeps; sw++) {
          line_sweep(L, w, w1, 0, b, cur, oth, st);
          (*nl)++;
          R *tmp = cur;
          cur = oth;
          oth = tmp;
        }
        if (cur != res) PCK(cudaMemcpyAsync(res, cur, sizeof(R) * L.n, cudaMemcpyDeviceToDevice, st));
      }
      PCK(cudaGetLastError());
      break;
    }
    const PLevel &C = S->lv[l + 1];
    if (L.halved) {
      const MgLev<R> M = mglev<R>(L);
      PCK(mg_down_level(M, L, C.nz, b, res, lvp(C.b), st, nl));
      continue;
    }
    if (L.planar) {
      PCK(mg_down_planar(L, b, res, lvp(C.b), st, nl));
      continue;
    }
    const LevArgs<R> A = largs<R>(L);
    pre_smooth<R>(L, w, w1, b, lvp(L.e2), st, nl);
    k_residual<R><<<mg_grid(L.nx, L.ny, L.nz), dim3(MG_BX, MG_BY), 0, st>>>(A, b, lvp(L.e2), lvp(L.r));
    *nl += 1;
    PCK(restrict_chain<R>(L, C, lvp(L.r), lvp(L.t), lvp(C.b), st, nl));
    PCK(cudaGetLastError());
  }
  for (int l = nlev - 2; l >= 0; l--) {
    PLevel &L = S->lv[l];
    const PLevel &C = S->lv[l + 1];
    const R *b = (l == 0) ? b0 : lvp(L.b);
    R *res = (l == 0) ? out : lvp(L.e);
    if (L.halved) {
      const MgLev<R> M = mglev<R>(L);
      PCK(mg_up_level(S, M, L, l == 0, b, lvp(C.e), res, st, nl));
    } else if (L.planar) {
      PCK(mg_up_planar(S, L, l == 0, b, lvp(C.e), res, st, nl));
    } else {
      PCK(prolong_chain<R>(L, C, lvp(C.e), lvp(L.t), lvp(L.e2), st, nl));
      post_smooth<R>(L, w, w1, b, lvp(L.e2), res, st, nl);
    }
    PCK(cudaGetLastError());
  }
  return mg_dot(S, out, st, nl);
}

// The solve in three parts: set-up (b, x0 = p_old, r0 and the first
// convergence test), one PCG iteration (V-cycle, z.r, p update, A p, x and r
// updates, convergence test), and the write-back of p with its ghosts.
static cudaError_t solve_begin(PoissonSolver *S, const Geo &g, const Phys &ph, const double *rhs_p,
                               const void *u3, int u3_fp32, const double *u_inlet, const double *pres_old,
                               double rtol, const CgCtl &ctl, cudaStream_t st, long *nl) {
  const int N = S->N, rb = S->rblk;
  const PLevel &F = S->lv[0];
  if (u3_fp32)
    k_build_b<float><<<rb, PB, 0, st>>>(g, (ph.dx / ph.dt) / ph.dy, 1.0 / ph.dy, rhs_p,
                                        static_cast<const float *>(u3), u_inlet, pres_old, S->bvec, S->x, S->bin,
                                        S->part, S->counter, S->s);
  else
    k_build_b<double><<<rb, PB, 0, st>>>(g, (ph.dx / ph.dt) / ph.dy, 1.0 / ph.dy, rhs_p,
                                         static_cast<const double *>(u3), u_inlet, pres_old, S->bvec, S->x, S->bin,
                                         S->part, S->counter, S->s);
  k_init_r<<<rb, PB, 0, st>>>(F.nx, F.ny, F.nz, F.cx, F.cy, F.cz, 1.0 / (double)N, rtol, ctl, S->s, S->bvec,
                              S->x, S->r, S->r32, S->part, S->counter);
  *nl += 2;
  return cudaGetLastError();
}

static cudaError_t solve_iteration(PoissonSolver *S, const CgCtl &ctl, cudaStream_t st, long *nl) {
  const int N = S->N, rb = S->rblk;
  const PLevel &F = S->lv[0];
  if (S->fp32) {
    float *z = static_cast<float *>(S->z);
    PCK(vcycle<float>(S, S->r32, z, st, nl));
    k_pupdate<float><<<nblocks(N), PB, 0, st>>>(N, S->s, z, S->p);
  } else {
    double *z = static_cast<double *>(S->z);
    PCK(vcycle<double>(S, S->r, z, st, nl));
    k_pupdate<double><<<nblocks(N), PB, 0, st>>>(N, S->s, z, S->p);
  }
  if (S->fp32) k_apply_dot<false><<<rb, PB, 0, st>>>(F.nx, F.ny, F.nz, F.cx, F.cy, F.cz, S->p, S->q, S->part, S->counter, S->s);
  else k_apply_dot<true><<<rb, PB, 0, st>>>(F.nx, F.ny, F.nz, F.cx, F.cy, F.cz, S->p, S->q, S->part, S->counter, S->s);
  k_axpy<<<rb, PB, 0, st>>>(N, ctl, S->s, S->p, S->q, S->x, S->r, S->r32, S->part, S->counter);
  *nl += 3;
  return cudaGetLastError();
}

static cudaError_t solve_end(PoissonSolver *S, const Geo &g, const Phys &ph, double *pres, cudaStream_t st,
                             long *nl) {
  k_sumx<<<S->rblk, PB, 0, st>>>(S->N, S->x, S->part, S->counter, S->s);
  dim3 grd((g.nx + 2 + 31) / 32, (g.ny + 2 + 3) / 4, g.nz + 2);
  k_writeback<<<grd, dim3(32, 4), 0, st>>>(g, ph.dy, 1.0 / (double)S->N, S->s, S->x, S->bin, pres);
  *nl += 2;
  return cudaGetLastError();
}

cudaError_t poisson_solve(PoissonSolver *S, const Geo &g, const Phys &ph,
                          const double *rhs_p, const void *u3, int u3_fp32,
                          const double *u_inlet, const double *pres_old,
                          double *pres, double rtol, int maxits, int *its,
                          double *rnorm, double *bnorm, int *reason,
                          cudaStream_t st, long *nl) {
  const CgCtl ctl = {maxits, 0, 0};
  PCK(solve_begin(S, g, ph, rhs_p, u3, u3_fp32, u_inlet, pres_old, rtol, ctl, st, nl));
  while (true) {
    PCK(cudaMemcpyAsync(S->s_host, S->s, sizeof(double) * S_COUNT, cudaMemcpyDeviceToHost, st));
    PCK(cudaStreamSynchronize(st));
    if (S->s_host[S_REASON] != 0.0) break;
    PCK(solve_iteration(S, ctl, st, nl));
  }
  PCK(solve_end(S, g, ph, pres, st, nl));
  *its = (int)S->s_host[S_IT];
  *rnorm = sqrt(S->s_host[S_RR]);
  *bnorm = sqrt(S->s_host[S_BB]);
  *reason = (int)S->s_host[S_REASON];
  return cudaSuccess;
}

cudaError_t poisson_solve_capture(PoissonSolver *S, const Geo &g, const Phys &ph,
                                  const double *rhs_p, const void *u3, int u3_fp32,
                                  const double *u_inlet, const double *pres_old,
                                  double *pres, double rtol, int maxits,
                                  cudaStream_t st, long *nl_static, long *nl_body) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t graph = nullptr;
  PCK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &graph, nullptr, nullptr, nullptr));
  if (cs != cudaStreamCaptureStatusActive || !graph) return cudaErrorStreamCaptureUnmatched;
  CgCtl ctl = {maxits, 1, 0};
  PCK(cudaGraphConditionalHandleCreate(&ctl.cond, graph, 0, 0));
  PCK(solve_begin(S, g, ph, rhs_p, u3, u3_fp32, u_inlet, pres_old, rtol, ctl, st, nl_static));
  const cudaGraphNode_t *deps = nullptr;
  size_t ndeps = 0;
  PCK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &graph, &deps, nullptr, &ndeps));
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = ctl.cond;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t node;
  PCK(cudaGraphAddNode(&node, graph, deps, nullptr, ndeps, &cp));
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  if (!S->side) PCK(cudaStreamCreateWithFlags(&S->side, cudaStreamNonBlocking));
  PCK(cudaStreamBeginCaptureToGraph(S->side, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  const cudaError_t eb = solve_iteration(S, ctl, S->side, nl_body);
  cudaGraph_t out = nullptr;
  const cudaError_t ee = cudaStreamEndCapture(S->side, &out);
  PCK(eb);
  PCK(ee);
  PCK(cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
  return solve_end(S, g, ph, pres, st, nl_static);
}

cudaError_t poisson_read(PoissonSolver *S, cudaStream_t st, int *its, double *rnorm, double *bnorm,
                         int *reason, int *worst, double *its_total) {
  PCK(cudaMemcpyAsync(S->s_host, S->s, sizeof(double) * S_COUNT, cudaMemcpyDeviceToHost, st));
  PCK(cudaStreamSynchronize(st));
  *its = (int)S->s_host[S_IT];
  *rnorm = sqrt(S->s_host[S_RR]);
  *bnorm = sqrt(S->s_host[S_BB]);
  *reason = (int)S->s_host[S_REASON];
  *worst = (int)S->s_host[S_WORST];
  *its_total = S->s_host[S_ITS_TOTAL];
  return cudaSuccess;
}

cudaError_t poisson_reset_worst(PoissonSolver *S, cudaStream_t st) {
  static const double zero = 0.0;
  return cudaMemcpyAsync(S->s + S_WORST, &zero, sizeof(double), cudaMemcpyHostToDevice, st);
}

}  // namespace tpls
