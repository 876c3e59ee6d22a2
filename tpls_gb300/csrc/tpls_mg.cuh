// tpls_mg.cuh -- kernels of the symmetric red-black V-cycle on the levels
// whose three axes are all coarsened, or (FP64) x and y (csrc/k_pressure.cu
// chooses the path).
//
// Red points have (i + j + k) even.  The pre-smoothing starts from zero, red
// then black, so
//   e_red   = b / d,                 e_black = (b + sum c e_red) / d,
// and the residual it leaves is zero at the black points (just relaxed) and
//   r_red   = sum c e_black
// at the red ones (b - d e_red cancels).  After the coarse correction the
// black half-sweep reads red values only and the red one black values only,
// so the correction is needed at the red points alone:
//   e_red   = b / d + P e_c,  e_black = (b + sum c e_red) / d,
//   e_red   = (b + sum c e_black) / d.
// A large FP64 level is therefore five passes, k_mg_black, k_mg_restrict
// (residual and R = P^T/8 in one), k_mg_prolong and two k_mg_half, in place
// in one array instead of thirteen launches over five arrays, with about 18
// instead of 27 operations per point (those levels are bound by the FP64
// pipe).  FP32 levels and short FP64 ones run the same values in two launches
// of tiles (k_mg_down, k_mg_up, below).
//
// In the five passes each thread owns an x pair (2 i2, 2 i2 + 1) of one row and marches kz
// levels: one vector load per level brings the pair, which holds the relaxed
// point's own z neighbours of the levels around it and one x neighbour.
#pragma once
#include "tpls_common.cuh"

namespace tpls {

// a * b, not absorbed into a following sum
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

template <typename R>
struct Pair2;
template <>
struct Pair2<float> {
  using T = float2;
};
template <>
struct Pair2<double> {
  using T = double2;
};

// A level's extents, couplings, 1/diagonal by x and z class (first,
// interior, last) and coupling/diagonal of a neighbour of that class.
template <typename R>
struct MgLev {
  int nx, ny, nz;
  R cx, cy, cz;
  R inv[3][3], tx[3][3], ty[3][3], tz[3][3];
};

constexpr int MGP_X = 32, MGP_Y = 8;  // pairs x rows per block (256 threads)

// One-dimensional grids: block -> (x tile, y tile, chunk of kz levels).
struct MgBlk {
  int i2, j, k0, k1;
  bool in;
};
template <typename R>
__device__ __forceinline__ MgBlk mg_block(const MgLev<R> &L, int kz) {
  const int gx = (L.nx / 2 + MGP_X - 1) / MGP_X, gy = (L.ny + MGP_Y - 1) / MGP_Y;
  const int bx = blockIdx.x % gx, by = (blockIdx.x / gx) % gy, bz = blockIdx.x / (gx * gy);
  MgBlk B;
  B.i2 = bx * MGP_X + (threadIdx.x & 31);
  B.j = by * MGP_Y + (threadIdx.x >> 5);
  B.k0 = bz * kz;
  B.k1 = min(B.k0 + kz, L.nz);
  B.in = 2 * B.i2 < L.nx && B.j < L.ny;
  return B;
}
__device__ __forceinline__ int mg_zc(int k, int nz) { return k == 0 ? 0 : (k == nz - 1 ? 2 : 1); }

// e at the black points from the right-hand side alone (pre-smoothing from
// zero): e = (b + sum (c/d)_n b_n) / d over the red neighbours n.
__global__ void __launch_bounds__(256) k_mg_black(const __grid_constant__ MgLev<double> L, const double *__restrict__ b,
                                                  double *__restrict__ e, int kz) {
  const MgBlk B = mg_block(L, kz);
  if (!B.in) return;
  const int nx = L.nx, plane = nx * L.ny;
  const int jm = (B.j > 0) ? -nx : plane - nx, jp = (B.j < L.ny - 1) ? nx : nx - plane;
  int c = 2 * B.i2 + nx * B.j + plane * B.k0;  // the pair's even point
  const double2 zero = {0.0, 0.0};
  double2 pm = (B.k0 > 0) ? *reinterpret_cast<const double2 *>(b + c - plane) : zero;
  double2 p0 = *reinterpret_cast<const double2 *>(b + c);
  for (int k = B.k0; k < B.k1; k++, c += plane) {
    const double2 pp = (k < L.nz - 1) ? *reinterpret_cast<const double2 *>(b + c + plane) : zero;
    const int odd = 1 - ((B.j + k) & 1);  // the black point: 1 = the pair's odd one
    const int o = c + odd, zc = mg_zc(k, L.nz);
    const int xo = odd ? ((2 * B.i2 + 1 == nx - 1) ? 2 : 1) : (B.i2 == 0 ? 0 : 1);      // its x class
    const int xi = odd ? (B.i2 == 0 ? 0 : 1) : ((2 * B.i2 + 1 == nx - 1) ? 2 : 1);      // its pair's other point
    const bool outer = odd ? (2 * B.i2 + 2 < nx) : (B.i2 > 0);                          // neighbour outside the pair
    double acc = odd ? p0.y : p0.x;
    acc = fma(L.tx[xi][zc], odd ? p0.x : p0.y, acc);
    if (outer) acc = fma(L.tx[1][zc], b[odd ? c + 2 : c - 1], acc);
    acc = fma(L.ty[xo][zc], b[o + jm] + b[o + jp], acc);
    if (k > 0) acc = fma(L.tz[xo][mg_zc(k - 1, L.nz)], odd ? pm.y : pm.x, acc);
    if (k < L.nz - 1) acc = fma(L.tz[xo][mg_zc(k + 1, L.nz)], odd ? pp.y : pp.x, acc);
    e[o] = acc * L.inv[xo][zc];
    pm = p0;
    p0 = pp;
  }
}

// e at the red points = b / d + P e_c.  P is trilinear with weights 3/4 and
// 1/4 per axis (an index beyond a wall falls back on the wall's cell, y
// wraps): 64 P = sum of products of 3 and 1, marched up z with the y- and
// x-combined coarse values of three coarse levels in registers.  Z false: z is
// not coarsened, 16 P in the point's own level.
template <bool Z>
__global__ void __launch_bounds__(256) k_mg_prolong(const __grid_constant__ MgLev<double> L, const double *__restrict__ b,
                                                    const double *__restrict__ ec, double *__restrict__ e, int kz) {
  const MgBlk B = mg_block(L, kz);  // kz even
  if (!B.in) return;
  const int nx = L.nx, plane = nx * L.ny, ncx = nx / 2, ncy = L.ny / 2, ncz = Z ? L.nz / 2 : L.nz;
  const int y0 = B.j >> 1;
  int y1 = (B.j & 1) ? y0 + 1 : y0 - 1;
  y1 = y1 < 0 ? ncy - 1 : (y1 >= ncy ? 0 : y1);
  const int xl = max(B.i2 - 1, 0), xr = min(B.i2 + 1, ncx - 1);
  const double *r0 = ec + ncx * y0, *r1 = ec + ncx * y1;
  // y-combined columns, then the even point's (3 own + left) and the odd
  // point's (3 own + right) x combination at coarse level q
  auto combine = [&](int q, double &ev, double &od) {
    const int o = ncx * ncy * min(max(q, 0), ncz - 1);
    const double h = fma(3.0, r0[o + B.i2], r1[o + B.i2]);
    ev = fma(3.0, h, fma(3.0, r0[o + xl], r1[o + xl]));
    od = fma(3.0, h, fma(3.0, r0[o + xr], r1[o + xr]));
  };
  if constexpr (!Z) {
    int c = 2 * B.i2 + nx * B.j + plane * B.k0;
    for (int k = B.k0; k < B.k1; k++, c += plane) {
      const int odd = (B.j + k) & 1;  // the pair's red point
      double ev, od;
      combine(k, ev, od);
      const int x = odd ? ((2 * B.i2 + 1 == nx - 1) ? 2 : 1) : (B.i2 == 0 ? 0 : 1);
      e[c + odd] = fma(b[c + odd], L.inv[x][mg_zc(k, L.nz)], (odd ? od : ev) * (1.0 / 16.0));
    }
    return;
  }
  const int ja = B.j & 1;  // even level: the red point is the pair's odd one when j is odd
  double em, om, e0, o0, e1, o1;
  combine(B.k0 / 2 - 1, em, om);
  combine(B.k0 / 2, e0, o0);
  int c = 2 * B.i2 + nx * B.j + plane * B.k0;
  const int xe = B.i2 == 0 ? 0 : 1, xo = (2 * B.i2 + 1 == nx - 1) ? 2 : 1;
  for (int k = B.k0; k < B.k1; k += 2) {
    combine(k / 2 + 1, e1, o1);
    const double lo = ja ? fma(3.0, o0, om) : fma(3.0, e0, em);
    const double hi = ja ? fma(3.0, e0, e1) : fma(3.0, o0, o1);
    const int x0 = ja ? xo : xe, x1 = ja ? xe : xo;
    e[c + ja] = fma(b[c + ja], L.inv[x0][mg_zc(k, L.nz)], lo * (1.0 / 64.0));
    const int c1 = c + plane + 1 - ja;
    e[c1] = fma(b[c1], L.inv[x1][mg_zc(k + 1, L.nz)], hi * (1.0 / 64.0));
    em = e0;
    om = o0;
    e0 = e1;
    o0 = o1;
    c += 2 * plane;
  }
}

// One relaxed point of the pair at level k: e = (b + sum c e_n) / d; `odd`:
// which of the pair; pm, p0, pp: the pair at k-1, k, k+1.
template <typename R, typename V2>
__device__ __forceinline__ R mg_relax(const MgLev<R> &L, const MgBlk &B, const R *e, R rhs, int odd, int c, int jm,
                                      int jp, int k, V2 pm, V2 p0, V2 pp) {
  const int nx = L.nx, o = c + odd, zc = mg_zc(k, L.nz);
  const int xo = odd ? ((2 * B.i2 + 1 == nx - 1) ? 2 : 1) : (B.i2 == 0 ? 0 : 1);
  const bool outer = odd ? (2 * B.i2 + 2 < nx) : (B.i2 > 0);
  R sx = odd ? p0.x : p0.y;
  if (outer) sx += e[odd ? c + 2 : c - 1];
  R acc = fma(L.cx, sx, rhs);
  acc = fma(L.cy, e[o + jm] + e[o + jp], acc);
  acc = fma(L.cz, odd ? pm.y + pp.y : pm.x + pp.x, acc);  // zero beyond a wall
  return acc * L.inv[xo][zc];
}

// In-place half-sweep of one colour (0 red, 1 black).
template <typename R>
__global__ void __launch_bounds__(256) k_mg_half(const __grid_constant__ MgLev<R> L, int colour,
                                                 const R *__restrict__ b, R *e, int kz) {
  using V2 = typename Pair2<R>::T;
  const MgBlk B = mg_block(L, kz);
  if (!B.in) return;
  const int nx = L.nx, plane = nx * L.ny;
  const int jm = (B.j > 0) ? -nx : plane - nx, jp = (B.j < L.ny - 1) ? nx : nx - plane;
  int c = 2 * B.i2 + nx * B.j + plane * B.k0;
  const V2 zero = {(R)0, (R)0};
  V2 pm = (B.k0 > 0) ? *reinterpret_cast<const V2 *>(e + c - plane) : zero;
  V2 p0 = *reinterpret_cast<const V2 *>(e + c);
  for (int k = B.k0; k < B.k1; k++, c += plane) {
    const V2 pp = (k < L.nz - 1) ? *reinterpret_cast<const V2 *>(e + c + plane) : zero;
    const int odd = (B.j + k + colour) & 1;
    e[c + odd] = mg_relax(L, B, e, b[c + odd], odd, c, jm, jp, k, pm, p0, pp);
    pm = p0;
    p0 = pp;
  }
}

// FP32 levels of the five passes keep the arithmetic of the general passes:
// e = b / d at the red points, the black ones relaxed from them, both stored
// (the residual reads both).
__global__ void __launch_bounds__(256) k_mg_pre(const __grid_constant__ MgLev<float> L, const float *__restrict__ b,
                                                float *__restrict__ e, int kz) {
  const MgBlk B = mg_block(L, kz);
  if (!B.in) return;
  const int nx = L.nx, nz = L.nz, plane = nx * L.ny;
  const int jm = (B.j > 0) ? -nx : plane - nx, jp = (B.j < L.ny - 1) ? nx : nx - plane;
  int c = 2 * B.i2 + nx * B.j + plane * B.k0;
  const int xe = B.i2 == 0 ? 0 : 1, xo = (2 * B.i2 + 1 == nx - 1) ? 2 : 1;
  const float2 zero = {0.0f, 0.0f};
  float2 pm = (B.k0 > 0) ? *reinterpret_cast<const float2 *>(b + c - plane) : zero;
  float2 p0 = *reinterpret_cast<const float2 *>(b + c);
  for (int k = B.k0; k < B.k1; k++, c += plane) {
    const float2 pp = (k < nz - 1) ? *reinterpret_cast<const float2 *>(b + c + plane) : zero;
    const bool odd = !((B.j + k) & 1);  // the black point: the pair's odd one
    const int o = c + odd, zc = mg_zc(k, nz), xb = odd ? xo : xe, xr = odd ? xe : xo;
    const float red = mul_rn(odd ? p0.x : p0.y, L.inv[xr][zc]);
    float sx = red;
    if (odd ? (2 * B.i2 + 2 < nx) : (B.i2 > 0)) sx += mul_rn(b[odd ? c + 2 : c - 1], L.inv[1][zc]);
    float acc = fmaf(L.cx, sx, odd ? p0.y : p0.x);
    acc = fmaf(L.cy, mul_rn(b[o + jm], L.inv[xb][zc]) + mul_rn(b[o + jp], L.inv[xb][zc]), acc);
    const float zm = mul_rn(odd ? pm.y : pm.x, L.inv[xb][mg_zc(max(k - 1, 0), nz)]);
    const float zp = mul_rn(odd ? pp.y : pp.x, L.inv[xb][mg_zc(min(k + 1, nz - 1), nz)]);
    acc = fmaf(L.cz, zm + zp, acc);
    const float blk = acc * L.inv[xb][zc];
    *reinterpret_cast<float2 *>(e + c) = odd ? make_float2(red, blk) : make_float2(blk, red);
    pm = p0;
    p0 = pp;
  }
}

// One axis of the prolongation: fine index f between its cell and the next
// one on its side; beyond a wall the cell alone.
template <typename R>
__device__ __forceinline__ R mg_lerp(R a, R b, bool wall) {
  return fma(wall ? (R)0 : (R)0.25, b, mul_rn(wall ? (R)1 : (R)0.75, a));
}

// e at the red points: b / d plus the correction interpolated along z, then
// y, then x.
__global__ void __launch_bounds__(256) k_mg_prolong32(const __grid_constant__ MgLev<float> L,
                                                      const float *__restrict__ b, const float *__restrict__ ec,
                                                      float *__restrict__ e, int kz) {
  const MgBlk B = mg_block(L, kz);  // kz even
  if (!B.in) return;
  const int nx = L.nx, nz = L.nz, plane = nx * L.ny, ncx = nx / 2, ncy = L.ny / 2, ncz = nz / 2;
  const int y0 = B.j >> 1;
  int y1 = (B.j & 1) ? y0 + 1 : y0 - 1;
  y1 = y1 < 0 ? ncy - 1 : (y1 >= ncy ? 0 : y1);
  const int xs[3] = {max(B.i2 - 1, 0), B.i2, min(B.i2 + 1, ncx - 1)};
  float cm[6], c0[6], c1[6];  // columns (x left, own, right) of rows y0 and y1 at three coarse levels
  auto load = [&](int q, float (&v)[6]) {
    const float *p = ec + (size_t)ncx * ncy * min(max(q, 0), ncz - 1);
#pragma unroll
    for (int m = 0; m < 3; m++) {
      v[m] = p[ncx * y0 + xs[m]];
      v[3 + m] = p[ncx * y1 + xs[m]];
    }
  };
  load(B.k0 / 2 - 1, cm);
  load(B.k0 / 2, c0);
  const bool ja = B.j & 1;
  int c = 2 * B.i2 + nx * B.j + plane * B.k0;
  const int xe = B.i2 == 0 ? 0 : 1, xo = (2 * B.i2 + 1 == nx - 1) ? 2 : 1;
  for (int k = B.k0; k < B.k1; k += 2) {
    load(k / 2 + 1, c1);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const bool odd = (h == 0) ? ja : !ja;  // the red point: the pair's odd one
      const float(&n)[6] = h == 0 ? cm : c1;
      const bool wz = h == 0 ? k == 0 : k + 1 == nz - 1;
      const float own = mg_lerp(mg_lerp(c0[1], n[1], wz), mg_lerp(c0[4], n[4], wz), false);
      const float oth = mg_lerp(mg_lerp(odd ? c0[2] : c0[0], odd ? n[2] : n[0], wz),
                                mg_lerp(odd ? c0[5] : c0[3], odd ? n[5] : n[3], wz), false);
      const float p = mg_lerp(own, oth, odd ? B.i2 == ncx - 1 : B.i2 == 0);
      const int o = c + h * plane + odd;
      e[o] = mul_rn(b[o], L.inv[odd ? xo : xe][mg_zc(k + h, nz)]) + p;
    }
#pragma unroll
    for (int m = 0; m < 6; m++) {
      cm[m] = c0[m];
      c0[m] = c1[m];
    }
    c += 2 * plane;
  }
}

// Residual after the pre-smoothing and its restriction, R = P^T / 8.  A block
// covers 60 x 14 fine columns (30 x 7 coarse) and marches the fine levels of
// czb coarse ones.  A warp holds 32 x pairs of a row (the tile's 30 and one on
// each side) and two of the 16 rows (one halo row on each side), so x
// neighbours and x taps pass by shuffles, z neighbours stay in registers, and
// only the y taps go through shared memory (double-buffered: one barrier per
// level); the z taps are summed in registers.
// FP64: the residual is zero at the black points, r = sum c e_black at the
// red ones, and two of the four x taps hit red points; taps are 3 and 1 (4
// where a wall reflects the missing one), scaled by 1/512 at the end.  Bound
// by the FP64 pipe (about 6 operations per fine point, halo included).
// FP32 (arithmetic is 64 times cheaper): the residual of every point and all
// taps, by the operations of k_residual and k_restrict_axis in their order,
// equal to theirs bit for bit; bound by its loads.
// Z false (FP64): z is not coarsened, R = P^T / 4 level by level.
constexpr int MGR_FX = 60, MGR_FY = 14;

// Four taps of a coarse point in the general restriction's order; w0, w1: 1
// instead of 3/4 where a wall drops the tap beyond it (which is zero here).
template <typename R>
__device__ __forceinline__ R mg_taps(R w0, R w1, R am, R a0, R a1, R ap) {
  R v = mul_rn(w0, a0);
  v = fma(w1, a1, v);
  v = fma((R)0.25, am, v);
  return fma((R)0.25, ap, v);
}

template <typename R, bool Z>
__global__ void __launch_bounds__(256) k_mg_restrict(const __grid_constant__ MgLev<R> L, const R *__restrict__ b,
                                                     const R *__restrict__ e, R *__restrict__ bc, int czb) {
  using V2 = typename Pair2<R>::T;
  __shared__ R sx[2][MGR_FY + 2][32];
  const int nx = L.nx, ny = L.ny, nz = L.nz, plane = nx * ny;
  const int ncx = nx / 2, ncy = ny / 2, ncz = Z ? nz / 2 : nz;
  const int gx = (nx + MGR_FX - 1) / MGR_FX, gy = (ny + MGR_FY - 1) / MGR_FY;
  const int bx = blockIdx.x % gx, by = (blockIdx.x / gx) % gy, bz = blockIdx.x / (gx * gy);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int ic = bx * (MGR_FX / 2) - 1 + lane;  // the pair's coarse column: fine 2 ic, 2 ic + 1
  const bool col = ic >= 0 && ic < ncx;
  const int y0 = by * MGR_FY;
  const int kc0 = bz * czb, kc1 = min(kc0 + czb, ncz);
  const int ka = Z ? max(2 * kc0 - 1, 0) : kc0, kb = Z ? min(2 * kc1, nz - 1) : kc1 - 1;
  const V2 zero = {(R)0, (R)0};
  // this warp's two rows, 2 w and 2 w + 1 of the tile's 16 (fine y0 - 1 + row; past the grid's end they repeat rows)
  int o[2], om[2], op[2], jl[2];
  V2 em[2], e0[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    int j = y0 - 1 + 2 * w + q;
    j = j < 0 ? ny - 1 : (j >= ny ? (j - ny) % ny : j);
    jl[q] = j;
    o[q] = 2 * ic + nx * j;
    om[q] = 2 * ic + nx * (j > 0 ? j - 1 : ny - 1);
    op[q] = 2 * ic + nx * (j < ny - 1 ? j + 1 : 0);
    em[q] = (col && ka > 0) ? *reinterpret_cast<const V2 *>(e + o[q] + (size_t)plane * (ka - 1)) : zero;
    e0[q] = col ? *reinterpret_cast<const V2 *>(e + o[q] + (size_t)plane * ka) : zero;
  }
  const bool own = lane >= 1 && lane < 31 && col && w < MGR_FY / 2 && y0 / 2 + w < ncy;
  R *out = bc + ic + ncx * (y0 / 2 + w);
  const size_t cplane = (size_t)ncx * ncy;
  // FP64: acc = the coarse level being summed, up = the next one's first tap.  FP32: acc holds taps 2 and 3 (added
  // first, as the general pass does), up the first tap until they are complete.
  R acc = (R)0, up = (R)0, first = (R)0;
  for (int k = ka; k <= kb; k++) {
    const int buf = k & 1;
    const size_t pl = (size_t)plane * k;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const V2 ep = (col && k < nz - 1) ? *reinterpret_cast<const V2 *>(e + o[q] + pl + plane) : zero;
      const R xl = __shfl_up_sync(0xffffffffu, e0[q].y, 1), xr = __shfl_down_sync(0xffffffffu, e0[q].x, 1);
      R v;
      if constexpr (sizeof(R) == sizeof(double)) {
        const bool odd = (jl[q] + k) & 1;  // the pair's red point
        R r = (R)0;
        if (col) {
          const R ym = e[om[q] + odd + pl], yp = e[op[q] + odd + pl];
          // x neighbours: the pair's other point, and the one outside it (absent beyond a wall)
          const R xo = odd ? ((ic < ncx - 1) ? xr : (R)0) : ((ic > 0) ? xl : (R)0);
          r = L.cx * ((odd ? e0[q].x : e0[q].y) + xo);
          r = fma(L.cy, ym + yp, r);
          r = fma(L.cz, odd ? em[q].y + ep.y : em[q].x + ep.x, r);
        }
        // taps of 2 ic - 1 .. 2 ic + 2: red even points are 2 ic (3) and 2 ic + 2 (1), odd ones 2 ic + 1 (3), 2 ic - 1
        const R rl = __shfl_up_sync(0xffffffffu, r, 1), rr = __shfl_down_sync(0xffffffffu, r, 1);
        const bool wall = odd ? ic == ncx - 1 : ic == 0;
        v = fma(wall ? (R)4 : (R)3, r, odd ? rl : rr);
      } else {
        V2 r = zero;
        if (col) {
          const V2 ym = *reinterpret_cast<const V2 *>(e + om[q] + pl), yp = *reinterpret_cast<const V2 *>(e + op[q] + pl);
          const V2 bb = *reinterpret_cast<const V2 *>(b + o[q] + pl);
          const R d = (R)2 * (L.cx + L.cy + L.cz);
          const bool lo = k > 0, hi = k < nz - 1;
          R a = mul_rn(d, e0[q].x);
          a = fma(-L.cx, (ic > 0 ? xl : e0[q].x) + e0[q].y, a);
          a = fma(-L.cy, ym.x + yp.x, a);
          r.x = bb.x - fma(-L.cz, (lo ? em[q].x : e0[q].x) + (hi ? ep.x : e0[q].x), a);
          a = mul_rn(d, e0[q].y);
          a = fma(-L.cx, e0[q].x + (ic < ncx - 1 ? xr : e0[q].y), a);
          a = fma(-L.cy, ym.y + yp.y, a);
          r.y = bb.y - fma(-L.cz, (lo ? em[q].y : e0[q].y) + (hi ? ep.y : e0[q].y), a);
        }
        const R rl = __shfl_up_sync(0xffffffffu, r.y, 1), rr = __shfl_down_sync(0xffffffffu, r.x, 1);
        v = mg_taps(ic == 0 ? (R)1 : (R)0.75, ic == ncx - 1 ? (R)1 : (R)0.75, rl, r.x, r.y, rr);
      }
      sx[buf][2 * w + q][lane] = v;
      em[q] = e0[q];
      e0[q] = ep;
    }
    __syncthreads();
    if (own) {  // rows 2 w .. 2 w + 3 are fine rows 2 jc - 1 .. 2 jc + 2
      const R s0 = sx[buf][2 * w][lane], s1 = sx[buf][2 * w + 1][lane];
      const R s2 = sx[buf][2 * w + 2][lane], s3 = sx[buf][2 * w + 3][lane];
      if constexpr (sizeof(R) == sizeof(double)) {
        const R v = fma((R)3, s1 + s2, s0 + s3);
        if constexpr (!Z) {
          out[cplane * k] = v * (R)(1.0 / 64.0);
          continue;
        }
        const R wz = (k == 0 || k == nz - 1) ? (R)4 : (R)3;
        if (k & 1) {  // k = 2 kc + 1: third tap of kc, first of kc + 1
          acc = fma(wz, v, acc);
          up = v;
        } else {  // k = 2 kc: fourth tap of kc - 1, second of kc
          if (k > 2 * kc0) out[cplane * (k / 2 - 1)] = (acc + v) * (R)(1.0 / 512.0);
          acc = fma(wz, v, up);
        }
      } else {
        const R v = mg_taps((R)0.75, (R)0.75, s0, s1, s2, s3);
        if (k & 1) {
          acc = fma(k == nz - 1 ? (R)1 : (R)0.75, v, acc);
          up = v;
        } else {
          if (k > 2 * kc0) out[cplane * (k / 2 - 1)] = fma((R)0.25, v, fma((R)0.25, first, acc)) * (R)0.125;
          acc = mul_rn(k == 0 ? (R)1 : (R)0.75, v);
          first = up;
        }
      }
    }
  }
  if (Z && own && kc1 == ncz) {
    if constexpr (sizeof(R) == sizeof(double)) out[cplane * (ncz - 1)] = acc * (R)(1.0 / 512.0);
    else out[cplane * (ncz - 1)] = fma((R)0.25, first, acc) * (R)0.125;
  }
}

// ---------------------------------------------------------------------------
// The same level in two launches, for levels too small to fill the GPU: a
// block takes a coarse tile CX x CY x CZ with the fine points around it in
// shared memory and runs all the passes of the level on it, recomputing the
// halo.  All loads of a block are issued before the first is used.
// FP32: every value is formed by the operations of the general passes
// (k_rbgs, k_residual, k_restrict_axis, k_prolong_axis) in their order, so the
// result equals theirs bit for bit; products that a sum would absorb into one
// rounding are kept apart (mul_rn).  FP64: the fewer operations of the five
// passes above (a warp's FP64 instruction holds its scheduler's unit for about
// 80 cycles, which is what a small level waits for beside its launches).
template <int CX, int CY, int CZ>
struct MgTile {
  static constexpr int FX = 2 * CX, FY = 2 * CY, FZ = 2 * CZ;
  // down: b / e with three points around the tile; r with one
  static constexpr int DX = FX + 6, DY = FY + 6, DZ = FZ + 6, RX = FX + 2, RY = FY + 2, RZ = FZ + 2;
  static constexpr int DN = DX * DY * DZ, RN = RX * RY * RZ, XN = CX * RY * RZ, YN = CX * CY * RZ;
  // up: e with two points around the tile; the coarse tile with two
  static constexpr int EX = FX + 4, EY = FY + 4, EZ = FZ + 4, KX = CX + 4, KY = CY + 4, KZ = CZ + 4;
  static constexpr int EN = EX * EY * EZ, KN = KX * KY * KZ, ZN = KX * KY * EZ, SN = KX * EY * EZ;
  static_assert(XN + YN <= DN && KN + ZN <= EN, "reused shared memory");
};

// y wrap; a tile reaches no further than one period beyond either end (the
// smallest extents included: ny 4 and 2 coarse rows).  n even: the colour of a
// row survives.
__device__ __forceinline__ int mg_wrap(int j, int n) { return j < 0 ? j + n : (j >= n ? j - n : j); }
__device__ __forceinline__ int mg_xc(int i, int nx) { return i == 0 ? 0 : (i == nx - 1 ? 2 : 1); }

// The points of a level around a tile (its extents DX x DY x DZ from fine
// point x0, y0, z0 on; y periodic, zero beyond the x and z walls), all loads
// issued together.
template <int DX, int DY, int DZ, typename R>
struct MgLoad {
  static constexpr int N = DX * DY * DZ, LI = (N + 255) / 256;
  R v[LI];
  __device__ __forceinline__ void load(const R *__restrict__ b, int nx, int ny, int nz, int x0, int y0, int z0,
                                       int t) {
#pragma unroll
    for (int m = 0; m < LI; m++) {
      const int q = t + 256 * m, lz = q / (DX * DY), ly = q / DX % DY, lx = q % DX;
      const int i = x0 + lx, j = mg_wrap(y0 + ly, ny), k = z0 + lz;
      v[m] = (q < N && i >= 0 && i < nx && k >= 0 && k < nz) ? b[i + nx * (j + (size_t)ny * k)] : (R)0;
    }
  }
  __device__ __forceinline__ void store(R *s, int t) {
#pragma unroll
    for (int m = 0; m < LI; m++)
      if (t + 256 * m < N) s[t + 256 * m] = v[m];
  }
};

// The Gauss-Seidel value of local point q of a tile of row length DX and
// plane DXY (zeros beyond the x and z walls).
template <int DX, int DXY, typename R>
__device__ __forceinline__ R mg_tile_relax(const MgLev<R> &L, const R *e, int q, R rhs, int i, int k) {
  R acc = fma(L.cx, e[q - 1] + e[q + 1], rhs);
  acc = fma(L.cy, e[q - DX] + e[q + DX], acc);
  acc = fma(L.cz, e[q - DXY] + e[q + DXY], acc);
  return mul_rn(acc, L.inv[mg_xc(i, L.nx)][mg_zc(k, L.nz)]);
}

template <typename R, int CX, int CY, int CZ>
__global__ void __launch_bounds__(256) k_mg_down(const __grid_constant__ MgLev<R> L, const R *__restrict__ b,
                                                 R *__restrict__ bc) {
  using T = MgTile<CX, CY, CZ>;
  constexpr bool F32 = sizeof(R) == sizeof(float);
  __shared__ R se[T::DN];
  __shared__ R sr[T::RN];
  __shared__ R sb[F32 ? T::DN : 1];  // FP32: b, for the residual
  R *sx = se, *sy = se + T::XN;      // after the residual
  const int nx = L.nx, ny = L.ny, nz = L.nz;
  const int ncx = nx / 2, ncy = ny / 2, ncz = nz / 2;
  const int gx = (ncx + CX - 1) / CX, gy = (ncy + CY - 1) / CY;
  const int x0 = (blockIdx.x % gx) * T::FX, y0 = (blockIdx.x / gx % gy) * T::FY, z0 = blockIdx.x / (gx * gy) * T::FZ;
  const int t = threadIdx.x;
  {
    MgLoad<T::DX, T::DY, T::DZ, R> ld;
    ld.load(b, nx, ny, nz, x0 - 3, y0 - 3, z0 - 3, t);
    if constexpr (F32) {  // red points: b / d
      ld.store(sb, t);
#pragma unroll
      for (int m = 0; m < ld.LI; m++) {
        const int q = t + 256 * m, lz = q / (T::DX * T::DY), ly = q / T::DX % T::DY, lx = q % T::DX;
        const int i = x0 - 3 + lx, k = z0 - 3 + lz;
        if ((lx + ly + lz) & 1)  // i + j + k = lx + ly + lz - 9 even (x0, y0, z0 are even)
          ld.v[m] = mul_rn(ld.v[m], L.inv[mg_xc(i, nx)][mg_zc(k, nz)]);
      }
    }
    ld.store(se, t);
  }
  __syncthreads();
  // black points of the tile and two points around it
  for (int q = t; q < (T::DX - 2) / 2 * (T::DY - 2) * (T::DZ - 2); q += 256) {
    constexpr int HX = (T::DX - 2) / 2;
    const int lz = 1 + q / (HX * (T::DY - 2)), ly = 1 + q / HX % (T::DY - 2);
    const int lx = 2 + 2 * (q % HX) - ((ly + lz) & 1);  // lx + ly + lz even: i + j + k = lx + ly + lz - 9 odd
    const int i = x0 - 3 + lx, k = z0 - 3 + lz, o = lx + T::DX * (ly + T::DY * lz);
    if (i >= 0 && i < nx && k >= 0 && k < nz) {
      if constexpr (F32) {
        se[o] = mg_tile_relax<T::DX, T::DX * T::DY>(L, se, o, se[o], i, k);
      } else {  // from b alone: the red neighbours' 1/d is in the couplings (zeros beyond the walls)
        const int xc = mg_xc(i, nx), zc = mg_zc(k, nz);
        R acc = fma(L.tx[mg_xc(max(i - 1, 0), nx)][zc], se[o - 1], se[o]);
        acc = fma(L.tx[mg_xc(min(i + 1, nx - 1), nx)][zc], se[o + 1], acc);
        acc = fma(L.ty[xc][zc], se[o - T::DX] + se[o + T::DX], acc);
        acc = fma(L.tz[xc][mg_zc(max(k - 1, 0), nz)], se[o - T::DX * T::DY], acc);
        acc = fma(L.tz[xc][mg_zc(min(k + 1, nz - 1), nz)], se[o + T::DX * T::DY], acc);
        se[o] = acc * L.inv[xc][zc];
      }
    }
  }
  __syncthreads();
  if constexpr (F32) {  // the residual of every point
    const R d = (R)2 * (L.cx + L.cy + L.cz);
    for (int q = t; q < T::RN; q += 256) {
      const int lz = q / (T::RX * T::RY), ly = q / T::RX % T::RY, lx = q % T::RX;
      const int i = x0 - 1 + lx, k = z0 - 1 + lz;
      R r = (R)0;
      if (i >= 0 && i < nx && k >= 0 && k < nz) {
        const int o = (lx + 2) + T::DX * ((ly + 2) + T::DY * (lz + 2));
        const R v = se[o];
        const R xm = (i > 0) ? se[o - 1] : v, xp = (i < nx - 1) ? se[o + 1] : v;
        const R zm = (k > 0) ? se[o - T::DX * T::DY] : v, zp = (k < nz - 1) ? se[o + T::DX * T::DY] : v;
        R a = mul_rn(d, v);
        a = fma(-L.cx, xm + xp, a);
        a = fma(-L.cy, se[o - T::DX] + se[o + T::DX], a);
        r = sb[o] - fma(-L.cz, zm + zp, a);
      }
      sr[q] = r;
    }
  } else {  // of the red points: the sum of the black couplings
    constexpr int HX = T::RX / 2;
    for (int q = t; q < HX * T::RY * T::RZ; q += 256) {
      const int lz = q / (HX * T::RY), ly = q / HX % T::RY, lx = 2 * (q % HX) + 1 - ((ly + lz) & 1);
      const int i = x0 - 1 + lx, k = z0 - 1 + lz, o = (lx + 2) + T::DX * ((ly + 2) + T::DY * (lz + 2));
      R r = (R)0;
      if (i >= 0 && i < nx && k >= 0 && k < nz) {
        // beyond a wall the tile holds zeros
        r = L.cx * (se[o - 1] + se[o + 1]);
        r = fma(L.cy, se[o - T::DX] + se[o + T::DX], r);
        r = fma(L.cz, se[o - T::DX * T::DY] + se[o + T::DX * T::DY], r);
      }
      sr[lx + T::RX * (ly + T::RY * lz)] = r;  // lx + ly + lz odd: i + j + k even
    }
  }
  __syncthreads();
  for (int q = t; q < T::XN; q += 256) {
    const int ix = q % CX, row = q / CX, ic = x0 / 2 + ix;  // row = ly + RY lz
    const R *p = sr + T::RX * row + 2 * ix;
    if constexpr (F32) {
      sx[q] = mg_taps(ic == 0 ? (R)1 : (R)0.75, ic == ncx - 1 ? (R)1 : (R)0.75, p[0], p[1], p[2], p[3]);
    } else {  // taps 1 3 3 1, red where lx + ly + lz is odd; 4 where a wall reflects the missing one (zero here)
      const bool odd = !((row % T::RY + row / T::RY) & 1);
      const R w = (odd ? ic == 0 : ic == ncx - 1) ? (R)4 : (R)3;
      sx[q] = fma(w, odd ? p[1] : p[2], odd ? p[3] : p[0]);
    }
  }
  __syncthreads();
  for (int q = t; q < T::YN; q += 256) {
    const int ix = q % CX, iy = q / CX % CY, lz = q / (CX * CY);
    const R *p = sx + ix + CX * (2 * iy + T::RY * lz);
    if constexpr (F32) sy[q] = mg_taps((R)0.75, (R)0.75, p[0], p[CX], p[2 * CX], p[3 * CX]);
    else sy[q] = fma((R)3, p[CX] + p[2 * CX], p[0] + p[3 * CX]);
  }
  __syncthreads();
  for (int q = t; q < CX * CY * CZ; q += 256) {
    const int ix = q % CX, iy = q / CX % CY, iz = q / (CX * CY);
    const int ic = x0 / 2 + ix, jc = y0 / 2 + iy, kc = z0 / 2 + iz;
    if (ic < ncx && jc < ncy && kc < ncz) {
      const R *p = sy + ix + CX * (iy + CY * 2 * iz);
      const R p0 = p[0], p1 = p[CX * CY], p2 = p[2 * CX * CY], p3 = p[3 * CX * CY];
      R v;
      if constexpr (F32) {
        v = mg_taps(kc == 0 ? (R)1 : (R)0.75, kc == ncz - 1 ? (R)1 : (R)0.75, p0, p1, p2, p3) * (R)0.125;
      } else {
        v = fma(kc == 0 ? (R)4 : (R)3, p1, p0);
        v = (fma(kc == ncz - 1 ? (R)4 : (R)3, p2, p3) + v) * (R)(1.0 / 512.0);
      }
      bc[ic + ncx * (jc + (size_t)ncy * kc)] = v;
    }
  }
}

// Coarse tile with two cells around it, clamped at the walls, y periodic.
template <int KX, int KY, int KZ, typename R>
struct MgLoadCoarse {
  static constexpr int N = KX * KY * KZ, LI = (N + 255) / 256;
  R v[LI];
  __device__ __forceinline__ void load(const R *__restrict__ ec, int ncx, int ncy, int ncz, int x0, int y0, int z0,
                                       int t) {
#pragma unroll
    for (int m = 0; m < LI; m++) {
      const int q = t + 256 * m, lz = q / (KX * KY), ly = q / KX % KY, lx = q % KX;
      const int ic = min(max(x0 + lx, 0), ncx - 1), jc = mg_wrap(y0 + ly, ncy), kc = min(max(z0 + lz, 0), ncz - 1);
      v[m] = q < N ? ec[ic + ncx * (jc + (size_t)ncy * kc)] : (R)0;
    }
  }
};

// e of the tile after the coarse correction and the post-smoothing; every
// thread of the block returns from it with the tile in se (local point 2 =
// the tile's first), its right-hand side in sb.
template <typename R, int CX, int CY, int CZ>
__device__ __forceinline__ void mg_up_tile(const MgLev<R> &L, const R *__restrict__ b, const R *__restrict__ ec, R *se,
                                           R *ss, R *sb, int x0, int y0, int z0) {
  using T = MgTile<CX, CY, CZ>;
  constexpr bool F32 = sizeof(R) == sizeof(float);
  R *sk = se, *sz = se + T::KN;  // before the fine values
  const int nx = L.nx, ny = L.ny, nz = L.nz;
  const int ncx = nx / 2, ncy = ny / 2, ncz = nz / 2;
  const int t = threadIdx.x;
  {
    MgLoad<T::EX, T::EY, T::EZ, R> lb;
    MgLoadCoarse<T::KX, T::KY, T::KZ, R> lc;
    lc.load(ec, ncx, ncy, ncz, x0 / 2 - 2, y0 / 2 - 2, z0 / 2 - 2, t);
    lb.load(b, nx, ny, nz, x0 - 2, y0 - 2, z0 - 2, t);
#pragma unroll
    for (int m = 0; m < lc.LI; m++)
      if (t + 256 * m < lc.N) sk[t + 256 * m] = lc.v[m];
    lb.store(sb, t);
  }
  __syncthreads();
  // one axis of the interpolation: FP32 as the general passes (3/4 and 1/4; a cell at a wall alone), FP64 3 and 1 (the
  // wall's clamped cell counts twice), scaled by 1/64 at the end
  auto lerp = [](R a, R c, bool wall) -> R {
    if constexpr (F32) return mg_lerp(a, c, wall);
    else return fma((R)3, a, c);
  };
  // fine index f = f0 - 2 + l; its cell is local (l >> 1) + 1, the next one on
  // its side one below for even l, one above for odd
  for (int q = t; q < T::ZN; q += 256) {
    const int lz = q / (T::KX * T::KY), col = q % (T::KX * T::KY), c0 = (lz >> 1) + 1;
    const int c1 = (lz & 1) ? c0 + 1 : c0 - 1, kc1 = z0 / 2 - 2 + c1;
    sz[q] = lerp(sk[col + T::KX * T::KY * c0], sk[col + T::KX * T::KY * c1], kc1 < 0 || kc1 >= ncz);
  }
  __syncthreads();
  for (int q = t; q < T::SN; q += 256) {
    const int lx = q % T::KX, ly = q / T::KX % T::EY, lz = q / (T::KX * T::EY), c0 = (ly >> 1) + 1;
    const int c1 = (ly & 1) ? c0 + 1 : c0 - 1;
    const R *p = sz + lx + T::KX * T::KY * lz;
    ss[q] = lerp(p[T::KX * c0], p[T::KX * c1], false);
  }
  __syncthreads();
  // red points of the tile and two points around it: b / d + P e_c; black: zero until relaxed
  constexpr int HE = T::EX / 2;
  for (int q = t; q < HE * T::EY * T::EZ; q += 256) {
    const int lz = q / (HE * T::EY), ly = q / HE % T::EY, odd = (ly + lz) & 1, lx = 2 * (q % HE) + odd;
    const int i = x0 - 2 + lx, k = z0 - 2 + lz, o = lx + T::EX * (ly + T::EY * lz);
    R v = (R)0;
    if (i >= 0 && i < nx && k >= 0 && k < nz) {
      const int c0 = (lx >> 1) + 1, c1 = (lx & 1) ? c0 + 1 : c0 - 1, ic1 = x0 / 2 - 2 + c1;
      const R *p = ss + T::KX * (ly + T::EY * lz);
      const R d = L.inv[mg_xc(i, nx)][mg_zc(k, nz)], w = lerp(p[c0], p[c1], ic1 < 0 || ic1 >= ncx);
      if constexpr (F32) v = mul_rn(sb[o], d) + w;
      else v = fma(sb[o], d, w * (R)(1.0 / 64.0));
    }
    se[o] = v;
    se[o + 1 - 2 * odd] = (R)0;
  }
  __syncthreads();
  for (int q = t; q < (T::EX - 2) / 2 * (T::EY - 2) * (T::EZ - 2); q += 256) {
    constexpr int HX = (T::EX - 2) / 2;
    const int lz = 1 + q / (HX * (T::EY - 2)), ly = 1 + q / HX % (T::EY - 2);
    const int lx = 1 + 2 * (q % HX) + ((ly + lz) & 1);  // lx + ly + lz odd
    const int i = x0 - 2 + lx, k = z0 - 2 + lz, o = lx + T::EX * (ly + T::EY * lz);
    if (i >= 0 && i < nx && k >= 0 && k < nz)
      se[o] = mg_tile_relax<T::EX, T::EX * T::EY>(L, se, o, sb[o], i, k);
  }
  __syncthreads();
  for (int q = t; q < T::FX / 2 * T::FY * T::FZ; q += 256) {
    const int lz = 2 + q / (T::FX / 2 * T::FY), ly = 2 + q / (T::FX / 2) % T::FY;
    const int lx = 2 + 2 * (q % (T::FX / 2)) + ((ly + lz) & 1);  // even sum
    const int i = x0 - 2 + lx, k = z0 - 2 + lz, o = lx + T::EX * (ly + T::EY * lz);
    if (i < nx && y0 - 2 + ly < ny && k < nz) se[o] = mg_tile_relax<T::EX, T::EX * T::EY>(L, se, o, sb[o], i, k);
  }
  __syncthreads();
}

template <typename R, int CX, int CY, int CZ>
__global__ void __launch_bounds__(256) k_mg_up(const __grid_constant__ MgLev<R> L, const R *__restrict__ b,
                                               const R *__restrict__ ec, R *__restrict__ e) {
  using T = MgTile<CX, CY, CZ>;
  __shared__ R se[T::EN];
  __shared__ R ss[T::SN];
  __shared__ R sb[T::EN];
  const int gx = (L.nx / 2 + CX - 1) / CX, gy = (L.ny / 2 + CY - 1) / CY;
  const int x0 = (blockIdx.x % gx) * T::FX, y0 = (blockIdx.x / gx % gy) * T::FY, z0 = blockIdx.x / (gx * gy) * T::FZ;
  mg_up_tile<R, CX, CY, CZ>(L, b, ec, se, ss, sb, x0, y0, z0);
  for (int q = threadIdx.x; q < T::FX * T::FY * T::FZ; q += 256) {
    const int lx = q % T::FX, ly = q / T::FX % T::FY, lz = q / (T::FX * T::FY);
    if (x0 + lx < L.nx && y0 + ly < L.ny && z0 + lz < L.nz)
      e[x0 + lx + L.nx * (y0 + ly + (size_t)L.ny * (z0 + lz))] = se[lx + 2 + T::EX * (ly + 2 + T::EY * (lz + 2))];
  }
}

}  // namespace tpls
