// k_momentum.cu -- momentum operator and Crank-Nicolson sweeps
// (momentum_allflux.f90:22-471, jacobi_iteration_allflux.f90:21-311,
// sor_iteration_allflux.f90:19-377, main_ns_hybrid.F90:629-641,743-887).
//
// Velocity components are addressed in the reference's staggered index
// space: u(i,j,k) sits between p-cells (i,j+1,k+1) and (i+1,j+1,k+1),
// v(i,j,k) between (i,j,k+1) and (i,j+1,k+1), w(i,j,k) between (i,j+1,k)
// and (i,j+1,k+1); the viscosity field mu is on the p-grid with two
// periodic ghost rows, so every face viscosity of the reference is read
// directly.
//
// Red-black SOR: for an even iteration_time the colouring is the 3-D
// checkerboard mod(k+j+flg,2), every point of a colour is independent and
// one thread updates one point.  For an odd iteration_time the colouring is
// mod(j+flg,2) in every plane, so the reference's sequential loop lets a
// point see the already-relaxed point below it: a recurrence up each column,
// run in chunks (k_sweep.cu).
// Periodic ghost rows are written by the thread that writes the row they
// copy (legal for even ny: no point of the colour being relaxed reads a
// ghost row written in the same half-sweep); for odd ny the caller runs a
// separate exchange after each half-sweep instead.
#include "tpls_sweep.cuh"
#include "tpls_pair.cuh"

namespace tpls {

// ---------------------------------------------------------------------------
// get_conv_all / get_diffusion_all point forms.
template <typename T>
struct CDT {
  T conv, diff;
};

// INTERIOR: the caller knows 0 < k < nz-1, so the wall-level forms of u and
// v (k = 0, nz-1) are left out at compile time (if-converted, their FP64
// instructions would occupy GB300's FP64 pipe on every level).
template <typename T, bool INTERIOR = false>
__device__ __forceinline__ CDT<T> conv_diff(int comp, const Geo &g, T rdx, T rdy, T rdz,
                                            const T *__restrict__ U, const T *__restrict__ V,
                                            const T *__restrict__ W, const FcT<T> &f, int i, int j,
                                            int k) {
  const int sy = g.sy, sz = g.sz, nzu = g.nz;  // u/v have planes 0..nz-1
  const int c = TPLS_IDX(g, i, j, k);
  const T h = (T)0.5, two = (T)2, third = (T)(1.0 / 3.0);
  const bool kb = !INTERIOR && k == 0, kt = !INTERIOR && k == nzu - 1;
  CDT<T> r;
  if (comp == 0) {
    const T x = U[c];
    const T tempv = (V[c] + V[c + 1] + V[c + sy] + V[c + 1 + sy]) * (T)0.25;
    const T tempw = (W[c] + W[c + 1] + W[c + sz] + W[c + 1 + sz]) * (T)0.25;
    const T Xc = h * (U[c + 1] - U[c - 1]) * rdx * x;
    const T Yc = h * (U[c + sy] - U[c - sy]) * rdy * tempv;
    T dz_;
    if (kb) dz_ = (x + U[c + sz]) * (h * rdz);
    else if (kt) dz_ = -(x + U[c - sz]) * (h * rdz);
    else dz_ = h * (U[c + sz] - U[c - sz]) * rdz;
    const T t1 = Xc + Yc + dz_ * tempw;
    const T E = f.px * (U[c + 1] - x) * rdx, Wt = f.mx * (x - U[c - 1]) * rdx;
    const T N = f.py * (V[c + 1 + sy] - V[c + sy]) * rdx, S = f.my * (V[c + 1] - V[c]) * rdx;
    const T O = f.pz * (W[c + 1 + sz] - W[c + sz]) * rdx, I = f.mz * (W[c + 1] - W[c]) * rdx;
    r.conv = t1 - ((E - Wt) * rdx + (N - S) * rdy + (O - I) * rdz);
    // loads only the planes each form uses (no plane -1 at k = 0, no plane nz at k = nz-1)
    const T umz = kb ? -two * x + U[c + sz] * third : U[c - sz];
    const T upz = kt ? -two * x + U[c - sz] * third : U[c + sz];
    r.diff = (f.px * (U[c + 1] - x) - f.mx * (x - U[c - 1])) * (rdx * rdx) +
             (f.py * (U[c + sy] - x) - f.my * (x - U[c - sy])) * (rdy * rdy) +
             (f.pz * (upz - x) - f.mz * (x - umz)) * (rdz * rdz);
  } else if (comp == 1) {
    const T x = V[c];
    const T tempu = (U[c - 1 - sy] + U[c - 1] + U[c - sy] + U[c]) * (T)0.25;
    const T tempw = (W[c - sy] + W[c] + W[c - sy + sz] + W[c + sz]) * (T)0.25;
    const T Yc = h * (V[c + sy] - V[c - sy]) * rdy * x;
    const T Xc = h * (V[c + 1] - V[c - 1]) * rdx * tempu;
    T dz_;
    if (kb) dz_ = (x + V[c + sz]) * (h * rdz);
    else if (kt) dz_ = -(x + V[c - sz]) * (h * rdz);
    else dz_ = h * (V[c + sz] - V[c - sz]) * rdz;
    const T t1 = Xc + Yc + dz_ * tempw;
    const T E = f.px * (U[c] - U[c - sy]) * rdy, Wt = f.mx * (U[c - 1] - U[c - 1 - sy]) * rdy;
    const T N = f.py * (V[c + sy] - x) * rdy, S = f.my * (x - V[c - sy]) * rdy;
    const T O = f.pz * (W[c + sz] - W[c - sy + sz]) * rdy, I = f.mz * (W[c] - W[c - sy]) * rdy;
    r.conv = t1 - ((E - Wt) * rdx + (N - S) * rdy + (O - I) * rdz);
    // loads only the planes each form uses (no plane -1 at k = 0, no plane nz at k = nz-1)
    const T vmz = kb ? -two * x + V[c + sz] * third : V[c - sz];
    const T vpz = kt ? -two * x + V[c - sz] * third : V[c + sz];
    r.diff = (f.px * (V[c + 1] - x) - f.mx * (x - V[c - 1])) * (rdx * rdx) +
             (f.py * (V[c + sy] - x) - f.my * (x - V[c - sy])) * (rdy * rdy) +
             (f.pz * (vpz - x) - f.mz * (x - vmz)) * (rdz * rdz);
  } else {
    const T x = W[c];
    const T tempu = (U[c - 1 - sz] + U[c - 1] + U[c - sz] + U[c]) * (T)0.25;
    const T tempv = (V[c - sz] + V[c] + V[c + sy - sz] + V[c + sy]) * (T)0.25;
    const T Zc = h * (W[c + sz] - W[c - sz]) * rdz * x;
    const T Xc = h * (W[c + 1] - W[c - 1]) * rdx * tempu;
    const T Yc = h * (W[c + sy] - W[c - sy]) * rdy * tempv;
    const T t1 = Xc + Yc + Zc;
    const T E = f.px * (U[c] - U[c - sz]) * rdz, Wt = f.mx * (U[c - 1] - U[c - 1 - sz]) * rdz;
    const T N = f.py * (V[c + sy] - V[c + sy - sz]) * rdz, S = f.my * (V[c] - V[c - sz]) * rdz;
    const T O = f.pz * (W[c + sz] - x) * rdz, I = f.mz * (x - W[c - sz]) * rdz;
    r.conv = t1 - ((E - Wt) * rdx + (N - S) * rdy + (O - I) * rdz);
    r.diff = (f.px * (W[c + 1] - x) - f.mx * (x - W[c - 1])) * (rdx * rdx) +
             (f.py * (W[c + sy] - x) - f.my * (x - W[c - sy])) * (rdy * rdy) +
             (f.pz * (W[c + sz] - x) - f.mz * (x - W[c - sz])) * (rdz * rdz);
  }
  return r;
}

constexpr int MB_X = 32, MB_Y = 4;

// Domain of a component's conv/diff (get_conv_all ranges) and of the
// right-hand side kernel (whole face range the history arrays carry).
__device__ __forceinline__ bool cd_valid(int comp, const Geo &g, int i, int k) {
  if (comp == 0) return i <= g.nx - 1;
  if (comp == 2) return k >= 1 && k <= g.nz - 1;
  return true;
}

// FP64 stencils of the FP32-mixed form (TPLS_PART_MOM_STENCIL): conv and diff
// in FP64, the defect right-hand side b = R / diag of the FP32 sweeps stored
// FP32, R = dt (diff - AB3(conv) + AB3(csf)) (see k_mom_rhs_pair); the sweeps
// rebuild the coefficients themselves.
template <bool INTERIOR>
__device__ __forceinline__ void mom_b32_point(int comp, const Geo &g, const Phys &ph, const Helm &hm,
                                              const double *__restrict__ U, const double *__restrict__ V,
                                              const double *__restrict__ W, const double *__restrict__ mu,
                                              const double *__restrict__ fc, const double *__restrict__ c1,
                                              const double *__restrict__ c0, const double *__restrict__ s1,
                                              const double *__restrict__ s0, double *__restrict__ conv2,
                                              double *__restrict__ csf2, float *__restrict__ bdef, int i, int j,
                                              int k) {
  const int c = TPLS_IDX(g, i, j, k);
  CDT<double> cd = {0.0, 0.0};
  const bool valid = cd_valid(comp, g, i, k);
  Fc f;
  if (valid) {
    f = faces(comp, g, mu, i, j, k);
    // 1/dx, 1/dy, 1/dz from the host (the same IEEE quotients, not three FP64
    // divisions per point on GB300's FP64 pipe)
    cd = conv_diff<double, INTERIOR>(comp, g, hm.rdx, hm.rdy, hm.rdz, U, V, W, f, i, j, k);
  }
  // main_ns_hybrid.F90:629-641 face averages of the CSF force
  double s2;
  if (comp == 0) s2 = (fc[TPLS_IDX(g, i + 1, j + 1, k + 1)] + fc[TPLS_IDX(g, i, j + 1, k + 1)]) * 0.5;
  else if (comp == 1) s2 = (fc[TPLS_IDX(g, i, j + 1, k + 1)] + fc[TPLS_IDX(g, i, j, k + 1)]) * 0.5;
  else s2 = (fc[TPLS_IDX(g, i, j + 1, k + 1)] + fc[TPLS_IDX(g, i, j + 1, k)]) * 0.5;
  conv2[c] = cd.conv;
  csf2[c] = s2;
  if (valid) {
    const double abc = (23.0 / 12.0) * cd.conv - (4.0 / 3.0) * c1[c] + (5.0 / 12.0) * c0[c];
    const double abs_ = (23.0 / 12.0) * s2 - (4.0 / 3.0) * s1[c] + (5.0 / 12.0) * s0[c];
    const double diag = 1.0 + hm.ax2 * (f.px + f.mx) + hm.ay2 * (f.py + f.my) + hm.az2 * (f.pz + f.mz);
    bdef[rec_slot(g, c, i)] = (float)(ph.dt * (cd.diff - abc + abs_) / diag);
  }
}

// CC: the velocity component at compile time.  The wall levels of u and v
// (k = 0, nz-1) take their own copy of the point code by a block-uniform
// branch, so the interior levels carry none of the wall forms.
template <int CC>
__global__ void __launch_bounds__(MB_X *MB_Y)
    k_mom_b32(Geo g, Phys ph, Helm hm, const double *__restrict__ U, const double *__restrict__ V,
              const double *__restrict__ W, const double *__restrict__ mu, const double *__restrict__ fc,
              const double *__restrict__ c1, const double *__restrict__ c0, const double *__restrict__ s1,
              const double *__restrict__ s0, double *__restrict__ conv2, double *__restrict__ csf2,
              float *__restrict__ bdef) {
  const int i = blockIdx.x * MB_X + threadIdx.x + 1, j = blockIdx.y * MB_Y + threadIdx.y + 1;
  const int k = blockIdx.z;
  if (i > g.nx || j > g.ny) return;
  if (CC != 2 && (k == 0 || k == g.nz - 1))
    mom_b32_point<false>(CC, g, ph, hm, U, V, W, mu, fc, c1, c0, s1, s0, conv2, csf2, bdef, i, j, k);
  else
    mom_b32_point<true>(CC, g, ph, hm, U, V, W, mu, fc, c1, c0, s1, s0, conv2, csf2, bdef, i, j, k);
}

cudaError_t launch_mom_rhs64r32(int comp, const Geo &g, const Phys &ph, const double *u2, const double *v2,
                                const double *w2, const double *mu, const double *fcsf, const double *c1,
                                const double *c0, const double *s1, const double *s0, double *conv2,
                                double *csf2, float *bdef, cudaStream_t st) {
  const int nk = (comp == 2) ? g.nz + 1 : g.nz;
  dim3 grd((g.nx + MB_X - 1) / MB_X, (g.ny + MB_Y - 1) / MB_Y, nk), blk(MB_X, MB_Y);
  const Helm hm = helm_of(ph);
  if (comp == 0) k_mom_b32<0><<<grd, blk, 0, st>>>(g, ph, hm, u2, v2, w2, mu, fcsf, c1, c0, s1, s0, conv2, csf2, bdef);
  else if (comp == 1)
    k_mom_b32<1><<<grd, blk, 0, st>>>(g, ph, hm, u2, v2, w2, mu, fcsf, c1, c0, s1, s0, conv2, csf2, bdef);
  else k_mom_b32<2><<<grd, blk, 0, st>>>(g, ph, hm, u2, v2, w2, mu, fcsf, c1, c0, s1, s0, conv2, csf2, bdef);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// FP64 right-hand sides and sweep records (the FP64 form).  Bound by the FP64
// pipe, so written for few operations (74 per point against 105 in the point
// form above):
//   * a thread marches kc levels of a column: the z faces' viscosity sums,
//     shear and difference products of a level's upper face are the next
//     level's lower face;
//   * conv and diff share the normal stress p dE - m dW of the component's own
//     axis; every axis' scales (1/2 of the centred difference, 1/4 of a
//     four-cell average, the grid spacings) are one factor;
//   * the AB3 and Crank-Nicolson combination is a product and six FMAs on
//     factors that carry dt, then the sum with the state: begun from the state,
//     it is rounded seven times at the state's size (3012 us at 256x128x192, 3044
//     so); 1/diag comes from rcp_seed and one Newton step.
// No output is further from a long-double evaluation than with the point form
// (conv 0.70-0.95 of its RMS error, diff 0.99-1.00, the step's u3, v3, w3 0.73-0.99).
// All three components in one launch (gx blocks along x each).
//
// The record of one point (8 doubles): the neighbour coefficients divided by
// the Helmholtz diagonal (jacobi_iteration_allflux.f90:84-90), x_new = cxp
// x[i+1] + cxm x[i-1] + cyp x[j+1] + cym x[j-1] + czp x[k+1] + czm x[k-1] +
// rhs/diag.  For u and v the wall ghost rule `-2 x(0) + x(1)/3` (and its top
// mirror) is folded in: at k = 0 the czm slot multiplies the point itself and
// czp absorbs czm/3; at k = nz-1 the czp slot multiplies the point itself and
// czm absorbs czp/3.  Order (cxp, cxm, cyp, cym, czp, czm, b, 1.2 czm), the
// last the factor of the odd half-sweep's column recurrence.
struct MomK {
  double vx, vy, vz;           // centred difference x velocity (sum of four where averaged)
  double tx, ty, tz;           // shear of conv per axis: rd_own rd_axis (a quarter where averaged)
  double lx, ly, lz;           // rd_axis^2 of diff (a quarter where averaged)
  double ax, ay, az;           // dt/(2 d^2) (a quarter where averaged)
  double k2, k1, k0, hd, l2, l1, l0;  // AB3 conv, CN diff and AB3 csf factors, dt included
};
struct MomArgs {
  const double *U, *V, *W, *mu;
  const double *f[3], *c1[3], *c0[3], *s1[3], *s0[3];
  double *conv2[3], *csf2[3], *coef[3];
  MomK q[3];
};

// The z face of a level as the level above needs it: the four-cell (w: single)
// viscosity, its products with the shear difference and with the component's
// own difference, and what the next face is formed from.
struct MomFace {
  double m, sh, own;
};

// What a column's thread computes: the step's right-hand side and records, or
// conv or diff alone (into conv2, on the component's domain).
enum { MOM_RHS, MOM_CONV, MOM_DIFF };

template <int CC, int WHAT>
__device__ __forceinline__ void mom_column(const Geo &g, const MomArgs &A, int i, int j, int ka, int kb) {
  const int sy = g.sy, sz = g.sz, my = g.sym, mz = g.szm, nz = g.nz;
  const MomK &q = A.q[CC];
  const double *__restrict__ U = A.U, *__restrict__ V = A.V, *__restrict__ W = A.W;
  const double *__restrict__ S = (CC == 0) ? U : (CC == 1 ? V : W);
  // the cell on the far side of the face: +x (u), -y (v), +z (w) of the near one
  const int om = (CC == 0) ? 1 : (CC == 1 ? -my : mz);
  const int oq = (CC == 0) ? 1 : (CC == 1 ? -sy : -sz);  // and in the velocity arrays, towards the other face point
  const bool inside = CC != 0 || i <= g.nx - 1;
  const double *f = A.f[CC], *c1 = A.c1[CC], *c0 = A.c0[CC], *s1 = A.s1[CC], *s0 = A.s0[CC];
  double *conv2 = A.conv2[CC], *csf2 = A.csf2[CC], *coef = A.coef[CC];
  double x = 0.0, mn = 0.0, mf = 0.0, ws = 0.0, fz = 0.0;
  MomFace lo = {0.0, 0.0, 0.0};
  // near-cell viscosity index of level k (u, v: level k+1 of the p-grid; w: k)
  auto mi = [&](int k) { return TPLS_IDXM(g, i, j + 1, k + (CC == 2 ? 0 : 1)); };
  bool started = false;
  for (int k = ka; k <= kb; k++) {
    const int c = TPLS_IDX(g, i, j, k);
    const bool level = (CC != 2) || (k >= 1 && k <= nz - 1);
    double conv = 0.0, diff = 0.0;
    double px = 0.0, mx = 0.0, py = 0.0, myv = 0.0, pz = 0.0, mzv = 0.0, sx = 0.0, xc = 0.0;
    const bool valid = inside && level;
    if (valid) {
      if (!started) {  // the lower face of the chunk's first level
        started = true;
        x = S[c];
        mn = A.mu[mi(k)];
        mf = A.mu[mi(k) + om];
        if (CC == 2) {
          lo.m = mn;
          lo.own = mn * (x - S[c - sz]);
        } else {
          lo.m = (mn + mf) + (A.mu[mi(k) - mz] + A.mu[mi(k) - mz + om]);
          const double w0 = W[c], w1 = W[c + oq];
          ws = w0 + w1;
          lo.sh = lo.m * (CC == 0 ? w1 - w0 : w0 - w1);
          if (k > 0) lo.own = lo.m * (x - S[c - sz]);
        }
      }
      const double xe = S[c + 1], xw = S[c - 1], xn = S[c + sy], xs = S[c - sy];
      const double dE = xe - x, dW = x - xw, dN = xn - x, dS = x - xs;
      // viscosity sums of the faces, and the level's upper face
      const double *m = A.mu + mi(k);
      const double near = mn + mf;  // the two cells of this point's own face
      double mn1 = 0.0, mf1 = 0.0;
      MomFace hi;
      // dT: the component's difference over the upper face, dsh: the shear's; dB2: the centred difference's lower half
      double xt = 0.0, dT, dB2, dsh = 0.0, ws1 = 0.0;
      if (CC == 2) {
        hi.m = mf;  // mu of level k+1
        xt = S[c + sz];
        dT = xt - x;
        hi.sh = 0.0;
        hi.own = hi.m * dT;
        dB2 = x - S[c - sz];
        mn1 = mf;
        mf1 = m[2 * mz];
        px = near + (m[1] + m[1 + mz]);
        mx = near + (m[-1] + m[-1 + mz]);
        py = near + (m[my] + m[my + mz]);
        myv = near + (m[-my] + m[-my + mz]);
        pz = hi.m;
        mzv = lo.m;
        sx = near;
      } else {
        mn1 = m[mz];
        mf1 = m[mz + om];
        hi.m = near + (mn1 + mf1);
        const double w0 = W[c + sz], w1 = W[c + sz + oq];
        ws1 = w0 + w1;
        dsh = CC == 0 ? w1 - w0 : w0 - w1;
        hi.sh = hi.m * dsh;
        pz = hi.m;
        mzv = lo.m;
        if (CC == 0) {
          px = mf;
          mx = mn;
          py = near + (m[my] + m[my + 1]);
          myv = near + (m[-my] + m[-my + 1]);
        } else {
          px = near + (m[1] + m[1 - my]);
          mx = near + (m[-1] + m[-1 - my]);
          py = mn;
          myv = mf;
        }
        sx = near;
        dT = 0.0;
        dB2 = 0.0;
      }
      // z differences; at the walls of u and v the ghost -2 x + x(k+-1)/3
      double dz;
      if (CC == 2) {
        dz = dT + dB2;
      } else if (k == 0) {
        xt = S[c + sz];
        dT = xt - x;
        hi.own = hi.m * dT;
        lo.own = lo.m * (x - fma(1.0 / 3.0, xt, -2.0 * x));
        dz = x + xt;
      } else if (k == nz - 1) {
        const double xb = S[c - sz];
        dT = fma(1.0 / 3.0, xb, -2.0 * x) - x;
        hi.own = hi.m * dT;
        dz = -(x + xb);
      } else {
        xt = S[c + sz];
        dT = xt - x;
        hi.own = hi.m * dT;
        dz = xt - S[c - sz];
      }
      // velocities at the point (sums of four) and shear of the other two components
      double vx, vy, vz, shx, shy;
      if (CC == 0) {
        const double a0 = V[c], a1 = V[c + 1], b0 = V[c + sy], b1 = V[c + 1 + sy];
        vx = x;
        vy = (a0 + a1) + (b0 + b1);
        vz = ws + ws1;
        shx = 0.0;
        shy = fma(py, b1 - b0, -myv * (a1 - a0));
      } else if (CC == 1) {
        const double a0 = U[c - 1 - sy], a1 = U[c - 1], b0 = U[c - sy], b1 = U[c];
        vx = (a0 + a1) + (b0 + b1);
        vy = x;
        vz = ws + ws1;
        shx = fma(px, b1 - b0, -mx * (a1 - a0));
        shy = 0.0;
      } else {
        const double a0 = U[c - 1 - sz], a1 = U[c - 1], b0 = U[c - sz], b1 = U[c];
        const double d0 = V[c - sz], d1 = V[c], e0 = V[c + sy - sz], e1 = V[c + sy];
        vx = (a0 + a1) + (b0 + b1);
        vy = (d0 + d1) + (e0 + e1);
        vz = x;
        shx = fma(px, b1 - b0, -mx * (a1 - a0));
        shy = fma(py, e1 - e0, -myv * (d1 - d0));
      }
      const double nx_ = fma(px, dE, -mx * dW), ny_ = fma(py, dN, -myv * dS), nz_ = fma(hi.m, dT, -lo.own);
      // shear of conv (the component's own axis shares diff's normal stress), then its convective terms, the streamwise
      // one last: the sum is rounded at its full size once
      conv = -q.tx * (CC == 0 ? nx_ : shx);
      conv = fma(-q.ty, CC == 1 ? ny_ : shy, conv);
      conv = fma(-q.tz, CC == 2 ? nz_ : fma(hi.m, dsh, -lo.sh), conv);
      conv = fma(q.vz, dz * vz, conv);
      conv = fma(q.vy, (xn - xs) * vy, conv);
      conv = fma(q.vx, (xe - xw) * vx, conv);
      diff = q.lx * nx_;
      diff = fma(q.ly, ny_, diff);
      diff = fma(q.lz, nz_, diff);
      lo = hi;
      xc = x;
      x = xt;
      mn = mn1;
      mf = mf1;
      ws = ws1;
    }
    if (WHAT != MOM_RHS) {
      if (valid) conv2[c] = (WHAT == MOM_CONV) ? conv : diff;
      continue;
    }
    // main_ns_hybrid.F90:629-641 face averages of the CSF force
    double s2;
    if (CC == 0) s2 = (f[TPLS_IDX(g, i + 1, j + 1, k + 1)] + f[TPLS_IDX(g, i, j + 1, k + 1)]) * 0.5;
    else if (CC == 1) s2 = (f[TPLS_IDX(g, i, j + 1, k + 1)] + f[TPLS_IDX(g, i, j, k + 1)]) * 0.5;
    else {
      const double fn = f[TPLS_IDX(g, i, j + 1, k + 1)];
      if (k == ka) fz = f[TPLS_IDX(g, i, j + 1, k)];
      s2 = (fn + fz) * 0.5;
      fz = fn;
    }
    conv2[c] = conv;
    csf2[c] = s2;
    if (valid) {
      // main_ns_hybrid.F90:743-751 (AB3 convection and CSF, CN diffusion)
      double r = q.k2 * conv;
      r = fma(q.k1, c1[c], r);
      r = fma(q.k0, c0[c], r);
      r = fma(q.hd, diff, r);
      r = fma(q.l2, s2, r);
      r = fma(q.l1, s1[c], r);
      r = fma(q.l0, s0[c], r) + xc;
      // the own axis' two faces are the two cells `near` sums (u: px + mx, v: py + my, w: pz + mz)
      double d = fma(q.ax, CC == 0 ? sx : px + mx, 1.0);
      d = fma(q.ay, CC == 1 ? sx : py + myv, d);
      d = fma(q.az, CC == 2 ? sx : pz + mzv, d);
      double h;
      if (rcp_range(d)) {
        h = rcp_seed(d);
        h = fma(h, fma(-d, h, 1.0), h);
      } else {
        h = div_slow(1.0, d);
      }
      const double hx = q.ax * h, hy = q.ay * h, hz = q.az * h;
      double czp = hz * pz, czm = hz * mzv;
      if (CC != 2) {
        if (k == 0) {
          czp = fma(czm, 1.0 / 3.0, czp);
          czm = -2.0 * czm;
        } else if (k == nz - 1) {
          czm = fma(czp, 1.0 / 3.0, czm);
          czp = -2.0 * czp;
        }
      }
      double2 *o = reinterpret_cast<double2 *>(coef + 8 * (size_t)rec_slot(g, c, i));
      o[0] = make_double2(hx * px, hx * mx);
      o[1] = make_double2(hy * py, hy * myv);
      o[2] = make_double2(czp, czm);
      o[3] = make_double2(r * h, 1.2 * czm);
    }
  }
}

// Levels per thread of the marching kernels: 8, halved to no less than 2 while
// `columns` blocks of them give fewer than eight blocks per SM.
static int march_levels(int columns, int nz) {
  int kc = 8;
  while (kc > 2 && columns * ((nz + kc) / kc) < 8 * 152) kc /= 2;
  return kc;
}

__global__ void __launch_bounds__(MB_X *MB_Y)
    k_mom_rhs(Geo g, const __grid_constant__ MomArgs A, int gx, int kc) {
  const int comp = blockIdx.x / gx, i = (blockIdx.x - comp * gx) * MB_X + threadIdx.x + 1;
  const int j = blockIdx.y * MB_Y + threadIdx.y + 1;
  const int last = (comp == 2) ? g.nz : g.nz - 1, ka = blockIdx.z * kc, kb = min(ka + kc - 1, last);
  if (i > g.nx || j > g.ny || ka > last) return;
  if (comp == 0) mom_column<0, MOM_RHS>(g, A, i, j, ka, kb);
  else if (comp == 1) mom_column<1, MOM_RHS>(g, A, i, j, ka, kb);
  else mom_column<2, MOM_RHS>(g, A, i, j, ka, kb);
}

// Standalone get_conv_all / get_diffusion_all by the same columns, the three
// components in one launch: conv 600 us and diff 407 us at 192x96x144 (38 and
// 26 FP64 operations per point; the point form with both terms, a launch per
// component, 1363 us each).
template <int WHAT>
__global__ void __launch_bounds__(MB_X *MB_Y)
    k_conv_diff(Geo g, const __grid_constant__ MomArgs A, int gx, int kc) {
  const int comp = blockIdx.x / gx, i = (blockIdx.x - comp * gx) * MB_X + threadIdx.x + 1;
  const int j = blockIdx.y * MB_Y + threadIdx.y + 1;
  const int ka = blockIdx.z * kc, kb = min(ka + kc, g.nz) - 1;  // (w's level nz is a wall)
  if (i > g.nx || j > g.ny || ka > kb) return;
  if (comp == 0) mom_column<0, WHAT>(g, A, i, j, ka, kb);
  else if (comp == 1) mom_column<1, WHAT>(g, A, i, j, ka, kb);
  else mom_column<2, WHAT>(g, A, i, j, ka, kb);
}

static MomK mom_factors(const Helm &hm, double dt, int q) {
  const double rd[3] = {hm.rdx, hm.rdy, hm.rdz}, a2[3] = {hm.ax2, hm.ay2, hm.az2};
  double v[3], t[3], l[3], a[3];
  for (int d = 0; d < 3; d++) {
    const double s = (d == q) ? 1.0 : 0.25;
    v[d] = 0.5 * rd[d] * s;
    t[d] = rd[q] * rd[d] * s;
    l[d] = rd[d] * rd[d] * s;
    a[d] = a2[d] * s;
  }
  return {v[0], v[1], v[2], t[0], t[1], t[2], l[0], l[1], l[2], a[0], a[1], a[2],
          -dt * (23.0 / 12.0), dt * (4.0 / 3.0), -dt * (5.0 / 12.0), dt / 2.0,
          dt * (23.0 / 12.0), -dt * (4.0 / 3.0), dt * (5.0 / 12.0)};
}

cudaError_t launch_conv_diff(int want_conv, const Geo &g, const Phys &ph, const double *u2, const double *v2,
                             const double *w2, const double *mu, double *const out[3], cudaStream_t st) {
  const Helm hm = helm_of(ph);
  MomArgs A = {};
  A.U = u2;
  A.V = v2;
  A.W = w2;
  A.mu = mu;
  for (int q = 0; q < 3; q++) {
    A.conv2[q] = out[q];
    A.q[q] = mom_factors(hm, ph.dt, q);
  }
  const int gx = (g.nx + MB_X - 1) / MB_X, gy = (g.ny + MB_Y - 1) / MB_Y, kc = march_levels(3 * gx * gy, g.nz);
  const dim3 grd(3 * gx, gy, (g.nz + kc - 1) / kc), blk(MB_X, MB_Y);
  if (want_conv) k_conv_diff<MOM_CONV><<<grd, blk, 0, st>>>(g, A, gx, kc);
  else k_conv_diff<MOM_DIFF><<<grd, blk, 0, st>>>(g, A, gx, kc);
  return cudaGetLastError();
}

cudaError_t launch_mom_rhs(const Geo &g, const Phys &ph, const double *u2, const double *v2, const double *w2,
                           const double *mu, const MomFields &m, cudaStream_t st) {
  const Helm hm = helm_of(ph);
  MomArgs A;
  A.U = u2;
  A.V = v2;
  A.W = w2;
  A.mu = mu;
  for (int q = 0; q < 3; q++) {
    A.f[q] = m.fcsf[q];
    A.c1[q] = m.c1[q];
    A.c0[q] = m.c0[q];
    A.s1[q] = m.s1[q];
    A.s0[q] = m.s0[q];
    A.conv2[q] = m.conv2[q];
    A.csf2[q] = m.csf2[q];
    A.coef[q] = m.coef[q];
    A.q[q] = mom_factors(hm, ph.dt, q);
  }
  const int gx = (g.nx + MB_X - 1) / MB_X, gy = (g.ny + MB_Y - 1) / MB_Y;
  const int kc = march_levels(3 * gx * gy, g.nz);
  k_mom_rhs<<<dim3(3 * gx, gy, (g.nz + kc) / kc), dim3(MB_X, MB_Y), 0, st>>>(g, A, gx, kc);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// FP32 momentum stencils of the FP32-mixed form on the FP64 velocity state.
//
// Each FP64 value is split by integer operations into an FP32 pair
// (hi = the value truncated to 24 significant bits, lo = the FP32 rounding
// of the remainder), so no FP64 instruction is issued: on GB300 FP64
// arithmetic and FP64<->FP32 conversions share a pipe 64x slower than FP32.
// Neighbour differences are formed as (hi_a - hi_b) + (lo_a - lo_b), which
// carries the FP32 precision of the difference itself instead of that of
// the O(|u|) values: the stencils' cancellations (first and second
// differences of a smooth field) then cost 1e-7 of the difference, not of
// |u|.  Sums and products use the pair rounded to FP32.
__device__ __forceinline__ F2 ld2(const double *__restrict__ p) { return split_bits(__ldg(p)); }

// float constants of one step (computed on the host in FP64, then rounded)
struct MomF {
  float rdx, rdy, rdz, ax2, ay2, az2;
  double dt64;
};

// get_conv_all / get_diffusion_all point forms (momentum_allflux.f90:22-471)
// on split values; the same operations as conv_diff with every difference
// of two velocity values taken from the pairs.  At the walls (u, v: k = 0
// and nz-1) the ghost value -2 x + x(k+-1)/3 enters as the difference
// x(k+-1)/3 - 3 x.
__device__ __forceinline__ CDT<float> conv_diff_pair(int comp, const Geo &g, const MomF &m,
                                                     const double *__restrict__ U, const double *__restrict__ V,
                                                     const double *__restrict__ W, const FcT<float> &f, int i,
                                                     int j, int k) {
  const int sy = g.sy, sz = g.sz, nzu = g.nz;
  const int c = TPLS_IDX(g, i, j, k);
  const float h = 0.5f, third = (float)(1.0 / 3.0), rdx = m.rdx, rdy = m.rdy, rdz = m.rdz;
  CDT<float> r;
  if (comp == 0 || comp == 1) {
    const double *S = comp == 0 ? U : V;
    const F2 x = ld2(S + c), xe = ld2(S + c + 1), xw = ld2(S + c - 1), xn = ld2(S + c + sy), xs = ld2(S + c - sy);
    float dT, dB, dzc;  // x(k+1) - x, x - x(k-1) (ghosts at the walls), centred z difference term
    if (k == 0) {
      const F2 xt = ld2(S + c + sz);
      dT = dif(xt, x);
      dB = (3.0f * x.h - xt.h * third) + (3.0f * x.l - xt.l * third);
      dzc = (val(x) + val(xt)) * (h * rdz);
    } else if (k == nzu - 1) {
      const F2 xb = ld2(S + c - sz);
      dB = dif(x, xb);
      dT = (xb.h * third - 3.0f * x.h) + (xb.l * third - 3.0f * x.l);
      dzc = -(val(x) + val(xb)) * (h * rdz);
    } else {
      const F2 xt = ld2(S + c + sz), xb = ld2(S + c - sz);
      dT = dif(xt, x);
      dB = dif(x, xb);
      dzc = h * dif(xt, xb) * rdz;
    }
    const float dE = dif(xe, x), dW = dif(x, xw), dN = dif(xn, x), dS = dif(x, xs);
    float t1, E, Wt, N, Sf, O, I;
    if (comp == 0) {
      const F2 v0 = ld2(V + c), v1 = ld2(V + c + 1), v2 = ld2(V + c + sy), v3 = ld2(V + c + 1 + sy);
      const F2 w0 = ld2(W + c), w1 = ld2(W + c + 1), w2 = ld2(W + c + sz), w3 = ld2(W + c + 1 + sz);
      const float tempv = (val(v0) + val(v1) + val(v2) + val(v3)) * 0.25f;
      const float tempw = (val(w0) + val(w1) + val(w2) + val(w3)) * 0.25f;
      const float Xc = h * dif(xe, xw) * rdx * val(x);
      const float Yc = h * dif(xn, xs) * rdy * tempv;
      t1 = Xc + Yc + dzc * tempw;
      E = f.px * dE * rdx;
      Wt = f.mx * dW * rdx;
      N = f.py * dif(v3, v2) * rdx;
      Sf = f.my * dif(v1, v0) * rdx;
      O = f.pz * dif(w3, w2) * rdx;
      I = f.mz * dif(w1, w0) * rdx;
    } else {
      const F2 u0 = ld2(U + c - 1 - sy), u1 = ld2(U + c - 1), u2 = ld2(U + c - sy), u3 = ld2(U + c);
      const F2 w0 = ld2(W + c - sy), w1 = ld2(W + c), w2 = ld2(W + c - sy + sz), w3 = ld2(W + c + sz);
      const float tempu = (val(u0) + val(u1) + val(u2) + val(u3)) * 0.25f;
      const float tempw = (val(w0) + val(w1) + val(w2) + val(w3)) * 0.25f;
      const float Yc = h * dif(xn, xs) * rdy * val(x);
      const float Xc = h * dif(xe, xw) * rdx * tempu;
      t1 = Xc + Yc + dzc * tempw;
      E = f.px * dif(u3, u2) * rdy;
      Wt = f.mx * dif(u1, u0) * rdy;
      N = f.py * dN * rdy;
      Sf = f.my * dS * rdy;
      O = f.pz * dif(w3, w2) * rdy;
      I = f.mz * dif(w1, w0) * rdy;
    }
    r.conv = t1 - ((E - Wt) * rdx + (N - Sf) * rdy + (O - I) * rdz);
    r.diff = (f.px * dE - f.mx * dW) * (rdx * rdx) + (f.py * dN - f.my * dS) * (rdy * rdy) +
             (f.pz * dT - f.mz * dB) * (rdz * rdz);
  } else {
    const F2 x = ld2(W + c), xe = ld2(W + c + 1), xw = ld2(W + c - 1), xn = ld2(W + c + sy), xs = ld2(W + c - sy);
    const F2 xt = ld2(W + c + sz), xb = ld2(W + c - sz);
    const F2 u0 = ld2(U + c - 1 - sz), u1 = ld2(U + c - 1), u2 = ld2(U + c - sz), u3 = ld2(U + c);
    const F2 v0 = ld2(V + c - sz), v1 = ld2(V + c), v2 = ld2(V + c + sy - sz), v3 = ld2(V + c + sy);
    const float tempu = (val(u0) + val(u1) + val(u2) + val(u3)) * 0.25f;
    const float tempv = (val(v0) + val(v1) + val(v2) + val(v3)) * 0.25f;
    const float Zc = h * dif(xt, xb) * rdz * val(x);
    const float Xc = h * dif(xe, xw) * rdx * tempu;
    const float Yc = h * dif(xn, xs) * rdy * tempv;
    const float t1 = Xc + Yc + Zc;
    const float dE = dif(xe, x), dW = dif(x, xw), dN = dif(xn, x), dS = dif(x, xs);
    const float dT = dif(xt, x), dB = dif(x, xb);
    const float E = f.px * dif(u3, u2) * rdz, Wt = f.mx * dif(u1, u0) * rdz;
    const float N = f.py * dif(v3, v2) * rdz, Sf = f.my * dif(v1, v0) * rdz;
    const float O = f.pz * dT * rdz, I = f.mz * dB * rdz;
    r.conv = t1 - ((E - Wt) * rdx + (N - Sf) * rdy + (O - I) * rdz);
    r.diff = (f.px * dE - f.mx * dW) * (rdx * rdx) + (f.py * dN - f.my * dS) * (rdy * rdy) +
             (f.pz * dT - f.mz * dB) * (rdz * rdz);
  }
  return r;
}

// Right-hand side of the FP32-mixed form's sweeps with FP32 stencils.
// The sweeps solve for the defect d = x - X (X the FP64 state of the
// component): with diag x - sum(a_n x_n) = rhs and diag = 1 + sum(a_n), the
// defect equation's right-hand side is
//   R = (rhs - X) + sum(a_n (X_n - X)) = dt (diff - AB3(conv) + AB3(csf)),
// because sum(a_n (X_n - X)) = (dt/2) diff for the same ghost-substituted
// neighbours (main_ns_hybrid.F90:743-751 for rhs).  conv and diff come from
// the FP32 pair stencils; the CSF force, the AB3 histories and R stay FP64
// (eleven FP64 operations per point): the CSF force is large at the
// interface, where it is balanced by the pressure gradient outside R, so its
// rounding is not relative to the step's increment.  Stored: b = R / diag,
// one float per point in record-slot order (the sweeps recompute the
// coefficients from mu).  conv is stored into its FP64 history exactly.
// The three components in one launch (gx blocks along x each).  Neither the
// FP64 pipe (11 operations per point) nor the issue slots (700 instructions)
// are full: it waits for loads and FP64 results, so many blocks per SM pay more
// than registers do.  Blocks (registers, spilled bytes) and us at 512x256x256 and
// 192x96x112: 8 (60, 0) 3997, 256; 10 (48, 20) 3434, 221; 12 (40, 164) 3175, 205; 14 and 16
// (32, 248) 2767, 182.  (A launch per component, 9 blocks: 4050 at 512x256x256.)
// (The component stays a run-time value: as a template argument it changes
// which products the compiler contracts, by last bits that the FP32 sweeps
// amplify to their own accuracy.)
struct MomPairArgs {
  const double *U, *V, *W;
  const float *mu;
  const double *f[3], *c1[3], *c0[3], *s1[3], *s0[3];
  double *conv2[3], *csf2[3];
  float *b[3];
};
__global__ void __launch_bounds__(MB_X *MB_Y, 14)
    k_mom_rhs_pair(Geo g, MomF m, const __grid_constant__ MomPairArgs A, int gx) {
  const int comp = blockIdx.x / gx, i = (blockIdx.x - comp * gx) * MB_X + threadIdx.x + 1;
  const int j = blockIdx.y * MB_Y + threadIdx.y + 1, k = blockIdx.z;
  if (i > g.nx || j > g.ny || (comp != 2 && k == g.nz)) return;
  const double *fc = A.f[comp];
  const int c = TPLS_IDX(g, i, j, k);
  CDT<float> cd = {0.0f, 0.0f};
  const bool valid = cd_valid(comp, g, i, k);
  FcT<float> f;
  if (valid) {
    f = faces<float>(comp, g, A.mu, i, j, k);
    cd = conv_diff_pair(comp, g, m, A.U, A.V, A.W, f, i, j, k);
  }
  // main_ns_hybrid.F90:629-641 face averages of the CSF force
  double s2;
  if (comp == 0) s2 = (fc[TPLS_IDX(g, i + 1, j + 1, k + 1)] + fc[TPLS_IDX(g, i, j + 1, k + 1)]) * 0.5;
  else if (comp == 1) s2 = (fc[TPLS_IDX(g, i, j + 1, k + 1)] + fc[TPLS_IDX(g, i, j, k + 1)]) * 0.5;
  else s2 = (fc[TPLS_IDX(g, i, j + 1, k + 1)] + fc[TPLS_IDX(g, i, j + 1, k)]) * 0.5;
  const double conv = widen_bits(cd.conv);
  A.conv2[comp][c] = conv;
  A.csf2[comp][c] = s2;
  if (!valid) return;
  const double abc = (23.0 / 12.0) * conv - (4.0 / 3.0) * A.c1[comp][c] + (5.0 / 12.0) * A.c0[comp][c];
  const double abs_ = (23.0 / 12.0) * s2 - (4.0 / 3.0) * A.s1[comp][c] + (5.0 / 12.0) * A.s0[comp][c];
  const double R = m.dt64 * (widen_bits(cd.diff) - abc + abs_);
  const float diag = 1.0f + m.ax2 * (f.px + f.mx) + m.ay2 * (f.py + f.my) + m.az2 * (f.pz + f.mz);
  A.b[comp][rec_slot(g, c, i)] = round_bits(R) / diag;
}

cudaError_t launch_mom_rhs_pair(const Geo &g, const Phys &ph, const double *u2, const double *v2, const double *w2,
                                const float *mu, const MomFields &q, float *const b[3], cudaStream_t st) {
  const Helm hm = helm_of(ph);
  MomF m;
  m.rdx = (float)(1.0 / ph.dx);
  m.rdy = (float)(1.0 / ph.dy);
  m.rdz = (float)(1.0 / ph.dz);
  m.dt64 = ph.dt;
  m.ax2 = (float)hm.ax2;
  m.ay2 = (float)hm.ay2;
  m.az2 = (float)hm.az2;
  MomPairArgs A = {u2, v2, w2, mu};
  for (int c = 0; c < 3; c++) {
    A.f[c] = q.fcsf[c];
    A.c1[c] = q.c1[c];
    A.c0[c] = q.c0[c];
    A.s1[c] = q.s1[c];
    A.s0[c] = q.s0[c];
    A.conv2[c] = q.conv2[c];
    A.csf2[c] = q.csf2[c];
    A.b[c] = b[c];
  }
  const int gx = (g.nx + MB_X - 1) / MB_X;
  k_mom_rhs_pair<<<dim3(3 * gx, (g.ny + MB_Y - 1) / MB_Y, g.nz + 1), dim3(MB_X, MB_Y), 0, st>>>(g, m, A, gx);
  return cudaGetLastError();
}

// jacobi_iteration_allflux.f90:21-282 with the routine's own boundary rows
// (v, w): the per-routine entry.  A thread marches kc levels of a column.
// 149 us per component at 192x96x144 (29 FP64 operations per point; the point
// form with averages and a division 197).  The right-hand side is added last
// and the quotient rounded once, as in that form, whose error this has: as a
// product with 1/diag, begun from the right-hand side, 146 us and 1.1 times it.
template <int CC>
__global__ void __launch_bounds__(MB_X *MB_Y)
    k_ref_jacobi(Geo g, RefCoef s, const double *__restrict__ xo, double *__restrict__ x, int kc) {
  const int i = blockIdx.x * MB_X + threadIdx.x + 1, j = blockIdx.y * MB_Y + threadIdx.y + 1;
  const int nz = g.nz, k0 = (CC == 2) ? 1 : 0, iend = (CC == 0) ? g.nx - 1 : g.nx;
  const int ka = k0 + blockIdx.z * kc, kb = min(ka + kc, nz);
  if (i > iend || j > g.ny || ka >= kb) return;
  const int sy = g.sy, sz = g.sz;
  int c = TPLS_IDX(g, i, j, ka);
  const double *m = ref_cell<CC>(g, s, i, j, ka);
  double near, lo;
  ref_begin<CC>(g, m, near, lo);
  double xc = xo[c], zm = (CC == 2 || ka > 0) ? xo[c - sz] : 0.0;
  for (int k = ka; k < kb; k++) {
    double hi, near1, d;
    double t = ref_point<CC, false>(g, s, m, near, lo, 0.0, xo[c + 1], xo[c - 1], xo[c + sy], xo[c - sy], hi, near1, d);
    double zp = 0.0;
    if (CC == 2 || k < nz - 1) zp = xo[c + sz];
    // the no-slip ghost values below k = 0 and above k = nz-1 (jacobi_iteration_allflux.f90:63-73)
    double zt = zp, zb = zm;
    if (CC != 2 && k == 0) zb = fma(zp, 1.0 / 3.0, -2.0 * xc);
    if (CC != 2 && k == nz - 1) zt = fma(zm, 1.0 / 3.0, -2.0 * xc);
    t = fma(s.cz, fma(hi, zt, lo * zb), t);
    const double v = div_inf(t + s.rhs[c], d);
    x[c] = v;
    if (CC == 1) {  // jacobi_iteration_allflux.f90:178-189
      if (i == 1) x[c - 1] = v;
      if (i == g.nx) x[c + 1] = v;
    } else if (CC == 2) {  // jacobi_iteration_allflux.f90:257-279
      const bool l = (i == 1), r = (i == g.nx);
      if (l) x[c - 1] = v;
      if (r) x[c + 1] = v;
      if (k == 1 || k == nz - 1) {
        auto wall = [&](int o) {
          x[o] = 0.0;
          if (l) x[o - 1] = 0.0;
          if (r) x[o + 1] = 0.0;
        };
        if (k == 1) wall(c - sz);
        if (k == nz - 1) wall(c + sz);
      }
    }
    zm = xc;
    xc = zp;
    near = near1;
    lo = hi;
    c += sz;
    m += g.szm;
  }
}

cudaError_t launch_ref_jacobi(int comp, const Geo &g, const RefCoef &s, const double *xo, double *x,
                              cudaStream_t st) {
  const int gx = (g.nx + MB_X - 1) / MB_X, gy = (g.ny + MB_Y - 1) / MB_Y, kc = march_levels(gx * gy, g.nz);
  const dim3 grd(gx, gy, (g.nz + kc - 1) / kc), blk(MB_X, MB_Y);
  if (comp == 0) k_ref_jacobi<0><<<grd, blk, 0, st>>>(g, s, xo, x, kc);
  else if (comp == 1) k_ref_jacobi<1><<<grd, blk, 0, st>>>(g, s, xo, x, kc);
  else k_ref_jacobi<2><<<grd, blk, 0, st>>>(g, s, xo, x, kc);
  return cudaGetLastError();
}

// sor_iteration_allflux.f90:54-99 (and v, w): 3-D checkerboard half-sweep of
// the per-routine entry, its quotient as the Jacobi point's.  84 us per
// component at 192x96x144 (with averages and a division 105).
template <int CC>
__global__ void __launch_bounds__(MB_X *MB_Y)
    k_ref_even(Geo g, RefCoef s, double *__restrict__ x, int flg) {
  const int i2 = blockIdx.x * MB_X + threadIdx.x, j = blockIdx.y * MB_Y + threadIdx.y + 1;
  const int k = blockIdx.z + (CC == 2 ? 1 : 0), nz = g.nz, iend = (CC == 0) ? g.nx - 1 : g.nx;
  const int i = 2 * i2 + 1 + ((k + j + flg) & 1);
  if (i > iend || j > g.ny) return;
  const int sy = g.sy, sz = g.sz, c = TPLS_IDX(g, i, j, k);
  const double *m = ref_cell<CC>(g, s, i, j, k);
  double near, lo, hi, near1, d;
  ref_begin<CC>(g, m, near, lo);
  double t = ref_point<CC, false>(g, s, m, near, lo, 0.0, x[c + 1], x[c - 1], x[c + sy], x[c - sy], hi, near1, d);
  const double xc = x[c];
  double zp, zm;
  if (CC == 2) {
    zp = x[c + sz];
    zm = x[c - sz];
  } else {
    zp = (k < nz - 1) ? x[c + sz] : fma(x[c - sz], 1.0 / 3.0, -2.0 * xc);
    zm = (k > 0) ? x[c - sz] : fma(zp, 1.0 / 3.0, -2.0 * xc);
  }
  t = fma(s.cz, fma(hi, zp, lo * zm), t) + s.rhs[c];
  x[c] = fma(1.2, div_inf(t, d) - xc, xc);
}

cudaError_t launch_ref_even(int comp, const Geo &g, const RefCoef &s, double *x, int flg, cudaStream_t st) {
  const dim3 grd(((g.nx + 1) / 2 + MB_X - 1) / MB_X, (g.ny + MB_Y - 1) / MB_Y, comp == 2 ? g.nz - 1 : g.nz);
  const dim3 blk(MB_X, MB_Y);
  if (comp == 0) k_ref_even<0><<<grd, blk, 0, st>>>(g, s, x, flg);
  else if (comp == 1) k_ref_even<1><<<grd, blk, 0, st>>>(g, s, x, flg);
  else k_ref_even<2><<<grd, blk, 0, st>>>(g, s, x, flg);
  return cudaGetLastError();
}

RefCoef ref_coef(int comp, const Phys &ph, const double *rhs, const double *mu) {
  const Helm h = helm_of(ph);
  return {mu, rhs, h.ax2 * (comp == 0 ? 1.0 : 0.25), h.ay2 * (comp == 1 ? 1.0 : 0.25),
          h.az2 * (comp == 2 ? 1.0 : 0.25)};
}

// get_difference of up to three pairs of iterates (the sweeps' convergence
// diagnostic): out[q], q < nout, = sum (a-b)^2 over i 1..nx, j 1..ny, planes
// 0..nzp-1, 0 without a pair.  One launch: rows to warps in a fixed order, a partial per
// block, summed by the last block in a fixed order.  (A launch and one or two
// more for the sum per component took 75 us of a step at 128x64x96, 30 at
// 64x32x48; this 23 and 13.)  FP64 iterates are differenced and
// summed in FP64; FP32 iterates are differenced in FP32 and each thread sums
// its squares as an FP32 pair (error-free sums), widened at the end: no FP64
// instruction per point (with a warp's FP32 sum widened per 32 points 450 us at
// 512x256x256, 200 with pairs).
constexpr int DF_B = 256, DF_W = DF_B / 32;
// A thread's squares of one pair summed in FP64, where their FP32 sum is not
// finite (it overflowed, or a square is infinite or NaN: the pair's rounding is
// NaN then).  Out of the loop, in which a test per square doubled the time.
static __device__ __noinline__ double wide_squares(const Geo &g, const float *__restrict__ x,
                                                   const float *__restrict__ y, int nzp) {
  double s = 0.0;
  for (int row = blockIdx.x * DF_W + (threadIdx.x >> 5); row < g.ny * nzp; row += gridDim.x * DF_W) {
    const int k = row / g.ny, c0 = TPLS_IDX(g, 1, row - g.ny * k + 1, k);
    for (int i = threadIdx.x & 31; i < g.nx; i += 32) {
      const float d = x[c0 + i] - y[c0 + i];
      s += widen_bits(__fmul_rn(d, d));
    }
  }
  return s;
}
template <typename T>
__global__ void __launch_bounds__(DF_B)
    k_diff_set(Geo g, const __grid_constant__ DiffSet<T> s, int planes, double *__restrict__ part, unsigned *ctr,
               double *__restrict__ out, int nout) {
  __shared__ double sh[3][DF_B];
  __shared__ bool last;
  const int t = threadIdx.x, lane = t & 31, nb = gridDim.x;
  double acc[3] = {0.0, 0.0, 0.0};
  float hi[3] = {0.0f, 0.0f, 0.0f}, lo[3] = {0.0f, 0.0f, 0.0f};
  for (int row = blockIdx.x * DF_W + (t >> 5); row < g.ny * planes; row += nb * DF_W) {
    const int k = row / g.ny, c0 = TPLS_IDX(g, 1, row - g.ny * k + 1, k);
#pragma unroll
    for (int q = 0; q < 3; q++) {
      if (!s.a[q] || k >= s.nzp[q]) continue;
      const T *a = s.a[q] + c0, *b = s.b[q] + c0;
#pragma unroll 4
      for (int i = lane; i < g.nx; i += 32) {
        const T d = a[i] - b[i];
        if constexpr (sizeof(T) == sizeof(float)) {
          const float e = __fmul_rn(d, d), s1 = hi[q] + e, z = s1 - hi[q];  // hi + e = s1 + its rounding
          lo[q] += (hi[q] - (s1 - z)) + (e - z);
          hi[q] = s1;
        } else {
          acc[q] = fma(d, d, acc[q]);
        }
      }
    }
  }
  if constexpr (sizeof(T) == sizeof(float))
    for (int q = 0; q < 3; q++)
      acc[q] = hi[q] <= 0x1.fffffep127f ? widen_bits(hi[q]) + widen_bits(lo[q])
                                        : wide_squares(g, s.a[q], s.b[q], s.nzp[q]);
  // the block's sums, in lane 0 of warp 0: lane by lane over the warps, then one
  // warp's tree
  auto block = [&](double (&v)[3]) {
    __syncthreads();
    for (int q = 0; q < 3; q++) sh[q][t] = v[q];
    __syncthreads();
    if (t < 32)
      for (int q = 0; q < 3; q++) {
        double x = sh[q][t];
        for (int w = 1; w < DF_W; w++) x += sh[q][t + 32 * w];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        v[q] = x;
      }
  };
  block(acc);
  if (t == 0) {
    for (int q = 0; q < 3; q++) part[q * nb + blockIdx.x] = acc[q];
    __threadfence();
    last = atomicAdd(ctr, 1u) == (unsigned)nb - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int q = 0; q < 3; q++) {
    acc[q] = 0.0;
    for (int b = t; b < nb; b += DF_B) acc[q] += __ldcg(part + q * nb + b);
  }
  block(acc);
  if (t == 0) {
    for (int q = 0; q < nout; q++) out[q] = acc[q];
    *ctr = 0u;
  }
}

template <typename T>
cudaError_t launch_diff_set(const Geo &g, const DiffSet<T> &s, double *part, unsigned *ctr, double *out, int nout,
                            cudaStream_t st) {
  int planes = 0;
  for (int q = 0; q < 3; q++)
    if (s.a[q] && s.nzp[q] > planes) planes = s.nzp[q];
  const int need = (g.ny * planes + DF_W - 1) / DF_W, nb = need < 1 ? 1 : (need < DIFF_BLOCKS ? need : DIFF_BLOCKS);
  k_diff_set<T><<<nb, DF_B, 0, st>>>(g, s, planes, part, ctr, out, nout);
  return cudaGetLastError();
}
template cudaError_t launch_diff_set<double>(const Geo &, const DiffSet<double> &, double *, unsigned *, double *, int,
                                             cudaStream_t);
template cudaError_t launch_diff_set<float>(const Geo &, const DiffSet<float> &, double *, unsigned *, double *, int,
                                            cudaStream_t);

// ---------------------------------------------------------------------------
// pressure.f90:16-56 get_source_pres on the full p-grid (zero outside the
// interior, ghost rows included, as the routine itself leaves them).
template <typename T>
__global__ void k_source(Geo g, double rdx, double rdy, double rdz, double rdt, const T *__restrict__ U,
                         const T *__restrict__ V, const T *__restrict__ W, double *__restrict__ rhs) {
  const int i = blockIdx.x * MB_X + threadIdx.x, j = blockIdx.y * MB_Y + threadIdx.y;
  const int k = blockIdx.z;
  if (i > g.nx + 1 || j > g.ny + 1) return;
  double r = 0.0;
  if (i >= 1 && i <= g.nx && j >= 1 && j <= g.ny && k >= 1 && k <= g.nz) {
    const int jj = j, jm = (jj == 1) ? g.ny : jj - 1;
    r = (((double)U[TPLS_IDX(g, i, jm, k - 1)] - (double)U[TPLS_IDX(g, i - 1, jm, k - 1)]) * rdx +
         ((double)V[TPLS_IDX(g, i, jj, k - 1)] - (double)V[TPLS_IDX(g, i, jm, k - 1)]) * rdy +
         ((double)W[TPLS_IDX(g, i, jm, k)] - (double)W[TPLS_IDX(g, i, jm, k - 1)]) * rdz) *
        rdt;
  }
  rhs[TPLS_IDX(g, i, j, k)] = r;
}

template <typename T>
static cudaError_t source(const Geo &g, const Phys &ph, const T *u3, const T *v3, const T *w3, double *rhs_p,
                          cudaStream_t st) {
  dim3 grd((g.nx + 2 + MB_X - 1) / MB_X, (g.ny + 2 + MB_Y - 1) / MB_Y, g.nz + 2);
  k_source<T><<<grd, dim3(MB_X, MB_Y), 0, st>>>(g, 1.0 / ph.dx, 1.0 / ph.dy, 1.0 / ph.dz, 1.0 / ph.dt, u3, v3,
                                                w3, rhs_p);
  return cudaGetLastError();
}
cudaError_t launch_source(const Geo &g, const Phys &ph, const double *u3, const double *v3, const double *w3,
                          double *rhs_p, cudaStream_t st) {
  return source(g, ph, u3, v3, w3, rhs_p, st);
}

// pressure.f90:59-134 get_uvw_pres, written out of place into the next
// state's velocity arrays over x 0..nx+1 and every row (ghost rows as
// periodic copies).
template <typename T>
__global__ void k_project(Geo g, double dtdx, double dtdy, double dtdz, const T *__restrict__ U,
                          const T *__restrict__ V, const T *__restrict__ W, const double *__restrict__ P,
                          const double *__restrict__ uin, double *__restrict__ uo,
                          double *__restrict__ vo, double *__restrict__ wo) {
  const int i = blockIdx.x * MB_X + threadIdx.x, j = blockIdx.y * MB_Y + threadIdx.y;
  const int k = blockIdx.z;
  if (i > g.nx + 1 || j > g.ny + 1) return;
  const int jj = wrapy(j, g.ny);
  const int c = TPLS_IDX(g, i, j, k), cc = TPLS_IDX(g, i, jj, k);
  const int sy = g.sy, sz = g.sz;
  if (k <= g.nz - 1) {
    double u;
    if (i == 0) u = uin[k];
    else if (i == g.nx + 1) u = 0.0;
    else u = (double)U[cc] - dtdx * (P[cc + 1 + sy + sz] - P[cc + sy + sz]);
    uo[c] = u;
    vo[c] = (double)V[cc] - dtdy * (P[cc + sy + sz] - P[cc + sz]);
  }
  wo[c] = (double)W[cc] - dtdz * (P[cc + sy + sz] - P[cc + sy]);
}

template <typename T>
static cudaError_t project(const Geo &g, const Phys &ph, const T *u3, const T *v3, const T *w3, const double *p,
                           const double *u_inlet, double *u_out, double *v_out, double *w_out, cudaStream_t st) {
  dim3 grd((g.nx + 2 + MB_X - 1) / MB_X, (g.ny + 2 + MB_Y - 1) / MB_Y, g.nz + 1);
  k_project<T><<<grd, dim3(MB_X, MB_Y), 0, st>>>(g, ph.dt / ph.dx, ph.dt / ph.dy, ph.dt / ph.dz, u3, v3, w3, p,
                                                 u_inlet, u_out, v_out, w_out);
  return cudaGetLastError();
}
cudaError_t launch_project(const Geo &g, const Phys &ph, const double *u3, const double *v3, const double *w3,
                           const double *p, const double *u_inlet, double *u_out, double *v_out, double *w_out,
                           cudaStream_t st) {
  return project(g, ph, u3, v3, w3, p, u_inlet, u_out, v_out, w_out, st);
}


}  // namespace tpls
