// k_dim.cu -- the diffuse-interface (Cahn-Hilliard) update of
// cahn_hilliard_solver.f90:41-382 (`dim`), the alternative to the level-set
// update + redistancing selected by idm = dim (main_ns_hybrid.F90:595-612).
//
// One thread per interior point.  The routine fills ghost values by copies (z
// planes from k = 1 / nz, periodic y rows, x columns from i = 1 / nx) and an
// inlet profile; the thread that owns the source writes them, so each phase is
// one launch and no warp runs for the two ghost columns of a row.  Positions
// the routine leaves untouched keep their previous value, as the reference's
// arrays do.  The iterate is double-buffered.  FP64 throughout: this is the
// FP64 form's path, bound by the FP64 pipe on large grids and by launch and
// arithmetic latency on small ones.
#include "tpls_kernels.h"

namespace tpls {

constexpr int DM_BX = 32, DM_BY = 4;

// The thread's interior point; false outside the grid.
struct Pt {
  int i, j, k, c;
};
__device__ __forceinline__ bool dim_point(const Geo &g, Pt &p) {
  p.i = blockIdx.x * DM_BX + threadIdx.x + 1;
  p.j = blockIdx.y * DM_BY + threadIdx.y + 1;
  p.k = blockIdx.z + 1;
  p.c = TPLS_IDX(g, p.i, p.j, p.k);
  return p.i <= g.nx && p.j <= g.ny;
}

// w(q) for the point and the face ghosts that copy it: the x ghost columns
// (j 1..ny, k 1..nz), the y ghost rows (i 1..nx, k 1..nz) and the z ghost
// planes (i 1..nx, j 1..ny); corners and edges are not set.
template <typename F>
__device__ __forceinline__ void first_order(const Geo &g, const Pt &p, F w) {
  w(p.c);
  if (p.i == 1) w(p.c - 1);
  if (p.i == g.nx) w(p.c + 1);
  if (p.j == 1) w(p.c + g.sy * g.ny);
  if (p.j == g.ny) w(p.c - g.sy * g.ny);
  if (p.k == 1) w(p.c - g.sz);
  if (p.k == g.nz) w(p.c + g.sz);
}

// 7-point Laplacian of a (plus a constant add, the driver's phi2 + 0.5 taken
// on the fly) at an interior point, divisions by dx^2 as multiplications by
// the host's 1/dx/dx
__device__ __forceinline__ double lap7(const Geo &g, const DimK &q, const double *__restrict__ a, double add,
                                       int c) {
  const double p = a[c] + add;
  return ((a[c + 1] + add) - 2.0 * p + (a[c - 1] + add)) * q.rdx2 +
         ((a[c + g.sy] + add) - 2.0 * p + (a[c - g.sy] + add)) * q.rdy2 +
         ((a[c + g.sz] + add) - 2.0 * p + (a[c - g.sz] + add)) * q.rdz2;
}

// dsqrt(c1*c1*(1-|c1|)*(1-|c1|))
__device__ __forceinline__ double mob(double c1) { return fabs(c1 * (1.0 - fabs(c1))); }

// The inlet profile of level k is kept in an edge of the Laplacian's array,
// which no copy rule sets and no stencil reads: one tanh per level instead of
// one per inlet element and iteration.
__device__ __forceinline__ int inlet_slot(const Geo &g, int k) { return TPLS_IDX(g, 0, 0, k); }

// :110-172 bulkE0 and d2phi of C = phi + add, with their ghost copies
__global__ void __launch_bounds__(DM_BX *DM_BY)
    k_dim_prep(Geo g, DimK q, const double *__restrict__ phi, double add, double *__restrict__ e0,
               double *__restrict__ l0) {
  Pt t;
  if (!dim_point(g, t)) return;
  const double p = phi[t.c] + add;
  const double e = (1.0 - 3.0 * p + 2.0 * p * p) * p / 2.0, l = lap7(g, q, phi, add, t.c);
  first_order(g, t, [&](int o) {
    e0[o] = e;
    l0[o] = l;
  });
  if (t.i == 1 && t.j == 1) l0[inlet_slot(g, t.k)] = 0.5 + 0.5 * tanh((t.k * q.dz - 0.5 * q.dz - q.height) / q.zden);
}

// :174-233 source0 = 2 temp5 - ConvPrevPhi, ConvPrevPhi = temp5 (interior),
// and the part of the relaxed update (:286-317) that the iterations share:
//   base = alfa1/diagonal (2 C - C_old / 2 + dt source0)
__global__ void __launch_bounds__(DM_BX *DM_BY)
    k_dim_source(Geo g, DimK q, const double *__restrict__ phi, double add, const double *__restrict__ phio,
                 double addo, const double *__restrict__ e0, const double *__restrict__ l0,
                 const double *__restrict__ conv2, double *__restrict__ cprev, double *__restrict__ base) {
  Pt t;
  if (!dim_point(g, t)) return;
  const int c = t.c, k = t.k, sy = g.sy, sz = g.sz;
  const double p = phi[c] + add;
  const double a1 = mob(((phi[c - 1] + add) + p) / 2.0), a2 = mob(((phi[c + 1] + add) + p) / 2.0);
  const double a3 = mob(((phi[c - sy] + add) + p) / 2.0), a4 = mob(((phi[c + sy] + add) + p) / 2.0);
  const double a5 = mob((k == 1) ? p : ((phi[c - sz] + add) + p) / 2.0);
  const double a6 = mob(((phi[c + sz] + add) + p) / 2.0);
  const double bc = e0[c], lc = l0[c];
  const double temp1 = (a2 * (e0[c + 1] - bc) - a1 * (bc - e0[c - 1])) * q.rdx2 +
                       (a4 * (e0[c + sy] - bc) - a3 * (bc - e0[c - sy])) * q.rdy2 +
                       (a6 * (e0[c + sz] - bc) - a5 * (bc - e0[c - sz])) * q.rdz2;
  const double temp2 = (l0[c + 1] - 2.0 * lc + l0[c - 1]) * q.rdx2 + (l0[c + sy] - 2.0 * lc + l0[c - sy]) * q.rdy2 +
                       (l0[c + sz] - 2.0 * lc + l0[c - sz]) * q.rdz2;
  const double temp3 = (a2 * (l0[c + 1] - lc) - a1 * (lc - l0[c - 1])) * q.rdx2 +
                       (a4 * (l0[c + sy] - lc) - a3 * (lc - l0[c - sy])) * q.rdy2 +
                       (a6 * (l0[c + sz] - lc) - a5 * (lc - l0[c - sz])) * q.rdz2;
  const double temp4 = (temp1 - q.epn2 * temp3) * q.repn - q.c_nt2 * lc + q.c_en2 * temp2;
  const double temp5 = temp4 * q.rpe - conv2[c];
  const double source0 = temp5 * 2.0 - cprev[c];
  cprev[c] = temp5;
  base[c] = q.ar * (2.0 * p - 0.5 * (phio[c] + addo) + q.dt * source0);
}

// :243-283 d2phi = grad^2(phiNew) with its ghost copies
__global__ void __launch_bounds__(DM_BX *DM_BY)
    k_dim_lap(Geo g, DimK q, const double *__restrict__ pin, double *__restrict__ l) {
  Pt t;
  if (!dim_point(g, t)) return;
  const double v = lap7(g, q, pin, 0.0, t.c);
  first_order(g, t, [&](int o) { l[o] = v; });
}

// v clamped to [0, 1] as `if (v < 0) v = 0; if (v > 1) v = 1` does (NaN and -0
// stay), by the bit pattern
__device__ __forceinline__ double clamp01(double v) {
  const int hi = __double2hiint(v), lo = __double2loint(v), mag = hi & 0x7fffffff;
  const bool nan = mag > 0x7ff00000 || (mag == 0x7ff00000 && lo != 0);
  if (nan) return v;
  if (hi < 0) return (mag | lo) ? 0.0 : v;
  return (hi > 0x3ff00000 || (hi == 0x3ff00000 && lo != 0)) ? 1.0 : v;
}

// One SOR iteration's new iterate, every position (:286-360): interior
// updates (bulkE0 = grad^2(d2phi) formed on the fly), the z ghost copies, the
// periodic y rows (taken after the z copies and before this iteration's x
// columns), the inlet profile and the outlet copy; positions no rule sets keep
// the old value.  With the iterations' common part in `base` the update is 11
// FP64 operations: 18 iterations with their Laplacians at 64x32x48 measured
// 227 us, and 542 us with a thread per ghost element, the full
// expression and the inlet's tanh per element.
__global__ void __launch_bounds__(DM_BX *DM_BY)
    k_dim_update(Geo g, DimK q, const double *__restrict__ base, const double *__restrict__ pin,
                 const double *__restrict__ l, double *__restrict__ pout) {
  Pt t;
  if (!dim_point(g, t)) return;
  const int c = t.c, wrap = g.sy * g.ny;
  const double lc = l[c];
  double v = fma(q.c_p, pin[c], base[c]);
  v = fma(q.c_l, lc, v);
  v = fma(q.c_bx, fma(-2.0, lc, l[c + 1]) + l[c - 1], v);
  v = fma(q.c_by, fma(-2.0, lc, l[c + g.sy]) + l[c - g.sy], v);
  v = fma(q.c_bz, fma(-2.0, lc, l[c + g.sz]) + l[c - g.sz], v);
  v = clamp01(v);
  // w(q) for the element q of this level and of the ghost plane beside it
  auto planes = [&](int o, auto w) {
    w(o);
    if (t.k == 1) w(o - g.sz);
    if (t.k == g.nz) w(o + g.sz);
  };
  auto put = [&](int o) { pout[o] = v; };
  planes(c, put);
  if (t.j == 1) planes(c + wrap, put);
  if (t.j == g.ny) planes(c - wrap, put);
  if (t.i == 1 || t.i == g.nx) {
    const int x = (t.i == 1) ? c - 1 : c + 1;  // the x ghost element
    // beyond k 1..nz untouched; the y ghost rows copy the old rows ny and 1
    planes(x, [&](int o) { pout[o] = pin[o]; });
    if (t.j == 1) planes(x, [&](int o) { pout[o + wrap] = pin[o]; });
    if (t.j == g.ny) planes(x, [&](int o) { pout[o - wrap] = pin[o]; });
    pout[x] = (t.i == 1) ? l[inlet_slot(g, t.k)] : v;
  }
}

// :611 phi3 = phiNew - 0.5 (every position), written to the state phi2 and
// to the next step's starting guess
__global__ void __launch_bounds__(DM_BX *DM_BY)
    k_dim_finish(Geo g, const double *__restrict__ pfin, double *__restrict__ phi2, double *__restrict__ phi3) {
  const int i = blockIdx.x * DM_BX + threadIdx.x, j = blockIdx.y * DM_BY + threadIdx.y, k = blockIdx.z;
  if (i > g.nx + 1 || j > g.ny + 1) return;
  const int c = TPLS_IDX(g, i, j, k);
  const double v = pfin[c] - 0.5;
  phi2[c] = v;
  phi3[c] = v;
}

DimK dim_constants(const Phys &ph, double epn, double pe) {
  const double nmda = 0.25, tao = 0.25, alfa1 = 1.1;
  DimK q;
  q.rdx2 = 1.0 / ph.dx / ph.dx;
  q.rdy2 = 1.0 / ph.dy / ph.dy;
  q.rdz2 = 1.0 / ph.dz / ph.dz;
  q.epn2 = epn * epn;
  q.repn = 1.0 / epn;
  q.rpe = 1.0 / pe;
  q.c_nt2 = nmda * tao / 2.0;
  q.c_en2 = q.epn2 * nmda / 2.0;
  q.dt = ph.dt;
  // :236-238 (dx**2.d0 folds to dx*dx; dx**4.d0 is a pow)
  const double a1 = 1.0 / (ph.dx * ph.dx) + 1.0 / (ph.dy * ph.dy) + 1.0 / (ph.dz * ph.dz);
  const double a2 = 2.0 / pow(ph.dx, 4.0) + 2.0 / pow(ph.dy, 4.0) + 2.0 / pow(ph.dz, 4.0);
  const double diagonal = 1.5 + nmda / 2.0 / pe * ph.dt * (2.0 * tao * a1 + q.epn2 * (4.0 * a1 * a1 + a2));
  q.ar = alfa1 * (1.0 / diagonal);
  const double kc = ph.dt * nmda / 2.0 / pe;
  q.c_p = 1.0 - 1.5 * q.ar;
  q.c_l = q.ar * kc * tao;
  q.c_bx = -q.ar * kc * q.epn2 * q.rdx2;
  q.c_by = -q.ar * kc * q.epn2 * q.rdy2;
  q.c_bz = -q.ar * kc * q.epn2 * q.rdz2;
  q.dz = ph.dz;
  q.height = ph.height;
  q.zden = 2.0 * sqrt(2.0) * epn;
  return q;
}

static dim3 full_p_grid(const Geo &g) {
  return dim3((g.nx + 2 + DM_BX - 1) / DM_BX, (g.ny + 2 + DM_BY - 1) / DM_BY, g.nz + 2);
}

static dim3 interior_grid(const Geo &g) {
  return dim3((g.nx + DM_BX - 1) / DM_BX, (g.ny + DM_BY - 1) / DM_BY, g.nz);
}

cudaError_t launch_dim_prep(const Geo &g, const DimK &q, const double *phi, double add, double *e0, double *l0,
                            cudaStream_t st) {
  k_dim_prep<<<interior_grid(g), dim3(DM_BX, DM_BY), 0, st>>>(g, q, phi, add, e0, l0);
  return cudaGetLastError();
}
cudaError_t launch_dim_source(const Geo &g, const DimK &q, const double *phi, double add, const double *phio,
                              double addo, const double *e0, const double *l0, const double *conv2, double *cprev,
                              double *base, cudaStream_t st) {
  k_dim_source<<<interior_grid(g), dim3(DM_BX, DM_BY), 0, st>>>(g, q, phi, add, phio, addo, e0, l0, conv2, cprev,
                                                                 base);
  return cudaGetLastError();
}
cudaError_t launch_dim_lap(const Geo &g, const DimK &q, const double *pin, double *l, cudaStream_t st) {
  k_dim_lap<<<interior_grid(g), dim3(DM_BX, DM_BY), 0, st>>>(g, q, pin, l);
  return cudaGetLastError();
}
cudaError_t launch_dim_update(const Geo &g, const DimK &q, const double *base, const double *pin, const double *l,
                              double *pout, cudaStream_t st) {
  k_dim_update<<<interior_grid(g), dim3(DM_BX, DM_BY), 0, st>>>(g, q, base, pin, l, pout);
  return cudaGetLastError();
}
cudaError_t launch_dim_finish(const Geo &g, const double *pfin, double *phi2, double *phi3, cudaStream_t st) {
  k_dim_finish<<<full_p_grid(g), dim3(DM_BX, DM_BY), 0, st>>>(g, pfin, phi2, phi3);
  return cudaGetLastError();
}

}  // namespace tpls
