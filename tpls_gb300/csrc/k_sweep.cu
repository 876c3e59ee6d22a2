// k_sweep.cu -- Jacobi and red-black SOR sweeps of the Crank-Nicolson
// Helmholtz solve on precomputed per-point coefficient records
// (jacobi_iteration_allflux.f90:21-282, sor_iteration_allflux.f90:19-377,
// boundary rows of main_ns_hybrid.F90:756-887).
//
// k_mom_rhs writes, once per timestep, one record per point of a velocity
// component: the six neighbour coefficients and rhs/diag, already divided
// by the Helmholtz diagonal, and the odd half-sweep's factor 1.2 czm (see
// mom_column in k_momentum.cu).  A sweep
// point is then x_new = sum(c_n x_n) + b: seven FMAs instead of the face
// averages, diagonal and division of the reference's form, evaluated once
// per step instead of once per sweep: on GB300's FP64 pipe the 64-byte
// record is the cheaper side of that trade.  The FP32 sweeps of the
// FP32-mixed form take the other side: FP32 arithmetic is 64x faster, so
// they recompute the coefficients per point from the FP32 viscosity and read
// only b (4 bytes), cutting a Jacobi point from ~40 to ~16 bytes of traffic.
// Templated on the arithmetic type and the coefficient source (records,
// MuCoef, or for the per-routine odd half-sweep RefCoef).
#include <type_traits>
#include "tpls_sweep.cuh"

namespace tpls {

// bz = 1.2 zm, the factor of the odd half-sweep's column recurrence.  The
// FP64 records carry it in their eighth slot (written by k_mom_rhs by the
// same multiplication, so the values are identical), loaded with b instead
// of computed in every odd half-sweep on the FP64 pipe.
template <typename T>
struct Rec {
  T xp, xm, yp, ym, zp, zm, b, bz;
};

// record of point c of the FP64 sweeps (8 doubles; `stream` = evict-first loads)
__device__ __forceinline__ Rec<double> load_rec(const double *__restrict__ coef, int c, bool stream) {
  const double2 *r = reinterpret_cast<const double2 *>(coef + 8 * (size_t)c);
  const double2 a = stream ? __ldcs(r) : __ldg(r), b = stream ? __ldcs(r + 1) : __ldg(r + 1);
  const double2 d = stream ? __ldcs(r + 2) : __ldg(r + 2), e = stream ? __ldcs(r + 3) : __ldg(r + 3);
  Rec<double> q = {a.x, a.y, b.x, b.y, d.x, d.y, e.x, e.y};
  return q;
}

template <typename T>
__device__ __forceinline__ T rec_apply(const Rec<T> &q, T xp, T xm, T yp, T ym, T zp, T zm) {
  T v = fma(q.xp, xp, q.b);
  v = fma(q.xm, xm, v);
  v = fma(q.yp, yp, v);
  v = fma(q.ym, ym, v);
  v = fma(q.zp, zp, v);
  return fma(q.zm, zm, v);
}

// Coefficients of point (i, j, k): the FP64 form reads its record; the FP32
// sweeps recompute the six coefficients from the FP32 viscosity exactly as
// the right-hand side kernels do (face averages, diagonal, wall rule folded
// into the z slots for u and v) and read b alone.
__device__ __forceinline__ Rec<double> get_rec(int, const Geo &g, const double *__restrict__ coef, int c, int i,
                                               int, int, bool stream) {
  return load_rec(coef, rec_slot(g, c, i), stream);
}
__device__ __forceinline__ Rec<float> get_rec(int comp, const Geo &g, const MuCoef &s, int c, int i, int j, int k,
                                              bool stream) {
  const FcT<float> f = faces<float>(comp, g, s.mu, i, j, k);
  const float diag = 1.0f + s.ax2 * (f.px + f.mx) + s.ay2 * (f.py + f.my) + s.az2 * (f.pz + f.mz);
  const float r = __fdividef(1.0f, diag);  // diag >= 1: the fast reciprocal is within 2 ulp
  float czp = s.az2 * f.pz * r, czm = s.az2 * f.mz * r;
  if (comp != 2) {
    if (k == 0) {
      czp += czm * (float)(1.0 / 3.0);
      czm = -2.0f * czm;
    } else if (k == g.nz - 1) {
      czm += czp * (float)(1.0 / 3.0);
      czp = -2.0f * czp;
    }
  }
  const float *bp = s.b + rec_slot(g, c, i);
  Rec<float> q = {s.ax2 * f.px * r, s.ax2 * f.mx * r, s.ay2 * f.py * r, s.ay2 * f.my * r, czp, czm,
                  stream ? __ldcs(bp) : __ldg(bp), 1.2f * czm};
  return q;
}

// The per-routine entries (sor_iteration_allflux.f90 on host arrays): A and B
// of point (i, j, k) of the odd half-sweep from the FP64 viscosity (ref_point),
// x the field, zp its value above (unused at the wall levels of u and v).
// near and lo in, near1 and hi out, as ref_point.  (112 us per half-sweep of a
// component at 192x96x144, where the segment kernel's bound of 5 blocks, chosen
// for the record form, spills 424 bytes of a thread's 48 registers; with the
// coefficients normalised one by one by a division 163.)
template <int CC>
__device__ __forceinline__ void ref_odd(const Geo &g, const RefCoef &s, const double *__restrict__ x,
                                        const double *m, int c, int k, int k0, double xc, double zp, double near,
                                        double lo, double &near1, double &hi, double &A, double &B) {
  double h;
  double t =
      ref_point<CC, true>(g, s, m, near, lo, s.rhs[c], x[c + 1], x[c - 1], x[c + g.sy], x[c - g.sy], hi, near1, h);
  double below = lo;  // weight of the point below
  double zt = zp;
  if (CC != 2 && k == g.nz - 1) {  // ghost -2 x + x(k-1)/3 above
    zt = -2.0 * xc;
    below = fma(hi, 1.0 / 3.0, lo);
  }
  t = fma(s.cz, hi * zt, t);
  B = 0.0;
  if (k == k0) {  // the wall value (w) or the ghost -2 x + x(k+1)/3 (u, v) below
    const double zm = (CC == 2) ? x[c - g.sz] : fma(zp, 1.0 / 3.0, -2.0 * xc);
    t = fma(s.cz, lo * zm, t);
  } else {
    B = ((1.2 * s.cz) * h) * below;
  }
  A = fma(1.2, fma(t, h, -xc), xc);
}

// The FP64 sweeps run every component of the set in one launch (gx blocks
// along x each): the components are independent, and one after the other they
// left a small channel's SMs idle (32 blocks per launch at 64x32x48) and
// every launch with a tail of its own.
// Jacobi: x = J(xo) on a component's interior with its boundary rows, ghost
// rows included (out of place, so no row read is written); ZERO: xo = 0, so
// x = b, the records' other entries neither read nor multiplied.
template <int SW_X, int SW_Y, bool ZERO>
__global__ void __launch_bounds__(SW_X *SW_Y)
    k_jacobi_c(Geo g, Helm h, const __grid_constant__ SweepSet64 S, int gx, const double *__restrict__ P) {
  const int q3 = blockIdx.x / gx, comp = S.id[q3];
  const int i = (blockIdx.x - q3 * gx) * SW_X + threadIdx.x + 1, j = blockIdx.y * SW_Y + threadIdx.y + 1;
  const int k = blockIdx.z + (comp == 2 ? 1 : 0);
  const int iend = (comp == 0) ? g.nx - 1 : g.nx;
  if (i > iend || j > g.ny || k > g.nz - 1) return;
  const int c = TPLS_IDX(g, i, j, k), sy = g.sy, sz = g.sz;
  double *x = S.x[q3];
  double v;
  if constexpr (ZERO) {
    v = __ldg(S.coef[q3] + 8 * (size_t)rec_slot(g, c, i) + 6);
  } else {
    const double *__restrict__ xo = S.xo[q3];
    const Rec<double> q = get_rec(comp, g, S.coef[q3], c, i, j, k, false);
    const double xc = xo[c];
    double zp, zm;
    if (comp == 2) {
      zp = xo[c + sz];
      zm = xo[c - sz];
    } else {  // walls folded into the record: the z slot multiplies the point itself
      zp = (k == g.nz - 1) ? xc : xo[c + sz];
      zm = (k == 0) ? xc : xo[c - sz];
    }
    v = rec_apply(q, xo[c + 1], xo[c - 1], xo[c + sy], xo[c - sy], zp, zm);
  }
  put(g, x, i, j, k, v, 1);
  const bool edge = (i == 1) || (i >= g.nx - 1) || (comp == 2 && (k == 1 || k == g.nz - 1));
  if (edge) jacobi_bc(comp, g, h, x, (const double *)nullptr, P, i, j, k, v, 1);
}

// 3-D checkerboard half-sweep (even iteration_time), one thread per point
// of the colour.
template <int SW_X, int SW_Y>
__global__ void __launch_bounds__(SW_X *SW_Y)
    k_sor_even_c(Geo g, Helm h, const __grid_constant__ SweepSet64 S, int gx, const double *__restrict__ P, int flg,
                 int bc, int fuse) {
  const int q3 = blockIdx.x / gx, comp = S.id[q3];
  const int i2 = (blockIdx.x - q3 * gx) * SW_X + threadIdx.x, j = blockIdx.y * SW_Y + threadIdx.y + 1;
  const int k = blockIdx.z + (comp == 2 ? 1 : 0);
  const int iend = (comp == 0) ? g.nx - 1 : g.nx;
  if (i2 > (iend - 1) / 2 || j > g.ny || k > g.nz - 1) return;
  const int i = 2 * i2 + 1 + ((k + j + flg) & 1);
  double *__restrict__ x = S.x[q3];
  double v = 0;
  if (i <= iend) {
    const int c = TPLS_IDX(g, i, j, k), sy = g.sy, sz = g.sz;
    const Rec<double> q = get_rec(comp, g, S.coef[q3], c, i, j, k, false);
    const double xc = x[c];
    double zp, zm;
    if (comp == 2) {
      zp = x[c + sz];
      zm = x[c - sz];
    } else {
      zp = (k == g.nz - 1) ? xc : x[c + sz];
      zm = (k == 0) ? xc : x[c - sz];
    }
    const double res = rec_apply(q, x[c + 1], x[c - 1], x[c + sy], x[c - sy], zp, zm);
    v = xc + 1.2 * (res - xc);
    put(g, x, i, j, k, v, fuse);
  }
  if (bc) sor_bc(comp, g, h, x, (const double *)nullptr, P, i2, i, iend, v, j, k, fuse);
}

// Odd-iteration half-sweep (2-D colouring, sequential in k).  Within such a
// half-sweep every value a point reads is the pre-sweep value except the
// relaxed point below it in its own column, so the update is the recurrence
//   x_new(k) = A(k) + B(k) x_new(k-1),
//   A = x + 1.2 (partial - x),  B = 1.2 czm   (partial = all terms but czm),
// with A and B known before the sweep; the column is split into chunks whose
// recurrences run in parallel from a zero start and are then joined:
// x = y + P x_in, with y the chunk-local solution, P the product of the B
// factors since the chunk start and x_in the value entering the chunk.
// Coefficient records are streamed (evict-first) so the x field stays
// resident in L2.
//
// The kernel walks the column in super-chunks of SOC_SC levels with a
// carried value, so shared memory stays bounded for any column length (36 KB for
// FP64) and several blocks share an SM.  Per super-chunk:
//   1. produce: A and B of every (level, column) pair, a warp per level and
//      a lane per column, all pairs independent (their loads overlap);
//   2. scan: warp w runs the recurrence over its SOC_SC/SOC_W levels from a
//      zero start, keeping y(k) and P(k) = prod B in place of A and B;
//   3. each warp folds the chunk ends below it and the carried value into
//      x_in and writes x = y + P x_in with the boundary rows; the last
//      level's x is carried into the next super-chunk.
// The rounding differs from the level-by-level order (the oracle's) by a
// few ulp.
// FP64 columns of one or two super-chunks: the chunks are of equal length and
// so are the warps' runs in one (75 levels: 2 x 38 in runs of 5 instead of 64
// and 11 in runs of 8), since a chunk takes as long as its busiest warp's
// chain: 16 half-sweeps 453 -> 411 us at 100x50x75, 195 -> 172 at 37x19x23, 640 ->
// 627 at 128x64x96.  Longer columns, which run by segments, keep 64 and 8, known
// at compile time (3433 us at 256x128x192, 3482 with lengths at run time), and so
// does FP32: another split would round differently, which the FP32-mixed
// form's later steps amplify to its own accuracy.
constexpr int SOC_W = 8, SOC_SC = 64;
template <typename T>
__device__ __forceinline__ bool odd_even_split(int nz) {
  return sizeof(T) == 8 && nz <= 2 * SOC_SC;
}
template <typename T>
__device__ __forceinline__ int odd_chunk(int nz) {  // levels of a super-chunk
  return odd_even_split<T>(nz) ? (nz <= SOC_SC ? nz : (nz + 1) / 2) : SOC_SC;
}
template <typename T>
__device__ __forceinline__ int odd_run(int nz, int n) {  // levels of a warp in a super-chunk of n
  return odd_even_split<T>(nz) ? (n + SOC_W - 1) / SOC_W : SOC_SC / SOC_W;
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ double ld_acquire_f64(const double *p) {
  double v;
  asm volatile("ld.acquire.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_u32(unsigned *p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Phases 1 and 2 of one super-chunk (levels kc .. kc+n-1) of a tile: A and B
// of every (level, column) pair into sA/sB, then each warp's chunk scanned
// in place (y and P), its ends into ey/ep.  Synchronises the block.  A warp
// per level, all (level, column) pairs independent.
// The FP32 sweeps are bound by the latency of the loads, and more warps hide
// it better than more loads per warp: two levels at a time in 32 registers (8
// blocks, all 64 warps of an SM) measured 416 us per half-sweep of three
// components at 512x256x256, one at a time 421, four in flight at 40 registers (6
// blocks) 470.  Lanes past the row's end take the row's first point of this
// colour (and store nothing), which frees the loads of their predicates: 421
// against 444.
template <typename T, typename CS, int CC>
__device__ __forceinline__ void odd_produce_scan_levels(int comp, const Geo &g, const CS &coef,
                                                        const T *__restrict__ x, int i, int j, bool act, int k0,
                                                        int kc, int n, T (*sA)[32], T (*sB)[32], T (*ey)[32],
                                                        T (*ep)[32]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int sy_ = g.sy, sz = g.sz, nz = g.nz;
  constexpr int PER = SOC_SC / SOC_W;
  const int ic = (sizeof(T) == 4 && !act) ? 1 + ((i & 1) ^ 1) : i;
#pragma unroll(sizeof(T) == 4 ? 2 : 4)
  for (int r = 0; r < PER; r++) {
    const int lk = w + r * SOC_W, k = kc + lk;
    if (lk < n) {
      T A = 0, B = 0;
      if (sizeof(T) == 4 || act) {
        const int c = TPLS_IDX(g, ic, j, k);
        const T xc = x[c];
        T zp;
        if constexpr (std::is_same<CS, RefCoef>::value) {
          const double *m = ref_cell<CC>(g, coef, ic, j, k);
          double near, lo, near1, hi;
          ref_begin<CC>(g, m, near, lo);
          zp = (CC == 2 || k < nz - 1) ? x[c + sz] : 0.0;
          ref_odd<CC>(g, coef, x, m, c, k, k0, xc, zp, near, lo, near1, hi, A, B);
        } else {
          const Rec<T> q = get_rec(comp, g, coef, c, ic, j, k, true);
          if (comp == 2) zp = x[c + sz];
          else zp = (k == nz - 1) ? xc : x[c + sz];
          T part = fma(q.xp, x[c + 1], q.b);
          part = fma(q.xm, x[c - 1], part);
          part = fma(q.yp, x[c + sy_], part);
          part = fma(q.ym, x[c - sy_], part);
          part = fma(q.zp, zp, part);
          if (k == k0) {  // the point below is a wall value (w) or the point itself (u, v)
            const T zm = (comp == 2) ? x[c - sz] : xc;
            A = xc + (T)1.2 * (fma(q.zm, zm, part) - xc);
          } else {
            A = xc + (T)1.2 * (part - xc);
            B = (sizeof(T) == 8) ? q.bz : (T)1.2 * q.zm;
          }
        }
      }
      sA[lk][lane] = A;
      sB[lk][lane] = B;
    }
  }
  __syncthreads();
  const int per = odd_run<T>(g.nz, n), lb = w * per, le = min(n, lb + per);
  T yv = 0, pv = 1;
  for (int lk = lb; lk < le; lk++) {
    const T B = sB[lk][lane];
    yv = fma(B, yv, sA[lk][lane]);
    pv = B * pv;
    sA[lk][lane] = yv;
    sB[lk][lane] = pv;
  }
  ey[w][lane] = yv;  // an empty chunk passes x_in through (y 0, P 1)
  ep[w][lane] = pv;
  __syncthreads();
}

// The same for the FP64 sweeps (bound by the FP64 pipe): each warp marches
// up its own PER consecutive levels and steps its chunk's recurrence as it
// goes, B read from the record (bz), the point above a level becoming the
// next level's centre value, no block barrier between production and scan.
// The operations per level and their order are those above, so both forms
// give the results of the whole-column form bit for bit.  With B from the
// record and the segment kernel's once-per-block fold, this form measured
// 10% faster than the level form for the FP64 sweeps at 256x128x192 and
// 11% slower for the FP32 sweeps at 512x256x256.
template <typename T, typename CS, int CC>
__device__ __forceinline__ void odd_produce_scan(int comp, const Geo &g, const CS &coef, const T *__restrict__ x,
                                                 int i, int j, bool act, int k0, int kc, int n,
                                                 T (*sA)[32], T (*sB)[32], T (*ey)[32], T (*ep)[32]) {
  if constexpr (sizeof(T) == 4) {
    odd_produce_scan_levels<T, CS, CC>(comp, g, coef, x, i, j, act, k0, kc, n, sA, sB, ey, ep);
  } else {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int sy_ = g.sy, sz = g.sz, nz = g.nz;
    constexpr int PER = SOC_SC / SOC_W;
    const int lb = w * PER, le = min(n, lb + PER);
    T yv = 0, pv = 1;
    int c = act ? TPLS_IDX(g, i, j, kc + lb) : 0;
    T xc = (act && lb < le) ? x[c] : (T)0;
    constexpr bool REF = std::is_same<CS, RefCoef>::value;
    double near = 0.0, lo = 0.0;  // REF: viscosities carried up the column
    const double *m = nullptr;
    if constexpr (REF) {
      if (act && lb < le) {
        m = ref_cell<CC>(g, coef, i, j, kc + lb);
        ref_begin<CC>(g, m, near, lo);
      }
    }
#pragma unroll
    for (int l = 0; l < PER; l++) {
      const int lk = lb + l, k = kc + lk;
      if (lk < le) {
        T A = 0, B = 0;
        if (act) {
          T zp;
          if constexpr (REF) {
            double near1, hi;
            zp = (CC == 2 || k < nz - 1) ? x[c + sz] : 0.0;
            ref_odd<CC>(g, coef, x, m, c, k, k0, xc, zp, near, lo, near1, hi, A, B);
            near = near1;
            lo = hi;
            m += g.szm;
          } else {
            const Rec<T> q = get_rec(comp, g, coef, c, i, j, k, true);
            if (comp == 2) zp = x[c + sz];
            else zp = (k == nz - 1) ? xc : x[c + sz];
            T part = fma(q.xp, x[c + 1], q.b);
            part = fma(q.xm, x[c - 1], part);
            part = fma(q.yp, x[c + sy_], part);
            part = fma(q.ym, x[c - sy_], part);
            part = fma(q.zp, zp, part);
            if (k == k0) {
              const T zm = (comp == 2) ? x[c - sz] : xc;
              A = xc + (T)1.2 * (fma(q.zm, zm, part) - xc);
            } else {
              A = xc + (T)1.2 * (part - xc);
              B = q.bz;
            }
          }
          xc = zp;  // x(k+1), the centre of the next level (unused after k = nz-1)
          c += sz;
        }
        yv = fma(B, yv, A);
        pv = B * pv;
        sA[lk][lane] = yv;
        sB[lk][lane] = pv;
      }
    }
    ey[w][lane] = yv;  // an empty chunk passes x_in through (y 0, P 1)
    ep[w][lane] = pv;
    __syncthreads();
  }
}

// x at the super-chunk's last level given the value entering it (what phase
// 3 writes there, by the same operations); 0 for a column outside the grid.
template <typename T>
__device__ __forceinline__ T odd_last_value(T xin, int n, bool col_in, T (*sA)[32], T (*sB)[32], T (*ey)[32],
                                            T (*ep)[32]) {
  const int lane = threadIdx.x & 31;
  constexpr int PER = SOC_SC / SOC_W;
  const int wl = (n - 1) / PER;
  for (int v = 0; v < wl; v++) xin = fma(ep[v][lane], xin, ey[v][lane]);
  return col_in ? fma(sB[n - 1][lane], xin, sA[n - 1][lane]) : (T)0;
}

// Boundary rows of a warp's levels lb .. le-1 (at most eight) of tile bx, after
// its writes: a lane per level, lanes 0-15 for the first pair and 16-31 for the
// last, so that the loads of all levels are in flight at once (by the pairs'
// own lanes, level after level, they took 4.6 of 14.4 us at 64x32x48, 16 of 50 at
// 192x96x112 in FP32; 16 half-sweeps now 222 instead of 237, and 608 instead of
// 730).  The point a boundary copies was relaxed here (in sA) or
// is of the other colour and final.  Nothing else in this sweep reads the
// boundary values of these levels.  first: the relaxed point of the first pair.
template <typename T>
__device__ __forceinline__ void odd_bc(int comp, const Geo &g, const Helm &h, T *__restrict__ x,
                                       const double *__restrict__ X, const double *__restrict__ P, int fuse, int bx,
                                       int first, int j, int iend, int kc, int lb, int le, T (*sA)[32]) {
  const int last = (iend - 1) / 2;
  if (bx != 0 && bx != last / 32) return;
  __syncwarp();
  const int lane = threadIdx.x & 31, right = lane >> 4, lk = lb + (lane & 15), i2 = right ? last : 0;
  if (lk >= le || bx != i2 / 32) return;
  const int ib = right ? iend : 1;
  const T src = (2 * i2 + first != ib) ? x[TPLS_IDX(g, ib, j, kc + lk)] : sA[lk][i2 & 31];
  sor_bc(comp, g, h, x, X, P, i2, ib, iend, src, j, kc + lk, fuse);
}

// Phase 3: each warp writes x = y + P x_in from the value entering its own
// chunk (given in xin for FP64; for FP32 xin enters the super-chunk and the
// warp folds the chunk ends below its own into it first), then the
// boundary rows of its levels.  Returns x at the super-chunk's last level
// for the warp that owns it (0 elsewhere).
template <typename T>
__device__ __forceinline__ T odd_write(int comp, const Geo &g, const Helm &h, T *__restrict__ x,
                                       const double *__restrict__ X, const double *__restrict__ P, int bc,
                                       int fuse, int i2, int i, int j, int iend, int npair, int kc, int n, T xin,
                                       T (*sA)[32], T (*sB)[32], T (*ey)[32], T (*ep)[32]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int PER = SOC_SC / SOC_W;
  const int lb = w * PER, le = min(n, lb + PER);
  T last = 0;
  if constexpr (sizeof(T) == 4)
    for (int v = 0; v < w; v++) xin = fma(ep[v][lane], xin, ey[v][lane]);
  if (i2 < npair) {
    for (int lk = lb; lk < le; lk++) {
      T v = 0;
      if (i <= iend) {
        v = fma(sB[lk][lane], xin, sA[lk][lane]);
        put(g, x, i, j, kc + lk, v, fuse);
      }
      sA[lk][lane] = v;  // kept for the boundary rows below
      if (lk == n - 1) last = v;
    }
  }
  if (bc) odd_bc<T>(comp, g, h, x, X, P, fuse, (i2 - lane) / 32, 1 + ((i & 1) ^ 1), j, iend, kc, lb, le, sA);
  return last;
}

// Shared memory of a block of the odd half-sweep: A and B (then y and P) of
// a super-chunk, the chunk ends, and the values carried between super-chunks
// or entering each warp's chunk (FP64) or the segment (FP32).
template <typename T>
struct OddShared {
  T A[SOC_SC][32], B[SOC_SC][32], ey[SOC_W][32], ep[SOC_W][32], xin[sizeof(T) == 8 ? SOC_W : 1][32];
};

// One tile: 32 columns (x pairs from bx*32) of row j = by+1, the whole
// column.  Every thread of the block runs it (it synchronises the block).
// The segment kernel below runs the same phases by the helpers above, one
// super-chunk per block.
template <typename T, typename CS, int CC>
__device__ __forceinline__ void sor_odd_c4_tile(int comp_, const Geo &g, const Helm &h, T *__restrict__ x,
                                                const CS &coef, const double *__restrict__ P,
                                                const double *__restrict__ X, int flg, int bc, int fuse, int bx,
                                                int by, OddShared<T> &sh) {
  const int comp = (CC >= 0) ? CC : comp_;
  T(&sA)[SOC_SC][32] = sh.A, (&sB)[SOC_SC][32] = sh.B, (&ey)[SOC_W][32] = sh.ey, (&ep)[SOC_W][32] = sh.ep;
  T(&scarry)[32] = sh.xin[0];
  const int j = by + 1;
  const int iend = (comp == 0) ? g.nx - 1 : g.nx;
  const int npair = (iend + 1) / 2;
  const int par = (j + flg) & 1;
  const int k0 = (comp == 2) ? 1 : 0, k1 = g.nz - 1;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i2 = bx * 32 + lane, i = 2 * i2 + 1 + par;
  const bool act = (i2 < npair) && (i <= iend);
  T carry = 0;  // x of the level below the super-chunk (k0 has B = 0)
  const int sc = odd_chunk<T>(g.nz);
  for (int kc = k0; kc <= k1; kc += sc) {
    const int n = min(sc, k1 - kc + 1);
    odd_produce_scan_levels<T, CS, CC>(comp, g, coef, x, i, j, act, k0, kc, n, sA, sB, ey, ep);  // 1. produce, 2. scan
    const int per = odd_run<T>(g.nz, n), lb = w * per, le = min(n, lb + per);
    // 3. fold and write
    T xin = carry;
    for (int v = 0; v < w; v++) xin = fma(ep[v][lane], xin, ey[v][lane]);
    if (i2 < npair) {
      for (int lk = lb; lk < le; lk++) {
        T v = 0;
        if (i <= iend) {
          v = fma(sB[lk][lane], xin, sA[lk][lane]);
          put(g, x, i, j, kc + lk, v, fuse);
        }
        sA[lk][lane] = v;  // kept for the boundary rows below
        if (lk == n - 1) scarry[lane] = v;
      }
    }
    if (bc) odd_bc<T>(comp, g, h, x, X, P, fuse, bx, 1 + par, j, iend, kc, lb, le, sA);
    __syncthreads();
    carry = scarry[lane];
  }
}

// Odd half-sweep with one block per super-chunk of a tile (segment), for
// columns of several segments (odd_set; FP64 records, the FP32 sweeps and the
// per-routine entries alike), so a launch has nz/64 times the blocks of
// the whole-column form and the blocks' load, scan and write phases
// overlap.
// The value entering a segment is the last value of the segment below it:
// segments are taken in ticket order, lowest segment of every tile first,
// so the block a segment waits for took its ticket earlier and is running;
// it publishes that value (the same operations as the whole-column form,
// so the results are bit-identical to it) as soon as it has its own
// entering value, before it writes.  The wait is bounded: if it runs out
// the block counts it in *kto, takes NaN as its entering value (the step's
// pressure solve then reports DIVERGED_NAN) and still publishes, so no
// later segment waits on it.
// The columns of every component of the set form one list of tiles.
template <typename T, typename CS, int CC>
__device__ __forceinline__ void sor_odd_segment(int comp_, const Geo &g, const Helm &h, T *__restrict__ x,
                                                const CS &coef, const double *__restrict__ P,
                                                const double *__restrict__ X, int flg, int bc, int fuse,
                                                const OddChain &oc, int limit, unsigned t, unsigned epoch, int nct,
                                                int seg, int bx, int j, OddShared<T> &sh) {
  const int comp = (CC >= 0) ? CC : comp_;
  T(&sA)[SOC_SC][32] = sh.A, (&sB)[SOC_SC][32] = sh.B, (&ey)[SOC_W][32] = sh.ey, (&ep)[SOC_W][32] = sh.ep;
  auto &sxin = sh.xin;
  const int iend = (comp == 0) ? g.nx - 1 : g.nx;
  const int npair = (iend + 1) / 2;
  const int par = (j + flg) & 1;
  const int k0 = (comp == 2) ? 1 : 0, k1 = g.nz - 1;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i2 = bx * 32 + lane, i = 2 * i2 + 1 + par;
  const bool act = (i2 < npair) && (i <= iend);
  const int kc = k0 + seg * SOC_SC, n = min(SOC_SC, k1 - kc + 1);
  if (n <= 0) return;  // w's columns are a level shorter: its last segment can be empty (none waits for it)
  constexpr int PER = SOC_SC / SOC_W;
  odd_produce_scan<T, CS, CC>(comp, g, coef, x, i, j, act, k0, kc, n, sA, sB, ey, ep);
  if (w == 0) {
    T xin = 0;  // k0 has B = 0
    if (seg > 0) {
      // every lane acquires the flag itself (one transaction per poll for
      // the warp) before reading its column's value
      const unsigned pt = t - (unsigned)nct;  // the segment below, same columns
      bool ok = true;
      int it = 0;
      while (ld_acquire_u32(&oc.flag[pt]) != epoch + 1u)
        if (++it >= limit) {
          ok = false;
          break;
        }
      xin = ok ? (T)ld_acquire_f64(&oc.incl[(size_t)pt * 32 + lane]) : (T)__longlong_as_double(0x7ff8000000000000ll);
      if (__any_sync(0xffffffffu, !ok) && lane == 0) atomicAdd(oc.kto, 1.0);
    }
    if constexpr (sizeof(T) == 8) {
      // FP64: the value entering every warp's chunk, the chunk ends below
      // it folded in order, once for the block instead of once per warp
      T xw = xin;
#pragma unroll
      for (int v = 0; v < SOC_W; v++) {
        sxin[v][lane] = xw;
        if (v + 1 < SOC_W) xw = fma(ep[v][lane], xw, ey[v][lane]);
      }
      if (seg < (k1 - k0) / SOC_SC) {  // a segment above waits for this one
        oc.incl[(size_t)t * 32 + lane] =
            act ? fma(sB[n - 1][lane], sxin[(n - 1) / PER][lane], sA[n - 1][lane]) : (T)0;
        __threadfence();
        __syncwarp();
        if (lane == 0) st_release_u32(&oc.flag[t], epoch + 1u);
      }
    } else {
      if (seg < (k1 - k0) / SOC_SC) {  // a segment above waits for this one
        oc.incl[(size_t)t * 32 + lane] = (double)odd_last_value<T>(xin, n, i2 < npair && i <= iend, sA, sB, ey, ep);
        __threadfence();
        __syncwarp();
        if (lane == 0) st_release_u32(&oc.flag[t], epoch + 1u);
      }
      sxin[0][lane] = xin;
    }
  }
  __syncthreads();
  odd_write<T>(comp, g, h, x, X, P, bc, fuse, i2, i, j, iend, npair, kc, n, sxin[sizeof(T) == 8 ? w : 0][lane], sA,
               sB, ey, ep);
}

// One component's work on a tile, the component a compile-time constant for
// the sweeps that form face viscosities (FP32, per-routine entries: these
// differ by component).
#define TPLS_BY_COMP(CALL)                        \
  do {                                            \
    if constexpr (!std::is_same<CS, const double *>::value) { \
      if (comp == 0) CALL(0);                     \
      else if (comp == 1) CALL(1);                \
      else CALL(2);                               \
    } else {                                      \
      CALL(-1);                                   \
    }                                             \
  } while (0)

// BC: with the boundary rows (the second half-sweep); the launches without
// them then carry none of their registers.
template <typename T, typename CS, bool BC>
__global__ void __launch_bounds__(SOC_W * 32, sizeof(T) == 4 ? 8 : 5)  // 32 / 48 registers: 8 / 5 blocks per SM
    k_sor_odd_seg(Geo g, Helm h, const __grid_constant__ SweepSet<T, CS> S, const double *__restrict__ P, int flg,
                  int fuse, OddChain oc, int gx, int limit) {
  __shared__ OddShared<T> sh;
  __shared__ unsigned s_t, s_ep;
  if (threadIdx.x == 0) {
    s_t = atomicAdd(&oc.ctr[0], 1u);
    s_ep = ld_acquire_u32(&oc.ctr[2]);
  }
  __syncthreads();
  const unsigned t = s_t, epoch = s_ep;
  const int nct = S.n * gx * g.ny;
  const int seg = (int)(t / (unsigned)nct), ct = (int)(t - (unsigned)seg * nct);
  const int q3 = ct / (gx * g.ny), tile = ct - q3 * gx * g.ny;
  const int comp = S.id[q3];
#define TPLS_SEG(CC)                                                                                              \
  sor_odd_segment<T, CS, CC>(comp, g, h, S.x[q3], S.coef[q3], P, S.X[q3], flg, BC, fuse, oc, limit, t, epoch, nct, \
                             seg, tile % gx, tile / gx + 1, sh)
  TPLS_BY_COMP(TPLS_SEG);
#undef TPLS_SEG
  if (threadIdx.x == 0) {  // the last block to leave resets the tickets and starts a new epoch
    __threadfence();
    if (atomicAdd(&oc.ctr[1], 1u) == gridDim.x - 1) {
      oc.ctr[0] = 0u;
      oc.ctr[1] = 0u;
      __threadfence();
      atomicAdd(&oc.ctr[2], 1u);
    }
  }
}

// (FP64: with a bound of 1 block per SM the compiler takes the registers of 2
// blocks and a half-sweep at 128x64x96 51 us instead of 40.5; bounds of 4 and
// 5 blocks measured 40.8 and 42.)
template <typename T, typename CS, bool BC>
__global__ void __launch_bounds__(SOC_W * 32, sizeof(T) == 4 ? 8 : 3)
    k_sor_odd_c4(Geo g, Helm h, const __grid_constant__ SweepSet<T, CS> S, const double *__restrict__ P, int gx,
                 int flg, int fuse) {
  __shared__ OddShared<T> sh;
  const int q3 = blockIdx.x / gx, bx = blockIdx.x - q3 * gx, comp = S.id[q3];
#define TPLS_COL(CC) \
  sor_odd_c4_tile<T, CS, CC>(comp, g, h, S.x[q3], S.coef[q3], P, S.X[q3], flg, BC, fuse, bx, blockIdx.y, sh)
  TPLS_BY_COMP(TPLS_COL);
#undef TPLS_COL
}

// Multi-instance odd half-sweep of the FP32 sweeps of a batch: the tiles of
// every member (32 columns of one row each) taken in order by an atomic
// ticket, as k_sweep4_multi.
template <int CC>
__global__ void __launch_bounds__(SOC_W * 32)
    k_odd_multi(const SweepMember *__restrict__ mem, const int *__restrict__ prefix, int n, int src, int flg,
                int bc, unsigned *ctr) {
  __shared__ OddShared<float> sh;
  __shared__ int s_t;
  const int total = prefix[n];
  for (;;) {
    if (threadIdx.x == 0) s_t = (int)atomicAdd(&ctr[0], 1u);
    __syncthreads();
    const int t = s_t;
    __syncthreads();
    if (t >= total) break;
    int m = 0;
    while (prefix[m + 1] <= t) m++;
    const SweepMember &M = mem[m];
    const int iend = (CC == 0) ? M.g.nx - 1 : M.g.nx;
    const int gx = ((iend + 1) / 2 + 31) / 32;
    const int lt = t - prefix[m];
    sor_odd_c4_tile<float, MuCoef, CC>(CC, M.g, M.h, M.x[CC][src], M.s[CC], M.P, M.X[CC], flg, bc, M.fuse,
                                       lt % gx, lt / gx, sh);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&ctr[1], 1u) == gridDim.x - 1) {
      ctr[0] = 0u;
      ctr[1] = 0u;
    }
  }
}

int odd_tiles(int comp, const Geo &g) {
  const int iend = (comp == 0) ? g.nx - 1 : g.nx;
  return (((iend + 1) / 2 + 31) / 32) * g.ny;
}

cudaError_t launch_odd_multi(int comp, const SweepMember *mem, const int *prefix, int n, int total_tiles, int src,
                             int flg, int bc, unsigned *ctr, int nblocks, cudaStream_t st) {
  const int nb = total_tiles < nblocks ? total_tiles : nblocks;
  if (nb <= 0) return cudaSuccess;
  if (comp == 0) k_odd_multi<0><<<nb, SOC_W * 32, 0, st>>>(mem, prefix, n, src, flg, bc, ctr);
  else if (comp == 1) k_odd_multi<1><<<nb, SOC_W * 32, 0, st>>>(mem, prefix, n, src, flg, bc, ctr);
  else k_odd_multi<2><<<nb, SOC_W * 32, 0, st>>>(mem, prefix, n, src, flg, bc, ctr);
  return cudaGetLastError();
}

// tile: the block shape (threads over i, or i pairs, by threads over j) the
// autotuner chooses among for the Jacobi and even-SOR kernels: 0 = 32x4 (the
// default), 1 = 32x8, 2 = 64x4, 3 = 16x8.
template <int BX, int BY>
static void jacobi_v(const Geo &g, const Helm &h, const SweepSet64 &s, const double *pres, bool zero,
                     cudaStream_t st) {
  const int gx = (g.nx + BX - 1) / BX;
  const dim3 grd(gx * s.n, (g.ny + BY - 1) / BY, g.nz), blk(BX, BY);
  if (zero) k_jacobi_c<BX, BY, true><<<grd, blk, 0, st>>>(g, h, s, gx, pres);
  else k_jacobi_c<BX, BY, false><<<grd, blk, 0, st>>>(g, h, s, gx, pres);
}
cudaError_t launch_jacobi_set(const Geo &g, const Phys &ph, const SweepSet64 &s, const double *pres, bool from_zero,
                              cudaStream_t st, const SweepTiles &t) {
  const Helm h = helm_of(ph);
  switch (t.jac) {
    case 1: jacobi_v<32, 8>(g, h, s, pres, from_zero, st); break;
    case 2: jacobi_v<64, 4>(g, h, s, pres, from_zero, st); break;
    case 3: jacobi_v<16, 8>(g, h, s, pres, from_zero, st); break;
    default: jacobi_v<32, 4>(g, h, s, pres, from_zero, st); break;
  }
  return cudaGetLastError();
}
cudaError_t launch_jacobi_set(const Geo &g, const Phys &ph, const SweepSet32 &s, const double *, bool, cudaStream_t st,
                              const SweepTiles &t) {
  return launch_sweep4(0, g, helm_of(ph), s, 0, 1, 1, t.jac, st);
}

template <int BX, int BY>
static void even_v(const Geo &g, const Helm &h, const SweepSet64 &s, const double *pres, int flg, int bc, int fuse,
                   cudaStream_t st) {
  const int gx = ((g.nx + 1) / 2 + BX - 1) / BX;
  k_sor_even_c<BX, BY><<<dim3(gx * s.n, (g.ny + BY - 1) / BY, g.nz), dim3(BX, BY), 0, st>>>(g, h, s, gx, pres, flg,
                                                                                          bc, fuse);
}
static cudaError_t even_set(const Geo &g, const Helm &h, const SweepSet64 &s, const double *pres, int flg, int bc,
                            int fuse, int tile, cudaStream_t st) {
  switch (tile) {
    case 1: even_v<32, 8>(g, h, s, pres, flg, bc, fuse, st); break;
    case 2: even_v<64, 4>(g, h, s, pres, flg, bc, fuse, st); break;
    case 3: even_v<16, 8>(g, h, s, pres, flg, bc, fuse, st); break;
    default: even_v<32, 4>(g, h, s, pres, flg, bc, fuse, st); break;
  }
  return cudaGetLastError();
}
// checkerboard half-sweep: four x points per thread (k_sweep32.cu)
static cudaError_t even_set(const Geo &g, const Helm &h, const SweepSet32 &s, const double *, int flg, int bc,
                            int fuse, int tile, cudaStream_t st) {
  return launch_sweep4(1, g, h, s, flg, bc, fuse, tile, st);
}

int odd_chain_segments(const Geo &g) {
  const int gx = (((g.nx + 1) / 2) + 31) / 32;  // v and w have the most pairs
  return 3 * ((g.nz - 1) / SOC_SC + 1) * gx * g.ny;
}

template <typename T, typename CS>
static cudaError_t odd_set(const Geo &g, const Helm &h, const SweepSet<T, CS> &s, const double *pres, int flg, int bc,
                           int fuse, cudaStream_t st, const OddChain *oc) {
  const int gx = ((g.nx + 1) / 2 + 31) / 32, nseg = (g.nz - 1) / SOC_SC + 1;
  const int blocks = nseg * s.n * gx * g.ny;
  constexpr bool rows = !std::is_same<CS, RefCoef>::value;  // the per-routine entries write no boundary rows
  // One block per segment, chained, for columns of 2 (FP32) or 3 (FP64) and
  // more segments.  With 2, half the blocks wait on the other half: the FP32
  // sweeps gain more from twice the blocks (16 half-sweeps at 192x96x112: 722
  // us, whole columns 764), the FP64 ones, bound by the FP64 pipe, do not
  // (128x64x96: 720, whole columns 646).
  if (oc && nseg >= (sizeof(T) == 4 ? 2 : 3) && oc->cap >= blocks) {
    if (rows && bc)
      k_sor_odd_seg<T, CS, rows><<<blocks, SOC_W * 32, 0, st>>>(g, h, s, pres, flg, fuse, *oc, gx, 1 << 20);
    else k_sor_odd_seg<T, CS, false><<<blocks, SOC_W * 32, 0, st>>>(g, h, s, pres, flg, fuse, *oc, gx, 1 << 20);
  } else {  // one block per 32 columns of a row, the column in super-chunks
    const dim3 grd(gx * s.n, g.ny);
    if (rows && bc) k_sor_odd_c4<T, CS, rows><<<grd, SOC_W * 32, 0, st>>>(g, h, s, pres, gx, flg, fuse);
    else k_sor_odd_c4<T, CS, false><<<grd, SOC_W * 32, 0, st>>>(g, h, s, pres, gx, flg, fuse);
  }
  return cudaGetLastError();
}

cudaError_t launch_sor_set(const Geo &g, const Phys &ph, const SweepSet64 &s, const double *pres, int flg,
                           int iteration_time, int bc, int fuse_ghosts, cudaStream_t st, const SweepTiles &t,
                           const OddChain *oc) {
  if (iteration_time % 2 == 0) return even_set(g, helm_of(ph), s, pres, flg, bc, fuse_ghosts, t.even, st);
  return odd_set(g, helm_of(ph), s, pres, flg, bc, fuse_ghosts, st, oc);
}
cudaError_t launch_sor_set(const Geo &g, const Phys &ph, const SweepSet32 &s, const double *pres, int flg,
                           int iteration_time, int bc, int fuse_ghosts, cudaStream_t st, const SweepTiles &t,
                           const OddChain *oc) {
  if (iteration_time % 2 == 0) return even_set(g, helm_of(ph), s, pres, flg, bc, fuse_ghosts, t.even, st);
  return odd_set(g, helm_of(ph), s, pres, flg, bc, fuse_ghosts, st, oc);
}

cudaError_t launch_ref_odd(int comp, const Geo &g, const RefCoef &r, double *x, int flg, cudaStream_t st,
                           const OddChain *oc) {
  SweepSet<double, RefCoef> s;
  s.n = 1;
  s.id[0] = comp;
  s.x[0] = x;
  s.coef[0] = r;
  return odd_set(g, Helm{}, s, nullptr, flg, 0, 0, st, oc);
}

MuCoef mu_coef(const Phys &ph, const float *mu, const float *b, const float4 *bco) {
  const Helm h = helm_of(ph);
  MuCoef m;
  m.mu = mu;
  m.b = b;
  m.bco = bco;
  m.ax2 = (float)h.ax2;
  m.ay2 = (float)h.ay2;
  m.az2 = (float)h.az2;
  return m;
}

// defect form: d = -X before the first sweep (the sweeps start from x = 0),
// x = X + d after the last (conversions by integer operations, tpls_pair.cuh)
__global__ void k_defect_init(const double *__restrict__ X, float *__restrict__ d, size_t n) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
    d[q] = -round_bits(X[q]);
}
__global__ void k_defect_apply(const double *__restrict__ X, const float *__restrict__ d, double *__restrict__ x,
                               size_t n) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
    x[q] = X[q] + widen_bits(d[q]);
}
cudaError_t launch_defect_init(const double *X, float *d, size_t n, cudaStream_t st) {
  k_defect_init<<<1216, 256, 0, st>>>(X, d, n);
  return cudaGetLastError();
}
cudaError_t launch_defect_apply(const double *X, const float *d, double *x, size_t n, cudaStream_t st) {
  k_defect_apply<<<1216, 256, 0, st>>>(X, d, x, n);
  return cudaGetLastError();
}

}  // namespace tpls
