"""Red-black levels of which x and y are coarsened and z is not (FP64,
csrc/tpls_mg.cuh with Z false).

CPU: the restriction and the prolongation, restated thread by thread, give the
general passes' values on ragged tiles and the smallest extents.  GPU: solves
on grids whose finest levels are of that kind, against the oracle's exact
solve."""
import numpy as np
import pytest

from tests.test_pressure_levels import _cls, _inv, _Kernels, _neighbours


def _general(b, ec, c):
    nz, ny, nx = b.shape
    inv = _inv(nx, nz, c)
    d = np.array([[[inv[_cls(i, nx), _cls(k, nz)] for i in range(nx)] for _ in range(ny)] for k in range(nz)])
    red = np.indices(b.shape).sum(0) % 2 == 0
    e = np.where(red, b * d, 0.0)
    e = np.where(red, e, (b + _neighbours(e, c)) * d)
    r = b - (e / d - _neighbours(e, c))

    def taps(n, periodic):
        R = np.zeros((n // 2, n))
        for q in range(n // 2):
            for f, w in ((2 * q - 1, 0.25), (2 * q, 0.75), (2 * q + 1, 0.75), (2 * q + 2, 0.25)):
                R[q, f % n if periodic else min(max(f, 0), n - 1)] += w
        return R
    Rx, Ry = taps(nx, False), taps(ny, True)
    bc = np.einsum("bj,ai,kji->kba", Ry, Rx, r) / 4
    e = e + np.einsum("bj,ai,kba->kji", Ry, Rx, ec)
    e = np.where(red, e, (b + _neighbours(e, c)) * d)
    return bc, np.where(red, (b + _neighbours(e, c)) * d, e)


class _Planar(_Kernels):
    def prolong(self, b, ec, e, kz):
        nx, ny, nz = self.n
        ncx, ncy = nx // 2, ny // 2
        for i2, j, k in self.pairs(kz):
            y0 = j >> 1
            y1 = (y0 + 1 if j & 1 else y0 - 1) % ncy
            odd = (j + k) & 1
            x1 = min(i2 + 1, ncx - 1) if odd else max(i2 - 1, 0)

            def column(x):
                return 3 * self.get(ec, ncx * ncy * k + ncx * y0 + x) + self.get(ec, ncx * ncy * k + ncx * y1 + x)
            o = 2 * i2 + odd + nx * (j + ny * k)
            xc = (2 if 2 * i2 + 1 == nx - 1 else 1) if odd else (0 if i2 == 0 else 1)
            e[o] = b[o] * self.inv[xc, _cls(k, nz)] + (3 * column(i2) + column(x1)) / 16

    def restrict(self, e, czb):
        nx, ny, nz = self.n
        cx, cy, cz = self.c
        ncx, ncy, gx, gy = nx // 2, ny // 2, (nx + 59) // 60, (ny + 13) // 14
        out = np.full(ncx * ncy * nz, np.nan)

        def at(i, row, k, there=True):
            return self.get(e, i + nx * row + nx * ny * k) if there else 0.0
        for blk in range(gx * gy * ((nz + czb - 1) // czb)):
            bx, by, bz = blk % gx, blk // gx % gy, blk // (gx * gy)
            y0 = by * 14
            for k in range(bz * czb, min(bz * czb + czb, nz)):
                sx = np.full((16, 32), np.nan)
                for row in range(16):
                    j = y0 - 1 + row
                    j = ny - 1 if j < 0 else (j - ny) % ny if j >= ny else j
                    odd, r = (j + k) & 1, np.full(32, np.nan)
                    for lane in range(32):
                        ic = bx * 30 - 1 + lane
                        if not 0 <= ic < ncx:
                            r[lane] = 0.0
                        elif lane != (31 if odd else 0):  # the shuffled neighbour is another warp's there
                            i = 2 * ic + odd
                            x = at(2 * ic + 1 - odd, j, k) + at(i + 1 if odd else i - 1, j, k,
                                                                i < nx - 1 if odd else i > 0)
                            r[lane] = cx * x + cy * (at(i, (j - 1) % ny, k) + at(i, (j + 1) % ny, k)) + cz * (
                                at(i, j, k - 1, k > 0) + at(i, j, k + 1, k < nz - 1))
                    for lane in range(1, 31):
                        wall = bx * 30 - 1 + lane == (ncx - 1 if odd else 0)
                        sx[row, lane] = (4 if wall else 3) * r[lane] + (r[lane - 1] if odd else r[lane + 1])
                for w in range(7):
                    for lane in range(1, 31):
                        ic, jc = bx * 30 - 1 + lane, y0 // 2 + w
                        if ic < ncx and jc < ncy:
                            s = sx[2 * w:2 * w + 4, lane]
                            out[ic + ncx * (jc + ncy * k)] = (3 * (s[1] + s[2]) + s[0] + s[3]) / 64
        return out


@pytest.mark.parametrize("size", [(4, 4, 3), (8, 6, 5), (66, 18, 7), (62, 16, 9), (6, 4, 17), (10, 4, 2)])
def test_planar_level_kernels_equal_the_general_passes(size):
    nx, ny, nz = size
    rng = np.random.default_rng(nx + 7 * nz)
    c = (1.3, 0.9, 1.1)
    b, ec = rng.normal(size=(nz, ny, nx)), rng.normal(size=(nz, ny // 2, nx // 2))
    bc, ref = _general(b, ec, c)
    K, flat = _Planar(nx, ny, nz, c), b.ravel()
    for kz, czb in ((2, 1), (8, 4)):
        e = K.black(flat, kz)
        got = K.restrict(e, czb)
        # a few dozen roundings of values of order 1
        assert np.max(np.abs(got - bc.ravel())) < 1e-13
        K.prolong(flat, ec.ravel(), e, kz)
        K.half(flat, e, 1, kz)
        K.half(flat, e, 0, kz)
        assert np.max(np.abs(e - ref.ravel())) < 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(64, 16, 15), (66, 34, 21), (126, 30, 9), (100, 50, 75), (40, 36, 50)])
def test_solves_on_planar_levels_match_the_exact_solve(size):
    """Solved to rtol 1e-13 (the preconditioner's precision does not enter
    the solution), as test_pressure_solve_tight: 1e-10 of the maximum."""
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz)
    rng = np.random.default_rng(nx)
    u3 = np.asfortranarray(st["U2"] + rng.normal(scale=1e-3, size=st["U2"].shape))
    u3[:, 0], u3[:, -1] = u3[:, -2], u3[:, 1]  # periodic rows, as the driver's exchange leaves them
    with TplsGpu(nx, ny, nz, p, uin) as g:
        o = Oracle(nx, ny, nz, p, uin)
        rhs = g.get_source_pres(u3, st["V2"], st["W2"], p.dx, p.dy, p.dz, p.dt)
        pold = np.zeros_like(st["PRES"], order="F")
        po, *_ = o.pressure_solve(pold, rhs, u3, uin, p.dx, p.dy, p.dz, p.dt)
        pg, its, _, reason = g.pressure_solve(pold, rhs, u3, uin, p.dx, p.dy, p.dz, p.dt, rtol=1e-13, maxits=400)
    assert reason == 2
    assert np.max(np.abs(pg - po)) <= 1e-10 * np.max(np.abs(po))
