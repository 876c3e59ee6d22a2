"""The red-black multigrid levels whose three axes are all halved
(csrc/tpls_mg.cuh).

CPU: the kernels' index arithmetic, restated thread by thread, stays inside
the arrays and their shared tiles and gives what the general path gives
(red-black half-sweeps, residual, restriction and prolongation as separate
passes over every point) on ragged tiles, single chunks and the smallest
extents.  GPU: solves that take those kernels, on extents at the edges of
their tiles, against the oracle's exact solve."""
import numpy as np
import pytest

EDGES = [(4, 4, 4), (8, 6, 4), (66, 18, 6), (64, 16, 20), (70, 34, 12), (6, 4, 34)]


def _inv(nx, nz, c):
    v = np.empty((3, 3))
    for a in range(3):
        for q in range(3):
            v[a, q] = 1.0 / (c[0] * (2 if a == 1 else 1) + 2 * c[1] + c[2] * (2 if q == 1 else 1))
    return v


def _cls(i, n):
    return 0 if i == 0 else 2 if i == n - 1 else 1


def _neighbours(e, c):
    """sum of coupling * neighbour, walls dropped, [k, j, i]."""
    s = c[1] * (np.roll(e, 1, 1) + np.roll(e, -1, 1))
    s[:, :, 1:] += c[0] * e[:, :, :-1]
    s[:, :, :-1] += c[0] * e[:, :, 1:]
    s[1:] += c[2] * e[:-1]
    s[:-1] += c[2] * e[1:]
    return s


def _general(b, ec, c):
    """Pre-smoothed residual restricted, and the corrected, post-smoothed
    iterate, pass by pass."""
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
                f = f % n if periodic else min(max(f, 0), n - 1)
                R[q, f] += w
        return R
    Rx, Ry, Rz = taps(nx, False), taps(ny, True), taps(nz, False)
    bc = np.einsum("ck,bj,ai,kji->cba", Rz, Ry, Rx, r) / 8
    e = e + np.einsum("ck,bj,ai,cba->kji", Rz, Ry, Rx, ec)
    e = np.where(red, e, (b + _neighbours(e, c)) * d)
    e = np.where(red, (b + _neighbours(e, c)) * d, e)
    return bc, e


class _Kernels:
    """tpls_mg.cuh on flat arrays; every index is checked."""

    def __init__(self, nx, ny, nz, c):
        self.n = (nx, ny, nz)
        self.c, self.inv = c, _inv(nx, nz, c)

    def pairs(self, kz):
        nx, ny, nz = self.n
        gx, gy = (nx // 2 + 31) // 32, (ny + 7) // 8
        for blk in range(gx * gy * ((nz + kz - 1) // kz)):
            bx, by, bz = blk % gx, blk // gx % gy, blk // (gx * gy)
            for t in range(256):
                i2, j = bx * 32 + t % 32, by * 8 + t // 32
                if 2 * i2 < nx and j < ny:
                    for k in range(bz * kz, min(bz * kz + kz, nz)):
                        yield i2, j, k

    @staticmethod
    def get(a, q):
        assert 0 <= q < a.size, q
        return a[q]

    def around(self, a, i2, j, k, odd):
        """own point, pair partner, outer x, y and z neighbours of one of the
        pair, as the kernels index them (None beyond a wall)."""
        nx, ny, nz = self.n
        plane = nx * ny
        c = 2 * i2 + nx * j + plane * k
        jm = -nx if j > 0 else plane - nx
        jp = nx if j < ny - 1 else nx - plane
        outer = 2 * i2 + 2 < nx if odd else i2 > 0
        o = c + odd
        return (o, self.get(a, c + 1 - odd), self.get(a, c + 2 if odd else c - 1) if outer else None,
                self.get(a, o + jm) + self.get(a, o + jp),
                self.get(a, o - plane) if k > 0 else None, self.get(a, o + plane) if k < nz - 1 else None)

    def black(self, b, kz):
        nx, ny, nz = self.n
        cx, cy, cz = self.c
        e = np.full(b.size, np.nan)
        for i2, j, k in self.pairs(kz):
            odd = 1 - ((j + k) & 1)
            o, xi, xout, y, zm, zp = self.around(b, i2, j, k, odd)
            xo = (2 if 2 * i2 + 1 == nx - 1 else 1) if odd else (0 if i2 == 0 else 1)
            xc = (0 if i2 == 0 else 1) if odd else (2 if 2 * i2 + 1 == nx - 1 else 1)
            zc = _cls(k, nz)
            v = b[o] + cx * self.inv[xc, zc] * xi + cy * self.inv[xo, zc] * y
            v += cx * self.inv[1, zc] * xout if xout is not None else 0.0
            v += cz * self.inv[xo, _cls(k - 1, nz)] * zm if zm is not None else 0.0
            v += cz * self.inv[xo, _cls(k + 1, nz)] * zp if zp is not None else 0.0
            e[o] = v * self.inv[xo, zc]
        return e

    def half(self, b, e, colour, kz):
        nx, ny, nz = self.n
        for i2, j, k in self.pairs(kz):
            odd = (j + k + colour) & 1
            o, xi, xout, y, zm, zp = self.around(e, i2, j, k, odd)
            xo = (2 if 2 * i2 + 1 == nx - 1 else 1) if odd else (0 if i2 == 0 else 1)
            v = b[o] + self.c[0] * (xi + (xout or 0.0)) + self.c[1] * y + self.c[2] * ((zm or 0.0) + (zp or 0.0))
            e[o] = v * self.inv[xo, _cls(k, nz)]

    def prolong(self, b, ec, e, kz):
        nx, ny, nz = self.n
        ncx, ncy, ncz = nx // 2, ny // 2, nz // 2
        for i2, j, k in self.pairs(kz):
            y0 = j >> 1
            y1 = (y0 + 1 if j & 1 else y0 - 1) % ncy
            xl, xr = max(i2 - 1, 0), min(i2 + 1, ncx - 1)

            def column(x, q):
                o = ncx * ncy * min(max(q, 0), ncz - 1)
                return 3 * self.get(ec, o + ncx * y0 + x) + self.get(ec, o + ncx * y1 + x)
            odd = (j & 1) if k % 2 == 0 else 1 - (j & 1)
            x1 = xr if odd else xl

            def both(q):
                return 3 * column(i2, q) + column(x1, q)
            v = 3 * both(k // 2) + both(k // 2 - 1 if k % 2 == 0 else k // 2 + 1)
            o = 2 * i2 + odd + nx * (j + ny * k)
            xc = (2 if 2 * i2 + 1 == nx - 1 else 1) if odd else (0 if i2 == 0 else 1)
            e[o] = b[o] * self.inv[xc, _cls(k, nz)] + v / 64

    def restrict(self, e, czb):
        nx, ny, nz = self.n
        cx, cy, cz = self.c
        plane, ncx, ncy, ncz = nx * ny, nx // 2, ny // 2, nz // 2
        gx, gy = (nx + 59) // 60, (ny + 13) // 14
        out = np.full(ncx * ncy * ncz, np.nan)

        def at(i, row, k, there=True):  # e or nothing beyond a wall
            return self.get(e, i + nx * row + plane * k) if there else 0.0
        for blk in range(gx * gy * ((ncz + czb - 1) // czb)):
            bx, by, bz = blk % gx, blk // gx % gy, blk // (gx * gy)
            y0, kc0 = by * 14, bz * czb
            kc1 = min(kc0 + czb, ncz)
            acc, up = np.zeros((8, 32)), np.zeros((8, 32))
            for k in range(max(2 * kc0 - 1, 0), min(2 * kc1, nz - 1) + 1):
                sx = np.full((16, 32), np.nan)
                for row in range(16):
                    j = y0 - 1 + row
                    j = ny - 1 if j < 0 else (j - ny) % ny if j >= ny else j
                    jm, jp = (j - 1) % ny, (j + 1) % ny
                    odd = (j + k) & 1
                    r = np.full(32, np.nan)
                    for lane in range(32):
                        ic = bx * 30 - 1 + lane
                        if not 0 <= ic < ncx:
                            r[lane] = 0.0
                            continue
                        i = 2 * ic + odd
                        # the x neighbour outside the pair comes by a shuffle: lane 0 has none on its left,
                        # lane 31 none on its right
                        lost = lane == (31 if odd else 0)
                        x = at(2 * ic + 1 - odd, j, k) + at(i + 1 if odd else i - 1, j, k,
                                                            i < nx - 1 if odd else i > 0)
                        r[lane] = np.nan if lost else cx * x + cy * (at(i, jm, k) + at(i, jp, k)) + cz * (
                            at(i, j, k - 1, k > 0) + at(i, j, k + 1, k < nz - 1))
                    for lane in range(1, 31):
                        ic = bx * 30 - 1 + lane
                        wall = ic == ncx - 1 if odd else ic == 0
                        sx[row, lane] = (4 if wall else 3) * r[lane] + (r[lane - 1] if odd else r[lane + 1])
                for w in range(7):
                    for lane in range(1, 31):
                        ic, jc = bx * 30 - 1 + lane, y0 // 2 + w
                        if ic >= ncx or jc >= ncy:
                            continue
                        v = 3 * (sx[2 * w + 1, lane] + sx[2 * w + 2, lane]) + sx[2 * w, lane] + sx[2 * w + 3, lane]
                        wz = 4 if k in (0, nz - 1) else 3
                        if k & 1:
                            acc[w, lane] += wz * v
                            up[w, lane] = v
                        else:
                            if k > 2 * kc0:
                                out[ic + ncx * (jc + ncy * (k // 2 - 1))] = (acc[w, lane] + v) / 512
                            acc[w, lane] = wz * v + up[w, lane]
                        if kc1 == ncz and k == nz - 1:
                            out[ic + ncx * (jc + ncy * (ncz - 1))] = acc[w, lane] / 512
        return out


class _Tiles:
    """k_mg_down / k_mg_up: a block's shared arrays as numpy arrays of the
    kernels' extents, filled and read by the kernels' local indices."""

    def __init__(self, nx, ny, nz, c, tile):
        self.n, self.c, self.inv, self.tile = (nx, ny, nz), c, _inv(nx, nz, c), tile

    def blocks(self):
        nx, ny, nz = self.n
        CX, CY, CZ = self.tile
        gx, gy, gz = ((n // 2 + t - 1) // t for n, t in zip(self.n, self.tile))
        for blk in range(gx * gy * gz):
            yield blk % gx * 2 * CX, blk // gx % gy * 2 * CY, blk // (gx * gy) * 2 * CZ

    def inside(self, i, k):
        return 0 <= i < self.n[0] and 0 <= k < self.n[2]

    def d(self, i, k):
        return self.inv[_cls(i, self.n[0]), _cls(k, self.n[2])]

    def load(self, a, i, j, k):
        nx, ny, nz = self.n
        assert -ny <= j < 2 * ny  # one wrap
        return _Kernels.get(a, i + nx * (j % ny + ny * k))

    def relax(self, e, l, rhs, i, k):
        z, y, x = l
        s = self.c[0] * (e[z, y, x - 1] + e[z, y, x + 1]) + self.c[1] * (e[z, y - 1, x] + e[z, y + 1, x])
        return (rhs + s + self.c[2] * (e[z - 1, y, x] + e[z + 1, y, x])) * self.d(i, k)

    @staticmethod
    def taps(w0, w1, p):
        return w0 * p[1] + w1 * p[2] + 0.25 * (p[0] + p[3])

    def down(self, b):
        nx, ny, nz = self.n
        CX, CY, CZ = self.tile
        ncx, ncy, ncz = nx // 2, ny // 2, nz // 2
        out = np.full(ncx * ncy * ncz, np.nan)
        for x0, y0, z0 in self.blocks():
            e = np.zeros((2 * CZ + 6, 2 * CY + 6, 2 * CX + 6))
            for z, y, x in np.ndindex(e.shape):
                i, j, k = x0 - 3 + x, y0 - 3 + y, z0 - 3 + z
                if self.inside(i, k):
                    v = self.load(b, i, j, k)
                    e[z, y, x] = v * self.d(i, k) if (i + j % ny + k) % 2 == 0 else v
            HX = (2 * CX + 4) // 2
            for q in range(HX * (2 * CY + 4) * (2 * CZ + 4)):
                z, y = 1 + q // (HX * (2 * CY + 4)), 1 + q // HX % (2 * CY + 4)
                x = 2 + 2 * (q % HX) - ((y + z) & 1)
                assert 1 <= x < e.shape[2] - 1
                i, k = x0 - 3 + x, z0 - 3 + z
                if self.inside(i, k):
                    e[z, y, x] = self.relax(e, (z, y, x), e[z, y, x], i, k)
            r = np.zeros((2 * CZ + 2, 2 * CY + 2, 2 * CX + 2))
            for z, y, x in np.ndindex(r.shape):
                i, j, k = x0 - 1 + x, y0 - 1 + y, z0 - 1 + z
                if self.inside(i, k):
                    o = (z + 2, y + 2, x + 2)
                    v = e[o]
                    xm, xp = (e[o[0], o[1], o[2] + s] if 0 <= i + s < nx else v for s in (-1, 1))
                    zm, zp = (e[o[0] + s, o[1], o[2]] if 0 <= k + s < nz else v for s in (-1, 1))
                    a = 2 * sum(self.c) * v - self.c[0] * (xm + xp) - self.c[2] * (zm + zp)
                    r[z, y, x] = self.load(b, i, j, k) - (a - self.c[1] * (e[o[0], o[1] - 1, o[2]]
                                                                         + e[o[0], o[1] + 1, o[2]]))
            sx = np.stack([self.taps(1 if x0 // 2 + x == 0 else 0.75, 1 if x0 // 2 + x == ncx - 1 else 0.75,
                                     [r[:, :, 2 * x + m] for m in range(4)]) for x in range(CX)], 2)
            sy = np.stack([self.taps(0.75, 0.75, [sx[:, 2 * y + m] for m in range(4)]) for y in range(CY)], 1)
            for z, y, x in np.ndindex(CZ, CY, CX):
                ic, jc, kc = x0 // 2 + x, y0 // 2 + y, z0 // 2 + z
                if ic < ncx and jc < ncy and kc < ncz:
                    out[ic + ncx * (jc + ncy * kc)] = 0.125 * self.taps(
                        1 if kc == 0 else 0.75, 1 if kc == ncz - 1 else 0.75, [sy[2 * z + m, y, x] for m in range(4)])
        return out

    def up(self, b, ec):
        nx, ny, nz = self.n
        CX, CY, CZ = self.tile
        ncx, ncy, ncz = nx // 2, ny // 2, nz // 2
        out = np.full(b.size, np.nan)

        def pair(l):  # local fine index -> its cell and the next one on its side
            c0 = (l >> 1) + 1
            return c0, c0 + 1 if l & 1 else c0 - 1

        def lerp(a, v, wall):
            return a if wall else 0.75 * a + 0.25 * v
        for x0, y0, z0 in self.blocks():
            K = np.zeros((CZ + 4, CY + 4, CX + 4))
            for z, y, x in np.ndindex(K.shape):
                ic, kc = min(max(x0 // 2 - 2 + x, 0), ncx - 1), min(max(z0 // 2 - 2 + z, 0), ncz - 1)
                assert -ncy <= y0 // 2 - 2 + y < 2 * ncy
                K[z, y, x] = _Kernels.get(ec, ic + ncx * ((y0 // 2 - 2 + y) % ncy + ncy * kc))
            Z = np.stack([lerp(K[pair(l)[0]], K[pair(l)[1]], not 0 <= z0 // 2 - 2 + pair(l)[1] < ncz)
                          for l in range(2 * CZ + 4)])
            S = np.stack([lerp(Z[:, pair(l)[0]], Z[:, pair(l)[1]], False) for l in range(2 * CY + 4)], 1)
            e = np.zeros((2 * CZ + 4, 2 * CY + 4, 2 * CX + 4))
            for z, y, x in np.ndindex(e.shape):
                i, j, k = x0 - 2 + x, y0 - 2 + y, z0 - 2 + z
                if (x + y + z) % 2 == 0 and self.inside(i, k):
                    assert (i + j % ny + k) % 2 == 0
                    c0, c1 = pair(x)
                    e[z, y, x] = self.load(b, i, j, k) * self.d(i, k) + lerp(S[z, y, c0], S[z, y, c1],
                                                                             not 0 <= x0 // 2 - 2 + c1 < ncx)
            HX = (2 * CX + 2) // 2
            for q in range(HX * (2 * CY + 2) * (2 * CZ + 2)):
                z, y = 1 + q // (HX * (2 * CY + 2)), 1 + q // HX % (2 * CY + 2)
                x = 1 + 2 * (q % HX) + ((y + z) & 1)
                i, j, k = x0 - 2 + x, y0 - 2 + y, z0 - 2 + z
                if self.inside(i, k):
                    e[z, y, x] = self.relax(e, (z, y, x), self.load(b, i, j, k), i, k)
            for q in range(CX * 2 * CY * 2 * CZ):
                z, y = 2 + q // (CX * 2 * CY), 2 + q // CX % (2 * CY)
                x = 2 + 2 * (q % CX) + ((y + z) & 1)
                i, j, k = x0 - 2 + x, y0 - 2 + y, z0 - 2 + z
                if i < nx and j < ny and k < nz:
                    e[z, y, x] = self.relax(e, (z, y, x), self.load(b, i, j, k), i, k)
            for z, y, x in np.ndindex(2 * CZ, 2 * CY, 2 * CX):
                if x0 + x < nx and y0 + y < ny and z0 + z < nz:
                    out[x0 + x + nx * (y0 + y + ny * (z0 + z))] = e[z + 2, y + 2, x + 2]
        return out


@pytest.mark.parametrize("tile", [(8, 2, 2)])
@pytest.mark.parametrize("size", [(4, 4, 4), (8, 6, 4), (34, 10, 10), (18, 4, 14), (6, 8, 6)])
def test_tile_kernels_equal_the_general_passes(size, tile):
    nx, ny, nz = size
    rng = np.random.default_rng(nx + ny)
    c = (1.3, 0.9, 1.1)
    b, ec = rng.normal(size=(nz, ny, nx)), rng.normal(size=(nz // 2, ny // 2, nx // 2))
    bc, ref = _general(b, ec, c)
    K = _Tiles(nx, ny, nz, c, tile)
    assert np.max(np.abs(K.down(b.ravel()) - bc.ravel())) < 1e-13
    assert np.max(np.abs(K.up(b.ravel(), ec.ravel()) - ref.ravel())) < 1e-13


@pytest.mark.parametrize("size", EDGES)
def test_halved_level_kernels_equal_the_general_passes(size):
    nx, ny, nz = size
    rng = np.random.default_rng(nx + 7 * nz)
    c = (1.3, 0.9, 1.1)
    b = rng.normal(size=(nz, ny, nx))
    ec = rng.normal(size=(nz // 2, ny // 2, nx // 2))
    bc, ref = _general(b, ec, c)
    K, flat = _Kernels(nx, ny, nz, c), b.ravel()
    for kz, czb in ((2, 1), (8, 4)):
        e = K.black(flat, kz)
        got = K.restrict(e, czb)  # reads black points only: the red ones are not set yet
        # a few dozen roundings of values of order 1
        assert np.max(np.abs(got - bc.ravel())) < 1e-13
        K.prolong(flat, ec.ravel(), e, kz)
        K.half(flat, e, 1, kz)
        K.half(flat, e, 0, kz)
        assert np.max(np.abs(e - ref.ravel())) < 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("size", [(64, 16, 16), (66, 34, 20), (130, 18, 36), (16, 64, 72), (130, 50, 60)])
def test_solves_on_halved_levels_match_the_exact_solve(size, precision):
    """Solved to rtol 1e-13 (the preconditioner's precision does not enter
    the solution), as test_pressure_solve_tight: 1e-10 of the maximum."""
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz, precision=precision, fp64_parts=2 * precision)
    rng = np.random.default_rng(nx)
    u3 = np.asfortranarray(st["U2"] + rng.normal(scale=1e-3, size=st["U2"].shape))
    u3[:, 0], u3[:, -1] = u3[:, -2], u3[:, 1]  # periodic rows, as the driver's exchange leaves them
    with TplsGpu(nx, ny, nz, p, uin) as g:
        o = Oracle(nx, ny, nz, p, uin)
        rhs = g.get_source_pres(u3, st["V2"], st["W2"], p.dx, p.dy, p.dz, p.dt)
        pold = np.zeros_like(st["PRES"], order="F")
        po, *_ = o.pressure_solve(pold, rhs, u3, uin, p.dx, p.dy, p.dz, p.dt)
        pg, its, _, reason = g.pressure_solve(pold, rhs, u3, uin, p.dx, p.dy, p.dz, p.dt, rtol=1e-13, maxits=200)
    assert reason == 2 and its < 60
    assert np.max(np.abs(pg - po)) <= 1e-10 * np.max(np.abs(po))
