"""The coarsest multigrid level's lines as matrices of their modes
(csrc/tpls_modes.cuh: k_dense_build, k_mode_dense).

CPU: the folded matrices (even and odd part about the line's middle, one
matrix for the sine and cosine modes of a wavenumber), indexed as the kernels
do, give what the sweeps along the line give.  GPU: solves on grids of one
level with lines of up to 64 points, and just above or with more matrices than
the limit, against the oracle's exact solve."""
import numpy as np
import pytest

from tests.test_pressure_modes import W, SWEEPS, _cos, _fourier


def _line(al, be, g):
    e = g.copy()
    for _ in range(SWEEPS - 1):
        s = np.zeros_like(e)
        s[1:] += e[:-1]
        s[:-1] += e[1:]
        e = al * e + be * s + g
    return e


@pytest.mark.parametrize("nx", [1, 2, 5, 8, 33, 63, 64])
def test_folded_matrices_equal_the_sweeps(nx):
    ny, nz, c = 6, 3, (1.3, 0.9, 0.4)
    half = (nx + 1) // 2
    (_, lz), (_, ly) = _cos(nz), _fourier(ny)
    D = np.full(2 * half * half * (ny // 2 + 1) * nz, np.nan)
    nbx = np.array([(0 if nx == 1 else 1 if i in (0, nx - 1) else 2) for i in range(nx)])

    def factors(my, mz):
        wd = W / (c[0] * nbx + 2 * c[1] + c[2] * lz[mz])
        return (1 - W) + wd * c[1] * (2 - ly[my]), wd * c[0], wd
    for cl in range(ny // 2 + 1):
        for mz in range(nz):
            al, be, ga = factors(0 if cl == 0 else 2 * cl - 1, mz)
            for jp in range(2 * half):
                j, odd, jm = jp >> 1, jp & 1, nx - 1 - (jp >> 1)
                g = np.zeros(half)
                g[j] = (0.0 if odd else 1.0) if j == jm else 0.5
                g *= ga[:half]
                e = g.copy()
                for _ in range(SWEEPS - 1):  # on half the line
                    left, right = np.r_[0.0, e[:-1]], np.r_[e[1:], 0.0]
                    if nx > 1:
                        right[-1] = (e[-1] if nx % 2 == 0 else left[-1]) * (-1.0 if odd else 1.0)
                    e = al[:half] * e + be[:half] * (left + right) + g
                    if odd and nx % 2:
                        e[-1] = 0.0
                for i in range(half):
                    D[2 * (half * (j + half * (mz + nz * cl)) + i) + odd] = e[i]
    assert not np.isnan(D).any()
    rng = np.random.default_rng(nx)
    for my in range(ny):
        for mz in range(nz):
            x = rng.normal(size=nx)
            al, be, ga = factors(my, mz)
            d = D.reshape(-1, 2)[half * half * (mz + nz * ((my + 1) // 2)):][:half * half].reshape(half, half, 2)
            i = np.arange(half)
            im = nx - 1 - i
            ev, od = np.where(i == im, x[i], x[i] + x[im]), x[i] - x[im]
            e, o = ev @ d[:, :, 0], od @ d[:, :, 1]
            got = np.empty(nx)
            got[im] = e - o
            got[i] = e + o
            # forty sweeps and 64 products of values of order 1
            assert np.max(np.abs(got - _line(al, be, ga * x))) < 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(5, 9, 23), (33, 7, 11), (63, 5, 9), (65, 5, 9), (25, 25, 75), (63, 35, 75),
                                  (31, 69, 121)])
def test_solves_match_the_oracle(size):
    """Converged to 1e-13 on both sides; the tolerance is the per-routine
    parity tests' 1e-11 of the maximum."""
    from oracle.oracle import Oracle
    from tests._util import relmax
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz, p_rtol=1e-13, p_maxits=400)
    o = Oracle(nx, ny, nz, p, uin)
    o.set_state(st)
    o.step(1)
    rhs, u3, pold = o.get_field("RHS_P"), o.get_field("U3"), o.get_field("PRES_OLD")
    po, *_ = o.pressure_solve(pold, rhs, u3, uin, p.dx, p.dy, p.dz, p.dt)
    with TplsGpu(nx, ny, nz, p, uin) as g:
        pg, its, rn, reason = g.pressure_solve(pold, rhs, u3, uin, p.dx, p.dy, p.dz, p.dt, rtol=1e-13, maxits=400)
    assert reason == 2
    inner = (slice(1, nx + 1), slice(1, ny + 1), slice(1, nz + 1))
    assert relmax(pg - pg[inner].mean(), po - po[inner].mean(), inner) < 1e-11
