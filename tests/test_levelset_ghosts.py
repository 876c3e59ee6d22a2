"""Ghost elements written by the threads that own the interior (csrc/
k_levelset.cu): the periodic rows, the inlet and outlet columns (copied,
extrapolated from the next lane or, where the last column starts a warp,
recomputed) and the extrapolated planes, on rows that end before, at and just
past a block of 32 columns and 8 rows, against the oracle.

The tolerance is the per-routine parity tests' 1e-11 of the maximum."""
import numpy as np
import pytest

from tests._util import relmax

TOL = 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(31, 7, 12), (32, 8, 9), (33, 9, 12), (65, 3, 10), (64, 16, 9)])
def test_levelset_routines(size):
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz)
    rng = np.random.default_rng(nx + ny + nz)
    o = Oracle(nx, ny, nz, p, uin)
    phi = np.asfortranarray(st["PHI2"] + 0.2 * p.dx * rng.uniform(-1, 1, size=o.shape("p")))
    o.exchange2d(phi)
    conv = [np.asfortranarray(rng.normal(scale=1e-2, size=o.shape("p"))) for _ in range(3)]
    with TplsGpu(nx, ny, nz, p, uin) as g:
        rows = (slice(None), slice(1, ny + 1), slice(None))  # the oracle's own ghost rows are undefined here

        def periodic(x):
            return np.array_equal(x[:, 0], x[:, ny]) and np.array_equal(x[:, ny + 1], x[:, 1])
        a = o.do_tpls(phi, *conv, p.levelset, p.height, p.dx, p.dz, p.dt)
        b = g.do_tpls(phi, *conv, p.levelset, p.height, p.dx, p.dz, p.dt)
        assert relmax(b[0], a[0], rows) < TOL and periodic(b[0])
        assert abs(b[1] - a[1]) <= 1e-9 * abs(a[1])
        fo = o.get_csf(phi, p.dx, p.dy, p.dz, p.scap, p.smooth_width)
        fg = g.get_csf(phi, p.dx, p.dy, p.dz, p.scap, p.smooth_width)
        assert any(np.any(f[0, 1:-1] != 0) and np.any(f[-1, 1:-1] != 0) for f in fo)  # the band reaches both end columns
        for x, y in zip(fg, fo):
            assert relmax(x, y, rows) < TOL and periodic(x)


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(33, 9, 12), (64, 8, 9)])
def test_float_pair_redistancing_ghosts(size):
    """The float-pair iteration writes the same copies: periodic rows and the
    outlet column equal their sources to the bit."""
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz, precision=1, fp64_parts=0)
    with TplsGpu(nx, ny, nz, p, uin) as g:
        g.set_state(st)
        g.step(1)
        phi = g.get_field("PHI2")
        assert np.array_equal(phi[:, 0], phi[:, ny]) and np.array_equal(phi[:, ny + 1], phi[:, 1])
        assert np.array_equal(phi[nx + 1], phi[nx])
        k = np.arange(1, nz + 1)
        h = float(np.float32(p.dx))  # this form carries the spacing in FP32
        assert np.abs(phi[0, 1, 1:nz + 1] - ((k - 0.5) * h - p.height)).max() < 1e-12
