"""The per-routine momentum entries whose threads march up a column
(csrc/k_momentum.cu, csrc/k_sweep.cu): get_conv_all, get_diffusion_all,
do_jacobi_* and do_sor_* on random fields and a random positive viscosity
against the oracle, on grids whose columns end inside a run of 2, 4 and 8
levels and inside a segment of the odd half-sweep, and whose rows end just
past a block of 32 points.

Tolerance: at most 60 roundings of 2^-53 per value, on terms up to 100 times
the largest result: 7e-13 of the maximum, taken as 1e-12."""
import numpy as np
import pytest

from tests._util import relmax

TOL = 1e-12


@pytest.fixture(scope="module", params=[(33, 7, 21), (35, 66, 93), (33, 130, 150)], ids=lambda s: "x".join(map(str, s)))
def pair(request):
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = request.param
    p, uin, _ = make_case("A", nx=nx, ny=ny, nz=nz)
    o = Oracle(nx, ny, nz, p, uin)
    rng = np.random.default_rng(nx * ny * nz)

    def field(kind):
        a = np.asfortranarray(rng.normal(size=o.shape(kind)))
        o.exchange2d(a)
        return a
    va = np.asfortranarray(rng.uniform(0.5, 2.0, size=o.shape("va")) * 1e-2)
    f = {"va": va, "uvw": (field("uv"), field("uv"), field("w"))}
    for q, kind in enumerate(("uv", "uv", "w")):
        f[q] = (field(kind), field(kind), field(kind))
    with TplsGpu(nx, ny, nz, p, uin) as g:
        yield p, o, g, f


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["get_conv_all", "get_diffusion_all"])
def test_stencils(pair, which):
    p, o, g, f = pair
    ro = getattr(o, which)(f["va"], *f["uvw"], p.dx, p.dy, p.dz)
    rg = getattr(g, which)(f["va"], *f["uvw"], p.dx, p.dy, p.dz)
    for a, b in zip(rg, ro):
        assert relmax(a, b) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("comp", [0, 1, 2])
def test_sweeps(pair, comp):
    p, o, g, f = pair
    x, xo, rhs = f[comp]
    xa, xb = np.array(x, order="F"), np.array(x, order="F")
    getattr(o, "do_jacobi_" + "uvw"[comp])(xa, xo, rhs, f["va"], p.dx, p.dy, p.dz, p.dt)
    getattr(g, "do_jacobi_" + "uvw"[comp])(xb, xo, rhs, f["va"], p.dx, p.dy, p.dz, p.dt)
    assert relmax(xb, xa) < TOL
    for flg in (0, 1):
        for it in (1, 2):
            xa, xb = np.array(x, order="F"), np.array(x, order="F")
            getattr(o, "do_sor_" + "uvw"[comp])(xa, rhs, f["va"], p.dx, p.dy, p.dz, p.dt, flg, it)
            getattr(g, "do_sor_" + "uvw"[comp])(xb, rhs, f["va"], p.dx, p.dy, p.dz, p.dt, flg, it)
            assert relmax(xb, xa) < TOL, (flg, it)
