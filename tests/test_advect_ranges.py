"""The FP64 advection's weights (csrc/k_advect.cu) over the magnitudes of phi:
one where eps dominates every smoothness indicator, ordinary ones, one whose
weights leave the range of the fast quotient (its out-of-line division), and
fields of constants and jumps, on grids whose columns are cut into chunks of 2
to 16 levels with remainders.  Against the oracle, 1e-11 of the maximum as the
per-routine parity tests."""
import numpy as np
import pytest

from tests._util import interior_rows, relmax


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(34, 9, 7), (64, 32, 21), (130, 48, 35)])
@pytest.mark.parametrize("scale", [1e-9, 1.0, 1e6, 1e20])
def test_advection_over_magnitudes(size, scale):
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz)
    rng = np.random.default_rng(nx)
    phi = np.array(st["PHI2"], order="F")
    phi[nx // 2:, :, nz // 2:] = 0.25  # constant beyond a jump
    phi += rng.normal(scale=1e-2, size=phi.shape) * (phi != 0.25)
    phi[:, 0], phi[:, -1] = phi[:, -2], phi[:, 1]
    phi *= scale
    u, v, w = (np.array(st[k], order="F") for k in ("U2", "V2", "W2"))
    with TplsGpu(nx, ny, nz, p, uin) as g:
        a = g.do_advect_phi(phi, u.copy("F"), v.copy("F"), w.copy("F"), p.dx, p.dy, p.dz)
    b = Oracle(nx, ny, nz, p, uin).do_advect_phi(phi, u.copy("F"), v.copy("F"), w.copy("F"), p.dx, p.dy, p.dz)
    rows = interior_rows(ny)
    assert np.all(np.isfinite(a[rows]))
    assert relmax(a, b, rows) < 1e-11
