"""The FP64 advection's column chunks (adv_levels and k_advect, csrc/k_advect.cu):
grids whose columns are cut into chunks of several levels with a shorter last one,
down to a single level, against the oracle (1e-11 of the maximum, as the
per-routine parity tests)."""
import numpy as np
import pytest

from tests._util import interior_rows, relmax

GRIDS = [((250, 99, 31), 8), ((97, 130, 61), 6), ((160, 80, 128), 11)]


def _levels(nx, ny, nz):
    """adv_levels: the chunk with the least (blocks of the busiest of 152 SMs) x
    (faces per column), a lone block per SM counting 1.2 times."""
    gxy = -(-nx // 32) * -(-ny // 8)

    def cost(q):
        w = -(-gxy * -(-nz // q) // 152)
        return w * (3 * q + 1) * (1.2 if w == 1 else 1.0)
    return min(range(1, 17), key=cost)


@pytest.mark.parametrize("size,kc", GRIDS)
def test_grids_have_long_chunks_and_a_remainder(size, kc):
    assert _levels(*size) == kc and kc > 1 and size[2] % kc != 0


@pytest.mark.gpu
@pytest.mark.parametrize("size,kc", GRIDS)
def test_advection_in_chunks(size, kc):
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz)
    phi = np.array(st["PHI2"], order="F")
    phi += np.random.default_rng(nx).normal(scale=1e-2, size=phi.shape)
    phi[:, 0], phi[:, -1] = phi[:, -2], phi[:, 1]
    u, v, w = (np.array(st[k], order="F") for k in ("U2", "V2", "W2"))
    with TplsGpu(nx, ny, nz, p, uin) as g:
        a = g.do_advect_phi(phi, u.copy("F"), v.copy("F"), w.copy("F"), p.dx, p.dy, p.dz)
    b = Oracle(nx, ny, nz, p, uin).do_advect_phi(phi, u.copy("F"), v.copy("F"), w.copy("F"), p.dx, p.dy, p.dz)
    rows = interior_rows(ny)
    assert np.all(np.isfinite(a[rows]))
    assert relmax(a, b, rows) < 1e-11
