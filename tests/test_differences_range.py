"""Differences of the last two iterates (k_diff_set, csrc/k_momentum.cu) over the
magnitudes of the velocity: a uniform stream scaled from 1 to 1e24, without
surface tension, so that the step is linear in the scale.  The FP32-mixed form
sums FP32 squares: as the FP64 form's sum while a square is an FP32 value, infinity
(not NaN) beyond."""
import numpy as np
import pytest


def _err_u(size, scale, precision, fill=None):
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, _, st = make_case("A", nx=nx, ny=ny, nz=nz, precision=precision, mom=4)
    p.scap = 0.0
    with TplsGpu(nx, ny, nz, p, np.full(nz, scale)) as g:
        g.set_state({"PHI2": st["PHI2"]})
        u = np.full(g.shape("uv"), scale, order="F")
        if fill is not None:
            u[5, 4, 3] = fill
        g.set_field("U2", u)
        g.graphs_enable(False)
        g.step(1)
        return g.stats()["err_u"]


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(48, 16, 24), (37, 9, 150)])
def test_sum_of_squares_over_scales(size):
    """Tolerance: the iterates are the FP32-mixed form's own, 1e-5 of the FP64
    form's in the parity tests of the sweeps."""
    for scale in (1.0, 1e12, 1e15, 1e18):  # squares of 1e-2 to 1e34 and their sums beyond 2^96
        want = _err_u(size, scale, 0)
        assert abs(_err_u(size, scale, 1) - want) < 1e-5 * want
    assert _err_u(size, 1e24, 1) == np.inf  # squares of 1e46


@pytest.mark.gpu
def test_nan_stays_nan():
    assert np.isnan(_err_u((48, 16, 24), 1.0, 1, fill=np.nan))
