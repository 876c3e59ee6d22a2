"""The FP32 odd half-sweep in two segments per column (csrc/k_sweep.cu) and
the ends of its and the four-point kernels' rows (csrc/k_sweep32.cu), whose
lanes past the last point repeat a point of the row: wall-normal extents
around one and two segments of 64 levels (w's columns a level shorter), rows
that end on every position of a group of four points and just past a tile of
32 pairs or 32 groups, against the oracle."""
import pytest

from tests._util import relmax


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(8, 4, 65), (65, 6, 66), (130, 4, 97), (67, 4, 128), (126, 4, 129)])
def test_fp32_sweeps_by_segments(size):
    """One step of the FP32-mixed form to 1e-5 of the maximum (its stated
    accuracy)."""
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz, p_rtol=1e-13, p_maxits=400, precision=1, fp64_parts=2)
    p.mom_u, p.mom_v, p.mom_w = 30, 17, 2
    rows = (slice(None), slice(1, ny + 1), slice(None))
    o = Oracle(nx, ny, nz, p, uin)
    o.set_state(st)
    o.step(1)
    with TplsGpu(nx, ny, nz, p, uin) as g:
        g.set_state(st)
        g.step(1)
        for k in ("U2", "V2", "W2"):
            assert relmax(g.get_field(k), o.get_field(k), rows) < 1e-5, k
