"""The momentum sweeps of u, v and w in common launches (SweepSet,
csrc/k_sweep.cu, csrc/k_sweep32.cu).

CPU: the blocks of a set's odd half-sweep decode to every segment of every
component's columns exactly once, and a segment waits only on an earlier
ticket that publishes.  GPU: components with sweep counts of their own (one
leaves the launches before the others, one makes a single sweep), odd spanwise
extents and a wall-normal extent whose w columns have one segment less, against
the oracle."""
import numpy as np
import pytest

from tests._util import relmax

SC = 64


@pytest.mark.parametrize("ids", [(0, 1, 2), (0, 2), (1,)])
@pytest.mark.parametrize("size", [(64, 8, 193), (66, 5, 129), (8, 3, 192), (130, 4, 256)])
def test_segments_of_a_set_cover_every_column(size, ids):
    nx, ny, nz = size
    gx, nseg = ((nx + 1) // 2 + 31) // 32, (nz - 1) // SC + 1
    cap = 3 * nseg * gx * ny
    nct = len(ids) * gx * ny
    seen, published = set(), set()
    for t in range(nseg * nct):  # in ticket order
        assert t < cap
        seg, ct = divmod(t, nct)
        q, tile = divmod(ct, gx * ny)
        bx, j = tile % gx, tile // gx + 1
        comp = ids[q]
        k0, k1 = (1 if comp == 2 else 0), nz - 1
        n = min(SC, k1 - (k0 + seg * SC) + 1)
        if n <= 0:  # nothing there, and no segment above it
            assert comp == 2 and seg == nseg - 1
            continue
        if seg > 0:
            assert t - nct in published
        if seg < (k1 - k0) // SC:
            published.add(t)
        for k in range(k0 + seg * SC, k0 + seg * SC + n):
            assert (comp, bx, j, k) not in seen
            seen.add((comp, bx, j, k))
    assert len(seen) == sum(gx * ny * (nz - (c == 2)) for c in ids)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("size", [(64, 32, 48), (37, 19, 23), (16, 8, 193)])
def test_components_with_their_own_sweep_counts(size, precision):
    """One step; FP64 to 1e-11 as the per-step parity tests, FP32-mixed to
    1e-5 of the maximum (its stated accuracy)."""
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz, p_rtol=1e-13, p_maxits=400, precision=precision,
                           fp64_parts=2 * precision)
    p.mom_u, p.mom_v, p.mom_w = 30, 17, 2
    rows = (slice(None), slice(1, ny + 1), slice(None))
    o = Oracle(nx, ny, nz, p, uin)
    o.set_state(st)
    o.step(1)
    with TplsGpu(nx, ny, nz, p, uin) as g:
        g.set_state(st)
        g.step(1)
        for k in ("U2", "V2", "W2"):
            assert relmax(g.get_field(k), o.get_field(k), rows) < (1e-5 if precision else 1e-11), k
        if not precision:
            so, sg = o.stats(), g.stats()
            for k in ("err_u", "err_v", "err_w"):
                assert abs(sg[k] - so[k]) <= 1e-9 * max(so["err_w"], so[k]), k
