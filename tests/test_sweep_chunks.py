"""The FP64 odd half-sweep by whole columns in super-chunks of equal length
(csrc/k_sweep.cu): every level belongs to one warp's run of one chunk, and the
result is the oracle's, for columns around one and two chunks of 64 levels (w's
columns a level shorter) and shorter than the eight warps."""
import pytest

from tests._util import relmax


@pytest.mark.parametrize("nz", list(range(4, 130)))
def test_runs_cover_the_column(nz):
    m = (nz - 1) // 64 + 1
    sc = (nz + m - 1) // m
    assert sc <= 64
    for k0 in (0, 1):
        seen = []
        for kc in range(k0, nz, sc):
            n = min(sc, nz - kc)
            per = (n + 7) // 8
            assert per <= 8
            for w in range(8):
                seen += range(kc + w * per, kc + min(n, w * per + per))
        assert seen == list(range(k0, nz))


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(8, 4, 5), (10, 6, 17), (66, 5, 65), (9, 4, 66), (12, 3, 127)])
def test_whole_columns_match_the_oracle(size):
    """One step to 1e-11, as the per-step parity tests."""
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz, p_rtol=1e-13, p_maxits=400)
    rows = (slice(None), slice(1, ny + 1), slice(None))
    o = Oracle(nx, ny, nz, p, uin)
    o.set_state(st)
    o.step(1)
    with TplsGpu(nx, ny, nz, p, uin) as g:
        g.set_state(st)
        g.step(1)
        for k in ("U2", "V2", "W2"):
            assert relmax(g.get_field(k), o.get_field(k), rows) < 1e-11, k
