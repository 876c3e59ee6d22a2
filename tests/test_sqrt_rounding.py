"""sqrt_rn (csrc/tpls_pair.cuh), the redistancing's square root with one FP64
operation.

CPU: its arithmetic in numpy, with every error of the FP32 reciprocal root that
rsqrtf's two ulps allow, returns the correctly rounded root wherever it does
not defer to the library, and defers rarely.  GPU: a redistancing iteration
agrees with the oracle (whose sqrt is the C library's) to the last bit but for
FMA contraction, over fields whose gradients span the fast range and leave it
on both sides."""
import numpy as np
import pytest

from tests._util import interior_rows, relmax

F = np.float32


def _fma32(a, b, c):
    return F(a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64))


def _residual(a, s):  # a - s*s with one rounding
    c = 134217729.0 * s
    h = c - (c - s)
    l = s - h
    p = s * s
    return (a - p) - (((h * h - p) + 2 * h * l) + l * l)


def _sqrt_rn(a, ulps):
    b = a.view(np.uint64)
    e = ((b >> np.uint64(52)) & np.uint64(0x7FF)).astype(np.int64)
    rem = (b & np.uint64(0x1FFFFFFF)).astype(np.uint32)
    h = (((e - 896).astype(np.uint32) << np.uint32(23))
         | ((b >> np.uint64(29)) & np.uint64(0x7FFFFF)).astype(np.uint32)).view(F)
    l = F(rem.astype(F) * np.ldexp(1.0, (e - 1075).astype(int)).astype(F))
    r = (F(1 / np.sqrt(h.astype(np.float64))).view(np.int32) + ulps).view(F)
    hr, sh = F(F(0.5) * r), F(h * r)
    sl = F(F(_fma32(-sh, sh, h) + l) * hr)
    sb = sh.astype(np.float64).view(np.int64)
    scale = np.ldexp(1.0, (52 - (((sb >> 52) & 0x7FF) - 1023)).astype(int)).astype(F)
    s0 = sb + np.rint(F(sl * scale)).astype(np.int64)
    cu = F(F(F(_residual(a, s0.view(np.float64))) * hr) * scale)
    n = np.rint(cu)
    r0 = s0 + n.astype(np.int64)
    sure = np.abs(F(cu - n)) <= F(0.5) - F(np.abs(cu) * F(2.0 ** -20) + F(2.0 ** -16))
    sure &= (np.abs(cu) < 65536) & ((r0 >> 52) == (sb >> 52)) & ((s0 >> 52) == (sb >> 52))
    return sure, r0.view(np.float64)


@pytest.mark.parametrize("kind", ["one binade pair", "many magnitudes", "next to squares", "powers of four"])
def test_fast_square_root_is_correctly_rounded(kind):
    rng = np.random.default_rng(len(kind))
    n = 1_000_000
    if kind == "one binade pair":
        a = rng.uniform(1.0, 4.0, n)
    elif kind == "many magnitudes":
        a = 10.0 ** rng.uniform(-17.0, 17.0, n)
    elif kind == "next to squares":
        a = rng.uniform(1.0, 2.0, n) ** 2
    else:
        a = (1.0 + rng.integers(-1000, 1000, n) * 2.0 ** -52) * 4.0 ** rng.integers(-25, 25, n)
    sure, s = _sqrt_rn(a, rng.integers(-2, 3, n).astype(np.int32))
    assert np.array_equal(s[sure], np.sqrt(a[sure]))
    if kind in ("one binade pair", "many magnitudes"):
        assert np.mean(~sure) < 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-12, 1e-3, 1.0, 1e12])
def test_redistancing_over_gradient_magnitudes(scale):
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = 40, 18, 30
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz)
    rng = np.random.default_rng(5)
    phi = np.array(st["PHI2"], order="F") * scale
    phi[:, :, nz // 2:] += rng.normal(scale=1e-3 * scale, size=phi[:, :, nz // 2:].shape)
    phi[2:9, 3:9, 3:9] = 0.7 * scale  # zero gradients
    phi[:, 0], phi[:, -1] = phi[:, -2], phi[:, 1]
    zero = np.zeros_like(phi, order="F")
    args = (phi, zero, zero, zero, 3, p.height, p.dx, p.dz, p.dt)
    with TplsGpu(nx, ny, nz, p, uin) as g:
        a, ea = g.do_tpls(*args)
    b, eb = Oracle(nx, ny, nz, p, uin).do_tpls(*args)
    assert relmax(a, b, interior_rows(ny)) < 1e-14  # a few ulps of FMA contraction over three iterations
    assert abs(ea - eb) <= 1e-12 * abs(eb)
