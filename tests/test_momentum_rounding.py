"""Rounding of the FP64 momentum operators (csrc/k_momentum.cu, tpls_sweep.cuh):
bounds on single results, derived from the order of their operations, on inputs
that leave only the terms in question.  u = 2^-53 is half a unit in the last
place of a value in [1, 2); ``_half(x)`` half a unit of x.

* a Jacobi and a checkerboard point divide by the diagonal: from a zero field
  the result is the rounded quotient rhs / diagonal, infinities included;
* the difference of a z face's two products rounds one of them;
* convection rounds its streamwise product and the sum at full size, no other;
* the step's right-hand side adds the state last: one rounding at its size."""
from fractions import Fraction

import numpy as np
import pytest

LD = np.longdouble


def _half(x):
    return LD(0.5) * np.spacing(np.abs(np.asarray(x, dtype=np.float64))).astype(LD)


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _context(nx, ny, nz, **kw):
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz, mom=2)
    for k, v in kw.items():
        setattr(p, k, v)
    return TplsGpu(nx, ny, nz, p, uin), p, st


def _diagonal(comp, mu, p):
    a = [(p.dt / (d * d)) / 2.0 for d in (p.dx, p.dy, p.dz)]
    d = 1.0
    for axis in range(3):  # own axis: two cells; the others: two sums of four, a quarter in the factor
        d = _fma(a[axis], 2.0 * mu, d) if axis == comp else _fma(0.25 * a[axis], 8.0 * mu, d)
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(20, 9, 7), (37, 12, 23)])
@pytest.mark.parametrize("mu", [0.37, 3.1e-3])
def test_points_divide_by_the_diagonal(size, mu):
    """A quotient from a 44-bit reciprocal with its remainder corrected is the
    rounded one but for about one point in 2^34."""
    nx, ny, nz = size
    g, p, _ = _context(*size)
    va = np.full((nx + 4, ny + 4, nz + 2), mu, order="F")
    rng = np.random.default_rng(nx)
    for comp, c in enumerate("uvw"):
        k0, iend = (1 if c == "w" else 0), (nx - 1 if c == "u" else nx)
        inner = (slice(1, iend + 1), slice(1, ny + 1), slice(k0, nz))
        rhs = np.asfortranarray(rng.normal(size=g.shape("w" if c == "w" else "uv")))
        rhs[3, 2, k0 + 2], rhs[4, 3, k0 + 1], rhs[5, 4, k0 + 3] = np.inf, -np.inf, np.nan
        want = rhs[inner] / _diagonal(comp, mu, p)
        x = getattr(g, "do_jacobi_" + c)(np.zeros_like(rhs), np.zeros_like(rhs), rhs, va, p.dx, p.dy, p.dz, p.dt)
        assert np.array_equal(x[inner], want, equal_nan=True)
        i, j, k = np.indices(rhs.shape)[:, inner[0], inner[1], inner[2]]
        for flg in (0, 1):
            x = getattr(g, "do_sor_" + c)(np.zeros_like(rhs), rhs, va, p.dx, p.dy, p.dz, p.dt, flg, 2)
            relaxed = np.where((i + j + k + flg) % 2 == 1, 1.2 * want, 0.0)
            assert np.array_equal(x[inner], relaxed, equal_nan=True)
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nz", [23, 64, 150])
def test_z_difference_rounds_one_product(nz):
    """Viscosity and u of z alone, u in multiples of 2^-10 (exact differences):
    diffusion is lz (P dT - M dB) with P and M the four-cell sums."""
    nx, ny = 12, 7
    g, p, _ = _context(nx, ny, nz)
    for seed in range(4):
        rng = np.random.default_rng(seed)
        mu = rng.uniform(0.5, 1.0, size=nz + 2)
        va = np.asfortranarray(np.broadcast_to(mu, (nx + 4, ny + 4, nz + 2)))
        s = rng.integers(1, 1 << 20, size=nz) / 1024.0
        u = np.asfortranarray(np.broadcast_to(s, (nx + 2, ny + 2, nz)))
        du, _, _ = g.get_diffusion_all(va, u, np.zeros_like(u), g.zeros("w"), p.dx, p.dy, p.dz)
        k = np.arange(1, nz - 1)
        M, P = 2.0 * mu[k] + 2.0 * mu[k + 1], 2.0 * mu[k + 1] + 2.0 * mu[k + 2]
        dT, dB = s[k + 1] - s[k], s[k] - s[k - 1]
        rd = 1.0 / p.dz
        lz = LD(0.25 * (rd * rd))
        nz_ = LD(1) * P * dT.astype(LD) - M.astype(LD) * dB
        bound = lz * (_half(M * dB) + _half(nz_)) + _half(lz * nz_)
        got = du[1:nx, 1:ny + 1, 1:nz - 1]
        assert np.all(got == got[:1, :1])
        assert np.all(np.abs(got[0, 0].astype(LD) - lz * nz_) <= bound * LD(1.000001))
    g.close()


def _uniform_u(g, rng):
    """u in [1, 2), random: differences of its values are exact."""
    u = np.asfortranarray(rng.uniform(1.0, 2.0, size=g.shape("uv")))
    u[:, 0], u[:, -1] = u[:, -2], u[:, 1]
    return u


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(37, 12, 23), (64, 16, 40)])
def test_convection_rounds_the_streamwise_term_last(size):
    nx, ny, nz = size
    g, p, _ = _context(*size)
    u = _uniform_u(g, np.random.default_rng(nz))
    mu = 1e-9  # the stress: below 1e-6 of the convective term
    va = np.full((nx + 4, ny + 4, nz + 2), mu, order="F")
    cu, _, _ = g.get_conv_all(va, u, g.zeros("uv"), g.zeros("w"), p.dx, p.dy, p.dz)
    g.close()
    rd = 1.0 / p.dx
    U = u[:, 1:ny + 1].astype(LD)
    x, e, w = U[1:nx], U[2:nx + 1], U[:nx - 1]
    P = (e - w) * x
    stress = LD(rd * rd) * LD(mu) * ((e - x) - (x - w))
    want = LD(0.5 * rd) * P - stress
    bound = LD(0.5 * rd) * _half(P) + _half(want) + 8 * _half(stress)
    assert np.all(np.abs(cu[1:nx, 1:ny + 1].astype(LD) - want) <= bound * LD(1.000001))


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(37, 12, 23), (64, 16, 40), (20, 10, 150)])
def test_right_hand_side_adds_the_state_last(size):
    """Without viscosity and surface tension the sweeps leave u3 = u - dt
    AB3(conv): the increment is below 1e-2 of u, so its own roundings (16 of
    them at most) count 0.16 units and the sum's own half a unit."""
    nx, ny, nz = size
    g, p, st = _context(*size, re=1e25, dt=1e-5, scap=0.0)
    rng = np.random.default_rng(nz)
    u = _uniform_u(g, rng)
    g.set_state({**st, "U2": u, "V2": g.zeros("uv"), "W2": g.zeros("w")})
    old = {}
    for h in ("CONV0_U", "CONV1_U"):
        old[h] = np.asfortranarray(rng.normal(scale=50.0, size=u.shape))
        g.set_field(h, old[h])
    g.step(1)
    u3 = g.get_field("U3")
    g.close()
    inner = (slice(1, nx), slice(1, ny + 1))
    U = u.astype(LD)
    conv = LD(0.5) / LD(p.dx) * (U[2:nx + 1, 1:ny + 1] - U[:nx - 1, 1:ny + 1]) * U[inner]
    t = LD(p.dt) * (LD(23) / 12 * conv - LD(4) / 3 * old["CONV1_U"][inner] + LD(5) / 12 * old["CONV0_U"][inner])
    assert np.max(np.abs(t)) < 1e-2
    want = U[inner] - t
    assert np.all(np.abs(u3[inner].astype(LD) - want) <= _half(want) + 0.16 * LD(2.0 ** -53))
