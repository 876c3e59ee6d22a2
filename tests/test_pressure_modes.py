"""The coarsest multigrid level by modes (csrc/tpls_modes.cuh).

CPU: the transforms as the kernels index them (folded halves, mode groups,
paired points) and the x recurrences give what the damped z-line sweeps give.
GPU: solves on grids that take that path (one to eight points per lane) and on
one line too long for it, against the oracle's exact solve."""
import numpy as np
import pytest

SWEEPS, W = 40, 0.8


def _cos(n):
    k, i = np.arange(n)[:, None], np.arange(n)[None]
    Q = np.cos(np.pi * k * (i + 0.5) / n) * np.sqrt(2.0 / n)
    Q[0] = np.sqrt(1.0 / n)
    return Q, 4.0 * np.sin(np.pi * k[:, 0] / (2 * n)) ** 2


def _fourier(n):
    Q, lam = [np.full(n, np.sqrt(1.0 / n))], [0.0]
    i = np.arange(n)
    for m in range(1, (n + 1) // 2):
        for f in (np.cos, np.sin):
            Q.append(np.sqrt(2.0 / n) * f(2 * np.pi * m * i / n))
            lam.append(4.0 * np.sin(np.pi * m / n) ** 2)
    if n % 2 == 0:
        Q.append(np.sqrt(1.0 / n) * (-1.0) ** i)
        lam.append(4.0)
    return np.array(Q), np.array(lam)


def _sweeps(b, c):
    nz, ny, nx = b.shape
    nbx = np.array([(0 if nx == 1 else 1 if i in (0, nx - 1) else 2) for i in range(nx)])
    Tz = np.diag([0.0 if nz == 1 else 1.0 if k in (0, nz - 1) else 2.0 for k in range(nz)])
    Tz -= np.diag(np.ones(nz - 1), 1) + np.diag(np.ones(nz - 1), -1)
    D = [c[2] * Tz + (c[0] * n + 2 * c[1]) * np.eye(nz) for n in nbx]
    e = np.zeros_like(b)
    for _ in range(SWEEPS):
        r = b + c[1] * (np.roll(e, 1, 1) + np.roll(e, -1, 1))
        r[:, :, 1:] += c[0] * e[:, :, :-1]
        r[:, :, :-1] += c[0] * e[:, :, 1:]
        e = (1 - W) * e + W * np.stack([np.linalg.solve(D[i], r[:, :, i]) for i in range(nx)], 2)
    return e


def _modes_z(Q, a):
    n, out = len(Q), np.full_like(a, np.nan)
    for g in range(2 * ((n + 7) // 8)):
        par, m0 = g & 1, (g >> 1) * 8 + (g & 1)
        for m in range(m0, min(m0 + 8, n), 2):
            half = n // 2
            v = a[:half] + (-1) ** par * a[::-1][:half]
            acc = np.tensordot(Q[m, :half], v, 1)
            if n % 2 and not par:
                acc = acc + Q[m, half] * a[half]
            assert np.isnan(out[m]).all()
            out[m] = acc
    return out


def _points_z(Q, a):
    n, out = len(Q), np.full_like(a, np.nan)
    half = (n + 1) // 2
    for k in range(half):
        e, o = np.tensordot(Q[::2, k], a[::2], 1), np.tensordot(Q[1::2, k], a[1::2], 1)
        out[k], out[n - 1 - k] = e + o, e - o
        if k == n - 1 - k:
            assert np.max(np.abs(o)) < 1e-13  # odd modes vanish at the middle point
    return out


@pytest.mark.parametrize("size", [(5, 3, 7), (1, 4, 6), (37, 5, 1), (9, 2, 2), (12, 6, 17)])
def test_modes_equal_the_line_sweeps(size):
    nx, ny, nz = size
    c = (1.3, 0.9, 0.4)
    b = np.random.default_rng(nx).normal(size=(nz, ny, nx))
    (Qz, lz), (Qy, ly) = _cos(nz), _fourier(ny)
    t = np.einsum("mj,kji->kmi", Qy, _modes_z(Qz, b))
    nbx = np.array([(0 if nx == 1 else 1 if i in (0, nx - 1) else 2) for i in range(nx)])
    wd = W / (c[0] * nbx[None, None] + 2 * c[1] + c[2] * lz[:, None, None])
    al, be, ga = (1 - W) + wd * c[1] * (2 - ly)[None, :, None], wd * c[0], wd * t
    e = ga
    for _ in range(SWEEPS - 1):
        s = np.zeros_like(e)
        s[:, :, 1:] += e[:, :, :-1]
        s[:, :, :-1] += e[:, :, 1:]
        e = al * e + be * s + ga
    got = _points_z(Qz, np.einsum("mj,kmi->kji", Qy, e))
    assert np.max(np.abs(got - _sweeps(b, c))) < 1e-12  # a few hundred roundings of values of order 1


@pytest.mark.parametrize("nz", [1, 2, 5, 8, 9, 23, 75, 130])
def test_line_solve_in_runs_equals_the_tridiagonal_solve(nz):
    """k_line_jacobi3: eight runs of levels solved from zero and joined by the
    products of their multipliers (empty runs pass values through)."""
    W8, cz, dxy = 8, 0.7, 1.9
    run = (nz + W8 - 1) // W8
    d = dxy + cz * np.array([0.0 if nz == 1 else 1.0 if k in (0, nz - 1) else 2.0 for k in range(nz)])
    cp, inv = np.zeros(nz), np.zeros(nz)
    for k in range(nz):
        den = d[k] + (cz * cp[k - 1] if k else 0.0)
        cp[k], inv[k] = -cz / den, 1.0 / den
    pf, pb = np.zeros(nz), np.zeros(nz)
    runs = [(min(w * run, nz), min(min(w * run, nz) + run, nz)) for w in range(W8)]
    for k0, k1 in runs:
        for k in range(k0, k1):
            pf[k] = cz * inv[k] * (pf[k - 1] if k > k0 else 1.0)
        for k in range(k1 - 1, k0 - 1, -1):
            pb[k] = (-cp[k] if k < nz - 1 else 0.0) * (pb[k + 1] if k < k1 - 1 else 1.0)
    rhs = np.random.default_rng(nz).normal(size=nz)
    buf, se, sp = np.zeros(nz), np.zeros(W8), np.ones(W8)
    for w, (k0, k1) in enumerate(runs):
        y = 0.0
        for k in range(k0, k1):
            y = (cz * y + rhs[k]) * inv[k]
            buf[k] = y
        se[w], sp[w] = y, pf[k1 - 1] if k1 > k0 else 1.0
    se2, sp2 = np.zeros(W8), np.ones(W8)
    for w, (k0, k1) in enumerate(runs):
        v_in = 0.0
        for v in range(w):
            v_in = sp[v] * v_in + se[v]
        x = 0.0
        for k in range(k1 - 1, k0 - 1, -1):
            yk = pf[k] * v_in + buf[k]
            x = yk - (cp[k] * x if k < nz - 1 else 0.0)
            buf[k] = x
        se2[w], sp2[w] = x, pb[k0] if k1 > k0 else 1.0
    out = np.zeros(nz)
    for w, (k0, k1) in enumerate(runs):
        v_in = 0.0
        for v in range(W8 - 1, w, -1):
            v_in = sp2[v] * v_in + se2[v]
        out[k0:k1] = pb[k0:k1] * v_in + buf[k0:k1]
    A = np.diag(d) - cz * (np.diag(np.ones(nz - 1), 1) + np.diag(np.ones(nz - 1), -1))
    assert np.max(np.abs(out - np.linalg.solve(A, rhs))) < 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(31, 19, 23), (37, 9, 15), (101, 5, 21), (131, 9, 25), (259, 5, 9), (50, 25, 75)])
def test_solves_through_the_modes_match_the_exact_solve(size):
    """As test_pressure_solve_tight: rtol 1e-13, 1e-10 of the maximum."""
    from oracle.oracle import Oracle
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    nx, ny, nz = size
    p, uin, st = make_case("A", nx=nx, ny=ny, nz=nz)
    rng = np.random.default_rng(nx)
    u3 = np.asfortranarray(st["U2"] + rng.normal(scale=1e-3, size=st["U2"].shape))
    u3[:, 0], u3[:, -1] = u3[:, -2], u3[:, 1]
    with TplsGpu(nx, ny, nz, p, uin) as g:
        o = Oracle(nx, ny, nz, p, uin)
        rhs = g.get_source_pres(u3, st["V2"], st["W2"], p.dx, p.dy, p.dz, p.dt)
        pold = np.zeros_like(st["PRES"], order="F")
        po, *_ = o.pressure_solve(pold, rhs, u3, uin, p.dx, p.dy, p.dz, p.dt)
        pg, its, _, reason = g.pressure_solve(pold, rhs, u3, uin, p.dx, p.dy, p.dz, p.dt, rtol=1e-13, maxits=400)
    assert reason == 2
    assert np.max(np.abs(pg - po)) <= 1e-10 * np.max(np.abs(po))
