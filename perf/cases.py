"""Performance cases of the TPLS timestep: what a user of this package has it
do, through its public entry points (tpls_gb300.api, tpls_gb300.batch).

A case is a dict of plain values; ``kind`` says which use it stands for:

* ``step``   a channel whose state stays on the device: three timesteps (one
  per phase of the AB3 history), then phi, u, v, w, p into pinned host arrays,
  as a run that keeps an eye on its fields does;
* ``batch``  several small channels of uneven grids advanced together, as the
  parameter studies and the job server do;
* ``interface``  the per-routine calls of a driver that keeps its own time
  loop, on its host arrays: advection, the level-set update with redistancing
  (or the diffuse-interface update), surface tension and viscosity;
* ``momentum``  the driver's momentum calls on host arrays it has registered
  (device-resident behind their addresses): convection, diffusion, and two
  rounds of Jacobi and red-black sweeps of u, v and w, downloaded at the end;
* ``pressure``  the driver's pressure source and Poisson solve on host arrays.

Grids are cubic cells 1/nz; ``re`` and ``m``: Reynolds number and viscosity
ratio (200 and 2 where not given).  ``form``: ``fp64``, or ``mixed`` (FP32 stencils,
sweeps and multigrid levels on an FP64 state, redistancing in FP64: the setting
batched and served jobs run with).
"""
import math

import numpy as np
import torch

from tpls_gb300.api import FIELD_KIND, Params, TplsGpu, shape_of
from tpls_gb300.batch import Batch

OUT_FIELDS = ("PHI2", "U2", "V2", "W2", "PRES")
STEPS = 3
PI_SP = float(np.float32(3.1415926535))
WENO_EPS = float(np.float32(1.0e-7))
LS_ITERS, MOM_ITERS, DIM_ITERS = 10, 30, 18


def listed():
    return [
        # the smallest channel of the configurations: a step is hundreds of
        # short kernels, so launches and dependent latencies count
        {"name": "step64_small", "kind": "step", "form": "fp64", "nx": 64, "ny": 32, "nz": 48},
        # every extent odd: periodic rows exchanged by their own launches, and
        # no extent the multigrid can halve
        {"name": "step64_odd", "kind": "step", "form": "fp64", "nx": 37, "ny": 19, "nz": 23},
        # extents that halve once or twice and then turn odd
        {"name": "step64_ragged", "kind": "step", "form": "fp64", "nx": 100, "ny": 50, "nz": 75},
        # an ordinary grid between the two
        {"name": "step64_mid", "kind": "step", "form": "fp64", "nx": 128, "ny": 64, "nz": 96},
        # the FP64 headline grid
        {"name": "step64_channel", "kind": "step", "form": "fp64", "nx": 256, "ny": 128, "nz": 192},
        # one served job of the FP32-mixed form
        {"name": "mixed_job", "kind": "step", "form": "mixed", "nx": 192, "ny": 96, "nz": 112,
         "re": 350.0, "m": 6.0},
        # the FP32-mixed headline grid, the largest
        {"name": "mixed_channel", "kind": "step", "form": "mixed", "nx": 512, "ny": 256, "nz": 256,
         "re": 500.0, "m": 20.0},
        # a batch of uneven small channels, FP32-mixed
        {"name": "batch_mixed", "kind": "batch", "form": "mixed", "members": 8, "nx": 64, "ny": 32, "nz": 32},
        # a driver's own loop, routine by routine: level set
        {"name": "routines_interface", "kind": "interface", "method": "lsm", "nx": 128, "ny": 64, "nz": 96},
        # the other interface method
        {"name": "routines_dim", "kind": "interface", "method": "dim", "nx": 64, "ny": 32, "nz": 48},
        # the momentum routines on registered arrays
        {"name": "routines_momentum", "kind": "momentum", "nx": 192, "ny": 96, "nz": 144},
        # the pressure routines
        {"name": "routines_pressure", "kind": "pressure", "nx": 128, "ny": 64, "nz": 96},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the kinds above over their ranges of grids, with even
    and odd extents.  Grids with odd extents stay smaller: the pressure solve
    cannot coarsen them far, so they cost more per cell."""
    kind = rng.choice(["step", "step", "step", "batch", "interface", "momentum", "pressure"])
    case = {"kind": kind}
    if kind == "batch":
        return {**case, "form": "mixed", "members": rng.randint(4, 10), "nx": 32 * rng.randint(2, 4),
                "ny": 32 * rng.randint(1, 2), "nz": 16 * rng.randint(2, 5), "re": round(rng.uniform(100.0, 500.0))}
    odd = rng.random() < 0.35
    nx, ny, nz = _log_int(rng, 32, 320), _log_int(rng, 16, 160), _log_int(rng, 20, 200)
    if odd:
        while nx * ny * nz > 400_000:
            nx, ny, nz = max(24, nx * 4 // 5), max(9, ny * 4 // 5), max(12, nz * 4 // 5)
    else:  # multiples of 8, as grids are chosen for multigrid
        nx, ny, nz = (max(16, (n + 4) // 8 * 8) for n in (nx, ny, nz))
    if kind == "step":
        case["form"] = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "interface":
        case["method"] = rng.choice(["lsm", "lsm", "dim"])
    return {**case, "nx": nx, "ny": ny, "nz": nz, "re": round(rng.uniform(100.0, 500.0)),
            "m": round(rng.uniform(1.5, 10.0), 1)}


# ---- inputs -----------------------------------------------------------------

def _members(case):
    """Grids of the channels of a batch: the base grid and uneven multiples of
    its smallest step, in an order of their own."""
    return [(case["nx"] + 32 * (q % 4), case["ny"] + 32 * (q % 3 == 2), case["nz"] + 16 * ((q * 5) % 4))
            for q in range(case["members"])]


def _base_flow(nz, dz, re, m, height, sw):
    """u(z) of the two-layer channel driven by a unit pressure gradient:
    (mu u')' = -1 with the discretisation's wall ghosts, solved directly."""
    def mu(k):
        phi = dz * k - 0.5 * dz - height
        s = 0.0 if phi < -sw else 1.0 if phi > sw else \
            0.5 + phi / (2.0 * sw) + math.sin(PI_SP * phi / sw) / (2.0 * PI_SP)
        return (s + m * (1.0 - s)) / re
    v = [mu(k) for k in range(nz + 2)]
    A = np.zeros((nz, nz))
    for k in range(nz):
        lo, hi = 0.5 * (v[k] + v[k + 1]), 0.5 * (v[k + 2] + v[k + 1])
        A[k, k] += lo + hi
        for q, f, inner in ((k - 1, lo, k + 1), (k + 1, hi, k - 1)):
            if 0 <= q < nz:
                A[k, q] -= f
            else:  # ghost -2 u(wall) + u(inner)/3
                A[k, k] += 2.0 * f
                A[k, inner] -= f / 3.0
    return np.linalg.solve(A / dz ** 2, np.ones(nz))


def _channel(case, dims, seed, **kw):
    """Parameters, inlet profile and seeded fields of one channel, the fields
    as CUDA tensors indexed [z, y, x] (a C-ordered tensor of that shape is the
    Fortran-ordered host array of shape (x, y, z))."""
    nx, ny, nz = dims
    re, m = case.get("re", 200.0), case.get("m", 2.0)
    dx = dz = 1.0 / nz
    sw, height = 1.5 * dx, 0.5
    uz = _base_flow(nz, dz, re, m, height, sw)
    dt = min(0.2 * dx / float(np.abs(uz).max()), 0.5 * math.sqrt(dx ** 3 / (2.0 * math.pi)))
    par = dict(dx=dx, dy=dx, dz=dz, dt=dt, re=re, mu_plus=1.0, mu_minus=m, height=height, scap=1.0,
               smooth_width=sw, mom_u=MOM_ITERS, mom_v=MOM_ITERS, mom_w=MOM_ITERS, levelset=LS_ITERS,
               p_rtol=1e-5, p_maxits=200, **kw)
    rng = np.random.default_rng(seed)
    d, f64 = "cuda", torch.float64
    x = (torch.arange(nx + 2, device=d, dtype=f64) - 0.5) * dx
    y = (torch.arange(ny + 2, device=d, dtype=f64) - 0.5) * dx
    z = (torch.arange(nz + 2, device=d, dtype=f64) - 0.5) * dz
    Lx, Ly = nx * dx, ny * dx
    h = torch.full((ny + 2, nx + 2), height, device=d, dtype=f64)
    for _ in range(4):  # interface modes no shorter than the channel is high
        kx = int(rng.integers(1, max(2, min(5, int(Lx) + 1))))
        ky = int(rng.integers(0, max(1, min(5, int(Ly) + 1))))
        a, th = rng.uniform(0.0, 0.04), rng.uniform(0.0, 2.0 * math.pi)
        h += a * torch.cos(2.0 * math.pi * kx / Lx * x[None, :] + 2.0 * math.pi * ky / Ly * y[:, None] + th)
    gen = torch.Generator(device=d)
    gen.manual_seed(seed)

    def noise(*shape):
        return (2.0 * torch.rand(*shape, device=d, dtype=f64, generator=gen) - 1.0) * 1e-3
    u = torch.tensor(uz, device=d, dtype=f64)[:, None, None].expand(nz, ny + 2, nx + 2).clone()
    v = torch.zeros(nz, ny + 2, nx + 2, device=d, dtype=f64)
    w = torch.zeros(nz + 1, ny + 2, nx + 2, device=d, dtype=f64)
    u[:, 1:ny + 1, 1:nx] += noise(nz, ny, nx - 1)
    v[:, 1:ny + 1, 1:nx + 1] += noise(nz, ny, nx)
    w[1:nz, 1:ny + 1, 1:nx + 1] += noise(nz - 1, ny, nx)
    for q in (u, v, w):
        _wrap_y(q)
    p = (-(torch.arange(nx + 2, device=d, dtype=f64) * dx - 0.5 * dx)).expand(nz + 2, ny + 2, nx + 2).clone()
    return par, uz, {"PHI2": z[:, None, None] - h[None], "U2": u, "V2": v, "W2": w, "PRES": p}, gen


def _pinned(shape, fill=None):
    """A Fortran-ordered host array of that (x, y, z) shape in pinned memory."""
    t = torch.zeros(shape[::-1], dtype=torch.float64, pin_memory=True)
    if fill is not None:
        t.copy_(fill)
    return t.numpy().T


def _context(case, dims, seed):
    extra = {"precision": 1, "fp64_parts": 2} if case["form"] == "mixed" else {}
    par, uz, st, _ = _channel(case, dims, seed, **extra)
    g = TplsGpu(*dims, Params(**par), uz)
    for name, t in st.items():
        g.set_field(name, t.cpu().numpy().T)
    return g


def _member_seed(seed, q):
    return seed * 1000 + q


def prepare(case, seed):
    kind, dims = case["kind"], (case["nx"], case["ny"], case["nz"])
    if kind == "step":
        g = _context(case, dims, seed)
        return {"kind": kind, "g": g, "out": {f: _pinned(g.shape(FIELD_KIND[f])) for f in OUT_FIELDS}}
    if kind == "batch":
        gs = [_context(case, d, _member_seed(seed, q)) for q, d in enumerate(_members(case))]
        outs = [{f: _pinned(g.shape(FIELD_KIND[f])) for f in OUT_FIELDS} for g in gs]
        return {"kind": kind, "batch": Batch(gs), "members": gs, "outs": outs}
    par, uz, st, gen = _channel(case, dims, seed)
    g = TplsGpu(*dims, Params(**par), uz)
    s = {"kind": kind, "g": g, "par": par, "uin": uz}
    arr = {k: _pinned(t.shape[::-1], t) for k, t in _routine_inputs(case, par, st, gen).items()}
    shapes = {k: shape_of(k, *dims) for k in ("p", "uv", "w", "va")}
    if kind == "interface":
        s["method"] = case["method"]
        arr.update({k: _pinned(shapes["p"]) for k in ("conv", "phi3", "fx", "fy", "fz")}, va=_pinned(shapes["va"]))
    elif kind == "momentum":
        arr["va"] = _pinned(shapes["va"])
        arr.update({f"{a}_{c}": _pinned(shapes["w" if c == "w" else "uv"])
                    for a in ("conv", "diff", "a", "b") for c in "uvw"})
        for a in arr.values():
            g.register_host(a)
    else:
        arr.update({k: _pinned(shapes["p"]) for k in ("rhs_p", "pres")})
    s["arr"] = arr
    return s


def _routine_inputs(case, par, st, gen):
    """The driver's arrays before the calls: the fields, and the histories and
    right-hand sides that earlier calls of its loop would have left."""
    d, f64 = "cuda", torch.float64

    def rnd(like, scale):
        return (2.0 * torch.rand(like.shape, device=d, dtype=f64, generator=gen) - 1.0) * scale
    phi, u, v, w = st["PHI2"], st["U2"], st["V2"], st["W2"]
    if case["kind"] == "interface":
        c0, c1 = rnd(phi, 1e-2), rnd(phi, 1e-2)
        if case["method"] == "dim":  # the concentration across the interface
            C = 0.5 + 0.5 * torch.tanh(phi / (2.0 * math.sqrt(2.0) * 1.5 * par["dx"]))
            return {"phi": C, "u": u, "v": v, "w": w, "prev": c0}
        return {"phi": phi, "u": u, "v": v, "w": w, "c0": c0, "c1": c1}
    if case["kind"] == "momentum":
        return {"phi": phi, "u": u, "v": v, "w": w, "rhs_u": u + rnd(u, 1e-3), "rhs_v": v + rnd(v, 1e-3),
                "rhs_w": w + rnd(w, 1e-3)}
    u3, v3, w3 = u + rnd(u, 1e-3), v + rnd(v, 1e-3), w + rnd(w, 1e-3)
    w3[0] = w3[-1] = 0.0
    for q in (u3, v3, w3):
        _wrap_y(q)
    return {"u3": u3, "v3": v3, "w3": w3, "pres_old": st["PRES"]}


# ---- one pass ---------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "step":
        g = state["g"]
        g.step_async(STEPS)
        g.get_fields_into(state["out"])
        g.sync()
        return state["out"]
    if kind == "batch":
        state["batch"].step_async(STEPS)
        for g, out in zip(state["members"], state["outs"]):
            g.get_fields_into(out)
        for g in state["members"]:
            g.sync()
        return state["outs"]
    g, a, q = state["g"], state["arr"], state["par"]
    dx, dy, dz, dt = q["dx"], q["dy"], q["dz"], q["dt"]
    if kind == "interface":
        conv = g.do_advect_phi(a["phi"], a["u"], a["v"], a["w"], dx, dy, dz, conv2_phi=a["conv"])
        if state["method"] == "dim":
            new, prev = g.dim(a["phi"], a["phi"], conv, a["prev"], a["phi"], DIM_ITERS, 1.5 * dz, 1000.0,
                              q["height"], dx, dy, dz, dt)
            return {"conv": conv, "new": new, "prev": prev}
        phi3, err = g.do_tpls(a["phi"], a["c0"], a["c1"], conv, LS_ITERS, q["height"], dx, dz, dt, phi3=a["phi3"])
        g.get_csf(phi3, dx, dy, dz, q["scap"], q["smooth_width"], fx=a["fx"], fy=a["fy"], fz=a["fz"])
        g.get_viscosity(a["phi"], q["smooth_width"], q["re"], q["mu_minus"], q["mu_plus"], viscosity_aug=a["va"])
        return {"conv": conv, "phi3": phi3, "err": err, "fx": a["fx"], "fy": a["fy"], "fz": a["fz"], "va": a["va"]}
    if kind == "momentum":
        g.get_viscosity(a["phi"], q["smooth_width"], q["re"], q["mu_minus"], q["mu_plus"], viscosity_aug=a["va"])
        vel = (a["va"], a["u"], a["v"], a["w"], dx, dy, dz)
        g.get_conv_all(*vel, out=tuple(a["conv_" + c] for c in "uvw"))
        g.get_diffusion_all(*vel, out=tuple(a["diff_" + c] for c in "uvw"))
        for c in "uvw":
            jac, sor = getattr(g, "do_jacobi_" + c), getattr(g, "do_sor_" + c)
            new, old = a["a_" + c], a["b_" + c]
            for it in (1, 2):
                jac(new, old, a["rhs_" + c], a["va"], dx, dy, dz, dt)
                sor(new, a["rhs_" + c], a["va"], dx, dy, dz, dt, 0, it)
                sor(new, a["rhs_" + c], a["va"], dx, dy, dz, dt, 1, it)
                new, old = old, new
        names = ["va"] + [f"{p}_{c}" for p in ("conv", "diff", "a", "b") for c in "uvw"]
        for n in names:
            g.download_host(a[n])
        return {n: a[n] for n in names}
    g.get_source_pres(a["u3"], a["v3"], a["w3"], dx, dy, dz, dt, rhs=a["rhs_p"])
    g.pressure_solve(a["pres_old"], a["rhs_p"], a["u3"], state["uin"], dx, dy, dz, dt, pres=a["pres"])
    return {"rhs_p": a["rhs_p"], "pres": a["pres"]}


def work(case):
    """Bytes: the arrays each call takes and gives, once (a timestep: the 20
    state fields in and out).  Flops per cell: the operators as the routines
    state them (advection 300, a redistancing iteration 25, right-hand sides
    500, a Jacobi sweep 13 and two half-sweeps 16 per component, a pressure
    iteration 80)."""
    grids = _members(case) if case["kind"] == "batch" else [(case["nx"], case["ny"], case["nz"])]
    n = float(sum(nx * ny * nz for nx, ny, nz in grids))
    if case["kind"] in ("step", "batch"):
        flops = 300 + LS_ITERS * 25 + 500 + 3 * (MOM_ITERS // 2) * 29 + 6 * 80
        return {"bytes": n * (STEPS * 40 * 8 + 5 * 8), "flops": n * STEPS * flops}
    if case["kind"] == "interface":
        if case["method"] == "dim":
            return {"bytes": n * 8 * 8, "flops": n * (300 + DIM_ITERS * 40)}
        return {"bytes": n * 8 * 13, "flops": n * (300 + LS_ITERS * 25 + 60)}
    if case["kind"] == "momentum":
        return {"bytes": n * 8 * 20, "flops": n * (300 + 3 * 2 * 29 * 3)}
    return {"bytes": n * 8 * 6, "flops": n * (10 + 6 * 80)}


# ---- the same in plain torch, 64 bits ---------------------------------------
# Arrays are [z, y, x] with the ghost planes of the package's host arrays; J is
# the slice of the interior rows 1..ny.

J = slice(1, -1)


def _wrap_y(a):
    a[:, 0] = a[:, -2]
    a[:, -1] = a[:, 1]
    return a


def _weno5(pos, m2, m1, c0, p1, p2, p3):
    a, b, c, d, e = (torch.where(pos, s, t) for s, t in ((m2, p3), (m1, p2), (c0, p1), (p1, c0), (p2, m1)))
    q1 = 13.0 / 12.0 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2 + WENO_EPS
    q2 = 13.0 / 12.0 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2 + WENO_EPS
    q3 = 13.0 / 12.0 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2 + WENO_EPS
    w1, w2, w3 = 0.1 / q1 ** 2, 0.6 / q2 ** 2, 0.3 / q3 ** 2
    f1 = a / 3 - 7 * b / 6 + 11 * c / 6
    f2 = -b / 6 + 5 * c / 6 + d / 3
    f3 = c / 3 + 5 * d / 6 - e / 6
    return (w1 * f1 + w2 * f2 + w3 * f3) / (w1 + w2 + w3)


def _exact_advect(phi, u, v, w, q):
    nz, ny, nx = phi.shape[0] - 2, phi.shape[1] - 2, phi.shape[2] - 2
    below = torch.arange(ny, device=phi.device)  # row j - 1 of rows 1..ny, periodic
    below[0] = ny
    c = phi[1:-1, J]
    ur = u[:, below][:, :, :nx + 1]
    fx = torch.where(ur >= 0, c[:, :, :nx + 1], c[:, :, 1:nx + 2])
    s = slice(3, nx - 1)
    fx[:, :, s] = _weno5(ur[:, :, s] >= 0, *(c[:, :, 3 + o:nx - 1 + o] for o in range(-2, 4)))
    gx = ur * fx
    rows = phi[1:-1, J, 1:-1]
    vr = v[:, J, 1:-1]  # face above row j
    gy = vr * _weno5(vr >= 0, *(torch.roll(rows, -o, 1) for o in range(-2, 4)))
    wr = w[:, below][:, :, 1:-1]
    col = phi[:, J, 1:-1]
    fz = 0.5 * (col[:-1] + col[1:])
    s = slice(3, nz - 1)
    fz[s] = _weno5(wr[s] >= 0, *(col[3 + o:nz - 1 + o] for o in range(-2, 4)))
    gz = wr * fz
    out = torch.zeros_like(phi)
    out[1:-1, J, 1:-1] = ((gx[:, :, 1:] - gx[:, :, :-1]) / q["dx"] + (gy - torch.roll(gy, 1, 1)) / q["dy"]
                          + (gz[1:] - gz[:-1]) / q["dz"])
    return out


def _level_ghosts(a, inlet):
    """Inlet value, outlet copy, linear z ghosts, periodic rows."""
    a[1:-1, J, 0] = inlet[1:-1, None]
    a[1:-1, J, -1] = a[1:-1, J, -2]
    a[0, J] = 2.0 * a[1, J] - a[2, J]
    a[-1, J] = 2.0 * a[-2, J] - a[-3, J]
    return _wrap_y(a)


def _exact_levelset(phi, c0, c1, c2, q, iters):
    k = torch.arange(phi.shape[0], device=phi.device, dtype=torch.float64)
    a = torch.empty_like(phi)
    a[1:-1, J, 1:-1] = (phi - q["dt"] * (23.0 / 12.0 * c2 - 4.0 / 3.0 * c1 + 5.0 / 12.0 * c0))[1:-1, J, 1:-1]
    _level_ghosts(a, (k * q["dz"] - 0.5 * q["dz"]) - q["height"])
    h = q["dx"]
    inlet = (k * h - 0.5 * h) - q["height"]

    def stencil(a):
        m = a[1:-1, J, 1:-1]
        return m, ((a[1:-1, J, :-2], a[1:-1, J, 2:]), (a[1:-1, :-2, 1:-1], a[1:-1, 2:, 1:-1]),
                   (a[:-2, J, 1:-1], a[2:, J, 1:-1]))
    m, nb = stencil(a)
    near = torch.zeros_like(m, dtype=torch.bool)
    big = torch.full_like(m, h)
    g2 = torch.zeros_like(m)
    for lo, hi in nb:
        near |= (m * lo <= 0) | (m * hi <= 0)
        big = torch.maximum(big, torch.maximum((hi - m).abs(), (lo - m).abs()))
        g2 += (hi - lo) ** 2
    dist = h * m / torch.maximum(big, 0.5 * torch.sqrt(g2))
    sign = torch.sign(m)
    err = 0.0
    for _ in range(iters):
        m, nb = stencil(a)
        g2 = torch.zeros_like(m)
        for lo, hi in nb:
            up = torch.where(sign > 0, m - torch.minimum(lo, hi), torch.maximum(lo, hi) - m)
            g2 += torch.clamp(up, min=0.0) ** 2
        dc = torch.where(near, sign * m.abs() - dist, sign * (torch.sqrt(g2) - h))
        b = torch.empty_like(a)
        b[1:-1, J, 1:-1] = m - 0.3 * dc
        _level_ghosts(b, inlet)
        err = float(((a - b)[:, J, 1:-1] ** 2).sum())
        a = b
    return a, err


def _exact_csf(f, q):
    dx, dy, dz, sw = q["dx"], q["dy"], q["dz"], q["smooth_width"]

    def at(i, j, k):
        n = f.shape
        return f[1 + k:n[0] - 1 + k, 1 + j:n[1] - 1 + j, 1 + i:n[2] - 1 + i]
    m = at(0, 0, 0)
    gx, gy, gz = ((at(1, 0, 0) - at(-1, 0, 0)) / (2 * dx), (at(0, 1, 0) - at(0, -1, 0)) / (2 * dy),
                  (at(0, 0, 1) - at(0, 0, -1)) / (2 * dz))
    xx = (at(1, 0, 0) - 2 * m + at(-1, 0, 0)) / dx ** 2
    yy = (at(0, 1, 0) - 2 * m + at(0, -1, 0)) / dy ** 2
    zz = (at(0, 0, 1) - 2 * m + at(0, 0, -1)) / dz ** 2
    xy = (at(1, 1, 0) - at(-1, 1, 0) - at(1, -1, 0) + at(-1, -1, 0)) / (4 * dx * dy)
    xz = (at(1, 0, 1) - at(-1, 0, 1) - at(1, 0, -1) + at(-1, 0, -1)) / (4 * dx * dz)
    yz = (at(0, 1, 1) - at(0, -1, 1) - at(0, 1, -1) + at(0, -1, -1)) / (4 * dy * dz)
    n2 = gx ** 2 + gy ** 2 + gz ** 2
    flat = n2 < 1e-10
    n2 = torch.where(flat, torch.ones_like(n2), n2)
    kap = -((xx + yy + zz) / n2.sqrt() - (gx * gx * xx + gy * gy * yy + gz * gz * zz) / n2 ** 1.5
            - 2 * (gx * gy * xy + gx * gz * xz + gy * gz * yz) / n2 ** 1.5)
    kap = torch.where(flat, torch.zeros_like(kap), kap).clamp(max=1.0 / min(dx, dy, dz))
    delta = torch.where(m.abs() <= sw, (1 + torch.cos(PI_SP * m / sw)) / (2 * sw), torch.zeros_like(m))
    out = []
    for g in (gx, gy, gz):
        r = torch.zeros_like(f)
        r[1:-1, J, 1:-1] = delta * q["scap"] * kap * g
        r[0], r[-1] = 2 * r[1] - r[2], 2 * r[-2] - r[-3]
        r[:, :, 0], r[:, :, -1] = 2 * r[:, :, 1] - r[:, :, 2], 2 * r[:, :, -2] - r[:, :, -3]
        out.append(_wrap_y(r))
    return out


def _exact_viscosity(phi, q):
    """On x 0..nx+1 with two periodic rows on each side."""
    sw = q["smooth_width"]
    s = 0.5 + phi / (2 * sw) + torch.sin(PI_SP * phi / sw) / (2 * PI_SP)
    s = torch.where(phi < -sw, torch.zeros_like(s), torch.where(phi > sw, torch.ones_like(s), s))
    mu = ((q["mu_plus"] * s + q["mu_minus"] * (1 - s)) / q["re"])[:, J]
    ny = mu.shape[1]
    return mu[:, torch.arange(-2, ny + 2, device=phi.device) % ny].contiguous()


class _Momentum:
    """Component c of the velocity: the operators on its points (i 1..nx, u
    1..nx-1; rows 1..ny; planes 0..nz-1, w 1..nz-1)."""

    def __init__(self, c, mu, q):
        self.c, self.q = c, q
        self.nz, self.ny, self.nx = mu.shape[0] - 2, mu.shape[1] - 4, mu.shape[2] - 2
        self.k0 = 1 if c == "w" else 0
        self.nk, self.ni = self.nz - self.k0, self.nx - (c == "u")

        def m(i, j, k):
            return mu[1 + k:1 + k + self.nk, 3 + j:3 + j + self.ny, 1 + i:1 + i + self.ni]
        a = m(0, 0, 0)
        o = {"u": (1, 0, 0), "v": (0, -1, 0), "w": (0, 0, 1)}[c]  # the cell on the other side of the face
        b = m(*o)

        def edge(i, j, k):
            return 0.25 * (a + b + m(i, j, k) + m(i + o[0], j + o[1], k + o[2]))
        x = (b, a) if c == "u" else (edge(1, 0, 0), edge(-1, 0, 0))
        y = (a, b) if c == "v" else (edge(0, 1, 0), edge(0, -1, 0))
        z = (b, a) if c == "w" else (edge(0, 0, 1), edge(0, 0, -1))
        self.faces = x + y + z

    def at(self, a, i, j, k):
        """a at the points shifted by (i, j, k); a carries one more plane on
        each side of its own."""
        lo = self.k0 + k + 1
        return a[lo:lo + self.nk, 1 + j:1 + j + self.ny, 1 + i:1 + i + self.ni]

    def conv_diff(self, u, v, w):
        q, c = self.q, self.c
        rx, ry, rz = 1.0 / q["dx"], 1.0 / q["dy"], 1.0 / q["dz"]
        px, mx, py, my, pz, mz = self.faces

        def padded(a):
            zero = torch.zeros_like(a[:1])
            return torch.cat([zero, a, zero])
        U, V, W = padded(u), padded(v), padded(w)
        S = {"u": U, "v": V, "w": W}[c]
        at = self.at
        x, up, dn = at(S, 0, 0, 0), at(S, 0, 0, 1).clone(), at(S, 0, 0, -1).clone()
        cz = 0.5 * (up - dn)
        if c != "w":  # walls
            cz[0], cz[-1] = 0.5 * (x[0] + up[0]), -0.5 * (x[-1] + dn[-1])
            dn[0], up[-1] = -2 * x[0] + up[0] / 3, -2 * x[-1] + dn[-1] / 3
        dE, dW, dN, dS = at(S, 1, 0, 0) - x, x - at(S, -1, 0, 0), at(S, 0, 1, 0) - x, x - at(S, 0, -1, 0)
        diff = ((px * dE - mx * dW) * rx * rx + (py * dN - my * dS) * ry * ry
                + (pz * (up - x) - mz * (x - dn)) * rz * rz)

        def mean(a, offs):
            return 0.25 * sum(at(a, *o) for o in offs)
        if c == "u":
            vel = (x, mean(V, [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0)]),
                   mean(W, [(0, 0, 0), (1, 0, 0), (0, 0, 1), (1, 0, 1)]))
            E, Wt = px * dE * rx, mx * dW * rx
            N, Sf = py * (at(V, 1, 1, 0) - at(V, 0, 1, 0)) * rx, my * (at(V, 1, 0, 0) - at(V, 0, 0, 0)) * rx
            T, B = pz * (at(W, 1, 0, 1) - at(W, 0, 0, 1)) * rx, mz * (at(W, 1, 0, 0) - at(W, 0, 0, 0)) * rx
        elif c == "v":
            vel = (mean(U, [(-1, -1, 0), (-1, 0, 0), (0, -1, 0), (0, 0, 0)]), x,
                   mean(W, [(0, -1, 0), (0, 0, 0), (0, -1, 1), (0, 0, 1)]))
            E, Wt = px * (at(U, 0, 0, 0) - at(U, 0, -1, 0)) * ry, mx * (at(U, -1, 0, 0) - at(U, -1, -1, 0)) * ry
            N, Sf = py * dN * ry, my * dS * ry
            T, B = pz * (at(W, 0, 0, 1) - at(W, 0, -1, 1)) * ry, mz * (at(W, 0, 0, 0) - at(W, 0, -1, 0)) * ry
        else:
            vel = (mean(U, [(-1, 0, -1), (-1, 0, 0), (0, 0, -1), (0, 0, 0)]),
                   mean(V, [(0, 0, -1), (0, 0, 0), (0, 1, -1), (0, 1, 0)]), x)
            E, Wt = px * (at(U, 0, 0, 0) - at(U, 0, 0, -1)) * rz, mx * (at(U, -1, 0, 0) - at(U, -1, 0, -1)) * rz
            N, Sf = py * (at(V, 0, 1, 0) - at(V, 0, 1, -1)) * rz, my * (at(V, 0, 0, 0) - at(V, 0, 0, -1)) * rz
            T, B = pz * (up - x) * rz, mz * (x - dn) * rz
        conv = (0.5 * (dE + dW) * rx * vel[0] + 0.5 * (dN + dS) * ry * vel[1] + cz * rz * vel[2]
                - ((E - Wt) * rx + (N - Sf) * ry + (T - B) * rz))
        return conv, diff

    def place(self, a, like):
        """a on the points, zero elsewhere."""
        out = torch.zeros_like(like)
        out[self.k0:self.k0 + self.nk, J, 1:1 + self.ni] = a
        return out

    def coefficients(self, rhs):
        """x_new = sum(coef * neighbour) + b, the wall ghosts folded in (the
        outer z slot of a wall level multiplies the point itself)."""
        q = self.q
        s = [0.5 * q["dt"] / q[d] ** 2 for d in ("dx", "dx", "dy", "dy", "dz", "dz")]
        a = [si * f for si, f in zip(s, self.faces)]
        r = 1.0 / (1.0 + sum(a))
        a = [x * r for x in a]
        if self.c != "w":
            a[4][0] += a[5][0] / 3
            a[5][0] *= -2
            a[5][-1] += a[4][-1] / 3
            a[4][-1] *= -2
        self.coef = a
        self.b = r * rhs[self.k0:self.k0 + self.nk, J, 1:1 + self.ni]
        i = torch.arange(1, 1 + self.ni, device=rhs.device)[None, None]
        j = torch.arange(1, 1 + self.ny, device=rhs.device)[None, :, None]
        k = torch.arange(self.k0, self.k0 + self.nk, device=rhs.device)[:, None, None]
        self.ij, self.ijk = (i + j) % 2, (i + j + k) % 2

    def _terms(self, x):
        """The point itself and its neighbours (+x, -x, +y, -y, +z, -z)."""
        p, n = x[self.k0:self.k0 + self.nk, J, 1:1 + self.ni], slice(self.k0, self.k0 + self.nk)
        if self.c == "w":
            up, dn = x[2:2 + self.nk, J, 1:1 + self.ni], x[:self.nk, J, 1:1 + self.ni]
        else:
            up, dn = torch.cat([p[1:], p[-1:]]), torch.cat([p[:1], p[:-1]])
        return p, (x[n, J, 2:2 + self.ni], x[n, J, :self.ni], x[n, 2:, 1:1 + self.ni], x[n, :-2, 1:1 + self.ni], up, dn)

    def jacobi(self, old, new):
        _, nb = self._terms(old)
        v = self.b + sum(c * x for c, x in zip(self.coef, nb))
        new[self.k0:self.k0 + self.nk, J, 1:1 + self.ni] = v

    def half_sweep(self, x, flg, it):
        p, nb = self._terms(x)
        if it % 2 == 0:  # checkerboard
            v = self.b + sum(c * y for c, y in zip(self.coef, nb))
            v = torch.where(self.ijk != flg, p + 1.2 * (v - p), p)
        else:  # columns, upwards
            part = self.b + sum(c * y for c, y in zip(self.coef[:5], nb[:5]))
            A, B = p + 1.2 * (part - p), 1.2 * self.coef[5]
            v = torch.empty_like(p)
            v[0] = torch.addcmul(A[0], B[0], nb[5][0])
            for k in range(1, self.nk):
                torch.addcmul(A[k], B[k], v[k - 1], out=v[k])
            v = torch.where(self.ij != flg, v, p)
        x[self.k0:self.k0 + self.nk, J, 1:1 + self.ni] = v

    def rows(self, x, pres, own=False):
        """The boundary rows after a sweep; own: those the routine itself
        writes, without the driver's pressure outlet of u."""
        n = slice(self.k0, self.k0 + self.nk)
        if self.c != "u":
            x[n, J, 0], x[n, J, -1] = x[n, J, 1], x[n, J, -2]
        elif not own:
            x[:, J, 0] = x[:, J, 1]
            P, nx = pres[1:-1, J], self.nx
            x[:, J, nx] = x[:, J, nx - 1] + self.q["dt"] / self.q["dx"] * (P[..., nx + 1] + P[..., nx - 1]
                                                                           - 2 * P[..., nx])
            x[:, J, nx + 1] = 0.0
        if self.c == "w":
            x[0, J], x[-1, J] = 0.0, 0.0

    def solve(self, like, pres, iters):
        x = [torch.zeros_like(like), torch.zeros_like(like)]
        for it in range(1, iters // 2 + 1):
            old, new = x[(it - 1) % 2], x[it % 2]
            self.jacobi(old, new)
            self.rows(new, pres)
            _wrap_y(new)
            for flg in (0, 1):
                self.half_sweep(new, flg, it)
                if flg:
                    self.rows(new, pres)
                _wrap_y(new)
        return new


def _exact_source(u, v, w, q):
    nz, ny = u.shape[0], u.shape[1] - 2
    below = torch.arange(ny, device=u.device)
    below[0] = ny
    out = torch.zeros(nz + 2, ny + 2, u.shape[2], device=u.device, dtype=u.dtype)
    ub, wb = u[:, below], w[:, below]
    out[1:-1, J, 1:-1] = ((ub[..., 1:-1] - ub[..., :-2]) / q["dx"] + (v[:, J] - v[:, below])[..., 1:-1] / q["dy"]
                          + (wb[1:] - wb[:-1])[..., 1:-1] / q["dz"]) / q["dt"]
    return out


def _exact_pressure(rhs, u, uin, pold, q):
    """Direct solution of the interior system (cosines in x and z, Fourier in
    y) with the interior mean of pold, and its ghosts."""
    nz, ny, nx = (n - 2 for n in rhs.shape)
    row = torch.arange(ny, device=rhs.device)  # u row of p row j + 1
    row[0] = ny
    bin_ = (q["dx"] / q["dt"]) / q["dy"] * (uin[:, None] - u[:, row, 0])
    b = -rhs[1:-1, J, 1:-1].clone()
    b[..., 0] += bin_ / q["dy"]
    b -= b.mean()

    def cosines(n):
        k = torch.arange(n, device=rhs.device, dtype=torch.float64)[:, None]
        i = torch.arange(n, device=rhs.device, dtype=torch.float64)[None]
        Q = torch.cos(math.pi * k * (i + 0.5) / n) * math.sqrt(2.0 / n)
        Q[0] = math.sqrt(1.0 / n)
        return Q, 4.0 * torch.sin(math.pi * k[:, 0] / (2 * n)) ** 2
    (Qx, lx), (Qz, lz) = cosines(nx), cosines(nz)
    m = torch.arange(ny // 2 + 1, device=rhs.device, dtype=torch.float64)
    ly = 4.0 * torch.sin(math.pi * m / ny) ** 2
    # the operator as the reference assembles it: 1/dy^2 along x, 1/dx^2 along y
    lam = lx[None, None] / q["dy"] ** 2 + ly[None, :, None] / q["dx"] ** 2 + lz[:, None, None] / q["dz"] ** 2
    lam[0, 0, 0] = 1.0
    t = torch.fft.rfft(torch.einsum("ck,kjm->cjm", Qz, b @ Qx.T), dim=1) / lam
    t[0, 0, 0] = 0.0
    x = torch.einsum("ck,cjm->kjm", Qz, torch.fft.irfft(t, n=ny, dim=1)) @ Qx
    x += pold[1:-1, J, 1:-1].mean() - x.mean()
    p = torch.empty_like(rhs)
    p[1:-1, J, 1:-1] = x
    p[1:-1, J, 0] = x[..., 0] + q["dy"] * bin_
    p[1:-1, J, -1] = x[..., -1]
    p[0, J], p[-1, J] = p[1, J], p[-2, J]
    return _wrap_y(p)


def _exact_steps(case, dims, seed, steps):
    q, uz, s, _ = _channel(case, dims, seed)
    uin = torch.tensor(uz, device="cuda", dtype=torch.float64)
    phi, u, v, w, p = (s[f] for f in OUT_FIELDS)
    vel = {"u": u, "v": v, "w": w}
    zero = {c: (torch.zeros_like(a), torch.zeros_like(a)) for c, a in vel.items()}
    conv, force = dict(zero), dict(zero)  # (older, newer)
    cphi = (torch.zeros_like(phi), torch.zeros_like(phi))
    pold = torch.zeros_like(phi)

    def ab3(new, old):
        return 23.0 / 12.0 * new - 4.0 / 3.0 * old[1] + 5.0 / 12.0 * old[0]
    for _ in range(steps):
        mu = _exact_viscosity(phi, q)
        c2 = _exact_advect(phi, vel["u"], vel["v"], vel["w"], q)
        phi, _ = _exact_levelset(phi, cphi[0], cphi[1], c2, q, LS_ITERS)
        cphi = (cphi[1], c2)
        fx, fy, fz = _exact_csf(phi, q)
        out = {}
        for c, a in vel.items():
            mom = _Momentum(c, mu, q)
            cv, df = (mom.place(t, a) for t in mom.conv_diff(vel["u"], vel["v"], vel["w"]))
            # the force between the two cells of each face, rows j + 1
            f2 = torch.zeros_like(a)
            if c == "u":
                f2[:, J, 1:-1] = 0.5 * (fx[1:-1, 2:, 2:] + fx[1:-1, 2:, 1:-1])
            elif c == "v":
                f2[:, J, 1:-1] = 0.5 * (fy[1:-1, 2:, 1:-1] + fy[1:-1, J, 1:-1])
            else:
                f2[:, J, 1:-1] = 0.5 * (fz[1:, 2:, 1:-1] + fz[:-1, 2:, 1:-1])
            rhs = a - q["dt"] * ab3(cv, conv[c]) + 0.5 * q["dt"] * df + q["dt"] * ab3(f2, force[c])
            conv[c], force[c] = (conv[c][1], cv), (force[c][1], f2)
            mom.coefficients(rhs)
            out[c] = mom.solve(a, p, MOM_ITERS)
        u3, v3, w3 = out["u"], out["v"], out["w"]
        p = _exact_pressure(_exact_source(u3, v3, w3, q), u3, uin, pold, q)
        rx, ry, rz = q["dt"] / q["dx"], q["dt"] / q["dy"], q["dt"] / q["dz"]
        u3, v3, w3 = u3.clone(), v3.clone(), w3.clone()
        u3[:, J, :-1] -= rx * (p[1:-1, 2:, 1:] - p[1:-1, 2:, :-1])
        u3[..., 0], u3[..., -1] = uin[:, None], 0.0
        v3[:, J] -= ry * (p[1:-1, 2:] - p[1:-1, J])
        w3[:, J] -= rz * (p[1:, 2:] - p[:-1, 2:])
        vel = {"u": _wrap_y(u3), "v": _wrap_y(v3), "w": _wrap_y(w3)}
        pold = p
    return dict(zip(OUT_FIELDS, (phi, vel["u"], vel["v"], vel["w"], p)))


def _host_order(v):
    return v.permute(2, 1, 0) if isinstance(v, torch.Tensor) else v


def exact(case, seed):
    """What run() returns for the first pass on these inputs."""
    kind, dims = case["kind"], (case["nx"], case["ny"], case["nz"])
    if kind == "step":
        r = _exact_steps(case, dims, seed, STEPS)
    elif kind == "batch":
        return [{f: _host_order(a) for f, a in _exact_steps(case, d, _member_seed(seed, q), STEPS).items()}
                for q, d in enumerate(_members(case))]
    else:
        q, uz, st, gen = _channel(case, dims, seed)
        a = _routine_inputs(case, q, st, gen)
        if kind == "interface":
            r = {"conv": _exact_advect(a["phi"], a["u"], a["v"], a["w"], q)}
            if case["method"] == "dim":
                r.update(new=None, prev=None)
            else:
                r["phi3"], r["err"] = _exact_levelset(a["phi"], a["c0"], a["c1"], r["conv"], q, LS_ITERS)
                r["fx"], r["fy"], r["fz"] = _exact_csf(r["phi3"], q)
                r["va"] = torch.nn.functional.pad(_exact_viscosity(a["phi"], q), (1, 1))
        elif kind == "momentum":
            mu = _exact_viscosity(a["phi"], q)
            r = {"va": torch.nn.functional.pad(mu, (1, 1))}
            for c in "uvw":
                mom = _Momentum(c, mu, q)
                r["conv_" + c], r["diff_" + c] = (mom.place(t, a[c]) for t in mom.conv_diff(a["u"], a["v"], a["w"]))
                mom.coefficients(a["rhs_" + c])
                new, old = torch.zeros_like(a[c]), torch.zeros_like(a[c])
                first = new
                for it in (1, 2):
                    mom.jacobi(old, new)
                    mom.rows(new, None, own=True)
                    for flg in (0, 1):
                        mom.half_sweep(new, flg, it)
                    new, old = old, new
                r["a_" + c], r["b_" + c] = first, new if new is not first else old
        else:
            rhs = _exact_source(a["u3"], a["v3"], a["w3"], q)
            uin = torch.tensor(uz, device="cuda", dtype=torch.float64)
            r = {"rhs_p": rhs, "pres": _exact_pressure(rhs, a["u3"], uin, a["pres_old"], q)}
    return {k: _host_order(v) for k, v in r.items()}
