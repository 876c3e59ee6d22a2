"""The per-routine entries on arrays in the host layout (csrc/tpls_api.cu):
plain host arrays (copied in and out) and registered ones (the kernels work on
the device mirrors themselves) give the same values bit for bit, also where an
output is an input as well (then everything is copied), and where several
arrays live in one registered buffer."""
import numpy as np
import pytest

from tpls_gb300.api import TplsGpu
from tpls_gb300.channel import make_case

SIZES = [(37, 19, 23), (64, 8, 130)]


def _arrays(g, st, seed):
    rng = np.random.default_rng(seed)

    def rnd(kind, s=1.0):
        return np.asfortranarray(rng.normal(scale=s, size=g.shape(kind)))
    a = {"phi": np.array(st["PHI2"], order="F"), "va": np.asfortranarray(rng.uniform(0.01, 0.02, size=g.shape("va")))}
    for n, kind in (("u", "uv"), ("v", "uv"), ("w", "w")):
        a[n] = np.array(st[n.upper() + "2"], order="F") + rnd(kind, 1e-2)
        a["x" + n], a["o" + n], a["r" + n], a["c" + n] = rnd(kind), rnd(kind), rnd(kind), rnd(kind)
    for n in ("conv", "c0", "c1", "phi3", "fx", "fy", "fz", "prev", "new", "rhs"):
        a[n] = rnd("p", 1e-2)
    return a


def _calls(g, p, a):
    d = (p.dx, p.dy, p.dz)
    g.exchange2d(a["ru"])
    g.do_advect_phi(a["phi"], a["u"], a["v"], a["w"], *d, conv2_phi=a["conv"])
    g.do_tpls(a["phi"], a["c0"], a["c1"], a["conv"], 5, p.height, p.dx, p.dz, p.dt, phi3=a["phi3"])
    g.get_csf(a["phi3"], *d, p.scap, p.smooth_width, fx=a["fx"], fy=a["fy"], fz=a["fz"])
    g.get_viscosity(a["phi"], p.smooth_width, p.re, p.mu_minus, p.mu_plus, viscosity_aug=a["va"])
    vel = (a["va"], a["u"], a["v"], a["w"])
    g.get_conv_all(*vel, *d, out=(a["cu"], a["cv"], a["cw"]))
    out = [g.get_diffusion_all(*vel, *d)]
    for n in "uvw":
        getattr(g, "do_jacobi_" + n)(a["x" + n], a["o" + n], a["r" + n], a["va"], *d, p.dt)
        for it in (1, 2):
            getattr(g, "do_sor_" + n)(a["x" + n], a["r" + n], a["va"], *d, p.dt, it % 2, it)
    # the new iterate is also the old one: every array is copied
    g.do_jacobi_u(a["ou"], a["ou"], a["ru"], a["va"], *d, p.dt)
    g.get_source_pres(a["xu"], a["xv"], a["xw"], *d, p.dt, rhs=a["rhs"])
    out.append(g.get_difference(a["xu"], a["ou"]))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("how", ["each", "one buffer"])
def test_registered_arrays_give_the_same_values(size, how):
    p, uin, st = make_case("A", nx=size[0], ny=size[1], nz=size[2])
    with TplsGpu(*size, p, uin) as g:
        plain = _arrays(g, st, 5)
        reg = {k: v.copy(order="F") for k, v in plain.items()}
        if how == "each":
            for x in reg.values():
                g.register_host(x)
        else:
            buf = np.concatenate([x.ravel(order="F") for x in reg.values()])
            at = 0
            for k, x in reg.items():
                reg[k] = buf[at:at + x.size].reshape(x.shape, order="F")
                at += x.size
            g.register_host(buf)
        r0, r1 = _calls(g, p, plain), _calls(g, p, reg)
        g.download_host()
        for k in plain:
            assert np.array_equal(plain[k], reg[k]), k
        assert all(np.array_equal(x, y) for x, y in zip(r0[0], r1[0])) and r0[1] == r1[1]
