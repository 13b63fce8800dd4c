"""The one-pass forms of rk, rk_2fl and the ghost fills against the oracle's
restatement and against the passes they stand in for.

Bounds: as in test_gpu_procedures.py (rk_2fl 1e-13, rk 1e-12 of the field's
maximum); the one-launch ghost fill is bit-equal to the oracle's stages.
"""
import numpy as np
import pytest

import oracle as O
from cansfz import case as C

from test_gpu_parity import _nml, _rand_fields, _rel

pytestmark = pytest.mark.gpu


class _Shifted(C.DeviceField):
    """A field whose base address is a multiple of 8 bytes only."""

    def __init__(self, shape, device="cuda"):
        import torch

        self.shape = tuple(shape)
        self.t = torch.zeros(int(np.prod(shape)) + 1, dtype=torch.float64, device=device)[1:]


@pytest.mark.parametrize("ng,opts,shifted", [((24, 16, 20), "", False), ((10, 2, 9), "", False), ((36, 10, 13), "", True),
                                             ((70, 6, 24), "balanced", False), ((24, 14, 9), "balanced", True),
                                             ((24, 16, 20), "buoyancy", False), ((300, 2, 9), "", False)])
def test_rk_with_pn_equal_p(ng, opts, shifted):
    """rk called with pn = p, two calls (the history): the oracle, and the
    same call with a copy of p as pn, which takes the pass-by-pass route."""
    p = _nml(*ng, "PPPPNN", l=(1.0, 0.75, 1.2))
    p.balanced = int(opts == "balanced")
    p.scalar = p.boussinesq = int(opts == "buoyancy")
    p.beta12[:] = [0.01, 0.02]
    rng, f, psi = _rand_fields(p, 22)
    psio = np.asfortranarray(np.clip(psi + 0.05 * rng.standard_normal(psi.shape), 0, 1))
    u, v, w, fx, fy, fz, pp, po, kap, s = (f(0.2) for _ in range(10))
    o = O.Case(p)
    ref = [a.copy(order="F") for a in (u, v, w)]
    cases = [C.Case(p), C.Case(p)]
    mk = (lambda a: _Shifted(a.shape).set(a)) if shifted else cases[0].field
    dev = {k: mk(a) for k, a in dict(psi=psi, psio=psio, fx=fx, fy=fy, fz=fz, p=pp, po=po, k=kap, s=s).items()}
    other = mk(pp)
    vel = [[mk(a) for a in (u, v, w)] for _ in cases]
    sc = (dev["s"], s) if opts == "buoyancy" else (None, None)
    for rkpar, dt, dt_r in (([1.0, 0.0], 1e-3, 1.0), ([1.4, -0.4], 1.2e-3, 1.2)):
        for g, pn, uvw in zip(cases, (dev["p"], other), vel):
            g.call("rk", list(rkpar), dt, dt_r, [0.0, 0.0, 0.0], dev["psi"], dev["k"], dev["p"], pn, dev["po"], sc[0],
                   dev["psio"], dev["fx"], dev["fy"], dev["fz"], *uvw)
        o.call("rk", np.array(rkpar), dt, dt_r, np.zeros(3), psi, kap, pp, pp, po, sc[1], psio, fx, fy, fz, *ref)
        for a, b, c in zip(vel[0], vel[1], ref):
            inner = (slice(1, -1),) * 3
            assert _rel(a.get()[inner], c[inner]) < 1e-12
            assert _rel(a.get()[inner], b.get()[inner]) < 1e-12
            ghosts = np.ones(c.shape, bool)
            ghosts[inner] = False
            assert np.array_equal(a.get()[ghosts], b.get()[ghosts])


@pytest.mark.parametrize("ng,vof", [((36, 10, 13), False), ((10, 2, 9), False), ((36, 10, 13), True), ((64, 16, 24), True),
                                    ((126, 2, 9), False), ((128, 2, 9), False), ((300, 4, 7), False), ((1024, 2, 5), True)])
def test_rk_2fl_in_one_pass(ng, vof):
    p = _nml(*ng, "PPPPNN", l=(1.0, 0.75, 1.2), vof=vof)
    g, o = C.Case(p), O.Case(p)
    rng, f, psi = _rand_fields(p, 21)
    u, v, w, nx, ny, nz, phi = (f(0.3) for _ in range(7))
    psi[0, 0, 0] = 1.5  # a ghost beyond [0, 1]: clip_field works on the whole array
    dev = [g.field(a) for a in (u, v, w, nx, ny, nz, phi)]
    psig, ref = g.field(psi), psi.copy(order="F")
    fg, fo = [g.field() for _ in range(3)], [o.empty() for _ in range(3)]
    for rkpar, dt in (([1.0, 0.0], 2e-3), ([1.45, -0.45], 1.7e-3)):
        g.call("rk_2fl", list(rkpar), dt, 0.7, 0.013, 1.0, *dev, psig, *fg)
        o.call("rk_2fl", np.array(rkpar), dt, 0.7, 0.013, 1.0, u, v, w, nx, ny, nz, phi, ref, *fo)
        assert _rel(psig.get(), ref) < 1e-13
        assert psig.get().min() >= 0.0 and psig.get().max() <= 1.0
        for a, b in zip(fg, fo):
            assert _rel(a.get()[1:-1, 1:-1, 1:-1], b[1:-1, 1:-1, 1:-1]) < 1e-13


@pytest.mark.parametrize("cbcpre", ["PPPPNN", "NNPPNN", "DDPPNN", "PPNNNN", "PPPPPP", "NNNNNN", "DDNNDD", "PPPPDD"])
@pytest.mark.parametrize("ng", [(24, 16, 20), (6, 2, 3), (36, 6, 9)])
def test_ghost_fills_in_one_launch(cbcpre, ng):
    p = _nml(*ng, cbcpre, l=(1.0, 0.75, 1.2))
    for q in range(18):
        p.bcvel[q] = 0.1 * q - 0.3
    for q in range(6):
        p.bcpre[q] = 0.2 * q if cbcpre[q] == "D" else 0.0
    g, o = C.Case(p), O.Case(p)
    _, f, _ = _rand_fields(p, 31)
    for which in range(6):
        a = f()
        ag = g.field(a)
        g.call("boundp", which, ag)
        o.call("boundp", which, a)
        assert np.array_equal(ag.get(), a), which
    for correc in (0, 1):
        uvw = [f() for _ in range(3)]
        dev = [g.field(a) for a in uvw]
        g.call("bounduvw", correc, *dev)
        o.call("bounduvw", correc, *uvw)
        for a, b in zip(dev, uvw):
            assert np.array_equal(a.get(), b), correc


@pytest.mark.parametrize("ng", [(24, 16, 20), (126, 6, 9), (128, 14, 5), (10, 2, 9), (300, 2, 7), (6, 36, 3)])
def test_correc_in_rows_and_in_tiles(ng):
    """correc's two block shapes, ghost ranges included (its divisions by rho0
    and the oracle's round alike: one rounding per operation)."""
    p = _nml(*ng, "PPPPNN", l=(1.0, 0.75, 1.2))
    g, o = C.Case(p), O.Case(p)
    _, f, _ = _rand_fields(p, 41)
    pp, u, v, w = (f() for _ in range(4))
    dev = [g.field(a) for a in (u, v, w)]
    g.call("correc", 0.013, g.field(pp), *dev)
    o.call("correc", 0.013, pp, u, v, w)
    for a, b in zip(dev, (u, v, w)):
        assert _rel(a.get(), b) < 1e-14
