"""Timed workloads of the framework, through its public entry points.

A case is a dict of plain values.  `kind` selects what one pass does:

  step      a whole simulation segment: set_fields from device arrays (with the
            scalar where there is one), prepare, `steps` time steps,
            get_fields back into device arrays
  ensemble  the same for a set of independent cases of uneven grids advanced
            together (cansfz_ensemble_*)
  dropin    `steps` time steps through the per-procedure entries, in the order
            in which a driver that keeps its own loop calls them
  solve     fillps + the FP64 Poisson solve + the pressure's ghost fill
  refined   the FP32 spectral solve with FP64-residual refinement sweeps

`exact` restates the same passes in plain torch in 64 bits.
"""
import ctypes as ct
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cans-fizzy_b200"))

from cansfz import case as C  # noqa: E402
from cansfz import lib as L  # noqa: E402
from cansfz import namelist, params  # noqa: E402

EPS = 2.220446049250313e-16
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(kind, nx, ny, nz, **kw):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "lx": 1.0, "ly": 1.0, "lz": 1.0, "form": "fp64",
         "capture": "acdi", "fluid": "droplets", "drops": 8, "rmin": 0.1, "rmax": 0.18, "gr": 0.0, "xwalls": False,
         "scalar": False, "opentop": False, "sweeps": -1, "steps": 8, "cases2d": 0, "cases3d": 0}
    c.update(kw)
    return c


def listed():
    return [
        # the 2-D convention (ny = 2) of the reference's own regression tests,
        # and the smallest member of the ensemble: a step is a chain of short kernels
        _case("step", 64, 2, 128, ly=2.0 / 64, lz=2.0, fluid="bubble", drops=1, name="bubble 2-D 64x2x128"),
        # the 3-D rising bubble of the parity configuration
        _case("step", 64, 64, 128, lz=2.0, fluid="bubble", drops=1, rmin=0.25, rmax=0.25, name="bubble 64x64x128"),
        # the headline workload, plain FP64 and mixed precision
        _case("step", 256, 256, 256, drops=64, rmin=0.03, rmax=0.06, name="droplets 256^3"),
        _case("step", 256, 256, 256, drops=64, rmin=0.03, rmax=0.06, form="mixed", name="droplets 256^3 mixed"),
        # the largest configuration: THINC/QQ transport
        _case("step", 512, 512, 256, lx=2.0, ly=2.0, drops=64, rmin=0.03, rmax=0.06, capture="thinc",
              name="thinc 512x512x256"),
        # dispersed wall-bounded shear flow: stretched z, lines of 512 points, mixed precision
        _case("step", 512, 256, 256, lx=2.0, drops=200, rmin=0.04, rmax=0.08, gr=1.5, fluid="shear", form="mixed",
              name="shear 512x256x256 mixed"),
        # a differentially heated cavity with walls in x (cosine transforms),
        # the scalar, the buoyancy, and sizes that fill no tile
        _case("step", 90, 50, 70, drops=3, rmin=0.15, rmax=0.2, xwalls=True, scalar=True, fluid="bubble",
              name="cavity 90x50x70 scalar"),
        # a parameter study: independent small cases of uneven grids in one graph
        _case("ensemble", 0, 0, 0, cases2d=12, cases3d=12, fluid="bubble", name="ensemble 24"),
        # a host program that keeps its own time loop and calls procedure by procedure
        _case("dropin", 48, 40, 56, steps=2, drops=4, name="procedures 48x40x56"),
        _case("dropin", 128, 128, 128, steps=2, drops=16, rmin=0.06, rmax=0.1, name="procedures 128^3"),
        # the projection's solve alone, with an open top (a well-posed system:
        # no free constant in the result), and the refined FP32 solve of the same system
        _case("solve", 256, 256, 256, opentop=True, name="poisson 256^3"),
        _case("refined", 256, 256, 256, opentop=True, sweeps=1, name="poisson 256^3 refined"),
    ]


def _smooth(n):
    for q in (2, 3, 5, 7):
        while n % q == 0:
            n //= q
    return n == 1


def _len(rng, lo, hi):
    """An even line length with factors 2, 3, 5 and 7, spread over log(lo..hi)."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    while n % 2 or not _smooth(n):
        n += 1
    return n


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["dropin", "solve", "refined", "ensemble"])
    if kind == "ensemble":
        return _case("ensemble", 0, 0, 0, cases2d=rng.randint(2, 12), cases3d=rng.randint(2, 12), fluid="bubble")
    cap = {"step": 2.4e7, "dropin": 4e6, "solve": 3e7, "refined": 2e7}[kind]
    while True:
        nx, ny = _len(rng, 24, 512), _len(rng, 24, 384)
        nz = int(math.exp(rng.uniform(math.log(20), math.log(384))))
        if rng.random() < 0.5:
            nz = max(16, nz - nz % 16)
        two_d = kind == "step" and rng.random() < 0.2
        if two_d:
            ny = 2
        if 2e4 * (0.5 if two_d else 1.0) < nx * ny * nz <= cap:
            break
    d = 1.0 / nx
    kw = {"lx": 1.0, "ly": ny * d, "lz": nz * d}
    small = min(kw["lx"], kw["lz"]) if two_d else min(kw.values())
    kw.update(rmin=0.2 * small, rmax=0.25 * small, drops=1)
    if kind == "step":
        kw["capture"] = rng.choice(["acdi", "acdi", "thinc"])
        kw["form"] = rng.choice(["fp64", "fp64", "mixed"])
        kw["fluid"] = rng.choice(["droplets", "bubble"])
        kw["xwalls"] = rng.random() < 0.25
        kw["scalar"] = rng.random() < 0.25
        kw["gr"] = rng.choice([0.0, 0.0, round(rng.uniform(0.5, 1.5), 2)])
        kw["steps"] = rng.choice([5, 8])
        if kw["form"] == "mixed" and nx * ny > 4096 and rng.random() < 0.3:
            kw["sweeps"] = 1
    elif kind == "dropin":
        kw["steps"] = rng.randint(1, 3)
        kw["capture"] = rng.choice(["acdi", "thinc"])
    else:
        kw["opentop"] = True
        if kind == "refined":
            kw["sweeps"] = rng.randint(1, 2)
    return _case(kind, nx, ny, nz, **kw)


def _members(case, seed):
    """The cases of an ensemble: grids and physics drawn from one fixed seed
    (the sizes are part of the workload), initial fields from `seed`."""
    r = random.Random(4)
    out = []
    for q in range(case["cases2d"] + case["cases3d"]):
        two = q < case["cases2d"]
        n = r.choice([64, 96, 128, 192, 256] if two else [32, 48, 64, 96])
        m = _case("step", n, 2 if two else n, 2 * n, ly=2.0 / n if two else 1.0, lz=2.0, fluid="bubble", drops=1,
                  rmin=0.125, rmax=0.25, steps=case["steps"])
        m.update(rho2=1000.0 / r.choice([10.0, 100.0, 1000.0]), mu2=10.0 / r.choice([10.0, 100.0]),
                 sigma=r.uniform(1.0, 30.0))
        out.append((m, 1000 * seed + q))
    return out


# ---------------------------------------------------------------------------
# parameters and inputs
# ---------------------------------------------------------------------------
FLUIDS = {  # rho12, mu12, sigma, gravity
    "droplets": ((1000.0, 1.0), (100.0, 1.0), 1.0, -1.0),
    "bubble": ((1000.0, 100.0), (10.0, 1.0), 24.5, -0.98),
    "shear": ((10.0, 1.0), (1.0, 1.0), 0.5, 0.0),
}


def _physics(c):
    rho, mu, sigma, grav = FLUIDS[c["fluid"]]
    rho, mu = (rho[0], c.get("rho2", rho[1])), (mu[0], c.get("mu2", mu[1]))
    return rho, mu, c.get("sigma", sigma), grav, 12.0 if c["fluid"] == "shear" else 0.0


def _params(c):
    rho, mu, sigma, grav, bf = _physics(c)
    x = ("D", "N") if c["xwalls"] else ("P", "P")  # (velocity, scalar fields)
    top = "D" if c["opentop"] else "N"
    nor = lambda comp: ", ".join(  # noqa: E731
        "'%s','%s'" % (t, t) for t in (("D" if comp == 0 else "N") if c["xwalls"] else "P", "P", "D" if comp == 2 else "N"))
    text = f"""
&dns
ng(1:3) = {c['nx']}, {c['ny']}, {c['nz']}
l(1:3) = {c['lx']!r}, {c['ly']!r}, {c['lz']!r}
gtype = 1, gr = {c['gr']!r}
cfl = 0.5, dtmax = 1.e9, dt_f = -1.
icheck = {c['steps']}
cbcvel(0:1,1:3,1) = '{x[0]}','{x[0]}', 'P','P', 'D','D'
cbcvel(0:1,1:3,2) = '{x[0]}','{x[0]}', 'P','P', 'D','D'
cbcvel(0:1,1:3,3) = '{x[0]}','{x[0]}', 'P','P', 'D','{'N' if c['opentop'] else 'D'}'
cbcpre(0:1,1:3) = '{x[1]}','{x[1]}', 'P','P', 'N','{top}'
bforce(1:3) = {bf!r}, 0., 0.
gacc(1:3) = 0., 0., {grav!r}
/
&two_fluid
cbcpsi(0:1,1:3) = '{x[1]}','{x[1]}', 'P','P', 'N','N'
cbcnor(0:1,1:3,1) = {nor(0)}
cbcnor(0:1,1:3,2) = {nor(1)}
cbcnor(0:1,1:3,3) = {nor(2)}
rho12(1:2) = {rho[0]!r}, {rho[1]!r}
mu12(1:2) = {mu[0]!r}, {mu[1]!r}
ka12(1:2) = 0.02, 0.01
cp12(1:2) = 1., 2.
beta12(1:2) = 0.01, 0.02
sigma = {sigma!r}
psi_thickness_factor = {0.5 if c['capture'] == 'thinc' else 0.51}
/
&scalar
cbcsca(0:1,1:3) = '{'D' if c['xwalls'] else 'P'}','{'D' if c['xwalls'] else 'P'}', 'P','P', 'D','D'
bcsca(0:1,1:3) = {'1., 0.' if c['xwalls'] else '0., 0.'}, 0., 0., 1., 0.
/
&cansfz
interface_capturing_vof = {'T' if c['capture'] == 'thinc' else 'F'}
scalar = {'T' if c['scalar'] else 'F'}
boussinesq_buoyancy = {'T' if c['scalar'] else 'F'}
form = '{c['form']}'
refine_sweeps = {c['sweeps']}
/
"""
    return params.from_namelist(namelist.parse(text))


class Grid:
    """Axes and metrics on the GPU: index 0..n+1 in every direction."""

    def __init__(self, c):
        self.n = (c["nx"], c["ny"], c["nz"])
        self.l = (c["lx"], c["ly"], c["lz"])
        nx, ny, nz = self.n
        self.dl = [self.l[d] / self.n[d] for d in range(3)]
        k = np.arange(1, nz + 1)
        z0 = (k.astype(np.float32) / np.float32(nz)).astype(np.float64)
        gr = c["gr"]
        z = z0 if gr == 0.0 else 0.5 * (1.0 + np.tanh((z0 - 0.5) * gr) / np.tanh(gr / 2.0))
        zf = np.concatenate([[0.0], z * self.l[2], [0.0]])
        dzf = np.zeros(nz + 2)
        dzf[1:-1] = zf[1:-1] - zf[:-2]
        dzf[0], dzf[-1] = dzf[1], dzf[-2]
        dzc = np.zeros(nz + 2)
        dzc[:-1] = 0.5 * (dzf[:-1] + dzf[1:])
        dzc[-1] = dzc[-2]
        zc = np.concatenate([[-dzc[0] / 2.0], -dzc[0] / 2.0 + np.cumsum(dzc[:-1])])
        zf = np.concatenate([[0.0], np.cumsum(dzf[1:])])
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.dzc, self.dzf, self.dzci, self.dzfi = (dev(a) for a in (dzc, dzf, 1.0 / dzc, 1.0 / dzf))
        self.zc, self.zf = dev(zc), dev(zf)
        self.dlmax, self.dlmin = max(self.dl[0], self.dl[1], dzf.max()), min(self.dl[0], self.dl[1], dzf.min())

    def axis(self, d, face):
        if d == 2:
            return self.zf if face else self.zc
        i = torch.arange(self.n[d] + 2, dtype=F64, device="cuda")
        return (i if face else i - 0.5) * self.dl[d]

    def shape(self, d, a):
        return a.view([-1 if 2 - q == d else 1 for q in range(3)])


def _droplets(c, g, rng):
    """psi (halo layout) of `drops` spheres (cylinders along y in 2-D), apart
    from each other where they can be, min over spheres of a tanh profile."""
    eps = g.dlmax * (0.5 if c["capture"] == "thinc" else 0.51)
    two_d = c["ny"] == 2
    per = (not c["xwalls"], True, False)
    ctr, out = [], None
    for _ in range(c["drops"]):
        for _try in range(2000):
            r = rng.uniform(c["rmin"], c["rmax"])
            x = [rng.uniform(0.0, g.l[d]) if per[d] else rng.uniform(min(r + 2 * eps, 0.5 * g.l[d]), max(g.l[d] - r - 2 * eps, 0.5 * g.l[d]))
                 for d in range(3)]
            gap = []
            for y, ry in ctr:
                dd = [x[d] - y[d] for d in range(3)]
                dd = [v - g.l[d] * round(v / g.l[d]) if per[d] else v for d, v in enumerate(dd)]
                if two_d:
                    dd[1] = 0.0
                gap.append(math.sqrt(sum(v * v for v in dd)) - r - ry - 4 * eps)
            if not gap or min(gap) > 0:
                break
        ctr.append((x, r))
        sq = 0.0
        for d in range(3):
            if two_d and d == 1:
                continue
            a = g.axis(d, False) - x[d]
            if per[d]:
                a = a - g.l[d] * torch.round(a / g.l[d])
            sq = sq + g.shape(d, a * a)
        phi = torch.sqrt(sq) - r
        out = phi if out is None else torch.minimum(out, phi)
    psi = 0.5 * (1.0 + torch.tanh(out / (2.0 * eps)))
    if c["fluid"] != "bubble":
        psi = 1.0 - psi
    return psi.expand(c["nz"] + 2, c["ny"] + 2, c["nx"] + 2).contiguous()


def _velocity(c, g, rng):
    """A smooth random velocity of rms ~0.1, discretely divergence-free and
    zero through the walls: the curl of a potential on the cell edges.  In 2-D
    (ny = 2) nothing depends on y and v is the third component of the flow."""
    per = (not c["xwalls"], True, False)
    two_d = c["ny"] == 2

    def potential(comp):
        # on the cell edges along `comp`: centred along comp, faces elsewhere
        acc = 0.0
        for _ in range(4):
            term = rng.gauss(0.0, 1.0)
            for d in range(3):
                s = g.axis(d, d != comp) / g.l[d]
                if two_d and d == 1:
                    continue
                k = rng.randint(1, 3)
                if per[d]:
                    f = torch.cos(2 * math.pi * k * s + rng.uniform(0, 2 * math.pi))
                else:
                    f = torch.cos(math.pi * k * s) if d == comp else torch.sin(math.pi * k * s)
                term = term * g.shape(d, f)
            acc = acc + term
        return acc.expand(c["nz"] + 2, c["ny"] + 2, c["nx"] + 2)

    def diff(a, d):  # backward difference between faces i-1 and i, over the cell size
        m = a - torch.roll(a, 1, 2 - d)
        return m * g.shape(2, g.dzfi) if d == 2 else m / g.dl[d]

    A = [potential(q) for q in range(3)]
    u, v, w = diff(A[2], 1) - diff(A[1], 2), diff(A[0], 2) - diff(A[2], 0), diff(A[1], 0) - diff(A[0], 1)
    out = [f.contiguous() for f in (u, v, w)]  # (ghost planes: filled by the step's own boundary conditions)
    rms = torch.sqrt(sum((f[1:-1, 1:-1, 1:-1] ** 2).mean() for f in out) / 3.0)
    out = [f * (0.1 / rms) for f in out]
    out[2][0] = 0.0
    out[2][-2:] = 0.0
    if c["fluid"] == "shear":
        s = g.zc / g.l[2]
        out[0] = 0.1 * out[0] + g.shape(2, 6.0 * s * (1.0 - s))
    return [f.contiguous() for f in out]


def _scalar(c, g, rng):
    s = 1.0 - g.shape(0, g.axis(0, False)) / g.l[0] if c["xwalls"] else 1.0 - g.shape(2, g.zc) / g.l[2]
    wave = torch.sin(2 * math.pi * g.shape(1, g.axis(1, False)) / g.l[1] + rng.uniform(0, 6.0)) if c["ny"] > 2 else 0.0
    s = s + 0.05 * wave * torch.sin(math.pi * g.shape(2, g.zc) / g.l[2])
    return s.expand(c["nz"] + 2, c["ny"] + 2, c["nx"] + 2).contiguous()


def _inputs(c, seed):
    """u, v, w, p, psi (and s) in the halo layout, as torch tensors [k, j, i]."""
    g, rng = Grid(c), random.Random(seed)
    f = dict(zip("uvw", _velocity(c, g, rng)))
    f["psi"] = _droplets(c, g, rng)
    f["p"] = torch.zeros_like(f["psi"])
    if c["scalar"]:
        f["s"] = _scalar(c, g, rng)
    return g, f


def _noise(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.randn((c["nz"] + 2, c["ny"] + 2, c["nx"] + 2), generator=gen, device="cuda", dtype=F64)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
NAMES = ("u", "v", "w", "p", "psi")


def _p(t):
    return ct.c_void_p(t.data_ptr())


class _Segment:
    """One case of a step or an ensemble: the context, the initial fields and
    the buffers that receive the result."""

    def __init__(self, c, seed, out=None, own_stream=False):
        _, self.f = _inputs(c, seed)
        self.case = C.Case(_params(c), own_stream=own_stream)
        # the case's own stream, for what is done to its results
        self.stream = torch.cuda.ExternalStream(self.case.lib.cansfz_stream(self.case.h))
        self.out = out or {q: torch.empty_like(self.f["u"]) for q in (NAMES + ("s",) if c["scalar"] else NAMES)}

    def start(self):
        h, f = self.case.h, self.f
        L.check(self.case.lib.cansfz_set_fields(h, *[_p(f[q]) for q in NAMES], 1))
        if "s" in f:
            L.check(self.case.lib.cansfz_set_scalar(h, _p(f["s"]), 1))
        L.check(self.case.lib.cansfz_prepare(h))

    def finish(self):
        L.check(self.case.lib.cansfz_get_fields(self.case.h, *[_p(self.out[q]) for q in NAMES], 1))
        if "s" in self.f:
            L.check(self.case.lib.cansfz_get_aux(self.case.h, b"s", _p(self.out["s"]), 1))
        # the pressure is defined up to a constant (Neumann and periodic boundaries)
        p = self.out["p"]
        with torch.cuda.stream(self.stream):
            p.sub_(p[1:-1, 1:-1, 1:-1].mean())


class _Procedures:
    """A time loop of the caller's own over the per-procedure entries."""

    def __init__(self, c, seed):
        _, self.f0 = _inputs(c, seed)
        self.stream = torch.cuda.Stream()
        self.stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(self.stream):
            self.case = C.Case(_params(c))
        self.thinc = c["capture"] == "thinc"
        self.steps = c["steps"]
        z = lambda: torch.zeros_like(self.f0["u"])  # noqa: E731
        self.f = {q: z() for q in NAMES + ("psio", "po", "pp", "phi", "kappa", "nx", "ny", "nz", "fx", "fy", "fz")}
        g = Grid(c)
        self.seps = g.dlmax * (0.5 if self.thinc else 0.51)
        self.beta = 1.0
        torch.cuda.synchronize()

    def run(self):
        lib, h, f = self.case.lib, self.case.h, {k: _p(t) for k, t in self.f.items()}
        call = lambda name, *a: L.check(getattr(lib, "cansfz_" + name)(h, *a), name)  # noqa: E731

        def normals():
            call("boundp", 1, f["psi"])
            if self.thinc:
                call("vof_thinc_cmpt_phi", self.beta, f["psi"], f["phi"])
            else:
                call("acdi_cmpt_phi", self.seps, f["psi"], f["phi"])
            call("cmpt_norm_curv_youngs", f["phi"], f["nx"], f["ny"], f["nz"], f["kappa"])
            for which, q in ((2, "kappa"), (3, "nx"), (4, "ny"), (5, "nz")):
                call("boundp", which, f[q])

        def gamma():
            out = ct.c_double()
            call("acdi_set_gamma", 1.0, f["u"], f["v"], f["w"], out)
            return max(out.value, 1e-12)

        with torch.cuda.stream(self.stream):
            for q in NAMES:
                self.f[q].copy_(self.f0[q])
            call("bounduvw", 0, f["u"], f["v"], f["w"])
            call("boundp", 0, f["p"])
            self.f["po"].copy_(self.f["p"])
            normals()
            gam = 0.0 if self.thinc else gamma()
            dtmax, div = ct.c_double(), (ct.c_double(), ct.c_double())
            call("chkdt", f["u"], f["v"], f["w"], gam, self.seps, dtmax)
            dt = 0.5 * dtmax.value
            rk, rho_av = (ct.c_double * 2)(1.5, -0.5), (ct.c_double * 3)(0.0, 0.0, 0.0)
            for _ in range(self.steps):
                self.f["psio"].copy_(self.f["psi"])
                call("rk_2fl", rk, dt, gam, self.seps, self.beta, f["u"], f["v"], f["w"], f["nx"], f["ny"], f["nz"],
                     f["phi"], f["psi"], f["fx"], f["fy"], f["fz"])
                call("bounduvw", 0, f["fx"], f["fy"], f["fz"])
                normals()
                call("rk", rk, dt, 1.0, rho_av, f["psi"], f["kappa"], f["p"], f["p"], f["po"], None, f["psio"], f["fx"],
                     f["fy"], f["fz"], f["u"], f["v"], f["w"])
                call("bounduvw", 0, f["u"], f["v"], f["w"])
                call("fillps", 1.0 / dt, f["u"], f["v"], f["w"], f["pp"])
                call("updt_rhs_b", f["pp"])
                call("solver", f["pp"])
                call("boundp", 0, f["pp"])
                call("correc", dt, f["pp"], f["u"], f["v"], f["w"])
                call("bounduvw", 1, f["u"], f["v"], f["w"])
                self.f["po"].copy_(self.f["p"])
                call("updatep", f["pp"], f["p"])
                call("boundp", 0, f["p"])
                if not self.thinc:
                    gam = gamma()
            call("chkdt", f["u"], f["v"], f["w"], gam, self.seps, dtmax)
            call("chkdiv", f["u"], f["v"], f["w"], *div)
            p = self.f["p"]
            p.sub_(p[1:-1, 1:-1, 1:-1].mean())
        return {**{q: self.f[q] for q in NAMES}, "dtmax": np.array(dtmax.value)}


class _Solve:
    def __init__(self, c, seed):
        self.stream = torch.cuda.Stream()
        with torch.cuda.stream(self.stream):
            self.case = C.Case(_params(c))
            if c["kind"] == "solve":
                self.vel = [_noise(c, seed + q) for q in range(3)]
            else:
                self.rhs = _noise(c, seed)
            self.p = torch.zeros_like(_noise(c, seed))
        self.refined, self.sweeps = c["kind"] == "refined", c["sweeps"]
        torch.cuda.synchronize()

    def run(self):
        lib, h = self.case.lib, self.case.h
        if self.refined:
            L.check(lib.cansfz_solver_refined(h, _p(self.rhs), _p(self.p), self.sweeps))
        else:
            L.check(lib.cansfz_fillps(h, 100.0, *[_p(q) for q in self.vel], _p(self.p)))
            L.check(lib.cansfz_solver(h, _p(self.p)))
            L.check(lib.cansfz_boundp(h, 0, _p(self.p)))
        return self.p


class _Ensemble:
    def __init__(self, c, seed):
        members = _members(c, seed)
        sizes = [(m["nx"] + 2) * (m["ny"] + 2) * (m["nz"] + 2) for m, _ in members]
        self.out = {q: torch.zeros(sum(sizes), dtype=F64, device="cuda") for q in NAMES}
        self.segs, at = [], 0
        for (m, s), size in zip(members, sizes):
            shape = (m["nz"] + 2, m["ny"] + 2, m["nx"] + 2)
            view = {q: self.out[q][at:at + size].view(shape) for q in NAMES}
            self.segs.append(_Segment(m, s, out=view, own_stream=True))
            at += size
        torch.cuda.synchronize()
        for s in self.segs:
            s.start()
        self.ens = C.Ensemble([s.case for s in self.segs])

    def __del__(self):
        self.ens.close()  # before its cases


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        s = _Segment(case, seed)
    elif kind == "ensemble":
        s = _Ensemble(case, seed)
    elif kind == "dropin":
        s = _Procedures(case, seed)
    else:
        s = _Solve(case, seed)
    return {"kind": kind, "steps": case["steps"], "state": s}


def run(state):
    s, kind = state["state"], state["kind"]
    if kind == "step":
        s.start()
        L.check(s.case.step(state["steps"]), "step")
        s.finish()
        return s.out
    if kind == "ensemble":
        for q in s.segs:
            q.start()
        L.check(s.ens.step(state["steps"])[0], "ensemble step")
        for q in s.segs:
            q.finish()
        return s.out
    return s.run()


# ---------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: per time step 19 accesses of the state and 10 of the Poisson
    passes (each field of a step read or written once per use that a global
    solve separates), and the fields in and out of a segment; per procedure
    each argument once."""
    if case["kind"] == "ensemble":
        w = [work(m) for m, _ in _members(case, 0)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    cells = float(case["nx"] * case["ny"] * case["nz"])
    fft = 2.5 * 2 * (math.log2(max(case["nx"], 2)) + math.log2(max(case["ny"], 2)))
    steps = case["steps"]
    if case["kind"] == "step":
        per = 232.0 - (32.0 if case["form"] == "mixed" else 0.0) + (32.0 if case["scalar"] else 0.0)
        return {"bytes": cells * (steps * per + 80.0), "flops": cells * steps * (900.0 + fft)}
    if case["kind"] == "dropin":
        return {"bytes": cells * (steps * 576.0 + 80.0), "flops": cells * steps * (900.0 + fft)}
    if case["kind"] == "solve":
        return {"bytes": cells * (32.0 + 10 * 8.0), "flops": cells * (20.0 + fft)}
    return {"bytes": cells * (16.0 + case["sweeps"] * 24.0), "flops": cells * (1 + case["sweeps"]) * (20.0 + fft)}


def tolerance(case):
    """About four times the largest error against `exact`, and the largest
    difference between the solve's two line and two z algorithms, seen over
    listed and drawn cases.  FP64 steps: p, defined against the constant of the
    singular mode, 4e-11, the other fields below 1e-12.  The mixed form stores
    its intermediates in 32 bits (p 2e-8, a cell's velocity 5e-7).  A refinement
    sweep takes the FP32 solve's error from 5e-5 to 1e-8 and then 1e-10."""
    if case["kind"] == "solve":
        return {"rel": 2e-12, "max": 1e-11}
    if case["kind"] == "refined":
        return {"rel": 1e-7, "max": 1e-6} if case["sweeps"] == 1 else {"rel": 2e-9, "max": 2e-8}
    if case["kind"] == "dropin":
        return {"rel": 1e-11, "max": 1e-10}
    return {"rel": 2e-10, "max": 1e-9} if case["form"] == "fp64" else {"rel": 1e-7, "max": 2e-6}


# ---------------------------------------------------------------------------
# the same passes in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    def __init__(self, c, seed):
        self.c = c
        self.g, f = _inputs(c, seed)
        self.f = f
        self.rho, self.mu, self.sigma, self.grav, self.bf = _physics(c)
        self.per = (not c["xwalls"], True, False)
        self.seps = self.g.dlmax * (0.5 if c["capture"] == "thinc" else 0.51)
        self.thinc = c["capture"] == "thinc"
        self.first = True
        n = self.g.n
        self.basis = [self.modes(d) for d in range(2)]
        g = self.g
        self.za, self.zcc = g.dzfi[1:-1] * g.dzci[:-2], g.dzfi[1:-1] * g.dzci[1:-1]
        self.zb = -(self.za + self.zcc)
        self.zb[0] += self.za[0]
        self.zb[-1] += (-1.0 if c["opentop"] else 1.0) * self.zcc[-1]
        self.n = n

    # interior shifted by (a, b, c) cells along x, y, z
    @staticmethod
    def at(f, a=0, b=0, c=0):
        q = f.shape
        return f[1 + c:q[0] - 1 + c, 1 + b:q[1] - 1 + b, 1 + a:q[2] - 1 + a]

    def z(self, m, off=0):
        return m[1 + off:m.numel() - 1 + off].view(-1, 1, 1)

    # ghost fills -----------------------------------------------------------
    @staticmethod
    def line(f, d, i):
        return f.select(2 - d, i)

    def fill(self, f, rules, values=None):
        """Cell-centred ghosts: 'P', 'N' (zero gradient) or 'D' (value)."""
        for d in range(3):
            n = self.g.n[d]
            if rules[d][0] == "P":
                self.line(f, d, 0).copy_(self.line(f, d, n))
                self.line(f, d, n + 1).copy_(self.line(f, d, 1))
                continue
            for side, (gh, inn) in enumerate(((0, 1), (n + 1, n))):
                if rules[d][side] == "N":
                    self.line(f, d, gh).copy_(self.line(f, d, inn))
                else:
                    v = values[d][side] if values else 0.0
                    self.line(f, d, gh).copy_(2.0 * v - self.line(f, d, inn))

    def scalar_rules(self, wall="N"):
        return [("P", "P") if p else (wall, wall) for p in self.per]

    def fill_normal(self, f, comp):
        self.fill(f, [("P", "P") if p else (("D", "D") if d == comp else ("N", "N")) for d, p in enumerate(self.per)])

    def fill_vel(self, vel, correc=False):
        for q, f in enumerate(vel):
            for d in range(3):
                n = self.g.n[d]
                if self.per[d]:
                    self.line(f, d, 0).copy_(self.line(f, d, n))
                    self.line(f, d, n + 1).copy_(self.line(f, d, 1))
                elif d != q:
                    self.line(f, d, 0).copy_(-self.line(f, d, 1))
                    self.line(f, d, n + 1).copy_(-self.line(f, d, n))
                elif not correc:
                    self.line(f, d, 0).zero_()
                    self.line(f, d, n + 1).copy_(self.line(f, d, n - 1))
                    self.line(f, d, n).zero_()

    # phase field -----------------------------------------------------------
    def phi(self, psi):
        if self.thinc:
            q = psi.clamp(EPS, 1.0 - EPS)
            return 0.5 * torch.log(q / (1.0 - q))
        return self.seps * torch.log((psi + EPS) / (1.0 - psi + EPS))

    def youngs(self, phi):
        g = self.g
        lo = lambda a, d: a.narrow(2 - d, 0, a.shape[2 - d] - 1)  # noqa: E731
        hi = lambda a, d: a.narrow(2 - d, 1, a.shape[2 - d] - 1)  # noqa: E731
        dif = lambda a, d: hi(a, d) - lo(a, d)  # noqa: E731
        add = lambda a, d: hi(a, d) + lo(a, d)  # noqa: E731
        m = [0.25 * add(add(dif(phi, 0), 1), 2) / g.dl[0], 0.25 * add(add(dif(phi, 1), 0), 2) / g.dl[1],
             0.25 * add(add(dif(phi, 2), 0), 1) * g.dzci[:-1].view(-1, 1, 1)]
        norm = torch.sqrt(m[0] ** 2 + m[1] ** 2 + m[2] ** 2) + EPS
        m = [q / norm for q in m]
        nor = [0.125 * add(add(add(q, 0), 1), 2) for q in m]
        size = torch.sqrt(nor[0] ** 2 + nor[1] ** 2 + nor[2] ** 2) + EPS
        kap = -0.25 * (add(add(dif(m[0], 0), 1), 2) / g.dl[0] + add(add(dif(m[1], 1), 0), 2) / g.dl[1] +
                       add(add(dif(m[2], 2), 0), 1) * self.z(g.dzfi))
        out = []
        for q in nor + [kap]:
            f = torch.zeros_like(phi)
            self.at(f).copy_(q / size if q is not kap else q)
            out.append(f)
        for q in range(3):
            self.fill_normal(out[q], q)
        self.fill(out[3], self.scalar_rules())
        return out[:3], out[3]

    def interface(self):
        self.fill(self.f["psi"], self.scalar_rules())
        self.ph = self.phi(self.f["psi"])
        self.nor, self.kap = self.youngs(self.ph)

    def transport(self, gam):
        """Face fluxes (halo arrays, +face of each cell) and d(psi)/dt."""
        g, psi = self.g, self.f["psi"]
        fl, rate = [], 0.0
        for d, vel in enumerate((self.f["u"], self.f["v"], self.f["w"])):
            def cut(a, off):  # cells i (off 0) or i+1 (off 1) of the faces i = 0..n along d, interior across
                q = [slice(1, -1)] * 3
                q[2 - d] = slice(off, a.shape[2 - d] - 1 + off)
                return a[tuple(q)]
            uf = cut(vel, 0)
            if self.thinc:
                pos = uf > 0.0
                nn = torch.where(pos, cut(self.nor[d], 0), cut(self.nor[d], 1))
                dd = torch.where(pos, cut(self.ph, 0), cut(self.ph, 1))
                flux = uf / (1.0 + torch.exp(-2.0 * (nn * torch.where(pos, 0.5, -0.5) + dd)))
            else:
                dli = g.dzci[:-1].view(-1, 1, 1) if d == 2 else 1.0 / g.dl[d]
                nf = [0.5 * (cut(q, 0) + cut(q, 1)) for q in self.nor]
                rn = nf[d] / (torch.sqrt(nf[0] ** 2 + nf[1] ** 2 + nf[2] ** 2) + EPS)
                sharp = 0.25 * gam * (1.0 - torch.tanh(0.25 * (cut(self.ph, 0) + cut(self.ph, 1)) / self.seps) ** 2) * rn
                flux = 0.5 * (cut(psi, 0) + cut(psi, 1)) * uf - (gam * self.seps * (cut(psi, 1) - cut(psi, 0)) * dli - sharp)
            n = g.n[d]
            dv = flux.narrow(2 - d, 1, n) - flux.narrow(2 - d, 0, n)
            rate = rate - (dv * self.z(g.dzfi) if d == 2 else dv / g.dl[d])
            f = torch.zeros_like(psi)
            self.at(f).copy_(flux.narrow(2 - d, 1, n))
            fl.append(f)
        self.fill_vel(fl)
        return fl, rate

    # momentum --------------------------------------------------------------
    def momentum_rate(self, fl):
        """Advection and diffusion of the staggered velocity (one expression
        per pair of component q and direction d)."""
        g, at = self.g, self.at
        vel, psi = (self.f["u"], self.f["v"], self.f["w"]), self.f["psi"]
        rho, drho = self.rho[1], self.rho[0] - self.rho[1]
        mu, dmu = self.mu[1], self.mu[0] - self.mu[1]
        mass = [rho * v + drho * x for v, x in zip(vel, fl)]
        e = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
        sh = lambda f, *ws: at(f, *[sum(w[i] for w in ws) for i in range(3)])  # noqa: E731
        neg = lambda w: tuple(-x for x in w)  # noqa: E731
        o = (0, 0, 0)
        out = []
        for q in range(3):
            acc = 0.0
            for d in range(3):
                # spacings: dq along the component's own axis, dd of the difference between faces
                for s, side in ((1.0, o), (-1.0, neg(e[d]))):
                    if d == q:
                        flux = 0.25 * (sh(mass[d], side) + sh(mass[d], side, e[d])) * (sh(vel[q], side) + sh(vel[q], side, e[d]))
                        hi = 1.0 / g.dl[d] if d < 2 else self.z(g.dzfi, 1 if side == o else 0)
                        str_ = 2.0 * (sh(vel[q], side, e[d]) - sh(vel[q], side)) * hi
                        m = mu + dmu * sh(psi, side, e[d])
                    else:
                        flux = 0.25 * (sh(mass[d], side) + sh(mass[d], side, e[q])) * (sh(vel[q], side) + sh(vel[q], side, e[d]))
                        hd = 1.0 / g.dl[d] if d < 2 else self.z(g.dzci, 0 if side == o else -1)
                        hq = 1.0 / g.dl[q] if q < 2 else self.z(g.dzci)
                        str_ = (sh(vel[q], side, e[d]) - sh(vel[q], side)) * hd + (sh(vel[d], side, e[q]) - sh(vel[d], side)) * hq
                        m = mu + dmu * 0.25 * (sh(psi, side) + sh(psi, side, e[d]) + sh(psi, side, e[q]) + sh(psi, side, e[d], e[q]))
                    last = 1.0 / g.dl[d] if d < 2 else (self.z(g.dzci) if q == 2 else self.z(g.dzfi))
                    acc = acc + s * last * (-flux + str_ * m)
            out.append(acc)
        return out

    def others(self, q, ratio):
        g, at, psi = self.g, self.at, self.f["psi"]
        e = [(1, 0, 0), (0, 1, 0), (0, 0, 1)][q]
        h = 1.0 / g.dl[q] if q < 2 else self.z(g.dzci)
        rho0 = min(self.rho)
        half = 0.5 * (at(psi, *e) + at(psi))
        rho = self.rho[1] + (self.rho[0] - self.rho[1]) * half
        r = (self.bf if q == 0 else 0.0) + (rho * self.grav if q == 2 else 0.0)
        r = r + 0.5 * (at(self.kap, *e) + at(self.kap)) * self.sigma * 2.0 / sum(self.rho) * rho * (at(psi, *e) - at(psi)) * h
        p, po = self.f["p"], self.po
        dp = (at(p, *e) - at(p)) * h
        dpe = (1.0 + ratio) * dp - ratio * (at(po, *e) - at(po)) * h
        r = r - (dpe + rho / rho0 * (dp - dpe))
        if self.c["scalar"] and q == 2:
            b = self.rho[1] * 0.02 + (self.rho[0] * 0.01 - self.rho[1] * 0.02) * half
            r = r - self.grav * b * 0.5 * (at(self.f["s"], *e) + at(self.f["s"]))
        return r, rho

    def scalar_rate(self, fl, psi):
        g, at, s = self.g, self.at, self.f["s"]
        cp = (self.rho[0] * 1.0, self.rho[1] * 2.0)
        acc = 0.0
        for d, v in enumerate((self.f["u"], self.f["v"], self.f["w"])):
            e = [(1, 0, 0), (0, 1, 0), (0, 0, 1)][d]
            m = cp[1] * v + (cp[0] - cp[1]) * fl[d]
            for sg, o in ((1.0, (0, 0, 0)), (-1.0, tuple(-x for x in e))):
                nx = tuple(a + b for a, b in zip(o, e))
                h = 1.0 / g.dl[d] if d < 2 else self.z(g.dzci, 0 if sg > 0 else -1)
                ka = 0.01 + 0.01 * 0.5 * (at(psi, *nx) + at(psi, *o))
                flux = -0.5 * at(m, *o) * (at(s, *nx) + at(s, *o)) + ka * (at(s, *nx) - at(s, *o)) * h
                acc = acc + sg * flux * (1.0 / g.dl[d] if d < 2 else self.z(g.dzfi))
        return acc, cp

    # projection ------------------------------------------------------------
    def modes(self, d):
        """Eigenvalues and orthonormal eigenvectors of the second difference."""
        n = self.g.n[d]
        m = torch.zeros(n, n, dtype=F64)
        i = torch.arange(n)
        m[i, i] = -2.0
        m[i[:-1], i[1:]] += 1.0
        m[i[1:], i[:-1]] += 1.0
        if self.per[d]:
            m[0, n - 1] += 1.0
            m[n - 1, 0] += 1.0
        else:
            m[0, 0] += 1.0
            m[n - 1, n - 1] += 1.0
        lam, v = torch.linalg.eigh(m)
        return lam.cuda() / self.g.dl[d] ** 2, v.cuda()

    def poisson(self, rhs):
        """The interior solution of the 7-point Laplacian."""
        (lx, vx), (ly, vy) = self.basis
        h = torch.matmul(rhs, vx)
        h = torch.matmul(vy.T, h)
        lam = ly.view(-1, 1) + lx.view(1, -1)
        n = h.shape[0]
        a, b, c = self.za.tolist(), self.zb.tolist(), self.zcc.tolist()
        small = 1e-9 * float(lam.abs().max())
        zero = (lam.abs() < small) if not self.c["opentop"] else torch.zeros_like(lam, dtype=torch.bool)
        lam = torch.where(lam.abs() < small, torch.zeros_like(lam), lam)
        cp = torch.empty_like(h)
        for k in range(n):
            den = b[k] + lam if k == 0 else b[k] + lam - a[k] * cp[k - 1]
            if k == n - 1:
                den = torch.where(zero, torch.full_like(den, math.inf), den)
            cp[k] = c[k] / den
            h[k] = (h[k] if k == 0 else h[k] - a[k] * h[k - 1]) / den
        for k in range(n - 2, -1, -1):
            h[k] -= cp[k] * h[k + 1]
        return torch.matmul(vy, torch.matmul(h, vx.T))

    def divergence(self, vel):
        g, at, (u, v, w) = self.g, self.at, vel
        return (at(w) - at(w, 0, 0, -1)) * self.z(g.dzfi) + (at(v) - at(v, 0, -1)) / g.dl[1] + (at(u) - at(u, -1)) / g.dl[0]

    def pressure_rules(self):
        return [("P", "P") if p else ("N", "D" if d == 2 and self.c["opentop"] else "N") for d, p in enumerate(self.per)]

    # limits ----------------------------------------------------------------
    def gamma(self):
        at = self.at
        u, v, w = self.f["u"], self.f["v"], self.f["w"]
        q = (0.5 * (at(u) + at(u, -1))) ** 2 + (0.5 * (at(v) + at(v, 0, -1))) ** 2 + (0.5 * (at(w) + at(w, 0, 0, -1))) ** 2
        return max(math.sqrt(float(q.max())), float(np.float32(1e-12)))

    def dtmax(self, gam):
        g, at = self.g, self.at
        vel = (self.f["u"], self.f["v"], self.f["w"])
        e = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
        dti = 0.0
        for q in range(3):
            acc = 0.0
            for d in range(3):
                if d == q:
                    s = at(vel[d]).abs()
                else:
                    m = tuple(-x for x in e[d])
                    s = 0.25 * (at(vel[d]) + at(vel[d], *m) + at(vel[d], *e[q]) + at(vel[d], *[a + b for a, b in zip(m, e[q])])).abs()
                acc = acc + (s / g.dl[d] if d < 2 else s * self.z(g.dzci if q == 2 else g.dzfi))
            dti = max(dti, float(acc.max()))
        dl2 = g.dlmin ** 2
        visc = max(self.mu[0] / self.rho[0], self.mu[1] / self.rho[1]) * 6.0 / dl2
        cap = self.sigma / min(self.rho) / g.dlmin ** 3
        t = 0.5 * (dti + visc + math.sqrt((dti + visc) ** 2 + 4.0 * ((self.grav / g.dlmin) ** 2 + cap)))
        out = min(1.0 / t, 1.0 / (dti if self.thinc else gam * self.seps / dl2))
        if self.c["scalar"]:
            out = min(out, dl2 / max(0.02 / self.rho[0], 0.01 / (2.0 * self.rho[1])))
        return out

    # the time loop ---------------------------------------------------------
    def segment(self, steps, check):
        f, at = self.f, self.at
        self.fill_vel([f["u"], f["v"], f["w"]])
        self.fill(f["p"], self.pressure_rules())
        self.po = f["p"].clone()
        srules = [("P", "P") if p else ("D", "D") for p in self.per]
        sval = [(1.0, 0.0) if self.c["xwalls"] else (0.0, 0.0), (0.0, 0.0), (1.0, 0.0)]
        if self.c["scalar"]:
            self.fill(f["s"], srules, sval)
        self.interface()
        gam = 0.0 if self.thinc else self.gamma()
        dt = 0.5 * self.dtmax(gam)
        old = {}

        def ab2(name, r):
            prev = old.get(name, r)
            old[name] = r
            return dt * (1.5 * r - 0.5 * prev)

        for it in range(1, steps + 1):
            psio = f["psi"].clone()
            fl, rate = self.transport(gam)
            at(f["psi"]).copy_((at(psio) + ab2("psi", rate)).clamp(0.0, 1.0))
            self.interface()
            if self.c["scalar"]:
                r, cp = self.scalar_rate(fl, f["psi"])
                new, was = (cp[1] + (cp[0] - cp[1]) * at(q) for q in (f["psi"], psio))
                at(f["s"]).copy_((at(f["s"]) * was + ab2("s", r)) / new)
                self.fill(f["s"], srules, sval)
            rates = self.momentum_rate(fl)
            for q, name in enumerate("uvw"):
                e = [(1, 0, 0), (0, 1, 0), (0, 0, 1)][q]
                force, rho = self.others(q, 1.0)
                was = self.rho[1] + (self.rho[0] - self.rho[1]) * 0.5 * (at(psio, *e) + at(psio))
                at(f[name]).copy_((at(f[name]) * was + ab2(name, rates[q]) + dt * force) / rho)
            vel = [f["u"], f["v"], f["w"]]
            self.fill_vel(vel)
            pp = torch.zeros_like(f["p"])
            rho0 = min(self.rho)
            at(pp).copy_(self.poisson(rho0 / dt * self.divergence(vel)))
            self.fill(pp, self.pressure_rules())
            g = self.g
            f["u"][:, :, :-1] -= dt / rho0 * (pp[:, :, 1:] - pp[:, :, :-1]) / g.dl[0]
            f["v"][:, :-1] -= dt / rho0 * (pp[:, 1:] - pp[:, :-1]) / g.dl[1]
            f["w"][:-1] -= dt / rho0 * (pp[1:] - pp[:-1]) * g.dzci[:-1].view(-1, 1, 1)
            self.fill_vel(vel, correc=True)
            self.po = f["p"]
            f["p"] = self.po + pp
            self.fill(f["p"], self.pressure_rules())
            if not self.thinc:
                gam = self.gamma()
            if check and it == steps:
                dt = 0.5 * self.dtmax(gam)
        f["p"] -= at(f["p"]).mean()
        self.gam = gam
        return {q: f[q] for q in (NAMES + ("s",) if self.c["scalar"] else NAMES)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _Exact(case, seed).segment(case["steps"], True)
    if kind == "ensemble":
        got = [_Exact(m, s).segment(case["steps"], True) for m, s in _members(case, seed)]
        return {q: torch.cat([x[q].reshape(-1) for x in got]) for q in NAMES}
    if kind == "dropin":
        e = _Exact(case, seed)
        got = e.segment(case["steps"], False)
        return {**got, "dtmax": np.array(e.dtmax(e.gam))}
    e = _Exact(case, seed)
    if kind == "solve":
        rhs = min(e.rho) * 100.0 * e.divergence([_noise(case, seed + q) for q in range(3)])
    else:
        rhs = e.at(_noise(case, seed))
    p = torch.zeros_like(e.f["p"])
    e.at(p).copy_(e.poisson(rhs))
    e.fill(p, e.pressure_rules())
    return p
