"""The Poisson solve at the edges of its kernels' size ranges: the partitioned
z solve's chunks (shortest and longest columns, columns that the chunks do not
divide, a last tile of few columns, FP64 and FP32), thin domains, whose lowest
modes are the worst conditioned, and the two-pass transforms of 512 points
with a partial tile of lines.

The reference is the same discrete system (the eigenvalues and z coefficients
that the solver holds) solved in extended precision (64-bit significands).

Bounds, relative to the largest value of the solution.  Partitioned columns of
24 to 512 levels: each of the four transform passes rounds log2(n) <= 9 times,
a column's solve a few times per chunk: about 50 roundings of 1.1e-16, random in
sign, and the largest of up to 1e6 values 5 times their deviation: 1e-14.  One
column per thread (other lengths, and short columns of large grids): gaussel's order, whose pivots round
against a condition of (2 nz/pi)^2.  Column 0 of a problem without a Dirichlet
wall is singular and its constant is fixed by the rounded last pivot in
gaussel's order, as the oracle's: compared with the oracle apart.
"""
import math

import numpy as np
import pytest

import oracle as O
from cansfz import case as C

from test_gpu_parity import _nml

pytestmark = pytest.mark.gpu

EPS = 2.0**-53
L = np.longdouble

SHAPES = [
    # chunks: 24 levels is the first column the 8 chunks hold, 23 the last they do not
    ("PPPPNN", (12, 10, 23)), ("PPPPNN", (12, 10, 24)), ("PPPPNN", (12, 10, 25)), ("PPPPDD", (20, 6, 31)),
    ("PPPPNN", (64, 2, 65)), ("NNPPNN", (30, 14, 97)), ("PPPPNN", (16, 12, 128)), ("PPPPDD", (10, 10, 255)),
    # 16 chunks from 257 levels to 512, one column per thread beyond
    ("PPPPNN", (12, 10, 257)), ("PPPPNN", (16, 4, 384)), ("PPPPNN", (10, 6, 500)), ("DDNNDD", (12, 10, 512)),
    ("PPPPNN", (12, 10, 513)),
    # lines of 512 points in x and y, few lines and partial tiles
    ("PPPPNN", (512, 6, 9)), ("PPPPDD", (512, 10, 7)), ("NNPPNN", (6, 512, 10)), ("PPPPNN", (20, 512, 3)),
    ("PPPPNN", (512, 512, 4)),
    # both sides of the rule by which short columns of large grids go to the column solves
    ("PPPPNN", (128, 128, 40)), ("PPPPNN", (160, 128, 40)), ("PPPPNN", (160, 128, 52)), ("PPPPNN", (200, 196, 26)),
    ("PPPPNN", (256, 160, 26)), ("PPPPNN", (256, 160, 63)), ("PPPPNN", (256, 160, 64)),
]
# cubic cells, so that lambda*lz^2 of the lowest modes is small
THIN = [("PPPPNN", (512, 8, 24)), ("PPPPND", (512, 8, 24)), ("PPPPNN", (384, 8, 48)), ("PPPPND", (256, 8, 64)),
        ("PPPPNN", (128, 32, 100)), ("PPPPDD", (256, 8, 64))]


# ---------------------------------------------------------------------------
# the system in extended precision
# ---------------------------------------------------------------------------
def _kind(bc):
    return {"PP": 0, "NN": 1, "DD": 2}[bc]


def _lambda(n, kind, dl):
    """src/initsolver.f90:81-139, in the order of `_transform`."""
    if kind == 0:
        arg = [2.0 * m * math.pi / n for m in range(n // 2 + 1)] + [2.0 * (n - k) * math.pi / n for k in range(1, n // 2)]
    else:
        arg = [(m + (kind == 2)) * math.pi / n for m in range(n)]
    d = 1.0 / dl
    return np.array([-2.0 * (1.0 - math.cos(a)) * (d * d) for a in arg])


def _wall_basis(n, kind):
    """Orthonormal rows: the cosines of Neumann walls, the sines of Dirichlet walls."""
    pi, i = 4 * np.arctan(L(1)), np.arange(n)
    a = pi / (2 * n) * (((2 * i + 1) * (i[:, None] + (kind == 2))) % (4 * n))
    v = np.cos(a) if kind == 1 else np.sin(a)
    return v / np.sqrt((v * v).sum(axis=1, keepdims=True))


def _transform(f, axis, kind):
    """Along one axis: the cosine and then the sine coefficients of a periodic
    line, or those of the walls."""
    f = np.moveaxis(f, axis, 0)
    n = f.shape[0]
    if kind == 0:
        h = np.fft.rfft(f, axis=0)
        assert h.dtype == np.clongdouble
        h = np.concatenate([h.real, h.imag[1:n // 2]])
    else:
        h = np.tensordot(_wall_basis(n, kind), f, axes=1)
    return np.moveaxis(h, 0, axis)


def _inverse(h, axis, kind):
    h = np.moveaxis(h, axis, 0)
    n = h.shape[0]
    if kind == 0:
        c = np.zeros((n // 2 + 1,) + h.shape[1:], np.clongdouble)
        c.real = h[:n // 2 + 1]
        c.imag[1:n // 2] = h[n // 2 + 1:]
        f = np.fft.irfft(c, n, axis=0)
    else:
        f = np.tensordot(_wall_basis(n, kind).T, h, axes=1)
    return np.moveaxis(f, 0, axis)


def _exact(p, g, rhs, keep0=True):
    """The solution of the stored system; keep0: with column 0 (of a problem
    with a Dirichlet wall), else without it."""
    bc = [bytes(p.cbcpre[2 * d:2 * d + 2]).decode() for d in range(3)]
    n = list(p.ng)
    dl = [p.l[d] / n[d] for d in range(2)]
    kx, ky = _kind(bc[0]), _kind(bc[1])
    lam = _lambda(n[0], kx, dl[0])[:, None] + _lambda(n[1], ky, dl[1])
    dzci, dzfi = g["dzci"], g["dzfi"]
    a, c = dzfi[1:-1] * dzci[:-2], dzfi[1:-1] * dzci[1:-1]
    b = -(a + c)
    b[0] += a[0] * (-1.0 if bc[2][0] == "D" else 1.0)
    b[-1] += c[-1] * (-1.0 if bc[2][1] == "D" else 1.0)
    a, b, c, lam = (x.astype(L) for x in (a, b, c, lam))
    h = _transform(_transform(rhs.astype(L), 0, kx), 1, ky)
    if not keep0:
        h[0, 0] = 0
        lam[0, 0] = -1
    d = np.zeros_like(h)
    d[:, :, 0] = c[0] / (b[0] + lam)
    h[:, :, 0] /= b[0] + lam
    for k in range(1, n[2]):
        z = 1 / (b[k] + lam - a[k] * d[:, :, k - 1])
        d[:, :, k] = c[k] * z
        h[:, :, k] = (h[:, :, k] - a[k] * h[:, :, k - 1]) * z
    for k in range(n[2] - 2, -1, -1):
        h[:, :, k] -= d[:, :, k] * h[:, :, k + 1]
    return _inverse(_inverse(h, 1, ky), 0, kx)


def _case(cbcpre, ng, thin=False):
    p = _nml(*ng, cbcpre, l=tuple(n / 512.0 for n in ng) if thin else (1.0, 0.75, 1.2))
    rhs = np.zeros(tuple(n + 2 for n in ng), order="F")
    rhs[1:-1, 1:-1, 1:-1] = np.random.default_rng(5).standard_normal(p.n)
    return p, rhs


def _partitioned(ng):
    """The columns that the partitioned solve takes in FP64."""
    ncol, nz = ng[0] * ng[1], ng[2]
    if not 24 <= nz <= 512 or ncol % 4:
        return False
    return nz >= 64 or ncol <= 16384 or (nz >= 52 if ncol < 32768 else ncol <= 40000)


def _bound(ng):
    return 1e-14 if _partitioned(ng) else 4 * EPS * (2 * ng[2] / math.pi) ** 2 + 1e-14


def _well_posed(cbcpre):
    return cbcpre if "D" in cbcpre else cbcpre[:5] + "D"


# ---------------------------------------------------------------------------
@pytest.mark.parametrize("cbcpre,ng,thin", [(*s, False) for s in SHAPES] + [(*s, True) for s in THIN])
def test_solver(cbcpre, ng, thin):
    """With a Dirichlet wall (the top's where the shape has none): every mode,
    column 0 included, against the extended-precision solution."""
    p, rhs = _case(_well_posed(cbcpre), ng, thin)
    g = C.Case(p)
    pg = g.field(rhs)
    g.call("solver", pg)
    ref = _exact(p, g.grid(), rhs[1:-1, 1:-1, 1:-1])
    assert np.abs(pg.get()[1:-1, 1:-1, 1:-1] - ref).max() < _bound(ng) * np.abs(ref).max()


SINGULAR = [(*s, False) for s in SHAPES if "D" not in s[0]] + [(*s, True) for s in THIN if "D" not in s[0]]


@pytest.mark.parametrize("cbcpre,ng,thin", SINGULAR)
def test_solver_without_a_dirichlet_wall(cbcpre, ng, thin):
    """Column 0 is each level's sum over x and y, which is exact for whole
    numbers.  Where the sums are zero, so is column 0's solution, and the
    others are compared; with 1 added everywhere, which the last pivot blows
    up, column 0, constant included: a sum of nz equal signs, so nz roundings
    at most."""
    p, rhs = _case(cbcpre, ng, thin)
    inner = rhs[1:-1, 1:-1, 1:-1]
    inner[:] = np.rint(1024.0 * inner)
    inner[0, 0] -= inner.sum(axis=(0, 1))
    g, o = C.Case(p), O.Case(p)
    pg = g.field(rhs)
    g.call("solver", pg)
    ref = _exact(p, g.grid(), inner, keep0=False)
    assert np.abs(pg.get()[1:-1, 1:-1, 1:-1] - ref).max() < _bound(ng) * np.abs(ref).max()
    rhs[1:-1, 1:-1, 1:-1] += 1.0
    pg = g.field(rhs)
    g.call("solver", pg)
    o.call("solver", rhs)
    a, b = (f[1:-1, 1:-1, 1:-1].mean(axis=(0, 1)) for f in (pg.get(), rhs))
    assert np.abs(a - b).max() < 4 * EPS * (ng[2] + 50) * np.abs(b).max()


REFINED = [("PPPPDD", (12, 10, 24), False), ("PPPPDD", (20, 6, 31), False), ("PPPPDD", (64, 2, 65), False),
           ("PPPPDD", (10, 6, 500), False), ("PPPPDD", (512, 6, 9), False), ("PPPPND", (512, 8, 24), True),
           ("PPPPND", (256, 8, 64), True), ("PPPPND", (20, 512, 32), False), ("PPPPNN", (20, 512, 32), False),
           ("PPPPNN", (20, 6, 31), False), ("PPPPNN", (64, 64, 100), False),
           ("PPPPND", (512, 256, 24), False), ("PPPPND", (512, 270, 24), False)]


@pytest.mark.parametrize("cbcpre,ng,thin", REFINED)
def test_solver_refined(cbcpre, ng, thin):
    """The FP32 solve: transforms of 64 to 256 points as split-BF16 GEMMs keep
    16 bits of a line's largest mode, other lengths 24, and the white right-hand
    side's smallest modes are 1e-1 of that: 1e-4.  A sweep leaves the same
    fraction of its residual, in the worst mode ten times that: 1e-3 of the
    error before, and a second one 1e-3 of that, down to the FP64 rounding.
    Between Neumann walls, with the sums of each level zero, the pinned column
    0 is a constant, which is removed."""
    p, rhs = _case(cbcpre, ng, thin)
    singular = "D" not in cbcpre
    inner = rhs[1:-1, 1:-1, 1:-1]
    if singular:
        inner[:] = np.rint(1024.0 * inner)
        inner[0, 0] -= inner.sum(axis=(0, 1))
    g = C.Case(p)
    rg, pg = g.field(rhs), g.field()
    ref = _exact(p, g.grid(), inner, keep0=not singular)
    for sweeps, bound in ((0, 1e-4), (1, 1e-7), (2, 1e-10)):
        g.call("solver_refined", rg, pg, sweeps)
        got = pg.get()[1:-1, 1:-1, 1:-1]
        if singular:
            got = got - got.mean()
        assert np.abs(got - ref).max() < bound * np.abs(ref).max(), sweeps


@pytest.mark.parametrize("ng", [(64, 2, 65), (12, 10, 257), (96, 64, 128)])
def test_column_solve_chosen_later(ng):
    """zsolve = 1 on a case whose columns the partitioned solve takes: the
    elimination factors are evaluated when the plan asks for them (FP64, and
    FP32 where that solver has run or runs later)."""
    p, rhs = _case("PPPPND", ng)
    ref = _exact(p, C.Case(p).grid(), rhs[1:-1, 1:-1, 1:-1])
    for refined_first in (False, True):
        g = C.Case(p)
        rg, pg = g.field(rhs), g.field()
        if refined_first:
            g.call("solver_refined", rg, pg, 1)
        q = g.plan()
        q.zsolve = 1
        g.set_plan(q)
        g.call("solver_refined", rg, pg, 1)
        assert np.abs(pg.get()[1:-1, 1:-1, 1:-1] - ref).max() < 1e-6 * np.abs(ref).max()
        pg = g.field(rhs)
        g.call("solver", pg)
        got = pg.get()[1:-1, 1:-1, 1:-1]
        assert np.abs(got - ref).max() < (4 * EPS * (2 * ng[2] / math.pi) ** 2 + 1e-14) * np.abs(ref).max()


def test_no_factors_where_the_partitioned_solve_takes_the_columns():
    """Two spectral-size arrays less than a case whose columns are one level
    too long for it."""
    import torch

    def used(nz):
        free = torch.cuda.mem_get_info()[0]
        case = C.Case(_nml(96, 64, nz))
        used = free - torch.cuda.mem_get_info()[0]
        case.close()
        return used

    used(512)  # the first case loads the module
    cells = 96 * 64 * 512 * 8
    assert used(513) - used(512) > 1.5 * cells
