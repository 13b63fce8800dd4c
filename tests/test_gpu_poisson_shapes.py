"""The Poisson solve at the edges of its kernels' size ranges, against the
oracle: the partitioned z solve's chunks (shortest and longest columns,
columns that the chunks do not divide, a last tile of few columns, FP64 and
FP32), and the two-pass transforms of 512 points with a partial tile of lines.

Bounds: as in test_gpu_parity.test_poisson_bcs, 1e-12 of the largest stored
value (the constant of the singular mode included) for the FP64 solve.  One
refinement sweep of the FP32 solve leaves the square of its own relative error:
up to 7e-4 for a column of 500 levels (2^-24 times a condition number of about
(2 nz/pi)^2), squared 5e-7, bound 1e-6.  (Not for Neumann walls on a grid whose
single-precision z quotients make it slightly uneven: there the FP64 residual's
mean over the singular mode leaves 1e-6 and more whatever the sweeps, in either z solve.)
"""
import numpy as np
import pytest

import oracle as O
from cansfz import case as C

from test_gpu_parity import _nml

pytestmark = pytest.mark.gpu

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
]


def _system(cbcpre, ng):
    p = _nml(*ng, cbcpre, l=(1.0, 0.75, 1.2))
    rhs = np.zeros(tuple(n + 2 for n in ng), order="F")
    rhs[1:-1, 1:-1, 1:-1] = np.random.default_rng(5).standard_normal(p.n)
    if "D" not in cbcpre:
        rhs[1:-1, 1:-1, 1:-1] -= rhs[1:-1, 1:-1, 1:-1].mean()
    return p, rhs


def _compare(a, b, singular):
    a, b = a[1:-1, 1:-1, 1:-1], b[1:-1, 1:-1, 1:-1]
    scale = max(np.abs(a).max(), np.abs(b).max())
    if singular:
        a, b = a - a.mean(), b - b.mean()
    return np.abs(a - b).max(), scale, np.abs(b).max()


@pytest.mark.parametrize("cbcpre,ng", SHAPES)
def test_solver(cbcpre, ng):
    p, rhs = _system(cbcpre, ng)
    g, o = C.Case(p), O.Case(p)
    pg = g.field(rhs)
    g.call("solver", pg)
    o.call("solver", rhs)
    err, scale, _ = _compare(pg.get(), rhs, "D" not in cbcpre)
    assert err / scale < 1e-12


@pytest.mark.parametrize("cbcpre,ng", [("PPPPDD", (12, 10, 24)), ("PPPPDD", (20, 6, 31)), ("PPPPDD", (64, 2, 65)),
                                       ("PPPPDD", (10, 6, 500)), ("PPPPDD", (512, 6, 9)), ("PPPPNN", (20, 512, 32))])
def test_solver_refined(cbcpre, ng):
    p, rhs = _system(cbcpre, ng)
    g, o = C.Case(p), O.Case(p)
    rg, pg = g.field(rhs), g.field()
    g.call("solver_refined", rg, pg, 1)
    o.call("solver", rhs)
    err, _, size = _compare(pg.get(), rhs, "D" not in cbcpre)
    assert err / size < 1e-6
