"""The one-launch ghost fills against the oracle's stages (bit-equal)."""
import numpy as np
import pytest

import oracle as O
from cansfz import case as C

from test_gpu_parity import _nml, _rand_fields

pytestmark = pytest.mark.gpu


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
