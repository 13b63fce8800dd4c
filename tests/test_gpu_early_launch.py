"""Small grids, whose step is a chain of kernels that come onto the device
before their predecessor has ended, against the same steps without early
launches (an ensemble's graph has none): bit-equal over many steps, since the
launch shapes change no result.
"""
import numpy as np
import pytest

from cansfz import case as C
from cansfz import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("ng,l,two_d", [((16, 2, 32), (1.0, 0.125, 2.0), True), ((64, 2, 128), (1.0, 2.0 / 64, 2.0), True),
                                        ((32, 32, 32), (1.0, 1.0, 1.0), False)])
def test_many_steps_with_and_without_early_launch(ng, l, two_d, form):
    p, f = W._bubble_case(*ng, *l, 100.0, 10.0, 5.0, 0.4, two_d)
    p.form = form
    early, plain = C.Case(p, own_stream=True), C.Case(p, own_stream=True)
    for c in (early, plain):
        c.set_fields(*f)
        c.prepare()
    ens = C.Ensemble([plain], batch=1)
    for n in (1, 149, 150):
        assert early.step(n) == 0
        rc, _ = ens.step(n)
        assert rc == 0
        for nm in ("u", "v", "w", "p", "psi"):
            assert np.array_equal(early.get(nm), plain.get(nm)), (nm, n)
    a, b = early.diag(), plain.diag()
    assert (a.istep, a.dt, a.gam, a.divmax) == (b.istep, b.dt, b.gam, b.divmax)
    ens.close()


@pytest.mark.parametrize("ng", [(30, 200, 30), (250, 2, 40)])
def test_lines_of_runtime_length_between_early_launches(ng):
    """Transforms that are not launched early themselves, with kernels before
    and after them that are."""
    test_many_steps_with_and_without_early_launch(ng, (1.0, ng[1] / ng[0], ng[2] / ng[0]), ng[1] == 2, 0)
