"""fb_advance with dt following the CFL number (one wait per step, coefficients
built beside the kernels that do not need them) against the separate calls: the
same kernels in the same order, so the same bits; only the checkbcs norms (HIST
18, 19) are summed in another order.  A step whose dt is refused ends the call."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu

FIELDS = ("q2", "q3", "pr", "ru2", "ru3", "lmcc", "lmvel", "rigid", "press", "tau", "qb2n", "qb3n", "dq3x2o")


def _deck(nlm, nsst, cflmax, path):
    c = cases.tiny_cylinder(nlm=nlm) if nlm < 500 else cases.viv_cylinder(nlm=nlm, noise=1e-3)
    c.params.idtv = False
    c.params.nsst = nsst
    c.params.cflmax = cflmax
    c.params.dtmax = 0.02
    return c.write(str(path))


@pytest.mark.parametrize("nsst,report,nlm", [(3, False, 40), (1, True, 40), (3, True, 513), (3, False, 2049)])
def test_variable_dt_advance_equals_separate_calls(nsst, report, nlm, tmp_path):
    path = _deck(nlm, nsst, 0.25, tmp_path / "deck")
    a, b, c = (fb.Solver(path) for _ in range(3))
    for s in (a, b, c):
        s.set_report(report)
    rows = []
    for ns in range(7):
        a.fluid_tsch(ns)
        a.rigid(ns)
        rows.append(a.last_history())
    hist = np.concatenate([b.advance(0, 4), b.advance(4, 3)])
    ones = np.concatenate([c.advance(ns, 1) for ns in range(7)])
    np.testing.assert_array_equal(ones, hist)
    for f in FIELDS:
        np.testing.assert_array_equal(b.get(f), a.get(f), err_msg=f)
        np.testing.assert_array_equal(c.get(f), a.get(f), err_msg=f)
    rows, norms = np.stack(rows), [18, 19]
    np.testing.assert_array_equal(np.delete(hist, norms, 1), np.delete(rows, norms, 1))
    np.testing.assert_allclose(hist[:, norms], rows[:, norms], rtol=nlm * 2.0 ** -53, atol=0)
    for s in (a, b, c):
        s.close()


def test_refused_dt_ends_the_call(tmp_path):
    path = _deck(40, 3, 1e-12, tmp_path / "deck")   # dt = cflmax / cflm < 1e-8 from the second step on
    a, b = fb.Solver(path), fb.Solver(path)
    a.advance(0, 1)
    with pytest.raises(fb.FBError) as e:
        b.advance(0, 3)
    assert e.value.code == fb.FB_ERR_CFL
    for f in FIELDS:
        np.testing.assert_array_equal(b.get(f), a.get(f), err_msg=f)
    for s in (a, b):
        s.close()
