"""A refused variable dt (cflmax / cfl below 1e-8) ends its step between the
marker set-up and the forcing.  The context goes on working: a step taken after
it equals, bit for bit, the step of a context that was never refused, with the
markers where they were, moved, or given back after they had left the domain
(a refused step raises no error of the set-up that it did not come to use)."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu

FIELDS = ("q2", "q3", "pr", "ru2", "ru3", "lmcc", "lmvel", "lmnor", "rigid", "press", "tau", "qb2n", "qb3n", "dq3x2o")


def _refused(call):
    with pytest.raises(fb.FBError) as e:
        call()
    assert e.value.code == fb.FB_ERR_CFL


def _step(s, how):
    """A step at the deck's own dt (ns = 0), which no CFL number refuses."""
    if how == "advance":
        s.advance(0, 1)
    else:
        s.fluid_tsch(0)
        s.rigid(0)


@pytest.mark.parametrize("nlm", [40, 400])   # 400: cells with more touchers than a group's list holds
@pytest.mark.parametrize("how", ["advance", "separate"])
@pytest.mark.parametrize("move", [0.0, 0.04])
def test_steps_after_a_refused_dt(nlm, how, move, tmp_path):
    c = cases.tiny_cylinder(nlm=nlm)
    c.params.idtv = False
    c.params.cflmax = 1e-12
    path = c.write(str(tmp_path / "deck"))
    a, b = fb.Solver(path), fb.Solver(path)
    for s in (a, b):
        _step(s, how)
    for call in (lambda: b.advance(1, 3), lambda: b.fluid_tsch(1), lambda: b.advance(1, 1)):
        _refused(call)
    for s in (a, b):
        s.set("lmcc", s.get("lmcc") + move)
        for _ in range(2):
            _step(s, how)
    _refused(lambda: b.fluid_tsch(2))
    for s in (a, b):
        _step(s, how)
    for f in FIELDS:
        np.testing.assert_array_equal(b.get(f), a.get(f), err_msg=f)
    np.testing.assert_array_equal(b.last_history(), a.last_history())
    for s in (a, b):
        s.close()


def test_refused_with_markers_outside(tmp_path):
    c = cases.tiny_cylinder()
    c.params.idtv = False
    c.params.cflmax = 1e-12
    path = c.write(str(tmp_path / "deck"))
    a, b = fb.Solver(path), fb.Solver(path)
    for s in (a, b):
        s.advance(0, 1)
    lmcc = b.get("lmcc")
    b.set("lmcc", lmcc + 100.0)
    _refused(lambda: b.fluid_tsch(1))
    _refused(lambda: b.advance(1, 2))
    b.set("lmcc", lmcc)
    for s in (a, b):
        s.advance(0, 1)
        s.advance(0, 1)
    for f in FIELDS + ("scalars",):
        np.testing.assert_array_equal(b.get(f), a.get(f), err_msg=f)
    for s in (a, b):
        s.close()
