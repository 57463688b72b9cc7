"""What a step that ends with an error leaves behind: the same, whether it is
taken by fb_advance, by a batch, by the separate calls or stage by stage.

* A CFL number beyond the limit holds the forcing back in every substep.
* Loads whose probes fail leave press and tau as they were.
* At variable dt the step that raises an error is counted, with its history
  row, and the next one leaves no trace.
"""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu

STATE = ("q2", "q3", "pr", "ru2", "ru3", "lmcc", "lmvel", "lmnor", "rigid", "press", "tau", "qb2n", "qb3n", "dq3x2o")


def _open(c, path):
    s = fb.Solver(path)
    q2 = s.get("q2")
    q2[1:c.n3m + 1] += c.v_perturbation()
    s.set("q2", q2)
    return s


def _fails(call, code):
    with pytest.raises(fb.FBError) as e:
        call()
    assert e.value.code == code


def _uniform(nlm):
    """A cylinder on a grid uniform along z; finer for more than 2048 markers."""
    if nlm <= 500:
        c = cases.tiny_cylinder(n3m=96, nlm=nlm)
    else:
        c = cases.viv_cylinder(n3m=576, n2m=256, ywin=(-2.0, 2.0), zdom=(-3.0, 9.0), ydom=(-3.0, 3.0), nlm=nlm)
    c.zcoord = cases.uniform_axis(12.0, c.n3m)
    return c, 12.0 / c.n3m


def _move(c, y, z):
    """The body's centre at (y, z)."""
    c.vert = c.vert + (np.array([y, z]) - c.params.cmposi)
    c.params.cmposi = (y, z)


@pytest.mark.parametrize("how", ["advance", "fluid_tsch", "batch"])
@pytest.mark.parametrize("nsst", [3, 1])
def test_cfl_error_holds_the_forcing_back(how, nsst, tmp_path):
    if how == "batch" and nsst == 1:
        pytest.skip("batches are RK3")
    c = cases.tiny_cylinder()
    c.params.nsst = nsst
    c.params.cfllim = 1e-6
    path = c.write(str(tmp_path / "deck"))
    a, b = _open(c, path), _open(c, path)
    a.set_substep(0, 1)
    assert a.stage("cfl") == fb.FB_ERR_CFL
    for n in range(1, nsst + 1):
        a.set_substep(0, n)
        for st in ("boucdq", "nl_rhs", "lgrdistribution", "forcing", "helsolve", "divg", "phcalc", "updvp",
                   "pr_submean"):
            if st != "lgrdistribution" or n == 1:
                assert a.stage(st, n) == fb.FB_ERR_CFL
    if how == "batch":
        other = _open(c, path)
        batch = fb.Batch([b, other])
        assert batch.info()["groups"] == 1
        _fails(lambda: batch.advance(1), fb.FB_ERR_CFL)
        batch.close()
        other.close()
    else:
        _fails(lambda: b.advance(0, 1) if how == "advance" else b.fluid_tsch(0), fb.FB_ERR_CFL)
    # the stages' and the step's launches sum the same terms in other block
    # shapes (boucdq's flux, the pressure mean): a few roundings of order one
    # values, where a forced substep differs by the forcing itself, O(0.1)
    for f in ("q2", "q3", "pr"):
        np.testing.assert_allclose(b.get(f), a.get(f), rtol=0, atol=1e-11, err_msg=f)
    for s in (a, b):
        s.close()


@pytest.mark.parametrize("nlm", [40, 2048, 2049])
def test_failed_probes_leave_the_loads(nlm, tmp_path):
    # markers down to the fourth line from the inflow: supported, but a probe's
    # search needs five lines on either side.  They come last in the order of the
    # markers, so that with many of them others' probes have ended before
    c, h = _uniform(nlm)
    _move(c, 3.0, 0.5 + 3.6 * h)
    v = np.roll(c.vert[:-1], int(0.45 * nlm), axis=0)
    c.vert = np.concatenate([v, v[:1]])
    path = c.write(str(tmp_path / "deck"))
    a, b = _open(c, path), _open(c, path)
    before = np.linspace(1.0, 2.0, nlm)
    for s in (a, b):
        s.set("press", before)
    _fails(lambda: a.fluid_tsch(0), fb.FB_ERR_MARKER_OUT)
    _fails(lambda: a.rigid(0), fb.FB_ERR_MARKER_OUT)
    _fails(lambda: b.advance(0, 1), fb.FB_ERR_MARKER_OUT)
    np.testing.assert_array_equal(a.get("press"), before)
    for f in STATE:
        np.testing.assert_array_equal(b.get(f), a.get(f), err_msg=f)
    for s in (a, b):
        s.close()


@pytest.mark.parametrize("nsst", [3, 1])
def test_variable_dt_counts_the_failing_step(nsst, tmp_path):
    # the body drifts into the second cell at the upper wall, where the support
    # does not fit: the marker set-up of the step that follows raises the error
    c = cases.tiny_cylinder()
    c.params.idtv = False
    c.params.nsst = nsst
    c.params.cflmax = 0.25
    c.params.dtmax = 0.02
    c.params.cbody = False
    c.params.ipert = (1.0, 0.0, 0.0)
    c.params.kk = (0.0, 0.0, 0.0)
    rm = 0.5 * (c.ycoord[1:] + c.ycoord[:-1])
    _move(c, 0.5 * (rm[-3] + rm[-2]) - 0.5 - 0.05, 3.0)
    path = c.write(str(tmp_path / "deck"))
    a, b = _open(c, path), _open(c, path)
    rows, code = [], 0
    for ns in range(20):
        try:
            a.fluid_tsch(ns)
        except fb.FBError as e:
            code = e.code
        try:
            a.rigid(ns)
        except fb.FBError as e:
            assert e.code == code
        rows.append(a.last_history())
        if code:
            break
    assert code and len(rows) > 2
    _fails(lambda: b.advance(0, 20), code)
    np.testing.assert_array_equal(b.last_history(), rows[-1])
    for f in STATE:
        np.testing.assert_array_equal(b.get(f), a.get(f), err_msg=f)
    sa, sb = a.scalars(), b.scalars()
    for f in ("time", "dt", "dt_o", "cflm", "q3avg", "nbcv", "nbcw", "pravg"):
        assert sb[f] == sa[f], f
    for s in (a, b):
        s.close()
