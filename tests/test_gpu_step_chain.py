"""fb_advance's chain of launches (the end of a step beside the start of the
next one, the loads finished by the probes, one launch for their sums and the
rigid update) against the separate calls fb_fluid_tsch + fb_rigid: the same
arithmetic in the same order, so the same bits.  Only the checkbcs norms are
summed in another order (a sum of nlm non-negative terms: nlm 2^-53 relative at
most).  Marker counts at the edges of the closing launch (one block of 512
threads, at most 2048 markers; more take the two launches); a body at rest in
fluid at rest has no tangents (they carry over from nowhere)."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


def _open(c, path, rest):
    s = fb.Solver(path)
    if rest:
        for f in ("q2", "q3"):
            s.set(f, np.zeros((c.n3m + 2, c.n2m + 1)))
    else:
        q2 = s.get("q2")
        q2[1:c.n3m + 1] += c.v_perturbation()
        s.set("q2", q2)
    return s


@pytest.mark.parametrize("nlm,nsst,opts", [
    (40, 3, {}), (40, 1, {}), (40, 3, {"report": True}), (40, 3, {"rest": True}), (40, 3, {"cbody": False}),
    (40, 3, {"rtcoup": True}), (512, 3, {}), (513, 3, {}), (2048, 3, {}), (2049, 3, {"report": True})])
def test_advance_equals_separate_calls(nlm, nsst, opts, tmp_path):
    if nlm < 500:
        c = cases.tiny_cylinder(nlm=nlm)
    else:
        c = cases.viv_cylinder(nlm=nlm, noise=1e-3)
    c.params.nsst = nsst
    c.params.cbody = opts.get("cbody", True)
    c.params.rtcoup = opts.get("rtcoup", False)
    path = c.write(str(tmp_path / "deck"))
    steps = 5
    a, b = (_open(c, path, opts.get("rest", False)) for _ in range(2))
    for s in (a, b):
        s.set_report(opts.get("report", False))
    rows = []
    for ns in range(steps):
        a.fluid_tsch(ns)
        a.rigid(ns)
        rows.append(a.last_history())
    hist = np.concatenate([b.advance(0, 3), b.advance(3, 2)])
    for f in ("q2", "q3", "pr", "ru2", "ru3", "lmcc", "lmvel", "lmacc", "lmnor", "vert", "rigid", "press", "tau",
              "qb2n", "qb3n", "dq3x2o"):
        np.testing.assert_array_equal(b.get(f), a.get(f), err_msg=f)
    rows, norms = np.stack(rows), [18, 19]
    np.testing.assert_array_equal(np.delete(hist, norms, 1), np.delete(rows, norms, 1))
    np.testing.assert_allclose(hist[:, norms], rows[:, norms], rtol=nlm * 2.0 ** -53, atol=0)
    for s in (a, b):
        s.close()
