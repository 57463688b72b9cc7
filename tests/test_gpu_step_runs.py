"""A long fb_advance (several steps per graph launch from the 17th on) against
short calls with the same state: the same kernels in the same order, so the
same bits, with the remainders of the run length."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsst,report,nlm,steps", [(3, False, 40, 49), (3, True, 40, 56), (1, False, 40, 61),
                                                   (3, True, 2049, 50)])
def test_long_call_equals_short_calls(nsst, report, nlm, steps, tmp_path):
    c = cases.tiny_cylinder(nlm=nlm) if nlm < 500 else cases.viv_cylinder(nlm=nlm, noise=1e-3)
    c.params.nsst = nsst
    path = c.write(str(tmp_path / "deck"))
    a, b = fb.Solver(path), fb.Solver(path)
    for s in (a, b):
        s.set_report(report)
    short = [a.advance(n, min(10, 2 * steps + 20 - n)) for n in range(0, 2 * steps + 20, 10)]
    long = [b.advance(0, steps), b.advance(steps, steps + 20)]   # the second call has the run from its start
    np.testing.assert_array_equal(np.concatenate(long), np.concatenate(short))
    for f in ("q2", "q3", "pr", "ru2", "ru3", "lmcc", "lmvel", "rigid", "press", "tau"):
        np.testing.assert_array_equal(b.get(f), a.get(f), err_msg=f)
    for s in (a, b):
        s.close()
