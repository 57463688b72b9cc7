"""FB_SCALARS behind fb_advance: the values that the separate calls leave, the
substep coefficients (al, ga, ro) among them, whichever of fb_advance's graphs
were made in the call.  The checkbcs norms are summed in another order."""
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsst", [3, 1])
@pytest.mark.parametrize("vardt", [False, True])
@pytest.mark.parametrize("calls", [(1, 1), (3, 2), (60,)])
def test_scalars_after_advance(nsst, vardt, calls, tmp_path):
    c = cases.tiny_cylinder()
    c.params.nsst = nsst
    c.params.idtv = not vardt
    c.params.dtmax = 0.02
    path = c.write(str(tmp_path / "deck"))
    a, b = fb.Solver(path), fb.Solver(path)
    ns = 0
    for n in calls:
        b.advance(ns, n)
        for _ in range(n):
            a.fluid_tsch(ns)
            a.rigid(ns)
            ns += 1
    sa, sb = a.scalars(), b.scalars()
    for k in fb.SCALAR_NAMES:
        if k in ("nbcv", "nbcw"):
            assert sb[k] == pytest.approx(sa[k], rel=c.nlm * 2.0 ** -53, abs=0), k
        else:
            assert sb[k] == sa[k], k
    for s in (a, b):
        s.close()
