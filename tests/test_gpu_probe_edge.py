"""Loads of a body near the inflow whose probes reach the first two cells: the
wall-normal derivative there reads pr in row k = 0, which fb_advance brings up
to date later than the separate calls do.  Same kernels' arithmetic in the same
order, so the same bits (the checkbcs norms, HIST 18 and 19, are summed in
another order: nlm 2^-53)."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsst", [3, 1])
@pytest.mark.parametrize("nlm", [40, 2050])   # one closing launch, and the two launches beyond 2048 markers
def test_probes_at_the_inflow(nsst, nlm, tmp_path):
    if nlm <= 500:
        c = cases.tiny_cylinder(n3m=96, nlm=nlm)
    else:
        c = cases.viv_cylinder(n3m=576, n2m=256, ywin=(-2.0, 2.0), zdom=(-3.0, 9.0), ydom=(-3.0, 3.0), nlm=nlm)
    c.zcoord = cases.uniform_axis(12.0, c.n3m)
    h = 12.0 / c.n3m
    z = 6.5 * h + 0.5            # the leftmost marker in cell 7
    c.vert = c.vert + np.array([0.0, z - c.params.cmposi[1]])
    c.params.cmposi = (c.params.cmposi[0], z)
    c.params.kprobe = 4.9 ** 0.5   # probes 4.9 spacings off the surface: z = 1.6 h
    c.params.nsst = nsst
    path = c.write(str(tmp_path / "deck"))
    a, b = fb.Solver(path), fb.Solver(path)
    for s in (a, b):
        q2 = s.get("q2")
        q2[1:c.n3m + 1] += c.v_perturbation()
        s.set("q2", q2)
    rows = []
    for ns in range(4):
        a.fluid_tsch(ns)
        a.rigid(ns)
        rows.append(a.last_history())
    hist = b.advance(0, 4)
    for f in ("press", "tau", "rigid", "lmcc", "q2", "q3", "pr"):
        np.testing.assert_array_equal(b.get(f), a.get(f), err_msg=f)
    rows, norms = np.stack(rows), [18, 19]
    np.testing.assert_array_equal(np.delete(hist, norms, 1), np.delete(rows, norms, 1))
    np.testing.assert_allclose(hist[:, norms], rows[:, norms], rtol=nlm * 2.0 ** -53, atol=0)
    for s in (a, b):
        s.close()
