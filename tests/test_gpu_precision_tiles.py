"""The 3xTF32 products that add to an earlier result (the refinement sweeps, in
place and into dph) at grids that leave remainders of the 128-row and 32-column
parts of a tile, alone and grouped: the step stays within the form's tolerance
of the FP64 transforms, 1e-9 per step."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n3m,n2m", [(48, 31), (65, 33), (97, 128), (160, 129)])
def test_refined_steps_match_fp64(n3m, n2m, tmp_path):
    h = 3.0 / (n3m // 2) if n3m < 160 else 6.0 / (n3m // 2)
    wy = (n2m // 2) * h
    dom = dict(zdom=(-3.0, 9.0), ydom=(-3.0, 3.0)) if n3m < 97 else dict(zdom=(-9.0, 27.0), ydom=(-9.0, 9.0))
    c = cases.viv_cylinder(n3m=n3m, n2m=n2m, h=h, zwin=(-1.0, (n3m // 2) * h - 1.0), ywin=(-wy / 2, wy / 2), nlm=40,
                           dt=5e-3, noise=1e-3, **dom)
    path = c.write(str(tmp_path / "deck"))
    out = []
    for mode, grouped in ((fb.POISSON_FP64, False), (fb.POISSON_TF32X3, False), (fb.POISSON_TF32X3, True)):
        s = [fb.Solver(path) for _ in range(2 if grouped else 1)]
        for x in s:
            x.set_poisson(mode)
            q2 = x.get("q2")
            q2[1:c.n3m + 1] += c.v_perturbation()
            x.set("q2", q2)
        if grouped:
            b = fb.Batch(s)
            assert b.info()["groups"] == 1
            b.advance(5)
            b.close()
        else:
            s[0].advance(0, 5)
        out.append([s[-1].get(f)[1:n3m + 1, :n2m] for f in ("q2", "q3")])
        for x in s:
            x.close()
    for got in out[1:]:
        for a, b in zip(got, out[0]):
            assert np.max(np.abs(a - b)) <= 1e-9 * 5 * np.max(np.abs(b))
