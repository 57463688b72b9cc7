"""The Poisson mode solves (k_ymodes) at the edges of their forms -- lane chunks
of up to 9, 17 and 25 values in registers, two warps per mode up to 1088
unknowns, the chunk in shared memory beyond -- by the residual of the systems
they solve, (A_y + wr) x = h: a backward stable elimination of n unknowns leaves
at most about 10 rounding errors of the largest term per row."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n2m", [32, 287, 288, 289, 544, 545, 800, 801, 1087, 1088, 1089, 1300])
@pytest.mark.parametrize("form", [fb.POISSON_INT8X8, fb.POISSON_TF32X3])
def test_mode_solves(n2m, form, tmp_path):
    h = 4.0 / n2m
    c = cases.viv_cylinder(n3m=72, n2m=n2m, h=h, zwin=(-1.0, 36 * h - 1.0), ywin=(-(n2m // 4) * h, (n2m // 4) * h),
                           zdom=(-3.0, 9.0), ydom=(-3.0, 3.0), nlm=24, dt=0.1 * h)
    s = fb.Solver(c.write(str(tmp_path / "deck")))
    s.set_poisson(form)
    rng = np.random.default_rng(n2m)
    for f in ("q2", "q3"):
        s.set(f, rng.standard_normal((c.n3m + 2, n2m + 1)))
    s.set_substep(2, 1)
    assert s.stage("divg") == 0
    dph = s.get("dph")[1:c.n3m + 1, :n2m]
    assert s.stage("phcalc") == 0
    # the last solve's modes: x with phi = zmm x (INT8), to the transforms' accuracy
    if form == fb.POISSON_INT8X8:
        x = s.get("hmn").reshape(c.n3m, -1)[:, :n2m]
        b = s.get("zmmt") @ dph
        wr, am, ac, ap = s.get("wr"), s.get("amphj"), s.get("acphj"), s.get("apphj")
        diag = ac[:n2m][None, :] + wr[:, None]
        r = diag * x - b
        r[:, 1:] += am[1:n2m] * x[:, :-1]
        r[:, :-1] += ap[:n2m - 1] * x[:, 1:]
        r[np.argmin(np.abs(wr))] = 0.0            # the null mode, whose last unknown is pinned
        size = np.abs(diag * x) + np.abs(b)
        size[:, 1:] += np.abs(am[1:n2m] * x[:, :-1])
        size[:, :-1] += np.abs(ap[:n2m - 1] * x[:, 1:])
        # the transform's own error: 1e-15 of the sums it forms
        tol = 20 * 2.0 ** -53 * size.max(axis=1, keepdims=True) + 2e-15 * (np.abs(s.get("zmmt")) @ np.abs(dph))
        assert np.all(np.abs(r) <= tol)
    else:
        phi = s.get("dph")[1:c.n3m + 1, :n2m]
        s.set_poisson(fb.POISSON_FP64)
        for f in ("q2", "q3"):
            s.set(f, s.get(f))
        assert s.stage("divg") == 0 and s.stage("phcalc") == 0
        ref = s.get("dph")[1:c.n3m + 1, :n2m]
        # two refinement sweeps of the split transforms: 1e-6 of the FP64 solution, gradients only
        d = np.diff(phi - ref, axis=0)
        assert np.max(np.abs(d)) <= 1e-6 * np.max(np.abs(np.diff(ref, axis=0)))
    s.close()
