"""The windowed helsolve at the edges of its tiles (32 columns x 32 or 64 rows,
segments of 16) against the full line scans: both solve the same systems, the
windows cut influences below 2^-56, and each is a chain of at most n rounded
operations of a diagonally dominant system: 1e-13 of the largest increment."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n3m,n2m", [(48, 32), (49, 33), (63, 47), (65, 64), (97, 65), (577, 257), (640, 256)])
def test_windowed_helsolve_equals_scans(n3m, n2m, tmp_path, monkeypatch):
    h = 3.0 / (n3m // 2) if n3m < 160 else 12.0 / n3m
    dom = {} if n3m >= 160 else dict(zdom=(-3.0, 9.0), ydom=(-3.0, 3.0))
    wy = (n2m // 2) * h
    c = cases.viv_cylinder(n3m=n3m, n2m=n2m, h=h, zwin=(-1.0, (n3m // 2) * h - 1.0), ywin=(-wy / 2, wy / 2), nlm=40,
                           dt=0.1 * h, **dom)
    path = c.write(str(tmp_path / "deck"))
    out = []
    for mode in ("win", "scan"):
        monkeypatch.setenv("FRIBOIS2D_HELSOLVE", mode)
        s = fb.Solver(path)
        assert (s.dims()[7] != 0) == (mode == "win")
        rng = np.random.default_rng(n3m)
        for f in ("q2", "q3", "rhs2", "rhs3"):
            s.set(f, rng.standard_normal((n3m + 2, n2m + 1)))
        for f in ("dqb2s", "dqb2n", "dqb3s", "dqb3n"):
            s.set(f, rng.standard_normal(n2m + 1))
        before = [s.get(f) for f in ("q2", "q3")]
        s.set_substep(2, 1)
        assert s.stage("helsolve") == 0
        out.append([s.get(f) - b for f, b in zip(("q2", "q3"), before)])
        s.close()
    for a, b in zip(*out):
        # (the difference of q after and before carries q's own rounding)
        assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b)) + 4 * 2.0 ** -52
