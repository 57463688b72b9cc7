"""The grouped digit cut, whose row maxima divg and the mode solves accumulate,
at ragged edges of its blocks (32 rows x 128 columns), and the windowed
helsolve's form for windows of 9 and 10 rows, alone and in a group."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


def _solver(path, seed):
    s = fb.Solver(path)
    s.set_poisson(fb.POISSON_INT8X8)
    rng = np.random.default_rng(seed)
    q2 = s.get("q2")
    q2[2:-2, 2:-2] += 1e-3 * rng.standard_normal(q2[2:-2, 2:-2].shape)
    s.set("q2", q2)
    return s


@pytest.mark.parametrize("n3m,n2m,dt", [(48, 31, 5e-3), (65, 33, 5e-3), (127, 64, 4e-3), (129, 97, 0.02)])
def test_grouped_digits_equal_separate_runs(n3m, n2m, dt, tmp_path):
    h = 3.0 / (n3m // 2)
    wy = (n2m // 2) * h
    alone, together = [], []
    for i, re in enumerate((100.0, 130.0, 180.0)):
        c = cases.viv_cylinder(n3m=n3m, n2m=n2m, h=h, zwin=(-1.0, (n3m // 2) * h - 1.0), ywin=(-wy / 2, wy / 2),
                               zdom=(-3.0, 9.0), ydom=(-3.0, 3.0), nlm=40, dt=dt, noise=1e-3)
        c.params.visc = 1.0 / re
        path = c.write(str(tmp_path / f"deck{i}"))
        alone.append(_solver(path, i))
        together.append(_solver(path, i))
    window = alone[0].dims()[7]
    if n3m == 129:
        assert 9 <= max(window & 255, window >> 8) <= 10
    for s in alone:
        s.autotune()
        s.advance(0, 4)
    batch = fb.Batch(together)
    assert batch.info()["groups"] == 1
    batch.advance(1)   # twice: the maxima are cleared between the steps
    batch.advance(3)
    for a, b in zip(alone, together):
        for f in ("q2", "q3", "pr"):
            x, y = a.get(f), b.get(f)
            # the digits follow from the rows alone; sums over a grid (the
            # means) run in another order: a few 2^-52 of a field's size a step
            assert np.max(np.abs(x - y)) <= 1e-12 * np.max(np.abs(x)), f
    batch.close()
    for s in alone + together:
        s.close()


def test_window_form_of_ten_rows(tmp_path, monkeypatch):
    # as the other forms' comparison with the line scans: 1e-13 of the increment
    h = 3.0 / 64
    c = cases.viv_cylinder(n3m=129, n2m=97, h=h, zwin=(-1.0, 2.0), ywin=(-24 * h, 24 * h), zdom=(-3.0, 9.0),
                           ydom=(-3.0, 3.0), nlm=40, dt=0.02)
    path = c.write(str(tmp_path / "deck"))
    out = []
    for mode in ("win", "scan"):
        monkeypatch.setenv("FRIBOIS2D_HELSOLVE", mode)
        s = fb.Solver(path)
        w = s.dims()[7]
        assert (9 <= max(w & 255, w >> 8) <= 10) == (mode == "win")
        rng = np.random.default_rng(5)
        for f in ("q2", "q3", "rhs2", "rhs3"):
            s.set(f, rng.standard_normal((131, 98)))
        for f in ("dqb2s", "dqb2n", "dqb3s", "dqb3n"):
            s.set(f, rng.standard_normal(98))
        before = [s.get(f) for f in ("q2", "q3")]
        s.set_substep(2, 1)
        assert s.stage("helsolve") == 0
        out.append([s.get(f) - b for f, b in zip(("q2", "q3"), before)])
        s.close()
    for a, b in zip(*out):
        assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b)) + 4 * 2.0 ** -52
