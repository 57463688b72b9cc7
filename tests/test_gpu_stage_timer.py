"""fb_time_stage repeats a stage behind itself.  Its launches must be those of a
sequence of separate fb_stage calls (one warm-up, the captured repeats twice),
each of which sees what the one before stored: equal bits."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stage,fields", [
    ("nl_rhs", ("rhs2", "rhs3", "ru2", "ru3")), ("forcing", ("rhs2", "rhs3")), ("helsolve", ("q2", "q3")),
    ("updvp", ("q2", "q3", "pr")), ("loads", ("press", "tau", "bcerrv", "bcerrw"))])
@pytest.mark.parametrize("name", ["tiny", "384x256"])
def test_repeats_equal_separate_calls(stage, fields, name, tmp_path):
    c = cases.tiny_cylinder() if name == "tiny" else cases.viv_cylinder_384x256()
    path = c.write(str(tmp_path / "deck"))
    a, b = fb.Solver(path), fb.Solver(path)
    for s in (a, b):
        q2 = s.get("q2")
        q2[1:c.n3m + 1] += c.v_perturbation()
        s.set("q2", q2)
        s.advance(0, 2)
        s.set_substep(2, 2)
        for st in ("boucdq", "nl_rhs", "forcing"):
            assert s.stage(st, 2) == 0
    reps = 5
    b.time_stage(stage, 2, reps=reps)
    for _ in range(1 + 2 * reps):
        assert a.stage(stage, 2) == 0
    for f in fields:
        np.testing.assert_array_equal(b.get(f), a.get(f), err_msg=f)
    for s in (a, b):
        s.close()
