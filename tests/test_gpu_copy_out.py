"""Field reads through the pinned chunks (fields above 512 KiB) and the history
ring's runs: chunk remainders, one chunk more or less, a ring that wraps."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n3m,n2m", [(384, 160), (384, 256), (700, 511), (1000, 127)])
def test_field_round_trip(n3m, n2m, tmp_path):
    c = cases.viv_cylinder(n3m=n3m, n2m=n2m, h=12.0 / n3m, zwin=(-1.5, (n3m // 4) * 12.0 / n3m - 1.5),
                           ywin=(-(n2m // 4) * 6.0 / n3m, ((n2m // 4) - (n2m // 4) / 2) * 12.0 / n3m), nlm=60)
    s = fb.Solver(c.write(str(tmp_path / "deck")))
    rng = np.random.default_rng(n2m)
    for f in ("q2", "pr"):
        x = rng.standard_normal((n3m + 2, n2m + 1))
        s.set(f, x)
        np.testing.assert_array_equal(s.get(f), x)
        np.testing.assert_array_equal(s.get(f), x)
    s.close()


def test_history_ring_wraps(tmp_path):
    s = fb.Solver(cases.tiny_cylinder().write(str(tmp_path / "deck")))
    s.advance(0, 4000, history=False)
    h = s.advance(4000, 200)     # rows 4000 .. 4199 of a ring of 4096
    assert np.array_equal(h[1:, 0], h[:-1, 8]) and np.all(np.diff(h[:, 8]) > 0)
    np.testing.assert_array_equal(h[-1], s.last_history())
    s.close()
