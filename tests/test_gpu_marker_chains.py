"""The spreading chains by groups of lanes (k_spread_chains) at the edges of
its list (up to 64 touchers of a cell by the group; more, or cells with more
than 16 boxes, by one thread), and the nearest nodes found in the MLS set-up's
launch: whole steps against the oracle's sequential loops.  A cell's markers
are summed in marker order in both, so the agreement is that of any step (1e-10
each)."""
import numpy as np
import pytest

from fribois2d_b200 import case as cases
from paritylib import Pair, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlm", [12, 40, 180, 400, 700])
def test_step_with_marker_clusters_follows_oracle(nlm, tmp_path):
    p = Pair(cases.tiny_cylinder(nlm=nlm), str(tmp_path))
    steps = 3
    for ns in range(steps):
        assert p.o.step(ns) == 0
    h = p.s.advance(0, steps)
    for f in ("q2", "q3"):
        assert rel(p.s.get(f)[1:p.n3m + 1, :p.n2m], p.of(f)[1:p.n3m + 1, :p.n2m]) <= 1e-10 * steps, f
    sc, o = p.s.scalars(), p.o.scalars()
    # the CFL number of the last step's start and the mean w, from nl_rhs
    assert h[-1, 20] == sc["cflm"] == pytest.approx(o["cflm"], rel=1e-10)
    assert sc["q3avg"] == pytest.approx(o["q3avg"], rel=1e-10)
    p.s.close()
