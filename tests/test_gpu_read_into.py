"""Field reads into pinned and pageable memory of the caller, the same bits."""
import ctypes

import numpy as np
import pytest

import fribois2d_b200 as fb
from fribois2d_b200 import case as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 3])
def test_read_into_pinned_memory(offset, tmp_path):
    import torch
    c = cases.viv_cylinder(nlm=60)
    s = fb.Solver(c.write(str(tmp_path / "deck")))
    x = np.random.default_rng(0).standard_normal((c.n3m + 2, c.n2m + 1))
    s.set("q2", x)
    buf = torch.zeros(x.size + offset, dtype=torch.float64, pin_memory=True)
    dp = ctypes.POINTER(ctypes.c_double)
    ptr = ctypes.cast(buf.data_ptr() + 8 * offset, dp)
    assert fb.lib().fb_get_array(s.ctx, fb.IDS["q2"], ptr, x.size) == 0
    np.testing.assert_array_equal(buf.numpy()[offset:], x.reshape(-1))
    np.testing.assert_array_equal(s.get("q2"), x)
    s.close()
