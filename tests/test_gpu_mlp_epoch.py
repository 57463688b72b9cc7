"""Training by one launch per epoch (k_mlp_epoch) at the edges of its range:
input and output widths, one group of samples, ragged last groups, several
groups per cluster block, and a batch beyond the cluster's shared memory (the
per-minibatch launches).

Full-batch epochs are compared with Adam in 64 bits on the oracle's gradient.
The FP32 gradient sums are within 1e-5 of the largest gradient entry, so where
an entry is at least 1e-2 of that its normalised step is within 1e-3, and three
steps within 3e-3 of the learning rate; ten times that is allowed.
"""
import numpy as np
import pytest

import fribois2d_b200 as fb
from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


def _data(n, n_in, n_out, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, n_in)).astype(np.float32)
    return x, (np.sin(x @ rng.standard_normal((n_in, n_out))) + 0.5).astype(np.float32)


@pytest.mark.parametrize("n_in,n_out,batch", [(27, 2, 1), (27, 2, 16), (27, 2, 17), (27, 2, 100), (27, 2, 512),
                                              (1, 1, 40), (64, 8, 128), (64, 8, 250), (27, 2, 3000)])
def test_full_batch_epochs_follow_adam(n_in, n_out, batch):
    x, t = _data(batch, n_in, n_out, batch + n_in)
    m = fb.MLP(n_in, n_out, seed=5)
    p = m.params().astype(np.float64)
    lr, mom, var = 1e-3, 0.0, 0.0
    keep = np.ones(p.size, dtype=bool)
    for step in range(1, 4):
        loss, g = omlp.loss_and_grad(p, x.astype(np.float64), t.astype(np.float64))
        keep &= np.abs(g) >= 1e-2 * np.abs(g).max()
        mom = 0.9 * mom + 0.1 * g
        var = 0.999 * var + 0.001 * g * g
        p = p - lr * (mom / (1 - 0.9 ** step)) / (np.sqrt(var / (1 - 0.999 ** step)) + 1e-8)
    last = m.train(x, t, epochs=3, batch=batch, lr=lr, seed=1)
    got = m.params()
    assert keep.sum() > 10
    assert np.max(np.abs(got - p)[keep]) <= 3e-2 * lr
    assert last == pytest.approx(loss, rel=1e-4)
    m.close()


@pytest.mark.parametrize("batch", [5, 64, 200])
def test_minibatches_equal_separate_steps(batch):
    """Equal samples: an epoch of two minibatches and a remainder (dropped)
    is two full-batch epochs, bit for bit, and continues Adam's state."""
    x, t = _data(1, 27, 2, batch)
    out = []
    for n, epochs in ((2 * batch + batch // 2, 2), (batch, 4)):
        m = fb.MLP(27, 2, seed=3)
        m.train(np.repeat(x, n, 0), np.repeat(t, n, 0), epochs=epochs, batch=batch, lr=1e-3, seed=2)
        out.append(m.params())
        m.close()
    np.testing.assert_array_equal(out[0], out[1])
