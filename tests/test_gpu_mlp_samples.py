"""Minibatch training reads every sample once per epoch, and trains with more
samples than fit the device.

With a zero learning rate the reported loss is the mean over all samples of the
start parameters' squared errors; it is compared with the 64-bit value (FP32
forward pass and sums: 1e-5).  The samples' errors are all different, so a
sample read twice, or another's in its place, shows."""
import numpy as np
import pytest

import fribois2d_b200 as fb
from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n_out,batch", [(27, 2, 16), (27, 2, 100), (1, 1, 40), (64, 8, 250)])
def test_every_sample_counts_once(n_in, n_out, batch):
    n = 10 * batch
    rng = np.random.default_rng(batch)
    x = rng.standard_normal((n, n_in)).astype(np.float32)
    t = (rng.standard_normal((n, n_out)) * np.linspace(1.0, 30.0, n)[:, None]).astype(np.float32)
    m = fb.MLP(n_in, n_out, seed=4)
    want, _ = omlp.loss_and_grad(m.params().astype(np.float64), x.astype(np.float64), t.astype(np.float64))
    for epochs in (1, 3):
        assert m.train(x, t, epochs=epochs, batch=batch, lr=0.0, seed=epochs) == pytest.approx(want, rel=1e-5)
    m.close()


def test_samples_beyond_device_memory():
    import torch
    block, reps = 4096, 1440
    rng = np.random.default_rng(0)
    x0 = rng.standard_normal((block, 27)).astype(np.float32)
    t0 = rng.standard_normal((block, 2)).astype(np.float32)
    m = fb.MLP(27, 2, seed=4)
    want, _ = omlp.loss_and_grad(m.params().astype(np.float64), x0.astype(np.float64), t0.astype(np.float64))
    m.train(x0, t0, epochs=1, batch=128, lr=0.0)
    x, t = np.tile(x0, (reps, 1)), np.tile(t0, (reps, 1))    # 680 MB
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - (400 << 20), dtype=torch.uint8, device="cuda")
    assert m.train(x, t, epochs=1, batch=128, lr=0.0) == pytest.approx(want, rel=1e-4)
    del hog
    torch.cuda.empty_cache()
    m.close()
