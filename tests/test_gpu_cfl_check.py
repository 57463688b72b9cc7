"""fb_cfl_noalloc against the same expressions in numpy: rows and columns at the
edges of the kernel's pairs, passes and blocks (296 blocks, two rows and 1024
columns per pass), a NaN in the last cell, more consecutive calls than the
kernel has completion counters, and a captured call.

The CFL number is a maximum of unfused expressions: equal bits.  The mean is a
sum of n positive terms in another order: n 2^-53 relative at most."""
import ctypes

import numpy as np
import pytest

import fribois2d_b200 as fb

pytestmark = pytest.mark.gpu

DT, L2, L3 = 1e-3, 30.0, 40.0


def _call():
    f = fb.lib().fb_cfl_noalloc
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int] + \
        [ctypes.c_void_p] * 4 + [ctypes.c_double] * 3 + [ctypes.c_void_p] * 2
    return f


class Field:
    def __init__(self, n3m, n2m, pad, seed):
        import torch
        rng = np.random.default_rng(seed)
        self.n3m, self.n2m, self.pitch = n3m, n2m, n2m + 1 + pad
        self.h = dict(q2=rng.standard_normal((n3m + 2, self.pitch)), q3=1.5 + rng.random((n3m + 2, self.pitch)),
                      rc=np.cumsum(rng.random(n2m + 1)), zz=np.cumsum(rng.random(n3m + 1)),
                      u2=1.0 + rng.random(n2m), u3=1.0 + rng.random(n3m))
        self.d = {k: torch.from_numpy(v).cuda() for k, v in self.h.items()}
        self.out = torch.full((2,), -1.0, dtype=torch.float64, device="cuda")

    def launch(self, stream=None):
        p = {k: v.data_ptr() for k, v in self.d.items()}
        st = _call()(p["q2"], p["q3"], self.pitch, self.n2m + 1, self.n3m + 1, p["rc"], p["zz"], p["u2"], p["u3"],
                     DT, L2, L3, self.out.data_ptr(), stream)
        assert st == 0

    def check(self):
        n3m, n2m, h = self.n3m, self.n2m, self.h
        q2, q3 = h["q2"][1:, :n2m + 1], h["q3"][1:, :n2m]
        v = np.abs((q2[:n3m, :-1] + q2[:n3m, 1:]) * 0.5 * h["u2"][None, :])
        w = np.abs((q3[:n3m] + q3[1:]) * 0.5 * h["u3"][:, None])
        mean = np.sum(q3[:n3m] * np.diff(h["zz"])[:, None] * np.diff(h["rc"])[None, :]) / (L2 * L3)
        got = self.out.cpu().numpy()
        assert got[0] == np.max(v + w) * DT
        assert abs(got[1] - mean) <= n3m * n2m * 2.0 ** -53 * mean


@pytest.mark.parametrize("n3m,n2m,pad", [(1, 1, 0), (296, 255, 0), (297, 1023, 3), (591, 1025, 0), (593, 1, 7),
                                         (1500, 1500, 31), (8191, 40, 0)])
def test_sizes(n3m, n2m, pad):
    import torch
    f = Field(n3m, n2m, pad, n3m + n2m)
    for _ in range(2):
        f.out.fill_(-1.0)
        f.launch()
        torch.cuda.synchronize()
        f.check()
    f.d["q3"][n3m, n2m - 1] = float("nan")   # the last cell
    f.launch()
    torch.cuda.synchronize()
    assert f.out.cpu().numpy()[0] == float("inf")


def test_many_calls_of_changing_size():
    import torch
    fields = [Field(n3m, n2m, 0, n3m) for n3m, n2m in ((700, 30), (3, 500), (296, 64), (40, 40), (1000, 9))]
    for i in range(150):
        f = fields[i % 5]
        f.out.fill_(-1.0)
        f.launch()
        if i % 7 == 0 or i > 140:
            torch.cuda.synchronize()
            f.check()


def test_captured_call_clears_its_counter():
    """A replayed call starts from a cleared completion counter whatever an
    overlapping call has left in it: the graph clears it ahead of the kernel."""
    import torch
    rt = pytest.importorskip("cuda.bindings.runtime")
    f = Field(500, 300, 0, 1)
    f.launch()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        f.launch(torch.cuda.current_stream().cuda_stream)
    raw = rt.cudaGraph_t(init_value=int(g.raw_cuda_graph()))
    err, _, n = rt.cudaGraphGetNodes(raw, 0)
    err, nodes, n = rt.cudaGraphGetNodes(raw, n)
    kinds = [rt.cudaGraphNodeGetType(x)[1] for x in nodes]
    assert sorted(k.name for k in kinds) == ["cudaGraphNodeTypeKernel", "cudaGraphNodeTypeMemset"]
    g.instantiate()
    for _ in range(3):
        f.out.fill_(-1.0)
        g.replay()
        f.launch()          # calls between replays
        f.out.fill_(-1.0)
        g.replay()
        torch.cuda.synchronize()
        f.check()
