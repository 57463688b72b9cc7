"""The time step's INT8 transforms: 7 balanced base-256 digits per operand
(oracle/i8x8.py, ``gemm_balanced``).

Error bound of the scheme, per product term and relative to 2^(e + f): each
operand is rounded to half a unit of 2^-55 (2^-56; |a| < 1), the six dropped
digit pairs of the leading weight are at most 6 * 2^14 * 2^-70 and those below
it 5/256 of that and so on, in all under 9 * 2^-56; the seven FP64 additions and
the conversion round partial sums of at most sum |a||b|.  2^e is at most
2 / 0.994 of the row maximum.
"""
import numpy as np
import pytest

from oracle import i8x8


def _operands(M, N, K, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((M, K)) * np.exp(rng.uniform(-5, 5, (M, 1)))
    B = rng.standard_normal((N, K)) * np.exp(-rng.uniform(0, 6, (N, K)))
    A[0] = 0.0
    A[1] = np.sign(A[1]) * (1.0 - 2.0 ** -53)     # largest mantissas: the leading digit's edge
    A[2] = -np.abs(A[2]).max() * 0.996
    return A, B


@pytest.mark.parametrize("M,N,K", [(40, 30, 77), (64, 48, 1024)])
def test_balanced_product_error(M, N, K):
    A, B = _operands(M, N, K, M + N + K)
    for X in (A, B):
        e, D = i8x8.balanced_digits(X)
        assert all(d.min() >= -128 and d.max() <= 127 for d in D)
        back = sum(d.astype(np.longdouble) * 2.0 ** -(8 * i + 7) for i, d in enumerate(D))
        assert np.all(np.abs(back - X * np.ldexp(1.0, -e)[:, None]) <= 2.0 ** -56)
    ref = A.astype(np.longdouble) @ B.T.astype(np.longdouble)
    err = np.abs(i8x8.gemm_balanced(A, B) - ref)
    top = np.abs(A).max(axis=1)[:, None] * np.abs(B).max(axis=1)[None, :] * (2.0 / 0.994) ** 2
    assert np.all(err <= K * top * 9 * 2.0 ** -56 + 8 * 2.0 ** -53 * (np.abs(A) @ np.abs(B).T))
    # not worse than the 8 sign-magnitude digits it replaces
    assert np.linalg.norm(err.astype(float)) <= np.linalg.norm((i8x8.gemm(A, B) - ref).astype(float))


@pytest.mark.gpu
@pytest.mark.parametrize("width", [16, 32, 48, 64])
@pytest.mark.parametrize("n3m,n2m", [(48, 32), (131, 90), (257, 129)])
def test_step_transform_equals_restatement(n3m, n2m, width, tmp_path, monkeypatch):
    """One transform of the step (one to three k-blocks: pairs of digit slices
    that straddle k-blocks, an odd last slice) gives the restatement's bits."""
    import fribois2d_b200 as fb
    from fribois2d_b200 import case as cases
    monkeypatch.setenv("FRIBOIS2D_I8_TILE", str(width))
    c = cases.viv_cylinder(n3m=n3m, n2m=n2m, h=3.0 / (n3m // 2), zwin=(-1.0, 2.0),
                           ywin=(-1.5 * (n2m // 2) / (n3m // 2), 1.5 * (n2m // 2) / (n3m // 2)),
                           zdom=(-3.0, 9.0), ydom=(-3.0, 3.0), nlm=40)
    s = fb.Solver(c.write(str(tmp_path / "deck")))
    rng = np.random.default_rng(width)
    for f in ("q2", "q3"):
        s.set(f, s.get(f) + 0.1 * rng.standard_normal((c.n3m + 2, c.n2m + 1)))
    s.set_substep(2, 1)
    for stage in ("divg", "i8_split", "i8x8_gemm"):
        assert s.stage(stage) == 0
    dph = s.get("dph")[1:n3m + 1, :n2m]
    hmn = s.get("hmn").reshape(n3m, -1)[:, :n2m]
    np.testing.assert_array_equal(hmn, i8x8.gemm_balanced(np.ascontiguousarray(dph.T), s.get("zmmt")).T)
    s.close()
