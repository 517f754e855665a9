"""Block products over rows of every kind (runs of empty rows, rows around 8 and 32 entries, rows longer
than a warp's share, unsorted columns) and every number of right-hand sides a lane mapping ends at, column
by column against the oracle, bit for bit; the long sums of the fused dot products through the true
residual."""
import numpy as np
import pytest

import fiim_b200 as FB
import pyoracle as O
from test_gpu_batch import rounded
from test_gpu_products import rows_of

pytestmark = pytest.mark.gpu

LENGTHS = {
    "empty": lambda n, r: np.where(np.arange(n) % 71 == min(n - 1, 3), 2, 0),
    "edges": lambda n, r: r.choice([0, 1, 7, 8, 9, 31, 32, 33, 64], n),
    "uneven": lambda n, r: np.where(r.random(n) < 0.004, 3000, r.integers(0, 9, n)),
}


@pytest.mark.parametrize("kind", sorted(LENGTHS))
@pytest.mark.parametrize("n,k", [(1, 17), (33, 32), (900, 31), (6011, 1), (6011, 4), (6011, 9), (6011, 17), (6011, 32)])
def test_block_products_over_row_lengths(kind, n, k):
    r = np.random.default_rng(n + k)
    A, G, H = (rows_of(LENGTHS[kind](n, r), n, s) for s in (1, 2, 3))
    F = {"Gi": G[0], "Gj": G[1], "Gv": G[2], "IDv": r.standard_normal(n), "Hi": H[0], "Hj": H[1], "Hv": H[2]}
    X = r.standard_normal((n, k))
    X[n // 2, k // 2] = np.nan if n > 40 else 1.0
    for precision in ("fp64", "fp32"):
        S = FB.BlockSolver(A, F, k, precision=precision)
        Fr = rounded(F, precision)
        for op, ref in (("A", lambda u: O.csr_mv(*A, u)), ("M", lambda u: O.prec_apply(Fr, u))):
            want = np.stack([ref(np.ascontiguousarray(X[:, j])) for j in range(k)], axis=1)
            assert np.array_equal(S.apply(X, np.full((n, k), 7.0), op=op), want, equal_nan=True), (precision, op)
        S.close()


@pytest.mark.parametrize("n,k", [(5, 32), (1031, 17), (20011, 32), (20011, 3)])
def test_block_reductions_cover_every_row(n, k):
    """A = I + small uneven rows, M = I: the solve's true residual (a sum over all rows, taken on the
    device) equals the one formed here to the rounding of two sums of n terms, 2 n 2^-53 < 1e-11 each
    squared term, and the solution reaches the tolerance."""
    r = np.random.default_rng(n)
    lengths = LENGTHS["uneven"](n, r) if n > 100 else np.full(n, 2)
    rp, ci, v = rows_of(np.minimum(lengths, n) + 1, n, 7)
    v *= 0.2 / np.repeat(np.diff(rp), np.diff(rp))
    ci[rp[:-1]], v[rp[:-1]] = np.arange(n), 1.0
    one = np.arange(n + 1, dtype=np.int32)
    I = (one, one[:-1].copy(), np.ones(n))
    F = {"Gi": I[0], "Gj": I[1], "Gv": I[2], "IDv": np.ones(n), "Hi": I[0], "Hj": I[1], "Hv": I[2]}
    S = FB.BlockSolver((rp, ci, v), F, k)
    B, X = r.standard_normal((n, k)), np.zeros((n, k))
    res = S.solve(B, X, tol=1e-6, nmax=200)
    S.close()
    for j in range(k):
        b = np.ascontiguousarray(B[:, j])
        rel = np.linalg.norm(b - O.csr_mv(rp, ci, v, np.ascontiguousarray(X[:, j]))) / np.linalg.norm(b)
        assert res["info"][j] == 0 and rel < 1e-5
        assert abs(res["true_relres"][j] - rel) <= 1e-9 * rel + 1e-15


@pytest.mark.parametrize("shape", [None, "8,4", "16,2"])
@pytest.mark.parametrize("n,k", [(1, 4), (33, 1), (900, 16), (6011, 4), (6011, 9), (6012, 16), (70001, 3), (6011, 32)])
def test_rows_dealt_out_to_the_warps(monkeypatch, shape, n, k):
    """Matrices of even rows (one step of a warp after another, the last one partly filled) beside an
    uneven one (chunks): the same products, in every shape that serves k."""
    if shape:
        if k % int(shape.split(",")[1]):
            pytest.skip("the shape's vector width does not divide k")
        monkeypatch.setenv("FIIM_BLOCK_SHAPE", shape)
    r = np.random.default_rng(n + k)
    even = np.full(n, 7)
    A, G, H = rows_of(even, n, 1), rows_of(even, n, 2), rows_of(LENGTHS["uneven"](n, r), n, 3)
    F = {"Gi": G[0], "Gj": G[1], "Gv": G[2], "IDv": r.standard_normal(n), "Hi": H[0], "Hj": H[1], "Hv": H[2]}
    X = r.standard_normal((n, k))
    for precision in ("fp64", "fp32"):
        S = FB.BlockSolver(A, F, k, precision=precision)
        Fr = rounded(F, precision)
        for op, ref in (("A", lambda u: O.csr_mv(*A, u)), ("M", lambda u: O.prec_apply(Fr, u))):
            want = np.stack([ref(np.ascontiguousarray(X[:, j])) for j in range(k)], axis=1)
            assert np.array_equal(S.apply(X, np.full((n, k), 7.0), op=op), want), (precision, op)
        S.close()
