"""The kernel-level products without a lane count (one kernel for every matrix) against the oracle,
bit for bit: row lengths around the tile, runs of empty and of long rows, unsorted columns, and
entries outside the triangle."""
import numpy as np
import pytest
import torch

import fiim_b200 as FB
import pyoracle as O

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def rows_of(lengths, n, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    return rp, rng.integers(0, n, rp[-1]).astype(np.int32), rng.standard_normal(rp[-1])


LENGTHS = {
    "empty": lambda n, r: np.where(np.arange(n) % 7 == min(n - 1, 3), 2, 0),
    "short": lambda n, r: r.integers(0, 5, n),
    "tile": lambda n, r: r.choice([7, 8, 9, 255, 256, 257], n),      # tiles that end inside, at and after a row
    "long": lambda n, r: r.integers(200, 700, n),                     # a warp a row
    "uneven": lambda n, r: np.where(r.random(n) < 0.002, 5000, r.integers(1, 12, n)),
}


@pytest.mark.parametrize("kind", sorted(LENGTHS))
@pytest.mark.parametrize("n", [1, 31, 32, 33, 500, 40001])
def test_spmv_without_lanes(kind, n):
    r = np.random.default_rng(n)
    lengths = LENGTHS[kind](n, r)
    if lengths.sum() > 4_000_000:
        lengths = lengths[:n] // 8
    A = rows_of(lengths, n, n + 1)
    u = r.standard_normal(n)
    u[n // 2] = np.nan if n > 40 else 1.0
    y = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    FB.spmv(*[dev(a) for a in A], dev(u), y)
    assert np.array_equal(y.cpu().numpy(), O.csr_mv(*A, u), equal_nan=True)


@pytest.mark.parametrize("n,mean", [(1, 1), (33, 5), (700, 300), (20011, 6), (20011, 40)])
def test_prec_apply_filters_its_triangles(n, mean):
    """G and H with entries on both sides of the diagonal, columns in any order: only the upper (lower)
    ones count."""
    r = np.random.default_rng(n + mean)
    G, H = (rows_of(r.integers(0 if n > 1 else 1, 2 * mean + 1, n), n, s) for s in (1, 2))
    D, u = r.standard_normal(n), r.standard_normal(n)
    F = {"Gi": G[0], "Gj": G[1], "Gv": G[2], "IDv": D, "Hi": H[0], "Hj": H[1], "Hv": H[2]}
    want = O.prec_apply(F, u)
    z, tm = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    d = [dev(a) for a in (*G, D, *H, u)]
    FB.prec_apply(*d, z, tm)
    assert np.array_equal(z.cpu().numpy(), want)
    z.zero_()
    FB.prec_apply_noalloc(*d, z)
    assert np.array_equal(z.cpu().numpy(), want)
