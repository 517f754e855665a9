"""The GPU factor construction's ordering on the device against the host construction, array for
array: rows and columns with lists past one warp's, more entries than the first room, one row, and
arrays large enough for the staged copies."""
import numpy as np
import pytest

import fiim_b200 as FB

pytestmark = pytest.mark.gpu


def same(A, *args):
    host, gpu = FB.pdfiim_build(A, *args), FB.pdfiim_build(A, *args, gpu=True)
    for k in host:
        assert np.array_equal(host[k], gpu[k], equal_nan=True), k
    return host


def arrow(n, seed=0):
    """A dense first row and column over a band: row 0 of A^T and row 0 of G hold about n entries."""
    rng = np.random.default_rng(seed)
    rows = [sorted({0, max(i - 1, 0), i, min(i + 3, n - 1)}) if i else list(range(n)) for i in range(n)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    ci = np.concatenate(rows).astype(np.int32)
    v = rng.uniform(0.5, 1.0, len(ci))
    v[:n] = 0.1
    v[ci == np.repeat(np.arange(n), np.diff(rp))] = 6.0
    return rp, ci, v


@pytest.mark.parametrize("n", [1023, 1025, 5000])
def test_long_lists(n):
    F = same(arrow(n), 0.001, 1, 1, 1)
    assert np.diff(F["Gi"]).max() > 0.9 * n


def test_more_entries_than_the_first_room():
    A = FB.gen_poisson2d(40, 37)
    F = same(A, 0.0, 4, 1, 1)
    assert len(F["Gj"]) + len(F["Hj"]) > 4 * (len(A[1]) + 40 * 37)


@pytest.mark.parametrize("n", [1, 2, 33])
def test_small(n):
    same(FB.gen_poisson2d(n, 1), 0.05, 2, 2, 1)


@pytest.mark.parametrize("norm", ["I", "1", "2"])
def test_large_arrays(norm):
    same(FB.gen_convdiff3d(72, 0.4), 0.05, 2, 2, 1, -1, norm)


def test_many_rows_outgrow_both_smaller_capacities():
    """Five fill levels of the 7-point stencil reach up to 115 members: most of 21,952 rows are listed
    and built again at 64 and then at 128."""
    same(FB.gen_convdiff3d(28, 0.4), 0.02, 5, 1, 1)
