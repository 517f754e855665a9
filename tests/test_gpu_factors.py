"""The GPU factor construction's ordering on the device against the host construction, array for
array: rows and columns with lists past one warp's, more entries than the first room, one row, and
arrays large enough for the staged copies."""
import time

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


def test_large_factors_do_not_stay_on_the_device():
    """Between the two calls: factors past 512 MB wait in host memory, smaller ones on the device, and the
    second call copies either out as the host construction has them."""
    import ctypes as C

    import torch

    def sizes_only(A):
        ng, nh = C.c_int(0), C.c_int(0)
        FB._check(FB.lib().fiim_pdfiim_build_gpu(
            C.c_int(len(A[0]) - 1), FB._ptr(A[0]), FB._ptr(A[1]), FB._ptr(A[2]), C.c_int(1), C.c_int(1), C.c_int(1),
            C.c_double(0.05), C.c_int(-1), C.c_char(b"I"), C.c_char(b"B"), C.byref(ng), C.byref(nh),
            None, None, None, None, None, None, None))
        return 12 * (ng.value + nh.value)

    FB.pdfiim_build(FB.gen_poisson2d(40, 37), 0.05, 1, 1, 1, gpu=True)   # modules and pinned buffers
    for side, large in ((64, False), (184, True)):
        A = FB.gen_convdiff3d(side, 0.5)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        held = sizes_only(A)
        after = torch.cuda.mem_get_info()[0]
        assert (held > 512 << 20) == large
        assert before - after <= (4 << 20 if large else held + (32 << 20))
        same(A, 0.05, 1, 1, 1)
        assert before - torch.cuda.mem_get_info()[0] <= 4 << 20


def test_little_device_memory():
    """With the rest of the device taken: where only A, A^T and the entries fit, the first run counts, the
    second fills and the host orders, to the same arrays; where those do not fit, an error."""
    import torch
    A = FB.gen_convdiff3d(72, 0.4)
    n, nnz = 72 ** 3, len(A[1])
    host = same(A, 0.05, 2, 2, 1)
    entries = 12 * (len(host["Gj"]) + len(host["Hj"]))
    matrices = 24 * nnz + 60 * n
    assert 12 * 4 * (nnz + n) > entries + (16 << 20)     # the first room does not fit below
    for keep in (matrices + entries + (16 << 20), matrices // 2):
        torch.cuda.synchronize()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device="cuda")
        try:
            if keep > matrices:
                gpu = FB.pdfiim_build(A, 0.05, 2, 2, 1, gpu=True)
                assert all(np.array_equal(host[k], gpu[k]) for k in host)
            else:
                with pytest.raises(FB.FiimError, match="allocation"):
                    FB.pdfiim_build(A, 0.05, 2, 2, 1, gpu=True)
        finally:
            del hog
            torch.cuda.empty_cache()


def band(n, dense_column):
    """A band of four diagonals, with or without a first column that every row has."""
    i = np.arange(n)
    cols = np.stack([np.zeros(n, np.int64) if dense_column else i - 2, i - 1, i, i + 2], axis=1)
    keep = np.stack([i > 1, i > 0, i >= 0, i + 2 < n], axis=1)
    v = np.where(cols == i[:, None], 6.0, 0.4)
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    return rp, cols[keep].astype(np.int32), v[keep]


def test_a_list_of_many_thousand_entries():
    """Keys of three bytes, sorted in as many passes."""
    A = band(70001, True)
    assert np.bincount(A[1])[0] == 70001 and len(A[1]) > 1 << 16
    same(A, 0.001, 1, 1, 1)


def test_a_dense_column_costs_what_its_entries_do():
    """1.5 M rows: the ordering of one list with an entry a row is linear, so the construction takes no
    more than a few times what the band takes without that column (comparing all pairs: 40 times)."""
    times = {}
    for dense in (False, True):
        A = band(1_500_000, dense)
        t = []
        for _ in range(4):
            t0 = time.perf_counter()
            FB.pdfiim_build(A, 0.001, 1, 1, 1, gpu=True)
            t.append(time.perf_counter() - t0)
        times[dense] = min(t)
    assert times[True] < 8 * times[False], times
