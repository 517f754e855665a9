"""The reference-facing call over changing systems: one thread's solver is set up again in place for
another shape and reused for the same one, and every call equals a fresh solver's result bit for
bit, with the device-copy reuse on and off, from one thread and from several."""
import threading

import numpy as np
import pytest

import fiim_b200 as FB

pytestmark = pytest.mark.gpu


def system(kind):
    """Shapes that grow, shrink and change their layout: cluster-sized, mid-sized, symmetric storage."""
    side, seed = kind
    A = FB.gen_convdiff3d(side, 0.3 + 0.05 * seed)
    F = FB.pdfiim_build(A, 0.05, 2, 2, 1)
    return A, F, FB.rand_normal(side ** 3, seed)


KINDS = [(12, 1), (40, 2), (33, 3), (12, 4), (40, 5), (40, 2), (36, 6), (12, 1)]


def check(systems):
    for A, F, b in systems:
        n = len(b)
        with FB.Solver(A, F, variant="pdfiim") as S:
            y = np.zeros(n)
            r1 = S.solve(b, y, tol=1e-10, nmax=500)
        x = np.zeros(n)
        r = FB.EPBiCGSTAB_pdfiim(A, b, 1e-10, 500, (F["Gi"], F["Gj"], F["Gv"]), F["IDv"],
                                 (F["Hi"], F["Hj"], F["Hv"]), x)
        assert r[2] == r1["info"] == 0 and r[1] == r1["iter"] and np.array_equal(x, y)


@pytest.mark.parametrize("cache", [True, False])
def test_changing_shapes(cache):
    prev = FB.dropin_cache(cache)
    try:
        check([system(k) for k in KINDS])
    finally:
        FB.dropin_cache(prev)


def test_same_arrays_other_addresses():
    """The same system in other arrays, then the first arrays changed in place, then as they were."""
    A, F, b = system((34, 7))
    prev = FB.dropin_cache(True)
    try:
        copies = (tuple(a.copy() for a in A), {k: v.copy() for k, v in F.items()}, b)
        check([(A, F, b), copies, (A, F, b)])
        A[2][7] *= 1.5
        check([(A, F, b), copies])
    finally:
        FB.dropin_cache(prev)


def test_threads():
    errors = []

    def work(seed):
        try:
            check([system((20 + 8 * (seed % 3), seed)), system((34, seed)), system((16, seed))])
        except BaseException as e:   # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_a_thread_that_moves_to_another_device():
    """The same shape again after the thread's current device changed: solved there, and left current."""
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    s = system((33, 3))
    try:
        for dev in (0, 1, 0):
            torch.cuda.set_device(dev)
            before = torch.cuda.mem_get_info(dev)[0]
            check([s])
            assert torch.cuda.current_device() == dev
            if dev == 1:
                assert torch.cuda.mem_get_info(dev)[0] < before
    finally:
        torch.cuda.set_device(0)


PADDING = np.uint64(0xFFF7D1A6B00C5A1D).view(np.float64)   # a NaN: the sliced copies' mark of an empty slot


@pytest.mark.parametrize("points", [7, 19, 27])
def test_reloads_choose_the_form_a_fresh_solver_would(points):
    """One structure, its entries varying, constant and varying again, with and without an entry that holds
    the sliced copies' padding pattern: the kept solver takes the new values in the form that a fresh one
    would choose for them (shared blocks, a block a slice, the CSR streams), whose sums have different trees
    in part, so x is the fresh solver's bit for bit."""
    from test_gpu_slices import stencil
    from test_gpu_solve import identity_factors
    sides = (41, 37, 33)
    A = {kind: stencil(sides, points, kind) for kind in ("varying", "constant")}
    n = len(A["varying"][0]) - 1
    F, b = identity_factors(n), FB.rand_normal(n, 11)
    rng = np.random.default_rng(3)
    for kind in ("varying", "constant"):
        rp, ci, v = A[kind]
        v = v.copy()
        v[rng.integers(len(v))] = PADDING
        A[kind + " pad"] = (rp, ci, v)
        A[kind + " other"] = (rp, ci, A[kind][2] * 1.25)
    order = ["varying", "constant", "varying other", "varying pad", "varying", "constant pad", "constant",
             "constant other", "varying pad", "constant"]
    prev = FB.dropin_cache(False)
    try:
        for step, kind in enumerate(order):
            with FB.Solver(A[kind], F, variant="pdfiim") as S:
                y = np.full(n, 0.25)
                r1 = S.solve(b, y, tol=1e-9, nmax=60)
            x = np.full(n, 0.25)
            r = FB.EPBiCGSTAB_pdfiim(A[kind], b, 1e-9, 60, (F["Gi"], F["Gj"], F["Gv"]), F["IDv"],
                                     (F["Hi"], F["Hj"], F["Hv"]), x)
            assert np.array_equal(x, y, equal_nan=True) and r[1] == r1["iter"], (step, kind)
    finally:
        FB.dropin_cache(prev)


def test_a_smaller_system_gives_the_larger_ones_memory_back():
    """After a large system, a small one leaves no more on the device than 64 MB beyond its own."""
    import torch
    small, large = system((12, 1)), system((72, 2))
    free = []
    for s in (small, large, small):
        check([s])
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[1] > 100 << 20          # the large one's arena
    assert free[0] - free[2] <= 68 << 20


@pytest.mark.parametrize("points", [7, 27])
def test_reloads_into_shared_blocks(points):
    """Constant and layered entries, scaled, split into more kinds of slices and merged again: shared blocks
    take new values where the slices that share them stay alike, and are laid out again where not; x is a
    fresh solver's bit for bit."""
    from test_gpu_slices import stencil
    from test_gpu_solve import identity_factors
    A0 = stencil((41, 37, 33), points, "constant")
    n = len(A0[0]) - 1
    rows = np.repeat(np.arange(n), np.diff(A0[0]))
    layer = lambda k: 1.0 + (rows // (n // k + 1)) % 2   # noqa: E731
    values = [A0[2], A0[2] * 1.25, A0[2] * layer(5), A0[2] * layer(5) * 0.75, A0[2], A0[2] * layer(9),
              A0[2] * np.where(rows == 20011, 1.5, 1.0), A0[2] * 1.5]
    F, b = identity_factors(n), FB.rand_normal(n, 12)
    prev = FB.dropin_cache(False)
    try:
        for step, v in enumerate(values):
            A = (A0[0], A0[1], v)
            with FB.Solver(A, F, variant="pdfiim") as S:
                y = np.full(n, 0.25)
                r1 = S.solve(b, y, tol=1e-9, nmax=100)
                assert S.spmv_shape(0)[1] == 3 and S.matrix_bytes(0) < 8 * len(v)
            x = np.full(n, 0.25)
            r = FB.EPBiCGSTAB_pdfiim(A, b, 1e-9, 100, (F["Gi"], F["Gj"], F["Gv"]), F["IDv"],
                                     (F["Hi"], F["Hj"], F["Hv"]), x)
            assert r1["info"] == 0 and np.array_equal(x, y) and r[1] == r1["iter"], step
    finally:
        FB.dropin_cache(prev)
