"""The sliced forms of the solver's matrices: every way a matrix can be laid out gives the
CSR streams' products bit for bit (rows are summed in storage order in all of them), at sizes
around the slices' edges, with shared and with own blocks, and for vectors with infinities
and NaN, which must reach only the rows that have an entry there."""
import numpy as np
import pytest

import fiim_b200 as FB
import pyoracle as O
from test_gpu_solve import identity_factors

pytestmark = pytest.mark.gpu


def banded(n, offsets, value, drop=0.0, seed=0):
    """CSR with the diagonals `offsets`, entry value(row, offset), a share `drop` of the off-diagonal
    entries left out at random."""
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), len(offsets))
    d = np.tile(np.asarray(sorted(offsets)), n)
    keep = (rows + d >= 0) & (rows + d < n) & ((d == 0) | (rng.random(len(d)) >= drop))
    rows, d = rows[keep], d[keep]
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return rp.astype(np.int32), (rows + d).astype(np.int32), value(rows, d)


def product(A, u, monkeypatch, **env):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    n = len(A[0]) - 1
    with FB.Solver(A, identity_factors(n)) as S:
        y = S.apply(u, np.zeros(n), op="A")
        form = S.spmv_shape(0)[1]
    for k in env:
        monkeypatch.delenv(k)
    return y, form


def same(a, b):
    return np.array_equal(a, b, equal_nan=True)


KINDS = {
    # the same values in every row: all inner slices are one class
    "constant": lambda i, d: np.where(d == 0, 7.5, -1.0 - 0.25 * (d > 0)),
    # every slice differs
    "varying": lambda i, d: np.where(d == 0, 7.5, -1.0) + 1e-3 * np.sin(i * 1.7 + d),
    # two materials: a few hundred rows each
    "layers": lambda i, d: np.where(d == 0, 7.5, -1.0) * (1.0 + (i // 300) % 2),
}


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 1000, 4097])
def test_banded_products(monkeypatch, kind, n):
    offsets = [o for o in (-100, -33, -8, -1, 0, 1, 8, 32, 101) if abs(o) < n]
    A = banded(n, offsets, KINDS[kind])
    u = np.random.default_rng(n).standard_normal(n)
    ref = O.csr_mv(*A, u)
    for env in ({}, {"FIIM_DIA_SHARE": "0"}, {"FIIM_DIA_R": "1"}, {"FIIM_DIA_R": "2"}, {"FIIM_DIA": "0"}):
        y, form = product(A, u, monkeypatch, **env)
        assert same(y, ref), (env, form)


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_nonfinite_vector_entries(monkeypatch, kind, bad):
    """An infinity or NaN in the vector reaches exactly the rows with an entry in its column,
    whatever the padding of the slices around it."""
    n = 2000
    A = banded(n, (-45, -1, 0, 1, 44), KINDS[kind], drop=0.1, seed=3)
    u = np.random.default_rng(1).standard_normal(n)
    u[[0, 31, 32, 700, n - 1]] = bad
    ref = O.csr_mv(*A, u)
    assert np.isfinite(ref).sum() > n - 40
    for env in ({}, {"FIIM_DIA_SHARE": "0"}, {"FIIM_DIA": "0"}):
        y, form = product(A, u, monkeypatch, **env)
        assert same(y, ref), (env, form)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 1000, 4099])
@pytest.mark.parametrize("width,drop", [(9, 0.5), (33, 0.6), (64, 0.62), (65, 0.6)])
def test_packed_products(monkeypatch, n, width, drop):
    """Rows that hold a random part of 9 to 65 diagonals (a slice's records in one or two loads;
    65 in a full slice are one too many): packed slices where they serve, the same bits anyway,
    also with infinities in the vector."""
    rng = np.random.default_rng(width)
    offsets = [0] + [int(o) for o in rng.permutation(np.r_[-40:0, 1:41])[:width - 1]]
    A = banded(n, offsets, KINDS["varying"], drop=drop, seed=n)
    u = np.random.default_rng(n).standard_normal(n)
    u[n // 2] = np.inf
    ref = O.csr_mv(*A, u)
    forms = set()
    for env in ({}, {"FIIM_PACK": "0"}, {"FIIM_DIA": "0"}):
        y, form = product(A, u, monkeypatch, **env)
        forms.add(form)
        assert same(y, ref), (env, form)
    if n >= 1000 and width <= 64:
        assert 4 in forms
    if n >= 1000 and width == 65:
        assert 4 not in forms


def uneven_system(c=40):
    """3D convection-diffusion with a random coefficient field: the factors' slices do not share their
    diagonals closely (packed slices)."""
    A = FB.gen_convdiff3d(c, 0.5)
    n = c ** 3
    d = np.exp(0.5 * np.random.default_rng(2).standard_normal(n))
    A = (A[0], A[1], A[2] * d[A[1]] / d[np.repeat(np.arange(n), np.diff(A[0]))])
    return A, FB.pdfiim_build(A, 0.05, 2, 2, 1)


def test_packed_reload():
    """Drop-in calls over a system whose factors are served by packed slices: new values in the same
    structure, then other columns with the same row offsets; each equals a fresh solver's result
    bit for bit."""
    A, F = uneven_system()
    n = len(A[0]) - 1
    H = (F["Hi"], F["Hj"], F["Hv"])
    b = FB.rand_normal(n, 3)
    # other columns, the same row lengths: each row's second entry moves one column on where that is free
    moved = H[1].copy()
    first = H[0][:-1][np.diff(H[0]) > 2] + 1
    free = moved[first] + 1 < moved[first + 1]
    moved[first[free]] += 1
    assert free.sum() > 100
    prev = FB.dropin_cache(False)
    try:
        for Hj, Hv in ((H[1], H[2]), (H[1], H[2] * 1.25), (moved, H[2]), (H[1], H[2])):
            FF = dict(F, Hj=Hj, Hv=Hv)
            with FB.Solver(A, FF, variant="pdfiim") as S:
                y = np.zeros(n)
                r1 = S.solve(b, y, tol=1e-10, nmax=60)
                assert S.spmv_shape(2)[1] == 4
            x = np.zeros(n)
            r = FB.EPBiCGSTAB_pdfiim(A, b, 1e-10, 60, (F["Gi"], F["Gj"], F["Gv"]), F["IDv"], (H[0], Hj, Hv), x)
            assert np.array_equal(x, y, equal_nan=True) and r[1] == r1["iter"]
    finally:
        FB.dropin_cache(prev)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
def test_batch_with_and_without_shared_blocks(monkeypatch, precision):
    """A batch's solves with shared blocks and with every slice's own: the products are the same
    bits and the per-slice partial sums are grouped alike or by rows of the same slice, so the
    runs agree system by system to rounding, as do their iteration counts."""
    systems, bs = [], []
    for k, side in enumerate((9, 16, 33, 40)):
        A = FB.gen_convdiff2d(side, 1.0 + k, 0.3 * k, 0.5)
        systems.append((A, FB.pdfiim_build(A, 0.05, 2, 2, 1)))
        bs.append(FB.rand_normal(side * side, 40 + k))
    b, out = np.concatenate(bs), {}
    for share in ("1", "0"):
        monkeypatch.setenv("FIIM_DIA_SHARE", share)
        with FB.BatchSolver(systems, variant="pdfiim", precision=precision) as S:
            x = np.zeros(len(b))
            out[share] = (S.solve(b, x, tol=1e-10, nmax=500), x)
    assert np.array_equal(out["1"][0]["info"], out["0"][0]["info"]) and not out["1"][0]["info"].any()
    assert np.all(np.abs(out["1"][0]["iter"] - out["0"][0]["iter"]) <= 2)
    assert np.linalg.norm(out["1"][1] - out["0"][1]) <= 1e-7 * np.linalg.norm(out["0"][1])


def test_entries_outside_the_triangles_of_a_large_system():
    """G with entries below its diagonal and H with entries above: the solver reads the triangles only,
    through the sliced copies laid out of what is left, bit for bit as if they were given alone."""
    side = 48
    A = FB.gen_convdiff3d(side, 0.5)
    n = side ** 3
    F = FB.pdfiim_build(A, 0.05, 2, 2, 1)

    def widened(rp, ci, v, upper):
        rows = np.repeat(np.arange(n), np.diff(rp))
        other = np.arange(side, n) if upper else np.arange(n - side)      # one entry on the other side
        r = np.concatenate([rows, other])
        c = np.concatenate([ci, other - side if upper else other + side])
        w = np.concatenate([v, np.full(len(other), 3.0)])
        order = np.lexsort((c, r))
        ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
        return ptr, c[order].astype(np.int32), w[order]

    G, H = widened(F["Gi"], F["Gj"], F["Gv"], True), widened(F["Hi"], F["Hj"], F["Hv"], False)
    W = dict(F, Gi=G[0], Gj=G[1], Gv=G[2], Hi=H[0], Hj=H[1], Hv=H[2])
    b, out = FB.rand_normal(n, 9), []
    for f in (F, W):
        with FB.Solver(A, f, variant="pdfiim") as S:
            x = np.zeros(n)
            r = S.solve(b, x, tol=1e-10, nmax=300)
            out.append((r["iter"], x, S.spmv_shape(1)[1], S.spmv_shape(2)[1]))
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1]) and out[0][2:] == out[1][2:] == (3, 3)


def stencil(sides, points, kind):
    """The 7-, 19- or 27-point stencil on a box, with constant or varying entries."""
    nx, ny, nz = sides
    n = nx * ny * nz
    i = np.arange(n)
    at = (i // (nx * ny), i // nx % ny, i % nx)
    steps = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)
             if abs(a) + abs(b) + abs(c) <= {7: 1, 19: 2, 27: 3}[points]]
    inside = np.stack([np.all([(0 <= q + d) & (q + d < m) for q, d, m in zip(at, s, (nz, ny, nx))], axis=0)
                       for s in steps], axis=1)
    cols = np.stack([i + (s[0] * ny + s[1]) * nx + s[2] for s in steps], axis=1)
    v = np.stack([np.where(s == (0, 0, 0), 30.0, -1.0 / (1 + sum(map(abs, s)))) + 0.0 * i for s in steps], axis=1)
    if kind == "varying":
        v *= 1.0 + 0.1 * np.sin(0.7 * np.arange(n))[:, None]
    rp = np.concatenate([[0], np.cumsum(inside.sum(1))]).astype(np.int32)
    return rp, cols[inside].astype(np.int32), v[inside]


# the last box: several slices a warp of the products' grid
BOXES = [(37, 41, 23), (33, 32, 32), (67, 64, 63)]


def solves(monkeypatch, A, envs):
    """(iterations, x) of one solve with A served as each environment says."""
    n = len(A[0]) - 1
    b, out = FB.rand_normal(n, 5), []
    for env in envs:
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        x = np.full(n, 0.25)
        with FB.Solver(A, identity_factors(n)) as S:
            r = S.solve(b, x, tol=1e-11, nmax=100)
            assert S.spmv_shape(0)[1] == 3 and S.mode() < 2, env
        for k in env:
            monkeypatch.delenv(k)
        assert r["info"] == 0
        out.append((r["iter"], x))
    return b, out


@pytest.mark.parametrize("kind", ["constant", "varying"])
@pytest.mark.parametrize("sides", BOXES, ids=lambda s: "x".join(map(str, s)))
def test_sharing_leaves_the_iterates_alone(monkeypatch, sides, kind):
    """Seven diagonals: with shared blocks (one and two rows a lane) and with a block a slice, the sums that
    steer the solve have one tree, so x is the same bit for bit."""
    envs = ({}, {"FIIM_DIA_SHARE": "0"}, {"FIIM_DIA_R": "1"}, {"FIIM_DIA_SHARE": "0", "FIIM_DIA_R": "1"})
    _, out = solves(monkeypatch, stencil(sides, 7, kind), envs)
    for env, (its, x) in zip(envs[1:], out[1:]):
        assert its == out[0][0] and np.array_equal(x, out[0][1]), env


@pytest.mark.parametrize("points", [19, 27])
@pytest.mark.parametrize("sides", BOXES, ids=lambda s: "x".join(map(str, s)))
def test_wide_stencils_with_and_without_sharing(monkeypatch, sides, points):
    """More than eight diagonals: a block a slice means two rows a lane and another tree. Both solutions
    leave a residual below 1e-11 of the start's, and the symmetric A has 30 on its diagonal and at most 9
    beside it, so its inverse is at most 1 / 21: they differ by no more than twice that. One row a lane has
    the shared blocks' tree."""
    A = stencil(sides, points, "constant")
    n = len(A[0]) - 1
    b, out = solves(monkeypatch, A, ({}, {"FIIM_DIA_SHARE": "0"}, {"FIIM_DIA_SHARE": "0", "FIIM_DIA_R": "1"}))
    r0 = np.linalg.norm(b - O.csr_mv(*A, np.full(n, 0.25)))
    assert np.linalg.norm(out[0][1] - out[1][1]) <= 2 * 1e-11 * r0 / 21 + 1e-13 * np.linalg.norm(out[0][1])
    assert out[2][0] == out[0][0] and np.array_equal(out[2][1], out[0][1])


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("n", [1000, 4097])
def test_banded_matrices_are_served_by_the_sliced_copy(monkeypatch, kind, n):
    """Nine diagonals over full rows: form 3, with shared blocks (fewer bytes than the values) where every
    row is alike and a block a slice where none are; the CSR streams only where they are asked for."""
    A = banded(n, (-100, -33, -8, -1, 0, 1, 8, 32, 101), KINDS[kind])
    with FB.Solver(A, identity_factors(n)) as S:
        assert S.spmv_shape(0)[1] == 3
        if kind != "layers":
            assert (S.matrix_bytes(0) < 8 * len(A[1])) == (kind == "constant")
    for env in ("FIIM_DIA_SHARE", "FIIM_DIA"):
        monkeypatch.setenv(env, "0")
        with FB.Solver(A, identity_factors(n)) as S:
            assert S.spmv_shape(0)[1] == (3 if env == "FIIM_DIA_SHARE" else 0)
            assert S.matrix_bytes(0) >= 8 * len(A[1])
        monkeypatch.delenv(env)
