"""Measured cases of the solve phase: factored-approximate-inverse preconditioned BiCGSTAB.

A program that uses this library has a sparse system and its factors G, D^-1, H. It calls
the kernel-level products, keeps a solver handle and solves many right-hand sides, solves many
small systems or many right-hand sides at once, calls the reference's function with host
arrays, or builds the factors. Each case here is one such call.

The matrices are the ones this repository's benchmark and tests use (3D convection-diffusion
with constant coefficients, batches of 2D convection-diffusion systems, power-law rows) and a 3D
diffusion-convection operator with a random coefficient field on boxes with three different
sides, which is what a program with measured material data has.

Right-hand sides are made from a known solution, b = A x, so a solve's exact answer is x.
Tolerances are tight enough (1e-10 to 1e-13) that two correct solves agree to far more
digits than a stopping test at 1e-8 would leave.
"""
import concurrent.futures
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "computational-mathematics_b200"))
import fiim_b200 as FB  # noqa: E402


def listed():
    return [
        # One product of a small system through the kernel-level call: all latency.
        {"name": "spmv_small", "kind": "spmv", "nx": 33, "ny": 31, "nz": 5},
        # One product with uneven random rows (power-law lengths, cap 512), an odd row count.
        {"name": "spmv_power", "kind": "spmv_power", "n": 400003, "mean": 16.0},
        # The preconditioner product of a box-shaped 3D system, kernel-level call.
        {"name": "prec_box", "kind": "prec", "nx": 127, "ny": 96, "nz": 101},
        # A small system from host arrays, one after another through one handle.
        {"name": "solve_small", "kind": "solve", "field": "constant", "nx": 24, "ny": 24, "nz": 24, "memory": "host"},
        # An ordinary system with a random coefficient field.
        {"name": "solve_mid", "kind": "solve", "field": "random", "nx": 61, "ny": 47, "nz": 53, "memory": "device"},
        # The benchmark's own system: 128^3, constant coefficients.
        {"name": "solve_cube", "kind": "solve", "field": "constant", "nx": 128, "ny": 128, "nz": 128,
         "memory": "device"},
        # As large, with a random coefficient field and three different odd sides.
        {"name": "solve_box", "kind": "solve", "field": "random", "nx": 131, "ny": 113, "nz": 127,
         "memory": "device"},
        # FP32 inner solve verified in FP64, random coefficient field.
        {"name": "mixed_fp32", "kind": "mixed", "precision": "fp32", "nx": 97, "ny": 101, "nz": 90},
        # Many uneven 2D systems in one call, factors stored in FP32, FP64-verified.
        {"name": "batch_2d", "kind": "batch", "systems": 48, "lo": 32, "hi": 128, "precision": "fp32"},
        # 32 right-hand sides of one system with power-law rows, factors stored in FP32.
        {"name": "block_power", "kind": "block", "n": 200003, "rhs": 32, "precision": "fp32"},
        # The reference's own call with plain host arrays: everything goes up, x comes back.
        {"name": "dropin_box", "kind": "dropin", "nx": 70, "ny": 64, "nz": 59},
        # The factor construction on the GPU, for a nearly homogeneous material (so that the kept
        # pattern, hence the outputs' sizes, does not move with the seed).
        {"name": "factors_box", "kind": "factors", "nx": 61, "ny": 57, "nz": 50, "spread": 0.001},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """Three different sides of a box of lo..hi cells."""
    side = math.exp(rng.uniform(math.log(lo), math.log(hi))) ** (1 / 3)
    a, b = rng.uniform(0.8, 1.2), rng.uniform(0.85, 1.15)
    return {"nx": max(2, int(side * a)), "ny": max(2, int(side * b)), "nz": max(2, int(side / (a * b)))}


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv_power", "prec", "solve", "solve", "solve", "mixed", "batch", "block",
                       "dropin", "factors"])
    if kind in ("spmv", "prec"):
        return {"kind": kind, **_box(rng, 3000, 1200000)}
    if kind == "spmv_power":
        return {"kind": kind, "n": _log(rng, 5000, 400000), "mean": round(rng.uniform(4.0, 16.0), 2)}
    if kind == "solve":
        field = rng.choice(["constant", "random"])
        if field == "constant":
            s = _log(rng, 12, 120)
            return {"kind": kind, "field": field, "nx": s, "ny": s, "nz": s,
                    "memory": "host" if s < 30 else "device"}
        return {"kind": kind, "field": field, **_box(rng, 4000, 1500000), "memory": "device"}
    if kind == "mixed":
        return {"kind": kind, "precision": rng.choice(["fp32", "fp32", "bf16"]), **_box(rng, 60000, 900000)}
    if kind == "batch":
        return {"kind": kind, "systems": rng.randint(5, 48), "lo": 16, "hi": rng.randint(40, 128),
                "precision": rng.choice(["fp64", "fp32"])}
    if kind == "block":
        return {"kind": kind, "n": _log(rng, 10000, 200000), "rhs": rng.choice([3, 8, 16, 24, 32]),
                "precision": rng.choice(["fp64", "fp32"])}
    if kind == "factors":
        return {"kind": kind, **_box(rng, 5000, 260000), "spread": 0.001}
    return {"kind": kind, **_box(rng, 5000, 260000)}


# ------------------------------------------------------------------ matrices
def _stencil(c, rng):
    """7-point operator -div(k grad u) + w . grad u (first-order upwind) on a box with Dirichlet
    walls, k lognormal per cell, harmonic means at the faces, scaled by h^2. Returns the
    coefficients (n, 7) in ascending column order and the mask of the ones inside the box."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    k = np.exp(c.get("spread", 0.5) * rng.standard_normal((nz, ny, nx)))
    pe = 0.5
    n = nx * ny * nz
    vals, mask = np.zeros((n, 7)), np.ones((n, 7), bool)
    diag = np.zeros((nz, ny, nx))
    for axis, (lo, hi) in enumerate(((0, 6), (1, 5), (2, 4))):   # z, y, x
        pad = [(1, 1) if a == axis else (0, 0) for a in range(3)]
        kp = np.pad(k, pad, mode="edge")
        sl = lambda o: tuple(slice(o, o + k.shape[a]) if a == axis else slice(None) for a in range(3))  # noqa: E731
        kl, kh = kp[sl(0)], kp[sl(2)]
        tl, th = 2 * k * kl / (k + kl), 2 * k * kh / (k + kh)
        vals[:, lo], vals[:, hi] = -(tl + pe).ravel(), -th.ravel()
        diag += tl + th + pe
        at = np.arange(k.shape[axis])
        shape = [-1 if a == axis else 1 for a in range(3)]
        mask[:, lo] = np.broadcast_to((at > 0).reshape(shape), k.shape).ravel()
        mask[:, hi] = np.broadcast_to((at < len(at) - 1).reshape(shape), k.shape).ravel()
    vals[:, 3] = diag.ravel()
    return vals, mask


def _csr(c, vals, mask, first=0, last=7):
    """CSR arrays of the stencil columns [first, last)."""
    nx, ny = c["nx"], c["ny"]
    offsets = np.array([-nx * ny, -nx, -1, 0, 1, nx, nx * ny])[first:last]
    m = mask[:, first:last]
    cols = np.arange(len(vals))[:, None] + offsets[None, :]
    rp = np.concatenate([[0], np.cumsum(m.sum(1))])
    return rp.astype(np.int32), cols[m].astype(np.int32), vals[:, first:last][m]


def _power(c, rng):
    """Random columns, row lengths from a power law (cap 512) with the asked mean, a dominant diagonal."""
    n, mean = c["n"], c.get("mean", 16.0)
    w = rng.pareto(1.0, n) + 1.0
    length = np.minimum(np.maximum(1, w * (mean / 6.5)), 512).astype(np.int64)
    rows = np.repeat(np.arange(n), length)
    keys = rows * n + rng.integers(0, n, len(rows))
    keys = np.unique(np.concatenate([keys, np.arange(n) * (n + 1)]))
    rows, cols = keys // n, keys % n
    v = -rng.uniform(0.2, 1.0, len(keys))
    v[rows == cols] = 0.0
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    v[rows == cols] = 1.0 - np.add.reduceat(v, rp[:-1])
    return rp.astype(np.int32), cols.astype(np.int32), v


def _mul(A, x):
    """A x of a CSR matrix without empty rows; x may have several columns."""
    rp, ci, v = A
    if x.ndim == 1:
        return np.add.reduceat(v * x[ci], rp[:-1])
    return np.stack([np.add.reduceat(v * x[ci, j], rp[:-1]) for j in range(x.shape[1])], axis=1)


def _cells(c):
    return c["nx"] * c["ny"] * c["nz"]


def _solution(c, seed):
    """The known solution of a case, the first numbers drawn from its seed."""
    rng = np.random.default_rng(seed)
    n = _cells(c) if "nx" in c else c["n"]
    return rng, rng.standard_normal((n, c["rhs"]) if "rhs" in c else n)


def _matrix(c, rng):
    if c.get("field") == "constant":
        return FB.gen_convdiff3d(c["nx"], 0.5)
    return _csr(c, *_stencil(c, rng))


def _pdfiim(A):
    return FB.pdfiim_build(A, 0.05, 2, 2, 1, -1, "I", "B", gpu=True)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _dev_csr(A):
    return tuple(_dev(a) for a in A)


def _dev_factors(F):
    return {k: _dev(v) for k, v in F.items()}


def _factors2(c, vals, mask):
    """One-term factors of the stencil: G = I - U / d, H = I - L / d, D^-1 = 1 / d."""
    s = vals / vals[:, 3:4]
    s[:, 3] = 1.0
    return _csr(c, s, mask, 3, 7), 1.0 / vals[:, 3], _csr(c, s, mask, 0, 4)


def _batch_sides(c, seed):
    """The systems' generator parameters: side, diffusion, angle, cell Peclet number."""
    rng = np.random.default_rng(seed)
    for k in range(c["systems"]):
        side = int(np.random.default_rng(k).integers(c["lo"], c["hi"] + 1))   # the shapes belong to the case
        yield side, float(10 ** rng.uniform(-1, 1)), float(rng.uniform(0, 2 * np.pi)), float(rng.uniform(0.3, 1.0))


def _batch_solution(c, seed):
    sides = [p[0] for p in _batch_sides(c, seed)]
    return np.random.default_rng([seed, 1]).standard_normal(sum(s * s for s in sides)), sides


# ------------------------------------------------------------------ the interface
def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        x, sides = _batch_solution(c, seed)

        def system(p):
            A = FB.gen_convdiff2d(*p)
            return A, FB.acifim_build(A, 0.1, 0.05)

        with concurrent.futures.ThreadPoolExecutor(max(1, os.cpu_count() or 1)) as pool:
            systems = list(pool.map(system, _batch_sides(c, seed)))
        at = np.concatenate([[0], np.cumsum([s * s for s in sides])])
        b = np.concatenate([_mul(s[0], x[at[k]:at[k + 1]]) for k, s in enumerate(systems)])
        S = FB.BatchSolver(systems, variant="acifim", precision=c["precision"], memory="device", verified=True)
        return {"kind": kind, "S": S, "b": _dev(b), "x": _dev(np.zeros_like(b))}
    rng, x = _solution(c, seed)
    if kind in ("spmv", "spmv_power"):
        A = _dev_csr(_power(c, rng) if kind == "spmv_power" else _matrix(c, rng))
        return {"kind": kind, "A": A, "x": _dev(x), "y": _dev(np.zeros_like(x))}
    if kind == "prec":
        G, D, H = _factors2(c, *_stencil(c, rng))
        return {"kind": kind, "G": _dev_csr(G), "D": _dev(D), "H": _dev_csr(H), "r": _dev(x),
                "z": _dev(np.zeros_like(x)), "t": _dev(np.zeros_like(x))}
    if kind == "factors":
        return {"kind": kind, "A": _matrix(c, rng)}
    if kind == "block":
        A = _power({"n": c["n"], "mean": 12.0}, rng)
        F = FB.pdfiim_build(A, 0.1, 1, 1, 1, 32, "I", "B")
        b = _mul(A, x)
        S = FB.BlockSolver(_dev_csr(A), _dev_factors(F), c["rhs"], variant="afiim", precision=c["precision"],
                           memory="device", verified=True)
        return {"kind": kind, "S": S, "b": _dev(b), "x": _dev(np.zeros_like(b))}
    A = _matrix(c, rng)
    F, b = _pdfiim(A), _mul(A, x)
    if kind == "dropin":
        return {"kind": kind, "A": A, "b": b, "G": (F["Gi"], F["Gj"], F["Gv"]), "D": F["IDv"],
                "H": (F["Hi"], F["Hj"], F["Hv"])}
    precision = c["precision"] if kind == "mixed" else "fp64"
    if c.get("memory") == "host":
        return {"kind": kind, "S": FB.Solver(A, F, variant="pdfiim", precision=precision), "b": b}
    S = FB.Solver(_dev_csr(A), _dev_factors(F), variant="pdfiim", precision=precision, memory="device")
    return {"kind": kind, "S": S, "b": _dev(b), "x": _dev(np.zeros_like(b))}


def run(state):
    s, kind = state, state["kind"]
    if kind in ("spmv", "spmv_power"):
        FB.spmv(*s["A"], s["x"], s["y"])
        return s["y"]
    if kind == "prec":
        FB.prec_apply(*s["G"], s["D"], *s["H"], s["r"], s["z"], s["t"])
        return s["z"]
    if kind == "factors":
        return FB.pdfiim_build(s["A"], 0.06, 2, 2, 1, -1, "I", "B", gpu=True)
    if kind == "dropin":
        x = np.zeros(len(s["b"]))
        _, _, info = FB.EPBiCGSTAB_pdfiim(s["A"], s["b"], 1e-10, 1200, s["G"], s["D"], s["H"], x)
        return x, info
    tol = {"solve": 1e-10, "batch": 1e-13}.get(kind, 1e-12)
    if "x" not in s:   # host arrays
        x = np.zeros(len(s["b"]))
        return x, s["S"].solve(s["b"], x, tol=tol, nmax=1200)["info"]
    # A handle runs on its own stream: the caller's writes to x have to be done before the call.
    s["x"].zero_()
    torch.cuda.current_stream().synchronize()
    r = s["S"].solve(s["b"], s["x"], tol=tol, nmax=1200)
    return s["x"], r["info"]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        return _batch_solution(c, seed)[0], None
    if kind == "factors":
        return None   # a dense LU per row: minutes in plain numpy
    rng, x = _solution(c, seed)
    if kind == "spmv":
        return _mul(_matrix(c, rng), x)
    if kind == "spmv_power":
        return _mul(_power(c, rng), x)
    if kind == "prec":
        G, D, H = _factors2(c, *_stencil(c, rng))
        return _mul(G, D * _mul(H, x))
    return x, None


def work(case):
    """Every input read once and every output written once; the floating-point operations of the
    products and vector updates of a usual number of iterations (about the longest side's cells)."""
    c, kind = case, case["kind"]
    if kind == "batch":
        n = sum(p[0] ** 2 for p in _batch_sides(c, 0))
        side = c["hi"]
        return {"bytes": n * (12 * 5 + 8 * 11 + 24), "flops": side * n * (4 * 16 + 22)}
    n = _cells(c) if "nx" in c else c["n"]
    if kind == "spmv":
        return {"bytes": n * (12 * 7 + 4 + 16), "flops": 14 * n}
    if kind == "spmv_power":
        nnz = n * c["mean"]
        return {"bytes": 12 * nnz + 20 * n, "flops": 2 * nnz}
    if kind == "prec":
        return {"bytes": n * (12 * 8 + 8 + 24), "flops": 17 * n}
    if kind == "factors":
        return {"bytes": n * 12 * (7 + 6 + 11), "flops": n * 20 ** 3}
    if kind == "block":
        k = c["rhs"]
        return {"bytes": n * (12 * 13 + 8 * 12 + 16 * k), "flops": 10 * k * n * (4 * 25 + 22)}
    side = max(c["nx"], c["ny"], c["nz"])
    values = 8 if kind != "mixed" else 4
    return {"bytes": n * (12 * 7 + (values + 4) * 17 + 8 + 24), "flops": 0.8 * side * n * (4 * 24 + 22)}
