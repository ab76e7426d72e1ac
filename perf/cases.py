"""The work that programs built on this solver have it do, as timed cases.

Each case is one call (or one encode + solve) through the package's public
entry points, over the range of systems that the tests, the benchmark and the
reference's drivers use: 2D 5-point and 3D 7-point grids (constant, upwind and
variable-coefficient) and random sparse SPD systems, from about a thousand to
two million rows, in FP64 and in the mixed per-tile precisions.

Matrices are assembled on the GPU from the seed. Solves start from x0 = 0 with
b = A x*, x* ~ U[0, 1): x* is then the solution in 64 bits up to the rounding
of b. The tolerances are below the benchmark's 1e-10 so that x itself, and not
only the residual, is determined to about ten digits.
"""
import importlib
import math

import numpy as np
import torch

mf = importlib.import_module("mille-feillue_b200")

MAXITER = 60000

# kind: what is run. grid: points per side. decades: log10 of the ratio of the
# largest to the smallest face coefficient (variable-coefficient grids).
# velocity: the scale of the upwind grids' velocity.
LISTED = [
    # the smallest SpMV a program makes in a loop of its own: launch latency
    {"name": "spmv_grid2d_32", "kind": "spmv", "matrix": "grid2d", "grid": 32},
    # one product of the largest benchmark operator: memory bandwidth
    {"name": "spmv_grid3d_128", "kind": "spmv", "matrix": "grid3d", "grid": 128, "decades": 6.0},
    # a product without grid structure: scattered columns, x gathered
    {"name": "spmv_scattered_200k", "kind": "spmv", "matrix": "scattered", "n": 200000},
    # the smallest solve, ragged (rows not a multiple of the tile): latency
    {"name": "cg_grid2d_37", "kind": "cg", "matrix": "grid2d", "grid": 37, "tol": 1e-12},
    # the 2D Laplacian benchmark system: the matrix stays on the chip
    {"name": "cg_grid2d_256", "kind": "cg", "matrix": "grid2d", "grid": 256, "tol": 1e-13},
    # the nonsymmetric benchmark system (upwind convection-diffusion)
    {"name": "bicgstab_upwind_64", "kind": "bicgstab", "matrix": "upwind", "grid": 64, "velocity": 1.0,
     "tol": 1e-12},
    # a mid-size Jacobi-preconditioned solve on an odd grid
    {"name": "pcg_grid3d_75", "kind": "pcg", "matrix": "grid3d", "grid": 75, "decades": 6.0, "tol": 1e-13},
    # the headline system in FP64: larger than L2, streams every iteration
    {"name": "cg_grid3d_128", "kind": "cg", "matrix": "grid3d", "grid": 128, "decades": 6.0, "tol": 1e-13},
    # the headline system in the mixed per-tile precisions
    {"name": "cg_mixed_grid3d_128", "kind": "cg_mixed", "matrix": "grid3d", "grid": 128, "decades": 6.0, "tol": 1e-13},
    # many independent scattered SPD systems of a thousand to 2e5 rows in one launch
    {"name": "batch_cg_48", "kind": "batch", "count": 48, "lo": 1000, "hi": 200000, "tol": 1e-13},
    # sixteen right-hand sides of one system at once (host call)
    {"name": "multi_cg_grid3d_48x16", "kind": "multi", "matrix": "grid3d", "grid": 48, "decades": 4.0, "rhs": 16,
     "tol": 1e-13},
    # a program that meets each matrix once: host CSR, encode, solve, host x
    {"name": "encode_pcg_grid3d_100", "kind": "encode_pcg", "matrix": "grid3d", "grid": 100, "decades": 6.0,
     "tol": 1e-13},
]


def listed():
    return [dict(c) for c in LISTED]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds, sizes log-uniform over their ranges."""
    kind = rng.choice(["spmv", "spmv", "cg", "cg", "cg_mixed", "bicgstab", "pcg", "batch", "multi", "encode_pcg"])
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 48), "lo": _log_int(rng, 1000, 4000),
                "hi": _log_int(rng, 20000, 200000), "tol": 1e-13}
    c = {"kind": kind}
    if kind == "bicgstab":
        c.update(matrix="upwind", grid=_log_int(rng, 10, 90), velocity=round(rng.uniform(0.2, 2.0), 2), tol=1e-12)
        return c
    if kind == "cg_mixed":
        c.update(matrix="grid3d", grid=_log_int(rng, 24, 120))
    elif kind == "multi":
        c.update(matrix="grid3d", grid=_log_int(rng, 10, 48), rhs=rng.randint(2, 16))
    elif kind == "pcg" or kind == "encode_pcg":
        c.update(matrix="grid3d", grid=_log_int(rng, 10, 110))
    else:
        c.update(matrix=rng.choice(["grid2d", "grid3d", "scattered"]))
        if c["matrix"] == "grid2d":
            c.update(grid=_log_int(rng, 20, 600))
        elif c["matrix"] == "grid3d":
            c.update(grid=_log_int(rng, 10, 120))
        else:
            c.update(n=_log_int(rng, 1000, 200000))
    if c["matrix"] == "grid3d":
        c["decades"] = round(rng.uniform(0.0, 4.0 if kind == "multi" else 6.0), 2)
    if kind != "spmv":
        c["tol"] = 1e-13 if c["matrix"] != "grid2d" or c["grid"] > 100 else 1e-12
    return c


# ------------------------------------------------------------------ matrices
def _stencil_csr(n, cols, vals, live):
    """CSR (int32, int32, FP64 host arrays) of (n, k) entries in ascending columns, those with `live`."""
    rp = torch.zeros(n + 1, dtype=torch.int64, device=cols.device)
    rp[1:] = live.sum(1).cumsum(0)
    return (rp.to(torch.int32).cpu().numpy(), cols[live].to(torch.int32).cpu().numpy(), vals[live].cpu().numpy())


def _uniform(gen, n, dev):
    return torch.rand(n, dtype=torch.float64, generator=gen).to(dev)


def _grid2d(N, dev):
    r = torch.arange(N * N, device=dev)
    i, j = r % N, r // N
    cols = torch.stack([r - N, r - 1, r, r + 1, r + N], 1)
    live = torch.stack([j > 0, i > 0, i >= 0, i < N - 1, j < N - 1], 1)
    vals = torch.tensor([-1.0, -1.0, 4.0, -1.0, -1.0], dtype=torch.float64, device=dev).expand(N * N, 5)
    return cols, vals, live


def _grid3d_parts(N, dev):
    r = torch.arange(N ** 3, device=dev)
    i, j, k = r % N, (r // N) % N, r // (N * N)
    cols = torch.stack([r - N * N, r - N, r - 1, r, r + 1, r + N, r + N * N], 1)
    live = torch.stack([k > 0, j > 0, i > 0, i >= 0, i < N - 1, j < N - 1, k < N - 1], 1)
    return cols, live


def _upwind(N, velocity, gen, dev):
    """Upwind convection-diffusion, D = 1, h = 1, a velocity near (1, 0.5, 0.25) x its scale."""
    cols, live = _grid3d_parts(N, dev)
    v = velocity * (0.9 + 0.2 * torch.rand(3, dtype=torch.float64, generator=gen))
    v = (v * torch.tensor([1.0, 0.5, 0.25], dtype=torch.float64)).tolist()
    row = [-(1.0 + v[2]), -(1.0 + v[1]), -(1.0 + v[0]), 6.0 + sum(v), -1.0, -1.0, -1.0]
    return cols, torch.tensor(row, dtype=torch.float64, device=dev).expand(N ** 3, 7), live


def _grid3d(N, decades, gen, dev):
    """7-point Laplacian, face coefficients log-uniform over `decades` decades, Dirichlet boundaries."""
    cols, live = _grid3d_parts(N, dev)

    def faces(*shape):
        e = torch.rand(shape, dtype=torch.float64, generator=gen).to(dev)
        return 10.0 ** (decades * (e - 0.5))

    kx, ky, kz = faces(N, N, N + 1), faces(N, N + 1, N), faces(N + 1, N, N)
    f = [kz[:-1], ky[:, :-1], kx[:, :, :-1], kx[:, :, 1:], ky[:, 1:], kz[1:]]
    f = [a.reshape(-1) for a in f]
    diag = f[0] + f[1] + f[2] + f[3] + f[4] + f[5]
    return cols, torch.stack([-f[0], -f[1], -f[2], diag, -f[3], -f[4], -f[5]], 1), live


def _scattered_csr(n, gen, dev):
    """Random sparse SPD: 4..12 off-diagonal partners drawn per row, one weight in (-1, 0] per pair, the
    diagonal 0.01 above the sum of the magnitudes."""
    m = torch.randint(4, 13, (n,), generator=gen)
    i = torch.repeat_interleave(torch.arange(n), m)
    j = torch.randint(0, n - 1, (int(m.sum()),), generator=gen)
    j = j + (j >= i)
    pair = torch.unique((torch.minimum(i, j) * n + torch.maximum(i, j)).to(dev))
    w = -0.5 * _uniform(gen, pair.numel(), dev)
    a, b = pair // n, pair % n
    d = torch.arange(n, device=dev)
    key, order = torch.cat([a * n + b, b * n + a, d * n + d]).sort()
    vals = torch.cat([w, w, torch.zeros(n, dtype=torch.float64, device=dev)])[order]
    row = key // n
    counts = torch.bincount(row, minlength=n)
    rp = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    rp[1:] = counts.cumsum(0)
    vals[key % n == row] = 0.01 - torch.segment_reduce(vals, "sum", lengths=counts)
    return rp.to(torch.int32).cpu().numpy(), (key % n).to(torch.int32).cpu().numpy(), vals.cpu().numpy()


def _times(csr, x):
    """A x on the host, rows summed pairwise (np.add.reduceat)."""
    rp, ci, v = csr
    return np.add.reduceat(v * x[ci], rp[:-1].astype(np.int64))


def _csr(case, seed, dev):
    """(n, CSR) of the case's matrix. Every row holds its diagonal entry."""
    gen = torch.Generator().manual_seed(2 * seed)
    if case["matrix"] == "scattered":
        return case["n"], _scattered_csr(case["n"], gen, dev)
    N = case["grid"]
    if case["matrix"] == "grid2d":
        parts = _grid2d(N, dev)
    elif case["matrix"] == "upwind":
        parts = _upwind(N, case["velocity"], gen, dev)
    else:
        parts = _grid3d(N, case["decades"], gen, dev)
    n = parts[0].shape[0]
    return n, _stencil_csr(n, *parts)


def _xstar(n, seed, cols=None):
    gen = torch.Generator().manual_seed(2 * seed + 1)
    return torch.rand(n if cols is None else (cols, n), dtype=torch.float64, generator=gen).numpy()


def _batch_sizes(case):
    """Log-uniform sizes of the batch's systems, the same for every seed."""
    u = (np.arange(case["count"]) + 0.5) / case["count"]
    return [int(s) for s in np.exp(math.log(case["lo"]) + u * math.log(case["hi"] / case["lo"]))]


# ------------------------------------------------------------------- prepare
def prepare(case, seed):
    dev, kind = "cuda", case["kind"]
    s = {"kind": kind, "tol": case.get("tol")}
    if kind == "batch":
        mats, b = [], []
        for k, n in enumerate(_batch_sizes(case)):
            csr = _scattered_csr(n, torch.Generator().manual_seed(2 * (1009 * seed + k)), dev)
            mats.append(mf.Matrix.from_csr(n, n, *csr))
            b.append(_times(csr, _xstar(n, 1009 * seed + k)))
        s["batch"] = mf.Batch(mats)
        s["b"] = torch.from_numpy(np.concatenate(b)).to(dev)
        s["x"] = torch.empty_like(s["b"])
        return s
    n, csr = _csr(case, seed, dev)
    if kind == "spmv":
        s["tiles"] = mf.Tiles(csr=(n, n, *csr))
        s["x"] = torch.from_numpy(_xstar(n, seed)).to(dev)
        s["y"] = torch.empty_like(s["x"])
        return s
    if kind == "multi":
        X = _xstar(n, seed, case["rhs"])
        s["matrix"] = mf.Matrix.from_csr(n, n, *csr)
        s["b"] = np.asfortranarray(np.stack([_times(csr, x) for x in X], 1))
        return s
    b = _times(csr, _xstar(n, seed))
    if kind == "encode_pcg":
        s["csr"], s["b"] = (n, n, *csr), b
        return s
    s["tiles"] = mf.Tiles(csr=(n, n, *csr),
                          opts=mf.options(precision_mode=mf.MODE_MIXED_RULE) if kind == "cg_mixed" else None)
    s["b"] = torch.from_numpy(b).to(dev)
    s["x"] = torch.empty_like(s["b"])
    return s


# ----------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "spmv":
        s["tiles"].spmv_dev(s["x"].data_ptr(), s["y"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return s["y"]
    if kind == "batch":
        s["batch"].solve_cg_dev(s["b"].data_ptr(), s["x"].data_ptr(), tol=s["tol"], maxiter=MAXITER)
        return s["x"]
    if kind == "multi":
        return mf.solve_cg_multi(s["matrix"], s["b"], tol=s["tol"], maxiter=MAXITER)[0]
    if kind == "encode_pcg":
        return mf.Tiles(csr=s["csr"]).solve_pcg(s["b"], tol=s["tol"], maxiter=MAXITER)[0]
    t = s["tiles"]
    solve = {"cg": t.solve_cg_dev, "cg_mixed": t.solve_cg_dev, "pcg": t.solve_pcg_dev,
             "bicgstab": t.solve_bicgstab_dev}[kind]
    s["x"].zero_()
    solve(s["b"].data_ptr(), s["x"].data_ptr(), tol=s["tol"], maxiter=MAXITER)
    return s["x"]


# --------------------------------------------------------------- work, exact
def _rows_nnz(case):
    if case["kind"] == "batch":
        n = sum(_batch_sizes(case))
        return n, 17 * n
    if case["matrix"] == "scattered":
        return case["n"], 17 * case["n"]
    N = case["grid"]
    if case["matrix"] == "grid2d":
        return N * N, 5 * N * N - 4 * N
    return N ** 3, 7 * N ** 3 - 6 * N * N


def work(case):
    """Bytes: the matrix (CSR) and the vectors in and out once. Operations: the SpMVs and vector updates of
    about as many iterations as such a system takes."""
    n, nnz = _rows_nnz(case)
    cols, N, d = case.get("rhs", 1), case.get("grid", 0), case.get("decades", 0.0)
    bytes_ = 12 * nnz + 4 * n + 16 * n * cols
    kind = case["kind"]
    if kind == "spmv":
        return {"bytes": bytes_, "flops": 2 * nnz}
    if kind == "batch" or case["matrix"] == "scattered":
        its = 60
    elif kind in ("pcg", "encode_pcg"):
        its = N * (3.0 + 0.3 * d * d)
    elif kind == "bicgstab":
        its = 2.5 * N
    else:
        its = N * (2.5 + 0.95 * d * d)
    per = 2 * (2 * nnz + 10 * n) if kind == "bicgstab" else 2 * nnz + 10 * n
    return {"bytes": bytes_, "flops": its * per * cols}


def exact(case, seed):
    """SpMV: the product in 64 bits. Solves: the x* that b was made from."""
    if case["kind"] == "batch":
        return np.concatenate([_xstar(n, 1009 * seed + k) for k, n in enumerate(_batch_sizes(case))])
    n, _ = _rows_nnz(case)
    if case["kind"] == "multi":
        return np.ascontiguousarray(_xstar(n, seed, case["rhs"]).T)
    if case["kind"] == "spmv":
        _, csr = _csr(case, seed, "cuda")
        return _times(csr, _xstar(n, seed))
    return _xstar(n, seed)
