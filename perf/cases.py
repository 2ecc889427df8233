"""Performance cases: the calls a program makes on this library, through its
public Python entry points, at the sizes they are used at.

Kinds (``case["kind"]``):

* ``spmv``     -- ``CsrMatrix.spmv`` on a resident, autotuned matrix.
* ``spmm``     -- ``CsrMatrix.spmm``: k right-hand sides in one pass over A.
* ``cg``       -- ``CgSolver.solve`` with A and b resident (FP64 or mixed).
* ``cgd_host`` -- the drop-in ``cgd`` on host arrays, uploads included.
* ``serve``    -- a stream of uneven systems through the batching ``Server``.
* ``pagerank`` -- the drop-in ``pagerank`` on host arrays.
* ``rcm``      -- Cuthill-McKee order of a resident matrix, the permuted matrix
  and right-hand side, and one product with it.

Matrices: ``uniform`` (k uniformly drawn columns per row), ``powerlaw``
(Zipf-2.1 row lengths of a given mean, uniform columns) and 5- or 7-point
``diffusion`` operators on a grid, with face coefficients log-uniform in
[1/contrast, contrast] (contrast 1: the Laplacian).  Everything is drawn on
the GPU from the seed.

Solves stop at a relative residual of 1e-12 (1e-6 for float arrays), where x
is settled to well below its type's comparison bounds; at looser tolerances
the last digits of x depend on which iteration happened to meet the test.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gooseberry_b200 as gb

DEV = "cuda"


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # one latency-bound product: few rows, ten entries each
        {"name": "spmv_uniform_100k", "kind": "spmv", "matrix": "uniform", "n": 100_000,
         "mean": 10, "dtype": "f64"},
        # a web- or social-graph-like matrix, both value widths
        {"name": "spmv_powerlaw_8m", "kind": "spmv", "matrix": "powerlaw", "n": 8_000_000,
         "mean": 16, "dtype": "f64"},
        {"name": "spmv_powerlaw_2m_f32", "kind": "spmv", "matrix": "powerlaw", "n": 2_000_000,
         "mean": 16, "dtype": "f32"},
        # a banded operator larger than L2, as a time stepper or an outer solver applies it
        {"name": "spmv_laplace2d_4096", "kind": "spmv", "matrix": "diffusion", "dims": 2,
         "side": 4096, "contrast": 1.0, "dtype": "f64"},
        # several right-hand sides at once
        {"name": "spmm_laplace2d_1024_k8", "kind": "spmm", "matrix": "diffusion", "dims": 2,
         "side": 1024, "contrast": 1.0, "k": 8},
        # a small solve, where each iteration's latency is all there is
        {"name": "cg_diffusion2d_96", "kind": "cg", "matrix": "diffusion", "dims": 2, "side": 96,
         "contrast": 10.0, "mode": "f64"},
        # the benchmark's solve
        {"name": "cg_laplace2d_1024", "kind": "cg", "matrix": "diffusion", "dims": 2,
         "side": 1024, "contrast": 1.0, "mode": "f64"},
        # a variable-coefficient 3D solve, mixed precision; the matrix exceeds L2
        {"name": "cg_mixed_diffusion3d_160", "kind": "cg", "matrix": "diffusion", "dims": 3,
         "side": 160, "contrast": 100.0, "mode": "mixed"},
        # the reference's own call: host arrays in, host x out
        {"name": "cgd_host_diffusion2d_400", "kind": "cgd_host", "matrix": "diffusion",
         "dims": 2, "side": 400, "contrast": 10.0, "dtype": "f64"},
        # many users' systems, 1k to 262k rows, solved together
        {"name": "serve_mixed_48", "kind": "serve", "requests": 48, "lo": 32, "hi": 512,
         "mode": "mixed"},
        # ranking a graph read into host memory
        {"name": "pagerank_1m", "kind": "pagerank", "n": 1_000_000, "mean": 16},
        # renumbering a scrambled mesh before products with it
        {"name": "rcm_mesh2d_700", "kind": "rcm", "matrix": "diffusion", "dims": 2, "side": 700,
         "contrast": 10.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmm", "cg", "cg", "cg", "cgd_host", "serve", "pagerank",
                       "rcm"])
    if kind == "spmv":
        m = rng.choice(["uniform", "powerlaw", "diffusion"])
        dt = rng.choice(["f64", "f32"])
        if m == "diffusion":
            dims = rng.choice([2, 3])
            side = _log(rng, 64, 4000) if dims == 2 else _log(rng, 16, 200)
            return {"kind": kind, "matrix": m, "dims": dims, "side": side,
                    "contrast": rng.choice([1.0, 10.0, 100.0]), "dtype": dt}
        return {"kind": kind, "matrix": m, "n": _log(rng, 1_000, 4_000_000),
                "mean": rng.randint(4, 24), "dtype": dt}
    if kind == "spmm":
        dims = rng.choice([2, 3])
        return {"kind": kind, "matrix": "diffusion", "dims": dims,
                "side": _log(rng, 30, 1000) if dims == 2 else _log(rng, 10, 100),
                "contrast": rng.choice([1.0, 10.0]), "k": rng.randint(2, 16)}
    if kind == "cg":
        dims = rng.choice([2, 3])
        side = _log(rng, 16, 900) if dims == 2 else _log(rng, 8, 150)
        return {"kind": kind, "matrix": "diffusion", "dims": dims, "side": side,
                "contrast": rng.choice([1.0, 10.0]), "mode": rng.choice(["f64", "mixed"])}
    if kind == "cgd_host":
        return {"kind": kind, "matrix": "diffusion", "dims": 2, "side": _log(rng, 16, 600),
                "contrast": rng.choice([1.0, 10.0]), "dtype": rng.choice(["f64", "f32"])}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(8, 40), "lo": 32,
                "hi": rng.choice([128, 256, 512]), "mode": rng.choice(["mixed", "f64"])}
    if kind == "pagerank":
        return {"kind": kind, "n": _log(rng, 10_000, 800_000), "mean": rng.randint(4, 20)}
    dims = rng.choice([2, 3])
    return {"kind": kind, "matrix": "diffusion", "dims": dims,
            "side": _log(rng, 30, 700) if dims == 2 else _log(rng, 10, 75), "contrast": 10.0}


# ---- inputs ------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uniform(g, n, lo, hi):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo


def _grid(case):
    return (int(case["side"]),) * int(case["dims"])


def _stencil(shape, contrast, g):
    """The operator as (diagonal, [off-diagonal coefficients per axis]):
    one positive coefficient per face, Dirichlet faces on the diagonal."""
    lc = math.log(contrast)

    def faces(s):
        m = int(np.prod(s))
        return torch.exp(_uniform(g, m, -lc, lc)).reshape(s) if lc else torch.ones(
            s, device=DEV, dtype=torch.float64)

    diag = torch.zeros(shape, device=DEV, dtype=torch.float64)
    off = []
    for ax in range(len(shape)):
        s = list(shape)
        s[ax] += 1
        c = faces(s)
        diag += c.narrow(ax, 0, shape[ax]) + c.narrow(ax, 1, shape[ax])
        off.append(c.narrow(ax, 1, shape[ax] - 1).contiguous())
    return diag, off


def _stencil_csr(diag, off):
    """CSR (int32, int32, float64) of a stencil, columns ascending."""
    shape, dims = diag.shape, diag.dim()
    n = diag.numel()
    strides = [int(np.prod(shape[ax + 1:])) for ax in range(dims)]
    slots = [(ax, -1) for ax in range(dims)] + [(None, 0)] + [(ax, 1) for ax in reversed(range(dims))]
    cols = torch.empty((n, len(slots)), dtype=torch.int32, device=DEV)
    vals = torch.zeros((n, len(slots)), dtype=torch.float64, device=DEV)
    here = torch.zeros((n, len(slots)), dtype=torch.bool, device=DEV)
    row = torch.arange(n, dtype=torch.int32, device=DEV)
    for j, (ax, way) in enumerate(slots):
        cols[:, j] = row + (way * strides[ax] if way else 0)
        v, h = vals[:, j].view(shape), here[:, j].view(shape)
        if not way:
            v.copy_(diag)
            h.fill_(True)
        else:
            v, h = (t.narrow(ax, 1 if way < 0 else 0, shape[ax] - 1) for t in (v, h))
            v.copy_(-off[ax])
            h.fill_(True)
    rowptr = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    rowptr[1:] = torch.cumsum(here.sum(1), 0).to(torch.int32)
    return rowptr, cols[here], vals[here]


def _random_csr(case, g):
    """A CSR with uniformly drawn columns, ascending within each row."""
    n, nnz = int(case["n"]), int(case["n"]) * int(case["mean"])
    if case.get("matrix") == "uniform":
        length = torch.full((n,), int(case["mean"]), dtype=torch.int64, device=DEV)
    else:  # power law: Zipf exponent 2.1, capped, scaled to exactly nnz entries
        u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64).clamp_min(1e-12)
        w = (u ** (-1 / 1.1)).clamp_max(0.025 * n)
        length = 1 + (w * ((nnz - n) / w.sum())).floor().to(torch.int64)
        length[: nnz - int(length.sum())] += 1
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.cumsum(length, 0)
    key = torch.repeat_interleave(torch.arange(n, device=DEV) << 32, length, output_size=nnz)
    key += torch.randint(0, n, (nnz,), generator=g, device=DEV)
    cols = (key.sort().values & 0xFFFFFFFF).to(torch.int32)
    return rowptr.to(torch.int32), cols, _uniform(g, nnz, -1.0, 1.0)


def _csr(case, g):
    if case["matrix"] == "diffusion":
        return _stencil_csr(*_stencil(_grid(case), case["contrast"], g))
    return _random_csr(case, g)


def _sides(case):
    """Grid sides of a request stream: log-uniform, the same for every seed."""
    r = np.random.RandomState(int(case["requests"]))
    return [int(round(math.exp(v))) for v in r.uniform(
        math.log(case["lo"]), math.log(case["hi"]), int(case["requests"]))]


class _HostCsr:
    def __init__(self, rowptr, rowind, rowval):
        self.rowptr, self.rowind = (t.cpu().numpy().view(np.uint32) for t in (rowptr, rowind))
        self.rowval = rowval.cpu().numpy()


def _scramble(rowptr, cols, vals, g):
    """A symmetric random renumbering of a matrix."""
    n = rowptr.numel() - 1
    to = torch.randperm(n, generator=g, device=DEV)
    length = (rowptr[1:] - rowptr[:-1]).long()
    row = to[torch.repeat_interleave(torch.arange(n, device=DEV), length)]
    key, order = ((row << 32) + to[cols.long()]).sort()
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    return ptr.to(torch.int32), (key & 0xFFFFFFFF).to(torch.int32), vals[order]


def _graph(case, g):
    rowptr, cols, vals = _random_csr(case, g)
    return rowptr, cols, vals.abs() + 0.1


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("spmv", "spmm"):
        f32 = case.get("dtype") == "f32"
        rowptr, cols, vals = _csr(case, g)
        n = rowptr.numel() - 1
        if f32:
            A = gb.CsrMatrix.from_device(rowptr, cols, val32=vals.float())
        else:
            A = gb.CsrMatrix.from_device(rowptr, cols, val64=vals)
        dt = torch.float32 if f32 else torch.float64
        if kind == "spmm":
            k = int(case["k"])
            return {"kind": kind, "A": A, "k": k, "B": _uniform(g, n * k, -1.0, 1.0),
                    "out": torch.empty(n * k, dtype=dt, device=DEV)}
        A.autotune(f32=f32)
        return {"kind": kind, "A": A, "x": _uniform(g, n, -1.0, 1.0).to(dt),
                "y": torch.empty(n, dtype=dt, device=DEV)}
    if kind == "cg":
        rowptr, cols, vals = _csr(case, g)
        mixed = case["mode"] == "mixed"
        A = gb.CsrMatrix.from_device(rowptr, cols, val64=vals,
                                     val32=vals.float() if mixed else None)
        b = _uniform(g, rowptr.numel() - 1, -1.0, 1.0)
        return {"kind": kind, "S": gb.CgSolver(A, gb.CG_MIXED if mixed else gb.CG_F64), "b": b,
                "x": torch.empty_like(b)}
    if kind == "cgd_host":
        A = _HostCsr(*_csr(case, g))
        b = _uniform(g, len(A.rowptr) - 1, -1.0, 1.0).cpu().numpy()
        tol = 1e-12
        if case["dtype"] == "f32":
            A.rowval, b, tol = A.rowval.astype(np.float32), b.astype(np.float32), 1e-6
        return {"kind": kind, "A": A, "b": b, "error": tol * float(np.linalg.norm(b))}
    if kind == "serve":
        mode = gb.CG_MIXED if case["mode"] == "mixed" else gb.CG_F64
        reqs = []
        for side in _sides(case):
            A = _HostCsr(*_stencil_csr(*_stencil((side, side), 10.0, g)))
            reqs.append((A, _uniform(g, side * side, -1.0, 1.0).cpu().numpy()))
        return {"kind": kind, "reqs": reqs,
                "server": gb.Server(pool_bytes=2 << 30, max_slots=64, mode=mode)}
    if kind == "pagerank":
        return {"kind": kind, "A": _HostCsr(*_graph(case, g))}
    A = gb.CsrMatrix.from_device(*(_scramble(*_csr(case, g), g)))
    return {"kind": kind, "A": A, "x": _uniform(g, A.nrows, -1.0, 1.0)}


# ---- one pass ----------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "spmv":
        return state["A"].spmv(state["x"], state["y"])
    if kind == "spmm":
        return state["A"].spmm(state["B"], state["k"], out=state["out"])
    if kind == "cg":
        x, _ = state["S"].solve(state["b"], state["x"], tol=1e-12, relative=True, niter=20_000)
        return x
    if kind == "cgd_host":
        A = state["A"]
        x, _, _ = gb.cgd(A.rowptr, A.rowind, A.rowval, state["b"], state["error"], 20_000)
        return x
    if kind == "serve":
        srv = state["server"]
        for i, (A, b) in enumerate(state["reqs"]):
            srv.submit(i, A, b, tol=1e-12, niter=20_000)
        return [r.x for r in sorted(srv.drain(), key=lambda r: r.id)]
    if kind == "pagerank":
        A = state["A"]
        rank, _, _ = gb.pagerank(A.rowptr, A.rowind, A.rowval, 0.85, 1e-10, 200)
        return rank
    A, x = state["A"], state["x"]
    perm = A.cuthillmckee()
    px = gb.permute_vector(x, perm)
    return perm, px, A.permute(perm, perm).spmv(px)


# ---- what a pass cannot do without --------------------------------------------

def _shape(case):
    """Rows and entries of a case's matrix."""
    if case.get("matrix") == "diffusion":
        s, d = int(case["side"]), int(case["dims"])
        return s ** d, s ** d + 2 * d * (s - 1) * s ** (d - 1)
    return int(case["n"]), int(case["n"]) * int(case["mean"])


def _iterations(rows, dims, contrast):
    """About how many CG iterations a solve to 1e-12 takes (unpreconditioned:
    the grid's side times a factor that grows with the contrast)."""
    return int((4.5 if contrast <= 1 else 6.0 if contrast <= 10 else 21.0) * rows ** (1 / dims))


def _cg_work(n, nnz, iters, s=8):
    # per iteration: A once; p, r, x and A p each read or written as the
    # textbook recurrence needs them when nothing stays on the chip
    return {"bytes": float(iters) * (nnz * (4 + s) + 4 * (n + 1) + 8 * n * s),
            "flops": float(iters) * (2 * nnz + 10 * n)}


def work(case):
    kind = case["kind"]
    if kind == "serve":
        b = f = 0.0
        for s in _sides(case):
            w = _cg_work(s * s, 5 * s * s - 4 * s, _iterations(s * s, 2, 10.0),
                         4 if case["mode"] == "mixed" else 8)
            b, f = b + w["bytes"], f + w["flops"]
        return {"bytes": b, "flops": f}
    n, nnz = _shape(case)
    if kind in ("cg", "cgd_host"):
        narrow = case.get("mode") == "mixed" or case.get("dtype") == "f32"
        it = _iterations(n, int(case["dims"]), case["contrast"])
        return _cg_work(n, nnz, it, 4 if narrow else 8)
    if kind == "pagerank":
        return {"bytes": 21.0 * (nnz * 12 + 4 * (n + 1) + 16 * n) + 12.0 * nnz + 4 * (n + 1),
                "flops": 21.0 * (2 * nnz + 3 * n)}
    if kind == "rcm":  # the pattern once for the order, the matrix in and out, one product
        return {"bytes": 4.0 * nnz + 2 * (12.0 * nnz + 4 * n) + 12.0 * nnz + 44.0 * n,
                "flops": 2.0 * nnz}
    s = 4 if case.get("dtype") == "f32" else 8
    k = int(case.get("k", 1))
    return {"bytes": float(nnz * (4 + s) + 4 * (n + 1) + 2 * n * s * k), "flops": 2.0 * nnz * k}


# ---- the same results in 64 bits, in plain torch --------------------------------

def _apply(diag, off, x):
    y = diag * x
    for ax, c in enumerate(off):
        m = c.shape[ax]
        y.narrow(ax, 1, m).sub_(c * x.narrow(ax, 0, m))
        y.narrow(ax, 0, m).sub_(c * x.narrow(ax, 1, m))
    return y


def _solve(systems, bs):
    """Solutions of several stencil systems, as one block-diagonal Jacobi-
    preconditioned CG that is restarted on the true residual."""
    def amul(v):
        return [_apply(d, o, u) for (d, o), u in zip(systems, v)]

    def dots(u, v):  # one scalar per system
        return [torch.dot(p.reshape(-1), q.reshape(-1)) for p, q in zip(u, v)]

    inv = [1 / d for d, _ in systems]
    bs = [b.reshape(d.shape) for b, (d, _) in zip(bs, systems)]
    xs = [torch.zeros_like(b) for b in bs]
    for goal in (1e-11, 1e-5, 1e-3):
        r = [b - a for b, a in zip(bs, amul(xs))]
        z = [i * v for i, v in zip(inv, r)]
        p = [v.clone() for v in z]
        rz, first = dots(r, z), dots(r, r)
        for it in range(1, 20_000):
            q = amul(p)
            a = [u / torch.clamp_min(v, 1e-300) for u, v in zip(rz, dots(p, q))]
            for k in range(len(xs)):
                xs[k].addcmul_(a[k], p[k])
                r[k].addcmul_(a[k], q[k], value=-1)
                torch.mul(inv[k], r[k], out=z[k])
            new = dots(r, z)
            for k in range(len(xs)):
                p[k].mul_(new[k] / torch.clamp_min(rz[k], 1e-300)).add_(z[k])
            rz = new
            if it % 50 == 0:
                rr = torch.stack(dots(r, r)) / torch.clamp_min(torch.stack(first), 1e-300)
                if float(rr.max()) <= goal * goal:
                    break
    return [x.reshape(-1) for x in xs]


def _product(rowptr, cols, vals, x):
    n = rowptr.numel() - 1
    row = torch.repeat_interleave(torch.arange(n, device=DEV),
                                  (rowptr[1:] - rowptr[:-1]).long(), output_size=cols.numel())
    return torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(
        0, row, vals * x[cols.long()])


def exact(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("spmv", "spmm"):
        rowptr, cols, vals = _csr(case, g)
        n = rowptr.numel() - 1
        if kind == "spmm":
            k = int(case["k"])
            B = _uniform(g, n * k, -1.0, 1.0).view(k, n)
            return torch.stack([_product(rowptr, cols, vals, B[j]) for j in range(k)],
                               1).reshape(-1)
        x = _uniform(g, n, -1.0, 1.0)
        if case["dtype"] == "f32":
            vals, x = vals.float().double(), x.float().double()
        return _product(rowptr, cols, vals, x)
    if kind in ("cg", "cgd_host"):
        diag, off = _stencil(_grid(case), case["contrast"], g)
        b = _uniform(g, diag.numel(), -1.0, 1.0)
        if case.get("dtype") == "f32":
            diag, off, b = diag.float().double(), [c.float().double() for c in off], b.float().double()
        x, = _solve([(diag, off)], [b])
        return x.cpu().numpy() if kind == "cgd_host" else x
    if kind == "serve":
        systems, bs = [], []
        for side in _sides(case):
            systems.append(_stencil((side, side), 10.0, g))
            bs.append(_uniform(g, side * side, -1.0, 1.0))
        out = []
        for i in sorted(range(len(bs)), key=lambda i: bs[i].numel()):
            out.append((i, _solve([systems[i]], [bs[i]])[0].cpu().numpy()))
        return [x for _, x in sorted(out, key=lambda t: t[0])]
    if kind == "pagerank":
        rowptr, cols, vals = _graph(case, g)
        n = rowptr.numel() - 1
        c = cols.long()
        vals = vals / torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, c, vals)[c]
        rank = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
        for i in range(200):
            out = _product(rowptr, cols, vals, rank) * 0.85 + 0.15 / n
            if i % 10 == 0 and float(((rank - out) ** 2).sum()) <= 1e-20:
                return out.cpu().numpy()
            rank, out = out, rank
        return out.cpu().numpy()
    # an order is whole numbers, and the permuted vector and product follow it
    return None
