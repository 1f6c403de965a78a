"""The solves a program makes through this package, as cases that can be timed.

``listed()`` names them, ``draw(rng)`` gives another one of the same ranges,
``prepare(case, seed)`` makes the inputs and the analysed handle a program keeps,
``run(state)`` makes one call (or one forward and backward) and returns its
results, ``work(case)`` counts what the call cannot do without and
``exact(case, seed)`` solves the same systems in plain torch.

The matrices follow the repository's workload rules (capellinisptrsv_gb300/workloads.py):
off-diagonals U[-1, 1], diagonal 1 + sum of their magnitudes, columns uniform in
a band, or Zipf-distributed counts with half of the columns among the previous
32 rows.  They are drawn on the GPU from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import capellinisptrsv_gb300 as cs

DEV = "cuda"
DTYPES = {"f64": torch.float64, "f32": torch.float32}
NEAR = 32          # window of the Zipf matrices' near columns
ZIPF_S, ZIPF_CAP = 1.8, 512
FIXED = 1 << 40    # off-diagonals are multiples of 2^-40, so a row's sum of magnitudes is exact


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _case(name=None, *, call="solve", n=0, nsys=0, kind="band", kmin=1, kmax=5, band=0, dtype="f64", nrhs=1,
          fmt="csr", uplo="lower"):
    c = dict(call=call, n=n, nsys=nsys, kind=kind, kmin=kmin, kmax=kmax, band=band, dtype=dtype, nrhs=nrhs, fmt=fmt,
             uplo=uplo)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one small system by itself: a member of the batch, solved in a per-system loop
        _case("single_2k", n=2_003, kmin=3, kmax=12, band=250),
        # the plain 20,000-row system
        _case("plain_20k", n=20_000, kmin=1, kmax=5, band=2_000),
        # ragged rows (some without off-diagonals), odd sizes, single precision, upper, 3 right-hand sides
        _case("ragged_300k_f32_k3", n=300_007, kmin=0, kmax=20, band=30_011, dtype="f32", nrhs=3, uplo="upper"),
        # wide levels, few entries per row: the thread-per-row headline, both precisions
        _case("wide_4m_f64", n=4_194_304, kmin=1, kmax=7, band=65_536),
        _case("wide_4m_f32", n=4_194_304, kmin=1, kmax=7, band=65_536, dtype="f32"),
        # the same kind of matrix handed over by columns (the SyncFree_csc caller's format)
        _case("csc_1m5_f64", n=1_500_001, kmin=1, kmax=7, band=32_768, fmt="csc"),
        # long chains and heavy rows: the mix caller's matrices
        _case("zipf_1m_f64", n=1_048_576, kind="zipf", kmin=1),
        _case("zipf40_128k_f64", n=131_072, kind="zipf", kmin=38),
        # thousands of uneven systems in one graph-replayed launch
        _case("batch_2048_k1", call="graph", nsys=2_048, kmin=3, kmax=12),
        _case("batch_1024_k16", call="graph", nsys=1_024, kmin=3, kmax=12, nrhs=16),
        # forward and backward of the differentiable solve
        _case("grad_1m_k16", call="autograd", n=1_048_576, kmin=2, kmax=10, band=16_384, nrhs=16),
        # host arrays in, host arrays out (page-locked), as the reference's drivers are called
        _case("host_4m_f64", call="host", n=4_194_304, kmin=1, kmax=7, band=65_536),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["solve", "solve", "solve", "zipf", "graph", "autograd", "host"])
    dtype = rng.choice(["f64", "f64", "f32"])
    if what == "graph":
        nrhs = rng.choice([1, 4, 16, 32])
        return _case(call="graph", nsys=_log_int(rng, 256, 1_024 if nrhs <= 16 else 512), kmin=3, kmax=12, nrhs=nrhs)
    if what == "zipf":
        kmin = rng.choice([1, 1, 38])
        return _case(n=_log_int(rng, 20_000, 1_000_000 if kmin == 1 else 150_000), kind="zipf", kmin=kmin, dtype=dtype)
    kmin = rng.randint(0, 3)
    kmax = kmin + rng.randint(3, 12)
    if what == "host":
        n = _log_int(rng, 20_000, 3_000_000)
        return _case(call="host", n=n, kmin=kmin, kmax=kmax, band=max(1, n // rng.randint(8, 80)), dtype=dtype)
    if what == "autograd":
        n = _log_int(rng, 20_000, 800_000)
        return _case(call="autograd", n=n, kmin=kmin, kmax=kmax, band=max(1, n // rng.randint(8, 80)),
                     nrhs=rng.choice([1, 3, 4, 8, 16]))
    nrhs = rng.choice([1, 1, 1, 2, 3, 4, 8, 16, 20])
    n = _log_int(rng, 500, 3_000_000 // nrhs)
    return _case(n=n, kmin=kmin, kmax=kmax, band=max(1, n // rng.randint(8, 80)), dtype=dtype, nrhs=nrhs,
                 fmt=rng.choice(["csr", "csr", "csc"]), uplo=rng.choice(["lower", "lower", "upper"]))


# ---------------------------------------------------------------------------
# matrices
# ---------------------------------------------------------------------------

def _batch_sizes(nsys):
    # log-uniform in [500, 50,000], evenly spread, so the number of rows depends on the case alone
    u = (np.arange(nsys) + 0.5) / nsys
    return np.rint(np.exp(math.log(500) + u * math.log(100))).astype(np.int64)


def _zipf_weights(kmin):
    w = np.arange(1, ZIPF_CAP + 1, dtype=np.float64) ** -ZIPF_S
    return np.maximum(np.arange(1, ZIPF_CAP + 1), kmin), w / w.sum()


def _rows_and_entries(case):
    n = int(_batch_sizes(case["nsys"]).sum()) if case["nsys"] else case["n"]
    if case["kind"] == "zipf":
        k, w = _zipf_weights(case["kmin"])
        mean = float((k * w).sum())
    else:
        mean = (case["kmin"] + case["kmax"]) / 2
    return n, int(n * (mean + 1))


def _matrix(case, seed):
    """Lower-triangular CSR on the GPU: (n, rowptr int32, colidx int32, val f64), columns ascending, diagonal last."""
    gen = torch.Generator(device=DEV)
    # a training program keeps its structure and changes its values: there the structure is the case's own
    gen.manual_seed(17 if case["call"] == "autograd" else 1_000_003 * int(seed) + 17)
    if case["nsys"]:
        sizes = torch.from_numpy(_batch_sizes(case["nsys"])).to(DEV)
        sizes = sizes[torch.randperm(case["nsys"], generator=gen, device=DEV)]
        rowoff = torch.zeros(case["nsys"] + 1, dtype=torch.int64, device=DEV)
        rowoff[1:] = torch.cumsum(sizes, 0)
        n = int(rowoff[-1])
        i = torch.arange(n, device=DEV)
        first = torch.repeat_interleave(rowoff[:-1], sizes)
        low = torch.maximum(first, i - torch.repeat_interleave((sizes // 8).clamp(min=1), sizes))
    else:
        rowoff, n = None, case["n"]
        i = torch.arange(n, device=DEV)
        low = (i - case["band"]).clamp(min=0) if case["band"] else torch.zeros_like(i)
    keys = [i * n + i]
    if case["kind"] == "zipf":
        k, w = _zipf_weights(case["kmin"])
        at = torch.searchsorted(torch.from_numpy(np.cumsum(w)).to(DEV),
                                torch.rand(n, generator=gen, device=DEV, dtype=torch.float64))
        count = torch.minimum(torch.from_numpy(k).to(DEV)[at.clamp(max=ZIPF_CAP - 1)], i)
        near = torch.minimum((count + 1) // 2, i.clamp(max=NEAR))
        # `near` distinct ones of the previous 32 rows: those of the smallest random ranks
        rank = torch.rand(n, NEAR, generator=gen, device=DEV)
        back = torch.arange(1, NEAR + 1, device=DEV)
        rank = torch.where(back[None, :] <= i[:, None], rank, 2.0).argsort(dim=1).argsort(dim=1)
        r, c = torch.nonzero(rank < near[:, None], as_tuple=True)
        keys.append(r * n + (r - 1 - c))
        del rank
        far = count - near
        low = torch.zeros_like(i)
    else:
        span = case["kmax"] - case["kmin"] + 1
        far = case["kmin"] + (torch.rand(n, generator=gen, device=DEV, dtype=torch.float64) * span).long()
        far = torch.minimum(far, i - low)
    r = torch.repeat_interleave(i, far)
    u = torch.rand(r.numel(), generator=gen, device=DEV, dtype=torch.float64)
    lo = low[r]
    keys.append(r * n + lo + (u * (r - lo)).long().clamp(max=n - 1))
    del u, lo, r
    key = torch.unique(torch.cat(keys))   # sorted; the few columns drawn twice appear once
    del keys
    row = key // n
    col = key - row * n
    del key
    gen.manual_seed(1_000_003 * int(seed) + 23)
    m = torch.randint(-FIXED, FIXED + 1, (row.numel(),), generator=gen, device=DEV)
    diag = row == col
    m[diag] = 0
    total = torch.zeros(n, dtype=torch.int64, device=DEV).index_add_(0, row, m.abs())
    m[diag] = FIXED + total
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    val = m.to(torch.float64) / FIXED
    return n, rowptr.to(torch.int32), col.to(torch.int32), val, rowoff


def _inputs(case, seed):
    """The arrays handed to the package: (n, ptr, idx, val, rowoff, b, target)."""
    n, ptr, idx, val, rowoff = _matrix(case, seed)
    if (case["fmt"] == "csr") == (case["uplo"] == "upper"):
        # rows (columns) stored diagonal first: the lower matrix with both orders turned round
        ptr = (int(ptr[-1]) - ptr.flip(0)).contiguous()
        idx = (n - 1 - idx.flip(0)).contiguous()
        val = val.flip(0).contiguous()
    gen = torch.Generator(device=DEV)
    gen.manual_seed(1_000_003 * int(seed) + 29)
    shape = (n, case["nrhs"]) if case["nrhs"] > 1 else (n,)
    b = torch.randn(shape, generator=gen, device=DEV, dtype=torch.float64)
    target = torch.randn(shape, generator=gen, device=DEV, dtype=torch.float64) if case["call"] == "autograd" else None
    dt = DTYPES[case["dtype"]]
    return n, ptr, idx, val.to(dt), rowoff, b.to(dt), target


# ---------------------------------------------------------------------------
# one call
# ---------------------------------------------------------------------------

def prepare(case, seed):
    n, ptr, idx, val, rowoff, b, target = _inputs(case, seed)
    solver = cs.TriangularSolver(ptr, idx, val, n=n, fmt=case["fmt"], uplo=case["uplo"],
                                 sys_rowoff=None if rowoff is None else rowoff.cpu().numpy())
    s = {"call": case["call"], "solver": solver, "b": b}
    if case["call"] == "graph":
        s["x"] = torch.empty_like(b)
        s["stream"] = torch.cuda.Stream()
        s["stream"].wait_stream(torch.cuda.current_stream())
    elif case["call"] == "autograd":
        solver.reserve(case["nrhs"])
        s["val"] = val.requires_grad_(True)
        s["b"] = b.requires_grad_(True)
        s["target"] = target
    elif case["call"] == "host":
        s["b_host"] = b.cpu().pin_memory().numpy()
        s["x_host"] = torch.empty(b.shape, dtype=b.dtype).pin_memory().numpy()
    return s


def run(state):
    solver = state["solver"]
    if state["call"] == "solve":
        return solver.solve(state["b"])
    if state["call"] == "graph":
        return solver.graph_solve(state["b"], state["x"], state["stream"])
    if state["call"] == "host":
        return solver.solve_host(state["b_host"], state["x_host"])
    # one training step on 0.5 |x - target|^2
    x = cs.sptrsv(solver, state["val"], state["b"])
    grad_val, grad_b = torch.autograd.grad(x, (state["val"], state["b"]), x.detach() - state["target"])
    return {"x": x.detach(), "grad_val": grad_val, "grad_b": grad_b}


def work(case):
    n, nnz = _rows_and_entries(case)
    s, k = (8 if case["dtype"] == "f64" else 4), case["nrhs"]
    matrix, vector = 4 * (n + 1) + 4 * nnz + s * nnz, s * n * k
    if case["call"] == "autograd":
        # structure, values, b and target in; x, grad_b and grad_val out; two solves and the gradient's products
        return {"bytes": matrix + 4 * vector + s * nnz, "flops": k * (2 * (2 * nnz - n) + 2 * nnz + n)}
    return {"bytes": matrix + 2 * vector, "flops": k * (2 * nnz - n)}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------

def _fixed_point(n, row, col, off, diag, b):
    """x with diag x + (off-diagonals) x = b, by x <- (b - off x) / diag: the rows are
    diagonally dominant and the matrix triangular, so it settles to rounding."""
    order = torch.argsort(row, stable=True)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    a = torch.sparse_csr_tensor(ptr, col[order], off[order], size=(n, n))
    b = b.reshape(n, -1)
    x = b / diag[:, None]
    for step in range(4_000):
        y = (b - a @ x) / diag[:, None]
        if step % 8 == 7 and float((y - x).abs().max()) <= 1e-16 * float(y.abs().max()):
            return y
        x = y
    return None


def exact(case, seed):
    n, ptr, idx, val, _, b, target = _inputs(case, seed)
    lines = torch.repeat_interleave(torch.arange(n, device=DEV), (ptr[1:] - ptr[:-1]).long())
    idx, val, b = idx.long(), val.double(), b.double()
    row, col = (lines, idx) if case["fmt"] == "csr" else (idx, lines)
    on = row == col
    diag = torch.empty(n, dtype=torch.float64, device=DEV)
    diag[row[on]] = val[on]
    r, c, v = row[~on], col[~on], val[~on]
    x = _fixed_point(n, r, c, v, diag, b)
    if x is None:
        return None
    if case["call"] == "autograd":
        g = x - target.reshape(n, -1)
        y = _fixed_point(n, c, r, v, diag, g)
        if y is None:
            return None
        gv = torch.zeros_like(val)
        for j in range(x.shape[1]):
            gv -= y[row, j] * x[col, j]
        return {"x": x.reshape(b.shape), "grad_val": gv, "grad_b": y.reshape(b.shape)}
    x = x.reshape(b.shape)
    return x.cpu().numpy() if case["call"] == "host" else x
