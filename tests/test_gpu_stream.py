"""The stream kernel (wide levels and several right-hand sides, algorithm
"auto") at the edges of its slices, batches and lanes, against the oracle at the
suite's bars (relative infinity-norm error 1e-12 in FP64, 1e-5 in FP32)."""
from __future__ import annotations

import numpy as np
import pytest

import capellinisptrsv_gb300 as cs
import oracle
from conftest import rel_inf_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DEV = "cuda:0"
TOL = {np.float64: 1e-12, np.float32: 1e-5}


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


def blocks(nb, width, kmin, kmax, seed):
    """nb levels of `width` rows: row i has kmin..kmax distinct dependencies among
    the `width` rows before its level's first (the nearest of them in the previous
    level), rows of the first level none."""
    rng = np.random.default_rng(seed)
    n = nb * width
    i = np.arange(n)
    first = i // width * width
    cnt = np.where(first == 0, 0, rng.integers(kmin, kmax + 1, n))
    rows = np.repeat(i, cnt)
    # a random stride keeps the dependencies of a row distinct
    t = np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt)
    back = (np.repeat(rng.integers(0, width, n), cnt) + t * 37) % width
    cols = first[rows] - 1 - back
    v = rng.uniform(-1.0, 1.0, len(rows))
    diag = 1.0 + np.bincount(rows, np.abs(v), minlength=n)
    key = np.concatenate([rows * (n + 1.0) + cols, i * (n + 1.0) + i])
    order = np.argsort(key, kind="stable")
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(cnt + 1)
    return cs.CSRMatrix(n, rp, np.concatenate([cols, i])[order].astype(np.int32), np.concatenate([v, diag])[order])


MATRICES = {
    # (matrix, right-hand sides): which widths and row lengths reach the kernel depends on both
    "wide_short": (lambda: blocks(3, 12_293, 0, 7, 1), (1, 2, 3, 17)),      # ragged last slices, empty rows
    "wide_batch_edges": (lambda: blocks(3, 13_001, 8, 13, 2), (1, 4, 5)),   # 8 / 9 and 12 / 13 entries
    "wide_long": (lambda: blocks(3, 12_288, 20, 33, 3), (1, 16)),           # several batches
    "narrow_medium": (lambda: blocks(40, 301, 3, 10, 4), (3, 4, 8, 16, 31, 32, 33)),
    "narrow_short": (lambda: blocks(12, 2_003, 1, 6, 5), (8, 16)),
    "one_level": (lambda: cs.generate(n=20_003, kmin=0, kmax=0, band=1), (1, 5)),
}


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", list(MATRICES))
def test_stream_edges(name, dtype):
    make, ks = MATRICES[name]
    m = make()
    v = m.val.astype(dtype)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(v))
    rng = np.random.default_rng(23)
    for k in ks:
        ld = k + 2 if k % 2 else k  # odd counts also with a stride
        b = rng.standard_normal((m.n, k)).astype(dtype)
        bd = torch.zeros((m.n, ld), dtype=dev(b).dtype, device=DEV)[:, :k]
        bd.copy_(dev(b))
        x = torch.full((m.n, ld), 7.0, dtype=bd.dtype, device=DEV)
        got = host(s.solve(bd, x[:, :k])).copy()
        assert rel_inf_err(got, oracle.solve_csr_lower(m.rowptr, m.colidx, v, b)) <= TOL[dtype], k
        if ld > k:
            assert (host(x[:, k:]) == 7.0).all()
        y = host(s.solve_transpose(dev(b)))
        assert rel_inf_err(y, oracle.solve_csr_transpose(m.rowptr, m.colidx, v, b)) <= TOL[dtype], k
        # the row kernel sums in the same order
        s.set_algorithm("wrtfst")
        assert np.array_equal(host(s.solve(dev(b))), got)
        s.set_algorithm("auto")
    s.status()


def test_stream_follows_values_and_captures():
    """Refreshed values reach the layout; a caller's capture made before the layout
    exists solves with the row kernels, one made after it with the layout."""
    m = blocks(30, 701, 3, 10, 6)
    val = dev(m.val)
    b = np.random.default_rng(2).standard_normal((m.n, 8))
    bd, x = dev(b), torch.empty((m.n, 8), dtype=torch.float64, device=DEV)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), val)
    s.set_algorithm("wrtfst")
    s.reserve(8)
    s.set_algorithm("auto")
    st = torch.cuda.Stream()
    graphs = []
    for _ in range(2):
        st.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            s.solve(bd, x)
        graphs.append(g)
        s.solve(bd)  # builds the layout
    v2 = m.val * 1.5
    val.copy_(dev(v2))
    s.refresh_values(val)
    xo = oracle.solve_csr_lower(m.rowptr, m.colidx, v2, b)
    for g in graphs:
        x.zero_()
        g.replay()
        assert rel_inf_err(host(x), xo) <= 1e-12
    s.status()


def test_stream_nonfinite_rhs_and_timeout_hook():
    """An infinity and a NaN in b spread as in the oracle; the row that never
    publishes (debug hook) is still reported."""
    m = blocks(4, 12_500, 1, 9, 7)
    b = np.random.default_rng(3).standard_normal(m.n)
    b[100], b[200] = np.inf, np.nan
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
    x, xo = host(s.solve(dev(b))), oracle.solve_csr_lower(m.rowptr, m.colidx, m.val, b)
    assert np.array_equal(np.isfinite(x), np.isfinite(xo))
    ok = np.isfinite(xo)
    assert rel_inf_err(x[ok], xo[ok]) <= 1e-12
    s.debug_stuck_row(5, timeout_s=0.02)
    s.solve(dev(b))
    with pytest.raises(cs.CapspError):
        s.status()
    s.debug_stuck_row(-1, timeout_s=10.0)
    s.solve(dev(b))
    s.status()


def test_stream_beside_other_work():
    """The blocks may start behind another stream's work (the warps then take
    tickets), and two solves may run side by side."""
    m = blocks(20, 12_300, 3, 10, 9)
    b = np.random.default_rng(5).standard_normal((m.n, 4))
    bd, xo = dev(b), oracle.solve_csr_lower(m.rowptr, m.colidx, m.val, b)
    solvers = [cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val)) for _ in range(2)]
    outs = [torch.empty_like(bd) for _ in solvers]
    for s, x in zip(solvers, outs):
        s.set_timeout(5.0)
        s.solve(bd, x)
        s.status()
    streams = [torch.cuda.Stream() for _ in range(3)]
    w = torch.randn(4096, 4096, device=DEV, dtype=torch.bfloat16)
    torch.cuda.synchronize()
    for _ in range(5):
        with torch.cuda.stream(streams[2]):
            for _ in range(3):
                w @ w
        for s, x, st in zip(solvers, outs, streams):
            with torch.cuda.stream(st):
                x.zero_()
                s.solve(bd, x)
    torch.cuda.synchronize()
    for s, x in zip(solvers, outs):
        s.status()
        assert rel_inf_err(host(x), xo) <= 1e-12


def test_row_kernel_first_runs_inside_a_capture_after_stream_solves():
    """The scratch that warm-up solves in the stream kernel did not need is
    allocated without breaking the caller's capture."""
    m = cs.generate(n=60_000, kmin=1, kmax=5, band=30_000, seed=21)
    b = np.random.default_rng(21).standard_normal((m.n, 8)).astype(np.float32)
    v = m.val.astype(np.float32)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(v))
    bd = dev(b)
    x = torch.empty_like(bd)
    s.solve(bd, x)
    s.set_algorithm("wrtfst")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s.solve(bd, x)
    x.zero_()
    g.replay()
    assert rel_inf_err(host(x), oracle.solve_csr_lower(m.rowptr, m.colidx, v, b)) <= 1e-5
    s.status()
