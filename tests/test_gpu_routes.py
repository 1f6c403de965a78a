"""Solves on either side of the lines between the kernels of algorithm "auto",
against the oracle at the suite's bars (relative infinity-norm error 1e-12 in
FP64, 1e-5 in FP32)."""
from __future__ import annotations

import numpy as np
import pytest

import capellinisptrsv_gb300 as cs
import oracle
from conftest import rel_inf_err
from test_gpu_stream import blocks

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DEV = "cuda:0"
TOL = {np.float64: 1e-12, np.float32: 1e-5}


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


def grid(width, levels, backs):
    """`levels` levels of `width` rows: row i depends on the rows `backs` before it, the
    nearest of them `width` before."""
    n = width * levels
    rows, cols = [], []
    for d in backs:
        i = np.arange(d, n)
        rows.append(i)
        cols.append(i - d)
    i = np.arange(n)
    rows, cols = np.concatenate(rows + [i]), np.concatenate(cols + [i])
    order = np.argsort(rows * (n + 1.0) + cols, kind="stable")
    rows, cols = rows[order], cols[order]
    v = np.random.default_rng(width).uniform(-1.0, 1.0, len(rows))
    d = rows == cols
    v[d] = 0.0
    v[d] = 1.0 + np.bincount(rows, np.abs(v), minlength=n)
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(rows, minlength=n))
    return cs.CSRMatrix(n, rp, cols.astype(np.int32), v)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("width", [255, 256, 257])
def test_either_side_of_the_chain_kernels_line(width, dtype):
    """Rows of 2 and of 6 dependencies, some beyond the ring; more right-hand sides after fewer."""
    for backs in ((width, 12 * width), tuple(width * t + 3 * (t > 1) * t for t in (1, 2, 3, 5, 9, 14))):
        m = grid(width, 100, backs)
        v = m.val.astype(dtype)
        s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(v))
        assert s.info()["levels"] == 100
        for k in (1, 3, 16, 33):
            b = np.random.default_rng(k).standard_normal((m.n, k)).astype(dtype)
            xo = oracle.solve_csr_lower(m.rowptr, m.colidx, v, b)
            yo = oracle.solve_csr_transpose(m.rowptr, m.colidx, v, b)
            assert rel_inf_err(host(s.solve(dev(b))), xo) <= TOL[dtype], k
            assert rel_inf_err(host(s.solve_transpose(dev(b))), yo) <= TOL[dtype], k
        s.status()


def test_fp32_products_beyond_the_range_that_cancel():
    """b/d of -3e38 and a product of 4e38: the fused sum is 1e38, and so is the solve's
    (its remainder has no finite value).  Two levels of 64 rows: the chain kernel."""
    n = 128
    i = np.arange(n)
    rp = np.concatenate([i[:65], 64 + 2 * (i[:64] + 1)]).astype(np.int32)
    ci = np.concatenate([i[:64], np.stack([i[:64], i[64:]], 1).ravel()]).astype(np.int32)
    v = np.concatenate([np.ones(64), np.tile([-2.0, 1.0], 64)]).astype(np.float32)
    b = np.concatenate([np.full(64, 2e38), np.full(64, -3e38)]).astype(np.float32)
    s = cs.TriangularSolver(dev(rp), dev(ci), dev(v))
    x = host(s.solve(dev(b)))
    xo = oracle.solve_csr_lower(rp, ci, v.astype(np.float64), b.astype(np.float64))
    assert rel_inf_err(x, xo) <= 1e-5
    s.set_algorithm("wrtfst")
    assert rel_inf_err(host(s.solve(dev(b))), xo) <= 1e-5
    s.status()


def solve_longdouble(m, v, b):
    """Forward solve in extended precision (128-bit, or at least 80-bit, floats)."""
    v, x = v.astype(np.longdouble), b.astype(np.longdouble)
    for i in range(m.n):
        j0, j1 = m.rowptr[i], m.rowptr[i + 1] - 1
        x[i] = (x[i] - np.dot(v[j0:j1], x[m.colidx[j0:j1]])) / v[j1]
    return x


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("k", [1, 4])
def test_long_rows_are_as_exact_as_in_the_mixed_kernel(k, dtype):
    """Wide levels of 33 to 60 entries a row: the error is that of the mixed row kernel,
    which sums a row as a tree (a hundredth more for the order of equal terms)."""
    m = blocks(2, 12_800, 33, 60, 3)
    v = m.val.astype(dtype)
    b = np.random.default_rng(k).standard_normal((m.n, k)).astype(dtype)
    xo = solve_longdouble(m, v, b)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(v))
    err = {}
    for algorithm in ("auto", "mix"):
        s.set_algorithm(algorithm)
        d = host(s.solve(dev(b))).astype(np.longdouble) - xo
        err[algorithm] = float(np.sqrt((d * d).sum() / (xo * xo).sum()))
    assert err["auto"] <= 1.01 * err["mix"], err
    s.status()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind", ["zipf40", "band", "deep_band"])
def test_deep_matrices_are_solved_to_half_a_unit_in_the_last_place(kind, dtype):
    """The 2-norm of the error is below that of half a unit in the last place of every
    value: long rows do not add a rounding per entry."""
    m = {"zipf40": lambda: cs.generate("zipf40_1m", n=20_001, seed=3),
         "band": lambda: cs.generate(n=2_003, kmin=3, kmax=12, band=250, seed=3),
         "deep_band": lambda: cs.generate(n=20_000, kmin=3, kmax=9, band=60, seed=3)}[kind]()
    v = m.val.astype(dtype)
    b = np.random.default_rng(1).standard_normal(m.n).astype(dtype)
    xo = solve_longdouble(m, v, b)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(v))
    d = host(s.solve(dev(b))).astype(np.longdouble) - xo
    assert float(np.sqrt((d * d).sum() / (xo * xo).sum())) <= np.finfo(dtype).eps / 2
    s.status()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_nonfinite_right_hand_sides_in_deep_matrices(dtype):
    """An infinity and a NaN in b reach the rows that they reach in the oracle, no others."""
    m = cs.generate("zipf_1m", n=9_001, seed=5)
    v = m.val.astype(dtype)
    b = np.random.default_rng(5).standard_normal(m.n).astype(dtype)
    b[8_000], b[8_500] = np.inf, np.nan
    xo = oracle.solve_csr_lower(m.rowptr, m.colidx, v, b)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(v))
    x = host(s.solve(dev(b)))
    ok = np.isfinite(xo)
    assert 8_000 < ok.sum() < m.n - 2 and np.array_equal(np.isfinite(x), ok)
    assert rel_inf_err(x[ok], xo[ok]) <= TOL[dtype]
    s.status()
