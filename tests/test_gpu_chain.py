"""The chain kernel (levels of up to 256 rows, algorithm "auto"): the edges of
its chunks, ring and slots, against the oracle at the suite's bars (relative
infinity-norm error 1e-12 in FP64, 1e-5 in FP32)."""
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


def dense(n):
    """Full lower triangle: more near entries than a slot holds, one row per level."""
    rp = np.concatenate([[0], np.cumsum(np.arange(1, n + 1))]).astype(np.int32)
    ci = np.concatenate([np.arange(i + 1) for i in range(n)]).astype(np.int32)
    rng = np.random.default_rng(n)
    v = rng.uniform(-1.0, 1.0, len(ci))
    for i in range(n):
        v[rp[i + 1] - 1] = 1.0 + np.abs(v[rp[i]:rp[i + 1] - 1]).sum()
    return cs.CSRMatrix(n, rp, ci, v)


MATRICES = {
    # chunk edges (32 positions), the smallest solves, rows without dependencies
    "n1": lambda: cs.generate(n=1, kmin=0, kmax=0, band=1),
    "n31": lambda: cs.generate(n=31, kmin=0, kmax=3, band=5, seed=1),
    "n33": lambda: cs.generate(n=33, kmin=0, kmax=5, band=20, seed=2),
    "diagonal": lambda: cs.generate(n=100, kmin=0, kmax=0, band=1),
    # ring edges: the smallest ring, the largest one that holds the solve, one row more
    "n1024": lambda: cs.generate(n=1024, kmin=1, kmax=6, band=60, seed=3),
    "n1025": lambda: cs.generate(n=1025, kmin=1, kmax=6, band=60, seed=3),
    "n16384": lambda: cs.generate(n=16_384, kmin=1, kmax=6, band=900, seed=4),
    "n16385": lambda: cs.generate(n=16_385, kmin=1, kmax=6, band=900, seed=4),
    # wrapped rings: every entry near, far entries of light rows, far entries of heavy rows
    "wrap_near": lambda: cs.generate(n=30_011, kmin=1, kmax=4, band=300, seed=5),
    "wrap_far": lambda: cs.generate(n=40_003, kmin=1, kmax=5, band=0, seed=6),
    "deep_far_heavy": lambda: cs.generate("zipf40_1m", n=9_001 + 16_384, seed=7),
    # slots that overflow: all rows of a chunk, one row of it
    "dense": lambda: dense(700),
    "zipf": lambda: cs.generate("zipf_1m", n=20_001, seed=8),
}


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", list(MATRICES))
def test_chain_edges(name, dtype):
    m = MATRICES[name]()
    v = m.val.astype(dtype)
    rng = np.random.default_rng(17)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(v))
    for k, ld in ((1, 1), (3, 5), (18, 18)):
        b = rng.standard_normal((m.n, k)).astype(dtype)
        xo = oracle.solve_csr_lower(m.rowptr, m.colidx, v, b)
        bd = torch.zeros((m.n, ld), dtype=dev(b).dtype, device=DEV)[:, :k]
        bd.copy_(dev(b))
        x = torch.full((m.n, ld), 7.0, dtype=bd.dtype, device=DEV)
        got = s.solve(bd if k > 1 else dev(b[:, 0]), x[:, :k] if k > 1 else None)
        again = host(got).copy()
        assert rel_inf_err(again.reshape(m.n, k), xo.reshape(m.n, k)) <= TOL[dtype], (k, ld)
        if k > 1 and ld > k:
            assert (host(x[:, k:]) == 7.0).all()  # columns outside the solve stay as they were
        yo = oracle.solve_csr_transpose(m.rowptr, m.colidx, v, b)
        y = host(s.solve_transpose(dev(b)))
        assert rel_inf_err(y.reshape(m.n, k), yo.reshape(m.n, k)) <= TOL[dtype], (k, ld)
    s.status()


def test_chain_repeats_bit_for_bit_and_agrees_with_the_row_kernel():
    """Light rows are summed in storage order on either path."""
    m = cs.generate(n=20_000, kmin=1, kmax=7, band=1_500, seed=9)
    b = dev(cs.normal(m.n, seed=9))
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
    x1, x2 = host(s.solve(b)).copy(), host(s.solve(b)).copy()
    s.set_algorithm("wrtfst")
    x3 = host(s.solve(b))
    assert np.array_equal(x1.view(np.uint64), x2.view(np.uint64))
    assert np.array_equal(x1.view(np.uint64), x3.view(np.uint64))


@pytest.mark.parametrize("where", ["device", "host"])
def test_chain_values_follow_refresh_and_nonfinite_rhs(where):
    """New values reach the solve; an infinity and a NaN in b spread as in the oracle."""
    m = cs.generate(n=5_000, kmin=1, kmax=6, band=200, seed=10)
    a = (dev(m.rowptr), dev(m.colidx), dev(m.val)) if where == "device" else (m.rowptr, m.colidx, m.val)
    s = cs.TriangularSolver(*a)
    b = cs.normal(m.n, seed=10)
    s.solve(dev(b))
    v2 = m.val * np.where(np.arange(m.nnz) % 3 == 0, 1.25, 1.5)
    s.set_values(dev(v2) if where == "device" else v2)
    assert rel_inf_err(host(s.solve(dev(b))), oracle.solve_csr_lower(m.rowptr, m.colidx, v2, b)) <= 1e-12
    b[40], b[90] = np.inf, np.nan
    x, xo = host(s.solve(dev(b))), oracle.solve_csr_lower(m.rowptr, m.colidx, v2, b)
    assert np.array_equal(np.isfinite(x), np.isfinite(xo))
    ok = np.isfinite(xo)
    assert rel_inf_err(x[ok], xo[ok]) <= 1e-12
    s.status()


@pytest.mark.parametrize("name", ["n1025", "wrap_far", "zipf"])
def test_chain_timeout_is_reported(name):
    """A row that never publishes: its dependants' waits run out, TIMEOUT is
    reported, and the next solve is clean."""
    m = MATRICES[name]()
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
    b = cs.normal(m.n, seed=11)
    xo = oracle.solve_csr_lower(m.rowptr, m.colidx, m.val, b)
    s.debug_stuck_row(5, timeout_s=0.02)
    s.solve(dev(b))
    with pytest.raises(cs.CapspError) as e:
        s.status()
    assert e.value.status == 2
    s.debug_stuck_row(-1, timeout_s=10.0)
    assert rel_inf_err(host(s.solve(dev(b))), xo) <= 1e-12
    s.status()


@pytest.mark.parametrize("k", [28, 29, 32, 61])
@pytest.mark.parametrize("name", ["n33", "wrap_near", "wrap_far", "deep_far_heavy"])
def test_chain_clusters_of_five_and_four_blocks(name, k):
    """Each right-hand side comes out as when it is solved alone, bit for bit, on
    either side of the line between the cluster sizes and with a remainder."""
    m = MATRICES[name]()
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
    b = np.random.default_rng(k).standard_normal((m.n, k))
    x = host(s.solve(dev(b)))
    for r in (0, 27, k - 1):
        alone = host(s.solve(dev(b[:, r])))
        assert np.array_equal(x[:, r].view(np.uint64), alone.view(np.uint64)), r
    s.status()


@pytest.mark.parametrize("n", [131_072, 131_073])
def test_chain_marks_short_vectors_pending_itself(n):
    """Either side of the length up to which the kernel fills the publication
    vector; the second solve would read the first one's values where it did not."""
    m = cs.generate("zipf40_1m", n=n, seed=12)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
    for seed in (1, 2):
        b = cs.normal(m.n, seed=seed)
        x = host(s.solve(dev(b)))
        assert rel_inf_err(x, oracle.solve_csr_lower(m.rowptr, m.colidx, m.val, b)) <= 1e-12
    s.status()
