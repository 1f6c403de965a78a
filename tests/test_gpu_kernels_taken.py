"""The kernel, launches and plan that a solve reports, at sizes on either side of the
plans' edges: what the edge tests of each kernel rest on."""
from __future__ import annotations

import numpy as np
import pytest

import capellinisptrsv_gb300 as cs
import oracle
from conftest import rel_inf_err
from test_gpu_stream import MATRICES as STREAMS
from test_gpu_stream import blocks, dev, host

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = {np.float64: 1e-12, np.float32: 1e-5}



def far_blocks(nb, width, back):
    """Levels of `width` rows: a row depends on the one `width` before it and on five
    some `back` levels before."""
    n = width * nb
    rows, cols = [], []
    for d in [width] + [back * width + 7 * t for t in range(5)]:
        i = np.arange(d, n)
        rows.append(i)
        cols.append(i - d)
    i = np.arange(n)
    rows, cols = np.concatenate(rows + [i]), np.concatenate(cols + [i])
    order = np.argsort(rows * (n + 1.0) + cols, kind="stable")
    rows, cols = rows[order], cols[order]
    v = np.random.default_rng(nb).uniform(-1.0, 1.0, len(rows))
    d = rows == cols
    v[d] = 0.0
    v[d] = 1.0 + np.bincount(rows, np.abs(v), minlength=n)
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(rows, minlength=n))
    return cs.CSRMatrix(n, rp, cols.astype(np.int32), v)


CHAINS = {
    # the ring holds the solve up to 16,384 rows on deep matrices, 8,192 otherwise, and then
    # needs no publication vector; longer solves wrap a ring of 4,096
    "deep_16384": (lambda: cs.generate(n=16_384, kmin=2, kmax=8, band=120, seed=1), 16_384, False, 1),
    "deep_16385": (lambda: cs.generate(n=16_385, kmin=2, kmax=8, band=120, seed=1), 4_096, None, None),
    "hold_8192": (lambda: cs.generate(n=8_192, kmin=1, kmax=5, band=900, seed=2), 8_192, False, 1),
    "hold_8193": (lambda: cs.generate(n=8_193, kmin=1, kmax=5, band=900, seed=2), 4_096, None, None),
    # dependencies beyond the reach of 2,048: of light rows, of heavy ones
    "far_light": (lambda: far_blocks(120, 200, 15), 4_096, True, 1),
    "far_heavy": (lambda: cs.generate("zipf40_1m", n=25_385, seed=7), 4_096, True, 1),
    "far_long": (lambda: cs.generate("zipf_1m", n=131_073, seed=7), 4_096, True, 2),
}


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", list(CHAINS))
def test_chain_plans(name, dtype):
    make, ring, far, launches = CHAINS[name]
    m = make()
    v = m.val.astype(dtype)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(v))
    for k in (1, 3, 30):
        b = np.random.default_rng(k).standard_normal((m.n, k)).astype(dtype)
        x = host(s.solve(dev(b)))
        ran = s.last_solve()
        assert (ran["kernel"], ran["ring"]) == ("chain", ring)
        if far is not None:
            assert ran["far_entries"] == far
            assert ran["launches"] == (launches if k == 1 else 1 + far)
        assert rel_inf_err(x, oracle.solve_csr_lower(m.rowptr, m.colidx, v, b)) <= TOL[dtype], k
    s.status()


def test_kernels_by_shape_and_algorithm():
    m = blocks(3, 12_500, 1, 9, 4)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
    assert s.last_solve()["kernel"] == "none"
    b = dev(np.random.default_rng(4).standard_normal((m.n, 4)))
    x = s.solve(b)
    assert s.last_solve() == {"kernel": "stream", "launches": 2, "ring": 0, "far_entries": False}
    s.solve_transpose_grad(b, x)
    assert s.last_solve()["launches"] == 3
    s.set_algorithm("wrtfst")
    s.solve(b)
    assert s.last_solve()["kernel"] == "row"
    s.set_algorithm("syncfree_csc")
    s.solve_transpose(b)
    assert s.last_solve()["kernel"] == "column"
    narrow = blocks(30, 701, 1, 4, 5)
    s = cs.TriangularSolver(dev(narrow.rowptr), dev(narrow.colidx), dev(narrow.val))
    s.solve(dev(cs.normal(narrow.n, seed=5)))
    assert s.last_solve()["kernel"] == "row"  # one right-hand side on levels of 701 rows
    # "auto" before and after the first solve: the row kernels' choice
    assert s.info()["algorithm"] == 1


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", ["wide_short", "wide_batch_edges", "narrow_medium", "one_level"])
def test_stream_tickets_give_what_turns_give(name, dtype):
    """The share-out that is used where the blocks do not start together."""
    make, ks = STREAMS[name]
    m = make()
    v = m.val.astype(dtype)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(v))
    for k in ks:
        b = dev(np.random.default_rng(k).standard_normal((m.n, k)).astype(dtype))
        s.debug_stream_tickets(False)
        x = host(s.solve(b)).copy()
        taken = s.last_solve()["kernel"]
        s.debug_stream_tickets(True)
        assert np.array_equal(host(s.solve(b)), x), k
        # 33 go as 32 and one: the kernel is chosen for the 32
        assert taken == s.last_solve()["kernel"] == "stream", (k, taken)
    s.status()
