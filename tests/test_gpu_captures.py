"""Solves and value refreshes inside a caller's CUDA-graph captures, replayed
after the handle has gone on to other right-hand sides, against the oracle
(relative infinity-norm error 1e-12 in FP64)."""
from __future__ import annotations

import numpy as np
import pytest

import capellinisptrsv_gb300 as cs
import oracle
from conftest import rel_inf_err
from test_gpu_stream import blocks, dev, host

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def capture(f):
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        f()
    torch.cuda.synchronize()
    return g


def test_captured_refresh_reaches_every_later_solve():
    """One right-hand side needs no stream layout; 16 would build one, after the
    refresh was captured.  Replays with new values must reach the solves of both."""
    m = blocks(30, 701, 3, 10, 6)
    val = dev(m.val)
    rng = np.random.default_rng(4)
    b1, b16 = rng.standard_normal(m.n), rng.standard_normal((m.n, 16))
    bd1, bd16 = dev(b1), dev(b16)
    x1 = torch.empty_like(bd1)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), val)
    s.solve(bd1, x1)

    def step():
        s.refresh_values(val)
        s.solve(bd1, x1)

    g = capture(step)
    assert rel_inf_err(host(s.solve(bd16)), oracle.solve_csr_lower(m.rowptr, m.colidx, m.val, b16)) <= 1e-12
    for scale in (1.5, 0.75):
        v = m.val * np.where(np.arange(m.nnz) % 2 == 0, scale, 2.0)
        val.copy_(dev(v))
        g.replay()
        assert rel_inf_err(host(x1), oracle.solve_csr_lower(m.rowptr, m.colidx, v, b1)) <= 1e-12
        assert rel_inf_err(host(s.solve(bd16)), oracle.solve_csr_lower(m.rowptr, m.colidx, v, b16)) <= 1e-12
    s.status()


@pytest.mark.parametrize("k", [1, 16])
def test_transpose_built_after_a_captured_refresh_follows_it(k):
    """The transposed view does not exist when the refresh is captured."""
    m = blocks(30, 701, 3, 10, 8)
    val = dev(m.val)
    b = np.random.default_rng(k).standard_normal((m.n, k))
    bd = dev(b)
    x = torch.empty_like(bd)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), val)
    s.solve(bd, x)

    def step():
        s.refresh_values(val)
        s.solve(bd, x)

    g = capture(step)
    assert rel_inf_err(host(s.solve_transpose(bd)),
                       oracle.solve_csr_transpose(m.rowptr, m.colidx, m.val, b)) <= 1e-12
    v = m.val * np.where(np.arange(m.nnz) % 2 == 0, 1.5, 2.0)
    val.copy_(dev(v))
    g.replay()
    assert rel_inf_err(host(x), oracle.solve_csr_lower(m.rowptr, m.colidx, v, b)) <= 1e-12
    assert rel_inf_err(host(s.solve_transpose(bd)), oracle.solve_csr_transpose(m.rowptr, m.colidx, v, b)) <= 1e-12
    s.status()


@pytest.mark.parametrize("eager", [(), (2, 5, 32)])
def test_captured_solves_keep_their_scratch(eager):
    """One right-hand side takes the row kernels, 16 the stream kernel, 8 the row kernels
    again, with larger scratch: first needed inside a capture whose graph, like an
    earlier one, points at the smaller.  `eager`: row-kernel solves that outgrow it later."""
    m = blocks(12, 1_500, 1, 6, 9)
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
    rng = np.random.default_rng(9)
    b = {k: rng.standard_normal((m.n, k)) for k in (1, 8, 16)}
    bd = {k: dev(b[k]) for k in b}
    x = {k: torch.empty_like(bd[k]) for k in b}
    want = {k: oracle.solve_csr_lower(m.rowptr, m.colidx, m.val, b[k]) for k in b}
    for k in (1, 16):
        s.solve(bd[k], x[k])
    first = capture(lambda: s.solve(bd[1], x[1]))
    second = capture(lambda: (s.solve(bd[1], x[1]), s.solve(bd[8], x[8])))
    s.set_algorithm("wrtfst")
    for k in eager:
        s.solve(dev(rng.standard_normal((m.n, k))))
    for g, ks in ((first, (1,)), (second, (1, 8)), (first, (1,))):
        for k in ks:
            x[k].zero_()
        g.replay()
        for k in ks:
            assert rel_inf_err(host(x[k]), want[k]) <= 1e-12
    s.status()
