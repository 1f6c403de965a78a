"""Dependency waits that run out of their budget: what the stream and chain kernels report."""
from __future__ import annotations

import re

import numpy as np
import pytest

import capellinisptrsv_gb300 as cs
import oracle
from conftest import rel_inf_err
from test_gpu_chain import dense
from test_gpu_stream import blocks, dev, host

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def reported(m, s, b, stuck):
    """(row, row it waited on) of a solve in which row `stuck` never publishes; the next solve is clean."""
    xo = oracle.solve_csr_lower(m.rowptr, m.colidx, m.val, b)
    s.debug_stuck_row(stuck, timeout_s=0.02)
    s.solve(dev(b))
    with pytest.raises(cs.CapspError) as e:
        s.status()
    assert e.value.status == 2
    s.debug_stuck_row(-1, timeout_s=10.0)
    assert rel_inf_err(host(s.solve(dev(b))), xo) <= 1e-12
    s.status()
    return tuple(int(v) for v in re.search(r"row/column (-?\d+) waiting on (-?\d+)", str(e.value)).groups())


def check(m, got, stuck):
    row, on = got
    deps = m.colidx[m.rowptr[row]:m.rowptr[row + 1] - 1]
    assert 0 <= row < m.n and (on in deps or row == on == stuck), (row, on, deps)


@pytest.mark.parametrize("k", [1, 4, 16])
def test_stream_reports_the_waiting_row(k):
    """Not a lane of the same warp that is done, and not padding."""
    m = blocks(6, 12_301, 3, 11, 12)
    stuck = int(m.colidx[m.rowptr[15_000]])
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
    b = np.random.default_rng(k).standard_normal((m.n, k))
    check(m, reported(m, s, b, stuck), stuck)


def test_graph_replays_report_too():
    """The hook inside the handle's own capture, where AUTO otherwise takes the stream kernel."""
    m = blocks(6, 12_301, 3, 11, 12)
    b = np.random.default_rng(2).standard_normal((m.n, 4))
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
    st = torch.cuda.Stream()
    bd = dev(b)
    x = torch.empty_like(bd)
    torch.cuda.synchronize()
    s.debug_stuck_row(int(m.colidx[m.rowptr[15_000]]), timeout_s=0.02)
    s.graph_solve(bd, x, st)
    with pytest.raises(cs.CapspError) as e:
        s.status(st)
    assert e.value.status == 2
    s.debug_stuck_row(-1, timeout_s=10.0)
    s.graph_solve(bd, x, st)
    s.status(st)
    assert rel_inf_err(host(x), oracle.solve_csr_lower(m.rowptr, m.colidx, m.val, b)) <= 1e-12


CHAINS = {
    # near entries only; far entries, folded by a lane or by a warp; entries walked in global memory
    "near": lambda: cs.generate(n=1_025, kmin=1, kmax=6, band=60, seed=3),
    "far": lambda: cs.generate("zipf40_1m", n=25_385, seed=7),
    "far_light": lambda: cs.generate(n=60_000, kmin=6, kmax=12, band=9_000, seed=8),
    "spilled": lambda: dense(700),
}


@pytest.mark.parametrize("k", [1, 3])
@pytest.mark.parametrize("name", list(CHAINS))
def test_chain_reports_the_waiting_row(name, k):
    """Rows, not positions of the level order nor places in the ring."""
    m = CHAINS[name]()
    s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
    rng = np.random.default_rng(k)
    for stuck in (m.colidx[m.rowptr[m.n // 3]], m.colidx[m.rowptr[m.n - 3] + 1]):
        check(m, reported(m, s, rng.standard_normal((m.n, k)), int(stuck)), int(stuck))
