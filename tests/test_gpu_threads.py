"""Host threads that solve side by side, each with handles and a stream of its own."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import capellinisptrsv_gb300 as cs
import oracle
from conftest import rel_inf_err
from test_gpu_stream import dev

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_chain_solves_of_different_plans_in_two_threads():
    """The plans' launches differ in shared memory (ring, slots); neither thread's may
    depend on what the other launched last."""
    plans = [cs.generate("zipf_1m", n=9_001, seed=1), cs.generate(n=2_003, kmin=3, kmax=12, band=250, seed=2)]
    failures = []

    def work(m):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                s = cs.TriangularSolver(dev(m.rowptr), dev(m.colidx), dev(m.val))
                b = cs.normal(m.n, seed=3)
                bd, x = dev(b), torch.empty(m.n, dtype=torch.float64, device="cuda:0")
                xo = oracle.solve_csr_lower(m.rowptr, m.colidx, m.val, b)
                for _ in range(3_000):
                    s.solve(bd, x)
                s.status()
                if rel_inf_err(x.cpu().numpy(), xo) > 1e-12:
                    failures.append("wrong result")
        except Exception as e:  # noqa: BLE001 - the failure is reported in the main thread
            failures.append(repr(e))

    threads = [threading.Thread(target=work, args=(m,)) for m in plans]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
