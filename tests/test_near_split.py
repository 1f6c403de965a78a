"""The near/far split of the level layout (host side of the chain kernel)."""
from __future__ import annotations

import numpy as np
import pytest

import capellinisptrsv_gb300 as cs
from capellinisptrsv_gb300.solver import level_layout, level_schedule, near_split


@pytest.mark.parametrize("group,span", [(32, 64), (32, 0), (8, 100), (32, 10_000)])
@pytest.mark.parametrize("kind", ["zipf", "band", "diagonal"])
def test_near_split(kind, group, span):
    kw = {"zipf": dict(workload="zipf_1m", n=3_001), "band": dict(n=3_001, kmin=0, kmax=9, band=400),
          "diagonal": dict(n=257, kmin=0, kmax=0, band=1)}[kind]
    m = cs.generate(kw.pop("workload", None), seed=4, **kw)
    _, order, position, _ = level_schedule(m.n, m.rowptr, m.colidx)
    ptr, idx, _, _ = level_layout(m.n, m.rowptr, m.colidx, order, position)
    first, near = near_split(m.n, ptr, idx, span, group)
    total = 0
    for p in range(m.n):
        reach = p // group * group - span
        deps = idx[ptr[p]:ptr[p + 1]]
        assert first[p] == ptr[p] + int(np.sum(deps < reach))
        total += int(np.sum(deps >= reach))
    assert near == total
