"""Host side of the chain and stream kernels: the near/far split and the slices of a level layout."""
from __future__ import annotations

import numpy as np
import pytest

import capellinisptrsv_gb300 as cs
from capellinisptrsv_gb300.solver import level_layout, level_schedule, near_split, stream_layout


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


@pytest.mark.parametrize("kind", ["zipf", "band", "diagonal"])
def test_stream_layout(kind):
    """Slices of 8 rows of one level, most dependencies first, ties in position order."""
    kw = {"zipf": dict(workload="zipf_1m", n=3_001), "band": dict(n=3_001, kmin=0, kmax=9, band=400),
          "diagonal": dict(n=257, kmin=0, kmax=0, band=1)}[kind]
    m = cs.generate(kw.pop("workload", None), seed=5, **kw)
    _, order, position, start = level_schedule(m.n, m.rowptr, m.colidx)
    start = start[1:]
    ptr, _, _, _ = level_layout(m.n, m.rowptr, m.colidx, order, position)
    slices, pos, entries = stream_layout(start, ptr)
    cnt = np.diff(ptr)
    k = at = 0
    for a, b in zip(start[:-1], start[1:]):
        want = sorted(range(a, b), key=lambda p: (-min(int(cnt[p]), 63), p))
        rows = (b - a + 7) // 8
        want += [-1] * (8 * rows - len(want))
        assert pos[k:k + rows].ravel().tolist() == want
        for s in range(k, k + rows):
            longest = max((int(cnt[p]) for p in pos[s] if p >= 0), default=0)
            assert slices[s].tolist() == [at, longest]
            at += 8 * longest
        k += rows
    assert k == len(slices) and entries == at
