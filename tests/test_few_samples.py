"""Binning of few samples by counting, against the sort that bins more of them.

The same samples followed by left-out ones beyond the counting form's limit (65535 samples) are binned
by the sort; both keep each cell's samples in index order, so gridded sums, degridded values and the
counts of left-out samples are equal, bit for bit.
"""
from __future__ import annotations

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n,support,g,groups,tuning", [
    (1, 0, 1, 1, (8, -1, 0, 0)),            # one point, one cell
    (255, 3, 64, 1, (16, -1, 32, 32)),      # crowded: units of split cells
    (256, 10, 130, 2, (8, 0, 0, 40)),       # one block, ragged last tiles
    (257, 10, 4096, 1, (16, -1, 0, 32)),    # two blocks, 4096 cells: counts in both arrays
    (9000, 90, 700, 3, (8, 1, 16, 0)),      # up to 28 tiles a footprint, several plane groups
    (65535, 2, 500, 2, (16, 0, 0, 64)),     # the most samples
])
def test_counted_plan_equals_sorted_plan(tcv, cuda_ok, n, support, g, groups, tuning):
    import torch

    from tconvolve import _lib, raw

    rng = np.random.default_rng(n + g)
    s = 2 * support + 1
    planes = 2 * groups
    c_len = 64 * planes * s * s
    tab = torch.from_numpy(rng.standard_normal((c_len, 2)).astype(np.float32)).cuda().view(torch.complex64).reshape(-1)
    code = _lib.CTYPE_BY_NAME["c64"]
    iu = (support + rng.integers(0, g - s + 1, n)).astype(np.int32)
    iv = rng.integers(0, g - s + 1, n).astype(np.int32)
    if n > 1:
        iu[rng.integers(0, n, n // 50 + 1)] = support - 1  # left out: a footprint past the edge
    coff = (rng.integers(0, 64 * planes, n) * s * s).astype(np.int32)
    vis = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    field = torch.from_numpy((rng.standard_normal(g * g) + 1j * rng.standard_normal(g * g)).astype(np.complex64)).cuda()
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    pad = 65536 - n
    runs = []
    for extra in (0, pad):
        u = np.concatenate([iu, np.full(extra, -1, np.int32)])
        v = np.concatenate([iv, np.zeros(extra, np.int32)])
        co = np.concatenate([coff, np.zeros(extra, np.int32)])
        x = np.concatenate([vis, np.ones(extra, np.complex64)])
        plan = raw.Plan(d(u), d(v), d(co), support, g, c_len, tuning=tuning)
        grid = torch.zeros(g * g, dtype=torch.complex64, device="cuda")
        plan.grid(d(x), tab, code, grid)
        out = torch.empty(n + extra, dtype=torch.complex64, device="cuda")
        plan.degrid(field, tab, code, out)
        runs.append((grid.cpu().numpy(), out.cpu().numpy()[:n], plan.rejected() - extra))
    assert np.count_nonzero(runs[0][0]) > 0
    assert runs[0][2] == runs[1][2]
    assert np.array_equal(runs[0][0], runs[1][0])
    assert np.array_equal(runs[0][1], runs[1][1])
