"""Variable-width plans binned by distinct footprint (both passes sample-parallel).

Samples that share a footprint (position, table offset, width) are gridded once with the sum of their
data and degridded once.  Bars: grid and samples within the FP32 path's parity bar (relative L2 1e-5) of
the FP64 oracle; samples of one footprint get the same bits; two runs give the same bits; left-out
samples are counted and degrid to 0, as in plans binned by sample.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import REL_L2_FP32

pytestmark = pytest.mark.gpu

WIDTHS = np.array([1, 3, 9, 33, 65, 9], np.int32)  # two planes of one width


def _planes():
    size = 4 * WIDTHS.astype(np.int64) ** 2  # four kernels per plane
    off0 = np.concatenate([[0], np.cumsum(size)[:-1]]).astype(np.int32)
    return off0, int(size.sum())


@pytest.mark.parametrize("n,distinct,g,bad", [
    (1, 1, 130, 0), (300, 300, 130, 0), (5000, 1, 130, 0), (5000, 40, 131, 0), (20000, 3000, 257, 500), (700, 50, 130, 700),
])
@pytest.mark.parametrize("tuning", [(8, -1, 512, 128, 3), (8, 1, 0, 0, 3), (8, 32, 64, 64, 3)])
def test_repeated_footprints(tcv, orc, cuda_ok, n, distinct, g, bad, tuning):
    import torch

    from tconvolve import raw

    rng = np.random.default_rng(n + distinct)
    off0, c_len = _planes()
    c = (rng.standard_normal(c_len) + 1j * rng.standard_normal(c_len)).astype(np.complex64)
    wp0 = rng.integers(0, WIDTHS.size, distinct)
    s0 = WIDTHS[wp0]
    iu0 = rng.integers(s0 // 2, g - s0 // 2)          # columns iu - s/2 .. iu + s/2
    iv0 = rng.integers(0, g - s0 + 1)                 # rows iv .. iv + s - 1
    co0 = off0[wp0] + rng.integers(0, 4, distinct) * s0 * s0
    pick = rng.integers(0, distinct, n) if distinct < n else np.arange(n)
    iu, iv, wp, co = (a[pick].astype(np.int32) for a in (iu0, iv0, wp0, co0))
    out_of = rng.choice(n, bad, replace=False)
    for j, k in enumerate(out_of):  # one way of being left out each: position, plane, table
        if j % 4 == 0:
            iu[k] = -1
        elif j % 4 == 1:
            iv[k] = g
        elif j % 4 == 2:
            wp[k] = WIDTHS.size
        else:
            co[k] = c_len
    good = np.ones(n, bool)
    good[out_of] = False
    data = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    start = (rng.standard_normal(g * g) + 1j * rng.standard_normal(g * g)).astype(np.complex64)

    d = lambda a: torch.from_numpy(a.copy()).cuda()  # noqa: E731
    plan = raw.VarPlan(d(iu), d(iv), d(co), d(wp), WIDTHS, off0, g, c_len, tuning=tuning)
    assert plan.rejected() == bad
    runs = []
    for _ in range(2):
        grid, out = d(start), torch.full((n,), 7.0, dtype=torch.complex64, device="cuda")
        plan.grid(d(data), d(c), tcv.C64, grid)
        plan.degrid(grid, d(c), tcv.C64, out)
        runs.append((grid.cpu().numpy(), out.cpu().numpy()))
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
    got, vis = runs[0]
    assert not vis[~good].any()
    iu, iv, wp, co, pick = iu[good], iv[good], wp[good], co[good], pick[good]
    ref = start.astype(np.complex128)
    if good.any():
        ref = ref + orc.cur_grid_f64(data[good], iu, iv, wp, co, WIDTHS, c, g)
        same = np.zeros(distinct, np.complex64)
        same[pick] = vis[good]
        assert np.array_equal(same[pick], vis[good])
        ref_vis = orc.cur_degrid_f64(got, g, iu, iv, wp, co, WIDTHS, c)
        assert orc.rel_l2(vis[good], ref_vis) <= REL_L2_FP32
    assert orc.rel_l2(got, ref.reshape(got.shape)) <= REL_L2_FP32
