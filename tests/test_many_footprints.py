"""Variable-width plans on both sides of the sample count from which they are binned by distinct footprint
(2^18), and the work units of the fewer ones, sized by the pairs in their cells.

Bars: grid and samples within the FP32 path's parity bar (relative L2 1e-5) of the FP64 oracle; samples of one
footprint get the same value, bit for bit; two runs give the same bits; left-out samples are counted and
degrid to 0.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import REL_L2_FP32

WIDTHS = np.array([1, 3, 9, 17, 5, 9], np.int32)  # two planes of one width


@pytest.mark.gpu
@pytest.mark.parametrize("tuning", [(8, -1, 512, 128, 3), (8, 0, 0, 0, 3), (8, 32, 16, 64, 3)])
@pytest.mark.parametrize("n,distinct,bad", [
    (2**18 - 1, 40000, 300), (2**18, 40000, 300), (2**18, 1, 0), (2**18, 2**18, 0), (300001, 7, 299990), (2**18, 5, 2**18),
    (40000, 40000, 100), (700, 3, 700),
])
def test_either_side(tcv, orc, cuda_ok, n, distinct, bad, tuning):
    import torch

    from tconvolve import raw

    rng, g = np.random.default_rng(n + distinct), 257
    size = 4 * WIDTHS.astype(np.int64) ** 2  # four kernels per plane
    off0 = np.concatenate([[0], np.cumsum(size)[:-1]]).astype(np.int32)
    c_len = int(size.sum())
    c = (rng.standard_normal(c_len) + 1j * rng.standard_normal(c_len)).astype(np.complex64)
    wp0 = rng.integers(0, WIDTHS.size, distinct)
    s0 = WIDTHS[wp0]
    iu0, iv0 = rng.integers(s0 // 2, g - s0 // 2), rng.integers(0, g - s0 + 1)
    co0 = off0[wp0] + rng.integers(0, 4, distinct) * s0 * s0
    pick = rng.integers(0, distinct, n) if distinct < n else np.arange(n)
    iu, iv, wp, co = (a[pick].astype(np.int32) for a in (iu0, iv0, wp0, co0))
    out_of = rng.choice(n, bad, replace=False)
    iu[out_of[::2]], co[out_of[1::2]] = -1, c_len
    good = np.ones(n, bool)
    good[out_of] = False
    z = lambda m: (rng.standard_normal(m) + 1j * rng.standard_normal(m)).astype(np.complex64)  # noqa: E731
    data, start = z(n), z(g * g)

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
    ref = start.astype(np.complex128)
    if good.any():
        iu, iv, wp, co, pick = iu[good], iv[good], wp[good], co[good], pick[good]
        ref = ref + orc.cur_grid_f64(data[good], iu, iv, wp, co, WIDTHS, c, g)
        same = np.zeros(distinct, np.complex64)
        same[pick] = vis[good]
        assert np.array_equal(same[pick], vis[good])
        assert orc.rel_l2(vis[good], orc.cur_degrid_f64(got, g, iu, iv, wp, co, WIDTHS, c)) <= REL_L2_FP32
    assert orc.rel_l2(got, ref.reshape(got.shape)) <= REL_L2_FP32
