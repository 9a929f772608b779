"""The work units of a plan built without a tuning.

A plan without a tuning degrids cells that many samples crowd into in units of some samples, and grids
a few busy tiles in slices of their rows, so that they still fill the device.  Bars: the plan never outgrows the allocation-free entry's scratch where cells whole fit
it (host arithmetic); crowded samples grid and degrid within the parity bar of the FP32 path
(relative L2 1e-5 of the oracle), the same bits on every run.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import REL_L2_FP32


def test_default_units_keep_what_fits(tcv):
    from tconvolve._lib import TcvTuning

    L = tcv.lib()
    whole = TcvTuning(16, 32, 0, 0, 0)
    limit = L.tcv_static_scratch_bytes()
    for n in (1, 100, 16000, 60000, 100000, 160000, 269745, 400000, 2000000):
        for support, g in ((0, 128), (3, 64), (14, 256), (22, 1024), (64, 4096), (64, 16384), (200, 8192)):
            s = 2 * support + 1
            a = L.tcv_plan_workspace_bytes_tuned(n, support, g, 64 * s * s * 9, ctypes.byref(whole))
            b = L.tcv_plan_workspace_bytes(n, support, g, 64 * s * s * 9)
            assert b >= a > 0
            assert a > limit or b <= limit, (n, support, g)


@pytest.mark.gpu
@pytest.mark.parametrize("n,support,g,spread", [
    (63, 10, 64, 1),        # one cell, under two units: not cut
    (64, 10, 64, 1),        # exactly two units of 32
    (5000, 10, 129, 40),    # ragged counts, tiles at the grid's edge
    (20000, 3, 100, 50),
    (3000, 64, 300, 20),
])
def test_crowded_samples_match_oracle(tcv, orc, cuda_ok, n, support, g, spread):
    import torch

    from tconvolve import raw

    rng = np.random.default_rng(n)
    s, planes = 2 * support + 1, 2
    c_len = 64 * planes * s * s
    table64 = rng.standard_normal(c_len).astype(np.float32).astype(np.float64)  # real, as the attic table
    table = table64.astype(np.complex64)
    lo, hi = support, g - 1 - 2 * support
    at = lambda: np.clip(lo + rng.integers(0, max(1, min(spread, hi - lo + 1)), n), lo, hi).astype(np.int32)  # noqa: E731
    iu, iv = at(), at()
    coff = (rng.integers(0, 64 * planes, n) * s * s).astype(np.int32)
    vis = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    start = (rng.standard_normal(g * g) + 1j * rng.standard_normal(g * g)).astype(np.complex64)

    d = lambda a: torch.from_numpy(a.copy()).cuda()  # noqa: E731
    diu, div, dco, dc = d(iu), d(iv), d(coff), d(table)
    runs = []
    for _ in range(2):
        grid, out = d(start), torch.zeros(n, dtype=torch.complex64, device="cuda")
        raw.grid_raw(d(vis), support, dc, tcv.C64, 1.0, dco, diu, div, grid, g)
        raw.degrid_raw(grid, g, support, dc, tcv.C64, 1.0, dco, diu, div, out)
        runs.append((grid.cpu().numpy(), out.cpu().numpy()))
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
    grid64 = start.astype(np.complex128)
    orc.grid_f64(vis, support, table64, coff, iu, iv, grid64, g)
    out64 = orc.degrid_f64(grid64, g, support, table64, coff, iu, iv)
    assert orc.rel_l2(runs[0][0], grid64) <= REL_L2_FP32
    assert orc.rel_l2(runs[0][1], out64) <= REL_L2_FP32


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [8, 16, 32])
@pytest.mark.parametrize("form", ["c64", "r32", "rbf16"])
@pytest.mark.parametrize("n,support", [(1, 10), (257, 10), (3000, 3), (1500, 40)])
def test_whole_cells_in_slices_keep_their_bits(tcv, orc, cuda_ok, rows, form, n, support):
    """A plan group with few busy tiles is gridded in slices of its tiles; samples of zero data all over
    the grid make many tiles busy, which grids them whole.  The crowd's points get the same bits."""
    import torch

    from tconvolve import _lib, raw

    rng = np.random.default_rng(n + support)
    g, s = 2048, 2 * support + 1
    c_len = 64 * s * s
    c64 = torch.from_numpy(rng.standard_normal(c_len).astype(np.float32).astype(np.complex64)).cuda()
    code = _lib.CTYPE_BY_NAME[form]
    tab, scale = (c64, 1.0) if form == "c64" else raw.convert_c(c64, code)[:2]
    iu = (700 + rng.integers(0, 60, n)).astype(np.int32)
    iv = (900 + rng.integers(0, 60, n)).astype(np.int32)
    far = np.arange(support, g - s, 32 if support < 30 else 60, dtype=np.int32)
    fu, fv = (a.ravel().astype(np.int32) for a in np.meshgrid(far, far))
    coff = (rng.integers(0, 64, n) * s * s).astype(np.int32)
    vis = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    grids = []
    for crowd in (True, False):
        u, v, co, x = iu, iv, coff, vis
        if not crowd:
            u, v = np.concatenate([iu, fu]), np.concatenate([iv, fv])
            co = np.concatenate([coff, np.zeros(fu.size, np.int32)])
            x = np.concatenate([vis, np.zeros(fu.size, np.complex64)])
        plan = raw.Plan(d(u), d(v), d(co), support, g, c_len, tuning=(rows, -1, 0, 0))
        grid = torch.zeros(g * g, dtype=torch.complex64, device="cuda")
        plan.grid(d(x), tab, code, grid, scale)
        assert plan.rejected() == 0
        grids.append(grid.cpu().numpy())
    assert np.count_nonzero(grids[0]) > 0
    assert np.array_equal(grids[0], grids[1])
