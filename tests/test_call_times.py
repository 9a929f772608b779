"""Calls whose time is held against another form of the same work, measured side by side on the device.

Each bar is the ratio that the two forms' passes over memory or launches give, with a margin for noise;
medians of several runs of both in turn.
"""
from __future__ import annotations

import statistics

import pytest

pytestmark = pytest.mark.gpu


def _us(f, g, reps=9):
    """Median device times of f and g, run in turn."""
    import torch

    def once(h):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda.synchronize()
        a.record()
        h()
        b.record()
        b.synchronize()
        return 1000 * a.elapsed_time(b)

    for h in (f, g, f, g):
        once(h)
    t = [(once(f), once(g)) for _ in range(reps)]
    return tuple(statistics.median(x) for x in zip(*t))


def test_scaled_conversion_is_two_passes(tcv, cuda_ok):
    """An FP16 table takes a pass for its scale and the conversion: 8 + 8 + 2 bytes an entry where a float
    table takes 8 + 4, so 1.5 times the time, less what both have in common.  Bar: 1.5."""
    import torch

    from tconvolve import _lib, raw

    c = torch.zeros(33 * 64 * 129 * 129, dtype=torch.complex64, device="cuda")
    c.real.uniform_(-1.0, 1.0)
    two, one = _us(lambda: raw.convert_c(c, _lib.CTYPE_BY_NAME["rf16"]), lambda: raw.convert_c(c, _lib.CTYPE_BY_NAME["r32"]))
    assert two <= 1.5 * one, (two, one)


def _clean(tcv, width, d, niters):
    """Medians of AUTO and of a launch per iteration."""
    import torch

    from tconvolve.hogbom import Workspace, deconvolve_device
    from tconvolve.workload import synthetic_psf

    L = tcv.lib()
    p = torch.from_numpy(synthetic_psf(width).ravel()).cuda()
    m, r, ws = torch.zeros_like(d), torch.empty_like(d), Workspace(width)

    def form(strategy):
        def run():
            L.tcv_hogbom_set_strategy(strategy)
            deconvolve_device(d, width, p, width, m, r, niters, 0.1, 0.0, work=ws)

        return run

    try:
        return _us(form(0), form(1))
    finally:
        L.tcv_hogbom_set_strategy(0)


@pytest.mark.parametrize("width,niters", [(1900, 100), (2600, 100), (4096, 40), (4096, 100)])
def test_clean_of_a_flat_image(tcv, cuda_ok, width, niters):
    """CLEAN of noise, which is what later cycles find: put-off updates would bring most blocks up to date again
    and again, so it is a pass over the image an iteration.  Bar: a tenth over a launch per iteration."""
    import torch

    d = torch.randn(width * width, generator=torch.Generator("cuda").manual_seed(width), device="cuda")
    auto, each = _clean(tcv, width, d, niters)
    assert auto <= 1.1 * each, (auto, each)


@pytest.mark.parametrize("width,niters", [(1900, 1), (4096, 1), (4096, 5)])
def test_clean_of_few_iterations(tcv, cuda_ok, width, niters):
    """A few iterations do not pay for bringing all blocks up to date at the end.  Bar: a tenth over a launch
    per iteration."""
    import torch

    from tconvolve.workload import synthetic_dirty

    auto, each = _clean(tcv, width, torch.from_numpy(synthetic_dirty(width, 20, 1e-3, seed=5).ravel()).cuda(), niters)
    assert auto <= 1.1 * each, (auto, each)


@pytest.mark.parametrize("run,part", [(1, 0.02), (1, 0.06), (0, 0.02)])
def test_new_plan_of_a_short_track(tcv, cuda_ok, run, part):
    """A plan of a short stretch of the 12 h track, made for one gridding pass, both passes sample-parallel:
    binning costs about what it costs a plan that degrids by tiles (binned by sample, gridded alike with units
    of 512 samples).  Bar: a tenth over that."""
    import torch

    from tconvolve import current, raw

    b = current.Benchmark()
    b.setRunType(run)
    b.init()
    geo, n = b.geometry(), int(part * b.nVisibilitiesGridded())
    iu, iv, wp, co = (torch.from_numpy(a[:n].copy()).cuda() for a in b.offsets())
    (s_size, off0), c = b.planes(), torch.from_numpy(b.C()).cuda()
    b.close()
    data = torch.ones(n, dtype=torch.complex64, device="cuda")
    grid = torch.zeros(int(geo.g_size) ** 2, dtype=torch.complex64, device="cuda")
    plans = [raw.VarPlan(iu, iv, co, wp, s_size, off0, int(geo.g_size), int(geo.c_len), tuning=(8, -1, 512, 128, k)) for k in (3, 1)]
    vp = lambda t: raw._ptr(t)  # noqa: E731

    def once(plan):
        def run_():
            assert tcv.lib().tcv_plan_bin(plan.handle, vp(iu), vp(iv), vp(co), raw._stream()) == 0
            plan.grid(data, c, tcv.C64, grid)

        return run_

    both, one = _us(once(plans[0]), once(plans[1]))
    assert both <= 1.1 * one, (both, one)


@pytest.mark.parametrize("form", ["rbf16", "rf16"])
def test_gridding_in_slices_by_table_form(tcv, cuda_ok, form):
    """A few busy tiles are gridded in slices with several samples' entries in flight; a 16-bit entry is half
    a float one's bytes.  Bar: a tenth over the float table's time."""
    import numpy as np
    import torch

    from tconvolve import _lib, raw

    rng, n, support, g, planes = np.random.default_rng(2), 60000, 32, 1024, 9
    s = 2 * support + 1
    c = torch.zeros(64 * planes * s * s, dtype=torch.complex64, device="cuda")
    c.real.uniform_(-1.0, 1.0)
    d = lambda a: torch.from_numpy(a.astype(np.int32)).cuda()  # noqa: E731
    plan = raw.Plan(d(160 + rng.integers(0, 700, n)), d(128 + rng.integers(0, 700, n)),
                    d(rng.integers(0, 64 * planes, n) * s * s), support, g, c.numel())
    vis, grid = torch.ones(n, dtype=torch.complex64, device="cuda"), torch.zeros(g * g, dtype=torch.complex64, device="cuda")

    def of(name):
        tab, scale, _ = raw.convert_c(c, _lib.CTYPE_BY_NAME[name])
        return lambda: plan.grid(vis, tab, _lib.CTYPE_BY_NAME[name], grid, scale)

    half, full = _us(of(form), of("r32"))
    assert half <= 1.1 * full, (half, full)
