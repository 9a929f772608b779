"""A workspace that a program keeps serves every sample count up to the one it was made for.

A plan without a tuning takes smaller degridding units for fewer samples, so its own size can be larger
for fewer; it then gives units up.  Bar: the same bits as in a workspace of its own size.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest


# a count whose units are half those of the larger one; whole cells' size (the tuned entry with its
# defaults), in which no unit fits
@pytest.mark.gpu
@pytest.mark.parametrize("n,made_for", [(53200, 53300), (53200, 0), (700, 0), (1, 0)])
def test_kept_workspace(tcv, cuda_ok, n, made_for):
    import torch

    from tconvolve._lib import TcvTuning

    L, support, g, planes = tcv.lib(), 22, 1024, 9
    s = 2 * support + 1
    c_len = 64 * planes * s * s
    whole = TcvTuning(0, 0, 0, 0, 0)
    own = L.tcv_plan_workspace_bytes(n, support, g, c_len)
    kept = (L.tcv_plan_workspace_bytes(made_for, support, g, c_len) if made_for else
            L.tcv_plan_workspace_bytes_tuned(n, support, g, c_len, ctypes.byref(whole)))
    assert kept < own  # what this test is about
    rng = np.random.default_rng(n)
    d = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    iu = d(rng.integers(support, support + 300, n).astype(np.int32))
    iv = d(rng.integers(0, 300, n).astype(np.int32))
    co = d((rng.integers(0, 64 * planes, n) * s * s).astype(np.int32))
    z = lambda m: d((rng.standard_normal(m) + 1j * rng.standard_normal(m)).astype(np.complex64))  # noqa: E731
    tab, vis, field = z(c_len), z(n), z(g * g)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    got = []
    for nb in (own, kept):
        work = torch.empty(nb, dtype=torch.uint8, device="cuda")
        grid, out = torch.zeros(g * g, dtype=torch.complex64, device="cuda"), torch.zeros(n, dtype=torch.complex64, device="cuda")
        assert L.tcv_grid_raw(vp(vis), n, support, vp(tab), tcv.C64, 1.0, c_len, vp(co), vp(iu), vp(iv), vp(grid), g,
                              vp(work), nb, st) == 0
        assert L.tcv_degrid_raw(vp(field), g, support, vp(tab), tcv.C64, 1.0, c_len, vp(co), vp(iu), vp(iv), vp(out), n,
                                vp(work), nb, st) == 0
        got.append((grid.cpu().numpy(), out.cpu().numpy()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    small = torch.empty(256, dtype=torch.uint8, device="cuda")
    assert L.tcv_degrid_raw(vp(field), g, support, vp(tab), tcv.C64, 1.0, c_len, vp(co), vp(iu), vp(iv), vp(out), n,
                            vp(small), 256, st) == 7  # TCV_ERR_WORKSPACE


@pytest.mark.gpu
def test_find_peak_in_a_small_workspace(tcv, orc, cuda_ok):
    """A peak's scan keeps a candidate per CTA: 8 KiB, not a deconvolution's workspace."""
    import torch

    L, a = tcv.lib(), np.random.default_rng(4).standard_normal(3_000_001).astype(np.float32)
    d, work = torch.from_numpy(a).cuda(), torch.empty(8192, dtype=torch.uint8, device="cuda")
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    v, p = ctypes.c_float(), ctypes.c_int64()
    assert L.tcv_find_peak(vp(d), a.size, ctypes.byref(v), ctypes.byref(p), vp(work), 8192, None) == 0
    assert (v.value, p.value) == orc.find_peak(a)
    assert L.tcv_find_peak(vp(d), a.size, ctypes.byref(v), ctypes.byref(p), vp(work), 4096, None) == 7  # TCV_ERR_WORKSPACE
