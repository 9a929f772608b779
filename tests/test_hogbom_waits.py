"""Hogbom CLEAN: the bounded waits of every form whose CTAs wait for one another.

Each form is told to wait for one candidate or arrival more than is ever made, with a short limit.  Every CTA
must give up and return, the loop stops after its first iteration, later launches do nothing and the
result reports TCV_ERR_TIMEOUT.  With the default wait restored, a run in the same workspace equals a
launch per iteration (no waits), bit for bit.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AUTO, PER_LAUNCH, PERSISTENT = 0, 1, 2


def _check(strategy, w, limit_ns, niters=150):
    import torch

    from tconvolve._lib import lib
    from tconvolve.hogbom import Workspace, deconvolve_device
    from tconvolve.workload import synthetic_dirty, synthetic_psf

    L = lib()
    d = torch.from_numpy(synthetic_dirty(w, 15, 1e-3, seed=21).ravel()).cuda()
    p = torch.from_numpy(synthetic_psf(w).ravel()).cuda()
    m, r, ws = torch.zeros_like(d), torch.empty_like(d), Workspace(w)
    try:
        L.tcv_hogbom_set_strategy(strategy)
        assert L.tcv_hogbom_set_wait(limit_ns, 1) == 0
        deconvolve_device(d, w, p, w, m, r, niters, 0.1, 0.0, work=ws)
        torch.cuda.synchronize()  # returns: every CTA left its kernel
        done, stop = ctypes.c_int(), ctypes.c_int()
        st = L.tcv_hogbom_result(ctypes.c_void_p(ws.buf.data_ptr()), ctypes.byref(done), ctypes.byref(stop), None, None, None)
        assert (st, done.value, stop.value) == (5, 1, -1)  # TCV_ERR_TIMEOUT
        assert L.tcv_hogbom_set_wait(2_000_000_000, 0) == 0
        runs = []
        for form in (strategy, PER_LAUNCH):
            L.tcv_hogbom_set_strategy(form)
            m.zero_()
            deconvolve_device(d, w, p, w, m, r, niters, 0.1, 0.0, work=ws)
            assert ws.result()["done"] == niters
            runs.append((m.cpu().numpy(), r.cpu().numpy()))
    finally:
        L.tcv_hogbom_set_wait(2_000_000_000, 0)
        L.tcv_hogbom_set_strategy(AUTO)
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])


# one cluster; several clusters; put-off updates (the leading cluster)
@pytest.mark.parametrize("width", [128, 700, 2100])
@pytest.mark.parametrize("limit_ns", [0, 1_000_000])
def test_waits_run_out(tcv, cuda_ok, width, limit_ns):
    _check(AUTO, width, limit_ns)


# the persistent form has waits at every size: widths that the registers do not hold, and odd ones
@pytest.mark.parametrize("width", [1793, 2048, 2601, 4096])
def test_persistent_form_is_cooperative(tcv, cuda_ok, width):
    _check(PERSISTENT, width, 1_000_000, niters=20)
