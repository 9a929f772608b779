"""Hogbom CLEAN beyond the register-resident sizes: put-off updates, passes over the image, and the changes
from one to the other, on images at the edges of both.

Bar: bit-exact against the oracle (model, residual, every iteration's peak, the counts), whichever form an
iteration takes.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W = 2100


def _bright(sources=6, noise=1e-3, seed=3, w=W):
    from tconvolve.workload import synthetic_dirty

    return synthetic_dirty(w, sources, noise, seed=seed)


def _check(orc, dirty, psf, niters, threshold=0.0, gain=0.1):
    import torch

    from tconvolve.hogbom import deconvolve_device

    w, p = dirty.shape[0], psf.shape[0]
    d, k = torch.from_numpy(dirty.ravel().copy()).cuda(), torch.from_numpy(psf.ravel().copy()).cuda()
    m, r = torch.zeros_like(d), torch.empty_like(d)
    hv = torch.zeros(max(niters, 1), dtype=torch.float32, device="cuda")
    hp = torch.zeros(max(niters, 1), dtype=torch.int32, device="cuda")
    res = deconvolve_device(d, w, k, p, m, r, niters, gain, threshold, hist=(hv, hp)).result()
    o = orc.hogbom(dirty, psf, niters, gain, threshold)
    n = o["done"]
    assert (res["done"], res["stopped_at"], res["skipped_rows"]) == (n, o["stopped_at"], o["skipped_rows"])
    assert res["psf_peak_pos"] == o["psf_peak_pos"]
    assert np.array_equal(hp.cpu().numpy()[:n], o["hist_pos"][:n]) and np.array_equal(hv.cpu().numpy()[:n], o["hist_val"][:n])
    for got, want in ((m, o["model"]), (r, o["residual"])):
        assert np.array_equal(got.cpu().numpy(), want.ravel(), equal_nan=True)
    return o


# one iteration, a launch less and more, a ring of pending updates less and more, several rings
@pytest.mark.parametrize("niters", [1, 2, 15, 17, 127, 128, 129, 300])
def test_put_off_rings(tcv, orc, cuda_ok, niters):
    from tconvolve.workload import synthetic_psf

    _check(orc, _bright(20), synthetic_psf(W), niters)


# a threshold met at the first peak, inside the first launch, at a launch's and a ring's end, in a later ring
@pytest.mark.parametrize("stop", [0, 5, 16, 37, 128, 137])
def test_put_off_stops(tcv, orc, cuda_ok, stop):
    from tconvolve.workload import synthetic_psf

    dirty, psf = _bright(20), synthetic_psf(W)
    peaks = np.abs(orc.hogbom(dirty, psf, stop + 1, 0.1, 0.0)["hist_val"])
    threshold = np.nextafter(peaks[stop], np.float32(np.inf)) if stop == 0 else np.float32(peaks[stop] + peaks[:stop].min()) / 2
    assert _check(orc, dirty, psf, 300, float(threshold))["stopped_at"] == stop


@pytest.mark.parametrize("kind", ["ties", "nan", "inf", "inf psf", "nan psf", "flat psf", "off diagonal", "corner psf",
                                  "small psf", "large psf", "tiny", "negative", "zeros", "whole gain", "no gain"])
def test_put_off_images(tcv, orc, cuda_ok, kind):
    from tconvolve.workload import synthetic_psf

    dirty, psf, n, gain = _bright(), synthetic_psf(W), 60, 0.1
    if kind == "ties":  # the first index wins, over blocks, warps and the cluster's CTAs
        dirty = np.zeros((W, W), np.float32)
        dirty[5:2100:190, 7:2100:310] = 1.0
        dirty[100:2100:400, 9:2100:610] = -1.0
    elif kind == "nan":
        dirty[1000, 990:1010] = dirty[40, 50] = np.nan
        dirty[2099, 2099] = np.nan
    elif kind == "inf":  # the peak is infinite: the update turns its surroundings into NaN
        dirty[800, 900] = np.inf
        n = 4
    elif kind == "inf psf":
        psf[W // 2 + 3, W // 2 + 40] = np.inf
        n = 4
    elif kind == "nan psf":
        psf[W // 2 + 70, W // 2 - 40] = np.nan
    elif kind == "flat psf":  # every update reaches every block in full
        psf = np.full((W, W), 0.5, np.float32)
        psf[W // 2, W // 2] = 1.0
    elif kind == "off diagonal":  # rows of the PSF that the reference's row index leaves out
        psf = np.ascontiguousarray(np.roll(np.roll(psf, 210, axis=1), -130, axis=0))
    elif kind == "corner psf":  # no row left in
        psf = np.ascontiguousarray(np.roll(np.roll(psf, W // 2 - 1, axis=1), -W // 2, axis=0))
    elif kind == "small psf":
        psf = synthetic_psf(33)
    elif kind == "large psf":
        psf = synthetic_psf(4301)
    elif kind == "tiny":  # subnormal values and products
        dirty = (dirty * np.float32(1e-39)).astype(np.float32)
    elif kind == "negative":
        dirty = -dirty
    elif kind == "zeros":
        dirty = np.zeros((W, W), np.float32)
    elif kind == "whole gain":
        gain = 1.0
    elif kind == "no gain":
        gain, n = 0.0, 20
    _check(orc, dirty, psf, n, gain=gain)


# a flat image from the start, and one bright source over noise: flat before the first ring ends
@pytest.mark.parametrize("width,bright,niters,threshold", [
    (2100, 0.0, 140, 0.0), (2099, 0.0, 20, 4.9), (2100, 60.0, 300, 0.0), (2099, 60.0, 129, 0.0), (2100, 60.0, 300, 4.2),
    (4100, 0.0, 12, 0.0), (4100, 60.0, 140, 0.0),
])
def test_passes_take_over(tcv, orc, cuda_ok, width, bright, niters, threshold):
    from tconvolve.workload import synthetic_psf

    dirty = np.random.default_rng(width).standard_normal((width, width)).astype(np.float32)
    psf = synthetic_psf(1051)
    dirty[200:1251, 500:1551] += np.float32(bright) * psf
    _check(orc, dirty, psf, niters, threshold)


# a captured call replays as it ran: launches each, passes, put-off updates, passes that take over
@pytest.mark.parametrize("width,niters,noise", [(2100, 2, 0.0), (2100, 5, 0.0), (2100, 150, 0.0), (2100, 20, 1.0), (2099, 20, 0.0)])
def test_captured_call(tcv, cuda_ok, width, niters, noise):
    import torch

    from tconvolve.hogbom import Workspace, deconvolve_device
    from tconvolve.workload import synthetic_psf

    host = np.random.default_rng(7).standard_normal((width, width)).astype(np.float32)
    d = torch.from_numpy((host * np.float32(noise) if noise else _bright(w=width)).ravel().copy()).cuda()
    p = torch.from_numpy(synthetic_psf(width).ravel()).cuda()
    m, r, ws = torch.zeros_like(d), torch.empty_like(d), Workspace(width)
    deconvolve_device(d, width, p, width, m, r, niters, 0.1, 0.0, work=ws)
    want = (m.clone(), r.clone())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        m.zero_()
        deconvolve_device(d, width, p, width, m, r, niters, 0.1, 0.0, work=ws)
    for _ in range(2):
        m.fill_(3.0)
        r.fill_(3.0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(m, want[0]) and torch.equal(r, want[1])
        assert ws.result()["done"] == niters
