"""Hogbom CLEAN with put-off updates (the cooperative loop): sizes and images at its edges.

Bar: bit-exact against the oracle (model, residual, every iteration's peak): the updates of a pixel
are applied in order with the reference's roundings, whenever they are applied.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(dirty, psf, niters, gain=0.1, threshold=0.0):
    import torch

    from tconvolve.hogbom import deconvolve_device

    w, p = dirty.shape[0], psf.shape[0]
    d, k = torch.from_numpy(dirty.ravel().copy()).cuda(), torch.from_numpy(psf.ravel().copy()).cuda()
    m, r = torch.zeros_like(d), torch.empty_like(d)
    hv = torch.zeros(max(niters, 1), dtype=torch.float32, device="cuda")
    hp = torch.zeros(max(niters, 1), dtype=torch.int32, device="cuda")
    ws = deconvolve_device(d, w, k, p, m, r, niters, gain, threshold, hist=(hv, hp))
    return m.cpu().numpy(), r.cpu().numpy(), hv.cpu().numpy(), hp.cpu().numpy(), ws.result()


def _check(orc, dirty, psf, niters, threshold=0.0):
    m, r, hv, hp, res = _run(dirty, psf, niters, threshold=threshold)
    o = orc.hogbom(dirty, psf, niters, 0.1, threshold)
    n = o["done"]
    assert res["done"] == n and res["stopped_at"] == o["stopped_at"] and res["skipped_rows"] == o["skipped_rows"]
    assert np.array_equal(hp[:n], o["hist_pos"][:n]) and np.array_equal(hv[:n], o["hist_val"][:n])
    same = lambda a, b: np.array_equal(a, b.reshape(a.shape), equal_nan=True)  # noqa: E731
    assert same(m, o["model"]) and same(r, o["residual"])


# one block, ragged blocks, a block more than a power of two, blocks of 64 (more than 128 of 32 per
# side); PSFs smaller and larger than the image and of other block sizes; more iterations than the
# ring of pending updates holds
@pytest.mark.parametrize("width,psf,niters", [
    (1, 1, 5), (5, 3, 20), (31, 31, 60), (32, 64, 60), (33, 17, 60), (97, 195, 1030), (257, 257, 2100),
    (300, 40, 400), (64, 4100, 30), (4100, 64, 60), (4099, 4099, 12),
    # the residual in registers: each number of columns and rows per thread
    (600, 600, 40), (1025, 515, 30), (1430, 715, 40), (1537, 1537, 12), (2000, 333, 30), (2048, 2049, 10), (2049, 2048, 20),
])
def test_sizes(tcv, orc, cuda_ok, width, psf, niters):
    from tconvolve.workload import synthetic_dirty, synthetic_psf

    dirty = synthetic_dirty(width, 8, 1e-2, seed=width) if width > 4 else np.full((1, 1), 0.75, np.float32)
    _check(orc, dirty, synthetic_psf(psf), niters)


@pytest.mark.parametrize("kind", ["zeros", "equal", "noise", "nan", "inf", "flat psf", "off diagonal", "tiny"])
def test_images(tcv, orc, cuda_ok, kind):
    from tconvolve.workload import synthetic_dirty, synthetic_psf

    w, n = 160, 80
    rng = np.random.default_rng(5)
    dirty, psf = synthetic_dirty(w, 12, 1e-3, seed=3), synthetic_psf(w)
    if kind == "zeros":  # every candidate is zero: the peak is (0, index 0) as findPeak returns it
        dirty = np.zeros((w, w), np.float32)
    elif kind == "equal":  # ties everywhere: the first index wins
        dirty = np.where(rng.random((w, w)) < 0.5, 1.0, -1.0).astype(np.float32)
    elif kind == "noise":
        dirty = rng.standard_normal((w, w)).astype(np.float32)
    elif kind == "nan":
        dirty[40, 50] = dirty[100:140, 33] = np.nan
    elif kind == "inf":  # the peak is infinite: the update turns its surroundings into NaN
        dirty[80, 80] = np.inf
        n = 4
    elif kind == "flat psf":  # every update reaches every block in full
        psf = np.full((w, w), 0.5, np.float32)
        psf[w // 2, w // 2] = 1.0
    elif kind == "off diagonal":
        psf = np.ascontiguousarray(np.roll(np.roll(psf, 21, axis=1), -13, axis=0))
    elif kind == "tiny":  # subnormal values and products
        dirty, psf = (dirty * np.float32(1e-39)).astype(np.float32), psf
    _check(orc, dirty, psf, n)


@pytest.mark.parametrize("width,psf,niters,threshold", [
    (2100, 2100, 260, 0.0),   # noise: many blocks stay hot, passes take over at iteration 128, mid-ring end
    (2099, 1050, 257, 0.0),   # a ragged width, one iteration in the last ring
    (2100, 2101, 400, 4.16),  # the threshold stops a launch of passes
])
def test_passes_take_over(tcv, orc, cuda_ok, width, psf, niters, threshold):
    from tconvolve.workload import synthetic_psf

    dirty = np.random.default_rng(width + psf).standard_normal((width, width)).astype(np.float32)
    _check(orc, dirty, synthetic_psf(psf), niters, threshold)
