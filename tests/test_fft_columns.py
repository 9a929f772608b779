"""Image transforms of the sizes whose columns are transformed whole, against double precision.

Bar: relative L2 of 0.6 u log2(points), u = 2^-24, the rounding error of a single-precision transform
whose stages each round once or twice.
"""
from __future__ import annotations

import math

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [256, 512, 1024, 2048])
def test_whole_columns(tcv, cuda_ok, n):
    import torch

    from tconvolve import major

    rng = np.random.default_rng(n)
    bar = 0.6 * 2.0 ** -24 * math.log2(n * n)
    shift = np.fft.fftshift
    x = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))).astype(np.complex64)
    m = rng.standard_normal((n, n)).astype(np.float32)
    err = lambda got, ref: np.linalg.norm(got.reshape(n, n) - ref) / np.linalg.norm(ref)  # noqa: E731
    for forward in (True, False):
        g = torch.from_numpy(x.reshape(-1).copy()).cuda()
        major.fft_exec(g, n, forward)
        f = np.fft.fft2 if forward else lambda a: np.fft.ifft2(a) * float(n * n)
        assert err(g.cpu().numpy(), shift(f(shift(x.astype(np.complex128))))) <= bar
    grid = torch.empty(n * n, dtype=torch.complex64, device="cuda")
    major.grid_from_image(torch.from_numpy(m.reshape(-1)).cuda(), n, grid)
    assert err(grid.cpu().numpy(), shift(np.fft.fft2(shift(m.astype(np.float64))))) <= bar
    image = torch.empty(n * n, dtype=torch.float32, device="cuda")
    major.image_from_grid(grid, n, float(n) ** -2.0, image)
    assert err(image.cpu().numpy(), m) <= 2 * bar
