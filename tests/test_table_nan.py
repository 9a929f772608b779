"""A table of which some planes are not numbers: its sum, and with it the whole table, is not one.

A negative baseline makes the w cell negative and its square root not a number on every plane but
w = 0 (Benchmark.cc:236-265 as written).  Bar: the same values as the oracle's, which adds in order.
"""
from __future__ import annotations

import numpy as np
import pytest


# the plane w = 0 (numbers) comes last, in the middle, and alone; tables of one block and of several
@pytest.mark.gpu
@pytest.mark.parametrize("cell,w,numbers", [(100.0, 2, False), (20.0, 2, False), (100.0, 3, False), (100.0, 1, True)])
def test_sum_of_planes_that_are_not_numbers(tcv, orc, cuda_ok, cell, w, numbers):
    from tconvolve import raw

    c, sum_c = raw.init_c(1.4e9 / 2.998e8, cell, -2000, w)
    ref_c, *_, ref_sum = orc.init_c(orc.Config(10, w, 1, 4096, cell, -2000))
    assert np.isfinite(ref_sum) == numbers == bool(np.isfinite(sum_c))
    assert np.array_equal(np.isnan(c.cpu().numpy().real), np.isnan(ref_c.real))
