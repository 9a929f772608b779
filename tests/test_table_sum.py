"""The table's normalising sum: a float sum in index order, computed in parallel on the device.

Bar: bit-exact.  sumC equals the oracle's sequential float sum for the same table geometry, and the
normalised tables agree as the table's own bar says (CUDA's and the C library's cos / exp may round
a value differently near a float boundary: at most 1 entry in 2^20, by 1 ulp); where such an entry
differs the sum is compared with a sequential float sum of the device's own values instead.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (cell, planes): one plane (starts with underflowed zeros), an even and odd plane count, tables of
# one block, of many blocks and of several chunks per block, and sums past saturation
@pytest.mark.parametrize("cell,w", [(200.0, 1), (5.0, 1), (100.0, 2), (60.0, 5), (20.0, 17), (7.5, 12), (5.0, 33)])
def test_sum_is_the_sequential_float_sum(tcv, orc, cuda_ok, cell, w):
    from tconvolve import raw

    freq0 = 1.4e9 / 2.998e8
    c, sum_c = raw.init_c(freq0, cell, 2000, w)
    ref_c, *_, ref_sum = orc.init_c(orc.Config(10, w, 1, 4096, cell))
    got = c.cpu().numpy()
    a, b = got.view(np.uint32), np.ascontiguousarray(ref_c).view(np.uint32)
    diff = np.nonzero(a != b)[0]
    assert diff.size <= max(1, a.size >> 20)
    if diff.size == 0:
        assert np.float32(sum_c) == np.float32(ref_sum)
    else:  # the values before normalisation are not kept: the scale they were given is
        assert abs(float(sum_c) / float(ref_sum) - 1) < 1e-6
