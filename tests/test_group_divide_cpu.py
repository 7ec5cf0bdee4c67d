"""The arithmetic behind the look-up of a group (group_divide in csrc/radius_graph.cu), restated: from floor((2^32 - 1) / d) the upper
half of the product is the quotient or one less, for every 32-bit dividend.  The kernels' own division is run, in boxes of many
shapes, by test_look_up_of_a_group_in_thin_boxes."""

import numpy as np
import pytest


@pytest.mark.parametrize("d", [1, 2, 3, 5, 7, 63, 64, 65, 999, 1000, 65535, 65536, 65537, 2 ** 31 - 1, 2 ** 31, 2 ** 32 - 1])
def test_quotient_and_remainder(d):
    rng = np.random.default_rng(d % 1000)
    v = np.concatenate([np.arange(0, 2000), 2 ** 32 - 1 - np.arange(0, 2000), rng.integers(0, 2 ** 32, 200_000), d * rng.integers(0, 2 ** 32 // d, 2000)])
    v = np.concatenate([v, v + 1, v - 1]).clip(0, 2 ** 32 - 1).astype(np.uint64)
    by = np.uint64((2 ** 32 - 1) // d)
    q = (v * by) >> np.uint64(32)
    rest = v - q * np.uint64(d)
    late = rest >= d
    q, rest = q + late, rest - late * np.uint64(d)
    assert (q == v // np.uint64(d)).all() and (rest == v % np.uint64(d)).all()
