"""Subtile ranges whose bounds come out of numpy arrays: the products pass 64 bits, so they are taken in Python integers."""
from __future__ import annotations

import numpy as np
import pytest

from psuedocubes_b200.batch_experiment import tile_ranges
from psuedocubes_b200.focus import A619, B619, Config


@pytest.mark.parametrize('config', [Config(619, 10**27, 3 * 10**27, A619, B619), Config(619, 0, 10**20, A619 // 13, B619 * 13),
                                    Config(31, 0, 100000, 14 * 19, 9 * 13 * 31)], ids=['production', 'other-split', 'small'])
@pytest.mark.parametrize('kind', [np.int64, np.uint64])
def test_numpy_bounds_give_the_same_ranges(config, kind):
    first = config.B // 3
    span = min(config.B // 2, 10**10)
    for width in (span, -(-span // 7), -(-span // 63)):   # 64 subtiles at most
        want = [(v, min(v + width, first + span)) for v in range(first, first + span, width)]
        want = [(v, e, config.u_interval(v)[0], config.u_interval(e - 1)[1]) for v, e in want]
        for bounds in ((kind(first), first + span, width), (kind(first), kind(first + span), kind(width))):
            rows = tile_ranges(config, *bounds)
            assert rows == want
            assert all(type(x) is int for row in rows for x in row)
