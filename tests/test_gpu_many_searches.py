"""Sorted searches with more queries than the launch carries, up to and past the number that takes a lane per query."""
from __future__ import annotations

import numpy as np
import pytest

from psuedocubes_b200.gpu import DeviceArray

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('length', [0, 1, 7, 8, 1000, 300_001])
@pytest.mark.parametrize('n', [(1 << 17) - 1, 1 << 17, (1 << 17) + 1, 700_001])
def test_many_queries(runtime, length, n):
    rng = np.random.default_rng(length * 7 + n)
    values = np.sort(rng.integers(0, 3 * length + 2, size=length).astype(np.uint64) * np.uint64(1 << 40))   # duplicates among them
    queries = rng.integers(0, 3 * length + 3, size=n).astype(np.uint64) * np.uint64(1 << 40) + rng.integers(0, 3, size=n).astype(np.uint64)
    queries[:2] = 0, (1 << 64) - 1
    array = DeviceArray.from_host(runtime, values)
    assert np.array_equal(array.searchsorted(queries), np.searchsorted(values, queries).astype(np.uint64))
    if length > 8:
        part = array[3:length - 2]
        assert np.array_equal(part.searchsorted(queries), np.searchsorted(values[3:length - 2], queries).astype(np.uint64))

