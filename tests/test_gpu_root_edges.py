"""The cube-root sieve at the edges of its two kernels (tiles of 4,096 k values for lists and short counts,
long warp tasks for counts) and of its residue classes, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from psuedocubes_b200 import cubes

pytestmark = pytest.mark.gpu

TILE = 30 * 4096


@pytest.mark.parametrize('p', [2, 3, 4, 5, 7, 31, 257, 619, 1999, 2000])
def test_lists_at_class_and_tile_edges(runtime, oracle, p):
    for first, n in ((1, 1), (1, 31), (2, 29), (29, 3), (30, 1), (31, 30), (TILE - 1, 2), (TILE + 7, TILE - 14), (123457, TILE + 1),
                     (10**9 + 1, 3 * TILE + 11), (2**32 - 61, 61)):
        want = oracle.cube_roots(first, first + n - 1, p, listed=True)
        assert np.array_equal(cubes.list_roots(runtime, first, first + n - 1, p), want), (first, n)
        assert cubes.count_roots(runtime, first, first + n - 1, p) == len(want), (first, n)


@pytest.mark.parametrize('p', [5, 13, 619, 997, 1999])
def test_long_counts_match_oracle(runtime, oracle, p):
    """Ranges on both sides of the point where counting takes the long-task kernel (one task of 9, 5 or 3
    words per lane and class for each of 148 SMs), and across several tasks per warp."""
    for run in (9, 5, 3):
        point = 148 // 8 * 30 * 1024 * run
        for first, n in ((1, point - 12345), (7, point + 30 * 1024 * run + 1), (2**32 - 7 * point, 7 * point)):
            want = oracle.cube_roots(first, first + n - 1, p, threads=8)
            assert cubes.count_roots(runtime, first, first + n - 1, p) == want, (first, n)


def test_whole_range_count_matches_oracle(runtime, oracle):
    for p in (31, 619):
        assert cubes.count_roots(runtime, 1, 2**32 - 1, p) == oracle.cube_roots(1, 2**32 - 1, p, threads=8)


@pytest.mark.parametrize('p', [251, 257, 263, 443, 449, 1999])
def test_struck_primes_match_oracle(runtime, oracle, p):
    """No, one, two, 32 and 33 primes above the largest with a pattern, around whole tasks of 9,216 k values."""
    task = 30 * 9216
    for first, n in ((1, 20 * task), (30 * 10**6 + 1, 19 * task + 31), (2**32 - 21 * task + 1, 21 * task - 1)):
        want = oracle.cube_roots(first, first + n - 1, p, threads=8)
        assert cubes.count_roots(runtime, first, first + n - 1, p) == want, (first, n)
