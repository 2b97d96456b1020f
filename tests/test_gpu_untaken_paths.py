"""Paths that ordinary sizes seldom take: foci with and without bitset rings, root counts on both sides of the kernels' divide
on this device, and reports too long for the page-locked stage."""
from __future__ import annotations

import math
import random

import numpy as np
import pytest

from psuedocubes_b200 import cubes
from psuedocubes_b200.batched import BatchedEngine, Window
from psuedocubes_b200.focus import Config
from psuedocubes_b200.gpu import GPUFocus
from psuedocubes_b200.served import A_RINGS, B_RINGS

pytestmark = pytest.mark.gpu


def members(focus, low: int, high: int) -> np.ndarray:
    y = np.arange(low, high, dtype=np.int64)
    for q, residues in focus.rings:
        table = np.zeros(q, dtype=bool)
        table[list(residues)] = True
        y = y[table[y % q]]
    return y.astype(np.uint64)


# (rings of A, rings of B), table budget (0: the default), whether the foci of A and of B keep rings as bitset rows, or
# None where no division into wheel and rows fits the budget
FOCI = [((2, 2), 0, (False, False)), ((4, 3), 0, (False, False)), ((5, 4), 0, (False, False)), ((7, 5), 0, (False, False)),
        ((7, 5), 1 << 18, (True, True)), ((5, 4), 1 << 13, (True, True)), ((5, 4), 1 << 8, (None, None))]


@pytest.mark.parametrize('split, budget, rings', FOCI, ids=lambda x: str(x))
def test_foci_with_and_without_bitset_rings(runtime, split, budget, rings):
    """A focus without bitset rings keeps every wheel entry: its warps hold more than the 512 values of their stage."""
    config = Config(601, 10**20, 10**20 + 10**16, math.prod(A_RINGS[:split[0]]), math.prod(B_RINGS[:split[1]]))
    for focus, kept in zip(config.focuses(), rings):
        if kept is None:
            with pytest.raises(ValueError):
                GPUFocus(runtime, focus, budget)
            continue
        gpu = GPUFocus(runtime, focus, budget)
        assert (gpu.bitset_rings > 0) == kept
        low = focus.modulus - min(1000, focus.modulus // 2)
        high = low + min(2_000_000, 3000 * focus.modulus)
        want = members(focus, low, high)
        assert np.array_equal(gpu.window(low, high, cap=1 << 22).get(), want)
        if not kept and split != (7, 5):
            assert len(want) > 8 * 513


@pytest.mark.parametrize('p', [7, 619])
def test_counts_at_the_kernels_divide(runtime, oracle, p):
    """Counting takes long warp tasks of 9,216 k values of a class (30 numbers each) from one task per SM on."""
    groups = -(-runtime.sm_count // 8)                   # eight classes
    for tasks in (groups - 1, groups):
        for n in ((tasks * 9216 - 1) * 30, tasks * 9216 * 30, (tasks * 9216 + 1) * 30 + 7):
            for first in (1, 30 * 10**7 + 11):
                want = oracle.cube_roots(first, first + n - 1, p, threads=8)
                assert cubes.count_roots(runtime, first, first + n - 1, p) == want, (first, n)


@pytest.mark.parametrize('graph', [False, True])
def test_report_longer_than_the_stage(runtime, graph):
    """A window in so many subtiles that its counters and envelopes pass 4 MB, with more outputs than come along with them."""
    A, B = math.prod(A_RINGS[:5]), math.prod(B_RINGS[:4])
    engine = BatchedEngine(runtime)
    window = Window(139, 0, B, 10**9, 10**9 + 10**13, A, B)
    whole = engine.plan([window], None, output_cap=1 << 20)
    whole.run()
    counts, geometry, records = whole.raw()
    whole.close()
    batch = engine.plan([window], 5, output_cap=1 << 20)
    words = batch.ntiles * (batch.stride + 2)
    assert words * 8 > 4 << 20 and len(records) > 256
    batch.run(graph=graph)
    many, envelopes, split = batch.raw()
    batch.close()
    assert np.array_equal(many.sum(axis=0), counts[0])
    assert int(envelopes[:, 1].sum()) == int(geometry[0, 1])
    value = lambda r: sorted((int(b) & 0xFFFFFFFF) << 64 | int(a) for a, b in r)
    assert value(split) == value(records)
    rng = random.Random(4)
    config = window.config()
    for a, b in rng.sample(split.tolist(), 50):          # in the subtile that holds its v
        assert config.canonical((b & 0xFFFFFFFF) << 64 | a)[1] // 5 == b >> 32
