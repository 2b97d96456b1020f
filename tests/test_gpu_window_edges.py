"""Focus windows at the edges of the one-pass kernel: units of 4,096 wheel entries, warps of one and of several
units, warps too dense for their stage (a focus without T rings), and window ends on and beside wheel members."""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import pytest

from psuedocubes_b200.batched import BatchedEngine, Window
from psuedocubes_b200.focus import Config
from psuedocubes_b200.gpu import GPUFocus
from psuedocubes_b200.served import A_RINGS, B_RINGS

pytestmark = pytest.mark.gpu

SPLITS = [(2, 2), (4, 3), (5, 4), (7, 5)]


def members(focus, low: int, high: int) -> np.ndarray:
    """The focus values of [low, high), by their residues."""
    y = np.arange(low, high, dtype=np.int64)
    for q, residues in focus.rings:
        table = np.zeros(q, dtype=bool)
        table[list(residues)] = True
        y = y[table[y % q]]
    return y.astype(np.uint64)


@pytest.mark.parametrize('split', SPLITS, ids=lambda s: f'{s[0]}-{s[1]}')
@pytest.mark.parametrize('budget', [0, 1 << 16, 1 << 20])
def test_window_edges(runtime, split, budget):
    """``budget`` bounds the tables, so the same focus runs with and without T rings."""
    config = Config(601, 10**20, 10**20 + 10**16, math.prod(A_RINGS[:split[0]]), math.prod(B_RINGS[:split[1]]))
    rng = random.Random(hash(split) % 1000 + budget)
    for focus in config.focuses():
        try:
            gpu = GPUFocus(runtime, focus, budget)
        except ValueError:                               # no division into wheel and rows fits the budget
            continue
        M, per_unit = focus.modulus, max(1, 4096 * focus.modulus // focus.count)
        for span in (0, 1, 17, per_unit - 1, per_unit, per_unit + 1, 9 * per_unit, 40 * per_unit):
            span = min(span, 3_000_000, 4000 * M)
            low = rng.randrange(0, 3 * M)
            got = gpu.window(low, low + span, cap=1 << 22).get()
            assert np.array_equal(got, members(focus, low, low + span)), (M, low, span)
        # ends on a member, just past one, and on a period
        inside = members(focus, M, M + min(M, 200_000))
        for low, high in ((int(inside[0]), int(inside[-1])), (int(inside[0]) + 1, int(inside[-1]) + 1), (M, M + min(M, 200_000)),
                          (M - 1, M + 1)):
            got = gpu.window(low, high, cap=1 << 22).get()
            assert np.array_equal(got, members(focus, low, high)), (M, low, high)


def test_window_overflow_reports_the_count(runtime, focuses619):
    fa = focuses619[0]
    low, high = 10**17, 10**17 + 10**11
    whole = fa.window(low, high, cap=1 << 22).get()
    handle, count = ctypes.c_void_p(), ctypes.c_uint64()
    for cap in (0, 1, len(whole) - 1):
        code = runtime.lib.pc_focus_window(runtime.ctx, fa.handle, low, high, cap, ctypes.byref(handle), ctypes.byref(count))
        with pytest.raises(OverflowError):
            runtime.call(code)
        assert count.value == len(whole)
    assert np.array_equal(fa.window(low, high, cap=len(whole)).get(), whole)


def test_many_units_per_warp_match_oracle(focuses619, oracle619):
    """Spans whose units give each warp several, in the middle of a period and across many."""
    _, ofa, ofb = oracle619
    for focus, of, low, span in ((focuses619[0], ofa, 123456789012345678, 3 * 10**11), (focuses619[1], ofb, 400000000000000001, 10**11)):
        assert np.array_equal(focus.window(low, low + span, cap=1 << 24).get(), of.window(low, low + span, cap=1 << 24))


@pytest.mark.parametrize('n', [1, 31, 32, 33, 255, 256, 257, 1000])
def test_searchsorted_queries_at_the_launch_limit(runtime, focuses619, n):
    """Queries passed with the launch (up to 256) and uploaded, on a whole list and on a slice of it."""
    low = 10**17
    array = focuses619[0].window(low, low + 10**10, cap=1 << 22)
    host = array.get()
    rng = np.random.default_rng(n)
    q = rng.integers(low - 10**9, low + 11 * 10**9, size=n).astype(np.uint64)
    q[::3] = host[rng.integers(0, len(host), size=len(q[::3]))]
    assert np.array_equal(array.searchsorted(q), np.searchsorted(host, q))
    part = slice(len(host) // 3, len(host) // 2)
    assert np.array_equal(array[part].searchsorted(q), np.searchsorted(host[part], q))


@pytest.mark.parametrize('graph', [False, True], ids=['eager', 'graph'])
def test_one_window_and_several_agree(runtime, graph):
    """A plan of one window passes its descriptors with the launch, a plan of more uploads them."""
    engine = BatchedEngine(runtime)
    windows = [Window(p, 10**17 + k * 10**12, 10**17 + k * 10**12 + span)
               for k, (p, span) in enumerate(((619, 10**6), (547, 3 * 10**8), (619, 10**9)))]
    every = engine.plan(windows, width=10**8)
    for _ in range(3):                                   # with a graph: eager, capture, replay
        every.run(graph=graph)
    for w, row in zip(windows, every.results()):
        alone = engine.plan([w], width=10**8)
        for _ in range(3):
            alone.run(graph=graph)
        mine = alone.results()[0]
        for key in ('focus_u', 'focus_v', 'valid_focused_candidates', 'group_survivors', 'all_values'):
            assert mine[key] == row[key], (w, key)
        alone.close()
    every.close()
