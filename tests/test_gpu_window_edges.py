"""Focus windows at the edges of the one-pass kernel: units of 4,096 wheel entries, warps of one and of several
units, warps too dense for their stage (a focus without T rings), and window ends on and beside wheel members."""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import pytest

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
