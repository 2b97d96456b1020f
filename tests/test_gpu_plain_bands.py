"""The plain matcher on lists so long that each v row meets few of the u entries: rows in order, which let a CTA look for
the rows it shares positions with, against the same rows out of order, which do not, and against plain arithmetic."""
from __future__ import annotations

import ctypes
import random

import numpy as np
import pytest

from psuedocubes_b200 import _native as N
from psuedocubes_b200.focus import A619, B619, Config
from psuedocubes_b200.gpu import MASK, DeviceArray, Filters, GPUFocus

pytestmark = pytest.mark.gpu


def in_order(records: np.ndarray) -> bytes:
    rows = records.reshape(-1, 2)
    return rows[np.lexsort((rows[:, 0], rows[:, 1]))].tobytes()


class Lists:
    """A, B and (lo, hi] with u entries and v rows whose intervals meet them along a band."""
    def __init__(self, config, filters, us, vs, lo=None, hi=None):
        self.config, self.filters, self.us, self.vs = config, filters, us, vs
        self.lo, self.hi = config.lo if lo is None else lo, config.hi if hi is None else hi

    def run(self, runtime, vs, cap=1 << 18):
        f, counts, out, stats = self.filters, np.zeros(self.filters.ng + 3, dtype=np.uint64), np.zeros(2 * cap, dtype=np.uint64), N.Stats()
        du, dv = DeviceArray.from_host(runtime, self.us), DeviceArray.from_host(runtime, vs)
        runtime.call(runtime.lib.pc_run_plain(runtime.ctx, f.handle, du.handle, 0, len(self.us), dv.handle, 0, len(vs), self.lo & MASK,
                                              self.lo >> 64, self.hi & MASK, self.hi >> 64, counts, out, cap, ctypes.byref(stats)))
        n = int(counts[f.ng + 1])
        assert n <= cap
        return counts.tolist(), in_order(out[:2 * n]), stats.kernel_ms

    def positions(self):
        """Pairs with lo < u B - v A <= hi, from the exact ends of every row's interval."""
        A, B = self.config.A, self.config.B
        low = np.array([(self.lo + int(v) * A) // B for v in self.vs], dtype=np.uint64)
        high = np.array([(self.hi + int(v) * A) // B for v in self.vs], dtype=np.uint64)
        return int((np.searchsorted(self.us, high, 'right') - np.searchsorted(self.us, low, 'right')).sum())


def small(runtime, nu, nv, band, seed):
    """Arbitrary lists (duplicates among them) of a configuration of few filters, v rows of about ``band`` u entries."""
    config = Config(19, 0, 10**10, 14 * 19, 9 * 13)
    rng = np.random.default_rng(seed)
    vs = np.sort(rng.integers(0, 50 * nv, size=nv)).astype(np.uint64)
    top = 50 * nv * config.A // config.B
    us = np.sort(rng.integers(0, top + 1, size=nu)).astype(np.uint64)
    return Lists(config, Filters(runtime, config), us, vs, 3, 3 + max(1, band * top // nu) * config.B)


@pytest.mark.parametrize('nu, nv, band', [(16385, 16384, 1), (16385, 16384, 300), (1 << 18, 1024, 5), (2000, 140_001, 40),
                                          (20_000, 20_000, 600), (4_300_001, 63, 9), (4_300_001, 63, 100_000), (130, 2_100_000, 1)])
def test_ordered_rows_as_unordered_ones(runtime, nu, nv, band):
    lists = small(runtime, nu, nv, band, nu + nv + band)
    shuffled = np.random.default_rng(1).permutation(lists.vs)
    counts, values, _ = lists.run(runtime, lists.vs, 1 << 23)
    other, same, _ = lists.run(runtime, shuffled, 1 << 23)
    assert counts == other and values == same
    assert counts[0] == lists.positions() > 0


@pytest.mark.parametrize('primes', [(1021, 1019, 7, 2, 5), (7, 13, 37, 43, 61)], ids=['lookups', 'rows'])
@pytest.mark.parametrize('wrap', [False, True])
def test_entry_point_without_allocation(runtime, primes, wrap):
    """Host lists, in order and not; bounds so high that v A + hi could wrap are searched row by row."""
    rng = random.Random(sum(primes))
    A, B, nu, nv = (11 * 17, 19 * 23, 17_000, 17_000)
    if wrap:
        A = (1 << 64) - 59                               # prime
    vs = np.sort(np.random.default_rng(3).integers(10**6, 10**6 + 20 * nv, size=nv)).astype(np.uint64)
    ends = [int(v) * A // B for v in (vs[0], vs[-1])]
    us = np.sort(np.array([rng.randrange(ends[0], min(ends[1] + 900, 1 << 64)) for _ in range(nu)], dtype=np.uint64)) if ends[0] < 1 << 64 else \
        np.sort(np.random.default_rng(4).integers(0, 1 << 63, size=nu)).astype(np.uint64)
    lo, hi = 1000, 30_000 if not wrap else 1 << 70
    tables = np.array([int(rng.random() < 0.6) for q in primes for _ in range(q)], dtype=np.uint8)
    ng, cap = (len(primes) + 3) // 4, 1 << 18
    got = []
    for rows in (vs, np.random.default_rng(5).permutation(vs)):
        counts, out, err = np.zeros(ng + 3, dtype=np.uint64), np.zeros(2 * cap, dtype=np.uint64), ctypes.create_string_buffer(256)
        code = runtime.lib.pc_run_plain_static(0, us, nu, rows, nv, A, B, lo & MASK, lo >> 64, hi & MASK, hi >> 64,
                                               np.array(primes, dtype=np.uint32), len(primes), tables, counts, out, cap, err, 256)
        assert code == 0, err.value
        n = int(counts[ng + 1])
        assert n <= cap
        got.append((counts.tolist(), in_order(out[:2 * n])))
    assert got[0] == got[1]
    assert wrap or got[0][0][0] > 0


@pytest.mark.parametrize('hi', [10**27 + 10**23, 10**27 + 10**25])
def test_long_lists_take_the_time_of_their_positions(runtime, hi):
    """4.3e5 u entries and 6.8e5 v rows with 0.6 and 59 million positions: 33 ms when every CTA looks at every row."""
    config = Config(619, 10**27, hi, A619, B619)
    fa, fb = (GPUFocus(runtime, f) for f in config.focuses())
    low = 575222931200000000
    us = fa.window(config.u_interval(low)[0], config.u_interval(low + 7 * 10**10 - 1)[1], cap=1 << 22).get()
    vs = fb.window(low, low + 7 * 10**10, cap=1 << 22).get()
    lists = Lists(config, Filters(runtime, config), us, vs)
    counts, values, _ = lists.run(runtime, vs)
    other, same, _ = lists.run(runtime, np.random.default_rng(2).permutation(vs))
    assert counts == other and values == same and counts[0] == lists.positions()
    assert min(lists.run(runtime, vs)[2] for _ in range(3)) < 5
