"""A launch of many blocks with one much larger than the rest: its work is divided like everything else's."""
from __future__ import annotations

import numpy as np
import pytest

from psuedocubes_b200.batched import BatchedEngine, Window
from psuedocubes_b200.focus import B619

pytestmark = pytest.mark.gpu

LOW = 575222931200000000
WIDE = [Window(619, LOW + k * 5 * 10**10, LOW + (k + 1) * 5 * 10**10) for k in range(8)]


def few_u(span: int) -> Window:
    """Some twenty u entries and a v row per 10^5 of the span."""
    return Window(619, LOW, LOW + span, 10**27, 10**27 + 10**20, 14, B619)


def counters(engine: BatchedEngine, windows: list[Window], tuning=None) -> tuple[np.ndarray, np.ndarray, float]:
    batch = engine.plan(windows, None, tuning)
    times = []
    for _ in range(4):
        batch.run()
        times.append(batch.last_stats['kernel_ms'])
    counts, geometry, _ = batch.raw()
    got = counts.copy(), geometry.copy(), min(times)
    batch.close()
    return got


@pytest.mark.parametrize('place', [0, 4, 8])
def test_large_block_among_many(runtime, place):
    engine = BatchedEngine(runtime)
    each = {w: counters(engine, [w])[:2] for w in [*WIDE, few_u(10**11), few_u(10**12)]}
    _, _, without = counters(engine, WIDE)
    for extra in (few_u(10**11), few_u(10**12)):
        windows = [*WIDE[:place], extra, *WIDE[place:]]
        counts, geometry, ms = counters(engine, windows)
        for row, geo, w in zip(counts, geometry, windows):
            ng = (len(w.config().filter_order()) + 3) // 4
            assert np.array_equal(row[:ng + 3], each[w][0][0][:ng + 3]) and np.array_equal(geo, each[w][1][0])
        # 10^6 and 10^7 rows in one block: 5 and 45 ms of one CTA; the launch without them takes 2.7 ms
        assert ms < 2 * without, (place, ms, without)


def test_item_lengths_within_an_uneven_launch(runtime):
    engine = BatchedEngine(runtime)
    windows = [*WIDE, few_u(10**11)]
    counts, geometry, _ = counters(engine, windows)
    for v_chunk in (1000, 33):
        other, geo, _ = counters(engine, windows, dict(v_chunk=v_chunk))
        assert np.array_equal(counts, other) and np.array_equal(geometry, geo)
