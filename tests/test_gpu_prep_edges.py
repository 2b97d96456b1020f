"""Per-row bounds (k_vprep) in every way it finds them: rows as distances from their CTA's first row, staged or
not, rows of CTAs and warps that span segments, and moduli too large for 64-bit bounds."""
from __future__ import annotations

import random

import numpy as np
import pytest

from psuedocubes_b200.batch_experiment import MaskedMatcher, compare, prepare
from psuedocubes_b200.batched import BatchedEngine, Window
from psuedocubes_b200.focus import A619, B619, Config
from psuedocubes_b200.gpu import GPUFocus, Matcher
from psuedocubes_b200.run_production import compute_batch

pytestmark = pytest.mark.gpu

FIELDS = ('valid_focused_candidates', 'group_survivors', 'local_survivors', 'genuine_cubes', 'all_values', 'subtile_scopes')


def rows_span(rows: float) -> int:
    """A v span that holds about ``rows`` values of B619's focus."""
    return int(rows * 1.0368e5) + 1


@pytest.mark.parametrize('rows', [(3,), (20, 40, 11), (31, 32, 33, 64), (200, 300, 5, 700, 1), (1500, 2, 2, 2, 4000)], ids=str)
def test_windows_together_equal_windows_alone(runtime, rows):
    """Windows of a few rows to several CTAs' rows: one launch over all of them against one launch each."""
    rng = random.Random(sum(rows))
    engine = BatchedEngine(runtime)
    windows = []
    for k in range(40):
        span = rows_span(rows[k % len(rows)])
        first = rng.randrange(0, B619 - span)
        windows.append(Window(rng.choice((499, 547, 619)), first, first + span))
    batch = engine.plan(windows, width=10**7)
    batch.run()
    together = batch.results()
    batch.close()
    for w, row in list(zip(windows, together))[::7]:
        alone = engine.plan([w], width=10**7)
        alone.run()
        want = alone.results()[0]
        alone.close()
        assert all(row[k] == want[k] for k in FIELDS), w


@pytest.mark.parametrize('A, B, width', [(A619 // 13, B619 * 13, 10**9),            # B > 2^62: 128-bit bounds
                                         (A619, B619 // 163, 4 * 10**6),            # 57 u values per v row: not staged
                                         (A619 // 181 // 157, B619, 10**8)],
                         ids=['B>2^62', 'wide bounds', 'A<B'])
def test_masked_equals_plain_at_other_moduli(runtime, A, B, width):
    config = Config(619, 10**27, 10**27 + 10**25, A, B)
    af, bf = (GPUFocus(runtime, f) for f in config.focuses())
    first, end = B // 3, B // 3 + 5 * width + width // 3
    masked = MaskedMatcher(runtime, config).run(prepare(runtime, config, af, bf, first, end, width))
    plain = compute_batch(Matcher(runtime, config), af, bf, first, end, width)
    assert masked['valid_focused_candidates'] > 1000
    for key in FIELDS[:5]:
        assert masked[key] == plain[key], key


@pytest.mark.parametrize('tuning', [{}, dict(bitset_filters=4, block_words=16, threads=512), dict(bitset_filters=5, block_words=64, threads=512)],
                         ids=['default', '4x16', '5x64'])
def test_few_rows_per_block_equal_plain(runtime, tuning):
    """Windows of one to forty v rows (blocks whose rows are made for them alone, and whole blocks) against the
    plain per-tile loop."""
    rng = random.Random(len(tuning))
    engine = BatchedEngine(runtime)
    windows = []
    for rows in (1, 2, 5, 9, 12, 14, 16, 17, 18, 19, 20, 24, 30, 40):
        first = rng.randrange(0, B619 - 10**9)
        windows.append(Window(rng.choice((499, 547, 619)), first, first + rows_span(rows)))
    batch = engine.plan(windows, width=10**6, tuning=tuning)
    batch.run()
    for w, row in zip(windows, batch.results()):
        c = w.config()
        want = compute_batch(Matcher(runtime, c), *engine.focus_pair(c), w.first, w.end, 10**8)
        assert all(row[k] == want[k] for k in FIELDS[:4]), w
        assert sorted(row['all_values']) == sorted(want['all_values']), w
    batch.close()
