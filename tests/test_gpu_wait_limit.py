"""Passes whose CTAs wait for one another's counts give up when a wait runs out, and the call is refused: with a limit of no
polls, the first tile that finds its predecessor unfinished."""
from __future__ import annotations

import time

import numpy as np
import pytest

from psuedocubes_b200.batched import BatchedEngine, Window
from psuedocubes_b200.cubes import count_roots, list_roots
from psuedocubes_b200.focus import A619, B619, Config
from psuedocubes_b200.gpu import GPUFocus, Runtime

pytestmark = pytest.mark.gpu

LOW, DEFAULT = 575222931200000000, 1 << 22
ROOTS = (10**9 + 1, 10**9 + 20_000_000, 619)             # 160 tiles


@pytest.fixture
def runtime():
    own = Runtime(time.monotonic() + 300, 8 * 1024**3)
    yield own
    own.close()


def test_windows_and_lists_are_refused_and_work_again(runtime):
    config = Config(619, 10**27, 3 * 10**27, A619, B619)
    foci = [GPUFocus(runtime, f) for f in config.focuses()]
    spans = [(LOW, LOW + 10**11), (LOW, LOW + 3 * 10**11)]
    windows = [f.window(*s, cap=1 << 24).get() for f, s in zip(foci, spans)]
    roots, count = list_roots(runtime, *ROOTS), count_roots(runtime, *ROOTS)
    runtime.lib.pc_wait_limit(runtime.ctx, 0)
    for f, s in zip(foci, spans):
        with pytest.raises(ArithmeticError, match='did not finish'):
            f.window(*s, cap=1 << 24)
    with pytest.raises(ArithmeticError, match='did not finish'):
        list_roots(runtime, *ROOTS)
    runtime.lib.pc_wait_limit(runtime.ctx, DEFAULT)
    for f, s, want in zip(foci, spans, windows):
        assert np.array_equal(f.window(*s, cap=1 << 24).get(), want)
    assert np.array_equal(list_roots(runtime, *ROOTS), roots) and count_roots(runtime, *ROOTS) == count == len(roots)


def results(batch):
    counts, geometry, records = batch.raw()
    return counts.tolist(), geometry.tolist(), sorted(records.tolist())


@pytest.mark.parametrize('graph', [False, True])
def test_a_window_batch_that_gave_up_stays_refused(runtime, graph):
    engine = BatchedEngine(runtime)
    windows = [Window(p, LOW + k * 10**12, LOW + k * 10**12 + 2 * 10**10) for k, p in enumerate((619, 613, 499))]
    good = engine.plan(windows)
    good.run(graph=graph)
    want = results(good)
    batch = engine.plan(windows)
    runtime.lib.pc_wait_limit(runtime.ctx, 0)
    with pytest.raises(ArithmeticError, match='did not finish'):
        batch.run(graph=graph)
    runtime.lib.pc_wait_limit(runtime.ctx, DEFAULT)
    for _ in range(2):
        with pytest.raises(ArithmeticError, match='did not finish'):
            batch.run(graph=graph)
    batch.close()
    other = engine.plan(windows)
    other.run(graph=graph)
    good.run(graph=graph)
    assert results(other) == results(good) == want
    other.close()
    good.close()


@pytest.mark.parametrize('graph', [False, True])
def test_no_results_of_a_failed_run(runtime, graph):
    """A batch that has run and then gives up has no results: neither the old ones nor a mixture."""
    engine = BatchedEngine(runtime)
    batch = engine.plan([Window(619, LOW, LOW + 4 * 10**10)])
    batch.run(graph=graph)
    assert batch.positions() > 0
    runtime.lib.pc_wait_limit(runtime.ctx, 0)
    with pytest.raises(ArithmeticError, match='did not finish'):
        batch.run()                                      # a recorded graph keeps the limit it was recorded with
    runtime.lib.pc_wait_limit(runtime.ctx, DEFAULT)
    with pytest.raises(ValueError, match='has not run'):
        batch.raw()
    with pytest.raises(ArithmeticError, match='did not finish'):
        batch.run(graph=graph)
    with pytest.raises(ValueError, match='has not run'):
        batch.raw()
    batch.close()
