"""Survivor slices that a window batch outgrows: where larger ones do not fit the memory cap the run is refused, and the
batch works once there is room; runs with and without a recorded graph in any order give the same results."""
from __future__ import annotations

import ctypes
import time

import numpy as np
import pytest

from psuedocubes_b200.batched import BatchedEngine, Window
from psuedocubes_b200.gpu import DeviceArray, Runtime

pytestmark = pytest.mark.gpu

LOW = 575222931200000000
WINDOWS = [Window(p, LOW + k * 10**12, LOW + k * 10**12 + 10**10) for k, p in enumerate((619, 613, 499))]


@pytest.fixture
def runtime():
    own = Runtime(time.monotonic() + 300, 1 << 30)
    yield own
    own.close()


def left(runtime: Runtime) -> int:
    words = [ctypes.c_uint64() for _ in range(3)]
    runtime.lib.pc_mem_info(runtime.ctx, *[ctypes.byref(w) for w in words])
    return words[2].value - words[0].value


def results(batch):
    counts, geometry, records = batch.raw()
    return counts.tolist(), geometry.tolist(), sorted(records.tolist())


@pytest.mark.parametrize('graph', [False, True])
def test_a_batch_works_again_after_slices_did_not_fit(runtime, graph):
    engine = BatchedEngine(runtime)
    roomy = engine.plan(WINDOWS, None)
    roomy.run()
    want = results(roomy)
    roomy.close()
    batch = engine.plan(WINDOWS, None, dict(deep_records=1))
    taken = DeviceArray.from_host(runtime, np.zeros((left(runtime) - (1 << 20)) // 8, dtype=np.uint64))
    for _ in range(3):                                   # slices of 1,024 records and more take 2.4 MB
        with pytest.raises(MemoryError):
            batch.run(graph=graph)
    del taken
    for again in (graph, True, False):
        batch.run(graph=again)
        assert results(batch) == want
    batch.close()


def test_runs_with_and_without_a_graph_in_any_order(runtime):
    engine = BatchedEngine(runtime)
    batch = engine.plan(WINDOWS, None, dict(deep_records=3))
    batch.run()
    want = results(batch)
    for graph in (True, False, False, True, True, False, True):
        batch.run(graph=graph)
        assert results(batch) == want
    batch.close()
