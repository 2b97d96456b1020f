"""Calls on the runtime of a worker that runs leases on its helper thread: what a consumer of compute_leases asks for
between two receipts, and the receipts, are what they are without the other."""
from __future__ import annotations

import threading
import time

import numpy as np
import pytest

from psuedocubes_b200.batch_experiment import MaskedMatcher, prepare
from psuedocubes_b200.cubes import count_roots, list_roots
from psuedocubes_b200.focus import A619, B619, Config, Tile
from psuedocubes_b200.gpu import GPUFocus, Matcher, Runtime
from psuedocubes_b200.optimized import BATCH_WIDTH, compute_lease, compute_leases

pytestmark = pytest.mark.gpu

KEYS = ('focus_u', 'focus_v', 'cartesian_opportunities', 'valid_focused_candidates', 'genuine_cubes', 'local_survivors',
        'group_survivors', 'subtile_scopes', 'all_values')


def test_a_consumers_calls_do_not_mix_with_the_leases():
    runtime = Runtime(time.monotonic() + 600, 8 * 1024**3)
    config = Config(619, 10**27, 3 * 10**27, A619, B619)
    fa, fb = (GPUFocus(runtime, f) for f in config.focuses())
    masked, batches, plain = MaskedMatcher(runtime, config), MaskedMatcher(runtime, config), Matcher(runtime, config)
    low = 575222931200000000
    leases = [(low + k * 6 * BATCH_WIDTH, low + (k + 1) * 6 * BATCH_WIDTH) for k in range(10)]
    tile = Tile(low + 10**9 + 7, low + 10**9 + 7 + 30_000_000)

    def window(focus, width):
        return lambda: focus.window(low + 12345, low + 12345 + width, cap=1 << 22).get().tobytes()

    array = fb.window(low, low + 10**10, cap=1 << 22)
    queries = np.sort(np.random.default_rng(3).integers(low, low + 10**10, size=200).astype(np.uint64))
    calls = dict(window_u=window(fa, 10**9), window_v=window(fb, 7 * 10**9),
                 search=lambda: array.searchsorted(queries).tobytes(),
                 count=lambda: count_roots(runtime, 10**9 + 1, 10**9 + 5_000_000, 619),
                 list=lambda: list_roots(runtime, 10**9 + 1, 10**9 + 300_000, 547).tobytes(),
                 tile=lambda: [plain.tile(tile, fa, fb)[k] for k in ('valid_focused_candidates', 'group_survivors', 'all_values')],
                 batch=lambda: [batches.run(prepare(runtime, config, fa, fb, low, low + 10**9, 10**8))[k]
                                for k in ('valid_focused_candidates', 'group_survivors', 'all_values')])
    want = {name: call() for name, call in calls.items()}
    receipts = [compute_lease(masked, fa, fb, *lease) for lease in leases]
    done, wrong, rounds = threading.Event(), [], 0

    def consumer():
        nonlocal rounds
        while not done.is_set() or not rounds:
            for name, call in calls.items():
                got = call()
                if got != want[name]:
                    wrong.append(name)
            rounds += 1

    other = threading.Thread(target=consumer)
    other.start()
    try:
        for _ in range(4):
            for row, expected in zip(compute_leases(masked, fa, fb, leases), receipts):
                for key in KEYS:
                    assert row[key] == expected[key], key
    finally:
        done.set()
        other.join()
    assert not wrong and rounds
    runtime.close()
