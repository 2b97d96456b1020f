"""Focus windows and root lists in a context whose memory cap has room for their values and little else."""
from __future__ import annotations

import ctypes
import math
import time

import numpy as np
import pytest

from psuedocubes_b200.cubes import count_roots, list_roots
from psuedocubes_b200.focus import Config
from psuedocubes_b200.gpu import DeviceArray, GPUFocus, Runtime
from psuedocubes_b200.served import A_RINGS, B_RINGS

pytestmark = pytest.mark.gpu

SPARE = 4096                                             # beside the values: the window call's own words


def left(runtime: Runtime) -> int:
    words = [ctypes.c_uint64() for _ in range(3)]
    runtime.lib.pc_mem_info(runtime.ctx, *[ctypes.byref(w) for w in words])
    return words[2].value - words[0].value


@pytest.fixture(scope='module')
def tight():
    runtime = Runtime(time.monotonic() + 300, 64 << 20)
    config = Config(601, 10**20, 10**20 + 10**16, math.prod(A_RINGS[:5]), math.prod(B_RINGS[:4]))
    yield runtime, [GPUFocus(runtime, f) for f in config.focuses()]
    runtime.close()


def fill(runtime: Runtime, room: int) -> DeviceArray:
    """Takes all of the cap but ``room`` bytes (a multiple of 256)."""
    taken = DeviceArray.from_host(runtime, np.zeros((left(runtime) - room) // 8, dtype=np.uint64))
    assert left(runtime) == room
    return taken


@pytest.mark.parametrize('n', [100, 5000, 300_000])
def test_window_that_just_fits(tight, n):
    runtime, foci = tight
    for focus in foci:
        low = focus.modulus // 3
        high = low + int(n * focus.modulus / focus.count)
        want = focus.window(low, high, cap=1 << 22).get()
        exact = (8 * len(want) + 255) // 256 * 256
        taken = fill(runtime, exact + SPARE)
        assert np.array_equal(focus.window(low, high, cap=1 << 22).get(), want)
        assert np.array_equal(focus.window(low, high, cap=len(want)).get(), want)
        with pytest.raises(OverflowError):
            focus.window(low, high, cap=len(want) - 1)
        del taken
        assert left(runtime) > exact + SPARE


def test_refusals_without_room(tight):
    """A window that does not fit is a MemoryError; one over its own cap stays an OverflowError that reports the count."""
    runtime, foci = tight
    focus = foci[0]
    low = focus.modulus // 5
    high = low + int(50_000 * focus.modulus / focus.count)
    total = len(focus.window(low, high, cap=1 << 22))
    taken = fill(runtime, SPARE)
    with pytest.raises(MemoryError):
        focus.window(low, high, cap=1 << 22)
    handle, count = ctypes.c_void_p(), ctypes.c_uint64()
    for cap in (total - 1, total // 2, 100):
        code = runtime.lib.pc_focus_window(runtime.ctx, focus.handle, low, high, cap, ctypes.byref(handle), ctypes.byref(count))
        with pytest.raises(OverflowError):
            runtime.call(code)
        assert count.value == total and left(runtime) == SPARE
    del taken
    assert len(focus.window(low, high, cap=total)) == total


@pytest.mark.parametrize('p, n', [(5, 2_000_000), (619, 1_000_003), (2, 5000)])
def test_root_list_that_just_fits(tight, p, n):
    """8 KB beside the roots: the table of primes, the tile states and their rounding to 256 bytes."""
    runtime, _ = tight
    first = 10**9 + 1
    want = list_roots(runtime, first, first + n - 1, p)
    exact = (4 * len(want) + 255) // 256 * 256
    taken = fill(runtime, exact + 2 * SPARE)
    assert np.array_equal(list_roots(runtime, first, first + n - 1, p), want)
    assert count_roots(runtime, first, first + n - 1, p) == len(want)
    with pytest.raises(OverflowError):
        list_roots(runtime, first, first + n - 1, p, cap=len(want) - 1)
    del taken
    taken = fill(runtime, 2 * SPARE)
    with pytest.raises(OverflowError):
        list_roots(runtime, first, first + n - 1, p, cap=100)
    if exact > 2 * SPARE:
        with pytest.raises(MemoryError):
            list_roots(runtime, first, first + n - 1, p)
    del taken


@pytest.mark.parametrize('A, B, budget', [(2 * 5 * 11 * 17 * 23 * 29, 9, 0), (2 * 5 * 11 * 17 * 23 * 29 * 41, 9 * 7 * 13, 0),
                                          (599 * 593 * 2, 9 * 587, 0), (math.prod(A_RINGS[:7]), math.prod(B_RINGS[:6]), 0),
                                          (math.prod(A_RINGS[:7]), math.prod(B_RINGS[:6]), 1 << 20)])
def test_focus_tables_that_just_fit(A, B, budget):
    """A context with room for a focus's tables and 16 KB, far less than the scratch of their making on the device."""
    config = Config(619, 0, 10**9, A, B)
    for focus in config.focuses():
        roomy = Runtime(time.monotonic() + 300, 1 << 30)
        gpu = GPUFocus(roomy, focus, budget)
        span = min(3000 * focus.modulus, 50_000 * focus.modulus // focus.count)
        low = focus.modulus // 3
        want = gpu.window(low, low + span, cap=1 << 22).get()
        tables, shape = gpu.table_bytes, (gpu.wheel_modulus, gpu.wheel_size, gpu.bitset_rings, gpu.count)
        tight = Runtime(time.monotonic() + 300, tables // 256 * 256 + 4 * SPARE)
        other = GPUFocus(tight, focus, budget)
        assert (other.wheel_modulus, other.wheel_size, other.bitset_rings, other.count) == shape
        low_room = left(tight)
        assert 0 <= low_room <= 4 * SPARE
        few = want[:50]
        assert np.array_equal(other.window(low, int(few[-1]) + 1, cap=1 << 22).get(), few)
        del other
        tight.close()
        tight = Runtime(time.monotonic() + 300, max(256, tables // 256 * 256 - 1024))
        if tables > 4096:
            with pytest.raises(MemoryError):
                GPUFocus(tight, focus, budget)
        tight.close()
        del gpu
        roomy.close()
