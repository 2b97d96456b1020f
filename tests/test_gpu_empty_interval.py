"""pc_run_batch on intervals (lo, hi] that hold nothing because lo >= hi: no position, whatever lo is.  A lo of 2^64 B and
more has a bound floor((v A + lo) / B) that does not fit 64 bits."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from psuedocubes_b200 import _native as N
from psuedocubes_b200.focus import A619, B619, Config
from psuedocubes_b200.gpu import MASK, DeviceArray, Filters

pytestmark = pytest.mark.gpu

CONFIGS = [Config(619, 10**27, 3 * 10**27, A619, B619), Config(31, 0, 10**10, 14 * 19, 9 * 13 * 31)]


@pytest.mark.parametrize('config', CONFIGS, ids=lambda c: f'p{c.p}')
@pytest.mark.parametrize('nv', [5, 3000])
def test_no_position_between_lo_and_a_smaller_hi(runtime, config, nv):
    filters = Filters(runtime, config)
    first = config.B // 5
    span = min(config.B - first, 10**9)
    vs = np.unique(np.array([first + (span - 1) * k // (nv - 1) for k in range(nv)], dtype=np.uint64))
    low, high = config.u_interval(first)[0], config.u_interval(first + span - 1)[1]
    us = np.unique(np.array([low + (high - low) * k // 2500 for k in range(2500)], dtype=np.uint64))
    du, dv = (DeviceArray.from_host(runtime, x) for x in (us, vs))
    for lo in (config.hi, config.hi + 1, config.B << 64, (config.B << 64) + config.lo, (config.B << 66) + (config.B >> 1),
               (1 << 127) + 12345):
        if lo >> 128:
            continue
        counts, geometry = np.zeros(filters.ng + 3, dtype=np.uint64), np.zeros(2, dtype=np.uint64)
        out, n_out = np.zeros(2 * 64, dtype=np.uint64), ctypes.c_uint64()
        runtime.call(runtime.lib.pc_run_batch(
            runtime.ctx, filters.handle, None, du.handle, 0, len(us), dv.handle, 0, len(vs), lo & MASK, lo >> 64,
            config.hi & MASK, config.hi >> 64, first, span, 1, first + span, counts, geometry, out, 64,
            ctypes.byref(n_out), ctypes.byref(N.Stats())))
        assert not counts.any() and n_out.value == 0, hex(lo)
        assert geometry[1] == len(vs)
