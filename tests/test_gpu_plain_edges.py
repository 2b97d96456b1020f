"""The plain matcher at the edges of its split (1,024 u entries and 64 staged v rows per CTA, four filters
from residues) against plain integer arithmetic: every position of lists of arbitrary coordinates."""
from __future__ import annotations

import ctypes
import random

import numpy as np
import pytest

from psuedocubes_b200 import _native as N
from psuedocubes_b200.focus import A619, B619, Config
from psuedocubes_b200.gpu import MASK, DeviceArray, Matcher
from psuedocubes_b200.tables import allowed

pytestmark = pytest.mark.gpu

# residual filters: 1, 2, 3, 5, 6 (small moduli, 40-bit x) and 91 (production, 92-bit x)
CONFIGS = [Config(7, 0, 10**9, 14, 9), Config(13, 10**6, 10**9, 14, 9 * 13), Config(19, 10**6, 10**10, 14 * 19, 9 * 13),
           Config(31, 0, 10**10, 14 * 19, 9 * 13 * 31), Config(37, 5, 10**11, 14 * 19, 9 * 13 * 31),
           Config(619, 10**27, 3 * 10**27, A619, B619)]
SIZES = [(1, 1), (31, 65), (1023, 64), (1024, 63), (1025, 129), (2049, 3), (4097, 1), (5, 1500)]


def brute(c: Config, us: list[int], vs: list[int]) -> tuple[list[int], list[int]]:
    order, groups = c.filter_order(), c.filter_groups()
    tables = [set(allowed(q)) for q in order]
    counts, values = [0] * (len(groups) + 3), []
    for v in vs:
        for u in us:
            x = u * c.B - v * c.A
            if not c.lo < x <= c.hi:
                continue
            counts[0] += 1
            for i, (q, table) in enumerate(zip(order, tables)):
                if x % q not in table:
                    break
                if i % 4 == 3 or i + 1 == len(order):
                    counts[i // 4 + 1] += 1
            else:
                values.append(x)
    counts[len(groups) + 1] = len(values)
    return counts, sorted(values)


@pytest.mark.parametrize('config', CONFIGS, ids=lambda c: f'p{c.p}')
@pytest.mark.parametrize('size', SIZES, ids=lambda s: f'{s[0]}x{s[1]}')
def test_plain_split_edges(runtime, config, size):
    nu, nv = size
    rng = random.Random(nu * 7919 + nv * 31 + config.p)
    # v rows near one another (unsorted), u entries over the union of their intervals and a little beyond
    v0 = rng.randrange(0, max(1, config.B - 4 * nv))
    vs = [v0 + rng.randrange(0, 4 * nv) for _ in range(nv)]
    lo, hi = config.u_interval(min(vs))[0], config.u_interval(max(vs))[1]
    us = sorted(max(0, rng.randrange(lo - 3, hi + 3)) for _ in range(nu))
    m = Matcher(runtime, config)
    ng, cap = len(m.filter_groups), nu * nv
    counts, out = np.zeros(ng + 3, dtype=np.uint64), np.zeros(2 * cap, dtype=np.uint64)
    du, dv = (DeviceArray.from_host(runtime, np.array(x, dtype=np.uint64)) for x in (us, vs))
    runtime.call(runtime.lib.pc_run_plain(runtime.ctx, m.filters.handle, du.handle, 0, nu, dv.handle, 0, nv,
                                          config.lo & MASK, config.lo >> 64, config.hi & MASK, config.hi >> 64,
                                          counts, out, cap, ctypes.byref(N.Stats())))
    want, values = brute(config, us, vs)
    assert [int(n) for n in counts] == want
    assert sorted(int(a) | int(b) << 64 for a, b in out[:2 * len(values)].reshape(-1, 2)) == values


@pytest.mark.parametrize('config', CONFIGS, ids=lambda c: f'p{c.p}')
@pytest.mark.parametrize('size', [(127, 64), (128, 65), (129, 63), (257, 511), (1, 512), (130, 513), (40, 2100)],
                         ids=lambda s: f'{s[0]}x{s[1]}')
def test_plain_rows_edges(runtime, config, size):
    """The kernel for 64 and more v rows: chunks of 128 u entries, 32 v rows per warp, eight at a time."""
    test_plain_split_edges(runtime, config, size)


@pytest.mark.parametrize('nv', [63, 64, 200])
@pytest.mark.parametrize('primes', [(1021, 1019, 7, 2, 5), (1021, 1019, 7, 5, 3), (4093, 8191, 13), (1999, 47), (2039,)],
                         ids=lambda q: '-'.join(map(str, q)))
def test_plain_many_rows(runtime, primes, nv):
    """First filters whose residues are 2,048 and fewer rows, or more (the lookup kernel for every v list), with
    arbitrary residue tables, through the entry point that takes them."""
    rng = random.Random(sum(primes) + nv)
    A, B, nu = 11 * 17, 19 * 23, 300
    tables = [[int(rng.random() < 0.6) for _ in range(q)] for q in primes]
    vs = sorted(rng.randrange(10**9, 10**9 + 4 * nv) for _ in range(nv))
    us = sorted(rng.randrange(vs[0] * A // B, vs[-1] * A // B + 900) for _ in range(nu))
    lo, hi, ng, cap = 1000, 300_000, (len(primes) + 3) // 4, nu * nv
    counts, out, err = np.zeros(ng + 3, dtype=np.uint64), np.zeros(2 * cap, dtype=np.uint64), ctypes.create_string_buffer(256)
    code = runtime.lib.pc_run_plain_static(0, N.u64(us), nu, N.u64(vs), nv, A, B, lo, 0, hi, 0,
                                           np.array(primes, dtype=np.uint32), len(primes),
                                           np.array([b for t in tables for b in t], dtype=np.uint8), counts, out, cap, err, 256)
    assert code == 0, err.value
    want, values = [0] * (ng + 3), []
    for x in (u * B - v * A for v in vs for u in us):
        if lo < x <= hi:
            want[0] += 1
            for i, (q, table) in enumerate(zip(primes, tables)):
                if not table[x % q]:
                    break
                if i % 4 == 3 or i + 1 == len(primes):
                    want[i // 4 + 1] += 1
            else:
                values.append(x)
    want[ng + 1] = len(values)
    assert values and [int(n) for n in counts] == want
    assert sorted(out[:2 * len(values):2].tolist()) == sorted(values)
