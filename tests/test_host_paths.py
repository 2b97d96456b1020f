"""Host paths that work on many values at once against the definitions they replace."""
from __future__ import annotations

import random

import numpy as np

from psuedocubes_b200.accounting import digest, digest_decimals
from psuedocubes_b200.batch_experiment import outputs_by_tile, split_outputs, tile_ranges
from psuedocubes_b200.focus import A619, B619, Config
from psuedocubes_b200.predicate import is_perfect_cube, local3
from psuedocubes_b200.served import A_RINGS, B_RINGS, _A_PREFIXES, _B_PREFIXES, _count
from psuedocubes_b200.tables import allowed, ring_bytes, sieve_primes
from psuedocubes_b200.verify import _fails, local_and_cubes, local_test


def test_tile_ranges_are_the_u_intervals():
    rng = random.Random(7)
    configs = [Config(619, 10**27, 3 * 10**27, A619, B619), Config(31, 0, 100000, 14 * 19, 9 * 13 * 31),
               Config(619, 5, 10**20, A619 // 13, B619 * 13), Config(7, 0, 1000, 14, 9)]
    for c in configs:
        for _ in range(200):
            span = rng.randrange(1, min(c.B, 10**11) + 1)
            width = rng.choice([-(-span // 64), span, span + 5, rng.randrange(-(-span // 64), span + 1)])
            first = rng.randrange(0, c.B - span + 1)
            rows = tile_ranges(c, first, first + span, width)
            want = [(v, min(v + width, first + span)) for v in range(first, first + span, width)]
            assert rows == [(v, e, c.u_interval(v)[0], c.u_interval(e - 1)[1]) for v, e in want]


def test_local_test_is_local3():
    rng = random.Random(11)
    for p in (7, 13, 31, 619):
        values = [rng.randrange(1, 1 << rng.choice((5, 20, 64, 90, 96))) for _ in range(400)]
        values += [rng.randrange(1, 1 << 32) ** 3 for _ in range(200)] + [0, 1, 8, (1 << 64) - 1, 1 << 64, (1 << 96) - 1]
        ok, cubes = local_and_cubes(values, p)
        assert ok.tolist() == [local3(n, p) for n in values]
        assert cubes.tolist() == [is_perfect_cube(n) for n in values]
    assert local_test(np.zeros(0, dtype=np.uint64), np.zeros(0, dtype=np.uint64), 619).size == 0


def test_small_tables():
    for q in sieve_primes(700)[2:]:
        assert [i for i, x in enumerate(ring_bytes(q)) if x] == list(allowed(q))
        assert _fails(q).tolist() == [r == 0 or (q % 3 == 1 and pow(r, (q - 1) // 3, q) != 1) for r in range(q)]
    assert sieve_primes(1) == [] and sieve_primes(2) == [2]
    sieve_primes(50).append(0)                              # the caller's own list
    assert sieve_primes(50)[-1] == 47
    for rings, prefixes in ((A_RINGS, _A_PREFIXES), (B_RINGS, _B_PREFIXES)):
        for k, product, count, top in prefixes:
            assert product == np.prod([int(q) for q in rings[:k]], dtype=object) and top == max(rings[:k])
            assert count == np.prod([_count(q) for q in rings[:k]], dtype=object)


def test_digests_and_outputs():
    for values in ([], ['1'], ['12', '345', '6' * 30]):
        assert digest_decimals(values) == digest(values)
    records = np.array([[5, 3 << 32 | 1], [2, 3 << 32 | 1], [9, 0]], dtype=np.uint64)
    assert outputs_by_tile(records) == {3: [2 | 1 << 64, 5 | 1 << 64], 0: [9]}
    assert split_outputs(records, 5) == [[9], [], [], [2 | 1 << 64, 5 | 1 << 64], []]
