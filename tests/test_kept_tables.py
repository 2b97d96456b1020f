"""Tables kept between calls are bounded: checking against a large prime bound leaves no table per prime behind."""
from __future__ import annotations

import numpy as np

from psuedocubes_b200 import tables, verify
from psuedocubes_b200.predicate import primes_upto


def test_kept_tables_are_bounded():
    primes = [q for q in primes_upto(14_000) if q % 3 == 1]
    value = np.array([1], dtype=np.uint64), np.array([0], dtype=np.uint64)
    verify.verify_many(*value, primes[-1])
    for q in primes_upto(14_000):
        tables.ring_bytes(q)
        tables.sieve_primes(q)
    for kept, most in ((verify._fails, 1100), (tables.ring_bytes, 1100), (tables._primes, 32)):
        info = kept.cache_info()
        assert info.maxsize == most and info.currsize <= most
    assert len(primes_upto(14_000)) > 1600
