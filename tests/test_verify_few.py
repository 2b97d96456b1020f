"""A few values are checked one by one, more of them in arrays, with the same rows: whichever is less work for the prime
bound.  Four values below p = 31 took 114 us in arrays, 51 one by one."""
from __future__ import annotations

import pytest

from psuedocubes_b200 import batch_experiment
from psuedocubes_b200.focus import Config
from psuedocubes_b200.predicate import is_perfect_cube, local3
from psuedocubes_b200.verify import verify

CONFIG = Config(31, 0, 10**9, 14 * 19, 9 * 13 * 31)


@pytest.fixture(scope='module')
def survivors():
    return [n for n in range(10**6 + 1, 10**6 + 200_000, 2) if n % 9 in (1, 8) and local3(n, 31)]


@pytest.mark.parametrize('n, arrays', [(0, False), (1, False), (4, False), (46, False), (47, True), (120, True)])
def test_few_values_one_by_one(monkeypatch, survivors, n, arrays):
    """31 has 11 primes below it: 46 values are 506 tests, 47 are 517."""
    calls = []
    whole = batch_experiment.local_and_cubes
    monkeypatch.setattr(batch_experiment, 'local_and_cubes', lambda *a: calls.append(a) or whole(*a))
    values = survivors[:n]
    assert len(values) == n
    assert batch_experiment.verify_values(CONFIG, values) == [verify(x, 31) for x in values if not is_perfect_cube(x)]
    assert bool(calls) == arrays


@pytest.mark.parametrize('n', [2, 100])
def test_a_wrong_value_is_refused(survivors, n):
    for wrong in (survivors[0] + 1, 7**3 * 19, 10**9 + 1):
        with pytest.raises(ArithmeticError):
            batch_experiment.verify_values(CONFIG, survivors[:n - 1] + [wrong])
