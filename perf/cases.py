"""Timed cases of the sieve, through the entry points that a program calls.

A case is a dict of plain values whose ``kind`` names the entry point:

tile      ``Matcher.tile``: one plain tile of the per-tile loop (``compute_batch`` calls it tile by tile)
batch     ``prepare`` and ``MaskedMatcher.run`` / ``FusedMatcher.run``: one compute batch of up to 64 subtiles
lease     ``compute_lease``: one lease with its receipt
leases    ``compute_leases``: a worker that commits lease after lease
windows   uneven windows of mixed prime bounds, either planned afresh (``BatchedEngine.plan``, ``run``,
          ``results``) or a planned set replayed from its CUDA graph
served    ``ServedLoop.run``: range-certification requests released together to a resident loop
tables    ``GPUFocus`` twice and the residual filters (what a request with a new focus split needs before
          its first window), with one window of each focus read back
roots     ``count_roots`` / ``list_roots``: the genuine-cube control

A program opens one runtime and keeps its focus tables and matchers, so those are shared by the
cases of a process; everything drawn from the seed (where a range starts, the windows, the requests) is
the case's own.
"""
from __future__ import annotations

import math
import random
import time
from typing import Any

import numpy as np

from psuedocubes_b200.batch_experiment import FusedMatcher, MaskedMatcher, prepare as prepare_batch
from psuedocubes_b200.batched import DEFAULT_SETTINGS, BatchedEngine, WORKLOAD_PRIMES, seeded_windows
from psuedocubes_b200.cubes import count_roots, list_roots
from psuedocubes_b200.focus import A619, B619, Config, Tile
from psuedocubes_b200.gpu import Filters, GPUFocus, Matcher, Runtime
from psuedocubes_b200.optimized import BATCH_WIDTH, compute_lease, compute_leases
from psuedocubes_b200.served import A_RINGS, B_RINGS, SERVED_PRIMES, X_MAX, Request, ServedLoop, plan_request
from psuedocubes_b200.tables import allowed

LO, HI = 10**27, 3 * 10**27              # the production interval
ROOT_FIRST, ROOT_LAST = 1_000_000_001, 1_442_249_570   # its cube roots
M64 = (1 << 64) - 1


def listed() -> list[dict[str, Any]]:
    return [
        # the smallest call: a plain tile of 10^6 canonical v, as an overflow split or a short tail leaves
        dict(name='tile_1e6', kind='tile', p=547, width=1_000_003),
        # the production tile of the plain loop
        dict(name='tile_1e8', kind='tile', p=619, width=100_000_000),
        # the production compute batch: 64 subtiles of 10^8 v
        dict(name='batch_64x1e8', kind='batch', p=619, tiles=64, width=100_000_000, tail=0, engine='masked'),
        # a batch at another prime bound with fewer, odd subtiles and a short last one
        dict(name='batch_ragged', kind='batch', p=541, tiles=37, width=61_803_399, tail=23_456_789, engine='masked'),
        # a short lease that ends inside a batch (the end of an assigned range)
        dict(name='lease_24', kind='lease', p=619, batches=24, tail=1_234_567_891),
        # the headline workload: a worker running full production leases back to back
        dict(name='leases_3x256', kind='leases', p=619, count=3, batches=256),
        # the batched workload: 512 uneven windows, planned once and replayed
        dict(name='windows_512_replay', kind='windows', count=512, span_lo=6.0, span_hi=10.0, replay=True),
        # a smaller set of new windows, from plan to verified results
        dict(name='windows_48_fresh', kind='windows', count=48, span_lo=6.0, span_hi=10.0, replay=False),
        # range certification: requests of the workload's narrower spans, released together
        dict(name='served_12', kind='served', requests=12, span_lo=15.0, span_hi=17.0),
        # focus tables and filters of a served request's split (prefix lengths of the ring lists)
        dict(name='tables_7_6', kind='tables', p=601, a=7, b=6),
        # the genuine-cube control over all but a tenth of the production interval
        dict(name='roots_4e8', kind='roots', p=619, n=400_000_007, list=False),
        # the control's list of roots over a short interval
        dict(name='roots_list', kind='roots', p=619, n=1_000_003, list=True),
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict[str, Any]:
    kind = rng.choice(['tile', 'batch', 'batch', 'lease', 'lease', 'leases', 'windows', 'windows', 'served', 'tables',
                       'roots'])
    p = rng.choice(WORKLOAD_PRIMES)
    if kind == 'tile':
        return dict(kind=kind, p=p, width=_log(rng, 1e6, 2e8))
    if kind == 'batch':
        width = _log(rng, 1e6, 1e8)
        return dict(kind=kind, p=p, tiles=_log(rng, 1, 64), width=width, tail=rng.choice([0, rng.randrange(1, width)]),
                    engine=rng.choice(['masked', 'masked', 'masked', 'fused']))
    if kind == 'lease':
        return dict(kind=kind, p=p, batches=_log(rng, 1, 256), tail=rng.choice([0, rng.randrange(1, BATCH_WIDTH)]))
    if kind == 'leases':
        return dict(kind=kind, p=p, count=rng.choice([2, 3]), batches=_log(rng, 24, 256))
    if kind == 'windows':
        lo = rng.uniform(6.0, 8.0)
        return dict(kind=kind, count=_log(rng, 16, 512), span_lo=round(lo, 2), span_hi=round(rng.uniform(lo + 1, 10.0), 2),
                    replay=rng.random() < 0.5)
    if kind == 'served':
        lo = rng.uniform(15.0, 16.0)
        return dict(kind=kind, requests=_log(rng, 1, 16), span_lo=round(lo, 2), span_hi=round(rng.uniform(lo + 0.5, 17.5), 2))
    if kind == 'tables':
        return dict(kind=kind, p=rng.choice(SERVED_PRIMES), a=rng.randint(4, 10), b=rng.randint(4, 9))
    if rng.random() < 0.5:
        return dict(kind=kind, p=p, n=_log(rng, 1e5, 4e8), list=False)
    return dict(kind=kind, p=p, n=_log(rng, 1e4, 2e7), list=True)


# ------------------------------------------------------------------------------------------
# what a program keeps

class _Program:
    """One runtime with its production focus tables, matchers and window engine."""

    def __init__(self) -> None:
        self.runtime = Runtime(time.monotonic() + 24 * 3600, 16 * 1024**3)
        self.engine = BatchedEngine(self.runtime)
        self.kept: dict[tuple[str, int], Any] = {}

    def config(self, p: int) -> Config:
        return Config(p, LO, HI, A619, B619)

    def focuses(self, p: int) -> tuple[GPUFocus, GPUFocus]:
        return self.engine.focus_pair(self.config(p))

    def matcher(self, kind: Any, p: int) -> Any:
        key = (kind.__name__, p)
        if key not in self.kept:
            self.kept[key] = kind(self.runtime, self.config(p))
        return self.kept[key]


_program: _Program | None = None


def _the_program() -> _Program:
    global _program
    if _program is None:
        _program = _Program()
    return _program


def prepare(case: dict[str, Any], seed: int) -> dict[str, Any]:
    rng = random.Random(seed)
    prog = _the_program()
    kind = case['kind']
    state: dict[str, Any] = dict(case=case, program=prog)
    if kind == 'tile':
        first = rng.randrange(0, B619 - case['width'])
        state.update(matcher=prog.matcher(Matcher, case['p']), foci=prog.focuses(case['p']),
                     tile=Tile(first, first + case['width']))
    elif kind == 'batch':
        span = case['tiles'] * case['width'] - (case['width'] - case['tail'] if case['tail'] else 0)
        first = rng.randrange(0, (B619 - span) // case['width']) * case['width']
        engine = MaskedMatcher if case['engine'] == 'masked' else FusedMatcher
        state.update(matcher=prog.matcher(engine, case['p']), foci=prog.focuses(case['p']), first=first, end=first + span)
    elif kind in ('lease', 'leases'):
        count, width = case.get('count', 1), case['batches'] * BATCH_WIDTH
        first = rng.randrange(0, (B619 - count * width) // BATCH_WIDTH) * BATCH_WIDTH
        ranges = [(first + k * width, first + (k + 1) * width) for k in range(count)]
        if case.get('tail'):
            ranges[-1] = (ranges[-1][0], ranges[-1][1] - BATCH_WIDTH + case['tail'])
        state.update(matcher=prog.matcher(MaskedMatcher, case['p']), foci=prog.focuses(case['p']), ranges=ranges)
    elif kind == 'windows':
        windows = seeded_windows(case['count'], seed, (case['span_lo'], case['span_hi']))
        for p in WORKLOAD_PRIMES:
            prog.engine.family(prog.config(p))
        prog.focuses(WORKLOAD_PRIMES[0])
        state['windows'] = windows
        if case['replay']:
            state['plan'] = _plan(prog, windows)
            state['plan'].run(graph=True)
    elif kind == 'served':
        requests = []
        for k in range(case['requests']):
            lo = int(10 ** rng.uniform(20, math.log10(X_MAX)))
            hi = min(lo + int(10 ** rng.uniform(case['span_lo'], case['span_hi'])), X_MAX)
            requests.append(Request(k, rng.choice(SERVED_PRIMES), lo, hi))
        loop = prog.kept.get(('ServedLoop', 0))
        if loop is None:                     # a service keeps one loop and its resident tables
            loop = prog.kept[('ServedLoop', 0)] = ServedLoop(prog.runtime)
        state.update(loop=loop, requests=requests)
    elif kind == 'tables':
        A, B = math.prod(A_RINGS[:case['a']]), math.prod(B_RINGS[:case['b']])
        config = Config(case['p'], 10**20, 10**20 + 10**16, A, B)
        state.update(config=config, foci=config.focuses(),
                     lows=[rng.randrange(0, f.modulus) for f in config.focuses()])
    elif kind == 'roots':
        room = ROOT_LAST - ROOT_FIRST + 1 - case['n']
        first = ROOT_FIRST + rng.randrange(0, room + 1)
        state.update(first=first, last=first + case['n'] - 1)
    else:
        raise ValueError(f'unknown kind {kind}')
    return state


def _plan(prog: _Program, windows: list[Any]) -> Any:
    tuning = {k: v for k, v in DEFAULT_SETTINGS.items() if k != 'width'}
    return prog.engine.plan(windows, DEFAULT_SETTINGS['width'], tuning)


# ------------------------------------------------------------------------------------------
# one pass

def run(state: dict[str, Any]) -> Any:
    case, prog = state['case'], state['program']
    kind = case['kind']
    if kind == 'tile':
        af, bf = state['foci']
        return _result(state['matcher'].tile(state['tile'], af, bf))
    if kind == 'batch':
        m, (af, bf) = state['matcher'], state['foci']
        return _result(m.run(prepare_batch(m.runtime, m.config, af, bf, state['first'], state['end'], case['width'])))
    if kind == 'lease':
        af, bf = state['foci']
        return _result(compute_lease(state['matcher'], af, bf, *state['ranges'][0]))
    if kind == 'leases':
        af, bf = state['foci']
        return [_result(r) for r in compute_leases(state['matcher'], af, bf, state['ranges'])]
    if kind == 'windows':
        if case['replay']:
            state['plan'].run(graph=True)
            counts, geometry, records = state['plan'].raw()
            return [_padded(a.view(np.int64)) for a in (counts, geometry, records[np.lexsort(records.T)])]
        batch = _plan(prog, state['windows'])
        batch.run()
        rows = batch.results()
        batch.close()
        return _rows(rows)
    if kind == 'served':
        done = state['loop'].run(state['requests'], realtime=False)['results']
        return _rows([done[k] for k in sorted(done)])
    if kind == 'tables':
        rt = prog.runtime
        foci = [GPUFocus(rt, f) for f in state['foci']]
        filters = Filters(rt, state['config'])
        values = [_padded(f.window(low, low + _window_span(f.focus)).get().view(np.int64)) for f, low in zip(foci, state['lows'])]
        return [*values, *[f.count for f in foci], filters.ng]
    if case['list']:
        return _padded(list_roots(prog.runtime, state['first'], state['last'], case['p']).view(np.int32))
    return count_roots(prog.runtime, state['first'], state['last'], case['p'])


def _window_span(focus: Any) -> int:
    """A v or u span of about 4,096 focus values, at most a million coordinates."""
    return max(1, min(1_000_000, 4096 * focus.modulus // focus.count))


def _limbs(values: list[Any]) -> np.ndarray:
    out = np.array([v for x in map(int, values) for v in (x & M64, x >> 64)], dtype=np.uint64)
    return _padded(out.view(np.int64).reshape(-1, 2))


def _padded(rows: np.ndarray) -> np.ndarray:
    """The rows with their number, then zeros up to a size that does not change from seed to seed: outputs
    of one case have one shape."""
    n = len(rows)
    size = max(4096, 1 << int(1.3 * n).bit_length())
    out = np.zeros((size + 1, *rows.shape[1:]), dtype=rows.dtype)
    out[0], out[1:n + 1] = n, rows
    return out


def _result(row: dict[str, Any]) -> dict[str, Any]:
    """The numbers of a result or receipt: sums, group populations, subtile scopes, values, digests."""
    out = dict(sums=np.array([row[k] for k in ('focus_u', 'focus_v', 'cartesian_opportunities',
                                               'valid_focused_candidates', 'genuine_cubes', 'local_survivors')]),
               groups=np.array(row['group_survivors']), values=_limbs(row['all_values']))
    scopes = row.get('subtile_scopes')
    if scopes and 'transcript_sha256' in scopes[0]:
        out['transcript'] = np.frombuffer(bytes.fromhex(scopes[0]['transcript_sha256']), dtype=np.uint8)
    elif scopes:
        out['scopes'] = np.array([[s['valid_focused_candidates'], s['local_survivors'], *s['group_survivors']]
                                  for s in scopes])
    return out


def _rows(rows: list[dict[str, Any]]) -> dict[str, Any]:
    """The same for the rows of several windows or requests, whose filter lists differ in length."""
    return dict(sums=np.array([[r[k] for k in ('valid_focused_candidates', 'genuine_cubes', 'local_survivors')]
                               for r in rows]),
                groups=_padded(np.array([n for r in rows for n in r['group_survivors']])),
                values=_limbs([x for r in rows for x in (r['all_values'] if 'all_values' in r else r['values'])]))


# ------------------------------------------------------------------------------------------
# what a pass cannot do without

def _density(rings: tuple[int, ...]) -> float:
    return math.prod(len(allowed(q)) / q for q in rings)


DENSITY_A, DENSITY_B = _density(A_RINGS), _density(B_RINGS)


def _sieve(span: float, spans: int = 1, subtiles: float = 0.0, outputs: float = 0.0) -> dict[str, float]:
    """A v range of ``span``: its focus values once, its counters and outputs; 0.53 lane operations
    per focused position for the bitset intersection and the survivors."""
    values = span * DENSITY_B + (spans * (HI - LO) / B619 + span * A619 / B619) * DENSITY_A
    positions = span * DENSITY_B * (HI - LO) / B619 * DENSITY_A
    return dict(bytes=8 * values + 8 * 27 * subtiles + 16 * outputs, flops=0.53 * positions)


def work(case: dict[str, Any]) -> dict[str, float]:
    kind = case['kind']
    if kind == 'tile':
        return _sieve(case['width'], 1, 1)
    if kind == 'batch':
        return _sieve(case['tiles'] * case['width'], 1, case['tiles'])
    if kind in ('lease', 'leases'):
        n = case.get('count', 1)
        return _sieve(n * case['batches'] * BATCH_WIDTH, n, n * case['batches'] * 64)
    if kind == 'windows':
        a, b = case['span_lo'], case['span_hi']
        span = case['count'] * (10**b - 10**a) / ((b - a) * math.log(10))
        return _sieve(span, case['count'], case['count'] + span / DEFAULT_SETTINGS['width'])
    if kind == 'served':
        total = dict(bytes=0.0, flops=0.0)
        a, b = case['span_lo'], case['span_hi']
        for k in range(case['requests']):       # requests at even steps of the span's exponent
            span = 10 ** (a + (b - a) * (k + 0.5) / case['requests'])
            plan = plan_request(619, 10**26, 10**26 + int(span))
            positions = span * plan.density_a * plan.density_b
            total['bytes'] += 8 * (plan.count_a + plan.count_b)
            total['flops'] += 0.53 * positions
        return total
    if kind == 'tables':
        entries = sum(min(math.prod(len(allowed(q)) for q in rings), 32_000_000)
                      for rings in (A_RINGS[:case['a']], B_RINGS[:case['b']]))
        return dict(bytes=8.0 * entries + 8 * 8192, flops=0.0)
    n = case['n']
    groups = 40
    return dict(bytes=(4.0 * 0.0867 * n if case['list'] else 8.0) + 8 * groups, flops=3 * groups * n / 32)


# ------------------------------------------------------------------------------------------
# the same in plain numpy, where that takes seconds

def exact(case: dict[str, Any], seed: int) -> Any:
    kind = case['kind']
    rng = random.Random(seed)
    if kind == 'roots':
        first = ROOT_FIRST + rng.randrange(0, ROOT_LAST - ROOT_FIRST + 1 - case['n'] + 1)
        primes = [q for q in range(2, case['p'] + 1) if all(q % d for d in range(2, math.isqrt(q) + 1))]
        found, count, step = [], 0, 1 << 24
        for at in range(first, first + case['n'], step):
            stop = min(at + step, first + case['n'])
            keep = np.ones(stop - at, dtype=bool)
            for q in primes:
                keep[-at % q::q] = False
            if case['list']:
                found.append(np.flatnonzero(keep).astype(np.int64) + at)
            else:
                count += int(np.count_nonzero(keep))
        return _padded(np.concatenate(found).astype(np.int32)) if case['list'] else count
    if kind == 'tables':
        A, B = math.prod(A_RINGS[:case['a']]), math.prod(B_RINGS[:case['b']])
        lists = []
        for rings, coefficient in ((A_RINGS[:case['a']], B), (B_RINGS[:case['b']], -A)):
            M = math.prod(rings)
            low, count = rng.randrange(0, M), math.prod(len(allowed(q)) for q in rings)
            y = np.arange(max(1, min(1_000_000, 4096 * M // count)), dtype=np.int64) + low
            keep = np.ones(len(y), dtype=bool)
            for q in rings:
                table = np.zeros(q, dtype=bool)
                table[list(allowed(q))] = True
                keep &= table[(y % q) * (coefficient % q) % q]
            lists.append((y[keep], count))
        residuals = [q for q in (9, *(q for q in range(2, case['p'] + 1) if q != 3 and all(q % d for d in range(2, math.isqrt(q) + 1))))
                     if A % q and B % q]
        return [*[_padded(v) for v, _ in lists], *[n for _, n in lists], (len(residuals) + 3) // 4]
    return None
