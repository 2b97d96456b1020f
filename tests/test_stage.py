"""The page-locked stage of a context is lent to one call at a time: a call on a second thread gets none instead of
the memory in which the first one's results lie."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / 'psuedocubes_b200' / 'csrc'

PROGRAM = r'''
#include "stage.cuh"
#include <cstdio>
#include <thread>
#include <vector>

int main() {
    static uint64_t memory[64];
    StageBuffer none, buffer;
    if (StageLoan(none, [] { return (uint64_t *)nullptr; }).get()) return 1;     // cannot be had ...
    if (!StageLoan(none, [] { return memory; }).get()) return 2;                 // ... and is asked for again
    auto make = [] { return memory; };
    {
        StageLoan first(buffer, make);
        if (first.get() != memory) return 3;
        if (StageLoan(buffer, make).get()) return 4;                             // lent
        bool second = true;
        std::thread([&] { second = StageLoan(buffer, make).get() != nullptr; }).join();
        if (second) return 5;
        StageLoan moved(std::move(first));
        if (first.get() || moved.get() != memory || StageLoan(buffer, make).get()) return 6;
        first = std::move(moved);
        if (moved.get() || first.get() != memory || StageLoan(buffer, make).get()) return 7;
    }
    if (!StageLoan(buffer, make).get()) return 8;                                // given back
    std::vector<std::thread> threads;
    std::atomic<int> mixed{0}, got{0};
    for (uint64_t t = 1; t <= 4; ++t)
        threads.emplace_back([&, t] {
            for (int i = 0; i < 20000; ++i) {
                StageLoan loan(buffer, make);
                volatile uint64_t *w = loan.get();
                if (!w) continue;
                ++got;
                for (int k = 0; k < 64; ++k) w[k] = t;
                for (int k = 0; k < 64; ++k) mixed += w[k] != t;
            }
        });
    for (auto &t : threads) t.join();
    return mixed ? 9 : got ? 0 : 10;
}
'''


def test_stage_is_lent_to_one_call_at_a_time(tmp_path):
    compiler = shutil.which('g++')
    if compiler is None:
        pytest.skip('no C++ compiler')
    source, program = tmp_path / 'stage.cpp', tmp_path / 'stage'
    source.write_text(PROGRAM)
    subprocess.run([compiler, '-std=c++17', '-O2', '-pthread', f'-I{CSRC}', '-o', str(program), str(source)], check=True)
    assert subprocess.run([str(program)], timeout=120).returncode == 0


def test_every_use_of_the_stage_holds_a_loan():
    """No source keeps the buffer itself: its words are reached through a loan, or freed with the context."""
    for path in CSRC.glob('*.cu*'):
        if path.name == 'stage.cuh':
            continue
        for line in path.read_text().splitlines():
            code = line.split('//')[0]
            if 'stage.words' in code:
                assert 'cudaFreeHost' in code, (path.name, line)
            if 'pc_stage(' in code:
                assert 'StageLoan' in code or 'loan = ' in code, (path.name, line)
