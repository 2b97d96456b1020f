"""The division of the fused matcher's work among CTAs, run on the CPU: every row of every block is taken once, and no CTA
works much longer than its fair part, whatever the blocks' sizes."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / 'psuedocubes_b200' / 'csrc'

PROGRAM = r'''
#include "shares.cuh"
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

constexpr uint32_t GRID = 148, COST = 5596;

// Longest CTA over the fair part of all work, in rows; a share that starts inside a block builds the block again.
// Negative: a row was not taken, or taken twice.
double longest(const std::vector<uint64_t> &rows, Shares &d) {
    std::vector<uint64_t> prefix;
    uint64_t work = 0, largest = 0;
    for (uint64_t r : rows) {
        prefix.push_back(work);
        work += r ? r + COST : 0;
        largest = std::max(largest, r ? r + COST : 0);
    }
    d = divide_work(work, largest, rows.size(), GRID, COST);
    std::vector<uint64_t> taken(rows.size(), 0), next(rows.size(), 0), busy(GRID, 0);
    for (uint64_t share = 0; share < d.n; ++share) {
        uint64_t b, b_end, at = 0, at_end = 0, spent = 0;
        if (d.pairs) {
            b = share < d.pairs ? 2 * share : d.pairs + share;
            b_end = b + (share < d.pairs ? 2 : 1);
        } else {
            at = work * share / d.n, at_end = work * (share + 1) / d.n;
            b_end = b = std::upper_bound(prefix.begin(), prefix.end(), at) - prefix.begin() - 1;
            if (at != at_end) b_end = std::upper_bound(prefix.begin(), prefix.end(), at_end - 1) - prefix.begin();
        }
        if (b_end > rows.size()) return -1;
        for (uint64_t k = b; k < b_end; ++k) {
            uint32_t row = 0, end = (uint32_t)rows[k];
            if (!d.pairs) cut_rows(prefix[k] + COST, k == b ? at : 0, at_end, row, end);
            if (row >= end) continue;
            if (next[k] != row) return -2;               // shares take a block's rows in order, without gaps
            next[k] = end;
            taken[k] += end - row;
            spent += end - row + COST;
        }
        *std::min_element(busy.begin(), busy.end()) += spent;     // the CTA that is free first claims it
    }
    for (size_t k = 0; k < rows.size(); ++k)
        if (taken[k] != rows[k]) return -3;
    return *std::max_element(busy.begin(), busy.end()) / (work / (double)GRID);
}

int main() {
    std::mt19937_64 rng(5);
    auto check = [](const char *name, const std::vector<uint64_t> &rows, bool whole, double most) {
        Shares d{};
        const double l = longest(rows, d);
        printf("%s: %u shares, %u pairs, longest CTA %.3f of the fair part\n", name, d.n, d.pairs, l);
        return l > 0 && l <= most && (d.pairs != 0) == whole;
    };
    bool ok = true;
    std::vector<uint64_t> lease(10240, 1);
    for (size_t k = 0; k < lease.size(); ++k) lease[k] = std::min<uint64_t>({k * 27, (lease.size() - k) * 27, 28000});
    ok &= check("lease", lease, true, 1.05);
    std::vector<uint64_t> one(3000, 400);
    one[2999] = 1000000;
    ok &= check("one block of 1e6 rows, last", one, false, 1.15);
    std::rotate(one.begin(), one.end() - 1, one.end());
    ok &= check("one block of 1e6 rows, first", one, false, 1.15);
    one[0] = 9669254;
    ok &= check("one block of 9.7e6 rows", one, false, 1.15);
    std::vector<uint64_t> wide(3000, 0);
    for (auto &r : wide) r = rng() % 300000;
    ok &= check("up to 3e5 rows", wide, true, 1.15);
    std::vector<uint64_t> spread(5000, 0);
    for (auto &r : spread) r = (uint64_t)1 << rng() % 21;
    ok &= check("powers of two", spread, false, 1.25);
    std::vector<uint64_t> batch(57, 1000);
    ok &= check("batch", batch, false, 2.7);             // half the CTAs build a block that another one builds too
    ok &= check("one block", {5000000}, false, 1.3);
    for (int k = 0; k < 200; ++k) {                      // coverage: any sizes, empty blocks among them
        std::vector<uint64_t> any(1 + rng() % 6000);
        for (auto &r : any) r = rng() % 3 ? rng() % (1 + (rng() & ((uint64_t)1 << rng() % 22) - 1)) : 0;
        any[0] += 1;
        Shares d{};
        const double l = longest(any, d);
        if (l <= 0) printf("any %d: %f\n", k, l), ok = false;
    }
    return ok ? 0 : 1;
}
'''


def test_no_cta_waits_for_a_large_block(tmp_path):
    compiler = shutil.which('g++')
    if compiler is None:
        pytest.skip('no C++ compiler')
    source, program = tmp_path / 'shares.cpp', tmp_path / 'shares'
    source.write_text(PROGRAM)
    subprocess.run([compiler, '-std=c++17', '-O2', f'-I{CSRC}', '-o', str(program), str(source)], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout
