"""What the host knows of the flow table between submits (csrc/flow_bounds.h) against a model of the device: batches begin,
run and are waited for in any order; whenever nothing is in flight no entry may expire below the floor and no more may be
alive than the host says, and a sweep that would find something is asked for.  Host code only."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bnk_b200", "csrc")
PROGRAM = r"""
#include "flow_bounds.h"
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <vector>
constexpr long long S = 1000000000ll;
struct Batch { FlowWork w{}; bool began = false, ran = false, note = false, sweep = false, reported = false; long long now = 0; uint32_t n = 0; FlowReport r{}; };
int main(int, char **argv) {
    std::mt19937 rng(atoi(argv[1]));
    const int batches = atoi(argv[2]);
    auto below = [&](uint32_t n) { return (uint32_t)(rng() % n); };
    FlowBounds bounds(LLONG_MAX, 0);
    std::map<uint32_t, long long> table; // key -> expiry
    long long floor = LLONG_MAX, clock = 100 * S;
    std::vector<Batch> b(batches);
    int narrowed = 0, spared = 0;
    for (int step = 0; step < 8000; step++) {
        Batch &x = b[below(batches)];
        if (!x.began) {
            clock += below(3 * S);
            x.note = below(4) != 0;
            x.n = below(900);
            x.now = clock;
            x.began = true;
            x.ran = x.reported = x.sweep = false;
            const bool alone = [&] { for (Batch &y : b) if (&y != &x && y.began) return false; return true; }();
            if (x.note) {
                x.sweep = bounds.note_begins(x.w, x.n, x.now);
                bool expired = false;
                for (auto &e : table) expired |= x.now > e.second;
                if (alone && expired && table.size() + x.n > FlowBounds::kSweepThreshold && !x.sweep) return printf("no sweep, step %d\n", step), 1;
                spared += !x.sweep;
            } else {
                bounds.check_begins(x.w, x.now);
            }
        } else if (!x.ran) {
            for (uint32_t i = 0; i < x.n; i++) {
                const uint32_t key = below(20000);
                const long long exp = x.now + (key & 1 ? 120 : 30) * S;
                if (!x.note && !table.count(key)) continue;
                table[key] = exp;
                floor = std::min(floor, exp);
            }
            if (x.sweep && table.size() > FlowBounds::kSweepThreshold) {
                floor = LLONG_MAX;
                for (auto it = table.begin(); it != table.end();) {
                    if (x.now > it->second) it = table.erase(it);
                    else floor = std::min(floor, it++->second);
                }
            }
            if (x.note) {
                x.reported = true;
                x.r.live = table.size();
                x.r.floor = floor;
            }
            x.ran = true;
        } else {
            const uint64_t before = bounds.live_most();
            bounds.over(x.w, x.reported ? &x.r : nullptr);
            x.began = false;
            narrowed += bounds.live_most() < before;
            bool quiet = true;
            for (Batch &y : b) quiet &= !y.began;
            if (!quiet) continue;
            if (bounds.live_most() < table.size()) return printf("alive: %zu, said %llu, step %d\n", table.size(), (unsigned long long)bounds.live_most(), step), 1;
            for (auto &e : table)
                if (e.second < bounds.floor()) return printf("expiry below the floor, step %d\n", step), 1;
        }
    }
    printf("narrowed %d spared %d\n", narrowed, spared);
    return narrowed > 10 && spared > 10 ? 0 : 2;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("bounds")
    (d / "bounds.cpp").write_text(PROGRAM)
    exe = str(d / "bounds")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", CSRC, "-o", exe, str(d / "bounds.cpp")], check=True)
    return exe


@pytest.mark.parametrize("batches", [1, 2, 3])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_bounds_hold_whenever_nothing_is_in_flight(program, seed, batches):
    out = subprocess.run([program, str(seed), str(batches)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
