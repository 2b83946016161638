"""The order of a submit's copies and kernels over its streams (csrc/pieces.h, csrc/submit_order.h) with a CUDA runtime that
only keeps lists: every stream runs its operations in order, a stream that is waited for runs and the others only as far as
its events ask, and any call may fail.  Host code only."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bnk_b200", "csrc")

RUNTIME = r"""
#pragma once
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <deque>
#include <functional>
#include <vector>
enum cudaError_t { cudaSuccess, cudaErrorUnknown };
enum cudaMemcpyKind { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost };
struct Stream;
struct Event { std::vector<char> reached{1}; std::vector<Stream *> by{nullptr}; }; // of each record; none yet: reached
struct Op { std::function<void()> run; Event *wait = nullptr; size_t until = 0; bool blocked() const { return wait && !wait->reached[until]; } };
struct Stream { std::deque<Op> ops; };
typedef Stream *cudaStream_t;
typedef Event *cudaEvent_t;
inline int calls_left = 1 << 30; // the call after that many fails, and later ones do not
inline bool fails() { return --calls_left == -1; }
inline bool ready(Stream *s) { return !s->ops.empty() && !s->ops.front().blocked(); }
inline void one(Stream *s) { auto op = s->ops.front(); s->ops.pop_front(); if (op.run) op.run(); }
inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    if (fails()) return cudaErrorUnknown;
    st->ops.push_back({[=] { memcpy(d, s, n); }});
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    if (fails()) return cudaErrorUnknown;
    const size_t k = e->reached.size();
    e->reached.push_back(0);
    e->by.push_back(st);
    st->ops.push_back({[=] { e->reached[k] = 1; }});
    return cudaSuccess;
}
inline cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned) {
    if (fails()) return cudaErrorUnknown;
    st->ops.push_back({nullptr, e, e->reached.size() - 1});
    return cudaSuccess;
}
// Runs st until it is empty, and other streams only as far as that takes.
inline void advance(Stream *s) {
    while (!ready(s)) advance(s->ops.front().wait->by[s->ops.front().until]);
    one(s);
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    while (!st->ops.empty()) advance(st);
    return cudaSuccess;
}
"""
PROGRAM = r"""
#include "pieces.h"
#include "submit_order.h"
#include <cstdio>
#include <cstdlib>
#include <random>
#define TRY(x) do { if ((x) != cudaSuccess) return 1; } while (0)
struct Layout { std::vector<uint32_t> off, len; uint64_t ext; };
static Stream s, up, down;
static Event ev_up, ev_down;
// A submit as the library makes it: a kernel flips every byte of its packets and of their room.
static int submit(uint8_t *dev, uint8_t *host, const Layout &l, uint32_t more) {
    const PieceStreams ps{&up, &down, &ev_up, &ev_down};
    const uint32_t n = (uint32_t)l.off.size();
    Pieces pieces(l.off.data(), l.len.data(), n, more, l.ext);
    PieceCopies copies(ps, dev, host, &s);
    Piece p;
    pieces.next(p);
    TRY(copies.up(p));
    for (bool go = true; go;) {
        TRY(copies.is_up());
        if (fails()) return 1;
        s.ops.push_back({[=, &l] { for (uint32_t i = p.first; i < p.first + p.count; i++) for (uint32_t k = 0; k < l.len[i] + more; k++) dev[l.off[i] + k] ^= 0x5a; }});
        TRY(copies.down(p));
        go = pieces.next(p);
        if (go) TRY(copies.up(p));
    }
    TRY(copies.join());
    return 0;
}
static int pieces_test(uint32_t seed) {
    std::mt19937 rng(seed);
    const uint32_t more = seed & 1 ? 48 : 0, longest = seed % 3 == 0 ? 3'000'000 : seed % 3 == 1 ? 9000 : 70'000;
    Layout l;
    uint64_t at = (rng() % 64) * 16;
    while (at < 12'000'000) {
        const uint32_t len = rng() % longest;
        l.off.push_back((uint32_t)at);
        l.len.push_back(len);
        at = (at + len + more + 15 + rng() % 100) & ~15ull;
    }
    l.ext = (l.off.back() + (uint64_t)l.len.back() + more + 15) & ~15ull;
    std::vector<uint8_t> before(l.ext + 4096), host, dev(l.ext + 4096);
    for (auto &x : before) x = (uint8_t)rng();
    auto want = before;
    for (size_t i = 0; i < l.off.size(); i++) for (uint32_t k = 0; k < l.len[i] + more; k++) want[l.off[i] + k] ^= 0x5a;
    host = before;
    if (submit(dev.data(), host.data(), l, more)) return printf("fails\n"), 1;
    const int all_calls = (1 << 30) - calls_left;
    cudaStreamSynchronize(&s);
    if (host != want || !up.ops.empty() || !down.ops.empty()) return printf("wrong bytes or copies left\n"), 1;
    for (int k = 0; k < all_calls; k++) { // a call fails: whoever has waited for s has the ring back
        host = before;
        calls_left = k;
        submit(dev.data(), host.data(), l, more);
        calls_left = 1 << 30;
        cudaStreamSynchronize(&s);
        if (!up.ops.empty() || !down.ops.empty()) return printf("copies left behind call %d of %d\n", k, all_calls), 1;
    }
    return 0;
}
// Submits of batches in turn, in place on the shared stream or copied on their own, some failing half way: what is queued of a
// submit's kernels runs behind all kernels of those in front, and waiting for a batch waits for its kernels.
static int order_test(uint32_t seed) {
    std::mt19937 rng(seed);
    Stream shared, own[3];
    Event ev[3];
    SubmitOrder o[3] = {{&own[0], &ev[0], false}, {&own[1], &ev[1], false}, {&own[2], &ev[2], false}};
    std::vector<int> ran;
    int queued = 0, last = -1;
    for (int turn = 0; turn < 400; turn++) {
        const int b = turn % 3;
        cudaStreamSynchronize(o[b].run); // its earlier submit is waited for
        const bool direct = rng() % 2;
        std::vector<int> mine;
        const bool ok = [&] {
            SubmitOrder &x = o[b];
            x.begins(&own[b]);
            if (direct) x.begins(&shared);
            if (rng() % 4 == 0) calls_left = rng() % 3;
            if (last >= 0 && x.follow(o[last]) != cudaSuccess) return false;
            for (int k = 0; k < 2; k++) {
                if (rng() % 8 == 0) return false; // a launch fails
                const int id = queued++;
                mine.push_back(id);
                x.run->ops.push_back({[&ran, id] { ran.push_back(id); }});
            }
            if (direct) return true;
            if (x.kernels_end() != cudaSuccess) return false;
            x.run->ops.push_back({[] {}}); // the copy down
            return true;
        }();
        calls_left = 1 << 30;
        if (!ok && last >= 0) SubmitOrder::failed_behind(o[last]);
        last = b;
        if (rng() % 3 == 0) {
            cudaStreamSynchronize(o[b].run);
            for (int id : mine) { bool in = false; for (int r : ran) in |= r == id; if (!in) return printf("waited for, not run: %d\n", id), 1; }
        }
    }
    for (Stream *st : {&shared, &own[0], &own[1], &own[2]}) cudaStreamSynchronize(st);
    for (size_t i = 1; i < ran.size(); i++) if (ran[i] < ran[i - 1]) return printf("%d behind %d\n", ran[i], ran[i - 1]), 1;
    return (int)ran.size() != queued;
}
int main(int, char **argv) { return argv[1][0] == 'p' ? pieces_test(atoi(argv[2])) : order_test(atoi(argv[2])); }
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("streams")
    (d / "cuda_runtime.h").write_text(RUNTIME)
    (d / "streams.cpp").write_text(PROGRAM)
    exe = str(d / "streams")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", str(d), "-I", CSRC, "-o", exe, str(d / "streams.cpp")], check=True)
    return exe


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("what", ["pieces", "order"])
def test_streams(program, what, seed):
    out = subprocess.run([program, what, str(seed)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
