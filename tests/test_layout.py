"""How a batch's packets lie in its ring (host/scan.cpp) and which batches cross the link by neighbours (csrc/layout.h).  Host code only."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = """
#include "bnk_b200/csrc/layout.h"
extern "C" void look(const uint32_t *off, const uint32_t *len, uint32_t n, int open, uint32_t room, uint64_t *out) {
    const PacketScan r = scan_packets(off, len, n, room);
    const Layout l = layout_of(r, n, kMostRoom);
    const uint64_t v[] = {r.end, r.sum, r.longest, r.lowest, r.joined, r.in_order, l.dense, n && in_stream(l, n, open)};
    for (int i = 0; i < 8; i++) out[i] = v[i];
}
// tile and CTAs, and whether every tile has one that takes it, as the kernel deals them out
extern "C" void grid(uint32_t n, uint64_t bytes, uint32_t *out) {
    const StreamGrid g = stream_grid(n, bytes);
    const uint32_t tiles = (n + g.tile - 1) / g.tile, share = (tiles + g.ctas - 1) / g.ctas;
    out[0] = g.tile;
    out[1] = g.ctas;
    out[2] = (uint64_t)g.ctas * share >= tiles;
}
"""
ROOM = {False: 32, True: 0}  # behind a payload that is sealed; behind a message that is opened


@pytest.fixture(scope="module")
def look(tmp_path_factory):
    d = tmp_path_factory.mktemp("layout")
    (d / "look.cpp").write_text(PROGRAM)
    so = str(d / "look.so")
    subprocess.run(["g++", "-std=c++17", "-O3", "-fPIC", "-shared", "-I", ROOT, "-o", so, str(d / "look.cpp"),
                    os.path.join(ROOT, "bnk_b200", "host", "scan.cpp")], check=True)
    lib = C.CDLL(so)
    f = lib.look

    def call(off, length, opened):
        off, length = np.ascontiguousarray(off, np.uint32), np.ascontiguousarray(length, np.uint32)
        out = np.zeros(8, np.uint64)
        f(off.ctypes.data_as(C.c_void_p), length.ctypes.data_as(C.c_void_p), C.c_uint32(len(off)), C.c_int(opened), C.c_uint32(ROOM[opened]),
          out.ctypes.data_as(C.c_void_p))
        return dict(zip(("end", "sum", "longest", "lowest", "joined", "in_order", "dense", "stream"), map(int, out)))

    call.lib = lib
    return call


@pytest.mark.parametrize("opened", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 31, 33, 99, 1024, 1025, 1026, 3001])
def test_scan_is_what_it_says(look, n, opened):
    rng = np.random.default_rng(n)
    # the last: ends beyond 32 bits, lengths that no packet has
    for gaps, most in (((0, 1, 15, 16, 17, 31, 32), 200), ((-16, -1, 0, 16), 200), ((0,), 1500), ((0, 2**31), 200), ((0, 16), 1 << 26)):
        length, gap = rng.integers(0, most, n), rng.choice(gaps, n)
        room = ROOM[opened]
        off = np.zeros(n, np.int64)
        for i in range(1, n):  # in whole pieces, but for odd gaps; wrapped where 32 bits end
            off[i] = (((off[i - 1] + length[i - 1] + room + 15) & ~15) + gap[i]) % 2**32
        if rng.random() < 0.5:
            k = rng.permutation(n)
            off, length = off[k], length[k]
        joined = sum(int(b) - ((int(a) + int(k) + room + 15) & ~15) in (0, 16) for a, k, b in zip(off, length, off[1:]))
        got = look(off, length, opened)
        assert got["end"] == int((off + length).max()) and got["sum"] == int(length.sum()) and got["longest"] == int(length.max())
        assert got["lowest"] == int(off.min()) and got["joined"] == joined
        assert got["in_order"] == all(int(a) + int(k) + room <= int(b) for a, k, b in zip(off, length, off[1:]))


def _lies(n, size, step, order=None):
    off = np.arange(n, dtype=np.int64) * step
    return (off if order is None else off[order]), np.full(n, size)


@pytest.mark.parametrize("opened", [False, True])
def test_batches_whose_packets_join_go_by_neighbours(look, opened):
    extra = 32 if opened else 0  # a message and its payload
    rng = np.random.default_rng(1)
    for n, size, step in ((4096, 1420, 1472), (12_000, 1420, 1456), (9000, 64, 112), (16_000, 64, 96), (3000, 400, 432)):
        got = look(*_lies(n, size + extra, step), opened)
        assert got["dense"] and got["stream"], (n, size, step)
    # not: another order, in which every packet is a copy of its own; far apart, whichever of them comes first; in slots that are too
    # wide to join; few; long
    for name, n, size, step, order in (("falling", 9000, 64, 112, np.arange(9000)[::-1]), ("any order", 9000, 64, 112, rng.permutation(9000)),
                                       ("falling, apart", 4096, 300, 1024, np.arange(4096)[::-1]),
                                       ("apart, the last one first", 4096, 1420, 4096, np.r_[4095, 0:4095]), ("slots", 9000, 64, 128, None),
                                       ("slots", 16_000, 64, 128, None), ("few", 256, 1420, 1472, None), ("long", 1000, 1970, 2032, None)):
        got = look(*_lies(n, size + extra, step, order), opened)
        assert not got["stream"], name
        assert got["dense"] == (name in ("falling", "any order", "slots", "few")), name
    # very many small ones that do not join: as many bytes a copy as there is little to gain in pieces; in no order more
    for n, size, step, order, goes in ((20_000, 64, 128, None, False), (20_000, 150, 224, None, True), (80_000, 150, 224, None, False), (80_000, 300, 384, None, True),
                                       (16_000, 200, 240, rng.permutation(16_000), False), (16_000, 300, 352, rng.permutation(16_000), True)):
        assert look(*_lies(n, size + extra, step, order), opened)["stream"] == goes, (n, size)
    # large packets that do not join are sealed that way, and opened only where they would otherwise go in pieces
    got = look(*_lies(4096, 1300 + extra, 1472), opened)
    assert got["dense"] and got["stream"] == (not opened)
    assert look(*_lies(20_000, 1300 + extra, 1472), opened)["stream"]


@pytest.mark.parametrize("size", [60, 1420])
def test_grid_leaves_room_for_other_calls(look, size):
    out = (C.c_uint32 * 3)()
    for n in [*range(257, 3000), *range(3000, 1_000_000, 997)]:
        look.lib.grid(C.c_uint32(n), C.c_uint64(n * size), out)
        tile, ctas, covered = out
        assert tile in (4, 8, 16) and covered and 40 < ctas <= 143, n  # of 148 SMs
