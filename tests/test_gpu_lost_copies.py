"""What kernels do when a bulk copy over the link does not come.  The library here is a build of its own (_build.build_lost_copies)
that never asks for copies of LOST_BYTES and gives up waiting soon, so which packets are hit is a matter of their sizes."""
import os

import numpy as np
import pytest

from bnk_b200.filter import CompiledRule, PortRange, flatten_rules
from tests import helpers as H
from tests import reference_cases as RC

pytestmark = pytest.mark.gpu


def _load(monkeypatch, **kind):
    from bnk_b200 import _build, _lib

    if not os.path.exists(_build.lost_copies_path(**kind)):
        _build.build_lost_copies(**kind)
    monkeypatch.setattr(_lib, "_LIB", _lib.load(_build.lost_copies_path(**kind)))
    return _build.LOST_BYTES


@pytest.fixture
def lossy(gpu_lib, monkeypatch):
    return _load(monkeypatch)


@pytest.fixture
def gives_up(gpu_lib, monkeypatch):
    return _load(monkeypatch, gives_up=True)


def test_split_leaves_out_what_did_not_come(lossy, oracle):
    """Two super-packets of the same layout, one of them four bytes off the other's alignment: the copy of its last segment is
    one that does not come.  That segment is refused, its bytes of the super-packet on the device stay as they were, and
    everything else is split and sealed."""
    from bnk_b200 import Context
    from bnk_b200.device import F_NO_H2D
    from tests.test_gpu_gso import _tcp_super

    rng = np.random.default_rng(17)
    gso, hdr, stride = 1008, 40, 1152
    last = lossy - 16
    supers = [_tcp_super(rng, 2 * gso + last)[0] for _ in range(2)]
    src = [8, 4096 + 12]  # the payloads start 0 and 4 bytes behind a multiple of 16
    n = 6
    off = 8192 + H.layout_fixed(n, stride)
    lens = np.array([hdr + gso, hdr + gso, hdr + last] * 2, np.uint32)
    key = rng.integers(0, 256, (1, 32), dtype=np.uint8)
    from bnk_b200.device import GSO_SUPER_DTYPE

    def described(j, first):
        s = np.zeros(1, GSO_SUPER_DTYPE)
        s["src_off"], s["src_len"], s["first_pkt"], s["n_pkts"] = src[j], len(supers[j]), first, 3
        s["hdr_len"], s["gso_size"], s["csum_start"], s["csum_offset"], s["proto"] = hdr, gso, 20, 16, 6
        return s

    with Context(max_keypairs=1, mtu=1420, flow_capacity=0) as c:
        c.set_keypairs(0, key, key, np.array([3], np.uint32))
        b = c.batch(n, 8192 + n * stride)
        b.ring[:] = 0xA5
        b.off[:], b.len[:], b.slot[:], b.counter[:] = off, lens, 0, np.arange(n)
        b.upload(n)
        for s, at in zip(supers, src):
            b.ring[at:at + len(s)] = np.frombuffer(s, np.uint8)
        b.gso_split(np.concatenate([described(0, 0), described(1, 3)]), n)
        b.ring[:] = 0
        b.download(n)
        want = [s for p in supers for s in oracle.gso_split(p, hdr, gso, 20, 16, 6)]
        for i in range(n):
            got = b.ring[off[i] + 16:off[i] + 16 + lens[i]]
            if i < 5:
                assert got.tobytes() == want[i], i
            else:
                assert not got.any()
        # what the device holds of the second super-packet, through the first one's segments
        b.gso_split(described(1, 0), n, F_NO_H2D)
        b.download(n)
        held = supers[1][:hdr + 2 * gso] + b"\xa5" * last
        for i, w in enumerate(oracle.gso_split(held, hdr, gso, 20, 16, 6)):
            assert b.ring[off[i] + 16:off[i] + 16 + lens[i]].tobytes() == w, i
        b.seal(n, F_NO_H2D)
        assert list(np.flatnonzero(b.status)) == [5] and b.out_len[5] == 0
        b.close()


ROUND = 1984  # payload bytes a warp takes per round


# 8: a warp each, the descriptors with the launch and the header of a message ahead; 1024: tiles of four, so up to three packets
# lie behind the one that does not come; long: its second round does not come; and neighbours with this kernel asked for
@pytest.mark.parametrize("n,lost,long,stride", [(8, 3, False, 4096), (8, 0, True, 4096), (256, 255, False, 4096), (1024, 513, False, 4096),
                                                (1024, 515, True, 4096), (1024, 514, False, 1152)])
def test_seal_and_open_refuse_what_did_not_come(lossy, oracle, monkeypatch, n, lost, long, stride):
    from bnk_b200 import Context
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_NOTE_OUTBOUND, F_REPLAY, PKT_NOT_READ

    if stride < 4096:
        monkeypatch.setenv("BNK_AEAD_KERNEL", "wpp")  # read when a context is created
    rng = np.random.default_rng(n + lost)
    peers, now = 5, RC.T0
    keys = rng.integers(0, 256, (peers, 32), dtype=np.uint8)
    off, slot = H.layout_fixed(n, stride), rng.integers(0, peers, n).astype(np.uint32)
    refused = np.arange(n) == lost if n <= 256 else (np.arange(n) >= lost) & (np.arange(n) < lost // 4 * 4 + 4)
    with Context(max_keypairs=peers, mtu=0, flow_capacity=1 << 12, replay_ring_blocks=32) as c:
        c.set_keypairs(0, keys, keys, np.arange(peers, dtype=np.uint32))
        c.acl_set(True, flatten_rules([CompiledRule(srcs=["10.0.0.0/8"], proto="udp", ports=[PortRange(1, 9)])]))
        b = c.batch(n, n * stride)
        b.off[:], b.slot[:] = off, slot

        def lay_out(lens):
            b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
            for i in range(n):
                p = RC.udp(RC.SELF, RC.ip("10.0.0.0") + i, 7, 8)[:28]
                b.ring[off[i] + 16:off[i] + 44] = np.frombuffer(p[:2] + int(lens[i]).to_bytes(2, "big") + p[4:], np.uint8)
            b.len[:] = lens
            return np.array(b.ring)

        # ---- sealed ----
        lens = np.full(n, 1104, np.uint32)
        lens[lost] = (ROUND if long else 0) + lossy - 9
        ctr = np.array([np.count_nonzero(slot[:i] == slot[i]) for i in range(n)], np.uint64)
        plain = lay_out(lens)
        ring, st, ln = H.oracle_seal(oracle, keys, np.arange(peers), 0, plain, off, lens, slot, ctr)
        b.seal(n, F_ASSIGN_COUNTERS | F_NOTE_OUTBOUND, now)
        assert np.array_equal(b.status, np.where(refused, PKT_NOT_READ, st))
        assert np.array_equal(b.out_len, np.where(refused, 0, ln))
        assert H.spans_equal(np.array(b.ring), ring, off[~refused], ln[~refused]) == []
        kept = off + (16 + ROUND) * (long & (np.arange(n) == lost)).astype(np.uint32)  # the first round of a long message is out
        assert H.spans_equal(np.array(b.ring), plain, kept[refused], off[refused] + stride - kept[refused]) == []
        if long:
            assert H.spans_equal(np.array(b.ring), ring, off[[lost]], [16 + ROUND]) == []
        assert c.flows_count() == n - refused.sum() + long  # (its flow is in the first round)

        # ---- opened ----
        lens[lost] = (ROUND if long else 0) + lossy - 32 + (16 if long else 0)
        plain = lay_out(lens)
        ctr += 1000
        ring, st, ln = H.oracle_seal(oracle, keys, np.arange(peers), 0, plain, off, lens, slot, ctr)
        b.ring[:], b.len[:] = ring, ln
        want_ring, st, got_ctr, want_ln = H.oracle_open(oracle, keys, ring, off, ln, slot)
        b.open(n, F_REPLAY)
        st[refused] = PKT_NOT_READ
        want, state = H.oracle_replay(oracle, 32, slot, got_ctr, st)
        assert np.array_equal(b.status, want) and np.array_equal(b.out_len, np.where(refused, 0, want_ln))
        assert H.spans_equal(np.array(b.ring), want_ring, off[~refused], want_ln[~refused], 16) == []
        if long:
            ring[off[lost] + 16:off[lost] + 16 + ROUND] = 0
        assert H.spans_equal(np.array(b.ring), ring, off[refused], [stride] * refused.sum()) == []
        for s, r in state.items():
            last, words = c.replay_export(s)
            assert last == r.last and np.array_equal(words, r.ring())

        # ---- and the next submit is as any other ----
        lens[lost] = 700 if not long else ROUND + 732  # (copies of 704 and 736 bytes)
        plain = lay_out(lens)
        ring, st, ln = H.oracle_seal(oracle, keys, np.arange(peers), 0, plain, off, lens, slot, ctr)
        b.counter[:] = ctr
        b.seal(n)
        assert np.array_equal(b.status, st) and H.spans_equal(np.array(b.ring), ring, off, ln) == []
        b.close()


def _dense(c, oracle, keys, n, sizes, gaps, rng, first=0, ring_bytes=0):
    """A batch whose packets lie close together, its payloads and what sealing makes of it."""
    room = (sizes.astype(np.int64) + 47) // 16 * 16
    off = np.concatenate([[0], np.cumsum(room + gaps)])
    b = c.batch(n, max(int(off[-1]), ring_bytes))
    b.off[:], b.len[:], b.slot[:] = off[:-1], sizes, rng.integers(0, len(keys), n)
    b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
    ctr = np.array([first + np.count_nonzero(b.slot[:i] == b.slot[i]) for i in range(n)], np.uint64)
    ring, st, ln = H.oracle_seal(oracle, keys, np.arange(len(keys)), 0, b.ring, b.off, b.len, b.slot, ctr)
    assert (st == 0).all()
    return b, np.array(b.ring), ring, ln, ctr


# Packets of 1136 bytes, two a copy; the one that does not come lies by itself.  Tiles of 16 packets, one or three to a CTA: the
# copy behind the one that does not come is on its way already, and what would come next is not asked for.  (So few are opened by
# another kernel.)
@pytest.mark.parametrize("n,lost,stretch", [(1024, 518, 16), (1024, 1023, 16), (4096, 3 * 48 + 17, 48), (4096, 4095, 48)])
def test_neighbours_of_what_did_not_come(lossy, oracle, n, lost, stretch):
    from bnk_b200 import Context
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_REPLAY, PKT_NOT_READ

    rng = np.random.default_rng(n + lost)
    peers = 5
    keys = rng.integers(0, 256, (peers, 32), dtype=np.uint8)
    sizes, gaps = np.full(n, 1104, np.uint32), np.zeros(n, np.int64)
    sizes[lost] = lossy - 32
    gaps[max(lost - 1, 0)] = gaps[lost] = 32
    runs, tile = [], 16  # as they are asked for from the stretch's first packet on
    for t in range(lost // stretch * stretch, min(lost // stretch * stretch + stretch, n), tile):
        at, end = t, min(t + tile, n)
        while at < end:
            more = 2 if at + 1 < end and lost not in (at, at + 1) else 1
            runs.append(range(at, at + more))
            at += more
    which = next(k for k, r in enumerate(runs) if lost in r)
    refused = np.zeros(n, bool)
    for k, r in enumerate(runs):
        refused[list(r)] = k == which or k > which + 1
    with Context(max_keypairs=peers, mtu=0, flow_capacity=0, replay_ring_blocks=32) as c:
        c.set_keypairs(0, keys, keys, np.arange(peers, dtype=np.uint32))
        b, plain, ring, ln, ctr = _dense(c, oracle, keys, n, sizes, gaps, rng)
        b.status[:], b.out_len[:] = 0, 7
        b.seal(n, F_ASSIGN_COUNTERS)
        assert np.array_equal(b.status, np.where(refused, PKT_NOT_READ, 0)) and np.array_equal(b.out_len, np.where(refused, 0, ln))
        assert np.array_equal(b.counter, ctr)
        assert H.spans_equal(np.array(b.ring), ring, b.off[~refused], ln[~refused]) == []
        assert H.spans_equal(np.array(b.ring), plain, b.off[refused], ln[refused]) == []
        if n < 4096:
            return
        b.ring[:], b.len[:] = ring, ln
        want_ring, st, got, want_ln = H.oracle_open(oracle, keys, ring, b.off, ln, b.slot)
        b.open(n, F_REPLAY)
        want, state = H.oracle_replay(oracle, 32, b.slot, got, np.where(refused, PKT_NOT_READ, st))
        assert np.array_equal(b.status, want) and np.array_equal(b.out_len, np.where(refused, 0, want_ln))
        assert H.spans_equal(np.array(b.ring), want_ring, b.off[~refused], want_ln[~refused], 16) == []
        assert H.spans_equal(np.array(b.ring), ring, b.off[refused], ln[refused]) == []
        for s, r in state.items():
            last, words = c.replay_export(s)
            assert last == r.last and np.array_equal(words, r.ring())
        b.close()


@pytest.mark.parametrize("n", [4096, 5003])
def test_what_has_not_been_handed_out_is_refused(gives_up, oracle, n):
    """The warp that hands packets out gives up in the middle of the batch: what it has not sent back is refused, whatever the arrays
    held before, nothing of it is written, and the replay window does not take it for opened."""
    from bnk_b200 import Context
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_REPLAY, PKT_NOT_READ

    rng = np.random.default_rng(n)
    peers = 5
    keys = rng.integers(0, 256, (peers, 32), dtype=np.uint8)
    with Context(max_keypairs=peers, mtu=0, flow_capacity=0, replay_ring_blocks=32) as c:
        c.set_keypairs(0, keys, keys, np.arange(peers, dtype=np.uint32))
        b, plain, ring, ln, ctr = _dense(c, oracle, keys, n, np.full(n, 1104, np.uint32), np.zeros(n, np.int64), rng, 5000, 2048 * n)
        for p in range(peers):
            c.set_send_counter(p, 5000)
        b.status[:], b.out_len[:] = 0, 7
        b.seal(n, F_ASSIGN_COUNTERS)
        refused = np.array(b.status) == PKT_NOT_READ
        assert refused.any() and not b.status[~refused].any()
        assert np.array_equal(b.out_len, np.where(refused, 0, ln)) and np.array_equal(b.counter, ctr)
        assert H.spans_equal(np.array(b.ring), ring, b.off[~refused], ln[~refused]) == []
        assert H.spans_equal(np.array(b.ring), plain, b.off[refused], ln[refused]) == []
        want_ring, st, got, want_ln = H.oracle_open(oracle, keys, ring, b.off, ln, b.slot)
        # on the device, authentic packets everywhere: another kernel opens them, as they lie far apart
        dense = np.array(b.off)
        apart = H.layout_fixed(n, 2048)
        ctr -= np.uint64(5000)
        for i in range(n):
            b.ring[apart[i] + 16:apart[i] + 1120] = 0
        wide, st_wide, ln_wide = H.oracle_seal(oracle, keys, np.arange(peers), 0, b.ring, apart, b.len, b.slot, ctr)
        b.ring[:], b.off[:], b.len[:] = wide, apart, ln_wide
        b.open(n, F_REPLAY)
        _, state = H.oracle_replay(oracle, 32, b.slot, ctr, st_wide)
        assert not b.status.any()
        # and now neighbours, of counters that the window has not seen
        b.off[:] = dense
        for rep in range(2):
            b.ring[:], b.len[:], b.status[:] = ring, ln, 0
            b.open(n, F_REPLAY)
            refused = np.array(b.status) == PKT_NOT_READ
            assert refused.any()
            want, state = H.oracle_replay(oracle, 32, b.slot, got, np.where(refused, PKT_NOT_READ, st), state)
            assert np.array_equal(b.status, want) and np.array_equal(b.out_len, np.where(refused, 0, want_ln))
            assert H.spans_equal(np.array(b.ring), want_ring, b.off[~refused], want_ln[~refused], 16) == []
            assert H.spans_equal(np.array(b.ring), ring, b.off[refused], ln[refused]) == []
            for s, r in state.items():
                last, words = c.replay_export(s)
                assert last == r.last and np.array_equal(words, r.ring())
        b.close()


def test_a_wait_gives_up_after_a_time_that_callers_can_bear(lossy):
    """From the time that this build's waits take, that of the product's: between a tenth of a second, far above what a busy link
    keeps a packet waiting, and two seconds."""
    import re

    from bnk_b200 import Context, _build
    from bnk_b200.device import F_TIMED, PKT_NOT_READ

    text = open(os.path.join(_build.CSRC, "bulk.cuh")).read()
    turns = 1 << int(re.search(r"#define BNK_BULK_TURNS \(1u << (\d+)\)", text)[1])
    with Context(max_keypairs=1, mtu=0, flow_capacity=0) as c:
        key = np.zeros((1, 32), np.uint8)
        c.set_keypairs(0, key, key, np.zeros(1, np.uint32))
        b = c.batch(1, 1024)
        took = []
        for size, status in [(lossy, PKT_NOT_READ)] * 3 + [(lossy + 16, 0)] * 3:
            b.off[:], b.len[:], b.slot[:] = 0, size, 0
            b.seal(1, F_TIMED)
            assert b.status[0] == status
            took.append(b.last_kernel_ms())
        seconds = (min(took[:3]) - min(took[3:])) / 1e3 / (2 * _build.LOST_TURNS) * turns  # (it waits twice)
        assert 0.1 < seconds < 2, seconds
        b.close()
