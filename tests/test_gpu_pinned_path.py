"""Batches that stay in pinned memory: the warp-per-packet kernel at the edges of its rounds, the one-launch grouping at
the edges of its splits, and the flow table's sweep, against the CPU checker (bytes, statuses and counters are equal)."""
import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu

ROUND = 1984  # payload bytes a warp takes per round


def _expected_counters(slots, start, max_slots):
    """Consecutive per slot in batch order."""
    out, nxt = np.zeros(len(slots), np.uint64), dict(start)
    for i, s in enumerate(slots):
        if s < max_slots:
            out[i] = nxt.get(int(s), 0)
            nxt[int(s)] = nxt.get(int(s), 0) + 1
    return out, nxt


# 1 / 256 / 257: nonces inside the seal kernel or by the grouping launch; up to 1024 one CTA with one or two packets a thread,
# then 4, 8, 16 CTAs with one and 16 with two and four; 32769: the chain of kernels.  Keypairs: one, two and three digits.
@pytest.mark.parametrize("n,n_peers", [(1, 1), (256, 40), (257, 40), (512, 3), (513, 3), (1024, 600), (1025, 600), (2048, 9), (2049, 2000),
                                       (4096, 5), (4097, 5), (8192, 700), (8193, 3000), (16_384, 50), (16_385, 600_000), (32768, 300_000),
                                       (32769, 70)])
def test_counters_and_replay_at_the_edges_of_a_split(gpu_lib, oracle, n, n_peers):
    from bnk_b200 import Context
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_REPLAY, PKT_BAD_DESC

    rng = np.random.default_rng(n)
    c = Context(max_keypairs=n_peers, mtu=0, flow_capacity=0, replay_ring_blocks=32)
    try:
        used = min(n_peers, 200)
        keys = rng.integers(0, 256, (used, 32), dtype=np.uint8)
        first = n_peers - used  # the highest slots: every digit of the sort takes part
        c.set_keypairs(first, keys, keys, np.arange(used, dtype=np.uint32))
        size, stride = 20, 80
        b, r = c.batch(n, n * stride), c.batch(n, n * stride)
        state, start = {}, {}
        for turn in range(2):
            slots = (first + np.where(rng.random(n) < 0.3, used - 1, rng.integers(0, used, n))).astype(np.uint32)
            if n > 8:
                slots[rng.integers(0, n, 2)] = n_peers  # not a keypair
            b.ring[:] = rng.integers(0, 256, n * stride, dtype=np.uint8)
            b.off[:], b.len[:], b.slot[:], b.counter[:] = np.arange(n) * stride, size, slots, 77
            want_ctr, start = _expected_counters(slots, start, n_peers)
            real = slots < n_peers
            key_of = np.where(real, slots - np.uint32(first), 0).astype(np.uint32)
            ring, st, ln = H.oracle_seal(oracle, keys, np.arange(used), 0, b.ring, b.off, b.len, key_of, want_ctr)
            b.seal(n, F_ASSIGN_COUNTERS)
            assert np.array_equal(b.counter[real], want_ctr[real])  # (a packet without a keypair has no counter to report)
            assert np.array_equal(b.status, np.where(real, st, PKT_BAD_DESC)) and np.array_equal(b.out_len, np.where(real, ln, 0))
            assert H.spans_differ_count(np.array(b.ring), ring, b.off[real], ln[real]) == 0
            for s in (first, n_peers - 1):
                assert c.send_counter(s) == start.get(s, 0)
            # arrival: swaps, and copies of earlier packets in the place of a few
            order = np.arange(n)
            for i in rng.integers(0, n, n // 10):
                j = min(n - 1, int(i) + int(rng.integers(1, 70)))
                order[[i, j]] = order[[j, i]]
            again = rng.integers(0, n, n // 50)
            order[again] = order[np.maximum(again - rng.integers(1, 300, len(again)), 0)]
            r.ring[:] = np.array(b.ring).reshape(n, stride)[order].reshape(-1)
            r.off[:], r.len[:], r.slot[:] = b.off, 16 + 32 + 16, slots[order]
            _, st, ctr, ln = H.oracle_open(oracle, keys, r.ring, r.off, r.len, key_of[order])
            st[~real[order]] = PKT_BAD_DESC
            want, state = H.oracle_replay(oracle, 32, r.slot, ctr, st, state)
            r.open(n, F_REPLAY)
            assert np.array_equal(r.status, want), np.flatnonzero(r.status != want)[:8]
            assert np.array_equal(r.out_len[want == 0], ln[want == 0])
        for s in list(state)[:5]:
            last, ring = c.replay_export(s)
            assert last == state[s].last and np.array_equal(ring, state[s].ring())
    finally:
        c.close()


@pytest.mark.parametrize("n", [16, 17, 64, 65, 160, 161])  # sizes of the descriptors that go along with a launch
def test_counters_and_replay_at_the_edges_of_inline_descriptors(gpu_lib, oracle, n):
    test_counters_and_replay_at_the_edges_of_a_split(gpu_lib, oracle, n, 40)


@pytest.mark.parametrize("copies", [False, True])
def test_round_edges_and_forgeries_of_long_packets(gpu_lib, oracle, copies):
    from bnk_b200.device import F_NO_D2H, F_NO_H2D

    from bnk_b200 import Context

    rng = np.random.default_rng(3)
    lens = np.array([k * ROUND + d for k in (1, 2) for d in (-65, -64, -17, -16, -15, -1, 0, 1, 15, 16, 17, 64)] + [3 * ROUND + 5], np.uint32)
    n = len(lens)
    keys = rng.integers(0, 256, (3, 32), dtype=np.uint8)
    slots = rng.integers(0, 3, n).astype(np.uint32)
    ctr = rng.integers(0, 2**60, n, dtype=np.uint64)
    off = H.layout_packed(lens)
    with Context(max_keypairs=3, mtu=0, flow_capacity=0) as c:
        c.set_keypairs(0, keys, keys, np.arange(3, dtype=np.uint32))
        b = c.batch(n, H.ring_bytes_for(off, lens))
        b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
        b.off[:], b.len[:], b.slot[:], b.counter[:] = off, lens, slots, ctr
        plain = np.array(b.ring)
        ring, st, ln = H.oracle_seal(oracle, keys, np.arange(3), 0, plain, off, lens, slots, ctr)

        def call(f):
            if not copies:
                return f(n)
            b.upload(n)
            f(n, F_NO_H2D | F_NO_D2H)
            b.download(n)

        call(b.seal)
        assert np.array_equal(b.out_len, ln) and H.spans_equal(np.array(b.ring), ring, off, ln) == []
        hurt = np.arange(n) % 3 == 0  # a byte of the ciphertext, the first or a later round's
        for i in np.flatnonzero(hurt):
            b.ring[int(off[i]) + 16 + int(rng.integers(0, lens[i]))] ^= 1
        b.len[:] = ln
        want, st, _, _ = H.oracle_open(oracle, keys, b.ring, off, ln, slots)
        call(b.open)
        assert np.array_equal(b.status, st) and np.array_equal(st == oracle.AUTH_FAIL, hurt)
        assert H.spans_equal(np.array(b.ring), want, off, ln - 32, start=16) == []


def test_flows_noted_by_the_seal_kernel_and_swept(gpu_lib, oracle):
    """More than 4096 flows over a clock that passes their lifetimes, noted by seal submits and by filter submits in
    turn: the table equals the checker's map after every one."""
    from bnk_b200 import Context, gen
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_NOTE_OUTBOUND

    sec = 10**9
    rng = np.random.default_rng(8)
    with Context(max_keypairs=2, mtu=1420, flow_capacity=1 << 15) as c:
        keys = rng.integers(0, 256, (2, 32), dtype=np.uint8)
        c.set_keypairs(0, keys, keys, np.zeros(2, np.uint32))
        c.acl_set(True, None)
        f = oracle.Filter()
        f.set_rules([])
        now = 1_700_000_000 * sec
        for turn, (n, step) in enumerate([(100, 1), (3000, 1), (1500, 31), (200, 5), (2500, 20), (257, 40), (64, 120), (1, 1)]):
            now += step * sec
            proto = rng.choice(np.array([6, 17, 1], np.uint8), n)
            h = gen._headers(proto, np.full(n, gen.ip4(100, 64, 0, 1), np.uint64), rng.integers(1 << 30, 1 << 31, n).astype(np.uint64),
                             rng.integers(1, 65536, n).astype(np.uint64), rng.integers(1, 65536, n).astype(np.uint64))
            lens = np.full(n, 28, np.uint32)
            h[n // 2, 0] = 0x65  # not IPv4: nothing to note
            f.note_batch(np.ascontiguousarray(h), 28, lens, now)
            b = c.batch(n, n * 80)
            b.ring.reshape(n, 80)[:, 16:44] = h
            b.off[:], b.len[:], b.slot[:] = np.arange(n) * 80, lens, rng.integers(0, 3, n)  # slot 2: refused, noted all the same
            if turn % 3 == 2:
                b.filter_note(n, now)
            else:
                b.seal(n, F_ASSIGN_COUNTERS | F_NOTE_OUTBOUND, now)
            b.close()
            assert c.flows_count() == f.flow_count, turn
            assert H.flows_equal(c.flows_export(), f.flows()), turn


@pytest.mark.parametrize("copied", [False, True])  # how the results come back
def test_split_uploads_super_packets_only(gpu_lib, oracle, copied, monkeypatch):
    """The split and the seal behind it change packets, then messages, and not a byte beside them in the host ring, where
    slots stand back to back and device memory holds another use's bytes; a refused segment changes none.  The sealed
    messages are on the device too."""
    from bnk_b200 import Context
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_NO_H2D, F_REPLAY, F_USE_OUT_LEN, PKT_BAD_DESC, PKT_NO_KEYPAIR
    from tests.test_gpu_gso import _plan, _tcp_super

    if copied:
        monkeypatch.setenv("BNK_HOST_DIRECT_BYTES", "0")
    rng = np.random.default_rng(4)
    supers, meta = [], []
    for size, gso in [(40_000, 1251), (9000, 333), (1380, 1380), (7, 2)]:
        pkt, cs, hdr = _tcp_super(rng, size)
        supers.append(pkt)
        meta.append((hdr, gso, cs, 16, 6))
    sup, seg_len, n, ring_bytes = _plan(supers, meta, 1472)
    want = [s for p, m in zip(supers, meta) for s in oracle.gso_split(p, *m)]
    key = rng.integers(0, 256, (1, 32), dtype=np.uint8)
    with Context(max_keypairs=2, mtu=1420, flow_capacity=0) as c:
        c.set_keypairs(0, key, key, np.array([9], np.uint32))
        b = c.batch(n, ring_bytes + 64)
        off = H.layout_packed(seg_len, slack=48)
        off += (np.arange(n) >= n // 2).astype(np.uint32) * 64  # a gap in the middle
        b.off[:], b.len[:], b.slot[:] = off, 1400, 0
        b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
        b.upload(n)
        b.ring[:] = 0xEE
        for j, pkt in enumerate(supers):
            b.ring[int(sup[j]["src_off"]):int(sup[j]["src_off"]) + len(pkt)] = np.frombuffer(pkt, np.uint8)
        b.len[:] = seg_len
        b.len[3] += 1   # does not match the split
        b.slot[5] = 1   # no keys there
        before = np.array(b.ring)
        b.gso_split(sup, n)
        if copied:  # (a download between the two: the packets themselves)
            b.download(n)
            expect = np.array(before)
            for i in np.delete(np.arange(n), 3):
                expect[off[i] + 16:off[i] + 16 + len(want[i])] = np.frombuffer(want[i], np.uint8)
            assert np.array_equal(b.ring, expect)
            b.ring[:] = before
        b.seal(n, F_NO_H2D | F_ASSIGN_COUNTERS)
        assert b.status[3] == PKT_BAD_DESC and b.status[5] == PKT_NO_KEYPAIR
        good = np.delete(np.arange(n), [3, 5])
        assert (b.status[good] == 0).all()
        expect, ctr = np.array(before), 0
        for i in range(n):
            if i not in (3, 5):
                msg = oracle.wg_seal(key[0].tobytes(), 9, ctr, want[i], 1420)
                expect[off[i]:off[i] + len(msg)] = np.frombuffer(msg, np.uint8)
            ctr += i not in (3, 5)
        if copied:  # of the segment that the seal refused, what the split has made of it
            expect[off[5] + 16:off[5] + 16 + len(want[5])] = np.frombuffer(want[5], np.uint8)
        assert np.array_equal(b.ring, expect)
        b.open(n, F_NO_H2D | F_USE_OUT_LEN | F_REPLAY)
        assert (b.status[good] == 0).all()
        room = np.zeros(len(before), bool)
        for i in good:
            assert b.payload(i)[:len(want[i])] == want[i], i
            room[off[i]:off[i] + 32 + ((len(want[i]) + 15) & ~15)] = True
        room[off[5] + 16:off[5] + 16 + len(want[5])] = True
        assert np.array_equal(b.ring[~room], before[~room])


@pytest.mark.parametrize("n,sizes", [(4000, (1420, 1404, 1)), (12_000, (64, 300, 0)), (100, (65_000, 30_001, 9)), (2200, (65_000, 30_001, 9))])
def test_large_batches_in_pieces(gpu_lib, oracle, n, sizes, monkeypatch):
    """A batch that goes over the link in pieces, packets across the pieces' ends among them, with every option that has
    its own part in the loop: bytes, statuses and flows are the checker's, and nothing beside the packets changes."""
    from bnk_b200 import Context, gen
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_DEMUX_INDEX, F_NOTE_OUTBOUND, F_REPLAY, F_STATS

    monkeypatch.setenv("BNK_PIECES_FROM", str(1 << 20))
    rng = np.random.default_rng(n)
    lens = rng.choice(np.array(sizes, np.uint32), n)
    off = H.layout_packed(lens)
    now, peers = 1_700_000_000 * 10**9, 7
    keys = rng.integers(0, 256, (peers, 32), dtype=np.uint8)
    with Context(max_keypairs=peers, mtu=1420, flow_capacity=1 << 14) as c:
        c.set_keypairs(0, keys, keys, np.arange(100, 100 + peers, dtype=np.uint32))
        for p in range(peers):
            c.index_set(100 + p, p)
        c.acl_set(True, None)
        f = oracle.Filter()
        f.set_rules([])
        b = c.batch(n, H.ring_bytes_for(off, lens))
        b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
        for i in np.flatnonzero(lens >= 28)[::3]:
            o = int(off[i]) + 16
            h = gen._headers(np.array([17], np.uint8), *(np.array([v], np.uint64) for v in (1 << 20, rng.integers(1 << 30, 1 << 31), rng.integers(1, 65536), 53)))
            b.ring[o:o + 28] = h[0]
            f.note_outbound(h[0].tobytes(), now)
        for i in np.setdiff1d(np.flatnonzero(lens >= 28), np.flatnonzero(lens >= 28)[::3]):
            b.ring[int(off[i]) + 16] = 0x60
        b.off[:], b.len[:], b.slot[:] = off, lens, rng.integers(0, peers, n)
        slots, plain = np.array(b.slot), np.array(b.ring)
        ctr, _ = _expected_counters(slots, {}, peers)
        ring, st, ln = H.oracle_seal(oracle, keys, np.arange(100, 100 + peers), 1420, plain, off, lens, slots, ctr)
        b.seal(n, F_ASSIGN_COUNTERS | F_NOTE_OUTBOUND | F_STATS, now)
        assert b.stats()["by_status"][0] == n
        assert np.array_equal(b.counter, ctr) and np.array_equal(b.status, st) and np.array_equal(b.out_len, ln)
        assert np.array_equal(b.ring, ring)
        assert H.flows_equal(c.flows_export(), f.flows())
        hurt = rng.choice(n, max(1, n // 50), replace=False)
        for i in hurt:
            b.ring[int(off[i]) + int(ln[i]) - 1] ^= 1
        b.len[:], b.slot[:] = ln, 0
        want, st, ctr, ln2 = H.oracle_open(oracle, keys, b.ring, off, ln, slots)
        b.open(n, F_DEMUX_INDEX | F_REPLAY)
        assert np.array_equal(b.status, st) and np.array_equal(b.slot, slots) and np.array_equal(b.counter, ctr)
        assert np.array_equal(b.out_len, ln2) and np.array_equal(b.ring, want)
        assert set(np.flatnonzero(st == oracle.AUTH_FAIL)) == set(hurt)


def test_nothing_to_send_in_pieces(gpu_lib, monkeypatch):
    """An empty batch has no pieces, whatever size they start from."""
    from bnk_b200 import Context
    from bnk_b200.device import F_STATS

    monkeypatch.setenv("BNK_PIECES_FROM", "0")
    with Context(max_keypairs=1, flow_capacity=0) as c:
        b = c.batch(4, 4096)
        for f in (b.seal, b.open):
            f(0, F_STATS)
            assert b.stats()["packets"] == 0
            f(0)
