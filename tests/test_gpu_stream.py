"""Batches in pinned memory whose packets lie close together: several cross the link as one copy, so what is checked is where
such a stretch begins and ends, and that nothing but the messages changes, against the oracle."""
import numpy as np
import pytest

from tests import helpers as H
from tests import reference_cases as RC

pytestmark = pytest.mark.gpu

LONGEST = 1969  # of the packets that go this way


# Tiles of 4 to 16 packets, a last one that is not full; sizes whose neighbours just fill a stretch of 3200 bytes and do not (1504 and
# 1552 with their room), the smallest and the longest, whole pieces and parts of them; packets apart, out of order, and with nothing
# between them; 16 small ones a stretch for more CTAs.
@pytest.mark.parametrize("mtu", [0, 1420])
@pytest.mark.parametrize("n,sizes,gaps", [
    (400, (1456, 1504, 1505, 1552, 1568, 1969), (0, 16)),
    (513, (LONGEST, 0, 1, 15, 16, 17, 63, 64, 65, 1968, 1953), (0, 16, 32)),
    (1025, (1420, 576, 64, 1419), (0, 16, 0, 0, 48)),
    (1503, tuple(range(300, 800, 7)), (0,)),
    (9001, (64, 40, 52, 28), (0, 16)),
])
def test_seal_and_open_of_neighbours(gpu_lib, oracle, n, sizes, gaps, mtu):
    from bnk_b200 import Context
    from bnk_b200.device import (F_ASSIGN_COUNTERS, F_DEMUX_INDEX, F_NOTE_OUTBOUND, PKT_AUTH_FAIL, PKT_BAD_DESC, PKT_COUNTER_EXHAUSTED,
                                 PKT_MALFORMED, PKT_NO_KEYPAIR)
    from bnk_b200.filter import CompiledRule, PortRange, flatten_rules

    rng = np.random.default_rng(n + mtu)
    peers, now = 7, RC.T0
    keys = rng.integers(0, 256, (peers, 32), dtype=np.uint8)
    lens = rng.choice(np.asarray(sizes, np.uint32), n)
    lens[:len(sizes)] = sizes
    last = lens.astype(np.int64) % mtu if mtu else lens.astype(np.int64)  # padded is the last unit, as far as the MTU
    body = lens - last + (np.minimum((last + 15) & ~15, mtu) if mtu else (last + 15) & ~15)
    room = ((body + 32 + 15) & ~15) + rng.choice(np.asarray(gaps), n)
    at = np.concatenate([[0], np.cumsum(room)])
    off, ring_bytes = at[:-1].astype(np.uint32), int(at[-1]) + 16
    order = np.arange(n)
    for i in rng.integers(0, n - 1, n // 25):
        order[[i, i + 1]] = order[[i + 1, i]]
    off, lens = off[order], lens[order]
    slot = rng.integers(0, peers, n).astype(np.uint32)
    refused = rng.choice(n, 6, replace=False)
    with Context(max_keypairs=peers + 1, mtu=mtu, flow_capacity=1 << 15) as c:
        c.set_keypairs(0, keys, keys, 100 + np.arange(peers, dtype=np.uint32))
        c.acl_set(True, flatten_rules([CompiledRule(srcs=["10.0.0.0/8"], proto="udp", ports=[PortRange(1, 9)])]))
        for p in range(peers):
            c.index_set(100 + p, p)
        b = c.batch(n, ring_bytes)
        b.ring[:] = rng.integers(0, 256, ring_bytes, dtype=np.uint8)
        noted = np.flatnonzero(lens >= 28)[:3000]
        b.ring[off + 16] = 0  # no IPv4
        for i in noted:
            p = RC.udp(RC.SELF, RC.ip("10.0.0.0") + int(i), 7, 8)[:28]
            b.ring[off[i] + 16:off[i] + 44] = np.frombuffer(p[:2] + int(lens[i]).to_bytes(2, "big") + p[4:], np.uint8)

        def geometry(o, ln, sl):  # a place that is no place, one past the ring, no slot, a slot without keys
            o, ln, sl = o.copy(), ln.copy(), sl.copy()
            o[refused[0]] += 4
            o[refused[1]] = (ring_bytes - 16) & ~15
            sl[refused[2]], sl[refused[3]] = peers + 1, peers
            return o, ln, sl

        # ---- sealed: nonces of the caller's, then the library's own with the flows noted ----
        plain = np.array(b.ring)
        for own in (False, True):
            b.ring[:] = plain
            ctr = rng.integers(0, 2**60, n, dtype=np.uint64)
            ctr[refused[4]] = 2**64 - 2**13 - 1
            o, ln, sl = geometry(off, lens, slot)
            b.off[:], b.len[:], b.slot[:] = o, ln, sl
            if own:
                ctr = np.array([c.send_counter(p) for p in range(peers + 1)] + [0], np.uint64)[sl] + np.array(
                    [np.count_nonzero(sl[:i] == sl[i]) for i in range(n)], np.uint64)
                b.seal(n, F_ASSIGN_COUNTERS | F_NOTE_OUTBOUND, now)
                assert np.array_equal(b.counter[sl <= peers], ctr[sl <= peers])
            else:
                b.counter[:] = ctr
                b.seal(n)
            bad = refused[:4 if own else 5]
            good = np.ones(n, bool)
            good[bad] = False
            want = np.zeros(n, np.uint8)
            want[bad[:3]], want[bad[3]] = PKT_BAD_DESC, PKT_NO_KEYPAIR
            if not own:
                want[bad[4]] = PKT_COUNTER_EXHAUSTED
            ring, st, length = H.oracle_seal(oracle, keys, 100 + np.arange(peers), mtu, plain, off[good], lens[good], slot[good], ctr[good])
            assert (st == 0).all() and np.array_equal(b.status, want) and np.array_equal(b.out_len[good], length) and not b.out_len[bad].any()
            assert np.array_equal(b.ring, ring)  # between the messages nothing has changed either
        assert c.flows_count() == len(set(noted) - set(refused[:2]))

        # ---- opened, the slot given and looked up ----
        sealed = np.array(ring)
        back = np.flatnonzero(good)
        m = len(back)
        off, slot = off[back], slot[back]
        hurt = rng.random(m) < 0.05
        for i in np.flatnonzero(hurt):  # anywhere behind the header
            sealed[int(off[i]) + 16 + int(rng.integers(0, length[i] - 16))] ^= 1
        odd = rng.choice(np.flatnonzero(~hurt), 3, replace=False)
        sealed[off[odd[0]]] = 5              # no transport message
        length[odd[1]] = 31                  # too short for one
        for demux in (False, True):
            o = off.copy()
            o[odd[2]] += 8
            b.ring[:] = sealed
            b.off[:m], b.len[:m], b.slot[:m], b.slot[odd[1]] = o, length, slot, slot[odd[1]]
            b.open(m, F_DEMUX_INDEX if demux else 0)
            fine = np.ones(m, bool)
            fine[odd] = False
            ring, st, ctr, ln = H.oracle_open(oracle, keys, sealed, off[fine], length[fine], slot[fine])
            want = np.zeros(m, np.uint8)
            want[fine], want[odd] = st, (PKT_MALFORMED, PKT_MALFORMED, PKT_BAD_DESC)
            assert np.count_nonzero(st == PKT_AUTH_FAIL) == np.count_nonzero(hurt)
            assert np.array_equal(b.status[:m], want)
            assert np.array_equal(b.out_len[:m][fine], ln) and not b.out_len[odd].any() and np.array_equal(b.counter[:m][fine], ctr)
            if demux:
                assert np.array_equal(b.slot[:m][fine], slot[fine])
            ok = want == 0
            assert H.spans_equal(np.array(b.ring), ring, off[ok], b.out_len[:m][ok], 16) == []
            assert H.spans_differ_count(np.zeros_like(ring), np.array(b.ring), off[hurt], b.len[:m][hurt] - 32, 16) == 0  # forged: wiped
            changed = np.zeros(ring_bytes, bool)
            for x, k in zip(off[fine], length[fine]):
                changed[x + 16:x + k - 16] = True
            assert np.array_equal(np.array(b.ring)[~changed], sealed[~changed])
        b.close()


@pytest.mark.parametrize("n,size", [(4096, 1420), (9000, 64)])
def test_refused_descriptors_may_name_bytes_of_others(gpu_lib, oracle, n, size):
    """Some descriptors of a batch are placeholders that are refused, of no slot or of one without keys, and name a place at which
    another packet lies.  That packet is sealed and opened as if they were not there, whichever of the two is looked at first."""
    from bnk_b200 import Context
    from bnk_b200.device import PKT_BAD_DESC, PKT_NO_KEYPAIR

    rng = np.random.default_rng(n)
    peers, step = 5, (size + 47) // 16 * 16
    keys = rng.integers(0, 256, (peers, 32), dtype=np.uint8)
    good = rng.random(n) < 0.8
    off = np.zeros(n, np.uint32)
    off[good] = np.arange(good.sum()) * step
    # what a placeholder names: the first packet of the ring, the one behind its neighbour in front, or any
    names = rng.choice(3, n)
    behind = np.minimum(np.cumsum(good), good.sum() - 1) * step
    off[~good] = np.choose(names, [np.zeros(n), behind, rng.integers(0, good.sum(), n) * step])[~good]
    slot = np.where(good, rng.integers(0, peers, n), peers + rng.integers(0, 2, n)).astype(np.uint32)
    refused = np.where(slot == peers, PKT_NO_KEYPAIR, PKT_BAD_DESC)[~good]
    with Context(max_keypairs=peers + 1, mtu=0, flow_capacity=0) as c:
        c.set_keypairs(0, keys, keys, np.arange(peers, dtype=np.uint32))
        b = c.batch(n, int(good.sum()) * step)
        for rep in range(8):
            b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
            b.off[:], b.len[:], b.slot[:] = off, np.where(good, size, rng.choice([0, size], n)), slot
            b.counter[:] = rng.integers(0, 2**60, n, dtype=np.uint64)
            ctr = np.array(b.counter)
            ring, st, ln = H.oracle_seal(oracle, keys, np.arange(peers), 0, b.ring, off[good], b.len[good], slot[good], ctr[good])
            b.seal(n)
            assert np.array_equal(b.status[good], st) and np.array_equal(b.status[~good], refused)
            assert np.array_equal(b.out_len[good], ln) and not b.out_len[~good].any()
            assert np.array_equal(b.ring, ring), rep
            b.len[:] = step
            want, st, got, ln = H.oracle_open(oracle, keys, ring, off[good], b.len[good], slot[good])
            assert (st == 0).all()
            b.open(n)
            assert np.array_equal(b.status[good], st) and np.array_equal(b.status[~good], refused)
            assert np.array_equal(b.out_len[good], ln) and np.array_equal(b.counter[good], got)
            assert H.spans_differ_count(np.array(b.ring), want, off[good], ln, 16) == 0, rep
        b.close()


# Few and many peers: runs of a peer's packets that are longer than what the window looks back, and shorter; one cluster's work, and more
# than it takes; without the window the last checks run by themselves.
@pytest.mark.parametrize("n,peers,replay", [(5000, 7, True), (5000, 200, True), (5000, 200, False), (36_000, 300, True), (36_000, 300, False)])
def test_everything_on_behind_small_neighbours(gpu_lib, oracle, n, peers, replay):
    """Small packets that cross the link together, out of order, a few twice, a few damaged: receiver index, window, inner header, rules
    and reply flows say what the oracle says, and leave the same windows and flows behind."""
    from bnk_b200 import Context
    from bnk_b200.device import F_CHECK_INBOUND, F_DEMUX_INDEX, F_INNER_CHECK, F_REPLAY, PKT_BAD_INNER, PKT_FILTER_DENY, PKT_REPLAY
    from bnk_b200.filter import CompiledRule, PortRange, flatten_rules

    rng = np.random.default_rng(n + peers)
    keys = rng.integers(0, 256, (peers, 32), dtype=np.uint8)
    addr = RC.ip("100.64.0.0") + 16 + np.arange(peers) * 3
    rules = [("100.64.0.0/25", "udp", [(1, 20000), (40000, 50000)]), ("100.64.0.0/10", "tcp", [(22, 22), (50000, 60000)]), ("100.64.1.0/24", "icmp", [])]
    rules += [(f"100.64.{(k >> 8) & 255}.{k & 255}/32", "udp", [(20000, 30000 + k)]) for k in range(16, 16 + 3 * peers, 5)]
    # the packets, each from its peer's address but for some, and what the node has sent before
    m = n - n // 50
    slot = rng.integers(0, peers, m).astype(np.uint32)
    lens = rng.integers(28, 200, m)
    size = (lens + 47) // 16 * 16
    off = np.concatenate([[0], np.cumsum(size)])
    ring = rng.integers(0, 256, int(off[-1]), dtype=np.uint8)
    f = oracle.Filter()
    f.set_rules([([(RC.ip(s.split("/")[0]), int(s.split("/")[1]))], p, r) for s, p, r in rules])
    sent = []
    for i in range(m):
        src, sport, dport, kind = int(addr[slot[i]]), int(rng.integers(1, 9)), int(rng.integers(1, 65536)), rng.integers(0, 10)
        if rng.random() < 0.03:
            src += 1
        if kind == 0:
            p = RC.icmp_echo(src, RC.SELF, True)
        elif kind < 4 and lens[i] >= 40:
            p = RC.tcp(src, RC.SELF, sport, dport)
        else:
            p = RC.udp(src, RC.SELF, sport, dport)
        if rng.random() < 0.3:
            sent.append(RC.icmp_echo(RC.SELF, src, False) if kind == 0 else (RC.tcp if kind < 4 and lens[i] >= 40 else RC.udp)(RC.SELF, src, dport, sport))
        p = p[:2] + int(lens[i] + (rng.random() < 0.02)).to_bytes(2, "big") + p[4:]
        ring[off[i] + 16:off[i] + 16 + len(p)] = np.frombuffer(p, np.uint8)
    ctr = np.zeros(m, np.uint64)
    for p in range(peers):
        ctr[slot == p] = np.arange(np.count_nonzero(slot == p))
    sealed, st, ln = H.oracle_seal(oracle, keys, np.arange(peers), 0, ring, off[:-1], lens, slot, ctr)
    assert (st == 0).all() and np.array_equal(ln, size)
    # as they arrive
    order = np.argsort(np.arange(m) + np.where(rng.random(m) < 0.1, rng.integers(0, 300, m), 0), kind="stable")
    came = np.insert(order, rng.integers(0, m, n - m), rng.integers(0, m, n - m))
    at = np.concatenate([[0], np.cumsum(ln[came])]).astype(np.int64)
    ring = np.concatenate([sealed[off[i]:off[i] + ln[i]] for i in came])
    for i in rng.choice(n, n // 100, replace=False):
        ring[at[i] + 16 + int(rng.integers(0, ln[came[i]] - 16))] ^= 1
    off, lens, slot = at[:-1].astype(np.uint32), ln[came], slot[came]
    now = RC.T0
    plain, st, got, pt_len = H.oracle_open(oracle, keys, ring, off, lens, slot)
    want, state = H.oracle_replay(oracle, 32, slot, got, st) if replay else (st, {})
    for p in sent:
        f.note_outbound(p, now)
    for i in np.flatnonzero(want == oracle.OK):
        p = plain[off[i] + 16:off[i] + 16 + pt_len[i]].tobytes()
        total = oracle.inner_check(p, int(addr[slot[i]]))
        if total is None:
            want[i] = PKT_BAD_INNER
        else:
            pt_len[i] = total
            if not f.check_inbound(p[:total], now + RC.SEC):
                want[i] = PKT_FILTER_DENY
    with Context(max_keypairs=peers, mtu=0, flow_capacity=1 << 16, replay_ring_blocks=32) as c:
        c.set_keypairs(0, keys, keys, np.arange(peers, dtype=np.uint32))
        for p in range(peers):
            c.index_set(p, p)
            c.set_allowed_ip(p, int(addr[p]))
        c.acl_set(True, flatten_rules([CompiledRule(srcs=[s], proto=p, ports=[PortRange(*x) for x in r]) for s, p, r in rules]))
        note = c.batch(len(sent), 64 * len(sent))
        note.put_packets(sent, 64)
        note.filter_note(len(sent), now)
        b = c.batch(n, len(ring) + 64)
        b.ring[:len(ring)] = ring
        b.off[:], b.len[:], b.slot[:] = off, lens, 0xFFFFFFFF
        b.open(n, F_DEMUX_INDEX | F_INNER_CHECK | F_CHECK_INBOUND | (F_REPLAY if replay else 0), now + RC.SEC)
        assert np.array_equal(b.status, want) and np.array_equal(b.out_len, pt_len)
        for s in (0, oracle.AUTH_FAIL, PKT_BAD_INNER, PKT_FILTER_DENY) + ((PKT_REPLAY,) if replay else ()):
            assert np.count_nonzero(want == s) > 20, s
        ok = want == 0
        assert np.array_equal(b.slot, slot) and H.spans_differ_count(np.array(b.ring), plain, off[ok], pt_len[ok], 16) == 0
        for s, r in state.items():
            last, words = c.replay_export(s)
            assert last == r.last and np.array_equal(words, r.ring())
        assert H.flows_equal(c.flows_export(), f.flows())
        note.close()
        b.close()
