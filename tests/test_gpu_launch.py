"""Submits whose kernels are launched together through an executable graph (from the fourth of a kind on) do what they do
launch by launch: the same bytes, counters, verdicts and flows, in whatever order kinds and sizes come."""
import os

import numpy as np
import pytest

from tests import helpers as H
from tests import reference_cases as RC

pytestmark = pytest.mark.gpu


def _context(graphs, **kw):
    from bnk_b200 import Context

    old = os.environ.get("BNK_LAUNCH_GRAPHS")
    os.environ["BNK_LAUNCH_GRAPHS"] = str(graphs)
    try:
        return Context(**kw)
    finally:
        if old is None:
            del os.environ["BNK_LAUNCH_GRAPHS"]
        else:
            os.environ["BNK_LAUNCH_GRAPHS"] = old


def _passes(c, sizes, seed):
    """Rounds of note, seal (with flows), open (index, replay, inner header, rules), check and classify on one context."""
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_CHECK_INBOUND, F_DEMUX_INDEX, F_INNER_CHECK, F_NOTE_OUTBOUND, F_REPLAY
    from bnk_b200.filter import CompiledRule, PortRange, flatten_rules

    rng = np.random.default_rng(seed)
    peers = 7
    keys = rng.integers(0, 256, (peers, 32), dtype=np.uint8)
    c.set_keypairs(0, keys, keys, np.arange(peers, dtype=np.uint32) + 100)
    addr = [RC.ip("100.64.7.0") + p for p in range(peers)]
    for p in range(peers):
        c.index_set(100 + p, p)
        c.set_allowed_ip(p, addr[p])
        c.addr_set(bytes(10) + b"\xff\xff" + bytes([10, 0, 0, p]), 4000, p)
    c.acl_set(True, flatten_rules([CompiledRule(srcs=["100.64.7.0/30"], proto="udp", ports=[PortRange(1, 30000)])]))
    most = max(sizes)
    batches = [c.batch(most, most * 400) for _ in range(2)]
    got = []
    for r, n in enumerate(sizes):
        b, o = batches[r % 2], batches[1 - r % 2]
        now = RC.T0 + r * RC.SEC
        off = (np.arange(n, dtype=np.uint64) * 400).astype(np.uint32)
        slot = rng.integers(0, peers, n)
        lens = rng.integers(28, 340, n)
        b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
        for i in range(n):
            p = RC.udp(addr[slot[i]], RC.SELF, int(rng.integers(1, 9)), int(rng.integers(1, 60000)))[:28]
            p = p[:2] + int(lens[i]).to_bytes(2, "big") + p[4:]
            b.ring[int(off[i]) + 16:int(off[i]) + 44] = np.frombuffer(p, np.uint8)
        b.off[:n], b.len[:n], b.slot[:n] = off, lens, slot
        b.filter_note(n, now)
        b.seal(n, F_ASSIGN_COUNTERS | (F_NOTE_OUTBOUND if r % 3 else 0), now)
        got += [np.array(b.ring[:n * 400]), np.array(b.counter[:n]), np.array(b.out_len[:n]), np.array(b.status[:n])]
        o.ring[:n * 400] = b.ring[:n * 400]
        o.off[:n], o.len[:n] = off, b.out_len[:n]
        if n > 3:
            o.ring[int(off[n // 2]) + 20] ^= 1
        if r % 4 == 3 and n > 1:  # a message twice
            o.ring[:400] = o.ring[400:800]
            o.len[0] = o.len[1]
        o.open(n, F_DEMUX_INDEX | F_REPLAY | ((F_INNER_CHECK | F_CHECK_INBOUND) if r % 2 else 0), now)
        got += [np.array(o.ring[:n * 400]), np.array(o.counter[:n]), np.array(o.out_len[:n]), np.array(o.status[:n]), np.array(o.slot[:n])]
        b.len[:n] = lens
        b.src_addr[:n] = 0
        b.src_addr[:n, 10:12], b.src_addr[:n, 12], b.src_addr[:n, 15], b.src_addr[:n, 16], b.src_addr[:n, 17] = 255, 10, slot, 15, 160
        b.ring[off.astype(np.int64)] = 4
        b.slot[:n] = 99
        b.classify(n)
        got += [np.array(b.status[:n]), np.array(b.slot[:n])]
        o.len[:n] = lens
        o.filter_check(n, now)
        got.append(np.array(o.status[:n]))
    got.append(c.flows_export())
    for b in batches:
        b.close()
    return got


@pytest.mark.parametrize("sizes", [[1] * 10, [16, 17] * 6, [64, 65, 64] * 4, [160, 161] * 5, [256, 257] * 5, [700, 1025] * 5,
                                   [3, 300, 3, 3, 2000, 3, 300, 300, 3, 300, 2000, 2000, 2000, 3]], ids=str)
def test_same_results_launch_by_launch_and_through_graphs(gpu_lib, sizes):
    results = []
    for graphs in (0, 1, 1):  # the third context finds the second one's graphs gone
        with _context(graphs, max_keypairs=8, mtu=1420, flow_capacity=1 << 14) as c:
            results.append(_passes(c, sizes, len(sizes)))
            assert (c.graph_launch_count() > 0) == bool(graphs)
    for other in results[1:]:
        for x, y in zip(results[0], other):
            assert np.array_equal(x, y)


def test_batches_in_flight_and_contexts_beside_each_other(gpu_lib, oracle):
    """Graphs are shared by the contexts of a device: two contexts with up to four submits each in flight at once, sealed and
    opened, one context closed while the other's are in flight, every message and plaintext the checker's."""
    rng = np.random.default_rng(4)
    peers, n = 3, 40
    keys = [rng.integers(0, 256, (peers, 32), dtype=np.uint8) for _ in range(2)]
    off, slot = H.layout_fixed(n, 256), rng.integers(0, peers, n).astype(np.uint32)
    ridx = np.arange(peers, dtype=np.uint32) + 5
    made = [_context(1, max_keypairs=peers, flow_capacity=0) for _ in range(2)]
    batches = []
    for c, k in zip(made, keys):
        c.set_keypairs(0, k, k, ridx)
        batches.append([c.batch(n, n * 256) for _ in range(4)])
    for r in range(24):
        use = [(k, b) for k in range(len(made)) for b in batches[k][:1 + r % 4]]
        want = []
        for k, b in use:
            b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
            b.off[:], b.len[:], b.slot[:] = off, rng.integers(0, 200, n), slot
            b.counter[:] = rng.integers(0, 2**60, n, dtype=np.uint64)
            want.append((np.array(b.ring), *H.oracle_seal(oracle, keys[k], ridx, 1420, b.ring, off, b.len, slot, b.counter)))
        for k, b in use:
            b.seal(n, wait=False)
        for (k, b), (plain, ring, st, ln) in zip(use, want):
            b.wait()
            assert np.array_equal(b.status, st) and np.array_equal(b.out_len, ln)
            assert H.spans_equal(np.array(b.ring), ring, off, ln) == []
            b.len[:] = ln
        for k, b in use:
            b.open(n, wait=False)
        for i, ((k, b), (plain, ring, st, ln)) in reversed(list(enumerate(zip(use, want)))):
            b.wait()  # the second context's first
            ring, st, ctr, out = H.oracle_open(oracle, keys[k], ring, off, ln, slot)
            assert np.array_equal(b.status, st) and np.array_equal(b.counter, ctr) and np.array_equal(b.out_len, out)
            assert H.spans_equal(np.array(b.ring), ring, off, out, 16) == []
            if r == 15 and i == 4:  # four of the first context are in flight
                for x in batches.pop():
                    x.close()
                gone = made.pop()
                assert gone.graph_launch_count() > 20
                gone.close()
    assert made[0].graph_launch_count() > 50
    for b in batches[0]:
        b.close()
    made[0].close()


def test_graphs_made_while_other_threads_create_batches(gpu_lib):
    """Six threads make their batches, which synchronises the device, while the first of them already submit and their graphs
    are made; a process each time, as graphs are made once."""
    import subprocess

    from bnk_b200 import _build

    exe = _build.build_mt_stress()
    for _ in range(6):
        res = subprocess.run([exe, "6", "10", "128", "1420", "4"], capture_output=True, text=True, timeout=120)
        assert res.returncode == 0 and res.stdout.startswith("OK"), (res.returncode, res.stdout[-500:] + res.stderr[-2000:])
