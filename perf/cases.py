"""The work a user of this library has it do, as cases that can be timed and compared.

A VPN node's packets are in host memory: they come from a TUN device or a socket and go back there.  So every case
takes its packets from the batch's pinned ring (or from the caller's own buffers, for the queue and the dispatcher)
through the whole call and finds the results in host memory; only the rule check of very many headers is also run on
headers that already are on the device.  The calls are those of include/bnk_gpu.h, made through this package's
handles (Context, Batch) or, for the queue and the dispatcher, through the C ABI's binding itself.

Kinds of work, each over its range of sizes (see `draw`):

  seal      bnk_seal_submit on a ring of packets, nonces from the send counters; sealing works in place, so what a
            pass leaves in the ring is the next pass's payload
  tunnel    the data path of a node with everything on: outbound flows noted, counters, seal; the messages cross to
            the receiving ring out of order, a few twice, a few damaged; receiver index, open, replay window, inner
            header, inbound filter
  queue     several callers' batches outstanding on a seal queue and an open queue, caller-owned buffers
  dispatch  one large mixed batch in the caller's buffers through the multi-GPU dispatcher, sealed and opened
  gso       TCP / UDP super-packets split, noted and sealed on the device
  check     the ACL check of IP headers against a large rule table and a large flow table
  filter    what filteredTUN.Read and Write do: flows of whole packets noted, whole packets checked
  classify  datagrams told apart: disco, STUN, known peer, stranger
"""
import ctypes as C

import numpy as np

from bnk_b200 import Context, _lib, gen, slot_size
from bnk_b200.device import (ACL_TUPLE_DTYPE, F_ASSIGN_COUNTERS, F_CHECK_INBOUND, F_DEMUX_INDEX, F_INNER_CHECK, F_NO_H2D,
                             F_NOTE_OUTBOUND, F_REPLAY, F_SORT_BY_LENGTH, GSO_SUPER_DTYPE)

MTU = 1420
IMIX = (64, 576, 1420)  # at 7:4:1
MS = 1_000_000          # every pass happens a millisecond after the one before, as a clock has it
T0 = 1_700_000_000 * 10**9
NET = gen.ip4(100, 64, 0, 0)
SELF = gen.ip4(100, 64, 0, 1)


def listed():
    return [
        # a few small packets, as an interactive session or a handful of acknowledgements has them: the smallest call
        {"name": "seal_few", "kind": "seal", "n": 5, "size": 92, "peers": 3},
        # one tun.Device.Read of the upstream batch size, one busy peer, full-size packets
        {"name": "seal_read", "kind": "seal", "n": 128, "size": 1420, "peers": 1},
        # a bulk sender's ring: many peers, 186 MB each way
        {"name": "seal_ring", "kind": "seal", "n": 131072, "size": 1420, "peers": 8192},
        # the whole data path for the odd few packets of a quiet node
        {"name": "tunnel_few", "kind": "tunnel", "n": 9, "size": 300, "peers": 4, "rules": 40},
        # the whole data path for one upstream batch of full-size packets
        {"name": "tunnel_read", "kind": "tunnel", "n": 128, "size": 1420, "peers": 20, "rules": 500},
        # a hub's receive burst: 64/576/1420 bytes at 7:4:1, 256 peers, reordered, 1 % twice, 1 % damaged
        {"name": "tunnel_mix", "kind": "tunnel", "n": 4096, "size": 0, "peers": 256, "rules": 2000},
        # eight workers' upstream batches outstanding at once on a shared queue per direction
        {"name": "queue_8x128", "kind": "queue", "calls": 8, "n": 128, "size": 1420, "peers": 64},
        # a relay that gathers large batches in buffers of its own
        {"name": "dispatch", "kind": "dispatch", "n": 24576, "size": 1420, "peers": 256},
        # bulk TCP out of a host with segmentation offload: 64 KB super-packets, popular and rare peers
        {"name": "gso_tcp", "kind": "gso", "supers": 256, "segs": 47, "mss": 1380, "udp": False, "peers": 1000},
        # a large policy: 10,000 rules, 300,000 flows, a million headers on the device
        {"name": "check_headers", "kind": "check", "n": 1_000_000, "rules": 10_000, "nodes": 50_000, "flows": 300_000,
         "resident": True},
        # the TUN wrapper alone, on whole packets of mixed size
        {"name": "filter_packets", "kind": "filter", "n": 8192, "size": 0, "rules": 2000, "nodes": 5000},
        # a burst of received datagrams before any key is looked at
        {"name": "classify_burst", "kind": "classify", "n": 4096, "size": 0, "peers": 500},
    ]


def draw(rng):
    def span(lo, hi):  # spread over the logarithm
        return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))

    def size():
        return rng.choice([0, 1420, rng.randint(28, 1420)])

    kind = rng.choice(["seal", "seal", "tunnel", "tunnel", "queue", "dispatch", "gso", "check", "filter", "classify"])
    c = {"kind": kind}
    if kind == "seal":
        c.update(n=span(1, 120_000), size=size())
        c["peers"] = span(1, max(2, c["n"] // 4))
    elif kind == "tunnel":
        c.update(n=span(1, 16_384), size=size(), rules=span(10, 4000))
        c["peers"] = span(1, max(2, min(1000, c["n"] // 2)))
    elif kind == "queue":
        c.update(calls=rng.randint(1, 16), n=span(16, 256), size=size(), peers=span(2, 200))
    elif kind == "dispatch":
        c.update(n=span(200, 24_000), size=size(), peers=span(2, 400))
    elif kind == "gso":
        c.update(supers=span(1, 400), segs=rng.randint(2, 44), mss=rng.randint(536, 1380), udp=rng.random() < 0.3,
                 peers=span(1, 2000))
    elif kind == "check":
        c.update(n=span(1000, 900_000), rules=span(20, 10_000), nodes=span(100, 50_000), flows=span(100, 250_000),
                 resident=rng.random() < 0.5)
    elif kind == "filter":
        c.update(n=span(1, 16_384), size=size(), rules=span(10, 4000), nodes=span(20, 10_000))
    else:
        c.update(n=span(1, 50_000), size=size(), peers=span(2, 1000))
    return c


# ---------------------------------------------------------------------------------------
# what the cases share
# ---------------------------------------------------------------------------------------
class State:
    """What a program keeps between calls; closes its handles when it goes."""

    def __init__(self, *handles):
        self.handles = list(handles)

    def __del__(self):
        for h in self.handles:
            h.close()


class Handle:
    """A queue or dispatcher of the C ABI."""

    def __init__(self, ptr, destroy):
        self.ptr, self.destroy = ptr, destroy

    def close(self):
        if self.ptr:
            self.destroy(self.ptr)
            self.ptr = None


class Result(dict):
    """A pass's outputs by name.  They are views of the state's pinned memory, so the state lives as long as they do."""

    def __init__(self, state, arrays):
        super().__init__(arrays)
        self.state = state


def generator(seed):
    return np.random.Generator(np.random.PCG64(seed))


def random_bytes(g, n):
    return g.integers(0, 1 << 64, (n + 7) // 8, dtype=np.uint64).view(np.uint8)[:n]


def lengths(g, n, size):
    """Packet lengths: all of one size, or the 7:4:1 mix in random order."""
    if size:
        return np.full(n, size, np.uint32)
    return g.permutation(np.repeat(np.asarray(IMIX, np.uint32), (7, 4, 1))[np.arange(n) * 7 % 12])


def mean_length(size):
    return size if size else (7 * IMIX[0] + 4 * IMIX[1] + IMIX[2]) / 12


def pack(lens):
    """Offsets of packets laid back to back with room for header, padding and tag; the ring's length behind them."""
    end = np.cumsum((lens.astype(np.int64) + 48 + 15) & ~15)
    return np.concatenate([[0], end[:-1]]).astype(np.uint32), int(end[-1])


def headers(g, src, dst, sport, dport, proto, lens):
    """The first 28 bytes of IPv4 packets (TCP, UDP or ICMP)."""
    n = len(lens)
    h = np.zeros((n, 28), np.uint8)
    h[:, 0] = 0x45
    h[:, 2], h[:, 3] = lens >> 8, lens & 0xFF
    h[:, 8] = 64
    h[:, 9] = proto
    h[:, 12:16] = np.asarray(src, ">u4").reshape(-1, 1).view(np.uint8)
    h[:, 16:20] = np.asarray(dst, ">u4").reshape(-1, 1).view(np.uint8)
    h[:, 20:22] = np.asarray(sport, ">u2").reshape(-1, 1).view(np.uint8)
    h[:, 22:24] = np.asarray(dport, ">u2").reshape(-1, 1).view(np.uint8)
    h[proto == 1, 20:24] = (8, 0, 0, 0)
    return h


def put_headers(ring, off, h):
    ring[off.astype(np.int64)[:, None] + 16 + np.arange(h.shape[1])] = h


def protocols(g, n):
    return np.asarray((6, 17, 1), np.uint8)[g.choice(3, n, p=(0.6, 0.3, 0.1))]


def ports(g, n):
    return g.integers(1, 65536, n).astype(np.uint16)


def rule_table(g, rules, nodes):
    """Allowances of `rules` rules: mostly a few /32 sources and a port range each, one rule in a hundred a prefix."""
    per = np.minimum(64, g.geometric(0.25, rules))
    prefix = g.random(rules) < 0.01
    per[prefix] = 1
    of = np.repeat(np.arange(rules), per)
    proto, a, b = protocols(g, rules), ports(g, rules), ports(g, rules)
    b = np.where(g.random(rules) < 0.1, a, b)
    bits = np.where(prefix, g.integers(16, 25, rules), 32)
    t = np.zeros(len(of), ACL_TUPLE_DTYPE)
    t["addr"] = nodes[g.integers(0, len(nodes), len(of))] & ((0xFFFFFFFF << (32 - bits[of])) & 0xFFFFFFFF)
    t["prefix_len"], t["proto"] = bits[of], proto[of]
    icmp = proto[of] == 1
    t["port_first"] = np.where(icmp, 0, np.minimum(a, b)[of])
    t["port_last"] = np.where(icmp, 0, np.maximum(a, b)[of])
    return t


def node_addresses(g, n):
    return (NET + 256 + g.choice(1 << 21, n, replace=False)).astype(np.int64)


def note_flows(batch, ctx_now, src, dst, sport, dport, proto):
    """Opens outbound flows through a batch, as many at a time as it holds."""
    h = headers(None, src, dst, sport, dport, proto, np.full(len(proto), 28))
    room = min(batch.max_pkts, batch.ring_bytes // 48)
    for at in range(0, len(h), room):
        k = min(room, len(h) - at)
        batch.ring[:k * 48].reshape(k, 48)[:, 16:44] = h[at:at + k]
        batch.off[:k] = np.arange(k, dtype=np.uint32) * 48
        batch.len[:k] = 28
        batch.filter_note(k, ctx_now)
    batch.ring[:] = 0


def inbound(g, n, nodes, lens, flows):
    """Headers of received packets: 30 % replies to `flows` (src, dst, sport, dport, proto of the outbound packets), the
    rest fresh traffic from the nodes, one in twenty of those with a broken header."""
    src, proto, sport, dport = nodes[g.integers(0, len(nodes), n)], protocols(g, n), ports(g, n), ports(g, n)
    reply = g.random(n) < 0.3
    pick = g.integers(0, len(flows[0]), n)
    f_src, f_dst, f_sport, f_dport, f_proto = (f[pick] for f in flows)
    h = headers(g, np.where(reply, f_dst, src), np.where(reply, f_src, SELF), np.where(reply, f_dport, sport),
                np.where(reply, f_sport, dport), np.where(reply, f_proto, proto).astype(np.uint8), lens)
    bad = ~reply & (g.random(n) < 0.05)
    h[bad, 0] = np.asarray((0x65, 0x44, 0x45), np.uint8)[g.integers(0, 3, int(bad.sum()))]
    h[bad & (h[:, 0] == 0x45), 9] = 47
    return h


def new_flows(g, n, nodes):
    return (np.full(n, SELF), nodes[g.integers(0, len(nodes), n)], ports(g, n), ports(g, n), protocols(g, n))


# ---------------------------------------------------------------------------------------
# seal
# ---------------------------------------------------------------------------------------
def prepare_seal(case, g):
    n, peers = case["n"], case["peers"]
    lens = lengths(g, n, case["size"])
    off, ext = pack(lens)
    ctx = Context(max_keypairs=peers, mtu=MTU)
    s = State(ctx)
    keys = random_bytes(g, peers * 32)
    ctx.set_keypairs(0, keys, keys, g.integers(0, 1 << 32, peers, dtype=np.uint32))
    b = s.b = ctx.batch(n, ext)
    b.ring[:] = random_bytes(g, ext)
    b.off[:], b.len[:] = off, lens
    b.slot[:] = g.integers(0, peers, n)
    s.n, s.flags = n, F_ASSIGN_COUNTERS | (0 if case["size"] or n < 1024 else F_SORT_BY_LENGTH)
    s.out = {"ring": b.ring, "counter": b.counter.view(np.int64), "out_len": b.out_len, "status": b.status}
    return s


def run_seal(s):
    s.b.seal(s.n, s.flags)
    return Result(s, s.out)


# ---------------------------------------------------------------------------------------
# tunnel
# ---------------------------------------------------------------------------------------
def prepare_tunnel(case, g):
    n, peers = case["n"], case["peers"]
    lens = lengths(g, n, case["size"])
    off, ext = pack(lens)
    padded = np.minimum((lens.astype(np.int64) + 15) & ~15, MTU)
    slot = g.integers(0, peers, n).astype(np.uint32)
    # arrival order: one in twenty changes places with one up to 64 later; one in a hundred arrives once more
    order = np.arange(n)
    for p in g.integers(0, n, n // 20):
        q = min(n - 1, int(p) + 1 + int(g.integers(0, 64)))
        order[[p, q]] = order[[q, p]]
    twice = g.choice(n, n // 100, replace=False)
    twice_off = np.arange(len(twice), dtype=np.uint32) * np.uint32(slot_size(MTU))
    twice_ext = len(twice) * slot_size(MTU)
    came = np.concatenate([order, twice])
    where = np.argsort(np.concatenate([np.arange(n) * 2.0, np.argsort(order)[twice] * 2.0 + 61]), kind="stable")

    ctx = Context(max_keypairs=peers, mtu=MTU, flow_capacity=1 << 16)
    s = State(ctx)
    nodes = node_addresses(g, peers)
    keys = random_bytes(g, peers * 32)
    local = g.choice(1 << 31, peers, replace=False).astype(np.uint32)
    ctx.set_keypairs(0, keys, keys, local)  # the node's own messages come back to it: one index, one key per peer
    for p in range(peers):
        ctx.index_set(int(local[p]), p)
        ctx.set_allowed_ip(p, int(nodes[p]))
    ctx.acl_set(True, rule_table(g, case["rules"], nodes))
    m = len(came)
    s.tx, s.rx = (ctx.batch(m, ext + twice_ext) for _ in range(2))
    flows = new_flows(g, max(1, n // 3), nodes)
    note_flows(s.tx, T0, *flows)
    # a reply is a packet that a peer sends from its own address: of the flow that this node opened towards it
    h = headers(g, nodes[slot], np.full(n, SELF), ports(g, n), ports(g, n), protocols(g, n), lens)
    of_peer = {int(a): k for k, a in enumerate(flows[1])}
    for i in np.flatnonzero(g.random(n) < 0.3):
        k = of_peer.get(int(nodes[slot[i]]))
        if k is not None:
            h[i, 9] = flows[4][k]
            h[i, 20:22] = np.asarray([flows[3][k]], ">u2").view(np.uint8)
            h[i, 22:24] = np.asarray([flows[2][k]], ">u2").view(np.uint8)
    s.tx.ring[:ext] = random_bytes(g, ext)
    put_headers(s.tx.ring, off, h)
    s.n, s.m, s.ext, s.now = n, m, ext, T0
    s.off, s.len, s.slot = off, lens, slot
    s.came_from = came[where]
    s.came_off = np.concatenate([off[order], twice_off + np.uint32(ext)])[where].astype(np.uint32)
    s.twice = [(int(off[i]), int(o) + ext, int(padded[i]) + 32) for i, o in zip(twice, twice_off)]
    hurt = g.choice(n, n // 100, replace=False)
    s.hurt = off[hurt].astype(np.int64) + 16 + padded[hurt] + g.integers(0, 16, len(hurt))
    sort = 0 if case["size"] or n < 1024 else F_SORT_BY_LENGTH
    s.tx_flags = F_NOTE_OUTBOUND | F_ASSIGN_COUNTERS | sort
    s.rx_flags = F_DEMUX_INDEX | F_REPLAY | F_INNER_CHECK | F_CHECK_INBOUND | sort
    return s


def run_tunnel(s):
    tx, rx, n, m = s.tx, s.rx, s.n, s.m
    s.now += MS
    tx.off[:n], tx.len[:n], tx.slot[:n] = s.off, s.len, s.slot
    tx.seal(n, s.tx_flags, s.now)
    rx.ring[:s.ext] = tx.ring[:s.ext]  # the network
    for src, dst, k in s.twice:
        rx.ring[dst:dst + k] = tx.ring[src:src + k]
    if len(s.hurt):
        rx.ring[s.hurt] ^= 1
    rx.off[:], rx.len[:] = s.came_off, tx.out_len[s.came_from]
    rx.open(m, s.rx_flags, s.now)
    s.tx, s.rx = rx, tx  # what was received goes out with the next pass
    return Result(s, {"sealed": tx.ring, "counter": tx.counter[:n].view(np.int64), "sealed_len": tx.out_len[:n],
                      "seal_status": tx.status[:n], "opened": rx.ring, "opened_counter": rx.counter.view(np.int64),
                      "opened_len": rx.out_len, "open_status": rx.status, "slot": rx.slot})


# ---------------------------------------------------------------------------------------
# queue and dispatcher: caller-owned (pageable) buffers
# ---------------------------------------------------------------------------------------
def pointers(buf, offsets):
    return (np.uint64(buf.ctypes.data) + offsets.astype(np.uint64)).astype(np.uint64)


class Buffers:
    """Packets, messages and plaintexts in memory of the caller's own, with the arrays a call wants."""

    def __init__(self, g, n, size, peers):
        self.n = n
        self.len = lengths(g, n, size)
        step = np.arange(n, dtype=np.uint64) * np.uint64(MTU + 64)
        self.packets = random_bytes(g, n * (MTU + 64)).copy()
        self.sealed, self.opened = np.zeros_like(self.packets), np.zeros_like(self.packets)
        self.peer = g.integers(0, peers, n).astype(np.uint32)
        self.p_packets, self.p_sealed, self.p_opened = (pointers(b, step) for b in (self.packets, self.sealed, self.opened))
        self.sealed_len, self.opened_len = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
        self.seal_status, self.open_status = np.zeros(n, np.uint8), np.zeros(n, np.uint8)
        self.counter, self.opened_counter = np.zeros(n, np.uint64), np.zeros(n, np.uint64)
        self.opened_peer = np.zeros(n, np.uint32)

    def outputs(self):
        return [self.sealed, self.sealed_len, self.seal_status, self.counter.view(np.int64), self.opened, self.opened_len,
                self.open_status, self.opened_peer]


def prepare_queue(case, g):
    calls, n, peers = case["calls"], case["n"], case["peers"]
    L = _lib.lib()
    ctx = Context(max_keypairs=peers, mtu=MTU)
    keys = random_bytes(g, peers * 32)
    local = g.choice(1 << 31, peers, replace=False).astype(np.uint32)
    ctx.set_keypairs(0, keys, keys, local)
    for p in range(peers):
        ctx.index_set(int(local[p]), p)
    queues = []
    for open_side, flags in ((0, 0), (1, F_DEMUX_INDEX | F_REPLAY)):
        cfg = _lib.QueueCfg(C.sizeof(_lib.QueueCfg), 1024, MTU, 3, open_side, flags, 0, 0)
        q = C.c_void_p()
        _lib.check(L.bnk_queue_create(ctx._h, C.byref(cfg), C.byref(q)))
        queues.append(Handle(q, L.bnk_queue_destroy))
    s = State(*queues, ctx)
    s.L, s.q_seal, s.q_open = L, queues[0].ptr, queues[1].ptr
    s.all = Buffers(g, calls * n, case["size"], peers)
    s.calls = [slice(k * n, (k + 1) * n) for k in range(calls)]
    s.n = n
    a = s.all
    address = lambda v, k: v[s.calls[k]].ctypes.data  # noqa: E731 - the caller's arrays stay where they are
    s.seal_in = [[address(v, k) for v in (a.p_packets, a.len, a.peer)] for k in range(calls)]
    s.seal_out = [[address(v, k) for v in (a.p_sealed, a.sealed_len, a.counter)] + [None, address(a.seal_status, k)]
                  for k in range(calls)]
    s.open_in = [[address(v, k) for v in (a.p_sealed, a.sealed_len)] + [None] for k in range(calls)]
    s.open_out = [[address(v, k) for v in (a.p_opened, a.opened_len, a.opened_counter, a.opened_peer, a.open_status)]
                  for k in range(calls)]
    s.out = dict(enumerate(a.outputs()))
    return s


def through_queue(L, q, n, ins, outs):
    """Hands every caller's batch in and collects it; a queue that has no room is given it by collecting the oldest."""
    tickets, done = [], 0
    for args in ins:
        t = C.c_uint64()
        while (rc := L.bnk_queue_submit(q, *args, n, 0, C.byref(t))) == _lib.EBUSY:
            _lib.check(L.bnk_queue_wait(q, tickets[done], *outs[done]))
            done += 1
        _lib.check(rc)
        tickets.append(t)
    for k in range(done, len(tickets)):
        _lib.check(L.bnk_queue_wait(q, tickets[k], *outs[k]))


def run_queue(s):
    through_queue(s.L, s.q_seal, s.n, s.seal_in, s.seal_out)
    through_queue(s.L, s.q_open, s.n, s.open_in, s.open_out)
    return Result(s, s.out)


def prepare_dispatch(case, g):
    n, peers = case["n"], case["peers"]
    L = _lib.lib()
    devices = (C.c_int32 * 1)(0)
    per_gpu = _lib.Cfg(C.sizeof(_lib.Cfg), 0, peers, 128, MTU, 1 << 16, 0, 0)
    cfg = _lib.MgpuCfg(C.sizeof(_lib.MgpuCfg), 1, devices, 32768, MTU, peers, 0, per_gpu)
    m = C.c_void_p()
    _lib.check(L.bnk_mgpu_create(C.byref(cfg), C.byref(m)))
    s = State(Handle(m, L.bnk_mgpu_destroy))
    keys = random_bytes(g, peers * 32).reshape(peers, 32)
    local = g.choice(1 << 31, peers, replace=False)
    for p in range(peers):
        key = keys[p].ctypes.data
        _lib.check(L.bnk_mgpu_peer_set(m, p, key, key, int(local[p]), int(local[p]), 0))
    s.L, s.m, s.n = L, m, n
    a = s.all = Buffers(g, n, case["size"], peers)
    s.seal_args = [v.ctypes.data for v in (a.p_packets, a.len, a.peer)] + [n, 0, 0] + [
        v.ctypes.data for v in (a.p_sealed, a.sealed_len, a.counter, a.seal_status)]
    s.open_args = [v.ctypes.data for v in (a.p_sealed, a.sealed_len)] + [n, F_REPLAY, 0] + [
        v.ctypes.data for v in (a.p_opened, a.opened_len, a.opened_counter, a.opened_peer, a.open_status)]
    s.out = dict(enumerate(a.outputs()))
    return s


def run_dispatch(s):
    _lib.check(s.L.bnk_mgpu_seal(s.m, *s.seal_args))
    _lib.check(s.L.bnk_mgpu_open(s.m, *s.open_args))
    return Result(s, s.out)


# ---------------------------------------------------------------------------------------
# segmentation offload
# ---------------------------------------------------------------------------------------
def prepare_gso(case, g):
    n_super, segs, mss, udp, peers = case["supers"], case["segs"], case["mss"], case["udp"], case["peers"]
    hdr = 28 if udp else 40
    n = n_super * segs
    # the last segment of a super-packet is what is left over
    left = g.integers(1, mss + 1, n_super)
    payload = (segs - 1) * mss + left
    lens = np.full((n_super, segs), hdr + mss, np.uint32)
    lens[:, -1] = hdr + left
    lens = lens.reshape(-1)
    stride = slot_size(hdr + mss)
    off = (np.arange(n, dtype=np.int64) * stride).astype(np.uint32)
    room = (hdr + segs * mss + 15) & ~15
    ctx = Context(max_keypairs=peers, mtu=MTU, flow_capacity=1 << 16)
    s = State(ctx)
    nodes = node_addresses(g, peers)
    keys = random_bytes(g, peers * 32)
    ctx.set_keypairs(0, keys, keys, g.integers(0, 1 << 32, peers, dtype=np.uint32))
    ctx.acl_set(True, rule_table(g, 200, nodes))
    b = s.b = ctx.batch(n, n * stride + n_super * room)
    peer = gen.zipf_ranks(gen.SplitMix64(int(g.integers(0, 1 << 63))), n_super, peers)
    h = np.zeros((n_super, 40), np.uint8)
    h[:, :28] = headers(g, np.full(n_super, SELF), nodes[peer], ports(g, n_super), ports(g, n_super),
                        np.full(n_super, 17 if udp else 6, np.uint8), np.minimum(hdr + payload, 65535))
    h[:, 4:6] = g.integers(0, 256, (n_super, 2))
    if not udp:
        h[:, 24:32] = g.integers(0, 256, (n_super, 8))
        h[:, 32], h[:, 33] = 5 << 4, 0x18
    sup = s.supers = np.zeros(n_super, GSO_SUPER_DTYPE)
    at = n * stride + np.arange(n_super, dtype=np.int64) * room
    area = b.ring[n * stride:].reshape(n_super, room)
    area[:] = random_bytes(g, n_super * room).reshape(n_super, room)
    area[:, :hdr] = h[:, :hdr]
    sup["src_off"], sup["src_len"] = at, hdr + payload
    sup["first_pkt"], sup["n_pkts"] = np.arange(n_super) * segs, segs
    sup["hdr_len"], sup["gso_size"], sup["csum_start"] = hdr, mss, 20
    sup["csum_offset"], sup["proto"] = (6, 17) if udp else (16, 6)
    b.off[:], b.len[:], b.slot[:] = off, lens, np.repeat(peer, segs)
    s.n, s.now = n, T0
    s.out = {"ring": b.ring[:n * stride], "counter": b.counter.view(np.int64), "out_len": b.out_len, "status": b.status}
    return s


def run_gso(s):
    s.now += MS
    s.b.gso_split(s.supers, s.n)
    s.b.seal(s.n, F_NO_H2D | F_NOTE_OUTBOUND | F_ASSIGN_COUNTERS, s.now)
    return Result(s, s.out)


# ---------------------------------------------------------------------------------------
# packet filter, classification
# ---------------------------------------------------------------------------------------
def prepare_check(case, g):
    n, stride = case["n"], 48
    ctx = Context(max_keypairs=1, flow_capacity=1 << 20)
    s = State(ctx)
    nodes = node_addresses(g, case["nodes"])
    ctx.acl_set(True, rule_table(g, case["rules"], nodes))
    b = s.b = ctx.batch(n, n * stride)
    flows = new_flows(g, case["flows"], nodes)
    note_flows(b, T0, *flows)
    b.ring.reshape(n, stride)[:, 16:44] = inbound(g, n, nodes, np.full(n, 28), flows)
    b.off[:] = np.arange(n, dtype=np.uint32) * stride
    b.len[:] = np.where(g.random(n) < 0.01, 22, 28)
    s.n, s.now, s.flags = n, T0, 0
    if case["resident"]:
        b.upload(n)
        s.flags = F_NO_H2D
    return s


def run_check(s):
    s.now += MS
    s.b.filter_check(s.n, s.now, s.flags)
    return Result(s, {"status": s.b.status})


def prepare_filter(case, g):
    n = case["n"]
    ctx = Context(max_keypairs=1, flow_capacity=1 << 17)
    s = State(ctx)
    nodes = node_addresses(g, case["nodes"])
    ctx.acl_set(True, rule_table(g, case["rules"], nodes))
    flows = new_flows(g, n, nodes)
    for name in ("out", "into"):
        lens = lengths(g, n, case["size"])
        off, ext = pack(lens)
        b = ctx.batch(n, ext)
        b.ring[:] = random_bytes(g, ext)
        put_headers(b.ring, off, headers(g, *flows, lens) if name == "out" else inbound(g, n, nodes, lens, flows))
        b.off[:], b.len[:] = off, lens
        setattr(s, name, b)
    s.n, s.now = n, T0
    return s


def run_filter(s):
    s.now += MS
    s.out.filter_note(s.n, s.now)
    s.into.filter_check(s.n, s.now)
    return Result(s, {"status": s.into.status})


def prepare_classify(case, g):
    n, peers = case["n"], case["peers"]
    lens = lengths(g, n, case["size"]) + np.uint32(32)
    off, ext = pack(lens)
    ctx = Context(max_keypairs=max(peers, 8), mtu=MTU)
    s = State(ctx)
    addr = np.zeros((peers, 16), np.uint8)
    addr[:, 10:12] = 255
    addr[:, 12:] = random_bytes(g, peers * 4).reshape(peers, 4)
    port = ports(g, peers)
    for p in range(peers):
        ctx.addr_set(addr[p].tobytes(), int(port[p]), p)
    b = s.b = ctx.batch(n, ext)
    b.ring[:] = random_bytes(g, ext)
    o = off.astype(np.int64)
    what = g.random(n)
    start = np.zeros((n, 16), np.uint8)  # mostly transport messages
    start[:, 0] = 4
    start[:, 4:] = random_bytes(g, n * 12).reshape(n, 12)
    start[what < 0.02, :10] = np.frombuffer(b"bnk\0disco\0", np.uint8)
    stun = (what >= 0.02) & (what < 0.03)
    start[stun, :8] = (0, 1, 0, 0, 0x21, 0x12, 0xA4, 0x42)
    b.ring[o[:, None] + np.arange(16)] = start
    b.off[:], b.len[:] = off, lens
    who = g.integers(0, peers, n)
    b.src_addr[:, :16] = addr[who]
    b.src_addr[:, 16:18] = np.asarray(port[who], ">u2").reshape(-1, 1).view(np.uint8)
    b.src_addr[what > 0.97, 12:16] ^= 0x5A  # strangers
    s.n = n
    s.out = {"status": b.status, "slot": b.slot}
    return s


def run_classify(s):
    s.b.classify(s.n)
    return Result(s, s.out)


PREPARE = {"seal": prepare_seal, "tunnel": prepare_tunnel, "queue": prepare_queue, "dispatch": prepare_dispatch,
           "gso": prepare_gso, "check": prepare_check, "filter": prepare_filter, "classify": prepare_classify}
RUN = {"seal": run_seal, "tunnel": run_tunnel, "queue": run_queue, "dispatch": run_dispatch, "gso": run_gso,
       "check": run_check, "filter": run_filter, "classify": run_classify}


def prepare(case, seed):
    s = PREPARE[case["kind"]](case, generator(seed))
    s.run = RUN[case["kind"]]
    return s


def run(state):
    return state.run(state)


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def cipher_ops(length):
    """32-bit integer operations of ChaCha20-Poly1305 on one packet: 992 a cipher block (one more for the one-time key),
    40 a Poly1305 block (one more for the lengths)."""
    return (-(-length // 64) + 1) * 992 + (-(-length // 16) + 1) * 40


def mean_ops(size):
    if size:
        return cipher_ops(size)
    return (7 * cipher_ops(IMIX[0]) + 4 * cipher_ops(IMIX[1]) + cipher_ops(IMIX[2])) / 12


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    length = mean_length(case.get("size", 0))
    way = 2 * length + 32 + 25  # payload, message, descriptors and results of a packet sealed or opened
    if kind == "seal":
        return {"bytes": n * way, "flops": n * mean_ops(case["size"])}
    if kind in ("tunnel", "dispatch"):
        return {"bytes": 2 * n * way, "flops": 2 * n * mean_ops(case["size"])}
    if kind == "queue":
        k = n * case["calls"]
        return {"bytes": 2 * k * way, "flops": 2 * k * mean_ops(case["size"])}
    if kind == "gso":
        segs = case["supers"] * case["segs"]
        return {"bytes": segs * (2 * case["mss"] + 40 + 32 + 25), "flops": segs * cipher_ops(case["mss"] + 40)}
    if kind == "check":
        return {"bytes": n * (28 + 8 + 1), "flops": 0}
    if kind == "filter":
        return {"bytes": 2 * n * (28 + 8) + n, "flops": 0}
    return {"bytes": n * (20 + 20 + 8 + 5), "flops": 0}  # classify


def tolerance(case):
    return "exact"
