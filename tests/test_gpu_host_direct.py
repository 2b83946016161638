"""Batches run on the caller's pinned buffers (no copies) or through the copy engines.  Both
ways must give the same bytes, and a batch that ran without copies must still chain into device-resident calls."""
import os

import numpy as np
import pytest

from tests import helpers as H
from tests import reference_cases as RC

pytestmark = pytest.mark.gpu


def _context(direct_bytes, **kw):
    from bnk_b200 import Context

    old = os.environ.get("BNK_HOST_DIRECT_BYTES")
    os.environ["BNK_HOST_DIRECT_BYTES"] = str(direct_bytes)
    try:
        return Context(**kw)
    finally:
        if old is None:
            del os.environ["BNK_HOST_DIRECT_BYTES"]
        else:
            os.environ["BNK_HOST_DIRECT_BYTES"] = old


def _load(b, rng, n, n_peers):
    sizes = rng.choice([0, 1, 40, 576, 1300, 1420], n)
    off = (np.arange(n, dtype=np.uint64) * 1472).astype(np.uint32)
    for i in range(n):
        b.ring[int(off[i]) + 16:int(off[i]) + 16 + int(sizes[i])] = rng.integers(0, 256, int(sizes[i]), dtype=np.uint8)
    b.off[:n], b.len[:n] = off, sizes
    b.slot[:n] = rng.integers(0, n_peers, n)
    return off, sizes


@pytest.mark.parametrize("n", [1, 7, 64, 200, 256, 300])  # 300: more than go along with a launch
def test_same_bytes_with_and_without_copies(gpu_lib, oracle, n):
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_REPLAY

    n_peers = 9
    keys = np.random.default_rng(5).integers(0, 256, (n_peers, 32), dtype=np.uint8)
    results = []
    for direct_bytes in (0, 1 << 20):  # never / for everything this test sends
        rng = np.random.default_rng(77 + n)
        c = _context(direct_bytes, max_keypairs=n_peers, mtu=1420, flow_capacity=0)
        try:
            c.set_keypairs(0, keys, keys, np.arange(n_peers, dtype=np.uint32))
            b = c.batch(n, n * 1472)
            _load(b, rng, n, n_peers)
            plain = np.array(b.ring)
            b.seal(n, F_ASSIGN_COUNTERS)
            sealed = (np.array(b.ring), np.array(b.out_len[:n]), np.array(b.counter[:n]), np.array(b.status[:n]))
            # twice through open: the second time every packet is a replay
            b.len[:n] = b.out_len[:n]
            b.open(n, F_REPLAY)
            opened = (np.array(b.ring), np.array(b.out_len[:n]), np.array(b.status[:n]))
            b.ring[:] = sealed[0]
            b.open(n, F_REPLAY)
            again = np.array(b.status[:n])
            b.close()
            results.append((plain, sealed, opened, again))
        finally:
            c.close()
    (plain0, sealed0, opened0, again0), (plain1, sealed1, opened1, again1) = results
    assert np.array_equal(plain0, plain1)
    for x, y in zip(sealed0 + opened0, sealed1 + opened1):
        assert np.array_equal(x, y)
    assert (sealed0[3] == oracle.OK).all()
    assert set(np.unique(opened0[2])) <= {oracle.OK, oracle.KEEPALIVE}
    assert (again0 == oracle.REPLAY).all() and (again1 == oracle.REPLAY).all()
    # and the plaintext came back
    off = (np.arange(n, dtype=np.uint64) * 1472).astype(np.int64)
    rng = np.random.default_rng(77 + n)
    sizes = rng.choice([0, 1, 40, 576, 1300, 1420], n)
    for i in range(n):
        o, l = int(off[i]) + 16, int(sizes[i])
        assert np.array_equal(opened1[0][o:o + l], plain1[o:o + l]), i


def test_device_resident_call_after_a_batch_without_copies(gpu_lib, oracle):
    """seal without copies leaves the device ring behind; a following open that asks for no upload must still
    see the sealed bytes, and a download must not bring stale device bytes over the results."""
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_NO_D2H, F_NO_H2D

    n, n_peers = 48, 5
    rng = np.random.default_rng(9)
    keys = rng.integers(0, 256, (n_peers, 32), dtype=np.uint8)
    c = _context(1 << 20, max_keypairs=n_peers, mtu=1420, flow_capacity=0)
    try:
        c.set_keypairs(0, keys, keys, np.arange(n_peers, dtype=np.uint32))
        b = c.batch(n, n * 1472)
        off, sizes = _load(b, rng, n, n_peers)
        plain = np.array(b.ring)
        b.seal(n, F_ASSIGN_COUNTERS)               # no copies
        sealed = np.array(b.ring)
        assert not np.array_equal(sealed, plain)
        b.download(n)                              # nothing newer on the device
        assert np.array_equal(np.array(b.ring), sealed)
        b.len[:n] = b.out_len[:n]
        b.open(n, F_NO_H2D | F_NO_D2H)             # device-resident call: the library uploads first
        b.download(n)
        assert (np.array(b.status[:n]) != oracle.AUTH_FAIL).all()
        got = np.array(b.ring)
        for i in range(n):
            o, l = int(off[i]) + 16, int(sizes[i])
            assert np.array_equal(got[o:o + l], plain[o:o + l]), i
        b.close()
    finally:
        c.close()


def test_classify_and_gso_after_a_batch_without_copies(gpu_lib, oracle):
    """A submit that ran on the host arrays leaves every device descriptor behind.  classify and the GSO split
    upload only what they read; when the device copies are stale they must bring all descriptor fields along,
    or a device-resident seal after them would read old counters."""
    from bnk_b200.device import F_NO_D2H, F_NO_H2D

    n, n_peers = 32, 3
    rng = np.random.default_rng(21)
    keys = rng.integers(0, 256, (n_peers, 32), dtype=np.uint8)
    c = _context(1 << 20, max_keypairs=n_peers, mtu=1420, flow_capacity=0)
    try:
        c.set_keypairs(0, keys, keys, np.arange(n_peers, dtype=np.uint32))
        for i in range(n_peers):
            c.addr_set(bytes(10) + b"\xff\xff" + bytes([10, 0, 0, 1 + i]), 51820, i)
        b = c.batch(n, n * 1472)
        off, sizes = _load(b, rng, n, n_peers)
        sizes = np.maximum(sizes, 40)
        b.len[:n] = sizes
        b.counter[:n] = 1000 + np.arange(n)
        b.seal(n)                                   # host-direct: device descriptors are now behind
        first = np.array(b.ring)
        # new plaintext and new caller-chosen counters, written to the host arrays only
        for i in range(n):
            b.ring[int(off[i]) + 16:int(off[i]) + 16 + int(sizes[i])] = rng.integers(0, 256, int(sizes[i]), dtype=np.uint8)
        plain = np.array(b.ring)
        b.len[:n] = sizes
        b.counter[:n] = 5000 + np.arange(n)
        peers = rng.integers(0, n_peers, n)
        for i in range(n):
            b.src_addr[i, :] = 0
            b.src_addr[i, 10:12] = 0xFF
            b.src_addr[i, 12:16] = [10, 0, 0, 1 + int(peers[i])]
            b.src_addr[i, 16:18] = [51820 >> 8, 51820 & 255]
        b.classify(n)                               # uploads; must refresh counter/out_len/status too
        assert list(b.slot[:n]) == list(peers)
        b.seal(n, F_NO_H2D | F_NO_D2H)              # caller-supplied counters, read from the device copies
        b.download(n)
        assert (b.status[:n] == 0).all()
        assert (b.counter[:n] == 5000 + np.arange(n)).all()
        # (classify uploads datagrams, ring[off, off+len): the furthest packet's last 16 payload bytes, which lie
        # behind that span, are not part of its upload, so that one packet is left out of the byte comparison)
        for i in range(n - 1):
            o, l = int(off[i]) + 16, int(sizes[i])
            want = oracle.wg_seal(keys[int(peers[i])].tobytes(), int(peers[i]), 5000 + i, plain[o:o + l].tobytes(), 1420)
            assert b.message(i) == want, i
        assert not np.array_equal(np.array(b.ring), first)
        b.close()
    finally:
        c.close()


@pytest.mark.parametrize("between", ["seal", "open", "upload", "note", "check", "classify", "classify all", "split", "copied seal"])
def test_a_small_call_between_does_not_hide_what_is_behind(gpu_lib, oracle, between):
    """1000 packets sealed in place, then a copied call for ten of the batch, then all of them from the device: the ring and
    the descriptors that the device works on are those of the host arrays, beyond the ten too."""
    from bnk_b200.device import F_NO_D2H, F_NO_H2D, F_USE_OUT_LEN, GSO_SUPER_DTYPE

    n, few, size = 1000, 10, 300
    rng = np.random.default_rng(3)
    keys = rng.integers(0, 256, (2, 32), dtype=np.uint8)
    c = _context(1 << 20, max_keypairs=8, mtu=1420, flow_capacity=16)
    try:
        c.set_keypairs(0, keys, keys, np.arange(2, dtype=np.uint32))
        for p in range(2):
            c.addr_set(bytes(10) + b"\xff\xff" + bytes([10, 0, 0, 1 + p]), 51820, p)
        b = c.batch(n, n * 352)
        b.off[:], b.len[:], b.slot[:], b.counter[:] = np.arange(n) * 352, size, rng.integers(0, 2, n), np.arange(n)
        b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
        b.src_addr[:, 10:12], b.src_addr[:, 12:16], b.src_addr[:, 16:18] = 255, (10, 0, 0, 2), (51820 >> 8, 51820 & 255)
        plain = np.array(b.ring).reshape(n, 352)[:, 16:16 + size]
        b.seal(n)
        if between.startswith("classify"):
            if between == "classify all":
                slot = np.array(b.slot)
                b.classify(n)  # in place: the device has no source addresses
                b.slot[:] = slot
                b.upload(few)
            else:
                b.classify(few, F_NO_D2H)
        elif between == "split":
            b.gso_split(np.zeros(0, GSO_SUPER_DTYPE), few)
        elif between == "copied seal":  # results come down: nothing has to catch up for it, everything for what follows
            b.len[:few] = 200
            others = [c.batch(600, 600 * 800) for _ in range(4)]
            for o in others:
                o.seal(600, wait=False)
            b.seal(few)
            b.len[:few] = b.out_len[:few] - 32
            for o in others:
                o.wait()
        elif between == "upload":
            b.upload(few)
        elif between == "note":
            b.filter_note(few, 0, F_NO_D2H)
        elif between == "check":
            b.filter_check(few, 0, F_NO_D2H)
        else:
            getattr(b, between)(few, F_NO_D2H)
        if between == "classify all":
            b.classify(n, F_NO_H2D)
            assert (b.slot == 1).all() and (b.status == 0).all()
            return
        b.open(n, F_NO_H2D | F_USE_OUT_LEN | F_NO_D2H)
        b.download(n)
        assert (b.status[few:] == 0).all() and (b.out_len[few:] == 304).all()
        assert np.array_equal(b.ring.reshape(n, 352)[few:, 16:16 + size], plain[few:])
    finally:
        c.close()


@pytest.mark.parametrize("n,size,pieces_from", [(48, 300, None), (1000, 300, None), (12_000, 64, None), (24_000, 64, 1 << 20)])  # in place, and in pieces
def test_device_only_submits_need_no_wait(gpu_lib, oracle, monkeypatch, n, size, pieces_from):
    """A submit that touches no host array may follow any other without a wait in between."""
    from bnk_b200.device import F_ASSIGN_COUNTERS, F_NO_D2H, F_NO_H2D, F_REPLAY, F_USE_OUT_LEN

    rng = np.random.default_rng(n)
    stride = 48 + (size + 15) // 16 * 16
    keys = rng.integers(0, 256, (2, 32), dtype=np.uint8)
    if pieces_from:
        monkeypatch.setenv("BNK_PIECES_FROM", str(pieces_from))
    c = _context(512 << 20, max_keypairs=2, mtu=1420, flow_capacity=0)
    try:
        c.set_keypairs(0, keys, keys, np.arange(2, dtype=np.uint32))
        b = c.batch(n, n * stride)
        b.off[:], b.len[:], b.slot[:] = np.arange(n) * stride, size, rng.integers(0, 2, n)
        b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
        plain = np.array(b.ring).reshape(n, stride)[:, 16:16 + size]
        launched = c.launch_count()
        b.seal(n, F_ASSIGN_COUNTERS, wait=False)
        launched = c.launch_count() - launched  # for the nonces, up to 256 packets none, and for the packets, of pieces each one
        assert launched == 1 + (n > 256) if not pieces_from else launched > 2
        b.open(n, F_NO_H2D | F_NO_D2H | F_USE_OUT_LEN | F_REPLAY, wait=False)
        b.seal(n, F_NO_H2D | F_NO_D2H | F_ASSIGN_COUNTERS, wait=False)
        b.open(n, F_NO_H2D | F_NO_D2H | F_USE_OUT_LEN | F_REPLAY)
        b.download(n)
        assert (b.status == 0).all() and np.array_equal(b.ring.reshape(n, stride)[:, 16:16 + size], plain)
        assert sum(c.send_counter(p) for p in range(2)) == 2 * n
    finally:
        c.close()


@pytest.mark.parametrize("stride", [96, 512])  # packets that lie close together, and not
@pytest.mark.parametrize("look", ["note", "check", "classify"])
def test_heads_looked_at_and_then_sealed_on_the_device(gpu_lib, oracle, look, stride):
    """A look at the packets' heads, then a seal that takes the packets from the device: where the heads are read in place the
    packets go up behind the look, and from the second time on in front of it.  Every round has other packets, keypairs and
    nonces; some have the seal take the packets from the host."""
    from bnk_b200 import Context
    from bnk_b200.device import F_NO_H2D
    from bnk_b200.filter import CompiledRule, PortRange, flatten_rules

    rng = np.random.default_rng(stride)
    n, peers, size = 1500, 4, 60
    keys = rng.integers(0, 256, (peers, 32), dtype=np.uint8)
    off = H.layout_fixed(n, stride)
    with Context(max_keypairs=peers, mtu=0, flow_capacity=1 << 14) as c:
        c.set_keypairs(0, keys, keys, np.arange(peers, dtype=np.uint32))
        c.acl_set(True, flatten_rules([CompiledRule(srcs=["100.64.0.0/16"], proto="udp", ports=[PortRange(1, 30000)])]))
        b = c.batch(n, n * stride)
        f = oracle.Filter()
        f.set_rules([([(RC.ip("100.64.0.0"), 16)], "udp", [(1, 30000)])])
        for r, on_device in enumerate([True, True, True, False, True, False, False, True]):
            now = RC.T0 + r * RC.SEC
            b.ring[:] = rng.integers(0, 256, b.ring_bytes, dtype=np.uint8)
            packets = [RC.udp(RC.ip("100.64.0.0") + int(rng.integers(0, 1 << 17)), RC.SELF, int(rng.integers(1, 9)), int(rng.integers(1, 60000)))[:28]
                       for _ in range(n)]
            for o, p in zip(off, packets):
                b.ring[o + 16:o + 44] = np.frombuffer(p, np.uint8)
            b.off[:], b.len[:], b.slot[:] = off, size, rng.integers(0, peers, n)
            b.counter[:] = rng.integers(0, 2**60, n, dtype=np.uint64)
            if look == "note":
                b.filter_note(n, now)
                for p in packets:
                    f.note_outbound(p, now)
                assert H.flows_equal(c.flows_export(), f.flows())
            elif look == "check":
                b.filter_check(n, now)
                assert np.array_equal(b.status == 0, [f.check_inbound(p, now) for p in packets])
            else:
                slots = np.array(b.slot)
                b.classify(n)
                b.slot[:] = slots  # (an output of the call for known peers, of whom there are none)
            ring, st, ln = H.oracle_seal(oracle, keys, np.arange(peers), 0, b.ring, off, b.len, b.slot, b.counter)
            b.seal(n, F_NO_H2D if on_device else 0)
            assert np.array_equal(b.status, st) and np.array_equal(b.out_len, ln)
            assert H.spans_differ_count(np.array(b.ring), ring, off, ln) == 0, r
        b.close()
