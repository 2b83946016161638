"""What kernels do when a bulk copy over the link does not come.  The library here is a build of its own (_build.build_lost_copies)
that never asks for copies of LOST_BYTES and gives up waiting soon, so which packets are hit is a matter of their sizes."""
import os

import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.fixture
def lossy(gpu_lib, monkeypatch):
    from bnk_b200 import _build, _lib

    if not os.path.exists(_build.lost_copies_path()):
        _build.build_lost_copies()
    monkeypatch.setattr(_lib, "_LIB", _lib.load(_build.lost_copies_path()))
    return _build.LOST_BYTES


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
