"""ACL filter parity on the GPU: the reference's own cases through the Python mirror of its
interface, and configuration 3 against the CPU checker, verdict for verdict."""
import numpy as np
import pytest

from tests import reference_cases as RC

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu_lib):
    from bnk_b200 import Context

    c = Context(max_keypairs=4, flow_capacity=1 << 14)
    yield c
    c.close()


@pytest.fixture()
def make(ctx):
    from bnk_b200.filter import Filter

    made = []

    def _make():
        ctx.flows_clear()
        f = Filter(ctx, batch_pkts=8)
        made.append(f)
        return f

    yield _make
    for f in made:
        f._batch.close()


@pytest.mark.parametrize("case", RC.ALL_CASES, ids=lambda c: c.__name__)
def test_reference_cases(make, case):
    case(make)


def test_wrap_tun_cases(make):
    from bnk_b200.filter import wrap_tun

    RC.tun_case_drops_denied_inbound_writes(make, wrap_tun)
    RC.tun_case_read_records_outbound_flows(make, wrap_tun)


def _load_headers(b, hdr, lens):
    from bnk_b200 import gen

    n = len(lens)
    stride = gen.HDR_STRIDE
    view = b.ring[:n * stride].reshape(n, stride)
    view[:, 16:16 + hdr.shape[1]] = hdr
    b.off[:n] = (np.arange(n, dtype=np.uint64) * stride).astype(np.uint32)
    b.len[:n] = lens
    return n


def _run_config3(oracle, n_rules, n_nodes, n_out, n_in, seed=None, flow_capacity=1 << 20):
    """Every verdict of the inbound batch, of a late batch after the TTLs have run out and of the same batch
    again, and the flow count, against the CPU checker (whose rule walk runs on all host cores)."""
    from bnk_b200 import Context, gen
    from bnk_b200.device import F_STATS, PKT_FILTER_DENY, PKT_OK
    from bnk_b200.filter import flatten_rule_arrays

    w = gen.config3(n_rules, n_nodes, n_out, n_in, seed=seed)
    # CPU checker
    f = oracle.Filter()
    f.set_rules_arrays(w.rules.astype(oracle.RULE_DTYPE), w.srcs.astype(oracle.PREFIX_DTYPE),
                       w.ports.astype(oracle.PORT_DTYPE))
    f.note_batch(np.ascontiguousarray(w.outbound), 28, w.outbound_len, w.t0_ns)
    want = f.check_batch_mt(np.ascontiguousarray(w.inbound), 28, np.ascontiguousarray(w.inbound_len), w.t0_ns + RC.SEC)
    want_late = f.check_batch_mt(np.ascontiguousarray(w.late), 28, w.late_len, w.t0_ns + 10 * RC.MIN)
    want_again = f.check_batch_mt(np.ascontiguousarray(w.late), 28, w.late_len, w.t0_ns + 2 * RC.SEC)
    want_flows = f.flow_count
    # GPU
    c = Context(max_keypairs=4, flow_capacity=flow_capacity)
    try:
        c.acl_set(True, flatten_rule_arrays(w.rules, w.srcs, w.ports))
        cap = max(n_out, n_in)
        b = c.batch(cap, cap * gen.HDR_STRIDE)
        n = _load_headers(b, w.outbound, w.outbound_len)
        b.filter_note(n, w.t0_ns)
        n = _load_headers(b, w.inbound, w.inbound_len)
        b.filter_check(n, w.t0_ns + RC.SEC, F_STATS)
        got = (np.array(b.status[:n]) == PKT_OK).astype(np.uint8)
        stats = b.stats()
        assert stats["packets"] == n and stats["by_status"][PKT_OK] == int(got.sum())
        assert stats["by_status"][PKT_FILTER_DENY] == n - int(got.sum())
        n = _load_headers(b, w.late, w.late_len)
        b.filter_check(n, w.t0_ns + 10 * RC.MIN)
        got_late = (np.array(b.status[:n]) == PKT_OK).astype(np.uint8)
        b.filter_check(n, w.t0_ns + 2 * RC.SEC)
        got_again = (np.array(b.status[:n]) == PKT_OK).astype(np.uint8)
        got_flows = c.flows_count()
        got_table = c.flows_export()
    finally:
        c.close()
    assert np.array_equal(got, want), f"{np.flatnonzero(got != want)[:10]} differ"
    assert np.array_equal(got_late, want_late)
    assert np.array_equal(got_again, want_again)
    assert got_flows == want_flows
    # not only the verdicts: the whole flow table, key for key and expiry for expiry, equals the checker's map
    from tests.helpers import flows_equal

    assert len(got_table) == want_flows and flows_equal(got_table, f.flows())
    return w, got, want_late


def test_config3_small(oracle):
    w, want, late = _run_config3(oracle, 500, 2000, 6000, 20000, seed=77, flow_capacity=1 << 14)
    assert 0.25 < want.mean() < 0.9      # both verdicts well represented
    assert late.sum() < len(late)        # replies whose flow ran out are refused


def test_config3_full_size(oracle):
    """BASELINE configuration 3 at its stated size: 10,000 rules, 300,000 noted flows, 1,000,000 inbound
    headers; all 1,000,000 verdicts, the late batch and the flow count equal the CPU checker's."""
    w, got, late = _run_config3(oracle, 10_000, 50_000, 300_000, 1_000_000)
    assert len(got) == 1_000_000 and got.sum() > 300_000
    # size-independent properties over all 1,000,000 verdicts: malformed headers never pass ...
    # (a header cut to 22 bytes still parses when it is icmp, which needs one body byte only)
    bad = ((w.inbound_len < 24) & (w.inbound[:, 9] != 1)) | (w.inbound[:, 0] != 0x45) | ~np.isin(w.inbound[:, 9], (1, 6, 17))
    assert bad.sum() > 40_000 and got[bad].sum() == 0
    # ... and every exact mirror of a noted flow passes while its TTL runs
    reply = np.zeros(len(got), bool)
    key_out = {bytes(h[9:10]) + bytes(h[16:20]) + bytes(h[22:24]) + bytes(h[20:22]) for h in w.outbound[::7]}
    for i in range(0, len(got), 97):
        h = w.inbound[i]
        if not bad[i] and bytes(h[9:10]) + bytes(h[12:16]) + bytes(h[20:24]) in key_out:
            reply[i] = True
    assert reply.sum() > 100 and got[reply].all()


def test_flow_sweep_and_count(ctx):
    """filter.go:202-208 through the batch path: counts and the >4096 sweep follow the reference."""
    from bnk_b200.filter import Filter

    ctx.flows_clear()
    f = Filter(ctx, batch_pkts=5000)
    f.set_rules([])
    f.note_outbound_batch([RC.udp(RC.SELF, RC.PEER, 1 + i, 7) for i in range(4096)], RC.T0)
    assert ctx.flows_count() == 4096
    f.note_outbound(RC.udp(RC.SELF, RC.PEER, 5000, 7), RC.T0 + 10 * RC.SEC)
    assert ctx.flows_count() == 4097
    f.note_outbound(RC.udp(RC.SELF, RC.PEER, 5001, 7), RC.T0 + 31 * RC.SEC)
    assert ctx.flows_count() == 2
    assert not f.check_inbound(RC.udp(RC.PEER, RC.SELF, 7, 1), RC.T0 + 5 * RC.SEC)
    # duplicates inside one batch count once; the all-ones key has its own slot
    ctx.flows_clear()
    f.note_outbound_batch([RC.udp(RC.SELF, RC.PEER, 9, 9)] * 100 + [RC.udp(RC.SELF, 0xFFFFFFFF, 65535, 65535)] * 3, RC.T0)
    assert ctx.flows_count() == 2
    assert f.check_inbound(RC.udp(0xFFFFFFFF, RC.SELF, 65535, 65535), RC.T0 + RC.SEC)
    assert not f.check_inbound(RC.tcp(0xFFFFFFFF, RC.SELF, 65535, 65535), RC.T0 + RC.SEC)
    f._batch.close()


def test_flow_table_full_is_reported(gpu_lib):
    from bnk_b200 import Context
    from bnk_b200.device import BnkError
    from bnk_b200.filter import Filter

    c = Context(max_keypairs=4, flow_capacity=16)
    try:
        f = Filter(c, batch_pkts=64)
        f.set_rules([])
        with pytest.raises(BnkError) as e:
            f.note_outbound_batch([RC.udp(RC.SELF, RC.PEER, 1 + i, 7) for i in range(40)], RC.T0)
        assert e.value.code == -6
    finally:
        c.close()


def test_policy_to_verdicts_end_to_end(make):
    """Policy document -> Compile -> netmap -> ApplyNetmap -> GPU verdicts, the route of the reference's
    internal/dataplane/acl_integration_test.go:20-80 (tcp/7777 allowed, tcp/8888 blocked, replies pass)."""
    from bnk_b200 import acl

    nodes = [acl.NodeInfo("a", "100.64.0.1"), acl.NodeInfo("b", "100.64.0.2"), acl.NodeInfo("c", "100.64.0.3")]
    policy = acl.Policy(rules=[acl.Rule(["a"], ["b"], ["tcp/7777"])])
    compiled = acl.compile_policy(policy, nodes)
    a, b, c = RC.ip("100.64.0.1"), RC.ip("100.64.0.2"), RC.ip("100.64.0.3")
    f = make()
    acl.apply_netmap_filter(f, {"filter_enabled": True, "filter": acl.rules_to_netmap(compiled.get("b", []))})
    assert f.check_inbound(RC.tcp(a, b, 40000, 7777), RC.T0)
    assert not f.check_inbound(RC.tcp(a, b, 40000, 8888), RC.T0)
    assert not f.check_inbound(RC.tcp(c, b, 40000, 7777), RC.T0)
    # node a has no inbound rule at all under this policy: deny all but replies to what it opened
    acl.apply_netmap_filter(f, {"filter_enabled": True, "filter": acl.rules_to_netmap(compiled.get("a", []))})
    assert not f.check_inbound(RC.tcp(b, a, 7777, 40000, False), RC.T0)
    f.note_outbound(RC.tcp(a, b, 40000, 7777), RC.T0)
    assert f.check_inbound(RC.tcp(b, a, 7777, 40000, False), RC.T0 + RC.SEC)
    # the policy is withdrawn: allow all (flows are kept, rules are gone)
    acl.apply_netmap_filter(f, {"filter_enabled": False})
    assert f.check_inbound(RC.tcp(c, a, 1, 2), RC.T0)


def test_flow_table_export_and_import(gpu_lib, oracle):
    """State hand-over: the entries exported from one context, imported into a fresh one, give the same verdicts
    and the same table there (all three protocol classes, the all-ones key, a deleted entry is not exported)."""
    from bnk_b200 import Context
    from bnk_b200.filter import Filter
    from tests.helpers import flows_equal

    a = Context(max_keypairs=4, flow_capacity=1 << 10)
    b = Context(max_keypairs=4, flow_capacity=1 << 12)
    o = oracle.Filter()
    o.set_rules([])
    try:
        fa, fb = Filter(a, batch_pkts=64), Filter(b, batch_pkts=64)
        fa.set_rules([])
        fb.set_rules([])
        out = ([RC.udp(RC.SELF, RC.PEER, 1000 + i, 53) for i in range(20)] + [RC.tcp(RC.SELF, RC.OTHER, 2000 + i, 443) for i in range(20)]
               + [RC.icmp_echo(RC.SELF, RC.PEER, False), RC.udp(RC.SELF, 0xFFFFFFFF, 65535, 65535)])
        fa.note_outbound_batch(out, RC.T0)
        for p in out:
            o.note_outbound(p, RC.T0)
        # one udp flow runs out and is deleted by a lookup
        late = RC.udp(RC.PEER, RC.SELF, 53, 1000)
        assert not fa.check_inbound(late, RC.T0 + 31 * RC.SEC) and not o.check_inbound(late, RC.T0 + 31 * RC.SEC)
        table = a.flows_export()
        assert len(table) == 41 and flows_equal(table, o.flows())
        b.flows_import(table)
        assert b.flows_count() == 41 and flows_equal(b.flows_export(), o.flows())
        for pkt, want in ((RC.udp(RC.PEER, RC.SELF, 53, 1001), True), (late, False),
                          (RC.tcp(RC.OTHER, RC.SELF, 443, 2005, False), True), (RC.icmp_echo(RC.PEER, RC.SELF, True), True),
                          (RC.udp(0xFFFFFFFF, RC.SELF, 65535, 65535), True), (RC.tcp(RC.OTHER, RC.SELF, 443, 2999, False), False)):
            assert fb.check_inbound(pkt, RC.T0 + RC.SEC) == want == o.check_inbound(pkt, RC.T0 + RC.SEC)
        assert flows_equal(b.flows_export(), o.flows())  # the refreshed expiries too
        b.flows_import(table[:3])                         # importing a key again only moves its expiry
        assert b.flows_count() == 41
        fa._batch.close()
        fb._batch.close()
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("shape", ["few_lengths_listed", "many_keys_per_length", "everything_listed", "default_route"])
def test_rule_tables_with_many_prefix_lengths(gpu_lib, oracle, shape):
    """Rule tables with several prefix lengths in very different numbers: every verdict equals the checker's rule
    walk (acl.go:149-172: any prefix of any length that contains the source, filter.go:131-135).  Shapes: a handful
    of hand-written prefixes beside thousands of /32s; hundreds of keys in each of four lengths; only a few prefixes;
    a /0 rule.  (The index probes one hash table per prefix length in use; a variant that kept the rare lengths in a
    short list in shared memory passed the same test and was no faster.)"""
    from bnk_b200 import Context
    from bnk_b200.filter import Filter, CompiledRule, PortRange

    rng = np.random.default_rng({"few_lengths_listed": 1, "many_keys_per_length": 2, "everything_listed": 3,
                                 "default_route": 4}[shape])
    base = RC.ip("100.64.0.0")

    def host(k):
        return base + int(k)

    def pfx(addr, bits):
        import ipaddress
        return f"{ipaddress.ip_address(addr & ((0xffffffff << (32 - bits)) & 0xffffffff) if bits else 0)}/{bits}"

    rules = []
    if shape in ("few_lengths_listed", "default_route"):
        for k in rng.integers(1, 1 << 20, 3000):
            rules.append(CompiledRule(srcs=[pfx(host(k), 32)], proto=str(rng.choice(["tcp", "udp"])),
                                      ports=[PortRange(1, int(rng.integers(1, 40000)))]))
        for bits in (8, 12, 16, 20, 24, 28, 30):
            for _ in range(int(rng.integers(1, 6))):
                rules.append(CompiledRule(srcs=[pfx(host(rng.integers(1, 1 << 20)), bits)], proto="udp",
                                          ports=[PortRange(50, 60)]))
        if shape == "default_route":
            rules.append(CompiledRule(srcs=["0.0.0.0/0"], proto="icmp", ports=[]))
    elif shape == "many_keys_per_length":
        for bits in (24, 26, 28, 32):
            for k in rng.integers(1, 1 << 20, 400):
                rules.append(CompiledRule(srcs=[pfx(host(k), bits)], proto="tcp", ports=[PortRange(1000, 2000)]))
    else:
        for bits in (10, 16, 24, 32):
            for _ in range(5):
                rules.append(CompiledRule(srcs=[pfx(host(rng.integers(1, 1 << 20)), bits)], proto="tcp",
                                          ports=[PortRange(22, 22), PortRange(80, 90)]))
    c = Context(max_keypairs=4, flow_capacity=1 << 10)
    try:
        f = Filter(c, batch_pkts=4096)
        f.set_rules(rules)
        chk = oracle.Filter()
        chk.set_rules([([(RC.ip(s.split("/")[0]), int(s.split("/")[1])) for s in r.srcs], r.proto,
                        [(p.first, p.last) for p in r.ports]) for r in rules])
        # sources: half of them taken from the rules' own prefixes (inside and just outside), half anywhere
        pool = [RC.ip(s.split("/")[0]) for r in rules for s in r.srcs]
        pkts = []
        for k in range(4096):
            src = int(pool[int(rng.integers(0, len(pool)))]) + int(rng.integers(0, 3)) if k % 2 else host(rng.integers(1, 1 << 20))
            src &= 0xffffffff
            kind = int(rng.integers(0, 3))
            port = int(rng.choice([22, 55, 85, 1500, 30000, int(rng.integers(1, 65535))]))
            if kind == 0:
                pkts.append(RC.tcp(src, RC.SELF, 40000, port))
            elif kind == 1:
                pkts.append(RC.udp(src, RC.SELF, 40000, port))
            else:
                pkts.append(RC.icmp_echo(src, RC.SELF, False))
        got = f.check_inbound_batch(pkts, RC.T0)
        want = [chk.check_inbound(p, RC.T0) for p in pkts]
        assert got == want
        assert 50 < sum(want) < 4000
        f._batch.close()
    finally:
        c.close()


@pytest.mark.parametrize("room", [False, True])  # True: both buffers of the index were made with the context
@pytest.mark.parametrize("shape", ["hosts anywhere", "hosts of one stretch", "networks anywhere", "every length", "short only"])
def test_rule_tables_over_the_whole_address_space(gpu_lib, oracle, shape, room):
    """Tables whose prefixes lie anywhere (a block of the index for nearly every 65,536 addresses) or all in one such
    stretch, the first and the last address among them, set one after the other in one context."""
    from bnk_b200 import Context
    from bnk_b200.device import ACL_TUPLE_DTYPE

    rng = np.random.default_rng(len(shape))
    k = 90_000 if shape == "hosts anywhere" else 8000
    bits = {"hosts": np.full(k, 32), "networks": rng.integers(17, 25, k), "every": rng.integers(0, 33, k), "short": rng.integers(13, 17, k)}[shape.split()[0]]
    if shape == "every length":
        bits[bits < 9] += 12  # (or everything is allowed)
    addr = rng.integers(0, 1 << 32, k)
    if shape == "hosts of one stretch":
        addr = 0xC0A80000 + rng.integers(0, 1 << 16, k)
    addr[:2] = 0, 0xFFFFFFFF
    if shape == "every length":
        addr[k // 2:] = addr[:k // 2] ^ rng.integers(0, 1 << 12, k // 2)  # one inside the other
    addr &= (0xFFFFFFFF << (32 - bits)) & 0xFFFFFFFF
    n = 6000
    h = np.zeros((n, 28), np.uint8)
    for i in range(n):
        src = int(addr[rng.integers(0, k)] if i > 3 else (0, 0xFFFFFFFF, 0x80000000, 0x0000FFFF)[i])
        src = (src + int(rng.choice([0, 0, 1, 255, 256, 65535, 1 << 20]))) & 0xFFFFFFFF
        h[i] = np.frombuffer(RC.tcp(src, RC.SELF, 40000, 443)[:28], np.uint8)
    lens = np.full(n, 28, np.uint32)
    with Context(max_keypairs=1, flow_capacity=16, max_acl_tuples=100_000 if room else 0) as c:
        b = c.batch(n, n * 48)
        b.ring.reshape(n, 48)[:, 16:44] = h
        b.off[:], b.len[:] = np.arange(n) * 48, lens
        for part in (slice(0, k), slice(0, k // 3), slice(0, 1), slice(0, 0), slice(k // 2, k)):
            t = np.zeros(len(addr[part]), ACL_TUPLE_DTYPE)
            t["addr"], t["prefix_len"], t["proto"], t["port_first"], t["port_last"] = addr[part], bits[part], 6, 443, 443
            c.acl_set(True, t)
            chk = oracle.Filter()
            chk.set_rules([([(int(x), int(y)) for x, y in zip(addr[part], bits[part])], "tcp", [(443, 443)])])
            want = chk.check_batch_mt(np.ascontiguousarray(h), 28, lens, RC.T0)
            b.filter_check(n, RC.T0)
            assert np.array_equal(b.status == 0, want != 0), np.flatnonzero((b.status == 0) != (want != 0))[:5]
            assert len(t) < 4000 or 500 < (want != 0).sum() < n


@pytest.mark.parametrize("n", [1, 127, 128, 129, 5000])  # a CTA's statuses leave as one line
def test_nested_prefixes_and_merged_port_ranges(gpu_lib, oracle, n):
    """Prefixes of every length one inside the other, around the steps of the index (16, 24 bits), each with several port
    ranges that touch, overlap or leave a port between them: a packet is allowed by whichever contains it."""
    from bnk_b200 import Context
    from bnk_b200.device import F_NO_H2D
    from bnk_b200.filter import CompiledRule, PortRange, flatten_rules

    rng = np.random.default_rng(n)
    base = RC.ip("100.64.0.0")
    spots = base + rng.integers(0, 1 << 18, 12)  # prefixes crowd around these
    rules, chk_rules = [], []
    for bits in [0] + [int(b) for b in rng.integers(1, 33, 700)] + [15, 16, 17, 23, 24, 25, 31, 32] * 6:
        addr = int(spots[rng.integers(0, len(spots))]) ^ int(rng.integers(0, 1 << int(rng.integers(1, 20))))
        addr &= (0xffffffff << (32 - bits)) & 0xffffffff if bits else 0
        proto = str(rng.choice(["tcp", "udp", "icmp"], p=[0.5, 0.45, 0.05])) if bits > 8 else "udp"
        at, ranges = int(rng.integers(0, 65536)), []
        for _ in range(int(rng.integers(1, 6)) if proto != "icmp" else 0):
            end = min(65535, at + int(rng.choice([0, 1, 5, 300])))
            ranges.append((at, end))
            at = min(65535, end + int(rng.choice([0, 1, 2, 40])))
        rules.append(CompiledRule(srcs=[f"{addr >> 24}.{addr >> 16 & 255}.{addr >> 8 & 255}.{addr & 255}/{bits}"], proto=proto,
                                  ports=[PortRange(*r) for r in ranges]))
        chk_rules.append(([(addr, bits)], proto, ranges))
    chk = oracle.Filter()
    chk.set_rules(chk_rules)
    pick = rng.integers(0, len(chk_rules), n)
    h = np.zeros((n, 28), np.uint8)
    lens = np.full(n, 28, np.uint32)
    for i, k in enumerate(pick):  # sources inside and beside a prefix, ports at and beside the ends of a range
        (addr, bits), = chk_rules[k][0]
        src = (addr + int(rng.integers(-2, 3)) + int(rng.integers(0, 1 << min(32 - bits, 9)))) & 0xffffffff
        ends = [e for r in chk_rules[int(rng.choice(pick))][2] for e in r] or [80]
        port = (int(rng.choice(ends)) + int(rng.integers(-1, 2))) & 0xffff
        h[i] = np.frombuffer([RC.tcp, RC.udp, lambda a, b, c, d: RC.icmp_echo(a, b, False)][int(rng.integers(0, 3))](src, RC.SELF, 40000, port)[:28], np.uint8)
    want = chk.check_batch(np.ascontiguousarray(h), 28, lens, RC.T0)
    with Context(max_keypairs=1, flow_capacity=1 << 10) as c:
        c.acl_set(True, flatten_rules(rules))
        b = c.batch(n, n * 48)
        b.ring.reshape(n, 48)[:, 16:44] = h
        b.off[:], b.len[:] = np.arange(n) * 48, lens
        for flags in (0, F_NO_H2D):
            b.status[:] = 99
            b.filter_check(n, RC.T0, flags)
            assert np.array_equal(b.status == 0, want != 0), np.flatnonzero((b.status == 0) != (want != 0))[:5]
        assert n < 1000 or 200 < (want != 0).sum() < n - 200
        b.close()


@pytest.mark.parametrize("singles", [0, 1, 24, 256])
@pytest.mark.parametrize("longer", [False, True])
def test_single_addresses_of_a_block(gpu_lib, oracle, singles, longer):
    """Every address of a stretch of 256 and of its neighbours, of which some have rules of their own: 24 apart they share a mark in
    the index, and prefixes of 25 to 31 bits and one of 20 lie around them."""
    from bnk_b200 import Context
    from bnk_b200.device import F_NO_H2D
    from bnk_b200.filter import CompiledRule, PortRange, flatten_rules

    rng = np.random.default_rng(singles)
    block = RC.ip("100.64.37.0")
    of = [(int(a), 32, 100 + k % 3) for k, a in enumerate(block + rng.choice(256, singles, replace=False))]
    if longer:
        of += [(block + 24 * k & (0xffffffff << (32 - bits)) & 0xffffffff, bits, 200) for k, bits in enumerate(range(25, 32))] + [(block & 0xfffff000, 20, 300)]
    text = [f"{a >> 24}.{a >> 16 & 255}.{a >> 8 & 255}.{a & 255}/{bits}" for a, bits, _ in of]
    chk = oracle.Filter()
    chk.set_rules([([(a, bits)], "tcp", [(port, port)]) for a, bits, port in of])
    src = np.repeat(np.arange(block - 256, block + 512), 5)
    n = len(src)
    port = np.tile([100, 101, 102, 200, 300], n // 5)
    h = np.stack([np.frombuffer(RC.tcp(int(a), RC.SELF, 40000, int(p))[:28], np.uint8) for a, p in zip(src, port)])
    lens = np.full(n, 28, np.uint32)
    want = chk.check_batch(np.ascontiguousarray(h), 28, lens, RC.T0)
    with Context(max_keypairs=1, flow_capacity=1 << 10) as c:
        c.acl_set(True, flatten_rules([CompiledRule(srcs=[t], proto="tcp", ports=[PortRange(p, p)]) for t, (_, _, p) in zip(text, of)]))
        b = c.batch(n, n * 48)
        b.ring.reshape(n, 48)[:, 16:44] = h
        b.off[:], b.len[:] = np.arange(n) * 48, lens
        for flags in (0, F_NO_H2D):
            b.status[:] = 99
            b.filter_check(n, RC.T0, flags)
            assert np.array_equal(b.status == 0, want != 0), np.flatnonzero((b.status == 0) != (want != 0))[:5]
        assert ((want != 0).sum() >= singles) and (singles or longer or not want.any())
        b.close()


@pytest.mark.parametrize("n", [1025, 16384, 16385, 49152, 49153, 180000])  # a stretch of descriptors: 16,384, then double
@pytest.mark.parametrize("shuffled", [False, True])
def test_packets_close_together_go_up_stretch_by_stretch(gpu_lib, oracle, n, shuffled):
    """Headers 48 bytes apart, in ring order and not, on a device copy that holds others: every verdict is that of the
    header the host wrote."""
    from bnk_b200 import Context

    rng = np.random.default_rng(n)
    rule = ([(RC.ip("100.64.1.0"), 24)], "udp", [(1000, 1999)])
    chk = oracle.Filter()
    chk.set_rules([rule])
    h = np.zeros((n, 28), np.uint8)
    h[:] = np.frombuffer(RC.udp(RC.ip("100.64.1.1"), RC.SELF, 40000, 1000)[:28], np.uint8)
    h[:, 14] = rng.integers(1, 3, n)              # the source's third byte: in the prefix or beside it
    port = rng.integers(500, 2500, n)
    h[:, 22], h[:, 23] = port >> 8, port & 255
    lens = np.full(n, 28, np.uint32)
    want = chk.check_batch(h, 28, lens, RC.T0) != 0
    from bnk_b200.filter import CompiledRule, PortRange, flatten_rules

    with Context(max_keypairs=1, flow_capacity=1 << 10) as c:
        c.acl_set(True, flatten_rules([CompiledRule(srcs=["100.64.1.0/24"], proto="udp", ports=[PortRange(1000, 1999)])]))
        b = c.batch(n, n * 48)
        place = rng.permutation(n) if shuffled else np.arange(n)
        b.off[:], b.len[:] = place * 48, lens
        slots = b.ring.reshape(n, 48)
        slots[:] = 0
        b.filter_check(n, RC.T0)                  # the device's copy: headers that nothing allows
        assert (b.status != 0).all()
        slots[place, 16:44] = h
        b.filter_check(n, RC.T0)
        assert np.array_equal(b.status == 0, want), np.flatnonzero((b.status == 0) != want)[:5]
        assert 0.1 < want.mean() < 0.4
        b.close()


@pytest.mark.parametrize("n", [1, 511, 512, 513, 799])  # from 512 on, two lanes read a head that lies in pinned memory
def test_heads_of_packets_anywhere_in_the_ring(gpu_lib, oracle, n):
    """Whole packets in any order, at every 16 bytes of a line and up to the ring's last byte, some with IP options (ports
    beyond the first 32 bytes), some cut short, misplaced or outside the ring: flows and verdicts are the checker's."""
    from bnk_b200 import Context
    from bnk_b200.filter import CompiledRule, PortRange, flatten_rules
    from tests.helpers import flows_equal

    rng = np.random.default_rng(n)

    def packet(src, dst, sport, dport):
        p = bytearray([RC.udp, RC.tcp][int(rng.integers(0, 2))](src, dst, sport, dport)[:28])
        words = int(rng.choice([5, 5, 5, 6, 7, 8, 15]))  # options between the header and the ports
        p[0] = 0x40 | words
        p = p[:20] + bytes(rng.integers(0, 256, 4 * words - 20, dtype=np.uint8)) + p[20:] + bytes(int(rng.integers(0, 200)))
        return bytes(p[:int(rng.choice([0, 1, 19, 20, 4 * words, 4 * words + 3, 4 * words + 4]))] if rng.random() < 0.1 else p)

    peers = RC.ip("100.64.1.0") + rng.integers(0, 4, n)
    out = [packet(RC.SELF, int(p), 1000 + i, 53) for i, p in enumerate(peers)]
    into = [packet(int(p), RC.SELF, int(rng.choice([53, 54, 77])), 1000 + i) for i, p in enumerate(peers)]
    chk = oracle.Filter()
    chk.set_rules([([(RC.ip("100.64.1.2"), 32)], "tcp", [(1000, 1000 + n // 2)])])
    with Context(max_keypairs=1, flow_capacity=1 << 12) as c:
        c.acl_set(True, flatten_rules([CompiledRule(srcs=["100.64.1.2/32"], proto="tcp", ports=[PortRange(1000, 1000 + n // 2)])]))
        for inbound, pkts in ((False, out), (True, into)):
            order = rng.permutation(n)
            off, at = np.zeros(n, np.uint32), 0
            for i in order:
                off[i] = at
                at += 16 + ((len(pkts[i]) + 15) & ~15) + 16 * int(rng.integers(0, 9))
            ring = at - int(at - off[order[-1]] - 16 - ((len(pkts[order[-1]]) + 15) & ~15))  # the last packet ends where the ring does
            b = c.batch(n, ring)
            for i in range(n):
                b.ring[int(off[i]) + 16:int(off[i]) + 16 + len(pkts[i])] = np.frombuffer(pkts[i], np.uint8)
            wrong = rng.random(n) < 0.05
            bad = np.where(rng.random(n) < 0.5, off + 4, ring & 0xFFFFFFF0).astype(np.uint32)  # misplaced, or nothing behind it
            b.off[:], b.len[:] = np.where(wrong, bad, off), [len(p) for p in pkts]
            if inbound:
                b.filter_check(n, RC.T0 + 1)
                want = np.array([not w and chk.check_inbound(p, RC.T0 + 1) for w, p in zip(wrong, pkts)])
                assert np.array_equal(b.status == 0, want), np.flatnonzero((b.status == 0) != want)[:5]
                assert n < 500 or 0.1 * n < want.sum() < 0.5 * n  # a sixth replies, a sixteenth by the rule
            else:
                b.filter_note(n, RC.T0)
                for w, p in zip(wrong, pkts):
                    if not w:
                        chk.note_outbound(p, RC.T0)
            assert flows_equal(c.flows_export(), chk.flows())
            b.close()


@pytest.mark.parametrize("n", [1, 1025, 16385, 49153])
def test_packets_close_together_where_nothing_is_read_in_place(gpu_lib, oracle, n, monkeypatch):
    """The copies that bring heads up when pinned memory may not be read by the kernels."""
    monkeypatch.setenv("BNK_HOST_DIRECT_BYTES", "0")
    if n > 1:
        return test_packets_close_together_go_up_stretch_by_stretch(gpu_lib, oracle, n, True)
    for k in (1, 511, 799):
        test_heads_of_packets_anywhere_in_the_ring(gpu_lib, oracle, k)
