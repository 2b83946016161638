// Device side of the packet filter: the parser, the rule match and the reply-flow table (filter.Filter's f.flows,
// internal/filter/filter.go:26-38 of the reference), shared by the filter kernels and by the seal and open kernels
// that do their packets' filter work in passing.
//
// Flows.  Go's map[flowKey]time.Time becomes three open-addressing tables (tcp, udp, icmp) keyed by remote address | remote
// port | local port, claimed with a 64-bit compare-and-swap.  A deleted entry keeps its key with expiry FLOW_DEAD,
// which behaves like an absent key for every later lookup.  The live-entry count is kept exactly because the
// reference's expiry sweep depends on len(flows) > 4096.
#pragma once

#include <climits>

#include "bnk_internal.cuh"

constexpr unsigned long long FLOW_EMPTY = ~0ull;
constexpr long long FLOW_DEAD = LLONG_MIN;      // the key is there, the entry is deleted
constexpr long long FLOW_FRESH = LLONG_MIN + 1; // expiry of a slot no key has used yet
__host__ __device__ __forceinline__ bool flow_absent(long long exp) { return exp <= FLOW_FRESH; }
constexpr long long TTL_UDP = 30ll * 1000000000ll;  // filter.go:19
constexpr long long TTL_TCP = 120ll * 1000000000ll; // filter.go:20
constexpr long long TTL_ICMP = 30ll * 1000000000ll; // filter.go:21
constexpr long long TTL_LEAST = FlowBounds::kTtlLeast;
constexpr unsigned long long SWEEP_THRESHOLD = FlowBounds::kSweepThreshold;

// small device-side control block behind FilterTables::flow_live
struct FlowCtl {
    FlowReport rep;             // live count, floor of the expiries, overflow flag, per-class slot counts
    unsigned long long dropped; // entries the sweep under way has deleted
    long long next_floor;       // lowest expiry it has left
    uint32_t ticket;            // CTAs of the sweep that have finished
    uint32_t decided;           // 2: the sweep under way walks the table, 1: it does not, 0: no CTA has looked yet
    uint32_t moved;             // entries a compaction has re-inserted so far
};
__device__ __forceinline__ FlowCtl *flow_ctl(const FilterTables &ft) { return reinterpret_cast<FlowCtl *>(ft.flow_live); }

// Place of a flow key: the halves are spread by odd factors and finished in 32 bits (a 64-bit finaliser costs three
// times the instructions on a machine without a 64-bit multiplier).
__host__ __device__ __forceinline__ uint32_t flow_hash(uint64_t key) {
    uint32_t x = (uint32_t)(key >> 32) * 0x9e3779b1u ^ (uint32_t)key * 0x85ebca6bu;
    x ^= x >> 15;
    x *= 0x2c1b3c6du;
    x ^= x >> 12;
    x *= 0x297a2d39u;
    return x ^ (x >> 15);
}

struct Parsed {
    uint32_t src, dst;
    uint16_t sport, dport;
    uint8_t proto;
};
// filter.go:71-106 in two steps, so that the caller can fetch the ports from wherever it has them: w0..w4 are the first
// twenty bytes (present when len >= 20); returns the byte offset of the ports, 0 when none are needed, or
// kParseBad for a packet that does not parse.
constexpr uint32_t kParseBad = 0xffffffffu;
__device__ __forceinline__ uint32_t parse_ipv4_words(uint32_t w0, uint32_t w2, uint32_t w3, uint32_t w4, uint32_t len, Parsed &out) {
    if (len < 20) return kParseBad;
    if (((w0 & 0xffu) >> 4) != 4u) return kParseBad;
    const uint32_t ihl = (w0 & 0x0fu) * 4u;
    if (ihl < 20u || len < ihl) return kParseBad;
    out.proto = (uint8_t)((w2 >> 8) & 0xffu); // byte 9
    out.src = __byte_perm(w3, 0, 0x0123);     // bytes 12..15, big-endian
    out.dst = __byte_perm(w4, 0, 0x0123);
    out.sport = 0;
    out.dport = 0;
    const uint32_t body = len - ihl;
    if (out.proto == 6 || out.proto == 17) return body < 4 ? kParseBad : ihl; // ihl is a multiple of 4
    if (out.proto == 1) return body >= 1 ? 0u : kParseBad;
    return kParseBad;
}
__device__ __forceinline__ void parse_ports(uint32_t ports, Parsed &out) {
    out.sport = (uint16_t)(((ports & 0xffu) << 8) | ((ports >> 8) & 0xffu));
    out.dport = (uint16_t)((((ports >> 16) & 0xffu) << 8) | (ports >> 24));
}

__device__ __forceinline__ int proto_class(uint8_t proto) { return proto == 6 ? 0 : (proto == 17 ? 1 : 2); }
__device__ __forceinline__ long long flow_ttl(uint8_t proto) { // filter.go:108-117
    return proto == 6 ? TTL_TCP : (proto == 1 ? TTL_ICMP : TTL_UDP);
}
__device__ __forceinline__ unsigned long long flow_key(uint32_t remote, uint16_t rport, uint16_t lport) {
    return ((unsigned long long)remote << 32) | ((unsigned long long)rport << 16) | lport;
}

// One atomic per group of lanes that add to the same counter at the same point of the code, instead of one per
// lane: a batch of new flows otherwise sends a few hundred thousand atomics to two addresses (300,000 fresh flows
// took 0.7 ms that way).
template <typename T>
__device__ __forceinline__ void add_one_aggregated(T *counter) {
    const unsigned same = __match_any_sync(__activemask(), (unsigned long long)(uintptr_t)counter);
    if ((threadIdx.x & 31u) == (unsigned)(__ffs(same) - 1)) atomicAdd(counter, (T)__popc(same));
}
// No entry expires before rep.floor: whoever writes an expiry below it lowers it (rare: a fresh expiry lies at least
// the shortest lifetime ahead, and the floor is where the oldest entry stood at the last sweep).
__device__ __forceinline__ long long flow_floor(const FlowCtl *ctl) { return *(const volatile long long *)&ctl->rep.floor; }
__device__ __forceinline__ void flow_keep_floor(FlowCtl *ctl, long long exp, long long floor) {
    if (exp < floor) atomicMin(&ctl->rep.floor, exp);
}

// NoteOutbound (filter.go:189-209) of one flow by one thread, in three steps that each start with what the step
// before has asked memory for, so that a caller can do other work in between.
struct FlowNote {
    unsigned long long key = FLOW_EMPTY, old = FLOW_EMPTY;
    long long exp = 0, prev = 0;
    uint32_t h = 0;
    int cls = -1; // -1: nothing to note
    bool placed = false;

    __device__ __forceinline__ void begin(const FilterTables &ft, const Parsed &p, long long now) {
        cls = proto_class(p.proto);
        exp = now + flow_ttl(p.proto);
        key = flow_key(p.dst, p.dport, p.sport);
        h = flow_hash(key) & (ft.flow_capacity - 1);
        if (key != FLOW_EMPTY)
            old = atomicCAS(&ft.flow_slots[flow_region(ft, cls) + h].key, FLOW_EMPTY, key);
    }
    __device__ __forceinline__ void place(const FilterTables &ft) {
        if (cls < 0) return;
        if (key == FLOW_EMPTY) {
            prev = (long long)atomicExch((unsigned long long *)&ft.flow_special_exp[cls], (unsigned long long)exp);
            placed = true;
            return;
        }
        FlowSlot *const slots = ft.flow_slots + flow_region(ft, cls);
        for (uint32_t probe = 1; old != FLOW_EMPTY && old != key; probe++) {
            if (probe >= ft.flow_capacity) { // table full: the flow is not recorded, the host reports BNK_EFULL
                atomicAdd(&flow_ctl(ft)->rep.error, 1);
                return;
            }
            h = (h + 1) & (ft.flow_capacity - 1);
            old = atomicCAS(&slots[h].key, FLOW_EMPTY, key);
        }
        prev = (long long)atomicExch((unsigned long long *)&slots[h].exp, (unsigned long long)exp);
        placed = true;
    }
    __device__ __forceinline__ void count(const FilterTables &ft) {
        if (!placed) return;
        FlowCtl *const ctl = flow_ctl(ft);
        if (key != FLOW_EMPTY && old == FLOW_EMPTY) add_one_aggregated(&ctl->rep.used[cls]);
        if (flow_absent(prev)) add_one_aggregated(&ctl->rep.live);
        if (key != FLOW_EMPTY && prev == FLOW_DEAD) atomicSub(&ctl->rep.dead[cls], 1u); // a deleted entry is back
        flow_keep_floor(ctl, exp, flow_floor(ctl));
    }
};

// The state of the table after a batch, for the host (one thread, when all the batch's filter work is visible).
__device__ __forceinline__ void flow_report(const FlowCtl *ctl, FlowReport *host) {
    const volatile FlowReport *const r = &ctl->rep;
    FlowReport v;
    v.live = r->live;
    v.floor = r->floor;
    v.error = r->error;
    for (int c = 0; c < 3; c++) {
        v.used[c] = r->used[c];
        v.dead[c] = r->dead[c];
    }
    *host = v;
}

// ---- rules ----
// acl.CompiledRule.Match (acl.go:149-172) for every rule: a packet is allowed if any prefix that contains its source has
// an allowance for its protocol and port.  The longest such prefix is found directly: a table by the upper 16 address
// bits, where something longer than 16 exists in such a stretch a block by the next 8, and for prefixes longer than
// 24 a hash table, probed only for the lengths that occur among the 256 addresses around the packet's.  Every prefix
// names the next shorter one that contains it, so the others are reached without a further search.  Port ranges of a
// prefix are merged when the table is built.
// (Before: a probe of one hash table per prefix length in use and a walk over each match's allowances: ~2,300 warp
// instructions per warp at 10,000 rules, and 20 us for a packet whose source has a hundred rules.)
constexpr uint32_t kRuleBlock = 1u << 31; // in rule_top: a block follows; otherwise a group + 1 or 0
__host__ __device__ __forceinline__ uint32_t rule_hash(uint32_t addr, uint32_t len) { // a 32-bit finaliser
    uint32_t x = addr ^ (len * 0x9e3779b1u);
    x ^= x >> 16;
    x *= 0x85ebca6bu;
    x ^= x >> 13;
    x *= 0xc2b2ae35u;
    return x ^ (x >> 16);
}
// A block's entry says in bits 0 to 7 which lengths beyond 24 occur among its 256 addresses, and in the others that one of the single
// addresses has this remainder: with three or four of them a search in vain is spared seven times of eight.
__host__ __device__ __forceinline__ uint32_t rule_single_bit(uint32_t addr) { return 8u + (addr & 255u) % 24u; }
__host__ __device__ __forceinline__ uint32_t prefix_mask(uint32_t len) { return len == 0 ? 0u : 0xffffffffu << (32 - len); }
__device__ __forceinline__ bool port_in(uint32_t range, uint32_t port) { return port >= (range >> 16) && port <= (range & 0xffffu); }
__device__ __forceinline__ bool port_in_any(const uint32_t *ranges, uint32_t n, uint32_t port) {
    if (n <= 4) {
        const uint4 r = *reinterpret_cast<const uint4 *>(ranges);
        return port_in(r.x, port) || port_in(r.y, port) || port_in(r.z, port) || port_in(r.w, port);
    }
    uint32_t lo = 0, hi = n; // first range that starts beyond the port
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if ((ranges[mid] >> 16) <= port) lo = mid + 1;
        else hi = mid;
    }
    return lo > 0 && port <= (ranges[lo - 1] & 0xffffu);
}
struct GroupRead { // a RuleGroup in one 32-byte load
    uint32_t addr, len, parent, n_ports, tcp_at, udp_at, tcp0, udp0;
    __device__ __forceinline__ void from(const RuleGroup *g) {
        asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(addr), "=r"(len), "=r"(parent), "=r"(n_ports), "=r"(tcp_at), "=r"(udp_at), "=r"(tcp0), "=r"(udp0)
                     : "l"(__cvta_generic_to_global(g)));
    }
};
__device__ __forceinline__ bool rules_allow(const FilterTables &ft, const Parsed &p) {
    if (ft.rule_top == nullptr) return false;
    // Most policies name single addresses, so the first place that one could have in the table is asked for beside the top table,
    // and an entry is one load: 1,000,000 headers against 40,000 allowances checked in 47.9 us instead of 51.9, and with a block's
    // entry saying which single addresses there may be 46.9.  (The ranges of the prefixes around folded into a prefix's own saved
    // 0.8 us more; flows looked up in pairs, 32 bytes a load, 0.3; headers fetched ahead into L2 cost 3.)
    GroupRead e;
    uint32_t h = rule_hash(p.src, 32u) & ft.rule_long_mask;
    uint32_t g = ft.rule_top[p.src >> 16];
    e.from(&ft.rule_long[h]);
    bool have = false;
    if (g & kRuleBlock) {
        const uint2 blk = ft.rule_blocks[(size_t)(g & ~kRuleBlock) * 256u + ((p.src >> 8) & 255u)];
        g = blk.x;
        const bool single = (blk.y >> rule_single_bit(p.src)) & 1u;
        for (uint32_t lens = blk.y & (single ? 0xffu : 0x7fu); lens && !have;) { // bit k: prefixes of length 25 + k
            const uint32_t k = 31u - (uint32_t)__clz((int)lens), len = 25u + k, addr = p.src & prefix_mask(len);
            lens ^= 1u << k;
            if (len != 32u) {
                h = rule_hash(addr, len) & ft.rule_long_mask;
                e.from(&ft.rule_long[h]);
            }
            for (;;) { // it has empty places
                have = e.addr == addr && e.len == len;
                if (have || e.len == 0) break;
                h = (h + 1) & ft.rule_long_mask;
                e.from(&ft.rule_long[h]);
            }
        }
    }
    const bool tcp = p.proto == 6;
    for (;;) {
        if (!have) {
            if (g == 0) return false;
            e.from(&ft.rule_groups[g - 1]);
        }
        have = false;
        if (p.proto == 1) {
            if (e.parent >> 31) return true;
        } else {
            const uint32_t n = tcp ? e.n_ports & 0xffffu : e.n_ports >> 16;
            if (port_in(tcp ? e.tcp0 : e.udp0, p.dport)) return true;
            if (n > 1 && port_in_any(ft.rule_ports + (tcp ? e.tcp_at : e.udp_at), n, p.dport)) return true;
        }
        g = e.parent & 0x7fffffffu;
    }
}
// The reply-flow half of CheckInbound: is the packet the reply to a flow that is alive (the key mirrors NoteOutbound's)?
// In two steps, so that the first can wait for memory beside the search of the rules.
struct FlowReply {
    unsigned long long key, k;
    long long exp, *place;
    uint32_t h;
    int cls;

    __device__ __forceinline__ void begin(const FilterTables &ft, const Parsed &p) {
        cls = proto_class(p.proto);
        key = flow_key(p.src, p.sport, p.dport);
        h = flow_hash(key) & (ft.flow_capacity - 1);
        k = FLOW_EMPTY;
        exp = FLOW_FRESH;
        place = &ft.flow_special_exp[cls];
        if (ft.flow_capacity == 0) return;
        if (key == FLOW_EMPTY) {
            exp = *(volatile long long *)place;
        } else {
            FlowSlot *const at = ft.flow_slots + flow_region(ft, cls) + h;
            place = &at->exp;
            asm volatile("ld.volatile.global.v2.b64 {%0, %1}, [%2];" : "=l"(k), "=l"(exp) : "l"(__cvta_generic_to_global(at)));
        }
    }
    __device__ __forceinline__ uint8_t finish(const FilterTables &ft, uint8_t proto, long long now) {
        if (key != FLOW_EMPTY && k != key) {
            FlowSlot *const slots = ft.flow_slots + flow_region(ft, cls);
            exp = FLOW_FRESH;
            for (uint32_t probe = 1; k != FLOW_EMPTY && probe < ft.flow_capacity; probe++) {
                h = (h + 1) & (ft.flow_capacity - 1);
                k = slots[h].key;
                if (k == key) {
                    place = &slots[h].exp;
                    exp = *(volatile long long *)place;
                    break;
                }
            }
        }
        if (flow_absent(exp)) return BNK_PKT_FILTER_DENY;
        FlowCtl *const ctl = flow_ctl(ft);
        if (now < exp) { // strict: time.Before
            const long long fresh = now + flow_ttl(proto);
            *(volatile long long *)place = fresh; // keep-alive on traffic
            // The floor may come from L1, one word for all warps: a sweep that raises it meanwhile leaves it below `fresh`.
            flow_keep_floor(ctl, fresh, ctl->rep.floor);
            return BNK_PKT_OK;
        }
        // (not if another batch has recorded the flow again meanwhile)
        if ((long long)atomicCAS((unsigned long long *)place, (unsigned long long)exp, (unsigned long long)FLOW_DEAD) == exp) {
            atomicAdd(&ctl->rep.live, 0ull - 1ull);
            if (key != FLOW_EMPTY) atomicAdd(&ctl->rep.dead[cls], 1u);
        }
        return BNK_PKT_FILTER_DENY;
    }
};
// CheckInbound (filter.go:121-147) of a packet that parses, with enforcement on: a rule allows it, or it is a reply.
__device__ __forceinline__ uint8_t filter_verdict(const FilterTables &ft, const Parsed &p, long long now) {
    FlowReply reply;
    reply.begin(ft, p);
    if (rules_allow(ft, p)) return BNK_PKT_OK;
    return reply.finish(ft, p.proto, now);
}

// ---- the last word on an opened packet ----
// What the open kernel notes of a plaintext's headers is all that the checks behind the replay
// window need, so that they do not go back to the packet: over the host link that would be a read per packet.
//   x source address   y source port << 16 | destination port   z protocol | flags   w IPv4 total length
constexpr uint32_t kInnerParses = 1u << 8; // filter.parse accepts it
constexpr uint32_t kInnerWhole = 1u << 9;  // IPv4, 20 <= total length <= decrypted length
constexpr uint32_t kInnerJudged = 1u << 10, kInnerAllowed = 1u << 11; // the rules have been asked already, and allow it
struct VerdictArgs {
    FilterTables ft;
    const uint4 *inner;
    const uint32_t *slot;
    const uint32_t *allowed_ip;
    uint8_t *status;
    uint32_t *out_len;
    uint8_t *host_status; // the results' pinned arrays, written besides
    uint32_t *host_out_len;
    long long now;
    uint32_t n;
    bool inner_check, check_inbound;
};
__device__ __forceinline__ Parsed inner_parsed(const uint4 &h) {
    Parsed p;
    p.src = h.x;
    p.dst = 0;
    p.sport = (uint16_t)(h.y >> 16);
    p.dport = (uint16_t)h.y;
    p.proto = (uint8_t)h.z;
    return p;
}
// The last checks of packet i, which has been opened, as far as they leave no trace: its status and length, and whether it still
// depends on its flow (reply.finish).
__device__ __forceinline__ void checks_begin(const VerdictArgs &v, uint32_t i, uint32_t slot, uint8_t &found, uint32_t &len, uint8_t &proto,
                                             FlowReply &reply, bool &ask_flows) {
    found = BNK_PKT_OK;
    if (!v.inner_check && !v.check_inbound) return;
    const uint4 h = v.inner[i];
    const uint32_t allowed_ip = v.inner_check ? v.allowed_ip[slot] : 0u;
    proto = (uint8_t)h.z;
    if (v.check_inbound && v.ft.enforce) {
        if (h.z & kInnerParses) {
            const Parsed p = inner_parsed(h);
            reply.begin(v.ft, p);
            ask_flows = !((h.z & kInnerJudged) ? (h.z & kInnerAllowed) != 0 : rules_allow(v.ft, p));
        } else {
            found = BNK_PKT_FILTER_DENY;
        }
    }
    if (v.inner_check) { // cut to the IPv4 total length; the source must be the peer's address
        if ((h.z & kInnerWhole) && h.x != 0 && h.x == allowed_ip) {
            len = h.w;
        } else {
            found = BNK_PKT_BAD_INNER;
            ask_flows = false;
        }
    }
}
__device__ __forceinline__ void final_verdict(const VerdictArgs &v, uint32_t i) {
    uint8_t st = *(volatile uint8_t *)&v.status[i];
    uint32_t l = v.out_len[i];
    if (st == BNK_PKT_OK && (v.inner_check || v.check_inbound)) {
        uint8_t proto = 0;
        FlowReply reply;
        bool ask_flows = false;
        checks_begin(v, i, v.inner_check ? v.slot[i] : 0u, st, l, proto, reply, ask_flows);
        if (ask_flows) st = reply.finish(v.ft, proto, v.now);
        v.status[i] = st;
        v.out_len[i] = l;
    }
    if (v.host_status) {
        v.host_status[i] = st;
        v.host_out_len[i] = l;
    }
}
