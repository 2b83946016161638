// ACL packet filter for sm_100a: the per-packet work of filter.Filter
// (internal/filter/filter.go of the reference) and acl.CompiledRule.Match
// (internal/acl/acl.go:149-172), one thread per packet.
//
// Rules.  The reference scans every rule for every packet.  The verdict is an OR over rules, so scan order is free;
// here the flattened allowances (prefix, proto, port range) are grouped by prefix and the prefixes are indexed
// (filter_device.cuh).
//
// Flows: see filter_device.cuh.
// Go deletes map entries (filter.go:144, 202-208), so its map is bounded by the live
// flows; here deleted entries are counted per class, and once they fill a quarter of
// a class's region the surviving entries are re-inserted into the class's second,
// empty region and the two swap roles (filter_flows_maintain), between two batches.
#include <algorithm>
#include <cstring>
#include <vector>

#include "filter_device.cuh"

namespace {

// filter.go:71-106 of the packet at ring[o + 16 .. o + 16 + len), which has to lie in the ring.  Its first 32 bytes, which
// hold all of a packet without IP options, are asked for together: when the ring is in host memory a dependent read is
// another trip over the link (8192 whole packets noted and checked: 95 us with three dependent reads, 87 with one).
__device__ __forceinline__ bool parse_ipv4(const uint8_t *ring, uint32_t o, uint32_t len, uint64_t ring_bytes, Parsed &out) {
    if ((o & 15u) || (uint64_t)o + 16u + len > ring_bytes || len < 20) return false;
    const uint8_t *const p = ring + o + 16; // 16-byte aligned
    const bool both = (uint64_t)o + 48 <= ring_bytes;
    const uint4 a = *reinterpret_cast<const uint4 *>(p);
    uint4 b = make_uint4(0, 0, 0, 0);
    if (both) b = *reinterpret_cast<const uint4 *>(p + 16);
    else b.x = *reinterpret_cast<const uint32_t *>(p + 16);
    const uint32_t at = parse_ipv4_words(a.x, a.z, a.w, b.x, len, out);
    if (at == kParseBad) return false;
    if (at) parse_ports(both && at == 20 ? b.y : *reinterpret_cast<const uint32_t *>(p + at), out);
    return true;
}
// The same for a packet per lane (`have`: the lane has one), by all lanes of a warp: two lanes ask for a packet's two 16-byte
// halves in one instruction, so that halves in different sectors of one line are one request to the link all the same; a
// lane that asks for both makes two of them.  8192 whole packets noted and checked (two calls) 98 -> 76 us, 16,000 x 400 B
// 158 -> 106.  A ring on the device (1,000,000 headers 47.4 us, with pairs 48.3) and few packets (60 noted and checked 32.9
// us, 33.9) are not bound by requests, and the exchange between the lanes costs.  (One parser for both, taking the two
// halves, made the plain kernels up to 1 us slower on a few packets: those keep the code above.)
constexpr uint32_t kPairsFrom = 512;
struct HeadStage { // of one warp
    uint4 half[32][2];
};
__device__ __forceinline__ bool parse_ipv4_pairs(HeadStage &stage, const uint8_t *ring, bool have, uint32_t o, uint32_t len, uint64_t ring_bytes,
                                                 Parsed &out) {
    // (offsets and the ring's size are multiples of 16, so 20 bytes in the ring behind o + 16 are 32)
    have = have && !(o & 15u) && (uint64_t)o + 16u + len <= ring_bytes && len >= 20;
    const uint32_t lane = threadIdx.x & 31u, with = __ballot_sync(0xffffffffu, have);
    uint4 v[2];
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
        const uint32_t p = 16u * h + (lane >> 1), at = __shfl_sync(0xffffffffu, o, p);
        v[h] = make_uint4(0, 0, 0, 0);
        if ((with >> p) & 1u) v[h] = *reinterpret_cast<const uint4 *>(ring + at + 16u + 16u * (lane & 1u)); // 16-byte aligned
    }
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) stage.half[16u * h + (lane >> 1)][lane & 1u] = v[h];
    __syncwarp();
    if (!have) return false;
    const uint4 a = stage.half[lane][0], b = stage.half[lane][1];
    const uint32_t at = parse_ipv4_words(a.x, a.z, a.w, b.x, len, out);
    if (at == kParseBad) return false;
    if (at) parse_ports(at == 20 ? b.y : *reinterpret_cast<const uint32_t *>(ring + o + 16u + at), out);
    return true;
}

// ---- NoteOutbound, filter.go:189-209 ----------------------------------------------------
template <bool PAIRS>
__global__ void __launch_bounds__(128) filter_note_kernel(const __grid_constant__ FilterTables ft, const uint8_t *ring, const uint32_t *off,
                                   const uint32_t *len, uint32_t n, uint64_t ring_bytes, long long now, FlowReport *report, Done done) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    Parsed p;
    bool parses;
    if constexpr (PAIRS) {
        __shared__ HeadStage heads[4];
        parses = parse_ipv4_pairs(heads[threadIdx.x >> 5], ring, i < n, i < n ? off[i] : 0u, i < n ? len[i] : 0u, ring_bytes, p);
    } else {
        parses = i < n && parse_ipv4(ring, off[i], len[i], ring_bytes, p);
    }
    if (parses) {
        FlowNote note;
        note.begin(ft, p, now);
        note.place(ft);
        note.count(ft);
    }
    signal_done(done, report != nullptr, [&] { flow_report(flow_ctl(ft), report); });
}

// The reference sweeps expired flows whenever the map holds more than 4096 entries after an insert.  Within one batch
// (one `now`) that equals: insert everything, then sweep once if the count exceeds the threshold.  A sweep that
// starts at or before the floor of the expiries would find nothing and does not walk the table; the host, which
// knows a lower bound of the floor, does not even launch it (flow_note_begins).  One walk reads the expiries of the
// regions in use and leaves the floor at the lowest expiry it has seen, or at `beside`, which is what inserts and lookups
// that run beside it write at least.  Sweeps never run side by side (launch_flow_sweep); inserts and lookups may, so an
// entry is dropped only if it still is the one that was looked at.
__global__ void __launch_bounds__(256) filter_sweep_kernel(const __grid_constant__ FilterTables ft, long long now, long long beside,
                                                           FlowReport *report, Done done) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    FlowCtl *const ctl = flow_ctl(ft);
    __shared__ unsigned long long dropped_s;
    __shared__ long long floor_s;
    __shared__ uint32_t dead_s[3];
    __shared__ bool walk_s;
    if (threadIdx.x == 0) { // the first CTA to look decides for all: others insert and count meanwhile
        const uint32_t mine = *(volatile unsigned long long *)&ctl->rep.live > SWEEP_THRESHOLD && now > flow_floor(ctl) ? 2u : 1u;
        const uint32_t first = atomicCAS(&ctl->decided, 0u, mine);
        walk_s = (first ? first : mine) == 2u;
        dropped_s = 0;
        floor_s = LLONG_MAX;
        dead_s[0] = dead_s[1] = dead_s[2] = 0;
    }
    __syncthreads();
    const bool walk = walk_s;
    if (walk) {
        const size_t cap = ft.flow_capacity, total = 3 * cap;
        unsigned long long dropped = 0;
        long long floor = LLONG_MAX;
        for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < total + 3; k += (size_t)gridDim.x * blockDim.x) {
            const int cls = k < total ? (int)(k / cap) : 0;
            long long *const e = k < total ? &ft.flow_slots[flow_region(ft, cls) + (k - cls * cap)].exp : &ft.flow_special_exp[k - total];
            const long long exp = *e;
            if (flow_absent(exp)) continue;
            if (now > exp) {
                if ((long long)atomicCAS((unsigned long long *)e, (unsigned long long)exp, (unsigned long long)FLOW_DEAD) != exp) continue;
                dropped++;
                if (k < total) atomicAdd(&dead_s[cls], 1u);
            } else if (exp < floor) {
                floor = exp;
            }
        }
        if (dropped) atomicAdd(&dropped_s, dropped);
        atomicMin(&floor_s, floor);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (walk) {
            atomicAdd(&ctl->dropped, dropped_s);
            atomicMin(&ctl->next_floor, floor_s);
            for (int c = 0; c < 3; c++)
                if (dead_s[c]) atomicAdd(&ctl->rep.dead[c], dead_s[c]);
        }
        __threadfence();
        if (atomicAdd(&ctl->ticket, 1u) + 1u == gridDim.x) {
            __threadfence();
            if (walk) {
                atomicAdd(&ctl->rep.live, 0ull - *(volatile unsigned long long *)&ctl->dropped);
                const long long seen = *(volatile long long *)&ctl->next_floor;
                ctl->rep.floor = seen < beside ? seen : beside;
                ctl->dropped = 0;
                ctl->next_floor = LLONG_MAX;
            }
            ctl->ticket = ctl->decided = 0;
            __threadfence();
            if (report) flow_report(ctl, report);
            if (done.flag) {
                __threadfence_system();
                *(volatile uint32_t *)done.flag = done.value;
            }
        }
    }
}

// ---- CheckInbound, filter.go:121-147 -----------------------------------------------------
// only_status_ok: packets whose status is not BNK_PKT_OK are left alone (open pipeline).  host_status (may be null): the
// results' pinned array, which gets a CTA's 128 statuses as one line: 1,000,000 of them cost 20 us of link time beside
// the checks instead of a copy of 27 us behind them.
template <bool PAIRS>
__global__ void __launch_bounds__(128) filter_check_kernel(const __grid_constant__ FilterTables ft, const uint8_t *ring, const uint32_t *off,
                                    const uint32_t *len, uint8_t *status, uint32_t n, uint64_t ring_bytes,
                                    long long now, int only_status_ok, uint8_t *host_status, Done done) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ uint32_t line[32];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool have = i < n && !(only_status_ok && status[i] != BNK_PKT_OK);
    uint8_t verdict = BNK_PKT_OK; // filter.go:124-126: allow-all passes even unparseable packets
    if constexpr (PAIRS) {
        __shared__ HeadStage heads[4];
        Parsed p;
        if (ft.enforce && !parse_ipv4_pairs(heads[threadIdx.x >> 5], ring, have, have ? off[i] : 0u, have ? len[i] : 0u, ring_bytes, p))
            verdict = BNK_PKT_FILTER_DENY;
        else if (ft.enforce)
            verdict = filter_verdict(ft, p, now);
    }
    if (have) {
        if constexpr (!PAIRS) {
            Parsed p;
            if (ft.enforce)
                verdict = parse_ipv4(ring, off[i], len[i], ring_bytes, p) ? filter_verdict(ft, p, now) : (uint8_t)BNK_PKT_FILTER_DENY;
        }
        status[i] = verdict;
        reinterpret_cast<uint8_t *>(line)[threadIdx.x] = verdict;
    }
    if (host_status) {
        __syncthreads();
        const uint32_t first = blockIdx.x * blockDim.x + 4u * threadIdx.x;
        if (threadIdx.x < 32) {
            if (first + 4u <= n) *reinterpret_cast<uint32_t *>(host_status + first) = line[threadIdx.x];
            else
                for (uint32_t k = first; k < n; k++) host_status[k] = reinterpret_cast<uint8_t *>(line)[4u * threadIdx.x + (k - first)];
        }
    }
    signal_done(done, false, [] {});
}

__global__ void flows_fill_kernel(FilterTables ft) {
    const size_t total = (size_t)6 * ft.flow_capacity;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < total; k += (size_t)gridDim.x * blockDim.x) {
        ft.flow_slots[k] = FlowSlot{FLOW_EMPTY, FLOW_FRESH};
    }
    if (blockIdx.x == 0 && threadIdx.x < 3) ft.flow_special_exp[threadIdx.x] = FLOW_FRESH;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        FlowCtl v{};
        v.rep.floor = v.next_floor = LLONG_MAX;
        *flow_ctl(ft) = v;
    }
}

// ---- compaction: the entries of class `cls` that are not deleted move from the region in use to the class's
// other region, which is empty; the host then swaps the roles (filter_flows_maintain).  Expired entries that no
// sweep or lookup has deleted yet move along: they still count in len(f.flows), which decides the next sweep.
__global__ void flows_compact_kernel(FilterTables ft, int cls) {
    FlowCtl *ctl = flow_ctl(ft);
    const size_t from = flow_region(ft, cls), to = ((size_t)cls * 2 + (ft.flow_half[cls] ^ 1)) * ft.flow_capacity;
    FlowSlot *const slots = ft.flow_slots + to;
    uint32_t moved = 0;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < ft.flow_capacity; k += (size_t)gridDim.x * blockDim.x) {
        const unsigned long long key = ft.flow_slots[from + k].key;
        const long long exp = ft.flow_slots[from + k].exp;
        if (key == FLOW_EMPTY || flow_absent(exp)) continue;
        uint32_t h = flow_hash(key) & (ft.flow_capacity - 1);
        bool placed = false; // the target region starts empty and takes fewer entries than it has slots
        for (uint32_t probe = 0; probe < ft.flow_capacity && !placed; probe++) {
            if (atomicCAS(&slots[h].key, FLOW_EMPTY, key) == FLOW_EMPTY) placed = true;
            else h = (h + 1) & (ft.flow_capacity - 1);
        }
        if (!placed) {
            atomicAdd(&ctl->rep.error, 1);
            continue;
        }
        slots[h].exp = exp;
        moved++;
    }
    if (moved) atomicAdd(&ctl->moved, moved);
}
// wipes the region the class has just left and books the move
__global__ void flows_compact_finish_kernel(FilterTables ft, int cls) {
    FlowCtl *ctl = flow_ctl(ft);
    const size_t from = flow_region(ft, cls);
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < ft.flow_capacity; k += (size_t)gridDim.x * blockDim.x) {
        ft.flow_slots[from + k] = FlowSlot{FLOW_EMPTY, FLOW_FRESH};
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctl->rep.used[cls] = ctl->moved; // the kernel in front has finished: the count is final
        ctl->rep.dead[cls] = 0;
        ctl->moved = 0;
    }
}

// ---- per-batch counters (BNK_F_STATS): statuses and output bytes of the first n packets.  Every CTA adds its
// share to the device accumulators; the CTA that finishes last hands the totals to the host struct and leaves
// the accumulators zero for the next launch.
__global__ void __launch_bounds__(256) tally_kernel(const uint8_t *status, const uint32_t *out_len, uint32_t n,
                                                    unsigned long long *acc /* [16] statuses, [16] bytes, [17] ticket */,
                                                    bnk_batch_stats *host_out) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ unsigned int cnt[16];
    __shared__ unsigned long long bytes_s;
    __shared__ bool last;
    if (threadIdx.x < 16) cnt[threadIdx.x] = 0;
    if (threadIdx.x == 0) bytes_s = 0;
    __syncthreads();
    unsigned long long bytes = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint8_t st = status[i];
        add_one_aggregated(&cnt[st & 15u]); // nearly every lane hits the same bin
        if (st == BNK_PKT_OK) bytes += out_len[i];
    }
    for (int o = 16; o > 0; o >>= 1) bytes += __shfl_down_sync(0xffffffffu, bytes, o);
    if ((threadIdx.x & 31) == 0 && bytes) atomicAdd(&bytes_s, bytes);
    __syncthreads();
    if (threadIdx.x < 16 && cnt[threadIdx.x]) atomicAdd(&acc[threadIdx.x], (unsigned long long)cnt[threadIdx.x]);
    if (threadIdx.x == 0 && bytes_s) atomicAdd(&acc[16], bytes_s);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&acc[17], 1ull) + 1 == gridDim.x;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < 16) {
        host_out->by_status[threadIdx.x] = atomicExch(&acc[threadIdx.x], 0ull);
    } else if (threadIdx.x == 16) {
        host_out->bytes_out = atomicExch(&acc[16], 0ull);
        host_out->packets = n;
        acc[17] = 0;
    }
}

// ---- the rule index, from its prefixes ----
// The host sorts the prefixes by (address, length), which puts every prefix behind those that contain it and the ones of a
// stretch of 65,536 addresses next to each other; what the checks look up is filled in here.  On the host, with the
// blocks copied over, 10,000 prefixes spread over the whole address space took 3.3 ms, most of it for 20 MB of blocks.
struct RuleStretch { // upper 16 address bits under which something longer than 16 exists: its block's number is its place
    uint32_t hi, first, end; // prefixes [first, end)
};
struct RuleBuild {
    const RuleGroup *groups;
    const uint32_t *shorts;      // prefixes of up to 16 bits
    const RuleStretch *stretches;
    uint32_t n_groups, n_shorts, n_stretches;
    uint32_t *top;
    uint2 *blocks;
    RuleGroup *table; // all zero
    uint32_t mask;
};
constexpr uint32_t kTopCtas = 65536 / 256;
// prefix `g` (a number + 1; 0: none) or the next shorter one that contains `addr`
__device__ __forceinline__ uint32_t rule_containing(const RuleGroup *groups, uint32_t g, uint32_t addr) {
    while (g && (addr & prefix_mask(groups[g - 1].len)) != groups[g - 1].addr) g = groups[g - 1].parent & 0x7fffffffu;
    return g;
}
// CTAs [0, kTopCtas): rule_top; then a CTA per block; then the hash table, a thread per prefix
__global__ void __launch_bounds__(256) rule_build_kernel(const __grid_constant__ RuleBuild a) {
    const uint32_t tid = threadIdx.x;
    if (blockIdx.x < kTopCtas) {
        const uint32_t hi = blockIdx.x * 256u + tid, addr = hi << 16;
        uint32_t lo = 0, up = a.n_stretches;
        while (lo < up) {
            const uint32_t mid = (lo + up) / 2;
            if (a.stretches[mid].hi < hi) lo = mid + 1;
            else up = mid;
        }
        if (lo < a.n_stretches && a.stretches[lo].hi == hi) {
            a.top[hi] = kRuleBlock | lo;
            return;
        }
        lo = 0, up = a.n_shorts; // behind the last one that starts here or before
        while (lo < up) {
            const uint32_t mid = (lo + up) / 2;
            if (a.groups[a.shorts[mid]].addr <= addr) lo = mid + 1;
            else up = mid;
        }
        a.top[hi] = lo ? rule_containing(a.groups, a.shorts[lo - 1] + 1, addr) : 0u;
    } else if (blockIdx.x < kTopCtas + a.n_stretches) {
        const uint32_t k = blockIdx.x - kTopCtas;
        const RuleStretch s = a.stretches[k];
        const uint32_t addr = s.hi << 16 | tid << 8;
        uint32_t lo = s.first, up = s.end; // behind the last one at or before this address, of up to 24 bits if at it
        while (lo < up) {
            const uint32_t mid = (lo + up) / 2;
            const RuleGroup &g = a.groups[mid];
            if (g.addr < addr || (g.addr == addr && g.len <= 24)) lo = mid + 1;
            else up = mid;
        }
        const uint32_t x = lo > s.first ? rule_containing(a.groups, lo, addr) : a.groups[s.first].parent & 0x7fffffffu;
        uint32_t lens = 0;
        for (; lo < s.end && a.groups[lo].addr >> 8 == addr >> 8; lo++)
            lens |= 1u << (a.groups[lo].len - 25u) | (a.groups[lo].len == 32u ? 1u << rule_single_bit(a.groups[lo].addr) : 0u);
        a.blocks[(size_t)k * 256u + tid] = make_uint2(x, lens);
    } else {
        const uint32_t i = (blockIdx.x - kTopCtas - a.n_stretches) * 256u + tid;
        if (i >= a.n_groups) return;
        const RuleGroup g = a.groups[i];
        if (g.len <= 24) return;
        const unsigned long long key = (unsigned long long)g.len << 32 | g.addr;
        for (uint32_t h = rule_hash(g.addr, g.len) & a.mask;; h = (h + 1) & a.mask) { // a quarter full at most, and no key twice
            if (atomicCAS(reinterpret_cast<unsigned long long *>(&a.table[h]), 0ull, key) != 0ull) continue;
            uint2 *const rest = reinterpret_cast<uint2 *>(&a.table[h]);
            rest[1] = make_uint2(g.parent, g.n_ports);
            rest[2] = make_uint2(g.tcp_at, g.udp_at);
            rest[3] = make_uint2(g.tcp0, g.udp0);
            return;
        }
    }
}

} // namespace

// Where the parts of a rule index lie in its block of memory: what the host uploads, then what is built from it.
namespace {
struct RuleLayout {
    size_t groups = 0, ports, shorts, stretches, uploaded, top, table, blocks, total;
    RuleLayout(size_t n_blocks, size_t n_slots, size_t n_groups, size_t n_ports) {
        auto room = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
        ports = room(n_groups * sizeof(RuleGroup));
        shorts = ports + room(n_ports * sizeof(uint32_t));
        stretches = shorts + room(n_groups * sizeof(uint32_t));
        uploaded = top = stretches + room(n_blocks * sizeof(RuleStretch));
        table = top + room(65536 * sizeof(uint32_t));
        blocks = table + room(n_slots * sizeof(RuleGroup));
        total = blocks + room(n_blocks * 256 * sizeof(uint2));
    }
};
size_t rule_long_slots(size_t prefixes) { // a quarter full at most: the lanes of a warp wait for the longest of their walks
    size_t n = 4;
    while (n < prefixes * 4) n <<= 1;
    return n;
}
} // namespace

cudaError_t filter_tables_alloc(bnk_ctx *ctx) {
    FilterTables &ft = ctx->ft;
    ft = FilterTables{};
    const uint32_t cap = ctx->cfg.flow_capacity;
    ft.flow_capacity = cap;
    cudaError_t e;
    // one block: control block, special entries, slots
    const size_t head = 512;
    static_assert(sizeof(FlowCtl) <= 256, "control block");
    uint8_t *mem = nullptr;
    if ((e = cudaMalloc(&mem, head + (size_t)6 * cap * sizeof(FlowSlot))) != cudaSuccess) return e;
    ft.flow_live = reinterpret_cast<unsigned long long *>(mem);
    ft.flow_special_exp = reinterpret_cast<long long *>(mem + 256);
    if (cap) ft.flow_slots = reinterpret_cast<FlowSlot *>(mem + head);
    // With a stated rule-table capacity both buffer sets are allocated here, and a rule swap allocates nothing.
    if (const size_t cap_t = ctx->cfg.max_acl_tuples) {
        const size_t bytes = RuleLayout(std::min<size_t>(cap_t, 65536), rule_long_slots(cap_t), cap_t, 4 * cap_t).total;
        for (bnk_ctx::RuleSet &rs : ctx->rule_set) {
            if ((e = cudaMalloc(&rs.mem, bytes)) != cudaSuccess) return e;
            rs.cap = bytes;
        }
    }
    return filter_flows_clear(ctx, ctx->admin_stream);
}

void filter_tables_free(bnk_ctx *ctx) {
    FilterTables &ft = ctx->ft;
    cudaFree(ft.flow_live); // the block's beginning
    for (bnk_ctx::RuleSet &rs : ctx->rule_set) {
        cudaFree(rs.mem);
        for (cudaEvent_t ev : rs.in_use) cudaEventDestroy(ev);
        rs = bnk_ctx::RuleSet{};
    }
    ft = FilterTables{};
}

cudaError_t filter_flows_clear(bnk_ctx *ctx, cudaStream_t s) {
    ctx->ft.flow_half[0] = ctx->ft.flow_half[1] = ctx->ft.flow_half[2] = 0;
    for (auto &h : ctx->flow_dead_hint) h = 0;
    ctx->flow_errors_seen = 0;
    ctx->flow_bounds.set(LLONG_MAX, 0);
    ctx->sweep_now = LLONG_MIN;
    flows_fill_kernel<<<ctx->sm_count * 4, 256, 0, s>>>(ctx->ft);
    ctx->launches += 1;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(s);
}

cudaError_t filter_flow_stats(bnk_ctx *ctx, uint64_t *live, uint32_t used[3], uint32_t dead[3]) {
    FlowCtl ctl;
    cudaError_t e = cudaMemcpy(&ctl, ctx->ft.flow_live, sizeof ctl, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return e;
    *live = ctl.rep.live;
    for (int c = 0; c < 3; c++) {
        used[c] = ctl.rep.used[c];
        dead[c] = ctl.rep.dead[c];
    }
    return cudaSuccess;
}

// Export and import work on host copies of the tables: they are for tests and state hand-over, not for the packet
// path, and the caller has quiesced the context.  The host applies the same hash and the same probing as the kernels.
namespace {
struct FlowTablesHost {
    std::vector<FlowSlot> slots;
    long long special[3];
    FlowCtl ctl;
};
cudaError_t flows_download(bnk_ctx *ctx, FlowTablesHost &h) {
    const FilterTables &ft = ctx->ft;
    const size_t total = (size_t)6 * ft.flow_capacity;
    h.slots.resize(total);
    cudaError_t e = cudaSuccess;
    if (total) e = cudaMemcpy(h.slots.data(), ft.flow_slots, total * sizeof(FlowSlot), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(h.special, ft.flow_special_exp, sizeof h.special, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&h.ctl, ft.flow_live, sizeof h.ctl, cudaMemcpyDeviceToHost);
    return e;
}
int class_of(uint8_t proto) { return proto == 6 ? 0 : (proto == 17 ? 1 : 2); }
uint8_t proto_of(int cls) { return cls == 0 ? 6 : (cls == 1 ? 17 : 1); }
} // namespace

int filter_flows_export(bnk_ctx *ctx, bnk_flow_entry *out, size_t capacity, size_t *count) {
    FlowTablesHost h;
    if (flows_download(ctx, h) != cudaSuccess) return BNK_ECUDA;
    const FilterTables &ft = ctx->ft;
    size_t n = 0;
    auto emit = [&](int cls, unsigned long long key, long long exp) {
        if (n < capacity && out) {
            bnk_flow_entry e{};
            e.remote_addr = (uint32_t)(key >> 32);
            e.remote_port = (uint16_t)(key >> 16);
            e.local_port = (uint16_t)key;
            e.proto = proto_of(cls);
            e.expiry_unix_ns = exp;
            out[n] = e;
        }
        n++;
    };
    for (int cls = 0; cls < 3; cls++) {
        const size_t base = flow_region(ft, cls);
        for (size_t k = 0; k < ft.flow_capacity; k++) {
            const FlowSlot &v = h.slots[base + k];
            if (v.key != FLOW_EMPTY && !flow_absent(v.exp)) emit(cls, v.key, v.exp);
        }
        if (!flow_absent(h.special[cls])) emit(cls, FLOW_EMPTY, h.special[cls]);
    }
    *count = n;
    return BNK_SUCCESS;
}

int filter_flows_import(bnk_ctx *ctx, const bnk_flow_entry *entries, size_t n) {
    FlowTablesHost h;
    if (flows_download(ctx, h) != cudaSuccess) return BNK_ECUDA;
    const FilterTables &ft = ctx->ft;
    const uint32_t cap = ft.flow_capacity;
    for (size_t i = 0; i < n; i++) {
        const bnk_flow_entry &e = entries[i];
        if (e.proto != 6 && e.proto != 17 && e.proto != 1) return BNK_EINVAL;
        if (flow_absent(e.expiry_unix_ns)) return BNK_EINVAL;
        const int cls = class_of(e.proto);
        const unsigned long long key = ((unsigned long long)e.remote_addr << 32) | ((unsigned long long)e.remote_port << 16) | e.local_port;
        if (key == FLOW_EMPTY) {
            if (flow_absent(h.special[cls])) h.ctl.rep.live++;
            h.special[cls] = e.expiry_unix_ns;
            continue;
        }
        if (cap == 0) return BNK_EFULL;
        const size_t base = flow_region(ft, cls);
        uint32_t at = flow_hash(key) & (cap - 1);
        bool placed = false;
        for (uint32_t probe = 0; probe < cap && !placed; probe++, at = (at + 1) & (cap - 1)) {
            unsigned long long &k = h.slots[base + at].key;
            if (k != FLOW_EMPTY && k != key) continue;
            if (k == FLOW_EMPTY) {
                k = key;
                h.ctl.rep.used[cls]++;
            }
            long long &x = h.slots[base + at].exp;
            if (flow_absent(x)) h.ctl.rep.live++;
            if (x == FLOW_DEAD) h.ctl.rep.dead[cls]--;
            x = e.expiry_unix_ns;
            placed = true;
        }
        if (!placed) return BNK_EFULL;
    }
    h.ctl.rep.floor = LLONG_MIN; // unknown: the next sweep finds it
    ctx->flow_bounds.set(LLONG_MIN, h.ctl.rep.live);
    const size_t total = (size_t)6 * cap;
    cudaError_t e = cudaSuccess;
    if (total) e = cudaMemcpy(ft.flow_slots, h.slots.data(), total * sizeof(FlowSlot), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(ft.flow_special_exp, h.special, sizeof h.special, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(ft.flow_live, &h.ctl, sizeof h.ctl, cudaMemcpyHostToDevice);
    return e == cudaSuccess ? BNK_SUCCESS : BNK_ECUDA;
}

cudaError_t launch_flow_report(bnk_batch *b, cudaStream_t s) {
    const FlowCtl *ctl = reinterpret_cast<const FlowCtl *>(b->ctx->ft.flow_live);
    b->flow_reported = true;
    return cudaMemcpyAsync(b->h_flow, &ctl->rep, sizeof(FlowReport), cudaMemcpyDeviceToHost, s);
}

// Who has a clock behind that of a sweep waits for it.  (Clocks rise but for the order in which threads come by, so this is
// rare.)  Looked at behind flow_bounds' entry: a sweep that does not see that has left its clock here before.
static cudaError_t behind_newer_sweep(bnk_ctx *ctx, long long now, cudaStream_t s) {
    if (now >= ctx->sweep_now.load()) return cudaSuccess;
    std::lock_guard<std::mutex> g(ctx->sweep_mu); // its event is recorded
    return cudaStreamWaitEvent(s, ctx->ev_sweep, 0);
}
cudaError_t flow_note_begins(bnk_batch *b, uint32_t n, long long now, cudaStream_t s, bool &sweep) {
    sweep = b->ctx->flow_bounds.note_begins(b->flow_work, n, now);
    return behind_newer_sweep(b->ctx, now, s);
}
cudaError_t flow_check_begins(bnk_batch *b, long long now, cudaStream_t s) {
    b->ctx->flow_bounds.check_begins(b->flow_work, now);
    return behind_newer_sweep(b->ctx, now, s);
}
cudaError_t launch_flow_sweep(bnk_batch *b, long long now, const Done &done, cudaStream_t s) {
    bnk_ctx *ctx = b->ctx;
    std::lock_guard<std::mutex> g(ctx->sweep_mu);
    const long long latest = ctx->sweep_now.load();
    if (latest != LLONG_MIN) {
        const cudaError_t e = cudaStreamWaitEvent(s, ctx->ev_sweep, 0);
        if (e != cudaSuccess) return e;
    }
    ctx->sweep_now.store(std::max(latest, now));
    const long long beside = ctx->flow_bounds.beside(now);
    const size_t slots = (size_t)3 * ctx->ft.flow_capacity;
    const uint32_t grid = (uint32_t)std::min<size_t>(ctx->sm_count * 4, (slots + 1023) / 1024);
    b->flow_reported = true;
    ctx->launches += 1;
    const cudaError_t e = launch_after_kernel(filter_sweep_kernel, dim3(grid), dim3(256), s, ctx->ft, now, beside, b->h_flow, done);
    const cudaError_t r = cudaEventRecord(ctx->ev_sweep, s);
    return e != cudaSuccess ? e : r;
}

// Deleted entries keep their slots, so a class whose flows come and go (every connection brings a new source
// port) would fill up although few flows are alive, and a lookup that misses would walk longer and longer
// chains.  The submit that is about to record flows calls this first: when the device last reported that
// deleted entries fill a quarter of a class's region, the class is compacted on this batch's stream.  Kernels
// of other batches must not see the table half-moved, so the move is fenced against every other stream of the
// context on both sides, and submits are held off while the fences are placed (submit_mu, exclusive).
cudaError_t filter_flows_maintain(bnk_batch *b, cudaStream_t s) {
    bnk_ctx *ctx = b->ctx;
    const uint32_t cap = ctx->ft.flow_capacity;
    if (cap == 0) return cudaSuccess;
    const uint32_t limit = cap / 4;
    if (ctx->flow_dead_hint[0] < limit && ctx->flow_dead_hint[1] < limit && ctx->flow_dead_hint[2] < limit)
        return cudaSuccess;
    std::unique_lock<std::shared_mutex> tables(ctx->submit_mu);
    cudaError_t e;
    for (bnk_batch *o : ctx->batches) { // everything submitted so far finishes before the move
        for (cudaStream_t os : {o->stream, o->direct_stream}) {
            if (!os) continue;
            if ((e = cudaEventRecord(o->ev_fence, os)) != cudaSuccess) return e;
            if ((e = cudaStreamWaitEvent(s, o->ev_fence, 0)) != cudaSuccess) return e;
        }
    }
    for (int cls = 0; cls < 3; cls++) {
        if (ctx->flow_dead_hint[cls] < limit) continue;
        flows_compact_kernel<<<ctx->sm_count * 4, 256, 0, s>>>(ctx->ft, cls);
        flows_compact_finish_kernel<<<ctx->sm_count * 4, 256, 0, s>>>(ctx->ft, cls);
        ctx->launches += 2;
        ctx->ft.flow_half[cls] ^= 1; // launches from here on use the other region
        ctx->flow_dead_hint[cls] = 0;
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = cudaEventRecord(b->ev_fence, s)) != cudaSuccess) return e;
    for (bnk_batch *o : ctx->batches) // and nothing submitted later starts before it is done
        for (cudaStream_t os : {o->stream, o->direct_stream})
            if (os && os != s && (e = cudaStreamWaitEvent(os, b->ev_fence, 0)) != cudaSuccess) return e;
    return cudaSuccess;
}

cudaError_t launch_tally(bnk_batch *b, uint32_t n, cudaStream_t s) {
    bnk_ctx *ctx = b->ctx;
    uint32_t grid = (n + 1023) / 1024;
    if (grid == 0) grid = 1;
    if (grid > (uint32_t)ctx->sm_count * 4) grid = ctx->sm_count * 4;
    bnk_batch_stats *out = b->h_stats; // pinned memory has the same address on the device
    launch_kernel(n <= dependent_launch_up_to(), tally_kernel, dim3(grid), dim3(256), s, b->dev.status, b->dev.out_len, n,
                  b->d_stats, out);
    ctx->launches += 1;
    return cudaGetLastError();
}

// Builds the prefix-indexed rule table and swaps it in.  Runs per policy change
// (Engine.ApplyNetmap, internal/dataplane/engine.go:279-283), never per packet, and may run while packets
// flow: the reference swaps the table under the filter's mutex between two packets (filter.go:46-51); here
// the new table is uploaded into the buffer set that is not in use, on the admin stream, and the context's
// FilterTables (which every launch captures by value) switch over between two submits.  A batch submitted
// before the switch is judged by the old rules as a whole, one submitted after it by the new ones.
int filter_acl_upload(bnk_ctx *ctx, int enforce, const bnk_acl_tuple *tuples, size_t n) try {
    std::lock_guard<std::mutex> one_at_a_time(ctx->acl_mu);
    FilterTables &ft = ctx->ft;
    struct Item {
        uint64_t key, ent; // address << 8 | prefix length;  proto << 32 | first << 16 | last
    };
    std::vector<Item> items;
    items.reserve(n);
    for (size_t i = 0; i < n; i++) {
        const bnk_acl_tuple &t = tuples[i];
        if (t.prefix_len > 32) return BNK_EINVAL;
        if (t.proto != 6 && t.proto != 17 && t.proto != 1) continue; // can never equal a parsed protocol
        if (t.proto != 1 && t.port_first > t.port_last) continue;    // empty range
        items.push_back({(uint64_t)(t.addr & prefix_mask(t.prefix_len)) << 8 | t.prefix_len,
                         ((uint64_t)t.proto << 32) | ((uint64_t)t.port_first << 16) | t.port_last});
    }
    std::sort(items.begin(), items.end(), [](const Item &a, const Item &b) {
        return a.key != b.key ? a.key < b.key : a.ent < b.ent;
    });
    // One group per prefix, its ranges merged, in the order of (address, length): behind the prefixes that contain it, of
    // which `open` holds those that contain the last one.
    std::vector<RuleGroup> groups;
    std::vector<uint32_t> ports, open, shorts;
    std::vector<RuleStretch> stretches;
    size_t n_long = 0;
    for (size_t i = 0; i < items.size();) {
        const uint64_t key = items[i].key;
        const uint32_t number = (uint32_t)groups.size();
        RuleGroup g{};
        g.len = (uint32_t)key & 0xffu;
        g.addr = (uint32_t)(key >> 8);
        while (!open.empty() && (g.addr & prefix_mask(groups[open.back()].len)) != groups[open.back()].addr) open.pop_back();
        if (!open.empty()) g.parent = open.back() + 1;
        open.push_back(number);
        for (; i < items.size() && items[i].key == key && (items[i].ent >> 32) == 1; i++) g.parent |= 1u << 31; // icmp ignores ports
        for (const uint64_t proto : {6, 17}) {
            uint32_t count = 0, &at = proto == 6 ? g.tcp_at : g.udp_at;
            at = (uint32_t)ports.size();
            for (; i < items.size() && items[i].key == key && (items[i].ent >> 32) == proto; i++) {
                const uint32_t first = (uint32_t)items[i].ent >> 16, last = (uint32_t)items[i].ent & 0xffffu;
                if (count && first <= (ports.back() & 0xffffu) + 1) { // overlaps or continues the range before it
                    ports.back() = (ports.back() & 0xffff0000u) | std::max(last, ports.back() & 0xffffu);
                } else {
                    ports.push_back(first << 16 | last);
                    count++;
                }
            }
            (proto == 6 ? g.tcp0 : g.udp0) = count ? ports[at] : kNoPorts;
            g.n_ports |= count << (proto == 6 ? 0 : 16); // at most 32,768: there is a port between two ranges
            while (ports.size() & 3) ports.push_back(kNoPorts);
        }
        if (g.len <= 16) {
            shorts.push_back(number);
        } else {
            if (stretches.empty() || stretches.back().hi != g.addr >> 16) stretches.push_back({g.addr >> 16, number, number});
            stretches.back().end = number + 1;
        }
        n_long += g.len > 24;
        groups.push_back(g);
    }
    const size_t slots = rule_long_slots(n_long);
    const RuleLayout at(stretches.size(), slots, groups.size(), ports.size());
    std::vector<uint8_t> image(groups.empty() ? 0 : at.uploaded);
    const size_t index_bytes = groups.empty() ? 0 : at.total;
    if (index_bytes) {
        auto put = [&](size_t where, const auto &v) {
            if (!v.empty()) memcpy(image.data() + where, v.data(), v.size() * sizeof(v[0]));
        };
        put(at.groups, groups);
        put(at.ports, ports);
        put(at.shorts, shorts);
        put(at.stretches, stretches);
    }
    bnk_ctx::RuleSet &spare = ctx->rule_set[ctx->rule_cur ^ 1];
    // Kernels launched before the previous switch may still be reading the spare set: wait for those (the events
    // were recorded on the batches' streams at that switch), not for the whole device.
    for (cudaEvent_t ev : spare.in_use) {
        cudaEventSynchronize(ev);
        cudaEventDestroy(ev);
    }
    spare.in_use.clear();
    // A context created without max_acl_tuples grows the spare set here when a larger table arrives
    // (an allocation can stall the device for a moment; state the capacity to avoid that).
    if (index_bytes > spare.cap) {
        cudaFree(spare.mem);
        spare.mem = nullptr;
        spare.cap = 0;
        if (cudaMalloc(&spare.mem, index_bytes) != cudaSuccess) return BNK_ENOMEM;
        spare.cap = index_bytes;
    }
    cudaStream_t as = ctx->admin_stream;
    if (index_bytes) {
        RuleBuild b{};
        b.groups = reinterpret_cast<const RuleGroup *>(spare.mem + at.groups);
        b.shorts = reinterpret_cast<const uint32_t *>(spare.mem + at.shorts);
        b.stretches = reinterpret_cast<const RuleStretch *>(spare.mem + at.stretches);
        b.n_groups = (uint32_t)groups.size();
        b.n_shorts = (uint32_t)shorts.size();
        b.n_stretches = (uint32_t)stretches.size();
        b.top = reinterpret_cast<uint32_t *>(spare.mem + at.top);
        b.blocks = reinterpret_cast<uint2 *>(spare.mem + at.blocks);
        b.table = reinterpret_cast<RuleGroup *>(spare.mem + at.table);
        b.mask = (uint32_t)slots - 1;
        cudaError_t e = cudaMemcpyAsync(spare.mem, image.data(), image.size(), cudaMemcpyHostToDevice, as);
        if (e == cudaSuccess) e = cudaMemsetAsync(b.table, 0, slots * sizeof(RuleGroup), as);
        if (e != cudaSuccess) return BNK_ECUDA;
        const uint32_t table_ctas = n_long ? (b.n_groups + 255) / 256 : 0;
        rule_build_kernel<<<kTopCtas + b.n_stretches + table_ctas, 256, 0, as>>>(b);
        ctx->launches += 1;
        if (cudaGetLastError() != cudaSuccess) return BNK_ECUDA;
    }
    if (cudaStreamSynchronize(as) != cudaSuccess) return BNK_ECUDA;
    {
        std::unique_lock<std::shared_mutex> tables(ctx->submit_mu); // between two submits
        bnk_ctx::RuleSet &old = ctx->rule_set[ctx->rule_cur];
        for (bnk_batch *b : ctx->batches) { // what has been launched with the old set, per stream
            for (cudaStream_t bs : {b->stream, b->direct_stream}) {
                if (!bs) continue;
                cudaEvent_t ev;
                if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return BNK_ECUDA;
                cudaEventRecord(ev, bs);
                old.in_use.push_back(ev);
            }
        }
        ft.rule_top = index_bytes == 0 ? nullptr : reinterpret_cast<const uint32_t *>(spare.mem + at.top);
        ft.rule_blocks = reinterpret_cast<const uint2 *>(spare.mem + at.blocks);
        ft.rule_long = reinterpret_cast<const RuleGroup *>(spare.mem + at.table);
        ft.rule_long_mask = (uint32_t)slots - 1;
        ft.rule_groups = reinterpret_cast<const RuleGroup *>(spare.mem + at.groups);
        ft.rule_ports = reinterpret_cast<const uint32_t *>(spare.mem + at.ports);
        ft.enforce = enforce ? 1 : 0;
        ctx->rule_cur ^= 1;
    }
    return BNK_SUCCESS;
} catch (const std::exception &) { // a host allocation
    return BNK_ENOMEM;
}

static bool heads_in_pairs(const bnk_batch *b, uint32_t n) { return b->dev.ring == b->host.ring && n >= kPairsFrom; }

cudaError_t launch_filter_note(bnk_batch *b, uint32_t first, uint32_t n, long long now_ns, const Done &done, cudaStream_t s) {
    bnk_ctx *ctx = b->ctx;
    FlowReport *const report = done.flag ? b->h_flow : nullptr;
    if (report) b->flow_reported = true;
    launch_kernel(n <= dependent_launch_up_to(), heads_in_pairs(b, n) ? filter_note_kernel<true> : filter_note_kernel<false>, dim3((n + 127) / 128), dim3(128), s, ctx->ft,
        b->dev.ring, b->dev.off + first, b->dev.len + first, n, b->ring_bytes, now_ns, report, done);
    ctx->launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_filter_check(bnk_batch *b, uint32_t n, long long now_ns, bool only_status_ok, uint8_t *host_status,
                                const Done &done, cudaStream_t s) {
    bnk_ctx *ctx = b->ctx;
    if (n == 0) return cudaSuccess;
    // open pipeline: the packet handed to the filter is the decrypted payload of out_len bytes
    const uint32_t *lens = only_status_ok ? b->dev.out_len : b->dev.len;
    launch_kernel(n <= dependent_launch_up_to(), heads_in_pairs(b, n) ? filter_check_kernel<true> : filter_check_kernel<false>, dim3((n + 127) / 128), dim3(128), s, ctx->ft,
        b->dev.ring, b->dev.off, lens, b->dev.status, n, b->ring_bytes, now_ns, only_status_ok ? 1 : 0, host_status, done);
    ctx->launches += 1;
    return cudaGetLastError();
}
