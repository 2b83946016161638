// Internal declarations shared by the translation units of libbnkgpu.so.
// Nothing here is part of the C ABI (that is include/bnk_gpu.h).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <atomic>
#include <memory>
#include <mutex>
#include <shared_mutex>
#include <string>
#include <vector>

#include "../../include/bnk_gpu.h"
#include "flow_bounds.h"
#include "launch.h"
#include "pieces.h"
#include "submit_order.h"

// ---------------------------------------------------------------------------
// Device-resident tables of one context (one GPU).  All per-peer mutable state
// lives here, indexed by keypair slot, so that peers shard across GPUs with no
// exchange: keys, send counter, replay window.
// ---------------------------------------------------------------------------
// Next nonce of a keypair.  The packets of one seal launch read it and one of them moves it on, with nothing to order
// them by: so a launch never writes the entry its packets read.  The entry with the higher `seq` counts; the launch that
// carries the number q (ctx->seal_seq, rising) looks at entries below q only and writes the other one, as {value, q}.
// Kernels that separate their reads from their writes by a barrier change the entry in place.
struct alignas(32) SendCounter {
    struct alignas(16) Entry {
        uint64_t value, seq;
    } e[2];
};

struct KeypairTables {
    uint32_t *send_keys;    // [max_keypairs][8] little-endian words
    uint32_t *recv_keys;    // [max_keypairs][8]
    uint32_t *remote_index; // [max_keypairs] receiver index written into sealed headers
    SendCounter *send_counter; // [max_keypairs] next nonce to hand out
    uint64_t *replay_last;  // [max_keypairs] highest counter accepted
    uint64_t *replay_next;  // [max_keypairs] scratch: the value replay_last takes after the batch in flight
    uint64_t *replay_ring;  // [max_keypairs][ring_blocks] RFC 6479 bitmap ring
    uint32_t *allowed_ip;   // [max_keypairs] the peer's tunnel address, host order (0 = none)
    uint8_t *valid;         // [max_keypairs] 1 while the slot holds keys that bnk_keypair_set* put there
    // receiver index -> slot: open addressing, key = 1<<32 | index (0 = empty, 2<<32 = deleted)
    uint64_t *index_keys;   // [index_slots]
    uint32_t *index_vals;   // [index_slots]
    uint32_t index_slots;   // power of two
    // source address -> peer id (Bind.byAddr): open addressing over 32-byte entries
    struct AddrEntry {
        uint64_t hi, lo;   // the 16 address bytes as two little-endian words
        uint32_t port;     // port | 1<<16 when live, 2<<16 when deleted, 0 when empty
        uint32_t peer;
        uint64_t pad;
    };
    AddrEntry *addr_tab;    // [addr_slots]
    uint32_t addr_slots;    // power of two
};

// The allowances of one prefix.  Port ranges (first << 16 | last) are disjoint and in rising order; those of tcp and those
// of udp each start at a multiple of four in rule_ports and are filled up with kNoPorts to one.
struct alignas(32) RuleGroup {
    uint32_t addr, len;         // the prefix (hash table: len 0 = an empty place)
    uint32_t parent;            // the longest shorter prefix with allowances that contains this one, + 1; bit 31: icmp is allowed
    uint32_t n_ports;           // tcp's ranges | udp's << 16
    uint32_t tcp_at, udp_at;    // where they start in rule_ports
    uint32_t tcp0, udp0;        // the first of each (kNoPorts: none)
};
constexpr uint32_t kNoPorts = 0xffff0000u;

// Flattened, indexed ACL and the reply-flow table (filter_kernels.cu).
struct alignas(16) FlowSlot { // key and expiry side by side: a lookup's first probe is one 16-byte load
    unsigned long long key; // FLOW_EMPTY = all ones
    long long exp;          // in unix ns; FLOW_DEAD = deleted
};
struct FilterTables {
    // rule index (filter_device.cuh), one block of device memory
    const uint32_t *rule_top;    // [65536] by the upper 16 address bits; null when there are no rules
    const uint2 *rule_blocks;    // [blocks][256] by the next 8
    const RuleGroup *rule_long;  // hash table of the prefixes longer than 24
    uint32_t rule_long_mask;
    const RuleGroup *rule_groups;
    const uint32_t *rule_ports;
    int enforce;
    // flow table, one open-addressing region per protocol class (tcp, udp, icmp).  Every class has two
    // regions, [class][half][flow_capacity]; flow_half[class] says which one is in use, the other one is all
    // FLOW_EMPTY and receives the surviving entries when the class is compacted (filter_flows_compact).
    FlowSlot *flow_slots;   // [3][2][flow_capacity]
    uint32_t flow_capacity; // power of two
    uint8_t flow_half[3];
    unsigned long long *flow_live;  // device control block (FlowCtl): live entries (Go's len(f.flows)) and more
    long long *flow_special_exp;    // [3] entry for the one key that equals FLOW_EMPTY
};
// region of protocol class `cls` that is in use
__host__ __device__ inline size_t flow_region(const FilterTables &ft, int cls) {
    return ((size_t)cls * 2 + ft.flow_half[cls]) * ft.flow_capacity;
}
class CopyCrew;
struct bnk_ctx {
    bnk_cfg cfg;
    int device;
    KeypairTables kt;
    FilterTables ft;
    cudaStream_t admin_stream;
    cudaEvent_t timer_start;
    int sm_count;
    uint64_t host_direct_bytes; // batches up to this ring extent run on the caller's pinned buffers (BNK_HOST_DIRECT_BYTES)
    std::atomic<int> in_flight{0};           // batches submitted and not waited for
    std::atomic<uint64_t> direct_in_flight{0}; // ring bytes of those that run on the pinned buffers
    bool launch_graphs; // BNK_LAUNCH_GRAPHS
    int aead_mode; // 0 = choose by batch size and layout, 1 = always thread per packet, 2 = always warp per packet (BNK_AEAD_KERNEL)
    uint32_t aead_side_stream_from; // batches of at least this many packets run seal/open on the low-priority stream (BNK_AEAD_SIDE_STREAM_FROM; 0 = never)
    // ring extent from which a batch that is alone goes over the link in pieces (BNK_PIECES_FROM); of batches for aead_stream_kernel
    uint64_t pieces_from, stream_pieces_from;
    int prio_low, prio_high;        // stream priority range of the device
    std::atomic<uint64_t> launches, graph_launches;
    std::atomic<uint64_t> seal_seq{0}; // number of the last seal launch that handed out nonces itself (see SendCounter)
    std::mutex mu;
    std::string last_error;
    // Submits hold this shared while they queue their work; whoever changes what running kernels of other
    // batches could observe half-done (flow-table compaction) or swaps tables that launches capture by value
    // (rule table) holds it exclusively.
    std::shared_mutex submit_mu;
    std::vector<bnk_batch *> batches;       // every live batch of the context (guarded by mu)
    std::shared_ptr<CopyCrew> crew;         // helpers of its queues' copies, made with the first queue (guarded by mu)
    std::atomic<uint32_t> flow_dead_hint[3]; // deleted entries per class as last reported by the device
    FlowBounds flow_bounds;
    // Sweeps of the flow table run one behind the other, and work with an older clock than one of them behind it.
    std::mutex sweep_mu;
    cudaEvent_t ev_sweep;                  // behind the last one
    std::atomic<long long> sweep_now;      // latest clock of any
    std::atomic<int> flow_errors_seen;       // failed inserts already reported to a caller as BNK_EFULL
    // rule table: two device buffer sets, the one not in use receives the next upload
    struct RuleSet {
        uint8_t *mem = nullptr;
        size_t cap = 0;
        std::vector<cudaEvent_t> in_use; // recorded on every batch stream when the set was retired
    } rule_set[2];
    int rule_cur = 0;
    std::mutex acl_mu; // one bnk_acl_set at a time
    std::vector<KeypairTables::AddrEntry> addr_host; // host shadow of kt.addr_tab
    std::vector<uint64_t> index_keys_host; // host shadow of kt.index_keys (updates are rare: one per handshake)
    std::vector<uint32_t> index_vals_host; // host shadow of kt.index_vals
    uint32_t index_live, index_dead;       // entries of the receiver-index table in use / deleted but not yet reclaimed
    uint32_t addr_live, addr_dead;         // the same for the source-address table
};

struct DeviceBatch {
    uint8_t *ring;
    uint32_t *off, *len, *slot, *out_len;
    uint64_t *counter;
    uint8_t *status;
    uint8_t *src_addr;    // [max_pkts][BNK_SRC_ADDR_STRIDE]
    // scratch for grouping packets by keypair slot (group_kernels.cu)
    uint32_t *order;      // [max_pkts] packet indices, stable by slot
    uint32_t *order_tmp;  // [max_pkts]
    uint32_t *keys_tmp;   // [2][max_pkts] radix keys ping-pong
    // scratch of the replay window in its scan form (group_kernels.cu)
    uint64_t *sorted_counter;    // [max_pkts] counters in grouped order
    uint8_t *replay_state;       // [max_pkts] verdict per grouped position
    uint32_t *replay_hash;       // [replay_hash_capacity(max_pkts)] lowest position per (peer, counter)
    uint32_t *replay_tile_head;  // [tiles + 1] a run starts inside the tile; last entry: some packet needs the hash
    uint64_t *replay_tile_max;   // [tiles]
    uint64_t *replay_tile_carry; // [tiles]
    uint32_t *hist;       // [512 * chunks] digit-major histograms
    uint32_t *len_order;  // [max_pkts] packet indices ordered by length class
    uint4 *inner;         // [max_pkts] headers of opened packets on their way to the last checks
    uint32_t *counters32; // small scratch (bins)
    bnk_gso_super *gso;   // [max_pkts] super-packet descriptors of a GSO split
};

enum class Heads : uint8_t { none, in_place, copied }; // a submit that looks at the heads of many packets that lie close together
struct bnk_batch {
    bnk_ctx *ctx;
    uint32_t max_pkts;
    uint64_t ring_bytes;
    bnk_batch_view host; // pinned
    DeviceBatch dev;
    cudaStream_t stream;
    cudaStream_t aux_stream;   // grouping work that can run beside the open kernel
    // The seal/open launches of a large batch go to a stream of their own with the lowest priority, the short
    // kernels around them (grouping, counters, replay window, length classes) stay on `stream` / `aux_stream`
    // with the highest: a large seal/open launch fills every SM for hundreds of microseconds, and the short
    // kernels of the NEXT batch would otherwise get no SM until its last wave.  With priorities their CTAs take
    // the places seal/open CTAs leave as they retire, so the chain of one batch really runs beside the seal/open
    // kernel of another.
    cudaStream_t aead_stream;
    cudaEvent_t ev_aead_go, ev_aead_done;
    PieceStreams pieces; // of a batch large enough to go over the link that way
    cudaEvent_t ev_fork, ev_join;
    cudaEvent_t k_begin, k_end, t_end, a_begin, a_end;
    bool in_flight;
    // Submits ran on the host arrays: the device copies of the first `stale_pkts` packets and descriptors (of the first
    // `stale_src` source addresses) are behind.
    uint32_t stale_pkts, stale_src;
    Heads heads;           // what the last submit was, and ...
    bool heads_go_up;      // ... whether such submits leave the packets on the device (see heads_direct)
    uint64_t partial_to;   // below this place of the device ring only packets and super-packets are those of the host ring
    uint32_t split_sealed; // with partial_to: that many packets have been sealed since the split
    bool counted;        // this batch is one of ctx->in_flight
    uint64_t direct_counted; // what it adds to ctx->direct_in_flight
    // bnk_wait watches *h_done for done_seq when done_watched: the last kernel of the submit stores it (Done)
    uint32_t *h_done, *d_ticket;
    uint32_t done_seq, done_polls;
    bool done_watched;
    LaunchGraph *graph;  // what the submit in flight was launched through
    bool kernel_timed;
    bool aead_timed;
    bnk_gso_super *h_gso; // pinned staging for the super-packet descriptors
    uint8_t *h_desc, *d_desc; // one slab per side: off | len | slot | counter | out_len | status (npad entries each), then the ring
    uint32_t npad;
    size_t desc_room;  // bytes of the descriptor slab in front of the ring (same on both sides)
    bool joint_copy;   // descriptors and ring move as one copy
    FlowReport *h_flow; // pinned copy of the flow table's state after the batch's filter work
    bool stats_pending; // the last submit was made with BNK_F_STATS
    FlowWork flow_work; // its filter work that has not been waited for
    bool flow_reported; // the last submit queued a copy of the flow table's state into h_flow
    bnk_batch_stats *h_stats; // pinned; written by the tally kernel
    unsigned long long *d_stats; // device accumulators of the tally kernel (zero between launches)
    cudaEvent_t ev_fence; // orders this batch's stream against table maintenance on another stream
    // Submits in order over several batches (submit_order.h).  direct_stream: where such a batch runs when it stays in
    // pinned memory (shared with the batches it is ordered against; null: on its own stream).
    cudaStream_t direct_stream;
    SubmitOrder order;
    bool ordered; // between order_begin and order_end
    bnk_batch *behind;
};

// Small batches are two dependent launches with little work in each, so the gap between them counts.  A kernel
// launched through launch_after_kernel may be scheduled while the kernel in front of it on the stream is still
// running (programmatic dependent launch) and must call wait_for_kernel_in_front() before it touches anything
// that kernel writes: the wait ends when that kernel has finished and its writes are visible.  The kernel in front
// calls let_next_kernel_start() first thing, which allows the next one to be placed on the SMs (where it sits in
// its wait) as soon as all of this kernel's CTAs are resident; that hides the launch latency of the second kernel
// behind the first.  Launched the ordinary way, or with nothing of the kind behind it, both calls do nothing.
__device__ __forceinline__ void wait_for_kernel_in_front() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_kernel_start() { asm volatile("griddepcontrol.launch_dependents;"); }
// The chains of short kernels around a large batch (grouping, counters, replay window, length classes) are
// launched the same way while they are short: measured on 96,256 packets both sides of the pipeline got 7 % faster,
// on 1,048,576 packets 1 % slower.  With several large batches in flight it costs: CTAs that sit in their wait hold
// SM slots that the seal/open kernel of another batch could use (four batches of 262,144 mixed packets: 1.05 ms
// per step with dependent launches, 0.93 without).  Hence the limit.
inline uint32_t dependent_launch_up_to() {
    static const uint32_t v = [] {
        const char *m = getenv("BNK_DEPENDENT_LAUNCH_UP_TO"); // tuning aid
        return m ? (uint32_t)strtoul(m, nullptr, 0) : (1u << 17);
    }();
    return v;
}
template <typename... KArgs>
cudaError_t launch_after_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, const typename AsIs<KArgs>::type &...args) {
    return launch_shape(LaunchShape{nullptr, grid, block, 0, 1, true}, kernel, s, args...);
}
// the same launch with the ordinary full dependency when `dependent` is false
template <typename... KArgs>
cudaError_t launch_kernel(bool dependent, void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, const typename AsIs<KArgs>::type &...args) {
    return launch_shape(LaunchShape{nullptr, grid, block, 0, 1, dependent}, kernel, s, args...);
}

constexpr uint32_t kSlotNoKeypair = 0xfffffffeu; // demux found no keypair for the receiver index

// WireGuard padding: up to a multiple of 16, never beyond the MTU; a packet
// longer than the MTU is padded as if only its last MTU-sized unit counted.
__device__ __forceinline__ uint32_t wg_padded_len(uint32_t len, uint32_t mtu) {
    if (mtu == 0) return (len + 15u) & ~15u;
    uint32_t last = len > mtu ? len % mtu : len;
    uint32_t padded = (last + 15u) & ~15u;
    if (padded > mtu) padded = mtu;
    return len + (padded - last);
}

// ---------------------------------------------------------------------------
// Kernel launchers (each defined next to its kernels).  All are asynchronous on
// `s` and return the cudaError_t of the launch.
// ---------------------------------------------------------------------------
struct AeadResults { // where a packet's outcome goes; null members are left out
    uint64_t *counter;
    uint32_t *out_len;
    uint8_t *status;
    uint32_t *slot; // open side with demux
};
// How a batch's last kernel tells the host that everything before it is done: the CTA that finishes last stores
// `value` to a pinned word (bnk_wait watches it, which saves the ~3 us a stream synchronisation takes to notice).
struct Done {
    uint32_t *ticket; // device, zero between launches
    uint32_t *flag;   // pinned; null: nobody watches
    uint32_t value;
};
// By all threads of all CTAs, once, at the end; `last_words` (if `has_words`) runs in one thread when every CTA's work is
// visible on the device.  There is one fence that covers host memory, which takes 1.7 us (one in front of the last words as
// well: a packet sealed with its flow noted 18.9 us, without it 16.4).  Finding out who is last takes 0.75 us, but with a word
// per CTA, all watched by the host, every CTA has that fence: 128 x 1420 B sealed by 32 CTAs 19.7 us, so 23.0.
template <typename F>
__device__ __forceinline__ void signal_done(const Done &d, bool has_words, F last_words) {
    if (d.flag == nullptr) return;
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (gridDim.x != 1) {
        __threadfence();
        if (atomicAdd(d.ticket, 1u) + 1u != gridDim.x) return;
        *d.ticket = 0u;
    }
    if (has_words) {
        __threadfence();
        last_words();
    }
    __threadfence_system();
    *(volatile uint32_t *)d.flag = d.value;
}
struct HostDesc { // the descriptors where the host can read them
    const uint32_t *off, *len, *slot;
};
struct AeadArgs {
    const uint8_t *in;            // ring the input is read from and ...
    uint8_t *out, *out2;          // ... ring(s) the output goes to; thread per packet: in == out, no out2
    const uint32_t *off;
    const uint32_t *len;
    const uint32_t *slot;
    const uint64_t *counter;      // seal only
    AeadResults res[2];           // thread per packet: res[0] only, all members but slot set
    const uint32_t *keys;         // send keys (seal) or receive keys (open)
    const uint32_t *remote_index; // seal only
    const uint8_t *valid;         // per keypair slot: keys present
    const uint32_t *order;        // thread per packet: optional scheduling permutation, may be null
    const uint64_t *index_keys;   // with demux: the receiver-index table
    const uint32_t *index_vals;
    uint32_t index_slots;
    bool demux;                   // open, warp per packet: the slot comes from the header's receiver index
    bool inner_cut;               // packets will be cut to their IPv4 total length
    uint4 *inner;                 // open, warp per packet: headers of the plaintexts (see VerdictArgs); null: not wanted
    bool behind_kernel;           // a kernel of the same submit is in front
    bool over_link;               // a ring is in host memory
    bool from_host;               // the ring that is read and the descriptors are
    bool header_first;            // open of up to kRankMax packets with from_host: their headers are asked for ahead of them
    HostDesc host;                // with from_host
    uint64_t link_bytes;          // with over_link: bytes of the packets
    bool stream;                  // with from_host: it is a batch for kernel 3 (see in_stream)
    uint32_t n;
    uint32_t tile;                // set by the launcher
    uint32_t mtu;
    uint32_t max_slots;
    uint64_t ring_bytes;
    // Seal of up to kRankMax packets in pinned memory: nonces are handed out by the seal kernel itself (null: from counter[])
    SendCounter *send_counter;    // [max_slots]
    uint64_t seal_seq;
    // Seal in pinned memory with BNK_F_NOTE_OUTBOUND: the kernel records its packets' flows
    bool note;
    bool judge;                   // open: the packets will be checked against the rules
    long long now;
    FilterTables ft;
    FlowReport *flow_report;      // pinned, written before `done`; null: none
    Done done;
};
constexpr uint32_t kRankMax = 256;
cudaError_t launch_seal(const AeadArgs &a, cudaStream_t s, bnk_ctx *ctx);
cudaError_t launch_open(const AeadArgs &a, cudaStream_t s, bnk_ctx *ctx);

// group_kernels.cu
cudaError_t launch_group_by_slot(bnk_batch *b, uint32_t n, cudaStream_t s);
// slot / counter: the batch's arrays, wherever they are (device or pinned)
cudaError_t launch_assign_counters(bnk_batch *b, uint32_t n, const uint32_t *slot, uint64_t *counter, cudaStream_t s);
cudaError_t launch_replay(bnk_batch *b, uint32_t n, cudaStream_t s);
struct VerdictArgs;
// After the open kernel, up to kGroupMax packets: grouping, replay window (when `replay`) and the last checks in one launch.
constexpr uint32_t kGroupMax = 32768;
cudaError_t launch_open_tail(bnk_batch *b, uint32_t n, bool replay, const VerdictArgs *verdict, const Done &done, cudaStream_t s);
cudaError_t launch_verdict(bnk_ctx *ctx, const VerdictArgs &verdict, const Done &done, cudaStream_t s); // the last checks alone
cudaError_t group_kernels_init(); // once per context, for the current device
cudaError_t aead_kernels_init();
cudaError_t launch_length_order(bnk_batch *b, uint32_t n, const uint32_t *len, bool open_side, cudaStream_t s);
uint32_t group_sort_chunks(uint32_t max_pkts);
uint32_t replay_scan_tiles(uint32_t max_pkts);     // tiles of the running-maximum scan
uint32_t replay_hash_capacity(uint32_t max_pkts);  // entries of the duplicate-counter table

// filter_kernels.cu
// the inserts of packets [first, first + n); no sweep
cudaError_t launch_filter_note(bnk_batch *b, uint32_t first, uint32_t n, long long now_ns, const Done &done, cudaStream_t s);
cudaError_t launch_filter_check(bnk_batch *b, uint32_t n, long long now_ns, bool only_status_ok, uint8_t *host_status,
                                const Done &done, cudaStream_t s);
cudaError_t filter_tables_alloc(bnk_ctx *ctx);
void filter_tables_free(bnk_ctx *ctx);
int filter_acl_upload(bnk_ctx *ctx, int enforce, const bnk_acl_tuple *tuples, size_t n);
cudaError_t filter_flows_clear(bnk_ctx *ctx, cudaStream_t s);
cudaError_t filter_flow_stats(bnk_ctx *ctx, uint64_t *live, uint32_t used[3], uint32_t dead[3]);
int filter_flows_export(bnk_ctx *ctx, bnk_flow_entry *out, size_t capacity, size_t *count);
int filter_flows_import(bnk_ctx *ctx, const bnk_flow_entry *entries, size_t n);
cudaError_t launch_flow_report(bnk_batch *b, cudaStream_t s); // copies the flow table's control block to b->h_flow
// A submit is about to record up to n flows at `now` / to check packets at `now`, on stream s.  The former says whether the
// batch may have to sweep expired flows behind its inserts (launch_flow_sweep).
cudaError_t flow_note_begins(bnk_batch *b, uint32_t n, long long now, cudaStream_t s, bool &sweep);
cudaError_t flow_check_begins(bnk_batch *b, long long now, cudaStream_t s);
cudaError_t launch_flow_sweep(bnk_batch *b, long long now, const Done &done, cudaStream_t s);
// Rebuilds the regions whose deleted entries have piled up; called by a submit that feeds the flow table,
// before it takes submit_mu.  Returns without doing anything in the common case.
cudaError_t filter_flows_maintain(bnk_batch *b, cudaStream_t s);
// Per-status packet counts and byte total of the first n packets, into b->h_stats (one launch).
cudaError_t launch_tally(bnk_batch *b, uint32_t n, cudaStream_t s);

// inner_kernels.cu
cudaError_t launch_demux_index(bnk_batch *b, uint32_t first, uint32_t n, const uint32_t *len, cudaStream_t s); // packets [first, first + n)
cudaError_t launch_inner_check(bnk_batch *b, uint32_t n, cudaStream_t s);
cudaError_t launch_classify(bnk_batch *b, uint32_t n, const Done &done, cudaStream_t s);
// One 16-byte entry in one access, from and to the L2 that all SMs share.
__device__ __forceinline__ SendCounter::Entry counter_load(const SendCounter::Entry *p) {
    SendCounter::Entry v;
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }" : "=l"(v.value), "=l"(v.seq) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void counter_store(SendCounter::Entry *p, SendCounter::Entry v) {
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p), "l"(v.value), "l"(v.seq) : "memory");
}
struct CounterRead {
    SendCounter::Entry now;
    uint32_t at; // which entry that is
};
// The entry that counts, of those below `below` (~0: of both).
__device__ __forceinline__ CounterRead counter_read(const SendCounter *c, uint64_t below) {
    const SendCounter::Entry a = counter_load(&c->e[0]), b = counter_load(&c->e[1]);
    const bool first = a.seq < below && (b.seq >= below || a.seq >= b.seq);
    return CounterRead{first ? a : b, first ? 0u : 1u};
}
// nonce of the k-th packet of a run that starts at `base`: never past the message limit
__device__ __forceinline__ uint64_t saturating_counter(uint64_t base, uint32_t k) {
    const uint64_t c = base + k;
    return (c < base || c > BNK_REJECT_AFTER_MESSAGES) ? BNK_REJECT_AFTER_MESSAGES : c;
}
__host__ __device__ inline uint32_t addr_hash(uint64_t hi, uint64_t lo, uint32_t port) {
    uint64_t z = hi * 0x9e3779b97f4a7c15ull ^ (lo + 0xbf58476d1ce4e5b9ull) * 0x94d049bb133111ebull ^ ((uint64_t)port << 40);
    z ^= z >> 29;
    z *= 0xbf58476d1ce4e5b9ull;
    return (uint32_t)(z >> 32);
}
__host__ __device__ inline uint32_t index_hash(uint32_t index) {
    uint32_t z = index * 0x9e3779b1u;
    z ^= z >> 15;
    z *= 0x85ebca6bu;
    return z ^ (z >> 13);
}
// Receiver index -> keypair slot by a whole warp: the 32 places from the index's own on are looked at in one read, so
// a lookup is one trip to the table however long its probe chain (tables are at most half full).
__device__ __forceinline__ uint32_t demux_index_warp(const uint64_t *keys, const uint32_t *vals, uint32_t slots, uint32_t index) {
    const uint64_t key = (1ull << 32) | index;
    for (uint32_t base = 0; base < slots; base += 32) {
        const uint32_t h = (index_hash(index) + base + (threadIdx.x & 31u)) & (slots - 1);
        const uint64_t k = keys[h];
        const uint32_t v = vals[h];
        const uint32_t hit = __ballot_sync(0xffffffffu, k == key), empty = __ballot_sync(0xffffffffu, k == 0);
        const uint32_t at = __ffs(hit) - 1;
        if (hit && (empty == 0 || at < (uint32_t)__ffs(empty) - 1)) return __shfl_sync(0xffffffffu, v, at);
        if (empty) break;
    }
    return kSlotNoKeypair;
}

// gso_kernels.cu
cudaError_t launch_gso_split(bnk_batch *b, uint32_t n_super, uint32_t n_pkts, cudaStream_t s);
// The same with the descriptors and b->h_gso still in pinned memory: prepare, then the split, with the super-packets up or from
// the pinned ring.
bool gso_split_fits(const bnk_gso_super *supers, uint32_t n_super, uint32_t n_pkts, uint64_t ring_bytes);
cudaError_t launch_gso_prepare(bnk_batch *b, uint32_t n_super, uint32_t n_pkts, cudaStream_t s);
cudaError_t launch_gso_split_up(bnk_batch *b, uint32_t n_super, uint32_t n_pkts, const Done &done, cudaStream_t s);
cudaError_t launch_gso_split_in_place(bnk_batch *b, uint32_t n_super, uint32_t n_pkts, const Done &done, cudaStream_t s);
cudaError_t launch_packets_to_host(bnk_batch *b, uint32_t n, cudaStream_t s);
