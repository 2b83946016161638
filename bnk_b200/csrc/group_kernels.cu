// Per-keypair ordering work for sm_100a: grouping a batch by keypair slot while
// keeping arrival order (a stable least-significant-digit radix sort whose ranking
// step uses warp match/ballot instead of per-element atomics), handing out send
// counters, and walking the anti-replay window.
//
// Why a stable grouping: both the send counter (packets of one peer get
// consecutive nonces in batch order) and the replay window (verdicts depend on
// the arrival order of a peer's authenticated packets) are defined by a
// sequential walk per peer.  Different peers are independent, and inside a peer
// the walk has a parallel form: a packet's nonce is the peer's counter plus its
// rank in the peer's run, and the window's verdicts over a stretch of packets
// follow in closed form from the state at the start of the stretch.
#include <algorithm>

#include <cooperative_groups.h>

#include "filter_device.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr uint32_t kSortThreads = 256; // 8 warps per CTA
constexpr uint32_t kSortWarps = kSortThreads / 32;
constexpr uint32_t kMaxTiles = 32;     // a lane keeps up to 32 keys in registers
constexpr uint32_t kMaxDigitBits = 9;
constexpr uint32_t kMaxBins = 1u << kMaxDigitBits;
#ifndef BNK_SORT_MAX_CHUNKS
#define BNK_SORT_MAX_CHUNKS 320
#endif
constexpr uint32_t kBatchMaxChunks = BNK_SORT_MAX_CHUNKS; // ~2 CTAs per SM: enough to fill the GPU, few enough to scan quickly

struct SortKeySrc {
    const uint32_t *slot;
    uint32_t max_slots;
};

// Key of packet i: its keypair slot, or max_slots ("takes no part", sorts last).
__device__ __forceinline__ uint32_t slot_key(const SortKeySrc &k, uint32_t i) {
    const uint32_t s = k.slot[i];
    return s < k.max_slots ? s : k.max_slots;
}

// one shared-memory add per distinct digit in the warp instead of one per lane
__device__ __forceinline__ void warp_hist_add(uint32_t *cnt, uint32_t digit, bool have) {
    const uint32_t peers = __match_any_sync(0xffffffffu, have ? digit : 0xffffffffu);
    if (have && (__ffs(peers) - 1) == (int)(threadIdx.x & 31)) atomicAdd(&cnt[digit], __popc(peers));
}

// A CTA owns a chunk of 256 * TILES consecutive elements; warp w owns the 32 * TILES consecutive
// elements [w * 32 * TILES, (w + 1) * 32 * TILES) of it.

// --- pass step 1: per-chunk digit histogram -------------------------------------------
// grid = chunks, block = 256.  hist is digit-major: hist[digit * chunks + chunk].
template <uint32_t TILES>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(SortKeySrc src, const uint32_t *keys_in,
                                                                  uint32_t n, uint32_t shift, uint32_t bins,
                                                                  uint32_t chunks, uint32_t *hist) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ uint32_t cnt[kMaxBins];
    const uint32_t tid = threadIdx.x, chunk = blockIdx.x;
    for (uint32_t d = tid; d < bins; d += kSortThreads) cnt[d] = 0;
    __syncthreads();
    const uint32_t begin = chunk * (kSortThreads * TILES);
    const uint32_t end = min(n, begin + kSortThreads * TILES);
#pragma unroll
    for (uint32_t t = 0; t < TILES; t++) {
        const uint32_t i = begin + t * kSortThreads + tid;
        const bool have = i < end;
        uint32_t digit = 0;
        if (have) digit = ((keys_in ? keys_in[i] : slot_key(src, i)) >> shift) & (bins - 1);
        warp_hist_add(cnt, digit, have);
    }
    __syncthreads();
    for (uint32_t d = tid; d < bins; d += kSortThreads) hist[d * chunks + chunk] = cnt[d];
}

// --- pass step 2: per digit, exclusive prefix over the chunks -------------------------
// One warp per digit row (coalesced: the row is contiguous).  Row totals go to totals[digit]; the
// scatter kernel turns them into digit bases on its own.
__global__ void __launch_bounds__(kSortThreads) radix_rowscan_kernel(uint32_t *hist, uint32_t bins, uint32_t chunks,
                                                                     uint32_t *totals) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t d = (blockIdx.x * kSortThreads + threadIdx.x) >> 5;
    if (d >= bins) return;
    uint32_t *row = hist + (size_t)d * chunks;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < chunks; base += 32) {
        const uint32_t c = base + lane;
        const uint32_t v = c < chunks ? row[c] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        if (c < chunks) row[c] = carry + incl - v;
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) totals[d] = carry;
}

// --- exclusive scan of a small array by one CTA (length-class bins) ---------------------
__global__ void __launch_bounds__(1024) exclusive_scan_kernel(uint32_t *data, uint32_t n) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ uint32_t warp_off[32];
    __shared__ uint32_t carry_s;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) carry_s = 0;
    __syncthreads();
    for (uint32_t base = 0; base < n; base += 4096) {
        const uint32_t i0 = base + tid * 4;
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = (i0 + k < n) ? data[i0 + k] : 0u;
        const uint32_t mine = v[0] + v[1] + v[2] + v[3];
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        if (lane == 31) warp_off[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const uint32_t ws = warp_off[lane];
            uint32_t wi = ws;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= (uint32_t)o) wi += t;
            }
            warp_off[lane] = wi - ws;
        }
        __syncthreads();
        uint32_t run = carry_s + warp_off[warp] + (incl - mine);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i0 + k < n) data[i0 + k] = run;
            run += v[k];
        }
        __syncthreads();
        if (tid == 1023) carry_s = run; // carry + this tile's total
        __syncthreads();
    }
}

// --- pass step 3: stable scatter --------------------------------------------------------
// grid = chunks, block = 256.  (A) every warp counts the digits of its elements (kept in registers),
// (B) the counts become start positions: base of the digit (exclusive prefix of the row totals, done
// here per CTA) + the digit's elements in earlier chunks + the counts of the warps before,
// (C) every warp walks its elements in order, 32 at a time; lanes holding the same digit find each
// other with match_any and take consecutive positions, so equal digits keep their input order.
// No per-element atomics on global memory.
template <uint32_t TILES>
__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(SortKeySrc src, const uint32_t *keys_in,
                                                                     const uint32_t *vals_in, uint32_t n,
                                                                     uint32_t shift, uint32_t bins, uint32_t chunks,
                                                                     const uint32_t *hist, const uint32_t *totals,
                                                                     uint32_t *keys_out, uint32_t *vals_out) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ uint32_t cur[kSortWarps][kMaxBins];
    __shared__ uint32_t base_of[kMaxBins];
    __shared__ uint32_t warp_sum[kSortWarps];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, chunk = blockIdx.x;
    for (uint32_t d = tid; d < kSortWarps * kMaxBins; d += kSortThreads) (&cur[0][0])[d] = 0;
    __syncthreads();
    const uint32_t begin = chunk * (kSortThreads * TILES) + warp * (32 * TILES);
    const uint32_t end = min(n, (chunk + 1) * (kSortThreads * TILES));
    uint32_t key[TILES];
#pragma unroll
    for (uint32_t t = 0; t < TILES; t++) {
        const uint32_t i = begin + t * 32 + lane;
        const bool have = i < end;
        key[t] = have ? (keys_in ? keys_in[i] : slot_key(src, i)) : 0xffffffffu;
        warp_hist_add(cur[warp], (key[t] >> shift) & (bins - 1), have);
    }
    // digit bases: exclusive prefix over totals[0..bins), two digits per thread (bins <= 512)
    {
        const uint32_t d0 = 2 * tid, d1 = 2 * tid + 1;
        const uint32_t v0 = d0 < bins ? totals[d0] : 0u, v1 = d1 < bins ? totals[d1] : 0u;
        uint32_t incl = v0 + v1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        uint32_t before = 0;
        for (uint32_t w = 0; w < warp; w++) before += warp_sum[w];
        const uint32_t excl = before + incl - (v0 + v1);
        if (d0 < bins) base_of[d0] = excl;
        if (d1 < bins) base_of[d1] = excl + v0;
    }
    __syncthreads();
    for (uint32_t d = tid; d < bins; d += kSortThreads) {
        uint32_t run = base_of[d] + hist[d * chunks + chunk];
#pragma unroll
        for (uint32_t w = 0; w < kSortWarps; w++) {
            const uint32_t c = cur[w][d];
            cur[w][d] = run;
            run += c;
        }
    }
    __syncthreads();
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t *mine = cur[warp];
#pragma unroll
    for (uint32_t t = 0; t < TILES; t++) {
        const uint32_t i = begin + t * 32 + lane;
        const bool have = i < end;
        const uint32_t digit = have ? ((key[t] >> shift) & (bins - 1)) : 0xffffffffu;
        const uint32_t peers = __match_any_sync(0xffffffffu, digit);
        const uint32_t rank = __popc(peers & lt);
        uint32_t pos = 0;
        if (have) pos = mine[digit] + rank;
        __syncwarp();
        if (have && rank == 0) mine[digit] += __popc(peers);
        __syncwarp();
        if (have) {
            keys_out[pos] = key[t];
            vals_out[pos] = vals_in ? vals_in[i] : i;
        }
    }
}

// --- send counters ----------------------------------------------------------------------
// Packets of a slot get base, base+1, ... in batch order and the slot's counter moves past them, saturating
// at Reject-After-Messages (packets at or beyond it are refused by the seal kernel).  One thread per packet:
// in the sorted order a packet's rank inside its run is its position minus the start of the run, found by
// binary search, so a peer that owns most of a batch costs no more than any other.  The counters are read
// by the first kernel and advanced by the second, so no thread can see a counter that already moved.
__device__ __forceinline__ uint32_t run_start(const uint32_t *keys, uint32_t j) {
    const uint32_t key = keys[j];
    uint32_t lo = 0, hi = j; // first index in [0, j] whose key equals keys[j]
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (keys[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}
__global__ void assign_counters_kernel(const uint32_t *keys, const uint32_t *order, uint32_t n, uint32_t max_slots,
                                       const SendCounter *send_counter, uint64_t *counter_out) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t slot = keys[j];
    if (slot >= max_slots) return;
    counter_out[order[j]] = saturating_counter(counter_read(&send_counter[slot], ~0ull).now.value, j - run_start(keys, j));
}
__global__ void advance_counters_kernel(const uint32_t *keys, uint32_t n, uint32_t max_slots, SendCounter *send_counter) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t slot = keys[j];
    if (slot >= max_slots || (j + 1 < n && keys[j + 1] == slot)) return; // the last packet of a run moves the counter
    const CounterRead c = counter_read(&send_counter[slot], ~0ull);
    counter_store(&send_counter[slot].e[c.at], SendCounter::Entry{saturating_counter(c.now.value, j - run_start(keys, j) + 1), c.now.seq});
}

// --- anti-replay window, RFC 6479 -------------------------------------------------------
// The window is defined by a sequential walk over a peer's authenticated packets in arrival order: a counter
// above `last` moves the window (clearing the ring words the top passes), one more than a window behind is
// refused, and one in between is accepted unless its bit is already marked.  A GPU cannot afford the walk: a
// peer that owns a large batch would hold the batch up for about a microsecond per 32 packets, and a small
// batch of many peers would pay one dependent chain of loads per peer.  The verdicts have a closed form in
// terms of the state (last, ring) at the start of the batch.  With M_j = max(last, counters of the peer's
// earlier packets of the batch), packet j is accepted iff its counter is below the message limit and either
// exceeds M_j, or lies within the window behind M_j, was not marked in the ring at the start (only counters
// <= last can be) and does not repeat the counter of an earlier packet.  (A ring word that the walk would have
// cleared before reaching j lies more than a window behind M_j; an earlier packet with the same counter that
// was itself refused was refused for a reason that still holds at j.)  Afterwards last = M at the end of the
// run, the words the top moved over are cleared, and the accepted packets within a ring of the new top are
// marked.  Every term is data-parallel over the grouped order:
//   M_j                         a segmented exclusive running maximum (a scan),
//   "marked at the start"       a read of the ring as it was before the batch,
//   "repeats an earlier one"    the lowest grouped position holding the same (peer, counter), found with a
//                               hash table of positions; built only when some packet of the batch lies behind
//                               its M_j inside the window, which in-order traffic never does.
// Up to kGroupMax packets all of this runs in the cluster that sorted them (group_kernel); beyond, as kernels in
// stream order: scan_tiles (also lays the counters out in grouped order), scan_carry, classify, advance (new
// last, clears), hash_clear, hash_insert, finish (duplicate look-up, verdicts, marks).
constexpr uint32_t kScanTile = 1024; // grouped positions per CTA: 256 threads x 4
constexpr uint64_t kReplayNoPart = ~0ull; // grouped-order counter of a packet that takes no part
constexpr uint32_t kHashEmpty = 0xffffffffu;
enum : uint8_t { RP_NOPART = 0, RP_ACCEPT = 1, RP_REJECT = 2, RP_PENDING = 3 };

struct ReplayArgs {
    const uint32_t *keys;  // [n] keypair slots in grouped order
    const uint32_t *order; // [n] packet index of each grouped position
    uint32_t n, max_slots, ring_blocks;
    uint64_t *replay_last, *replay_next, *replay_ring;
    const uint64_t *counter; // per packet, as the open kernel left it
    uint8_t *status;         // per packet
    uint64_t *sorted_counter; // [n] scratch
    uint8_t *state;           // [n] scratch
    uint32_t *table;          // hash table of positions, `mask` + 1 entries
    uint32_t mask;
};

struct SegMax { // running maximum that restarts at every run head
    uint32_t f; // a head lies inside the span
    uint64_t m; // maximum since the last head (or over the whole span)
};
__device__ __forceinline__ SegMax seg_combine(SegMax a, SegMax b) { // a: earlier span, b: the span after it
    return SegMax{a.f | b.f, (b.f || b.m > a.m) ? b.m : a.m};
}
__device__ __forceinline__ SegMax seg_shfl_up(SegMax v, int o) {
    return SegMax{__shfl_up_sync(0xffffffffu, v.f, o), __shfl_up_sync(0xffffffffu, v.m, o)};
}
// Inclusive scan of one value per thread over a CTA of NW warps; returns the exclusive prefix of the calling
// thread and the total of the CTA.  `part` is NW entries of shared memory.
struct CtaSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
template <int NW, typename Sync = CtaSync>
__device__ __forceinline__ SegMax seg_block_exclusive(SegMax mine, SegMax *part, SegMax &total, Sync sync = Sync()) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SegMax inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const SegMax t = seg_shfl_up(inc, o);
        if (lane >= (uint32_t)o) inc = seg_combine(t, inc);
    }
    SegMax ex = seg_shfl_up(inc, 1);
    if (lane == 0) ex = SegMax{0u, 0ull};
    sync(); // `part` may still be read from an earlier call
    if (lane == 31) part[warp] = inc;
    sync();
    SegMax before{0u, 0ull};
    total = SegMax{0u, 0ull};
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        if ((uint32_t)w == warp) before = total;
        total = seg_combine(total, part[w]);
    }
    return seg_combine(before, ex);
}
// ITEMS consecutive grouped positions per thread.  e[k] = maximum of the values of the same run that lie in
// front of item k; total = the tile as one span; what lies in front of the tile comes in with tile_carry.
struct TileMax {
    SegMax ex;
    uint32_t headed; // bit k: a head lies at or before item k inside this thread
};
template <int ITEMS, int NW>
__device__ __forceinline__ TileMax tile_running_max(const bool (&head)[ITEMS], const uint64_t (&v)[ITEMS],
                                                    uint64_t (&e)[ITEMS], SegMax *part, SegMax &total) {
    SegMax run{0u, 0ull};
    TileMax t{SegMax{0u, 0ull}, 0u};
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (head[k]) run = SegMax{1u, 0ull};
        e[k] = run.m;
        t.headed |= run.f << k;
        if (v[k] > run.m) run.m = v[k];
    }
    t.ex = seg_block_exclusive<NW>(run, part, total);
    return t;
}
template <int ITEMS>
__device__ __forceinline__ void tile_carry(const TileMax &t, uint64_t carry, uint64_t (&e)[ITEMS]) {
    const uint64_t front = t.ex.f ? t.ex.m : (carry > t.ex.m ? carry : t.ex.m);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k)
        if (!((t.headed >> k) & 1u) && front > e[k]) e[k] = front;
}

// Counter of grouped position p, or kReplayNoPart.  Authenticated packets at or beyond the message limit are
// refused here: their verdict does not depend on the window and they leave no trace in it.
__device__ __forceinline__ uint64_t replay_gather(const ReplayArgs &a, uint32_t p, uint32_t slot, uint32_t pkt) {
    uint64_t c = kReplayNoPart;
    if (slot < a.max_slots) {
        const uint8_t st = a.status[pkt];
        if (st == BNK_PKT_OK || st == BNK_PKT_KEEPALIVE) {
            c = a.counter[pkt];
            if (c >= BNK_REJECT_AFTER_MESSAGES) {
                a.status[pkt] = BNK_PKT_REPLAY;
                c = kReplayNoPart;
            }
        }
    }
    a.sorted_counter[p] = c;
    return c;
}
// Verdict of position p as far as it can be told without the duplicate search; the last packet of a run also
// leaves the peer's next `last`.  e = running maximum of the run in front of p.
__device__ __forceinline__ uint8_t replay_classify(const ReplayArgs &a, uint32_t p, uint32_t slot, bool tail, uint64_t c, uint64_t e) {
    if (slot >= a.max_slots) return RP_NOPART;
    const uint64_t rmask = a.ring_blocks - 1, window = (uint64_t)(a.ring_blocks - 1) * 64u;
    const uint64_t last = a.replay_last[slot];
    const uint64_t M = e > last ? e : last;
    uint8_t st = RP_NOPART;
    uint64_t top = M;
    if (c != kReplayNoPart) {
        if (c > M) {
            st = RP_ACCEPT;
            top = c;
        } else if (M - c > window) st = RP_REJECT;
        else if (c <= last && ((a.replay_ring[(size_t)slot * a.ring_blocks + ((c >> 6) & rmask)] >> (c & 63u)) & 1ull))
            st = RP_REJECT;
        else st = RP_PENDING;
    }
    if (tail) a.replay_next[slot] = top;
    return st;
}
// Warp-wide over 32 consecutive positions (p = this lane's): the peers whose run ends here move their window.
__device__ __forceinline__ void replay_advance_warp(const ReplayArgs &a, uint32_t p) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t key = p < a.n ? a.keys[p] : 0xffffffffu;
    const bool is_tail = p < a.n && key < a.max_slots && (p + 1 == a.n || a.keys[p + 1] != key);
    uint32_t tails = __ballot_sync(0xffffffffu, is_tail);
    const uint64_t rmask = a.ring_blocks - 1;
    while (tails) {
        const uint32_t src = __ffs(tails) - 1;
        tails &= tails - 1;
        const uint32_t slot = __shfl_sync(0xffffffffu, key, src);
        uint64_t *ring = a.replay_ring + (size_t)slot * a.ring_blocks;
        const uint64_t last = a.replay_last[slot], next = a.replay_next[slot];
        const uint64_t top = last >> 6;
        uint64_t steps = (next >> 6) - top;
        if (steps > a.ring_blocks) steps = a.ring_blocks;
        for (uint64_t i = lane; i < steps; i += 32) ring[(top + 1 + i) & rmask] = 0ull;
        __syncwarp();
        if (lane == 0) a.replay_last[slot] = next;
    }
}
__device__ __forceinline__ uint32_t replay_hash(uint32_t slot, uint64_t c) {
    uint64_t x = c * 0x9E3779B97F4A7C15ull + slot;
    x ^= x >> 29;
    x *= 0xBF58476D1CE4E5B9ull;
    x ^= x >> 32;
    return (uint32_t)x;
}
// table[h] = lowest grouped position that holds the key (peer, counter); the key of an entry is read through
// the position it holds and never changes, so a probe may compare against whatever position it sees.
// Warp-wide (32 consecutive positions, `active` per lane): of the lanes that hold the same key only the lowest,
// which has the lowest position, goes to the table, so a burst of copies of one packet costs one atomic per
// warp instead of one per copy.
__device__ __forceinline__ void replay_hash_insert_warp(const ReplayArgs &a, uint32_t p, bool active) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t slot = active ? a.keys[p] : 0u;
    const uint64_t c = active ? a.sorted_counter[p] : 0ull;
    const unsigned long long tag = active ? (c * 0x9E3779B97F4A7C15ull + slot) : ~0ull - lane;
    const uint32_t same_tag = __match_any_sync(0xffffffffu, tag);
    const uint32_t first = __ffs(same_tag) - 1;
    const uint32_t first_slot = __shfl_sync(0xffffffffu, slot, first);
    const uint64_t first_c = __shfl_sync(0xffffffffu, c, first);
    if (!active || (lane != first && first_slot == slot && first_c == c)) return; // a lower lane carries this key
    uint32_t h = replay_hash(slot, c) & a.mask;
    for (uint32_t probes = 0; probes <= a.mask; ++probes, h = (h + 1) & a.mask) {
        uint32_t cur = *(volatile uint32_t *)&a.table[h];
        if (cur == kHashEmpty) {
            cur = atomicCAS(&a.table[h], kHashEmpty, p);
            if (cur == kHashEmpty) return;
        }
        if (a.keys[cur] == slot && a.sorted_counter[cur] == c) {
            atomicMin(&a.table[h], p);
            return;
        }
    }
}
__device__ __forceinline__ bool replay_hash_has_earlier(const ReplayArgs &a, uint32_t p, uint32_t slot, uint64_t c) {
    uint32_t h = replay_hash(slot, c) & a.mask;
    for (uint32_t probes = 0; probes <= a.mask; ++probes, h = (h + 1) & a.mask) {
        const uint32_t cur = *(volatile uint32_t *)&a.table[h];
        if (cur == kHashEmpty) return false;
        if (a.keys[cur] == slot && a.sorted_counter[cur] == c) return cur < p;
    }
    return false;
}
// Warp-wide: marks the accepted counters in the rings.  Lanes that hit the same ring word hand their bits to the lowest
// of them.
__device__ __forceinline__ void replay_mark_warp(const ReplayArgs &a, bool accepted, uint32_t slot, uint64_t c) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t rmask = a.ring_blocks - 1;
    const bool mark = accepted && (a.replay_last[slot] >> 6) - (c >> 6) < a.ring_blocks;
    const unsigned long long word = mark ? (unsigned long long)slot * a.ring_blocks + ((c >> 6) & rmask) : ~0ull - lane;
    const uint32_t group = __match_any_sync(0xffffffffu, word);
    const bool leader = mark && (uint32_t)(__ffs(group) - 1) == lane;
    uint32_t leaders = __ballot_sync(0xffffffffu, leader);
    const uint32_t bit_lo = mark && (c & 32u) == 0 ? 1u << (c & 31u) : 0u;
    const uint32_t bit_hi = mark && (c & 32u) != 0 ? 1u << (c & 31u) : 0u;
    unsigned long long *ring = reinterpret_cast<unsigned long long *>(a.replay_ring);
    if (__popc(leaders) <= 4) {
        while (leaders) {
            const uint32_t src = __ffs(leaders) - 1;
            leaders &= leaders - 1;
            const uint32_t members = __shfl_sync(0xffffffffu, group, src);
            const bool in = (members >> lane) & 1u;
            const uint32_t lo = __reduce_or_sync(0xffffffffu, in ? bit_lo : 0u);
            const uint32_t hi = __reduce_or_sync(0xffffffffu, in ? bit_hi : 0u);
            if (lane == src) atomicOr(&ring[word], ((unsigned long long)hi << 32) | lo);
        }
    } else if (mark) {
        atomicOr(&ring[word], ((unsigned long long)bit_hi << 32) | bit_lo);
    }
}
// Warp-wide over 32 consecutive positions: settles the pending verdicts, writes the refusals and marks the ring.
__device__ __forceinline__ void replay_finish_warp(const ReplayArgs &a, uint32_t p) {
    uint8_t st = p < a.n ? a.state[p] : (uint8_t)RP_NOPART;
    uint32_t slot = 0;
    uint64_t c = 0;
    if (st != RP_NOPART) {
        slot = a.keys[p];
        c = a.sorted_counter[p];
    }
    if (st == RP_PENDING) st = replay_hash_has_earlier(a, p, slot, c) ? RP_REJECT : RP_ACCEPT;
    if (st == RP_REJECT) a.status[a.order[p]] = BNK_PKT_REPLAY;
    replay_mark_warp(a, st == RP_ACCEPT, slot, c);
}
// The tile of the calling CTA (thread t: positions base..base+3): counters gathered when GATHER, else read
// back; running maximum with `carry` in front; returns the tile as one span.
template <bool GATHER>
__device__ __forceinline__ SegMax replay_tile(const ReplayArgs &a, uint32_t base, uint64_t carry, uint32_t (&slot)[4],
                                              uint64_t (&c)[4], uint64_t (&e)[4], SegMax *part) {
    bool head[4];
    uint64_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t p = base + k;
        head[k] = false;
        v[k] = 0;
        c[k] = kReplayNoPart;
        slot[k] = 0xffffffffu;
        if (p < a.n) {
            slot[k] = a.keys[p];
            head[k] = p == 0 || a.keys[p - 1] != slot[k];
            c[k] = GATHER ? replay_gather(a, p, slot[k], a.order[p]) : a.sorted_counter[p];
            if (c[k] != kReplayNoPart) v[k] = c[k];
        }
    }
    SegMax total;
    const TileMax t = tile_running_max<4, 8>(head, v, e, part, total);
    tile_carry<4>(t, carry, e);
    return total;
}

__global__ void __launch_bounds__(256) replay_scan_tiles_kernel(ReplayArgs a, uint32_t *tile_head, uint64_t *tile_max,
                                                                uint32_t *pending_flag) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ SegMax part[8];
    if (blockIdx.x == 0 && threadIdx.x == 0) *pending_flag = 0u;
    uint32_t slot[4];
    uint64_t c[4], e[4];
    const SegMax total = replay_tile<true>(a, blockIdx.x * kScanTile + threadIdx.x * 4u, 0ull, slot, c, e, part);
    if (threadIdx.x == 0) {
        tile_head[blockIdx.x] = total.f;
        tile_max[blockIdx.x] = total.m;
    }
}
// One CTA: carry[t] = running maximum that reaches tile t from the tiles in front of it.
__global__ void __launch_bounds__(1024) replay_scan_carry_kernel(const uint32_t *tile_head, const uint64_t *tile_max,
                                                                 uint32_t tiles, uint64_t *tile_carry) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ SegMax part[32];
    SegMax reached{0u, 0ull};
    for (uint32_t base = 0; base < tiles; base += 1024u) {
        const uint32_t t = base + threadIdx.x;
        SegMax mine{0u, 0ull};
        if (t < tiles) mine = SegMax{tile_head[t], tile_max[t]};
        SegMax total;
        const SegMax ex = seg_block_exclusive<32>(mine, part, total);
        if (t < tiles) tile_carry[t] = seg_combine(reached, ex).m;
        reached = seg_combine(reached, total);
    }
}
__global__ void __launch_bounds__(256) replay_classify_kernel(ReplayArgs a, const uint64_t *tile_carry,
                                                              uint32_t *pending_flag) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ SegMax part[8];
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * 4u;
    uint32_t slot[4];
    uint64_t c[4], e[4];
    replay_tile<false>(a, base, tile_carry[blockIdx.x], slot, c, e, part);
    bool pending = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (base + k >= a.n) continue;
        const bool tail = base + k + 1 == a.n || a.keys[base + k + 1] != slot[k];
        const uint8_t st = replay_classify(a, base + k, slot[k], tail, c[k], e[k]);
        a.state[base + k] = st;
        pending |= st == RP_PENDING;
    }
    if (__syncthreads_or(pending) && threadIdx.x == 0) *pending_flag = 1u;
}
__global__ void __launch_bounds__(256) replay_advance_kernel(ReplayArgs a) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    replay_advance_warp(a, blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void __launch_bounds__(256) replay_hash_clear_kernel(ReplayArgs a, const uint32_t *pending_flag) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    if (*pending_flag == 0u) return;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= a.mask; i += gridDim.x * blockDim.x) a.table[i] = kHashEmpty;
}
__global__ void __launch_bounds__(256) replay_hash_insert_kernel(ReplayArgs a, const uint32_t *pending_flag) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    if (*pending_flag == 0u) return;
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    replay_hash_insert_warp(a, p, p < a.n && a.state[p] != RP_NOPART);
}
__global__ void __launch_bounds__(256) replay_finish_kernel(ReplayArgs a) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    replay_finish_warp(a, blockIdx.x * blockDim.x + threadIdx.x);
}
// The last checks alone, one thread per packet.
__global__ void __launch_bounds__(256) verdict_kernel(const __grid_constant__ VerdictArgs v, Done done) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < v.n) final_verdict(v, i);
    signal_done(done, false, [] {});
}

// --- the whole ordering work of a batch of up to kGroupMax packets in one launch --------
// The same stable radix sort, the counters or the replay window behind it and the last checks behind that, by one
// cluster of up to 16 CTAs of 512 threads with 1 to 4 packets a thread.  As kernels in stream order this is up to
// twenty launches of a few microseconds' work each, and a batch of a few thousand packets spent more time in front of
// and between them than in them (a 4096-packet open with every check: 20 launches).  Keys and indices ping-pong
// between shared-memory buffers; the CTAs read each other's digit totals, and the scatter writes into the buffer of
// the CTA that a position belongs to, through distributed shared memory; cluster barriers stand where kernel
// boundaries stood.  Up to 256 packets the sort is a count: the place of a packet is the number of packets with a
// lower key, or the same key and a lower index.
constexpr uint32_t kGroupThreads = 512, kGroupWarps = kGroupThreads / 32, kGroupCtas = 16;
static_assert(kGroupMax == kGroupThreads * 4 * kGroupCtas, "4 packets a thread at most");

struct GroupArgs {
    SortKeySrc src;
    uint32_t n, passes, digit_bits, max_slots;
    // counters (send_counter != nullptr)
    SendCounter *send_counter;
    uint64_t *counter_out; // per packet
    // replay window (replay): rp.keys are written here
    uint32_t *keys_out;
    ReplayArgs rp;
    bool replay;
    VerdictArgs verdict; // n == 0: none
    Done done;
};

// A packet behind its window's top looks through so many of its peer's packets in front of it for its counter; only where that is
// not all of them is the table of positions built.  Opened with everything on, us with the table always / so: 2068 mixed packets of 256
// peers 88 / 82, 4136 109 / 103, 10,100 201 / 193, 16,160 of 1000 peers 287 / 262; of 8 peers, whose runs are longer, 4136 106 / 112.
constexpr uint32_t kLookBack = 64;
template <int ITEMS>
__global__ void __launch_bounds__(kGroupThreads, 1) group_kernel(const __grid_constant__ GroupArgs a) {
    let_next_kernel_start();    // seal side: the seal launch behind may take its place already
    wait_for_kernel_in_front(); // open side: statuses and counters come from the open launch in front
    constexpr uint32_t kChunk = kGroupThreads * ITEMS; // positions per CTA
    extern __shared__ __align__(16) uint32_t dyn[];
    auto kbuf = [&](uint32_t half) { return dyn + half * kChunk; };
    auto vbuf = [&](uint32_t half) { return dyn + (2 + half) * kChunk; };
    uint16_t *const cnt = reinterpret_cast<uint16_t *>(dyn + 4 * kChunk); // [kGroupWarps][kMaxBins]
    __shared__ uint32_t hist[kMaxBins], base_of[kMaxBins], warp_sum[kGroupWarps];
    __shared__ SegMax part[kGroupWarps];
    __shared__ SegMax cta_total;
    __shared__ uint32_t cta_head, cta_pending;
    const cg::cluster_group cluster = cg::this_cluster();
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ctas = gridDim.x, me = blockIdx.x;
    auto all_sync = [&] {
        if (ctas > 1) cluster.sync();
        else __syncthreads();
    };
    const uint32_t first = me * kChunk; // this CTA's positions (and, before the sort, its packets)
    const uint32_t mine = a.n > first ? min(kChunk, a.n - first) : 0u;
    if (a.replay) // (in case some packet turns out to need the table)
        for (uint32_t i = me * kGroupThreads + tid; i <= a.rp.mask; i += ctas * kGroupThreads) a.rp.table[i] = kHashEmpty;

    // ---- sort ----
    uint32_t f = 0; // which buffer holds the result
    if (a.n <= 256) { // one CTA
        const uint32_t key = tid < a.n ? slot_key(a.src, tid) : 0xffffffffu;
        if (tid < 256) kbuf(0)[tid] = key;
        __syncthreads();
        uint32_t place = 0;
        for (uint32_t j = 0; j < a.n; j++) {
            const uint32_t other = kbuf(0)[j];
            place += (other < key || (other == key && j < tid)) ? 1u : 0u;
        }
        f = 1;
        if (tid < a.n) {
            kbuf(1)[place] = key;
            vbuf(1)[place] = tid;
        }
        __syncthreads();
    } else {
        const uint32_t bins = 1u << a.digit_bits, lt = (1u << lane) - 1u;
        for (uint32_t p = 0; p < a.passes; p++, f ^= 1u) {
            const uint32_t shift = p * a.digit_bits;
            for (uint32_t d = tid; d < kGroupWarps * kMaxBins / 8; d += kGroupThreads) reinterpret_cast<uint4 *>(cnt)[d] = make_uint4(0, 0, 0, 0);
            __syncthreads();
            uint16_t *const my_cnt = cnt + warp * kMaxBins;
            uint32_t key[ITEMS], val[ITEMS], rank[ITEMS];
#pragma unroll
            for (int t = 0; t < ITEMS; t++) { // a warp owns 32 * ITEMS consecutive packets
                const uint32_t e = warp * (32 * ITEMS) + t * 32 + lane;
                const bool have = e < mine;
                key[t] = have ? (p == 0 ? slot_key(a.src, first + e) : kbuf(f)[e]) : 0xffffffffu;
                val[t] = have ? (p == 0 ? first + e : vbuf(f)[e]) : 0u;
                const uint32_t digit = have ? (key[t] >> shift) & (bins - 1) : 0xffffffffu;
                const uint32_t peers = __match_any_sync(0xffffffffu, digit);
                rank[t] = __popc(peers & lt);
                if (have) rank[t] += my_cnt[digit];
                __syncwarp();
                if (have && (peers & lt) == 0) my_cnt[digit] += (uint16_t)__popc(peers);
                __syncwarp();
            }
            __syncthreads();
            if (tid < bins) { // counts of the warps -> their starts inside the CTA's share of the digit
                uint32_t run = 0;
#pragma unroll
                for (uint32_t w = 0; w < kGroupWarps; w++) {
                    const uint32_t c = cnt[w * kMaxBins + tid];
                    cnt[w * kMaxBins + tid] = (uint16_t)run;
                    run += c;
                }
                hist[tid] = run;
            }
            all_sync();
            uint32_t before = 0, all = 0; // of digit `tid`: in the CTAs in front, in all CTAs
            if (tid < bins) {
                for (uint32_t c = 0; c < ctas; c++) {
                    const uint32_t v = ctas > 1 ? cluster.map_shared_rank(hist, c)[tid] : hist[tid];
                    if (c < me) before += v;
                    all += v;
                }
            }
            uint32_t incl = all;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += t;
            }
            if (lane == 31) warp_sum[warp] = incl;
            __syncthreads();
            for (uint32_t w = 0; w < warp; w++) before += warp_sum[w];
            if (tid < bins) base_of[tid] = before + incl - all;
            __syncthreads();
#pragma unroll
            for (int t = 0; t < ITEMS; t++) {
                const uint32_t e = warp * (32 * ITEMS) + t * 32 + lane;
                if (e < mine) {
                    const uint32_t digit = (key[t] >> shift) & (bins - 1);
                    const uint32_t pos = base_of[digit] + my_cnt[digit] + rank[t], to = pos / kChunk, at = pos % kChunk;
                    uint32_t *const kout = ctas > 1 ? cluster.map_shared_rank(kbuf(f ^ 1u), to) : kbuf(f ^ 1u);
                    uint32_t *const vout = ctas > 1 ? cluster.map_shared_rank(vbuf(f ^ 1u), to) : vbuf(f ^ 1u);
                    kout[at] = key[t];
                    vout[at] = val[t];
                }
            }
            all_sync();
        }
    }

    // ---- the grouped order: ITEMS consecutive positions a thread ----
    const uint32_t at0 = tid * ITEMS;
    uint32_t slot[ITEMS];
    bool head[ITEMS], tail[ITEMS];
    {
        uint32_t prev = 0xffffffffu;
        if (at0 > 0) prev = kbuf(f)[at0 - 1];
        else if (me > 0) prev = cluster.map_shared_rank(kbuf(f), me - 1)[kChunk - 1];
        uint32_t next = 0xffffffffu; // key behind the thread's last position
        if (at0 + ITEMS < mine) next = kbuf(f)[at0 + ITEMS];
        else if (at0 + ITEMS == kChunk && first + kChunk < a.n) next = cluster.map_shared_rank(kbuf(f), me + 1)[0];
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            slot[k] = at0 + k < mine ? kbuf(f)[at0 + k] : 0xffffffffu;
            head[k] = at0 + k < mine && ((first + at0 + k) == 0 || slot[k] != prev);
            prev = slot[k];
        }
#pragma unroll
        for (int k = 0; k < ITEMS; k++)
            tail[k] = at0 + k < mine && slot[k] != (k + 1 < ITEMS ? slot[k + 1] : next);
    }

    if (a.send_counter) {
        // start of the run a position lies in: running maximum of the head positions (+1; 0 = none yet)
        uint32_t run = 0;
#pragma unroll
        for (int k = 0; k < ITEMS; k++)
            if (head[k]) run = first + at0 + k + 1;
        uint32_t incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl = max(incl, t);
        }
        uint32_t front = __shfl_up_sync(0xffffffffu, incl, 1);
        if (lane == 0) front = 0;
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        uint32_t whole = 0;
        for (uint32_t w = 0; w < kGroupWarps; w++) {
            if (w < warp) front = max(front, warp_sum[w]);
            whole = max(whole, warp_sum[w]);
        }
        if (ctas > 1) {
            if (tid == 0) cta_head = whole;
            cluster.sync();
            for (uint32_t c = 0; c < me; c++) front = max(front, *cluster.map_shared_rank(&cta_head, c));
        }
        CounterRead counter[ITEMS];
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const uint32_t p = first + at0 + k;
            if (head[k]) front = p + 1;
            if (at0 + k >= mine || slot[k] >= a.max_slots) continue;
            counter[k] = counter_read(&a.send_counter[slot[k]], ~0ull);
            const uint32_t rank = p + 1 - front;
            a.counter_out[vbuf(f)[at0 + k]] = saturating_counter(counter[k].now.value, rank);
            counter[k].now.value = saturating_counter(counter[k].now.value, rank + 1);
        }
        all_sync(); // every counter is read
#pragma unroll
        for (int k = 0; k < ITEMS; k++)
            if (tail[k] && slot[k] < a.max_slots) counter_store(&a.send_counter[slot[k]].e[counter[k].at], counter[k].now);
    }

    // The window and the last checks wait for memory and for one another, so a thread keeps what it knows of its positions, asks
    // for all that nothing else has to be known for in front of a barrier, and the barriers are as few as the window's definition
    // wants: one for the running maximum, one behind the reads of the old window, one behind its move, one to put the results in
    // the packets' order.  (Each phase reading what the one before had left in memory, with a thread of its own: 2068 packets of 256
    // peers 33 us from the open kernel's end, now 22.)
    if (a.replay) {
        const ReplayArgs &r = a.rp;
        const uint64_t rmask = r.ring_blocks - 1, window = (uint64_t)(r.ring_blocks - 1) * 64u;
        uint64_t c[ITEMS], e[ITEMS], v[ITEMS], last[ITEMS];
        uint32_t pkt[ITEMS];
        uint8_t had[ITEMS], st[ITEMS]; // the packet's status so far; what the window says
#pragma unroll
        for (int k = 0; k < ITEMS; k++) { // asked for together
            pkt[k] = 0;
            c[k] = last[k] = 0;
            had[k] = BNK_PKT_BAD_DESC;
            if (at0 + k >= mine) continue;
            pkt[k] = vbuf(f)[at0 + k];
            had[k] = r.status[pkt[k]];
            c[k] = r.counter[pkt[k]];
            if (slot[k] < r.max_slots) last[k] = r.replay_last[slot[k]];
        }
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const bool authentic = at0 + k < mine && slot[k] < r.max_slots && (had[k] == BNK_PKT_OK || had[k] == BNK_PKT_KEEPALIVE);
            st[k] = authentic && c[k] >= BNK_REJECT_AFTER_MESSAGES ? RP_REJECT : RP_NOPART; // (whatever the window holds, and without a trace)
            if (!authentic || st[k] == RP_REJECT) c[k] = kReplayNoPart;
            v[k] = c[k] != kReplayNoPart ? c[k] : 0ull;
            if (at0 + k < mine) {
                a.keys_out[first + at0 + k] = slot[k];
                r.sorted_counter[first + at0 + k] = c[k];
                kbuf(f ^ 1u)[at0 + k] = (uint32_t)c[k]; // the counters in grouped order, beside the slots in kbuf(f)
                vbuf(f ^ 1u)[at0 + k] = (uint32_t)(c[k] >> 32);
            }
        }
        SegMax total;
        const TileMax t = tile_running_max<ITEMS, kGroupWarps>(head, v, e, part, total);
        if (tid == 0) {
            cta_total = total;
            cta_pending = 0;
        }
        all_sync();
        SegMax reached{0u, 0ull};
        for (uint32_t q = 0; q < me; q++) reached = seg_combine(reached, *cluster.map_shared_rank(&cta_total, q));
        tile_carry<ITEMS>(t, reached.m, e);
        bool pending = false;
#pragma unroll
        for (int k = 0; k < ITEMS; k++) { // e becomes the peer's `last` behind this packet
            e[k] = e[k] > last[k] ? e[k] : last[k];
            if (c[k] == kReplayNoPart) continue;
            if (c[k] > e[k]) {
                st[k] = RP_ACCEPT;
                e[k] = c[k];
            } else if (e[k] - c[k] > window ||
                       (c[k] <= last[k] && ((r.replay_ring[(size_t)slot[k] * r.ring_blocks + ((c[k] >> 6) & rmask)] >> (c[k] & 63u)) & 1ull))) {
                st[k] = RP_REJECT;
            } else { // accepted unless an earlier packet of the run has the same counter
                st[k] = RP_PENDING;
                const uint32_t at = at0 + k; // of this CTA; what lies in front of it is the end of the one before
                const auto looks = [&](const uint32_t *keys, const uint32_t *lo, const uint32_t *hi, uint32_t from, uint32_t to) {
#pragma unroll 1
                    for (uint32_t q = from; q-- > to;) {
                        if (keys[q] != slot[k]) return RP_ACCEPT; // the run has started behind it
                        if (lo[q] == (uint32_t)c[k] && hi[q] == (uint32_t)(c[k] >> 32)) return RP_REJECT;
                    }
                    return RP_PENDING;
                };
                const uint32_t *const keys = at >= kLookBack || me == 0 ? kbuf(f) : cluster.map_shared_rank(kbuf(f), me - 1);
                if (first + at < kLookBack || keys[(at - kLookBack) % kChunk] != slot[k]) { // the run starts within reach
                    st[k] = looks(kbuf(f), kbuf(f ^ 1u), vbuf(f ^ 1u), at, at > kLookBack ? at - kLookBack : 0u);
                    if (st[k] == RP_PENDING && me > 0)
                        st[k] = looks(cluster.map_shared_rank(kbuf(f), me - 1), cluster.map_shared_rank(kbuf(f ^ 1u), me - 1),
                                      cluster.map_shared_rank(vbuf(f ^ 1u), me - 1), kChunk, kChunk - (kLookBack - at));
                    if (st[k] == RP_PENDING) st[k] = RP_ACCEPT; // (it is the batch's first)
                }
                pending |= st[k] == RP_PENDING;
            }
        }
        if (__syncthreads_or(pending) && tid == 0) cta_pending = 1;
        all_sync(); // `last` and the rings are read
        bool any_pending = false;
        for (uint32_t q = 0; q < ctas; q++) any_pending |= (ctas > 1 ? *cluster.map_shared_rank(&cta_pending, q) : cta_pending) != 0;
#pragma unroll
        for (int k = 0; k < ITEMS; k++) { // the peers whose run ends here move their window, a lane each but for large steps
            const bool moves = tail[k] && slot[k] < r.max_slots;
            const uint64_t from = last[k] >> 6, passed = (e[k] >> 6) - from, steps = !moves ? 0u : passed < r.ring_blocks ? passed : r.ring_blocks;
            uint64_t *const ring = r.replay_ring + (moves ? (size_t)slot[k] * r.ring_blocks : 0u);
            if (steps <= 8)
                for (uint64_t i = 1; i <= steps; i++) ring[(from + i) & rmask] = 0ull;
            uint32_t large = __ballot_sync(0xffffffffu, steps > 8);
            while (large) {
                const uint32_t src = __ffs(large) - 1;
                large &= large - 1;
                uint64_t *const of = reinterpret_cast<uint64_t *>(__shfl_sync(0xffffffffu, (unsigned long long)ring, src));
                const uint64_t at = __shfl_sync(0xffffffffu, from, src), many = __shfl_sync(0xffffffffu, steps, src);
                for (uint64_t i = lane + 1; i <= many; i += 32) of[(at + i) & rmask] = 0ull;
            }
            if (moves) r.replay_last[slot[k]] = e[k];
            if (any_pending) replay_hash_insert_warp(r, first + at0 + k, c[k] != kReplayNoPart);
        }
        // The last checks want much of memory too, and none of it depends on what is being written.
        const VerdictArgs &w = a.verdict;
        uint32_t len[ITEMS], whole[ITEMS];
        uint8_t found[ITEMS], proto[ITEMS];
        FlowReply reply[ITEMS];
        bool ask_flows[ITEMS];
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            len[k] = whole[k] = proto[k] = 0;
            found[k] = had[k];
            ask_flows[k] = false;
            if (w.n == 0 || at0 + k >= mine) continue;
            len[k] = whole[k] = w.out_len[pkt[k]];
            if (had[k] == BNK_PKT_OK && st[k] != RP_REJECT) checks_begin(w, pkt[k], slot[k], found[k], len[k], proto[k], reply[k], ask_flows[k]);
        }
        all_sync(); // clears before marks, inserts before look-ups
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            if (st[k] == RP_PENDING) st[k] = replay_hash_has_earlier(r, first + at0 + k, slot[k], c[k]) ? RP_REJECT : RP_ACCEPT;
            replay_mark_warp(r, st[k] == RP_ACCEPT, slot[k], c[k]);
            if (at0 + k >= mine) continue;
            if (st[k] == RP_REJECT) {
                found[k] = BNK_PKT_REPLAY;
                len[k] = whole[k];
            } else if (ask_flows[k]) {
                found[k] = reply[k].finish(w.ft, proto[k], w.now);
            }
            r.status[pkt[k]] = found[k];
            if (w.n == 0) continue;
            w.out_len[pkt[k]] = len[k];
            if (w.host_status) { // to whose packet it is, so that what goes to the host goes in whole lines
                const uint32_t to = pkt[k] / kChunk, at = pkt[k] % kChunk;
                (ctas > 1 ? cluster.map_shared_rank(kbuf(f ^ 1u), to) : kbuf(f ^ 1u))[at] = len[k];
                (ctas > 1 ? cluster.map_shared_rank(vbuf(f ^ 1u), to) : vbuf(f ^ 1u))[at] = found[k];
            }
        }
        if (w.n && w.host_status) {
            all_sync();
            for (uint32_t i = tid; i < mine; i += kGroupThreads) {
                w.host_status[first + i] = (uint8_t)vbuf(f ^ 1u)[i];
                w.host_out_len[first + i] = kbuf(f ^ 1u)[i];
            }
        }
    }
    // (Nobody has looked into another's shared memory since the last barrier.)
    signal_done(a.done, false, [] {});
}

// --- what follows the open kernel of up to kTailMax packets -----------------------------
// Here nothing but latency counts, and group_kernel's phases wait for one another.  In this one CTA eight warps group the packets and run the replay window
// in registers and shared memory, while the other eight already look the packets' flows and rules up; who judges a
// packet then has everything in hand.
constexpr uint32_t kTailMax = 256;
struct HalfSync { // of the first 256 threads
    __device__ __forceinline__ void operator()() const { asm volatile("bar.sync 1, 256;" ::: "memory"); }
};
__global__ void __launch_bounds__(512) open_tail_kernel(const __grid_constant__ ReplayArgs r, const uint32_t *slots,
                                                        const __grid_constant__ VerdictArgs v, Done done) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ __align__(16) uint32_t key_of[kTailMax];
    __shared__ uint32_t sorted_key[kTailMax];
    __shared__ uint64_t sorted_ctr[kTailMax];
    __shared__ uint8_t sorted_pkt[kTailMax], refused[kTailMax];
    __shared__ SegMax part[8];
    const uint32_t tid = threadIdx.x, n = v.n;
    if (tid < kTailMax) { // ---- the replay window; the steps and their reasons are those of replay_*_kernel ----
        const HalfSync half_sync;
        const uint32_t lane = tid & 31;
        uint32_t key = 0xffffffffu;
        uint64_t c = kReplayNoPart;
        bool beyond = false; // authenticated, at or beyond the message limit
        if (tid < n) {
            const uint32_t slot = slots[tid];
            const uint8_t st = *(const volatile uint8_t *)&v.status[tid];
            const uint64_t ctr = r.counter[tid];
            key = min(slot, r.max_slots);
            if (key < r.max_slots && (st == BNK_PKT_OK || st == BNK_PKT_KEEPALIVE)) {
                beyond = ctr >= BNK_REJECT_AFTER_MESSAGES;
                if (!beyond) c = ctr;
            }
        }
        key_of[tid] = key;
        refused[tid] = beyond;
        half_sync();
        uint32_t place = 0; // packets with a lower key, or the same key and a lower index
        for (uint32_t j = 0; j < n; j += 4) {
            const uint4 other = *reinterpret_cast<const uint4 *>(&key_of[j]);
            place += (other.x < key + (j < tid)) + (other.y < key + (j + 1 < tid)) + (other.z < key + (j + 2 < tid)) + (other.w < key + (j + 3 < tid));
        }
        if (tid < n) {
            sorted_key[place] = key;
            sorted_ctr[place] = c;
            sorted_pkt[place] = (uint8_t)tid;
        }
        half_sync();
        const bool real = tid < n && sorted_key[tid] < r.max_slots; // from here on tid is a grouped position
        const uint32_t slot = real ? sorted_key[tid] : 0u;
        const bool head = tid < n && (tid == 0 || sorted_key[tid - 1] != sorted_key[tid]);
        const bool tail = real && (tid + 1 == n || sorted_key[tid + 1] != slot);
        c = real ? sorted_ctr[tid] : kReplayNoPart;
        const uint64_t rmask = r.ring_blocks - 1, window = (uint64_t)(r.ring_blocks - 1) * 64u;
        uint64_t *const ring = r.replay_ring + (size_t)slot * r.ring_blocks;
        const uint64_t last = real ? r.replay_last[slot] : 0;
        const uint64_t word = c != kReplayNoPart ? ring[(c >> 6) & rmask] : 0;
        SegMax mine{head, c != kReplayNoPart ? c : 0ull}, total;
        const SegMax ex = seg_block_exclusive<8>(mine, part, total, half_sync);
        const uint64_t e = head ? 0ull : ex.m, M = e > last ? e : last;
        uint8_t st = RP_NOPART;
        uint64_t top = M;
        if (c != kReplayNoPart) {
            if (c > M) {
                st = RP_ACCEPT;
                top = c;
            } else if (M - c > window || (c <= last && ((word >> (c & 63u)) & 1ull))) {
                st = RP_REJECT;
            } else { // accepted unless an earlier packet of the run has the same counter
                st = RP_ACCEPT;
                for (uint32_t q = tid; q-- > 0 && sorted_key[q] == slot;)
                    if (sorted_ctr[q] == c) {
                        st = RP_REJECT;
                        break;
                    }
            }
        }
        half_sync(); // `last` and the ring are read: the peers whose run ends here move their window
        uint32_t tails = __ballot_sync(0xffffffffu, tail && top != last);
        while (tails) {
            const uint32_t src = __ffs(tails) - 1;
            tails &= tails - 1;
            const uint32_t s = __shfl_sync(0xffffffffu, slot, src);
            const uint64_t from = __shfl_sync(0xffffffffu, last, src) >> 6, to = __shfl_sync(0xffffffffu, top, src) >> 6;
            const uint64_t steps = to - from < r.ring_blocks ? to - from : r.ring_blocks;
            for (uint64_t i = lane; i < steps; i += 32) r.replay_ring[(size_t)s * r.ring_blocks + ((from + 1 + i) & rmask)] = 0ull;
        }
        if (tail) r.replay_last[slot] = top;
        half_sync(); // clears before marks
        replay_mark_warp(r, st == RP_ACCEPT, slot, c);
        if (st == RP_REJECT) refused[sorted_pkt[tid]] = 1;
        __syncthreads();
    } else { // ---- the last checks of packet i ----
        const uint32_t i = tid - kTailMax;
        uint8_t st = BNK_PKT_BAD_DESC, found = BNK_PKT_OK; // found: what checks that leave no trace say of it
        uint32_t l = 0, len = 0;
        bool ask_flows = false;
        FlowReply reply;
        uint8_t proto = 0;
        if (i < n) {
            st = *(const volatile uint8_t *)&v.status[i];
            l = len = v.out_len[i];
            if (st == BNK_PKT_OK) checks_begin(v, i, slots[i], found, len, proto, reply, ask_flows);
        }
        __syncthreads();
        if (i < n) {
            uint8_t out = st;
            if (refused[i]) {
                out = BNK_PKT_REPLAY;
                len = l;
            } else if (st == BNK_PKT_OK) {
                out = found == BNK_PKT_OK && ask_flows ? reply.finish(v.ft, proto, v.now) : found;
            }
            v.status[i] = out;
            v.out_len[i] = len;
            if (v.host_status) {
                v.host_status[i] = out;
                v.host_out_len[i] = len;
            }
        }
    }
    signal_done(done, false, [] {});
}

// --- scheduling order by length class (mixed packet sizes) ------------------------------
// Packets with the same number of 64-byte cipher blocks end up next to each other so that
// the lanes of a seal/open warp finish together; classes in falling order of length.  Order inside a class does
// not matter.
constexpr uint32_t kLenBins = 1026;
__device__ __forceinline__ uint32_t len_bin(uint32_t len, bool open_side) {
    uint32_t body = open_side ? (len >= 32u ? len - 32u : 0u) : len;
    uint32_t blocks = (body + 63u) >> 6;
    return blocks > kLenBins - 1 ? kLenBins - 1 : blocks;
}
// Real traffic has a handful of sizes, so nearly all packets fall into three or four bins: atomics straight on
// the global bins serialise there (100,000 warp-level atomics on three addresses took 50 us per million
// packets).  A CTA counts its tile of 2048 packets in shared memory first (lanes with equal bins elect a leader)
// and touches a global bin once per tile; the scatter reserves a range per (tile, bin) the same way and ranks
// inside the range with the shared counters.
constexpr uint32_t kLenItems = 8; // packets per thread
constexpr uint32_t kLenTile = 256 * kLenItems;
__device__ __forceinline__ uint32_t len_tile_count(const uint32_t *len, uint32_t n, int open_side, uint32_t *h,
                                                   uint32_t (&bin)[kLenItems], uint32_t (&rank)[kLenItems]) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t first = blockIdx.x * kLenTile + threadIdx.x;
    for (uint32_t d = threadIdx.x; d < kLenBins; d += 256) h[d] = 0;
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kLenItems; k++) {
        const uint32_t i = first + k * 256u;
        const bool have = i < n;
        bin[k] = have ? len_bin(len[i], open_side) : 0xffffffffu;
        const uint32_t peers = __match_any_sync(0xffffffffu, bin[k]);
        const int leader = __ffs(peers) - 1;
        uint32_t at = 0;
        if (have && leader == (int)lane) at = atomicAdd(&h[bin[k]], __popc(peers));
        rank[k] = __shfl_sync(0xffffffffu, at, leader) + __popc(peers & ((1u << lane) - 1u)); // position inside the tile's bin
    }
    __syncthreads();
    return first;
}
__global__ void __launch_bounds__(256) len_hist_kernel(const uint32_t *len, uint32_t n, int open_side,
                                                       uint32_t *bins) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ uint32_t h[kLenBins];
    uint32_t bin[kLenItems], rank[kLenItems];
    len_tile_count(len, n, open_side, h, bin, rank);
    for (uint32_t d = threadIdx.x; d < kLenBins; d += 256)
        if (h[d]) atomicAdd(&bins[d], h[d]);
}
__global__ void __launch_bounds__(256) len_scatter_kernel(const uint32_t *len, uint32_t n, int open_side,
                                                          uint32_t *bins, uint32_t *order) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    __shared__ uint32_t h[kLenBins];
    uint32_t bin[kLenItems], rank[kLenItems];
    const uint32_t first = len_tile_count(len, n, open_side, h, bin, rank);
    for (uint32_t d = threadIdx.x; d < kLenBins; d += 256)
        if (h[d]) h[d] = atomicAdd(&bins[d], h[d]); // the tile's range in bin d starts here
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kLenItems; k++) {
        const uint32_t i = first + k * 256u;
        // longest class first: the launch then ends with the short packets, whose CTAs take a tenth of the time of
        // the long ones, instead of a last, half-empty wave of the longest
        if (i < n) order[n - 1u - (h[bin[k]] + rank[k])] = i;
    }
}

struct SortPlan {
    uint32_t passes, digit_bits;
};
SortPlan plan_for(uint32_t max_slots) {
    uint32_t bits = 1;
    while ((1ull << bits) <= (uint64_t)max_slots) bits++; // keys run 0..max_slots inclusive
    SortPlan p;
    p.passes = (bits + kMaxDigitBits - 1) / kMaxDigitBits;
    p.digit_bits = (bits + p.passes - 1) / p.passes;
    return p;
}

// elements per lane: the smallest power of two that keeps the chunk count at or below max_chunks
uint32_t tiles_for(uint32_t n, uint32_t max_chunks) {
    uint32_t tiles = 1;
    while (tiles < kMaxTiles && (n + kSortThreads * tiles - 1) / (kSortThreads * tiles) > max_chunks) tiles <<= 1;
    return tiles;
}
uint32_t chunks_for(uint32_t n, uint32_t tiles) { return (n + kSortThreads * tiles - 1) / (kSortThreads * tiles); }

struct SortBuffers {
    uint32_t *keys_a, *keys_b; // the sorted keys end up in keys_b
    uint32_t *vals_a, *order;  // the sorted packet indices end up in order
    uint32_t *hist;            // [bins * chunks]
    uint32_t *totals;          // [bins]
};

template <uint32_t TILES>
void sort_pass(const SortKeySrc &src, const uint32_t *kin, const uint32_t *vin, uint32_t n, uint32_t shift,
               uint32_t bins, uint32_t chunks, const SortBuffers &sb, uint32_t *kout, uint32_t *vout, cudaStream_t s) {
    launch_kernel(n <= dependent_launch_up_to(), radix_hist_kernel<TILES>, dim3(chunks), dim3(kSortThreads), s, src, kin,
        n, shift, bins, chunks, sb.hist);
    launch_kernel(n <= dependent_launch_up_to(), radix_rowscan_kernel,
        dim3((bins * 32 + kSortThreads - 1) / kSortThreads), dim3(kSortThreads), s, sb.hist, bins, chunks, sb.totals);
    launch_kernel(n <= dependent_launch_up_to(), radix_scatter_kernel<TILES>, dim3(chunks), dim3(kSortThreads), s, src,
        kin, vin, n, shift, bins, chunks, sb.hist, sb.totals, kout, vout);
}

// Stable sort of packet indices 0..n-1 by key.  Returns the number of kernel launches.
uint32_t group_sort(const SortKeySrc &src, uint32_t n, uint32_t max_chunks, const SortBuffers &sb, cudaStream_t s) {
    const SortPlan plan = plan_for(src.max_slots);
    const uint32_t bins = 1u << plan.digit_bits;
    const uint32_t tiles = tiles_for(n, max_chunks);
    const uint32_t chunks = chunks_for(n, tiles);
    // ping-pong so that the last pass lands in (keys_b, order)
    uint32_t *kbuf[2] = {sb.keys_b, sb.keys_a};
    uint32_t *vbuf[2] = {sb.order, sb.vals_a};
    const uint32_t *kin = nullptr, *vin = nullptr;
    for (uint32_t p = 0; p < plan.passes; p++) {
        const uint32_t shift = p * plan.digit_bits;
        const uint32_t o = (plan.passes - 1 - p) & 1u;
        switch (tiles) {
        case 1: sort_pass<1>(src, kin, vin, n, shift, bins, chunks, sb, kbuf[o], vbuf[o], s); break;
        case 2: sort_pass<2>(src, kin, vin, n, shift, bins, chunks, sb, kbuf[o], vbuf[o], s); break;
        case 4: sort_pass<4>(src, kin, vin, n, shift, bins, chunks, sb, kbuf[o], vbuf[o], s); break;
        case 8: sort_pass<8>(src, kin, vin, n, shift, bins, chunks, sb, kbuf[o], vbuf[o], s); break;
        case 16: sort_pass<16>(src, kin, vin, n, shift, bins, chunks, sb, kbuf[o], vbuf[o], s); break;
        default: sort_pass<32>(src, kin, vin, n, shift, bins, chunks, sb, kbuf[o], vbuf[o], s); break;
        }
        kin = kbuf[o];
        vin = vbuf[o];
    }
    return 3 * plan.passes;
}

// Dynamic shared memory of group_kernel<items>.
constexpr size_t group_smem(uint32_t items) { return (size_t)kGroupThreads * items * 16 + kGroupWarps * kMaxBins * 2; }
template <int ITEMS>
cudaError_t launch_group_items(const GroupArgs &a, uint32_t ctas, cudaStream_t s) {
    return launch_shape(LaunchShape{nullptr, dim3(ctas), dim3(kGroupThreads), (uint32_t)group_smem(ITEMS), ctas, true}, group_kernel<ITEMS>, s, a);
}
// One CTA up to 1024 packets (its barriers are cheaper than a cluster's: 600 opened in 37 us against 41), then as many as
// give every packet a thread, up to the 16 a cluster can have here (eight CTAs of two packets a thread and more: 2048
// opened in 54 us against 46, 4096 in 74 against 65, 32,768 in 259 against 243).
cudaError_t launch_group(const GroupArgs &a, cudaStream_t s) {
    uint32_t ctas = 1;
    while (ctas < kGroupCtas && a.n > std::max(ctas, 2u / ctas) * kGroupThreads) ctas *= 2;
    const uint32_t per_thread = (a.n + ctas * kGroupThreads - 1) / (ctas * kGroupThreads);
    if (per_thread <= 1) return launch_group_items<1>(a, ctas, s);
    if (per_thread <= 2) return launch_group_items<2>(a, ctas, s);
    return launch_group_items<4>(a, ctas, s);
}
cudaError_t launch_counters(bnk_ctx *ctx, const uint32_t *slot, uint32_t n, uint64_t *counter, cudaStream_t s) {
    const uint32_t max_slots = ctx->cfg.max_keypairs;
    const SortPlan plan = plan_for(max_slots);
    GroupArgs g{};
    g.src = SortKeySrc{slot, max_slots};
    g.n = n;
    g.passes = plan.passes;
    g.digit_bits = plan.digit_bits;
    g.max_slots = max_slots;
    g.send_counter = ctx->kt.send_counter;
    g.counter_out = counter;
    ctx->launches += 1;
    return launch_group(g, s);
}

} // namespace

cudaError_t group_kernels_init() {
    cudaError_t e = cudaFuncSetAttribute(group_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)group_smem(4));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(group_kernel<1>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(group_kernel<2>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(group_kernel<4>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

// words of histogram scratch a batch of max_pkts packets needs
uint32_t group_sort_chunks(uint32_t max_pkts) {
    const uint32_t worst = chunks_for(max_pkts, kMaxTiles);
    return (worst > kBatchMaxChunks ? worst : kBatchMaxChunks) + 1; // + one row of digit totals
}

// Sorts packet indices 0..n-1 by keypair slot, stable.  Leaves the sorted keys in
// dev.keys_tmp (second half) and the packet indices in dev.order.
cudaError_t launch_group_by_slot(bnk_batch *b, uint32_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    bnk_ctx *ctx = b->ctx;
    DeviceBatch &d = b->dev;
    SortKeySrc src{d.slot, ctx->cfg.max_keypairs};
    SortBuffers sb{d.keys_tmp, d.keys_tmp + b->max_pkts, d.order_tmp, d.order, d.hist + kMaxBins, d.hist};
    ctx->launches += group_sort(src, n, kBatchMaxChunks, sb, s);
    return cudaGetLastError();
}

cudaError_t launch_assign_counters(bnk_batch *b, uint32_t n, const uint32_t *slot, uint64_t *counter, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    bnk_ctx *ctx = b->ctx;
    DeviceBatch &d = b->dev;
    const SortKeySrc src{slot, ctx->cfg.max_keypairs};
    if (n <= kGroupMax) return launch_counters(ctx, slot, n, counter, s);
    SortBuffers sb{d.keys_tmp, d.keys_tmp + b->max_pkts, d.order_tmp, d.order, d.hist + kMaxBins, d.hist};
    ctx->launches += group_sort(src, n, kBatchMaxChunks, sb, s);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    launch_kernel(n <= dependent_launch_up_to(), assign_counters_kernel, dim3((n + 255) / 256), dim3(256), s,
        d.keys_tmp + b->max_pkts, d.order, n, ctx->cfg.max_keypairs, ctx->kt.send_counter, counter);
    launch_kernel(n <= dependent_launch_up_to(), advance_counters_kernel, dim3((n + 255) / 256), dim3(256), s,
        d.keys_tmp + b->max_pkts, n, b->ctx->cfg.max_keypairs, b->ctx->kt.send_counter);
    b->ctx->launches += 2;
    return cudaGetLastError();
}

uint32_t replay_scan_tiles(uint32_t max_pkts) { return (max_pkts + kScanTile - 1) / kScanTile; }
uint32_t replay_hash_capacity(uint32_t max_pkts) {
    uint32_t cap = 1024;
    while (cap < 2u * max_pkts && cap < 0x80000000u) cap <<= 1;
    return cap;
}
static ReplayArgs replay_args(bnk_batch *b, uint32_t n) {
    bnk_ctx *ctx = b->ctx;
    DeviceBatch &d = b->dev;
    uint32_t cap = 1024;
    while (cap < 2u * n) cap <<= 1; // at most half full
    ReplayArgs a{};
    a.keys = d.keys_tmp + b->max_pkts;
    a.order = d.order;
    a.n = n;
    a.max_slots = ctx->cfg.max_keypairs;
    a.ring_blocks = ctx->cfg.replay_ring_blocks;
    a.replay_last = ctx->kt.replay_last;
    a.replay_next = ctx->kt.replay_next;
    a.replay_ring = ctx->kt.replay_ring;
    a.counter = d.counter;
    a.status = d.status;
    a.sorted_counter = d.sorted_counter;
    a.state = d.replay_state;
    a.table = d.replay_hash;
    a.mask = cap - 1;
    return a;
}
cudaError_t launch_open_tail(bnk_batch *b, uint32_t n, bool replay, const VerdictArgs *verdict, const Done &done, cudaStream_t s) {
    bnk_ctx *ctx = b->ctx;
    DeviceBatch &d = b->dev;
    if (!replay) return launch_verdict(ctx, *verdict, done, s);
    if (n <= kTailMax) {
        VerdictArgs v{};
        if (verdict) v = *verdict;
        v.status = d.status;
        v.out_len = d.out_len;
        v.n = n;
        ctx->launches += 1;
        return launch_after_kernel(open_tail_kernel, dim3(1), dim3(512), s, replay_args(b, n), d.slot, v, done);
    }
    const SortPlan plan = plan_for(ctx->cfg.max_keypairs);
    GroupArgs g{};
    g.src = SortKeySrc{d.slot, ctx->cfg.max_keypairs};
    g.n = n;
    g.passes = plan.passes;
    g.digit_bits = plan.digit_bits;
    g.max_slots = ctx->cfg.max_keypairs;
    g.keys_out = d.keys_tmp + b->max_pkts;
    g.rp = replay_args(b, n);
    g.replay = true;
    if (verdict) g.verdict = *verdict;
    g.done = done;
    ctx->launches += 1;
    return launch_group(g, s);
}
cudaError_t launch_verdict(bnk_ctx *ctx, const VerdictArgs &v, const Done &done, cudaStream_t s) {
    ctx->launches += 1;
    return launch_after_kernel(verdict_kernel, dim3((v.n + 255) / 256), dim3(256), s, v, done);
}
// Expects launch_group_by_slot(b, n, ...) to have completed before this point of stream s.
cudaError_t launch_replay(bnk_batch *b, uint32_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    DeviceBatch &d = b->dev;
    const ReplayArgs a = replay_args(b, n);
    const uint32_t tiles = (n + kScanTile - 1) / kScanTile, grid = (n + 255) / 256;
    uint32_t *flag = d.replay_tile_head + replay_scan_tiles(b->max_pkts);
    launch_kernel(n <= dependent_launch_up_to(), replay_scan_tiles_kernel, dim3(tiles), dim3(256), s, a,
        d.replay_tile_head, d.replay_tile_max, flag);
    launch_kernel(n <= dependent_launch_up_to(), replay_scan_carry_kernel, dim3(1), dim3(1024), s, d.replay_tile_head,
        d.replay_tile_max, tiles, d.replay_tile_carry);
    launch_kernel(n <= dependent_launch_up_to(), replay_classify_kernel, dim3(tiles), dim3(256), s, a,
        d.replay_tile_carry, flag);
    launch_kernel(n <= dependent_launch_up_to(), replay_advance_kernel, dim3(grid), dim3(256), s, a);
    launch_kernel(n <= dependent_launch_up_to(), replay_hash_clear_kernel, dim3(b->ctx->sm_count * 4), dim3(256), s, a, flag);
    launch_kernel(n <= dependent_launch_up_to(), replay_hash_insert_kernel, dim3(grid), dim3(256), s, a, flag);
    launch_kernel(n <= dependent_launch_up_to(), replay_finish_kernel, dim3(grid), dim3(256), s, a);
    b->ctx->launches += 7;
    return cudaGetLastError();
}

cudaError_t launch_length_order(bnk_batch *b, uint32_t n, const uint32_t *len, bool open_side, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    DeviceBatch &d = b->dev;
    cudaError_t e = cudaMemsetAsync(d.counters32, 0, kLenBins * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    launch_kernel(n <= dependent_launch_up_to(), len_hist_kernel, dim3((n + kLenTile - 1) / kLenTile), dim3(256), s, len,
        n, open_side ? 1 : 0, d.counters32);
    launch_kernel(n <= dependent_launch_up_to(), exclusive_scan_kernel, dim3(1), dim3(1024), s, d.counters32, kLenBins);
    launch_kernel(n <= dependent_launch_up_to(), len_scatter_kernel, dim3((n + kLenTile - 1) / kLenTile), dim3(256), s,
        len, n, open_side ? 1 : 0, d.counters32, d.len_order);
    b->ctx->launches += 3;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------
// Send-counter hand-out for callers that must not allocate.
//
// The packet loop of a forwarder cannot afford cudaMalloc/cudaFree: both serialise the
// whole device, so one allocation stalls every other batch in flight, and a caller that
// keeps packets in device buffers of its own (for instance buffers a NIC writes into
// directly) has no bnk_batch whose creation would have set the grouping scratch aside.
// For those callers one group_kernel launch sorts in shared memory and writes nothing but their counters and the send
// counters.
// ---------------------------------------------------------------------------------------
namespace {

constexpr uint32_t kNoAllocMaxPkts = BNK_NOALLOC_MAX_PKTS;
static_assert(kNoAllocMaxPkts <= kGroupMax, "one launch");

int noalloc_fail(bnk_ctx *ctx, int code, const char *what, cudaError_t e = cudaSuccess) {
    std::lock_guard<std::mutex> g(ctx->mu);
    ctx->last_error = what;
    if (e != cudaSuccess) {
        ctx->last_error += ": ";
        ctx->last_error += cudaGetErrorString(e);
    }
    return code;
}

} // namespace

extern "C" int bnk_assign_counters_noalloc(bnk_ctx *ctx, void *stream, const uint32_t *dev_slot, uint32_t npkts,
                                           uint64_t *dev_counter) {
    if (!ctx) return BNK_EINVAL;
    if (!dev_slot || !dev_counter) return noalloc_fail(ctx, BNK_EINVAL, "bnk_assign_counters_noalloc: null buffer");
    if (npkts > kNoAllocMaxPkts)
        return noalloc_fail(ctx, BNK_EINVAL,
                            "bnk_assign_counters_noalloc: npkts exceeds BNK_NOALLOC_MAX_PKTS (16384); split the batch "
                            "or use bnk_seal_submit with BNK_F_ASSIGN_COUNTERS");
    if (npkts == 0) return BNK_SUCCESS;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return noalloc_fail(ctx, BNK_ECUDA, "cudaSetDevice", e);
    e = launch_counters(ctx, dev_slot, npkts, dev_counter, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return noalloc_fail(ctx, BNK_ECUDA, "kernel launch", e);
    return BNK_SUCCESS;
}
