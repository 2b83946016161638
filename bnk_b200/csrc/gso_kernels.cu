// Segmentation of TCP / UDP super-packets (IPv4) into MTU-sized packets, one warp per segment.
//
// Behaviour follows the split wireguard-go's Linux TUN code applies to a read that carries a virtio-net
// header (restated from its documented behaviour, golang.zx2c4.com/wireguard is not in the reference tree):
//   - every segment starts with the super-packet's IP header and transport header;
//   - IPv4: identification = first id + segment number, total length = header + segment payload,
//     header checksum recomputed;
//   - TCP: sequence number = first + segment number * gso_size, FIN and PSH survive on the last segment only;
//   - UDP: length = transport header + segment payload;
//   - transport checksum recomputed over pseudo header + transport header + payload.
// The work is a copy with a running one's-complement sum: HBM-bound, ~2 x segment bytes of traffic.
#include "bnk_internal.cuh"
#include "bulk.cuh"

namespace {

// one's-complement sum of big-endian 16-bit words, folded to 16 bits
__device__ __forceinline__ uint32_t fold16(uint64_t s) {
    s = (s & 0xffffffffull) + (s >> 32);
    s = (s & 0xffffffffull) + (s >> 32);
    uint32_t t = (uint32_t)s;
    t = (t & 0xffffu) + (t >> 16);
    t = (t & 0xffffu) + (t >> 16);
    return t;
}

struct SplitArgs {
    const bnk_gso_super *supers;
    uint32_t n_super;
    uint8_t *ring;
    const uint32_t *off, *len;
    uint32_t *slot;
    uint32_t n_pkts;
    uint64_t ring_bytes;
    const uint32_t *seg_super;
    const uint8_t *host_ring; // FROM_HOST
    Done done;
};
constexpr uint32_t kSplitWarps = 8;
constexpr uint32_t kSplitWindow = 2048; // FROM_HOST: a segment's payload, from the 16 bytes it starts in to those it ends in

// One segment, or packet that is none, by a warp.  FROM_HOST: the payload comes from the caller's pinned ring, in one bulk copy,
// and goes to the super-packet's place in the device ring besides (each word by the segment its first byte belongs to), which an
// upload would have filled; the headers are there already (gso_prepare_kernel).
template <bool FROM_HOST>
__device__ __forceinline__ void split_packet(const SplitArgs &a, uint32_t pkt, uint4 *stage, uint64_t *bar) {
    const bnk_gso_super *const supers = a.supers;
    const uint32_t n_super = a.n_super;
    uint8_t *const ring = a.ring;
    const uint32_t *const off = a.off, *const len = a.len;
    uint32_t *const slot = a.slot;
    const uint64_t ring_bytes = a.ring_bytes;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t j = a.seg_super[pkt];
    if (j >= n_super) { // not a segment of any super-packet: left alone
        if (!FROM_HOST) return;
        const uint32_t o = off[pkt], bytes = len[pkt];
        if ((o & 15u) || (uint64_t)o + 16 + bytes > ring_bytes) return;
        for (uint32_t q = 16u * lane; q < 16u + bytes; q += 512u)
            *reinterpret_cast<uint4 *>(ring + o + q) = *reinterpret_cast<const uint4 *>(a.host_ring + o + q);
        return;
    }
    const bnk_gso_super sp = supers[j];
    const uint32_t k = pkt - sp.first_pkt;
    const uint32_t hdr = sp.hdr_len, iph = sp.csum_start;
    const uint32_t data_at = hdr + k * sp.gso_size;
    bool ok = (sp.proto == 6 || sp.proto == 17) && iph >= 20 && hdr > iph && sp.gso_size > 0 && data_at < sp.src_len &&
              (sp.src_off & 3u) == 0 && (uint64_t)sp.src_off + sp.src_len <= ring_bytes &&
              sp.csum_offset + 2u <= hdr - iph && hdr - iph >= (sp.proto == 6 ? 20u : 8u) && ((hdr | iph) & 3u) == 0 &&
              (sp.csum_offset & 1u) == 0 && hdr <= 128u; // one header word per lane
    uint32_t seg_len = 0, total = 0;
    const uint32_t o = off[pkt];
    const uint64_t at = (uint64_t)sp.src_off + data_at; // of the payload, in the ring
    const uint8_t *payload = ring + at;
    bool came = true;
    if (FROM_HOST) { // (of such super-packets the host knows that they are whole and each segment fits the window)
        const uint64_t from = at & ~15ull, end = at + min((uint32_t)sp.gso_size, sp.src_len - data_at);
        const uint32_t bytes = (uint32_t)(((end + 15u) & ~15ull) - from);
        if (lane == 0) {
            bar_expect(bar, bytes);
            bulk_in(stage, a.host_ring + from, bytes, bar);
        }
        came = __all_sync(0xffffffffu, bar_wait(bar, 0));
        __syncwarp();
        payload = reinterpret_cast<const uint8_t *>(stage) + (at - from);
        const uint64_t word0 = (at + 3u) & ~3ull, whole = (uint64_t)sp.src_off + sp.src_len;
        for (uint64_t w = word0 + 4u * lane; came && w < end; w += 128u) {
            const uint8_t *const v = reinterpret_cast<const uint8_t *>(stage) + (w - from);
            if (w + 4u <= whole) *reinterpret_cast<uint32_t *>(ring + w) = *reinterpret_cast<const uint32_t *>(v);
            else
                for (uint64_t b = w; b < whole; b++) ring[b] = v[b - w];
        }
    }
    if (ok && came) {
        seg_len = min((uint32_t)sp.gso_size, sp.src_len - data_at);
        total = hdr + seg_len;
        ok = len[pkt] == total && (o & 15u) == 0 && (uint64_t)o + 16 + total + 32 <= ring_bytes && total <= 65535u;
    }
    if (!ok || !came) {
        if (lane == 0) slot[pkt] = 0xffffffffu; // the seal that follows reports BNK_PKT_BAD_DESC for it
        if (FROM_HOST && !came) bar_wait(bar, 0); // a copy that is still on its way must not meet the next kernel's shared memory
        return;
    }
    const uint8_t *in = ring + sp.src_off;
    uint8_t *out = ring + o + BNK_WG_HEADER;
    const bool last = data_at + seg_len == sp.src_len;

    // Headers: lane i takes header word i (IPv4 header and transport header are multiples of 4 bytes and together
    // at most 30 words), patches the field it holds and contributes its word to the IPv4 sum or to the transport
    // sum (source and destination address count for both: pseudo header).  The sums meet in the reductions below.
    const uint32_t ipw = iph >> 2, hw = hdr >> 2;
    uint64_t ip_sum = 0;  // IPv4 header, checksum field zero
    uint64_t hdr_sum = 0; // transport header + pseudo header, checksum field zero
    if (lane < hw) {
        uint32_t w = reinterpret_cast<const uint32_t *>(in)[lane];
        if (lane < ipw) {
            // words 0 (ver/ihl/tos/total length), 1 (id/flags/frag), 2 (ttl/proto/checksum), 3 src, 4 dst, options
            if (lane == 0) w = (w & 0x0000ffffu) | ((total >> 8) << 16) | ((total & 0xffu) << 24);
            else if (lane == 1) {
                const uint32_t id = (((w & 0xffu) << 8) | ((w >> 8) & 0xffu)) + k; // big-endian field in a little-endian word
                w = (w & 0xffff0000u) | ((id >> 8) & 0xffu) | ((id & 0xffu) << 8);
            } else if (lane == 2) w &= 0x0000ffffu; // checksum field cleared; lane 0 fills it in below
            ip_sum = (uint64_t)__byte_perm(w, 0, 0x4401) + (uint64_t)__byte_perm(w, 0, 0x4423);
            if (lane == 3 || lane == 4) hdr_sum = ip_sum;
        } else {
            const uint32_t t = lane - ipw;
            if (sp.proto == 6) {
                if (t == 1) {
                    const uint32_t seq = __byte_perm(w, 0, 0x0123) + k * sp.gso_size;
                    w = __byte_perm(seq, 0, 0x0123);
                } else if (t == 3 && !last) {
                    w &= ~(0x09u << 8); // flags are byte 13: FIN | PSH survive on the last segment only
                }
            } else if (t == 1) {
                const uint32_t ulen = hdr - iph + seg_len;
                w = (w & 0xffff0000u) | (ulen >> 8) | ((ulen & 0xffu) << 8);
            }
            if (t == (sp.csum_offset >> 2)) w &= (sp.csum_offset & 2u) ? 0x0000ffffu : 0xffff0000u; // checksum field cleared
            hdr_sum = (uint64_t)__byte_perm(w, 0, 0x4401) + (uint64_t)__byte_perm(w, 0, 0x4423);
        }
        reinterpret_cast<uint32_t *>(out)[lane] = w;
    }
    if (lane == 0) hdr_sum += sp.proto + (hdr - iph + seg_len);

    // payload copy + sum.  The destination starts on a word (headers are whole words); the source starts where the
    // segments before it end, at any byte of a word, so a word of the payload is cut out of two aligned words of the
    // source.
    const uint8_t *src = payload;
    uint8_t *dst = out + hdr;
    uint64_t sum = 0;    // of big-endian 16-bit words
    uint64_t le_sum = 0; // of the payload words as loaded (little-endian): the one's-complement sum commutes with the
                         // byte swap (RFC 1071, 2(B)), so the words are added raw and the folded sum is swapped once
    const uint32_t words = seg_len >> 2, shift = 8u * ((uint32_t)(uintptr_t)src & 3u);
    const uint32_t *s32 = reinterpret_cast<const uint32_t *>((uintptr_t)src & ~(uintptr_t)3u);
    uint32_t *d32 = reinterpret_cast<uint32_t *>(dst);
    auto word_at = [&](uint32_t i) { // behind a source that starts on a word there may be no further one
        const uint32_t lo = s32[i];
        return shift ? __funnelshift_r(lo, s32[i + 1], shift) : lo;
    };
    // several loads in flight per lane: the copy is latency-bound otherwise.  (Writing the destination in
    // aligned 16-byte chunks assembled from two aligned source lines was measured: 17 % slower.)
    constexpr uint32_t kInFlight = 4; // 2, 4 and 11 measure the same within noise
    uint32_t i = lane;
    for (; i + 32u * (kInFlight - 1) < words; i += 32u * kInFlight) {
        uint32_t w[kInFlight];
#pragma unroll
        for (uint32_t u = 0; u < kInFlight; u++) w[u] = word_at(i + 32u * u);
#pragma unroll
        for (uint32_t u = 0; u < kInFlight; u++) {
            d32[i + 32u * u] = w[u];
            le_sum += w[u];
        }
    }
    for (; i < words; i += 32) {
        const uint32_t w = word_at(i);
        d32[i] = w;
        le_sum += w;
    }
    for (uint32_t i = (words << 2) + lane; i < seg_len; i += 32) {
        const uint8_t v = src[i];
        dst[i] = v;
        sum += (i & 1u) ? v : ((uint32_t)v << 8);
    }
    le_sum = (le_sum & 0xffffffffull) + (le_sum >> 32); // 33 bits: 32 lanes of them still fit
    sum += hdr_sum; // both in 16-bit big-endian words
#pragma unroll
    for (int d = 16; d; d >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, d);
        le_sum += __shfl_xor_sync(0xffffffffu, le_sum, d);
        ip_sum += __shfl_xor_sync(0xffffffffu, ip_sum, d);
    }
    __syncwarp(); // the header words are in place before lane 0 writes the checksum bytes into them
    if (lane == 0) {
        const uint32_t ipc = ~fold16(ip_sum) & 0xffffu;
        out[10] = (uint8_t)(ipc >> 8);
        out[11] = (uint8_t)ipc;
        const uint32_t le = fold16(le_sum);
        const uint32_t c = ~fold16(sum + (((le & 0xffu) << 8) | (le >> 8))) & 0xffffu;
        out[iph + sp.csum_offset] = (uint8_t)(c >> 8);
        out[iph + sp.csum_offset + 1] = (uint8_t)c;
    }
}

template <bool FROM_HOST>
__global__ void __launch_bounds__(32 * kSplitWarps) gso_split_kernel(const __grid_constant__ SplitArgs a) {
    let_next_kernel_start();
    __shared__ __align__(128) uint4 stage[FROM_HOST ? kSplitWarps : 1][kSplitWindow / 16];
    __shared__ __align__(8) uint64_t bar[kSplitWarps];
    const uint32_t warp = threadIdx.x >> 5, pkt = blockIdx.x * kSplitWarps + warp;
    if (FROM_HOST) {
        if ((threadIdx.x & 31u) == 0) bar_init(&bar[warp]);
        bulk_fence_shared();
        __syncwarp();
    }
    wait_for_kernel_in_front();
    if (pkt < a.n_pkts) split_packet<FROM_HOST>(a, pkt, stage[FROM_HOST ? warp : 0], &bar[warp]);
    signal_done(a.done, false, [] {});
}

// In front of a split that reads the caller's pinned ring: what an upload would have brought of the descriptors, the super-packets'
// descriptors and headers, and the map from segment to super-packet.  (The super-packets come in batch order.)  A thread per
// packet, then a warp per super-packet.
struct PrepareArgs {
    const uint32_t *host_off, *host_len, *host_slot;
    uint32_t *off, *len, *slot, n_pkts;
    const bnk_gso_super *host_supers;
    bnk_gso_super *supers;
    uint32_t n_super;
    const uint8_t *host_ring;
    uint8_t *ring;
    uint32_t *seg_super;
};
__global__ void __launch_bounds__(256) gso_prepare_kernel(const __grid_constant__ PrepareArgs a) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    const uint32_t packet_ctas = (a.n_pkts + 255u) / 256u, lane = threadIdx.x & 31;
    if (blockIdx.x < packet_ctas) {
        const uint32_t i = blockIdx.x * 256u + threadIdx.x;
        if (i >= a.n_pkts) return;
        const uint32_t o = a.host_off[i], l = a.host_len[i], s = a.host_slot[i];
        a.off[i] = o;
        a.len[i] = l;
        a.slot[i] = s;
        return;
    }
    const uint32_t j = (blockIdx.x - packet_ctas) * 8u + (threadIdx.x >> 5);
    if (j >= a.n_super) return;
    constexpr uint32_t kWords = sizeof(bnk_gso_super) / 4;
    static_assert(sizeof(bnk_gso_super) == 4 * kWords && kWords <= 16, "two descriptors in the lanes of a warp");
    uint32_t w = 0; // lanes 0..: this one's words, lanes 16..: those of the one in front
    if (lane < kWords) w = reinterpret_cast<const uint32_t *>(a.host_supers + j)[lane];
    else if (j > 0 && lane >= 16u && lane < 16u + kWords) w = reinterpret_cast<const uint32_t *>(a.host_supers + j - 1)[lane - 16u];
    if (lane < kWords) reinterpret_cast<uint32_t *>(a.supers + j)[lane] = w;
    const uint32_t src = __shfl_sync(0xffffffffu, w, 0), first = __shfl_sync(0xffffffffu, w, 2), n = __shfl_sync(0xffffffffu, w, 3);
    const uint32_t hdr = __shfl_sync(0xffffffffu, w, 4) & 0xffffu; // words of the header, 32 at most
    const uint32_t before = __shfl_sync(0xffffffffu, w, 18) + __shfl_sync(0xffffffffu, w, 19); // where the one in front ends
    if (4u * lane < hdr) reinterpret_cast<uint32_t *>(a.ring + src)[lane] = reinterpret_cast<const uint32_t *>(a.host_ring + src)[lane];
    for (uint32_t k = before + lane; k < first + n; k += 32) a.seg_super[k] = k < first ? a.n_super : j;
    if (j + 1 == a.n_super)
        for (uint32_t k = first + n + lane; k < a.n_pkts; k += 32) a.seg_super[k] = a.n_super;
}

// segment -> super-packet index (n_super for packets that belong to none)
__global__ void gso_map_kernel(const bnk_gso_super *supers, uint32_t n_super, uint32_t n_pkts, uint32_t *seg_super) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_super) return;
    const bnk_gso_super sp = supers[j];
    for (uint32_t k = 0; k < sp.n_pkts; k++)
        if (sp.first_pkt + k < n_pkts) seg_super[sp.first_pkt + k] = j;
}

// What the device has made of the packets of a split, to the pinned ring, a warp per packet: the packet, or once a seal has
// run the message.  A packet that the split or the seal refused leaves no bytes.
__global__ void __launch_bounds__(256) packets_to_host_kernel(const uint8_t *ring, uint8_t *host_ring, const uint32_t *off,
                                                              const uint32_t *len, const uint32_t *slot, const uint8_t *status,
                                                              uint32_t n, uint64_t ring_bytes, uint32_t max_slots, uint32_t mtu, uint32_t sealed) {
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= n || slot[i] >= max_slots || (off[i] & 15u)) return;
    uint64_t at = off[i] + 16ull;
    uint32_t bytes = len[i];
    const uint8_t st = i < sealed ? status[i] : (uint8_t)BNK_PKT_BAD_DESC;
    if (st != BNK_PKT_BAD_DESC && st != BNK_PKT_NO_KEYPAIR && st != BNK_PKT_COUNTER_EXHAUSTED && st != BNK_PKT_MALFORMED &&
        st != BNK_PKT_NOT_READ) {
        at -= 16u;
        bytes = 16u + wg_padded_len(bytes, mtu) + 16u;
    }
    if (at + bytes > ring_bytes) return;
    for (uint32_t q = 16u * lane; q + 16u <= bytes; q += 512u)
        *reinterpret_cast<uint4 *>(host_ring + at + q) = *reinterpret_cast<const uint4 *>(ring + at + q);
    const uint32_t tail = (bytes & ~15u) + lane;
    if (tail < bytes) host_ring[at + tail] = ring[at + tail];
}

__global__ void fill_u32_kernel(uint32_t *p, uint32_t n, uint32_t v) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

} // namespace

cudaError_t launch_gso_split(bnk_batch *b, uint32_t n_super, uint32_t n_pkts, cudaStream_t s) {
    if (n_pkts == 0 || n_super == 0) return cudaSuccess;
    DeviceBatch &d = b->dev;
    uint32_t *seg_super = d.order_tmp; // grouping scratch is idle here
    launch_kernel(n_pkts <= dependent_launch_up_to(), fill_u32_kernel, dim3((n_pkts + 255) / 256), dim3(256), s,
        seg_super, n_pkts, n_super);
    launch_kernel(n_pkts <= dependent_launch_up_to(), gso_map_kernel, dim3((n_super + 127) / 128), dim3(128), s, d.gso,
        n_super, n_pkts, seg_super);
    b->ctx->launches += 2;
    return launch_gso_split_up(b, n_super, n_pkts, Done{}, s);
}

cudaError_t launch_gso_split_up(bnk_batch *b, uint32_t n_super, uint32_t n_pkts, const Done &done, cudaStream_t s) {
    DeviceBatch &d = b->dev;
    const SplitArgs a{d.gso, n_super, d.ring, d.off, d.len, d.slot, n_pkts, b->ring_bytes, d.order_tmp, nullptr, done};
    launch_kernel(n_pkts <= dependent_launch_up_to(), gso_split_kernel<false>, dim3((n_pkts + kSplitWarps - 1) / kSplitWarps),
        dim3(32 * kSplitWarps), s, a);
    b->ctx->launches += 1;
    return cudaGetLastError();
}

// Whether gso_split_kernel<true> can take them: in batch order, whole, and every segment in one window.
bool gso_split_fits(const bnk_gso_super *supers, uint32_t n_super, uint32_t n_pkts, uint64_t ring_bytes) {
    uint64_t next = 0;
    for (uint32_t j = 0; j < n_super; j++) {
        const bnk_gso_super &p = supers[j];
        const uint64_t segs = p.n_pkts, payload = (uint64_t)p.src_len - p.hdr_len;
        if (p.first_pkt < next || p.first_pkt + segs > n_pkts || segs == 0 || (p.src_off & 3u) || (uint64_t)p.src_off + p.src_len > ring_bytes ||
            (p.hdr_len & 3u) || p.hdr_len > 128u || p.hdr_len >= p.src_len || p.gso_size == 0 || p.gso_size + 32u > kSplitWindow ||
            segs != (payload + p.gso_size - 1) / p.gso_size)
            return false;
        next = p.first_pkt + segs;
    }
    return n_super != 0;
}
cudaError_t launch_gso_prepare(bnk_batch *b, uint32_t n_super, uint32_t n_pkts, cudaStream_t s) {
    DeviceBatch &d = b->dev;
    const bnk_batch_view &h = b->host;
    const PrepareArgs p{h.off, h.len, h.slot, d.off, d.len, d.slot, n_pkts, b->h_gso, d.gso, n_super, h.ring, d.ring, d.order_tmp};
    launch_kernel(false, gso_prepare_kernel, dim3((n_pkts + 255) / 256 + (n_super + 7) / 8), dim3(256), s, p);
    b->ctx->launches += 1;
    return cudaGetLastError();
}
cudaError_t launch_gso_split_in_place(bnk_batch *b, uint32_t n_super, uint32_t n_pkts, const Done &done, cudaStream_t s) {
    DeviceBatch &d = b->dev;
    const SplitArgs a{d.gso, n_super, d.ring, d.off, d.len, d.slot, n_pkts, b->ring_bytes, d.order_tmp, b->host.ring, done};
    launch_kernel(true, gso_split_kernel<true>, dim3((n_pkts + kSplitWarps - 1) / kSplitWarps), dim3(32 * kSplitWarps), s, a);
    b->ctx->launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_packets_to_host(bnk_batch *b, uint32_t n, cudaStream_t s) {
    const bnk_cfg &cfg = b->ctx->cfg;
    packets_to_host_kernel<<<(n + 7) / 8, 256, 0, s>>>(b->dev.ring, b->host.ring, b->dev.off, b->dev.len, b->dev.slot, b->dev.status, n,
                                                       b->ring_bytes, cfg.max_keypairs, cfg.mtu, b->split_sealed);
    b->ctx->launches += 1;
    return cudaGetLastError();
}
