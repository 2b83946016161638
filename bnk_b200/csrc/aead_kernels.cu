// Batched WireGuard transport-data seal / open for sm_100a.
//
// Work mapping: one thread owns one packet from the first ChaCha20 block to the
// Poly1305 tag, so every lane of a warp does useful 32-bit integer work on every
// instruction.  The path is bound by instruction issue on the integer pipes, not
// by HBM: ~19 integer operations per payload byte against ~2 bytes of traffic
// per payload byte, and the rotations of ChaCha20 issue at half rate on sm_100.
//
// Data movement is therefore kept to the fewest instructions: per 64-byte step a
// lane issues four 16-byte loads of its own packet ahead of the step's 80 quarter
// rounds (the rounds hide the latency; the two loads that share a 32-byte sector
// meet in L1) and four 16-byte stores after them (L2 merges the half sectors
// before they reach HBM).  No shared memory, no barriers, no cross-lane traffic:
// staging the 32 packets of a warp through shared memory so that global accesses
// are 512-byte wavefronts was measured and is 6 % slower, because its address
// arithmetic, shuffles and barriers cost issue slots that the rounds need.
//
// Arithmetic: ChaCha20 is RFC 8439 section 2.3 on 16 registers (rotations by 16
// and 8 are byte permutes, by 12 and 7 funnel shifts).  Poly1305 keeps h in five
// 32-bit limbs (radix 2^32) and multiplies with 32x32->64 multiply-adds on the
// FMA pipe.  The MAC input is ciphertext | zero pad to 16 | le64(0) | le64(ct_len),
// RFC 8439 section 2.8 with empty AAD; nonce = 32 zero bits | le64(counter) and the
// header is le32(4) | le32(receiver index) | le64(counter) (WireGuard whitepaper 5.4.6).
#include <algorithm>
#include <cstring>

#include "bulk.cuh"
#include "filter_device.cuh"
#include "layout.h"

namespace {

// Occupancy target for the register allocator: 4 CTAs of 128 threads per SM (up to 128 registers, no
// spills).  Measured within 2 % of each other: 3..6 CTAs of 128 threads, 3 CTAs of 256, 10 CTAs of 64.
#ifndef BNK_MIN_CTAS
#define BNK_MIN_CTAS 4
#endif
#ifndef BNK_WARPS_PER_CTA
#define BNK_WARPS_PER_CTA 4
#endif
constexpr int kWarpsPerCta = BNK_WARPS_PER_CTA;
constexpr int kThreads = kWarpsPerCta * 32;

// ---------------------------------------------------------------------------
// ChaCha20
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t rotl16(uint32_t x) { return __byte_perm(x, 0, 0x1032); }
__device__ __forceinline__ uint32_t rotl8(uint32_t x) { return __byte_perm(x, 0, 0x2103); }
__device__ __forceinline__ uint32_t rotl12(uint32_t x) { return __funnelshift_l(x, x, 12); }
__device__ __forceinline__ uint32_t rotl7(uint32_t x) { return __funnelshift_l(x, x, 7); }

// 12 instructions.  Exclusive-or, funnel shift and byte permute run on the ALU pipe only, at 64 lanes/clk/SM
// (two cycles per warp instruction per scheduler): 8 of them make a quarter round cost 16-17 cycles per warp,
// with the four additions riding along on the FMA pipe (the compiler already issues them there, so writing
// them as multiply-adds changes nothing).  The profiler agrees: issue slots 66 % busy, ALU pipe 75 %, top stall
// "math pipe throttle".  Moving a rotation to the multiplier (x * 2^n as a 64-bit product, low + high word) was
// measured too: each of the four rotations moved costs 9 % more time, the wide multiply being slower still.
#define BNK_QR(a, b, c, d) \
    a += b;                \
    d = rotl16(d ^ a);     \
    c += d;                \
    b = rotl12(b ^ c);     \
    a += b;                \
    d = rotl8(d ^ a);      \
    c += d;                \
    b = rotl7(b ^ c);

// One block: state = constants | key | block counter | 0 | counter lo | counter hi.
// (The first column round of columns 1, 2 and 3 reads constants, key and nonce only, so it is the same for every
// block of a packet.  Written out as a per-packet precomputation it compiles to the same register count as this
// form: the compiler already moves those 37 instructions out of the block loop.)
// UNROLL: double rounds per pass of the loop.  The throughput kernel wants all ten; a warp that computes one block and
// is done pays for fetching fifteen kilobytes of straight-line code instead (measured for one block of one warp: 1.7 us
// against 1.0 with one double round per pass).
template <int UNROLL = 10>
__device__ __forceinline__ void chacha20_block(uint32_t (&x)[16], const uint32_t (&k)[8], uint32_t blk,
                                               uint32_t n_lo, uint32_t n_hi) {
    x[0] = 0x61707865u;
    x[1] = 0x3320646eu;
    x[2] = 0x79622d32u;
    x[3] = 0x6b206574u;
#pragma unroll
    for (int i = 0; i < 8; i++) x[4 + i] = k[i];
    x[12] = blk;
    x[13] = 0u;
    x[14] = n_lo;
    x[15] = n_hi;
#pragma unroll UNROLL
    for (int r = 0; r < 10; r++) {
        BNK_QR(x[0], x[4], x[8], x[12])
        BNK_QR(x[1], x[5], x[9], x[13])
        BNK_QR(x[2], x[6], x[10], x[14])
        BNK_QR(x[3], x[7], x[11], x[15])
        BNK_QR(x[0], x[5], x[10], x[15])
        BNK_QR(x[1], x[6], x[11], x[12])
        BNK_QR(x[2], x[7], x[8], x[13])
        BNK_QR(x[3], x[4], x[9], x[14])
    }
    x[0] += 0x61707865u;
    x[1] += 0x3320646eu;
    x[2] += 0x79622d32u;
    x[3] += 0x6b206574u;
#pragma unroll
    for (int i = 0; i < 8; i++) x[4 + i] += k[i];
    x[12] += blk;
    x[14] += n_lo;
    x[15] += n_hi;
}

// ---------------------------------------------------------------------------
// Poly1305, radix 2^32.  r is clamped so r1..r3 are multiples of 4 and
// s_i = r_i + r_i/4 = 5*r_i/4 folds the 2^128-and-above partial products back
// (2^130 = 5 mod p).  h4 stays below 8 between blocks.
// ---------------------------------------------------------------------------
struct Poly {
    uint32_t h0, h1, h2, h3, h4;
    uint32_t r0, r1, r2, r3;
    uint32_t s1, s2, s3;
};

__device__ __forceinline__ void poly_init(Poly &p, uint32_t k0, uint32_t k1, uint32_t k2, uint32_t k3) {
    p.h0 = p.h1 = p.h2 = p.h3 = p.h4 = 0;
    p.r0 = k0 & 0x0fffffffu;
    p.r1 = k1 & 0x0ffffffcu;
    p.r2 = k2 & 0x0ffffffcu;
    p.r3 = k3 & 0x0ffffffcu;
    p.s1 = p.r1 + (p.r1 >> 2);
    p.s2 = p.r2 + (p.r2 >> 2);
    p.s3 = p.r3 + (p.r3 >> 2);
}

// h = (h + m + 2^128) * r, partially reduced.
__device__ __forceinline__ void poly_block(Poly &p, uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
    uint32_t h0 = p.h0, h1 = p.h1, h2 = p.h2, h3 = p.h3, h4 = p.h4;
    asm("add.cc.u32 %0, %0, %5;\n\t"
        "addc.cc.u32 %1, %1, %6;\n\t"
        "addc.cc.u32 %2, %2, %7;\n\t"
        "addc.cc.u32 %3, %3, %8;\n\t"
        "addc.u32 %4, %4, 1;"
        : "+r"(h0), "+r"(h1), "+r"(h2), "+r"(h3), "+r"(h4)
        : "r"(m0), "r"(m1), "r"(m2), "r"(m3));
    uint64_t d0 = (uint64_t)h0 * p.r0 + (uint64_t)h1 * p.s3 + (uint64_t)h2 * p.s2 + (uint64_t)h3 * p.s1;
    uint64_t d1 = (uint64_t)h0 * p.r1 + (uint64_t)h1 * p.r0 + (uint64_t)h2 * p.s3 + (uint64_t)h3 * p.s2 +
                  (uint64_t)h4 * p.s1;
    uint64_t d2 = (uint64_t)h0 * p.r2 + (uint64_t)h1 * p.r1 + (uint64_t)h2 * p.r0 + (uint64_t)h3 * p.s3 +
                  (uint64_t)h4 * p.s2;
    uint64_t d3 = (uint64_t)h0 * p.r3 + (uint64_t)h1 * p.r2 + (uint64_t)h2 * p.r1 + (uint64_t)h3 * p.r0 +
                  (uint64_t)h4 * p.s3;
    uint32_t top = h4 * p.r0;
    d1 += d0 >> 32;
    d2 += d1 >> 32;
    d3 += d2 >> 32;
    top += (uint32_t)(d3 >> 32);
    // everything at or above 2^130 comes back multiplied by 5
    uint32_t c = (top >> 2) + (top & ~3u);
    h0 = (uint32_t)d0;
    h1 = (uint32_t)d1;
    h2 = (uint32_t)d2;
    h3 = (uint32_t)d3;
    h4 = top & 3u;
    asm("add.cc.u32 %0, %0, %5;\n\t"
        "addc.cc.u32 %1, %1, 0;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.u32 %4, %4, 0;"
        : "+r"(h0), "+r"(h1), "+r"(h2), "+r"(h3), "+r"(h4)
        : "r"(c));
    p.h0 = h0;
    p.h1 = h1;
    p.h2 = h2;
    p.h3 = h3;
    p.h4 = h4;
}

// tag = ((h mod p) + pad) mod 2^128
__device__ __forceinline__ void poly_finish(const Poly &p, const uint32_t (&pad)[4], uint32_t (&tag)[4]) {
    uint32_t h0 = p.h0, h1 = p.h1, h2 = p.h2, h3 = p.h3, h4 = p.h4;
    uint32_t c = (h4 >> 2) * 5u;
    h4 &= 3u;
    asm("add.cc.u32 %0, %0, %5;\n\t"
        "addc.cc.u32 %1, %1, 0;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.u32 %4, %4, 0;"
        : "+r"(h0), "+r"(h1), "+r"(h2), "+r"(h3), "+r"(h4)
        : "r"(c));
    // g = h + 5; h >= p exactly when g reaches 2^130, and then h mod p = g - 2^130
    uint32_t g0, g1, g2, g3, g4;
    asm("add.cc.u32 %0, %5, 5;\n\t"
        "addc.cc.u32 %1, %6, 0;\n\t"
        "addc.cc.u32 %2, %7, 0;\n\t"
        "addc.cc.u32 %3, %8, 0;\n\t"
        "addc.u32 %4, %9, 0;"
        : "=r"(g0), "=r"(g1), "=r"(g2), "=r"(g3), "=r"(g4)
        : "r"(h0), "r"(h1), "r"(h2), "r"(h3), "r"(h4));
    if (g4 >> 2) {
        h0 = g0;
        h1 = g1;
        h2 = g2;
        h3 = g3;
    }
    asm("add.cc.u32 %0, %4, %8;\n\t"
        "addc.cc.u32 %1, %5, %9;\n\t"
        "addc.cc.u32 %2, %6, %10;\n\t"
        "addc.u32 %3, %7, %11;"
        : "=r"(tag[0]), "=r"(tag[1]), "=r"(tag[2]), "=r"(tag[3])
        : "r"(h0), "r"(h1), "r"(h2), "r"(h3), "r"(pad[0]), "r"(pad[1]), "r"(pad[2]), "r"(pad[3]));
}

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------
// keep the first k bytes (little-endian) of a word; k may be <= 0 or >= 4
__device__ __forceinline__ uint32_t keep_bytes(uint32_t w, int k) {
    if (k >= 4) return w;
    if (k <= 0) return 0u;
    return w & ((1u << (8 * k)) - 1u);
}

// ---------------------------------------------------------------------------
// Descriptor of one packet, validated; the outcome of a refused packet is recorded here.
// ---------------------------------------------------------------------------
struct Desc {
    uint32_t off, body /* bytes under the cipher */, in_len /* bytes to fetch */, n_lo, n_hi, slot;
    bool live;
};

template <bool OPEN>
__device__ __forceinline__ Desc load_desc(const AeadArgs &a, uint32_t pkt, bool have) {
    Desc d{0, 0, 0, 0, 0, 0, false};
    if (!have) return d;
    uint8_t st = BNK_PKT_OK;
    d.off = a.off[pkt];
    const uint32_t len = a.len[pkt];
    d.slot = a.slot[pkt];
    d.live = true;
    if ((d.off & 15u) || d.slot >= a.max_slots) {
        st = (OPEN && d.slot == kSlotNoKeypair) ? BNK_PKT_NO_KEYPAIR : BNK_PKT_BAD_DESC;
        d.live = false;
    } else if (!a.valid[d.slot]) {
        // never set, or cleared: the zeroed key of such a slot is public knowledge, so nothing is sealed
        // under it and nothing "authenticates" against it (wireguard-go drops traffic that has no keypair)
        st = BNK_PKT_NO_KEYPAIR;
        d.live = false;
    } else if (!OPEN) {
        d.body = wg_padded_len(len, a.mtu);
        d.in_len = len;
        const uint64_t ctr = a.counter[pkt];
        d.n_lo = (uint32_t)ctr;
        d.n_hi = (uint32_t)(ctr >> 32);
        if ((uint64_t)d.off + BNK_WG_HEADER + d.body + BNK_WG_TAG > a.ring_bytes || d.body < len) {
            st = BNK_PKT_BAD_DESC;
            d.live = false;
        } else if (ctr >= BNK_REJECT_AFTER_MESSAGES) {
            st = BNK_PKT_COUNTER_EXHAUSTED;
            d.live = false;
        }
    } else {
        if ((uint64_t)d.off + len > a.ring_bytes) {
            st = BNK_PKT_BAD_DESC;
            d.live = false;
        } else if (len < BNK_WG_HEADER + BNK_WG_TAG) {
            st = BNK_PKT_MALFORMED;
            d.live = false;
        } else {
            const uint4 hdr = *reinterpret_cast<const uint4 *>(a.out + d.off);
            d.n_lo = hdr.z;
            d.n_hi = hdr.w;
            a.res[0].counter[pkt] = ((uint64_t)hdr.w << 32) | hdr.z;
            if (hdr.x != 4u) {
                st = BNK_PKT_MALFORMED;
                d.live = false;
            } else {
                d.body = len - (BNK_WG_HEADER + BNK_WG_TAG);
                d.in_len = d.body;
            }
        }
    }
    if (!d.live) {
        a.res[0].status[pkt] = st;
        a.res[0].out_len[pkt] = 0;
        d.body = 0;
        d.in_len = 0;
    }
    return d;
}

// ---------------------------------------------------------------------------
// Kernel 1, thread per packet.  OPEN=false: seal in place.  OPEN=true: authenticate + decrypt in place.
// The throughput kernel: used when the batch is large enough to fill the GPU with one packet per thread.
// ---------------------------------------------------------------------------
template <bool OPEN>
__global__ void __launch_bounds__(kThreads, BNK_MIN_CTAS) aead_kernel(const __grid_constant__ AeadArgs a) {
    let_next_kernel_start();
    wait_for_kernel_in_front();
    const uint32_t idx = blockIdx.x * kThreads + threadIdx.x;
    const bool have = idx < a.n;
    const uint32_t pkt = have ? (a.order ? a.order[idx] : idx) : 0u;
    const Desc dsc = load_desc<OPEN>(a, pkt, have);
    const uint32_t off = dsc.off, body = dsc.body, in_len = dsc.in_len, n_lo = dsc.n_lo, n_hi = dsc.n_hi, slot = dsc.slot;
    const bool live = dsc.live;
    const uint32_t nblk = (body + 63u) >> 6;
    uint8_t *const data = a.out + (size_t)off + BNK_WG_HEADER; // 16-byte aligned

    uint32_t key[8];
    Poly poly;
    uint32_t pad[4] = {0, 0, 0, 0};
    if (live) {
        const uint4 *kp = reinterpret_cast<const uint4 *>(a.keys + (size_t)slot * 8);
        const uint4 ka = kp[0], kb = kp[1];
        key[0] = ka.x; key[1] = ka.y; key[2] = ka.z; key[3] = ka.w;
        key[4] = kb.x; key[5] = kb.y; key[6] = kb.z; key[7] = kb.w;
        uint32_t x[16];
        chacha20_block(x, key, 0u, n_lo, n_hi); // block 0 = one-time Poly1305 key
        poly_init(poly, x[0], x[1], x[2], x[3]);
        pad[0] = x[4]; pad[1] = x[5]; pad[2] = x[6]; pad[3] = x[7];
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) key[i] = 0;
        poly_init(poly, 0, 0, 0, 0);
    }

    // (Splitting off a branch-free loop over the whole blocks so that the Poly1305 multiplies can be scheduled
    // into the ChaCha20 rounds of the same thread, with the seal side absorbing the previous block's ciphertext,
    // was measured: no gain for seal, 10 % slower for open.  The warps of an SM already overlap the two phases.
    // Measured again on 1,048,576 x 1420 B with the comparisons peeled off the whole-block loop: seal 1.279 ms
    // against 1.276, open 1.383 against 1.261.  Feeding each Poly1305 column's carry into the next column's
    // first multiply-add instead of three 64-bit additions: seal 1.256, open 1.276: within the run-to-run spread.)
    for (uint32_t b = 0; b < nblk; b++) {
        const uint32_t base = b * 64u;
        uint32_t d[16];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            uint4 v = make_uint4(0, 0, 0, 0);
            // a chunk that starts inside the input is read whole: the bytes past in_len lie in the packet's own
            // padding / tag room and are masked below
            if (base + 16u * c < in_len) v = *reinterpret_cast<const uint4 *>(data + base + 16u * c);
            d[4 * c + 0] = v.x; d[4 * c + 1] = v.y; d[4 * c + 2] = v.z; d[4 * c + 3] = v.w;
        }
        uint32_t x[16];
        chacha20_block(x, key, b + 1u, n_lo, n_hi);
        if (base + 64u <= in_len) {
            // whole block of real bytes
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const uint32_t o0 = d[4 * c + 0] ^ x[4 * c + 0], o1 = d[4 * c + 1] ^ x[4 * c + 1];
                const uint32_t o2 = d[4 * c + 2] ^ x[4 * c + 2], o3 = d[4 * c + 3] ^ x[4 * c + 3];
                if (OPEN) poly_block(poly, d[4 * c + 0], d[4 * c + 1], d[4 * c + 2], d[4 * c + 3]);
                else poly_block(poly, o0, o1, o2, o3);
                *reinterpret_cast<uint4 *>(data + base + 16u * c) = make_uint4(o0, o1, o2, o3);
            }
        } else {
            // ragged end: bytes past in_len are zero padding (seal) and bytes past body do not exist
            const int in_left = (int)in_len - (int)base;
            const int body_left = (int)body - (int)base;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t o[4], m[4];
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    const int k = 16 * c + 4 * w;
                    const uint32_t in_w = keep_bytes(d[4 * c + w], in_left - k);
                    o[w] = keep_bytes(in_w ^ x[4 * c + w], body_left - k);
                    m[w] = OPEN ? in_w : o[w];
                }
                if (16 * c < body_left) poly_block(poly, m[0], m[1], m[2], m[3]);
                if (16 * c + 16 <= body_left) {
                    *reinterpret_cast<uint4 *>(data + base + 16u * c) = make_uint4(o[0], o[1], o[2], o[3]);
                } else if (16 * c < body_left) {
                    // last, partial chunk: byte stores
                    uint8_t *dst = data + base + 16u * c;
                    const int tail = body_left - 16 * c;
#pragma unroll
                    for (int k = 0; k < 15; k++)
                        if (k < tail) dst[k] = (uint8_t)(o[k >> 2] >> (8 * (k & 3)));
                }
            }
        }
    }

    if (!live) return;

    // ---- length block and tag ----
    // le64(aad_len = 0) | le64(body), with the 2^128 bit like every other block
    poly_block(poly, 0u, 0u, body, 0u);
    uint32_t tag[4];
    poly_finish(poly, pad, tag);
    uint8_t *tagp = data + body;

    if (!OPEN) {
        *reinterpret_cast<uint4 *>(a.out + off) = make_uint4(4u, a.remote_index[slot], n_lo, n_hi);
        if ((body & 3u) == 0) {
            uint32_t *t32 = reinterpret_cast<uint32_t *>(tagp);
            t32[0] = tag[0]; t32[1] = tag[1]; t32[2] = tag[2]; t32[3] = tag[3];
        } else {
#pragma unroll
            for (int w = 0; w < 4; w++)
#pragma unroll
                for (int k = 0; k < 4; k++) tagp[4 * w + k] = (uint8_t)(tag[w] >> (8 * k));
        }
        a.res[0].status[pkt] = BNK_PKT_OK;
        a.res[0].out_len[pkt] = BNK_WG_HEADER + body + BNK_WG_TAG;
    } else {
        uint32_t diff = 0;
        if ((body & 3u) == 0) {
            const uint32_t *t32 = reinterpret_cast<const uint32_t *>(tagp);
            diff = (t32[0] ^ tag[0]) | (t32[1] ^ tag[1]) | (t32[2] ^ tag[2]) | (t32[3] ^ tag[3]);
        } else {
#pragma unroll
            for (int w = 0; w < 4; w++)
#pragma unroll
                for (int k = 0; k < 4; k++) diff |= (uint32_t)(tagp[4 * w + k] ^ (uint8_t)(tag[w] >> (8 * k)));
        }
        if (diff == 0) {
            a.res[0].status[pkt] = body ? BNK_PKT_OK : BNK_PKT_KEEPALIVE;
            a.res[0].out_len[pkt] = body;
        } else {
            // forged or damaged: no plaintext may leave, wipe what the fused pass wrote
            uint8_t *dst = data;
            uint32_t k = 0;
            for (; k + 16u <= body; k += 16u) *reinterpret_cast<uint4 *>(dst + k) = make_uint4(0, 0, 0, 0);
            for (; k < body; k++) dst[k] = 0;
            a.res[0].status[pkt] = BNK_PKT_AUTH_FAIL;
            a.res[0].out_len[pkt] = 0;
        }
    }
}

// ---------------------------------------------------------------------------
// Poly1305 in radix 2^26 with both factors arbitrary: the warp-per-packet kernel multiplies by powers
// of r, which are not clamped, so the 5/4 trick of the radix-2^32 code above does not apply.
// Limbs of a product are below 2^26 (limb 1 may carry a few extra units); sums of two such values are
// valid left factors.
// ---------------------------------------------------------------------------
struct P26 {
    uint32_t v[5];
};
constexpr uint32_t kM26 = 0x3ffffffu;

__device__ __forceinline__ P26 p26_zero() { return P26{{0, 0, 0, 0, 0}}; }
__device__ __forceinline__ P26 p26_words(uint32_t t0, uint32_t t1, uint32_t t2, uint32_t t3, uint32_t hibit) {
    P26 m;
    m.v[0] = t0 & kM26;
    m.v[1] = ((t0 >> 26) | (t1 << 6)) & kM26;
    m.v[2] = ((t1 >> 20) | (t2 << 12)) & kM26;
    m.v[3] = ((t2 >> 14) | (t3 << 18)) & kM26;
    m.v[4] = (t3 >> 8) | (hibit << 24);
    return m;
}
__device__ __forceinline__ P26 p26_add(const P26 &x, const P26 &y) {
    P26 o;
#pragma unroll
    for (int i = 0; i < 5; i++) o.v[i] = x.v[i] + y.v[i];
    return o;
}
__device__ __forceinline__ P26 p26_mul(const P26 &x, const P26 &y) {
    const uint32_t s1 = y.v[1] * 5u, s2 = y.v[2] * 5u, s3 = y.v[3] * 5u, s4 = y.v[4] * 5u; // 2^130 = 5 (mod p)
    uint64_t d0 = (uint64_t)x.v[0] * y.v[0] + (uint64_t)x.v[1] * s4 + (uint64_t)x.v[2] * s3 + (uint64_t)x.v[3] * s2 +
                  (uint64_t)x.v[4] * s1;
    uint64_t d1 = (uint64_t)x.v[0] * y.v[1] + (uint64_t)x.v[1] * y.v[0] + (uint64_t)x.v[2] * s4 + (uint64_t)x.v[3] * s3 +
                  (uint64_t)x.v[4] * s2;
    uint64_t d2 = (uint64_t)x.v[0] * y.v[2] + (uint64_t)x.v[1] * y.v[1] + (uint64_t)x.v[2] * y.v[0] + (uint64_t)x.v[3] * s4 +
                  (uint64_t)x.v[4] * s3;
    uint64_t d3 = (uint64_t)x.v[0] * y.v[3] + (uint64_t)x.v[1] * y.v[2] + (uint64_t)x.v[2] * y.v[1] + (uint64_t)x.v[3] * y.v[0] +
                  (uint64_t)x.v[4] * s4;
    uint64_t d4 = (uint64_t)x.v[0] * y.v[4] + (uint64_t)x.v[1] * y.v[3] + (uint64_t)x.v[2] * y.v[2] + (uint64_t)x.v[3] * y.v[1] +
                  (uint64_t)x.v[4] * y.v[0];
    P26 o;
    d1 += d0 >> 26;
    d2 += d1 >> 26;
    d3 += d2 >> 26;
    d4 += d3 >> 26;
    const uint64_t t = (d0 & kM26) + (d4 >> 26) * 5u;
    o.v[0] = (uint32_t)t & kM26;
    o.v[1] = ((uint32_t)d1 & kM26) + (uint32_t)(t >> 26);
    o.v[2] = (uint32_t)d2 & kM26;
    o.v[3] = (uint32_t)d3 & kM26;
    o.v[4] = (uint32_t)d4 & kM26;
    return o;
}
// limbs of up to 32 bits -> limbs below 2^26 (limb 1 may keep a few extra units)
__device__ __forceinline__ P26 p26_carry(P26 h) {
    uint32_t c;
    c = h.v[0] >> 26; h.v[0] &= kM26; h.v[1] += c;
    c = h.v[1] >> 26; h.v[1] &= kM26; h.v[2] += c;
    c = h.v[2] >> 26; h.v[2] &= kM26; h.v[3] += c;
    c = h.v[3] >> 26; h.v[3] &= kM26; h.v[4] += c;
    c = h.v[4] >> 26; h.v[4] &= kM26; h.v[0] += c * 5u;
    c = h.v[0] >> 26; h.v[0] &= kM26; h.v[1] += c;
    return h;
}
// tag = ((h mod p) + pad) mod 2^128
__device__ __forceinline__ void p26_finish(const P26 &x, const uint32_t (&pad)[4], uint32_t (&tag)[4]) {
    uint32_t h0 = x.v[0], h1 = x.v[1], h2 = x.v[2], h3 = x.v[3], h4 = x.v[4], c;
    c = h1 >> 26; h1 &= kM26; h2 += c;
    c = h2 >> 26; h2 &= kM26; h3 += c;
    c = h3 >> 26; h3 &= kM26; h4 += c;
    c = h4 >> 26; h4 &= kM26; h0 += c * 5u;
    c = h0 >> 26; h0 &= kM26; h1 += c;
    // g = h + 5 - 2^130; g is non-negative exactly when h >= p
    uint32_t g0 = h0 + 5u; c = g0 >> 26; g0 &= kM26;
    uint32_t g1 = h1 + c;  c = g1 >> 26; g1 &= kM26;
    uint32_t g2 = h2 + c;  c = g2 >> 26; g2 &= kM26;
    uint32_t g3 = h3 + c;  c = g3 >> 26; g3 &= kM26;
    const uint32_t g4 = h4 + c - (1u << 26);
    if (!(g4 >> 31)) {
        h0 = g0; h1 = g1; h2 = g2; h3 = g3; h4 = g4;
    }
    const uint32_t w0 = h0 | (h1 << 26), w1 = (h1 >> 6) | (h2 << 20), w2 = (h2 >> 12) | (h3 << 14),
                   w3 = (h3 >> 18) | (h4 << 8);
    asm("add.cc.u32 %0, %4, %8;\n\t"
        "addc.cc.u32 %1, %5, %9;\n\t"
        "addc.cc.u32 %2, %6, %10;\n\t"
        "addc.u32 %3, %7, %11;"
        : "=r"(tag[0]), "=r"(tag[1]), "=r"(tag[2]), "=r"(tag[3])
        : "r"(w0), "r"(w1), "r"(w2), "r"(w3), "r"(pad[0]), "r"(pad[1]), "r"(pad[2]), "r"(pad[3]));
}

// ---------------------------------------------------------------------------
// Kernel 2, warp per packet: the kernel for batches too small to fill the GPU with one packet per thread, and for
// batches that stay in the caller's pinned memory (AeadArgs::in / out are then host addresses and the host link is
// the bound).
//
// A round covers up to 31 cipher blocks (1984 payload bytes; a full-size packet is one round).  One thread brings the
// round's bytes into shared memory with one bulk copy, and sends what leaves the round, put together in shared memory, with
// another: bytes behind the end of a message that share its last 16 are written back as they were read.  Over the link the
// copy engine of the SM asks for whole lines wherever a packet starts.  16-byte pieces asked for by the lanes do so only
// where the packets start on 32-byte sectors (plain copy through shared memory, 16,384 x 1440 B read and written: 1456 bytes
// apart 1030 us in pieces, 650 in bulk; 1536 bytes apart 645 either way; 4096 x 1440 B 1472 apart 186 and 165).
// Lane 0 computes cipher block 0 (the
// one-time Poly1305 key), lane j the round's block j, all in the same pass; on the seal side that needs no payload and
// is done while the payload is on its way.  For Poly1305 the round's 16-byte blocks are laid out from the right, four
// to a lane, the length block last in lane 31, so that every lane runs the same Horner steps from zero (the lane of the
// first block starts from the state carried in); lane j's sum is then multiplied by r^(4 (31 - j)), which again needs no
// payload, and the lanes' limbs are added up.
// A tag is checked before a one-round packet's plaintext is written.
//
// A warp takes tiles of a.tile consecutive packets (one in small batches); the descriptors of a tile lie in its
// lanes, and the next packet's bytes are on their way while one is computed.  Few warps are enough to keep the host
// link busy, and more of them in flight make it slower (read + write of 4096 x 1440 B in pieces: 172 us from 16 CTAs of 8
// warps, 184 from 148, 225 from 512), so the grid is capped for host-resident rings (wpp_grid).
//
// Loops are kept rolled: a warp of a small batch runs its code once, from a cold instruction cache.
// ---------------------------------------------------------------------------
constexpr uint32_t kWppWarps = 4; // one per scheduler: the warps of a small batch then share none
// Descriptors of a batch in host memory that go along with the launch, where they would be a trip over the link.  The
// driver and the GPU's front end handle a launch's parameters word by word, so there are several sizes (launch_wpp).
template <uint32_t N> // packets there is room for
struct InlineDesc {
    uint32_t off[N], len[N], slot[N];
};
template <>
struct InlineDesc<0> {};
constexpr uint32_t kRoundBlocks = 31;
constexpr uint32_t kRoundBytes = kRoundBlocks * 64;
constexpr uint32_t kStagePieces = 128; // header, 124 of the body, 2 that the tag may touch, rounded up to a line (no swizzle: a
                                       // bulk copy fills it, and the four-way bank conflicts of the lanes' loads are 0.1 us of 5)

__device__ __forceinline__ void copy_async16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// Round `rnd` of a packet: its first byte in the ring (the header's in round 0), and which 16-byte piece of the stage its
// first body byte is.
struct Round {
    uint64_t at;
    uint32_t body;
    __device__ __forceinline__ Round(uint32_t off, uint32_t rnd) {
        at = rnd == 0 ? (uint64_t)off : (uint64_t)off + BNK_WG_HEADER + (uint64_t)rnd * kRoundBytes;
        body = rnd == 0 ? 1u : 0u;
    }
};

// Word `lane` (0..15) of the 64 bytes that start at a piece.
__device__ __forceinline__ uint32_t stage_word(const uint4 *stage, uint32_t piece) {
    const uint32_t lane = threadIdx.x & 31;
    return reinterpret_cast<const uint32_t *>(&stage[piece])[lane & 15u];
}

// r^(4 e) for the lane's e = 31 - lane, one bit of e per step: pw goes through r^4, r^8, r^16 ...
struct LanePower {
    P26 p, pw;
    uint32_t bits; // of e still to come
    __device__ __forceinline__ void begin(const P26 &r) {
        p = p26_zero();
        p.v[0] = 1u;
        pw = p26_mul(r, r);
        pw = p26_mul(pw, pw);
        bits = 31u - (threadIdx.x & 31u);
    }
    __device__ __forceinline__ void step() {
        const P26 t = p26_mul(p, pw);
        if (bits & 1u) p = t;
        bits >>= 1;
        pw = p26_mul(pw, pw);
    }
};

// Poly1305's r and pad out of cipher block 0, which lane 0 holds.
__device__ __forceinline__ P26 one_time_key(const uint32_t (&x)[16], uint32_t (&pad)[4]) {
    const uint32_t k0 = __shfl_sync(0xffffffffu, x[0], 0), k1 = __shfl_sync(0xffffffffu, x[1], 0);
    const uint32_t k2 = __shfl_sync(0xffffffffu, x[2], 0), k3 = __shfl_sync(0xffffffffu, x[3], 0);
#pragma unroll
    for (int i = 0; i < 4; i++) pad[i] = __shfl_sync(0xffffffffu, x[4 + i], 0);
    return p26_words(k0 & 0x0fffffffu, k1 & 0x0ffffffcu, k2 & 0x0ffffffcu, k3 & 0x0ffffffcu, 0u);
}
// What a lane does with its part of one round: `data` is the stage at the round's body of rb bytes, x the lane's keystream,
// `steps` what is left of the powers, beside() runs between the cipher and Poly1305.  The body's ciphertext or plaintext and, on
// the seal side, the tag are in the stage afterwards.  True: the tag is wrong, and the body is zeros.
template <bool OPEN, typename F>
__device__ __forceinline__ bool cipher_and_mac(uint4 *const data, uint32_t rb, uint32_t body, bool last, uint32_t (&x)[16], const P26 &r,
                                               P26 &state, LanePower &power, uint32_t steps, const uint32_t (&pad)[4], bool broken, F beside) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t data_blocks = (rb + 15u) >> 4, blocks = data_blocks + (last ? 1u : 0u);
    const bool works = lane != 0 && (lane - 1u) * 64u < rb;
    const int body_left = (int)rb - (int)(lane - 1u) * 64;
    uint8_t *const end_byte = reinterpret_cast<uint8_t *>(data) + rb + lane; // byte `lane` behind the round's body
    const bool in_last_piece = lane < ((0u - rb) & 15u);                    // it shares the body's last piece
    uint8_t tag_byte = 0;
    bool forged = false;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        if (!works || 16 * c >= body_left) continue;
        uint4 *const p = &data[4u * (lane - 1u) + c];
        const uint4 v = *p;
        x[4 * c + 0] ^= v.x;
        x[4 * c + 1] ^= v.y;
        x[4 * c + 2] ^= v.z;
        x[4 * c + 3] ^= v.w;
        if (!OPEN) *p = make_uint4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
    }
    if (!OPEN) { // Poly1305 pads its last block with zeros
        __syncwarp();
        if (in_last_piece) *end_byte = 0;
    }
    beside();
    __syncwarp();
    // ---- Poly1305 over the ciphertext in the stage ----
    P26 V = p26_zero();
    const int b0 = (int)(4u * lane + blocks) - 128; // the lane's first block; negative: none
    if (b0 <= 0 && b0 > -4) V = state;              // (zero in round 0)
#pragma unroll 1
    for (int s = 0; s < 4; s++) {
        const int blk = b0 + s;
        uint4 m = make_uint4(0u, 0u, body, 0u); // le64(0) | le64(body)
        if (blk >= 0 && (uint32_t)blk < data_blocks) {
            m = data[blk];
            const int left = (int)rb - 16 * blk;
            if (OPEN && left < 16) {
                m.x = keep_bytes(m.x, left);
                m.y = keep_bytes(m.y, left - 4);
                m.z = keep_bytes(m.z, left - 8);
                m.w = keep_bytes(m.w, left - 12);
            }
        }
        const P26 next_v = p26_mul(p26_add(V, p26_words(m.x, m.y, m.z, m.w, 1u)), r);
        if (blk >= 0) V = next_v;
        if (OPEN && steps) { // beside the Horner step: neither waits for the other
            power.step();
            steps--;
        }
    }
    if (OPEN && steps) power.step();
    V = p26_mul(V, power.p);
#pragma unroll
    for (int d = 16; d; d >>= 1) { // limbs below 2^27: the sum of 32 of them fits a word
#pragma unroll
        for (int i = 0; i < 5; i++) V.v[i] += __shfl_xor_sync(0xffffffffu, V.v[i], d);
    }
    state = p26_carry(V);
    // ---- tag, output ----
    if (last) {
        uint32_t tag[4];
        p26_finish(state, pad, tag);
        const uint32_t tw = (lane & 8u) ? ((lane & 4u) ? tag[3] : tag[2]) : ((lane & 4u) ? tag[1] : tag[0]);
        const uint8_t tb = (uint8_t)(tw >> (8u * (lane & 3u)));
        if (OPEN) {
            tag_byte = *end_byte;
            forged = __any_sync(0xffffffffu, lane < 16u && tag_byte != tb) || broken;
        } else if (lane < 16u) {
            *end_byte = tb;
        }
    }
    if (OPEN) {
        __syncwarp(); // ciphertext and tag are read
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (works && 16 * c < body_left)
                data[4u * (lane - 1u) + c] =
                    forged ? make_uint4(0, 0, 0, 0) : make_uint4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
        __syncwarp();
        if (last && in_last_piece) *end_byte = tag_byte; // what is not plaintext goes back as it came
    }
    return forged;
}
// The flow of a packet whose payload starts at stage[piece] (the IPv4 header and the ports lie in 64 bytes).
__device__ __forceinline__ void note_head(FlowNote &note, const AeadArgs &a, const uint4 *stage, uint32_t piece, uint32_t len) {
    const uint32_t word = stage_word(stage, piece);
    Parsed p;
    const uint32_t at = parse_ipv4_words(__shfl_sync(0xffffffffu, word, 0), __shfl_sync(0xffffffffu, word, 2),
                                         __shfl_sync(0xffffffffu, word, 3), __shfl_sync(0xffffffffu, word, 4), len, p);
    const uint32_t ports = __shfl_sync(0xffffffffu, word, (at >> 2) & 15u);
    if (at != kParseBad && (threadIdx.x & 31) == 0) {
        if (at) parse_ports(ports, p);
        note.begin(a.ft, p, a.now);
    }
}
// What the last checks want of the plaintext of `body` bytes that starts at stage[piece].
__device__ __forceinline__ uint4 inner_head(const AeadArgs &a, const uint4 *stage, uint32_t piece, uint32_t body) {
    const uint32_t word = stage_word(stage, piece);
    const uint32_t w0 = __shfl_sync(0xffffffffu, word, 0), w3 = __shfl_sync(0xffffffffu, word, 3);
    const uint32_t total = ((w0 >> 8) & 0xff00u) | (w0 >> 24); // bytes 2,3 big-endian
    const bool is_whole = body >= 20 && ((w0 & 0xffu) >> 4) == 4u && total >= 20 && total <= body;
    Parsed p{};
    const uint32_t at = parse_ipv4_words(w0, __shfl_sync(0xffffffffu, word, 2), w3, __shfl_sync(0xffffffffu, word, 4),
                                         a.inner_cut && is_whole ? total : body, p);
    const uint32_t ports = __shfl_sync(0xffffffffu, word, (at >> 2) & 15u);
    if (at != kParseBad && at) parse_ports(ports, p);
    return make_uint4(__byte_perm(w3, 0, 0x0123), (uint32_t)p.sport << 16 | p.dport,
                      p.proto | (at != kParseBad ? kInnerParses : 0u) | (is_whole ? kInnerWhole : 0u), total);
}

// Seal batches of up to kRankMax packets in pinned memory hand out their nonces here (a.send_counter): a warp counts the
// packets of its slot in front of its own, and the last packet of a slot moves the counter past them all (SendCounter
// says why nobody has to wait for that).  A grouping launch in front took 5 us.
// NOTE: the flows of the packets are recorded from the bytes in the stage, each step of the table's atomics behind a
// piece of the cipher work.
template <bool OPEN, bool NOTE, uint32_t INLINE>
__global__ void __launch_bounds__(32 * kWppWarps, 4) aead_wpp_kernel(const __grid_constant__ AeadArgs a,
                                                                      const __grid_constant__ InlineDesc<INLINE> desc) {
    static_assert(!(OPEN && NOTE), "flows are recorded on the seal side");
    let_next_kernel_start(); // open side: the grouping + replay launch behind may take its place already
    // What a ring in device memory holds may come from the kernel in front; a pinned ring and its descriptors are the
    // host's, and only the counters of a seal come from there.
    if (!a.from_host) wait_for_kernel_in_front();
    __shared__ __align__(128) uint4 stage_all[kWppWarps][2][kStagePieces];
    __shared__ __align__(16) uint4 key_all[kWppWarps][2][2];
    __shared__ __align__(8) uint64_t bar_all[kWppWarps][2];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t T = INLINE ? 1u : a.tile, tiles = (a.n + T - 1) / T, step = gridDim.x * kWppWarps;
    uint32_t parity = 0;  // bit b: of the phase that stage b's next wait is for
    uint32_t awaited = 0; // bit b: copies into stage b are on their way
    bool broken = false;  // what was asked for has not come: nothing is read or written any more
    if (lane < 2) bar_init(&bar_all[warp][lane]);
    bulk_fence_shared();
    __syncwarp();

    struct Tile { // one packet's descriptor in each of the first T lanes
        uint32_t off, len, slot, valid, remote;
        uint64_t ctr;
    };
    auto load_tile = [&](uint32_t t) {
        Tile d{0, 0, 0, 0, 0, 0};
        const uint32_t i = t * T + lane;
        if (t < tiles && lane < T && i < a.n) {
            if constexpr (INLINE != 0) {
                d.off = desc.off[i];
                d.len = desc.len[i];
                d.slot = desc.slot[i];
            } else {
                d.off = a.off[i];
                d.len = a.len[i];
                if (!OPEN || !a.demux) d.slot = a.slot[i];
            }
        }
        return d;
    };
    auto load_keypair = [&](Tile &d, uint32_t t) { // what hangs on the slot: asked for once the slot is there
        const uint32_t i = t * T + lane;
        if (!OPEN && a.send_counter == nullptr && t < tiles && lane < T && i < a.n) d.ctr = a.counter[i];
        if (!(OPEN && a.demux) && d.slot < a.max_slots) {
            d.valid = a.valid[d.slot];
            if (!OPEN) d.remote = a.remote_index[d.slot];
        }
    };
    // Starts the copies of a packet's keys (when the slot is known) and of its first round into stage `buf`, which has been read
    // out.  The round is one copy: it reaches the link as whole lines wherever the packet starts, and takes one instruction.
    // header_first: a message's header comes with the keys besides.  Nonce and receiver index are all that the keystream and
    // Poly1305's powers need, and they are computed while the rest is on its way, as on the seal side: 128 x 1420 B opened by
    // receiver index 24.5 us -> 22.8, 9 x 300 B with everything on 21.1 -> 19.9.  (With the rest in pieces
    // asked for by the lanes this gains nothing where the slot has to be looked up: loads come back in the order they were
    // issued, those of the index table behind the packet's.)  It is a request more for each packet, which many threads feel:
    // see open_direct.
    const bool header_first = OPEN && INLINE != 0 && a.header_first;
    __shared__ uint4 header_all[OPEN && INLINE != 0 ? kWppWarps : 1];
    auto fetch = [&](uint32_t off, uint32_t len, uint32_t slot, uint32_t buf) {
        if ((!OPEN || !a.demux) && slot < a.max_slots && lane < 2)
            copy_async16(&key_all[warp][buf][lane], a.keys + (size_t)slot * 8 + 4u * lane);
        if (header_first && lane == 0 && !(off & 15u) && len >= BNK_WG_HEADER + BNK_WG_TAG && (uint64_t)off + len <= a.ring_bytes)
            copy_async16(&header_all[warp], a.in + off);
        copy_async_commit();
        if (broken) return;
        awaited |= 1u << buf;
        if (lane != 0) return;
        const Round r(off, 0);
        uint32_t from = 0, end = 0; // pieces
        if (!(off & 15u)) {
            if (OPEN) {
                const uint32_t body = len - (BNK_WG_HEADER + BNK_WG_TAG);
                if (len >= BNK_WG_HEADER + BNK_WG_TAG && (uint64_t)off + len <= a.ring_bytes)
                    end = r.body + (((body <= kRoundBytes ? body + BNK_WG_TAG : kRoundBytes) + 15u) >> 4);
            } else if ((uint64_t)off + BNK_WG_HEADER + len <= a.ring_bytes) {
                from = r.body;
                end = r.body + ((min(len, kRoundBytes) + 15u) >> 4);
                const uint32_t body = wg_padded_len(len, a.mtu); // a message that ends inside a piece: as far as that
                if (body <= kRoundBytes && (body & 15u) && (uint64_t)off + BNK_WG_HEADER + body + BNK_WG_TAG <= a.ring_bytes)
                    end = r.body + ((body + BNK_WG_TAG + 15u) >> 4);
            }
        }
        bar_expect(&bar_all[warp][buf], 16u * (end - from));
        if (end > from) bulk_in(&stage_all[warp][buf][from], a.in + r.at + 16u * from, 16u * (end - from), &bar_all[warp][buf]);
    };
    auto arrived = [&](uint32_t buf) { // the packet is in the stage
        if (!broken) broken = !bar_wait(&bar_all[warp][buf], (parity >> buf) & 1u);
        broken = __any_sync(0xffffffffu, broken);
        if (broken) return;
        parity ^= 1u << buf;
        awaited &= ~(1u << buf);
        __syncwarp();
    };

    uint32_t t = blockIdx.x * kWppWarps + warp, buf = 0;
    Tile cur = load_tile(t);
    // Loads come back in the order they were issued, also those from the device's own memory behind those over the link:
    // what hangs on the slot is asked for before the payload, unless the kernel in front has still to write it.
    __shared__ uint32_t slots[INLINE ? INLINE : 1];
    CounterRead counter{};
    const bool hands_out = INLINE && !OPEN && a.send_counter;
    if (OPEN || !a.behind_kernel || !a.from_host) load_keypair(cur, t);
    if (hands_out && t < tiles && lane == 0 && cur.slot < a.max_slots) counter = counter_read(&a.send_counter[cur.slot], a.seal_seq);
    if (t < tiles) fetch(__shfl_sync(0xffffffffu, cur.off, 0), __shfl_sync(0xffffffffu, cur.len, 0),
                         __shfl_sync(0xffffffffu, cur.slot, 0), 0);
    if (a.from_host) wait_for_kernel_in_front();
    if (!OPEN && a.behind_kernel && a.from_host) load_keypair(cur, t);
    if constexpr (INLINE && !OPEN) {
        if (hands_out) { // one tile of one packet per warp
            for (uint32_t i = threadIdx.x; i < a.n; i += blockDim.x) slots[i] = desc.slot[i];
            __syncthreads();
            if (t < tiles) {
                const uint32_t mine = slots[t];
                uint32_t before = 0, all = 0;
#pragma unroll 1
                for (uint32_t base = 0; base < a.n; base += 32) {
                    const uint32_t same = __ballot_sync(0xffffffffu, base + lane < a.n && slots[base + lane] == mine);
                    all += __popc(same);
                    before += __popc(base + 32 <= t ? same : base > t ? 0u : same & ((1u << (t - base)) - 1u));
                }
                cur.ctr = saturating_counter(counter.now.value, before);
                if (before + 1 == all && lane == 0 && mine < a.max_slots) // the last packet of its slot moves the counter on
                    counter_store(&a.send_counter[mine].e[counter.at ^ 1u],
                                  SendCounter::Entry{saturating_counter(counter.now.value, all), a.seal_seq});
            }
        }
    }
    __shared__ uint32_t cta_len[kWppWarps];
    __shared__ uint64_t cta_ctr[kWppWarps];
    __shared__ uint8_t cta_status[kWppWarps], cta_has[kWppWarps];
    const bool by_cta = T == 1 && tiles <= step; // one packet per warp: the CTA's results leave together
    for (; t < tiles; t += step) {
        const uint32_t in_tile = min(T, a.n - t * T);
        Tile next = load_tile(t + step);
        uint32_t res_len = 0, res_slot = 0, res_status = BNK_PKT_OK; // of the packet of this lane
        bool has_counter = !OPEN && cur.slot < a.max_slots;
        uint64_t res_ctr = cur.ctr;
#pragma unroll 1
        for (uint32_t k = 0; k < in_tile; k++, buf ^= 1u) {
            const uint32_t off = __shfl_sync(0xffffffffu, cur.off, k), len = __shfl_sync(0xffffffffu, cur.len, k);
            uint32_t slot = __shfl_sync(0xffffffffu, cur.slot, k);
            bool ahead = true; // another packet's copies are on their way behind this one's
            if (lane == 0) bulk_out_read(); // of the other stage, which the packet before has left
            __syncwarp();
            if (k + 1 < in_tile) {
                fetch(__shfl_sync(0xffffffffu, cur.off, k + 1), __shfl_sync(0xffffffffu, cur.len, k + 1),
                      __shfl_sync(0xffffffffu, cur.slot, k + 1), buf ^ 1u);
            } else if (t + step < tiles) {
                load_keypair(next, t + step);
                fetch(__shfl_sync(0xffffffffu, next.off, 0), __shfl_sync(0xffffffffu, next.len, 0),
                      __shfl_sync(0xffffffffu, next.slot, 0), buf ^ 1u);
            } else {
                ahead = false;
            }
            uint4 *const stage = stage_all[warp][buf];
            uint8_t *const stage_bytes = reinterpret_cast<uint8_t *>(stage);
            Round rd(off, 0);

            // ---- what the descriptor says (the same for all lanes) ----
            uint8_t st = BNK_PKT_OK;
            uint32_t body = 0, in_len = 0, n_lo = 0, n_hi = 0;
            uint4 ka = make_uint4(0, 0, 0, 0), kb = ka; // the keys, and whether there are any, of a slot that is looked up
            uint8_t valid = 0;
            if (OPEN) {
                if (ahead) copy_async_wait<1>();
                else copy_async_wait<0>();
                __syncwarp();
                if (!header_first) arrived(buf);
                const bool in_ring = (uint64_t)off + len <= a.ring_bytes, whole = in_ring && len >= BNK_WG_HEADER + BNK_WG_TAG;
                uint4 hdr = make_uint4(0, 0, 0, 0);
                if (!(off & 15u) && whole) hdr = header_first ? header_all[warp] : stage[0];
                if (a.demux) {
                    slot = 0; // descriptors refused below for other reasons
                    if (!(off & 15u) && whole) slot = demux_index_warp(a.index_keys, a.index_vals, a.index_slots, hdr.y);
                    if (slot < a.max_slots) { // asked for together
                        const uint4 *const kp = reinterpret_cast<const uint4 *>(a.keys + (size_t)slot * 8);
                        valid = a.valid[slot];
                        ka = kp[0];
                        kb = kp[1];
                    }
                }
                if (broken) st = BNK_PKT_NOT_READ;
                else if ((off & 15u) || slot >= a.max_slots) st = slot == kSlotNoKeypair ? BNK_PKT_NO_KEYPAIR : BNK_PKT_BAD_DESC;
                else if (!(a.demux ? valid : __shfl_sync(0xffffffffu, cur.valid, k))) st = BNK_PKT_NO_KEYPAIR;
                else if (!in_ring) st = BNK_PKT_BAD_DESC;
                else if (!whole) st = BNK_PKT_MALFORMED;
                else {
                    n_lo = hdr.z;
                    n_hi = hdr.w;
                    if (lane == k) {
                        res_ctr = ((uint64_t)hdr.w << 32) | hdr.z;
                        has_counter = true;
                    }
                    if (hdr.x != 4u) st = BNK_PKT_MALFORMED;
                    body = in_len = len - (BNK_WG_HEADER + BNK_WG_TAG);
                }
            } else {
                const uint64_t ctr = __shfl_sync(0xffffffffu, cur.ctr, k);
                n_lo = (uint32_t)ctr;
                n_hi = (uint32_t)(ctr >> 32);
                body = wg_padded_len(len, a.mtu);
                in_len = len;
                if ((off & 15u) || slot >= a.max_slots) st = BNK_PKT_BAD_DESC;
                else if (!__shfl_sync(0xffffffffu, cur.valid, k)) st = BNK_PKT_NO_KEYPAIR;
                else if ((uint64_t)off + BNK_WG_HEADER + body + BNK_WG_TAG > a.ring_bytes || body < len) st = BNK_PKT_BAD_DESC;
                else if (ctr >= BNK_REJECT_AFTER_MESSAGES) st = BNK_PKT_COUNTER_EXHAUSTED;
            }
            if (lane == k) {
                res_slot = slot;
                res_status = st;
                res_len = 0;
            }
            FlowNote note;
            auto note_begin = [&] {
                if (!NOTE || broken || (off & 15u) || (uint64_t)off + BNK_WG_HEADER + len > a.ring_bytes) return;
                note_head(note, a, stage, rd.body, len);
            };
            if (st != BNK_PKT_OK) { // the next packet's copies are in the other stage
                if (header_first) arrived(buf);
                if (!OPEN) {
                    arrived(buf);
                    note_begin();
                    note.place(a.ft);
                    note.count(a.ft);
                }
                __syncwarp();
                continue;
            }

            uint32_t key[8];
            {
                if (!OPEN || !a.demux) {
                    if (!OPEN) {
                        if (ahead) copy_async_wait<1>();
                        else copy_async_wait<0>();
                        __syncwarp();
                    }
                    ka = key_all[warp][buf][0];
                    kb = key_all[warp][buf][1];
                }
                key[0] = ka.x; key[1] = ka.y; key[2] = ka.z; key[3] = ka.w;
                key[4] = kb.x; key[5] = kb.y; key[6] = kb.z; key[7] = kb.w;
            }
            const uint32_t remote = OPEN ? 0u : __shfl_sync(0xffffffffu, cur.remote, k);
            P26 r = p26_zero(), state = p26_zero();
            LanePower power;
            uint32_t pad[4] = {0, 0, 0, 0};
            bool forged = false;
#pragma unroll 1
            for (uint32_t rnd = 0;; rnd++) {
                const uint32_t done = rnd * kRoundBytes;
                const uint32_t rb = min(body - done, kRoundBytes); // body bytes of this round
                const bool last = body - done <= kRoundBytes;
                const uint32_t blocks = ((rb + 15u) >> 4) + (last ? 1u : 0u);
                // ---- keystream: lane 0 block 0, lane j the j-th block of the round ----
                uint32_t x[16];
                chacha20_block<1>(x, key, lane == 0 ? 0u : rnd * kRoundBlocks + lane, n_lo, n_hi);
                uint32_t steps = 0; // of the lanes' powers: as many as there are bits in the number of lanes that hold blocks
                if (rnd == 0) {
                    r = one_time_key(x, pad);
                    power.begin(r);
                    steps = last ? 32u - __clz((blocks + 3u) / 4u - 1u) : 5u;
                    if (!OPEN || header_first) {
#pragma unroll 1
                        for (; steps; steps--) power.step();
                        arrived(buf);
                        note_begin();
                    }
                } else { // longer packets: the further rounds are fetched when their turn comes
                    rd = Round(off, rnd);
                    const uint32_t bytes = OPEN ? rb + (last ? BNK_WG_TAG : 0u) : (in_len > done ? min(in_len - done, kRoundBytes) : 0u);
                    const bool to_tag = !OPEN && last && (rb & 15u);
                    const uint32_t end = rd.body + (((to_tag ? rb + BNK_WG_TAG : bytes) + 15u) >> 4);
                    __syncwarp();
                    if (!broken) {
                        awaited |= 1u << buf;
                        if (lane == 0) {
                            bulk_out_read();
                            bar_expect(&bar_all[warp][buf], 16u * end);
                            if (end) bulk_in(stage, a.in + rd.at, 16u * end, &bar_all[warp][buf]);
                        }
                    }
                    arrived(buf);
                }
                // ---- cipher ----
                if (!OPEN && in_len < body) { // WireGuard's padding: zeros behind the payload
                    const uint32_t at = in_len + lane - done;
                    if (lane < 16u && in_len + lane >= done && at < rb)
                        stage_bytes[16u * rd.body + at] = 0;
                    __syncwarp();
                }
                forged = cipher_and_mac<OPEN>(&stage[rd.body], rb, body, last, x, r, state, power, steps, pad, broken, [&] {
                    if (NOTE && rnd == 0) note.place(a.ft);
                });
                if (!OPEN && rnd == 0 && lane == 0) {
                    stage[0] = make_uint4(4u, remote, n_lo, n_hi);
                }
                __syncwarp();
                if (OPEN && a.inner && rnd == 0 && !forged) {
                    const uint4 inner = inner_head(a, stage, rd.body, body);
                    if (lane == 0) a.inner[(size_t)t * T + k] = inner;
                }
                // The last piece goes out whole where the bytes behind the message were read from the same place.
                const uint32_t out_bytes = OPEN ? rb : rb + (last ? BNK_WG_TAG : 0u);
                const bool other_place = a.in != a.out;
                const uint32_t out_end = rd.body + ((out_bytes + (other_place ? 0u : 15u)) >> 4);
                const uint32_t out_from = OPEN ? rd.body : 0u; // (the open side's header stays)
                bulk_fence_shared();
                __syncwarp();
                if (lane == 0 && out_end > out_from && !broken) {
                    bulk_out(a.out + rd.at + 16u * out_from, &stage[out_from], 16u * (out_end - out_from));
                    if (a.out2) bulk_out(a.out2 + rd.at + 16u * out_from, &stage[out_from], 16u * (out_end - out_from));
                    bulk_out_commit();
                }
                if (other_place && lane < (out_bytes & 15u) && !broken) {
                    const uint8_t v = stage_bytes[16u * out_end + lane];
                    a.out[rd.at + 16u * out_end + lane] = v;
                    if (a.out2) a.out2[rd.at + 16u * out_end + lane] = v;
                }
                if (last) break;
            }
            if (OPEN && forged && body > kRoundBytes) { // the earlier rounds' plaintext is out already: wipe it
                uint8_t *const data = a.out + (size_t)off + BNK_WG_HEADER, *const data2 = a.out2 + (size_t)off + BNK_WG_HEADER;
                const uint32_t end = body - (body - 1u) % kRoundBytes - 1u; // what lies in the rounds before the last
                if (lane == 0) bulk_out_done(); // it is, and the zeros come behind it
                bulk_fence();
                __syncwarp();
                for (uint32_t q = lane * 16u; q < end; q += 512u) {
                    *reinterpret_cast<uint4 *>(data + q) = make_uint4(0, 0, 0, 0);
                    if (a.out2) *reinterpret_cast<uint4 *>(data2 + q) = make_uint4(0, 0, 0, 0);
                }
            }
            if (lane == k && broken) {
                res_status = BNK_PKT_NOT_READ;
            } else if (lane == k) {
                res_status = OPEN ? (forged ? BNK_PKT_AUTH_FAIL : body ? BNK_PKT_OK : BNK_PKT_KEEPALIVE) : BNK_PKT_OK;
                res_len = OPEN ? (forged ? 0u : body) : BNK_WG_HEADER + body + BNK_WG_TAG;
            }
            if (NOTE) note.count(a.ft);
            __syncwarp(); // the stage may be filled again
        }
        if (by_cta) {
            if (lane == 0) {
                cta_len[warp] = res_len;
                cta_ctr[warp] = res_ctr;
                cta_status[warp] = (uint8_t)res_status;
                cta_has[warp] = has_counter;
                if (a.res[0].slot) a.res[0].slot[t] = res_slot;
                if (a.res[1].slot) a.res[1].slot[t] = res_slot;
            }
        } else if (lane < in_tile) {
            const uint32_t i = t * T + lane;
#pragma unroll
            for (int d = 0; d < 2; d++) {
                const AeadResults &o = a.res[d];
                if (o.status) o.status[i] = (uint8_t)res_status;
                if (o.out_len) o.out_len[i] = res_len;
                if (o.counter && has_counter) o.counter[i] = res_ctr;
                if (o.slot) o.slot[i] = res_slot;
            }
        }
        cur = next;
    }
    if (lane == 0) bulk_out_done();
    for (uint32_t b = 0; broken && b < 2; b++) // a copy that is still on its way must not meet the next kernel's shared memory
        if ((awaited >> b) & 1u) bar_wait(&bar_all[warp][b], (parity >> b) & 1u);
    if (by_cta) {
        __syncthreads();
        const uint32_t i = blockIdx.x * kWppWarps + threadIdx.x;
        if (threadIdx.x < kWppWarps && i < a.n) {
#pragma unroll
            for (int d = 0; d < 2; d++) {
                const AeadResults &o = a.res[d];
                if (o.status) o.status[i] = cta_status[threadIdx.x];
                if (o.out_len) o.out_len[i] = cta_len[threadIdx.x];
                if (o.counter && cta_has[threadIdx.x]) o.counter[i] = cta_ctr[threadIdx.x];
            }
        }
    }
    signal_done(a.done, NOTE && a.flow_report, [&] { flow_report(flow_ctl(a.ft), a.flow_report); });
}

// ---------------------------------------------------------------------------
// Kernel 3, a stream of packets through each CTA: batches beyond kRankMax packets in pinned memory whose packets lie close
// together in the ring.
//
// There the link is the bound (without any cipher work kernel 2 takes as long), and what counts is how it is asked: in whole
// lines, few of them twice, and with about half a megabyte outstanding in all.  So the first warp brings neighbouring packets up
// as one copy, up to kStreamRun bytes of them, into one of kStreamStages stages, the other warps take the packets of a stage one
// by one, and the whole stretch goes back as one copy: bytes between packets as they were read.  Packets that are refused stay out of
// it, as their descriptors may name bytes of another packet, which has been worked on meanwhile.  The warps that compute are as
// many whatever the size of the packets, which a warp that fetched for itself could not have: with kernel 2's warp for each few
// packets either the requests of all of them are on the link at once, and the writes come afterwards, or small packets wait
// for warps.  At most kStreamAhead copies of a CTA are on their way up, however many of its stages are worked on.
// Plain copies in place, us for 1024 / 4096 / 12,000 packets of 1420 B 1472 apart: a packet at a time, two for each of 256 warps
// 62 / 176 / 482, two neighbours at a time, three stages in 64 CTAs 53 / 164 / 453; with 16 neighbours in 16 CTAs, as many
// bytes, 58 / 169 / 455, in 64 61 / 202 / 499.  9000 of 64 B: a packet at a time 74, 32 at a time 40.
//
// A CTA's packets lie next to each other, which counts when a core has just written them: the open of 1024 x 1420 B 67 us, with
// tiles dealt out in turn 75 (12,000 alike either way, 493 and 490).  A tile of a.tile packets is what the first warp has in its
// lanes: descriptors, of two tiles further ahead as well, since they come over the link behind all that has been asked for; and
// results, until a tile's leave together.
// ---------------------------------------------------------------------------
constexpr uint32_t kStreamWarps = 17, kStreamWorkers = kStreamWarps - 1;
constexpr uint32_t kStreamStages = 6, kStreamAhead = 2, kStreamRun = 3200;
constexpr uint32_t kStreamGap = kJoinGap;  // what may lie between neighbours: no message, wherever its descriptor is, fits in there
// Turns of the first warp in which nothing has happened: seconds.  (A build for tests has it give up at once.)
#ifndef BNK_STREAM_IDLE
#define BNK_STREAM_IDLE (1u << 25)
#endif
static_assert(kStreamRun >= kRoundBytes + BNK_WG_HEADER + 2 * BNK_WG_TAG && kStreamRun % 128 == 0, "a packet of one round fits");
struct StreamRun { // neighbours in a stage
    uint32_t count;        // 0: no more come
    uint32_t first, base;  // the first one, and where it starts in the ring
    uint32_t bytes;        // in the stage; 0: of a packet that lies outside of the ring
    uint32_t turn;         // the worker that takes the first
    bool asked, ends_tile; // asked: the bytes are, or were, on their way
    uint32_t off[32], len[32], slot[32], end[32];
    uint64_t counter[32]; // of a seal; then the results
    uint32_t out_len[32];
    uint8_t status[32], has_counter[32], worked_on[32];
};
struct StreamShared {
    alignas(128) uint4 stage[kStreamStages][(kStreamRun + 64) / 16]; // (a look at a packet's head may go 64 bytes beyond its start)
    StreamRun run[kStreamStages];
    uint64_t ready[kStreamStages], full[kStreamStages], over[kStreamStages]; // a run is described, has come, is worked on
    volatile bool ended; // no more runs come
};
// A wait for the first warp, whose own waits for copies end after bar_wait's time.
__device__ __forceinline__ bool bar_wait_warp(const StreamShared &sh, uint64_t *bar, uint32_t parity) {
    for (uint32_t k = 0; k < 2 * kStreamStages + 2; k++) {
        if (bar_wait(bar, parity)) return true;
        if (sh.ended) return false;
    }
    return false;
}

// The first warp.
template <bool OPEN>
__device__ __forceinline__ void stream_feed(const AeadArgs &a, StreamShared &sh) {
    const uint32_t lane = threadIdx.x & 31, T = a.tile, all = (a.n + T - 1) / T, share = (all + gridDim.x - 1) / gridDim.x;
    uint32_t t = blockIdx.x * share; // the tile that is given out
    const uint32_t tiles = min(all, t + share);
    struct Tile { // a packet's descriptor in each of the first T lanes
        uint32_t off, len, slot;
        uint64_t ctr;
    };
    auto load_tile = [&](uint32_t t) {
        Tile d{0, 0, 0, 0};
        const uint32_t i = t * T + lane;
        if (t < tiles && lane < T && i < a.n) {
            d.off = a.off[i];
            d.len = a.len[i];
            if (!OPEN || !a.demux) d.slot = a.slot[i];
            if (!OPEN && !a.behind_kernel) d.ctr = a.counter[i]; // the host's
        }
        return d;
    };
    uint32_t j = 0; // the tile's next packet
    Tile cur = load_tile(t), next = load_tile(t + 1), after = load_tile(t + 2);
    uint32_t end = 0; // of this lane's packet in the ring, in whole pieces; 0: outside of it
    bool joins = false; // it can come with the one in front
    auto look = [&] {
        const uint64_t room = OPEN ? cur.len : (uint64_t)BNK_WG_HEADER + cur.len;
        end = 0;
        if (lane < T && t * T + lane < a.n && !(cur.off & 15u) && cur.off + room <= a.ring_bytes && (!OPEN || cur.len >= BNK_WG_HEADER + BNK_WG_TAG)) {
            const uint32_t body = OPEN ? cur.len - (BNK_WG_HEADER + BNK_WG_TAG) : wg_padded_len(cur.len, a.mtu);
            const uint64_t message = (uint64_t)BNK_WG_HEADER + body + BNK_WG_TAG;
            const uint64_t size = cur.off + message <= a.ring_bytes && message > room ? message : room;
            if (body <= kRoundBytes && size <= kStreamRun) end = cur.off + (((uint32_t)size + 15u) & ~15u);
        }
        const uint32_t before = __shfl_up_sync(0xffffffffu, end, 1);
        joins = lane > 0 && end && before && cur.off >= before && cur.off - before <= kStreamGap;
    };
    look();
    // Runs are given to the stages in turn: `asked` of them have been, `sent` are on their way back (or have nothing to send).
    uint32_t turn = 0, asked = 0, sent = 0;
    bool fetches = true; // until a copy does not come
    const auto passed = [&](uint64_t *bars, uint32_t run) { // the same for all lanes
        const bool v = __any_sync(0xffffffffu, bar_test(&bars[run % kStreamStages], run / kStreamStages & 1u));
        __syncwarp();
        return v;
    };
    auto ask = [&] {
        const uint32_t s = asked % kStreamStages, in_tile = min(T, a.n - t * T), base = __shfl_sync(0xffffffffu, cur.off, j);
        StreamRun &r = sh.run[s];
        const uint32_t chain = __ballot_sync(0xffffffffu, lane > j && lane < in_tile && joins && end - base <= kStreamRun) >> j >> 1;
        const uint32_t count = (uint32_t)__ffs(~chain); // and the first itself
        const uint32_t to = __shfl_sync(0xffffffffu, end, j + count - 1), bytes = to ? to - base : 0u;
        if (lane >= j && lane < j + count) {
            r.off[lane - j] = cur.off;
            r.len[lane - j] = cur.len;
            r.slot[lane - j] = cur.slot;
            r.end[lane - j] = end;
            if (!OPEN) r.counter[lane - j] = cur.ctr;
        }
        if (lane == 0) {
            r.count = count;
            r.first = t * T + j;
            r.base = base;
            r.bytes = bytes;
            r.turn = turn;
            r.asked = fetches;
            r.ends_tile = j + count == in_tile;
            if (fetches) {
                bar_expect(&sh.full[s], bytes);
                if (bytes) bulk_in(sh.stage[s], a.in + base, bytes, &sh.full[s]);
            }
        }
        __syncwarp();
        if (lane == 0) bar_arrive(&sh.ready[s]);
        asked++;
        turn = (turn + count) % kStreamWorkers;
        j += count;
        if (j < in_tile) return;
        t++;
        j = 0;
        cur = next;
        next = after;
        after = load_tile(t + 2);
        look();
    };
    uint32_t res_len = 0, res_status = BNK_PKT_OK, res_slot = 0, res_has = 0;
    uint64_t res_ctr = 0;
    auto put_results = [&](uint32_t i) {
#pragma unroll
        for (int d = 0; d < 2; d++) {
            const AeadResults &o = a.res[d];
            if (o.status) o.status[i] = (uint8_t)res_status;
            if (o.out_len) o.out_len[i] = res_len;
            if (o.counter && res_has) o.counter[i] = res_ctr;
            if (o.slot) o.slot[i] = res_slot;
        }
    };
    auto send = [&] { // the oldest run, which has been worked on
        StreamRun &r = sh.run[sent % kStreamStages];
        const uint32_t count = r.count, first = r.first & (T - 1), k = lane - first;
        if (lane >= first && k < count) {
            res_len = r.out_len[k];
            res_status = r.status[k];
            res_slot = r.slot[k];
            res_ctr = r.counter[k];
            res_has = r.has_counter[k];
        }
        // (No worker waits for a packet that is refused for its descriptor; and where one has given up, the bytes are as they came.)
        const bool whole = __any_sync(0xffffffffu, r.asked && bar_wait(&sh.full[sent % kStreamStages], sent / kStreamStages & 1u));
        if (!whole) fetches = false;
        const uint32_t goes = __ballot_sync(0xffffffffu, whole && lane < count && r.worked_on[lane]);
        if (lane == 0) {
            for (uint32_t left = goes; left;) { // as a rule one copy of all of them
                const uint32_t k = __ffs(left) - 1, many = __ffs(~(left >> k)) - 1, from = r.off[k] - r.base; // (a run has at most 16)
                bulk_out(a.out + r.off[k], sh.stage[sent % kStreamStages] + from / 16, r.end[k + many - 1] - r.off[k]);
                left &= ~(((1u << many) - 1u) << k);
            }
            bulk_out_commit();
        }
        if (r.ends_tile && lane < first + count) put_results(r.first - first + lane);
        __syncwarp();
        sent++;
    };
    for (uint32_t idle = 0; (t < tiles || sent < asked) && idle < BNK_STREAM_IDLE;) {
        // a stage is free, or will be as soon as the copy out of it has read it, and not too much is on its way
        const bool room = asked < kStreamStages || asked - kStreamStages < sent;
        if (t < tiles && room && (!fetches || asked < kStreamAhead || passed(sh.full, asked - kStreamAhead))) {
            if (asked >= kStreamStages && lane == 0) {
                if (sent - (asked - kStreamStages) >= 2) bulk_out_read_but_last();
                else bulk_out_read();
            }
            __syncwarp();
            ask();
            idle = 0;
        } else if (sent < asked && passed(sh.over, sent)) {
            send();
            idle = 0;
        } else {
            __nanosleep(32);
            idle++;
        }
    }
    if (lane == 0) {
        sh.ended = true;
        if (asked < kStreamStages || asked - kStreamStages < sent) { // in the stage that every worker looks at next
            sh.run[asked % kStreamStages].count = 0;
            bar_arrive(&sh.ready[asked % kStreamStages]);
        }
        bulk_out_done();
    }
    for (uint32_t run = sent; run < asked; run++) // a copy that is still on its way must not meet the next kernel's shared memory
        if (sh.run[run % kStreamStages].asked) bar_wait(&sh.full[run % kStreamStages], run / kStreamStages & 1u);
    const uint32_t left = sent < asked ? sh.run[sent % kStreamStages].first : t * T + j, all_mine = min(a.n, tiles * T);
    if (left >= all_mine) return;
    // It has given up.  The results of the last tile that are known, and for all that has not been sent what it is.
    wait_for_kernel_in_front();
    if (lane < (left & (T - 1))) put_results((left & ~(T - 1)) + lane);
    for (uint32_t i = left + lane; i < all_mine; i += 32) {
        res_status = BNK_PKT_NOT_READ;
        res_len = 0;
        res_slot = OPEN && a.demux ? 0u : a.slot[i];
        res_has = !OPEN && res_slot < a.max_slots;
        if (!OPEN) res_ctr = a.counter[i];
        put_results(i);
    }
}

// The others.
template <bool OPEN, bool NOTE>
__device__ __forceinline__ void stream_work(const AeadArgs &a, StreamShared &sh, uint32_t worker) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t s = 0, parity = 0;;) {
        StreamRun &r = sh.run[s];
        if (!bar_wait_warp(sh, &sh.ready[s], parity)) return;
        const uint32_t count = r.count;
        if (count == 0) return;
        uint4 inner = make_uint4(0, 0, 0, 0); // the n-th of this run's plaintexts of this warp in lane n
        uint32_t inner_of = 0, n_inner = 0;
#pragma unroll 1
        for (uint32_t k = (worker + kStreamWorkers - r.turn) % kStreamWorkers; k < count; k += kStreamWorkers) {
            const uint32_t off = r.off[k], len = r.len[k], pkt = r.first + k;
            uint32_t slot = r.slot[k];
            const bool in_stage = r.bytes != 0;
            uint4 *const stage = sh.stage[s] + (in_stage ? (off - r.base) >> 4 : 0u); // the header, and then the body
            bool broken = false, looked = false;
            auto arrived = [&] {
                if (!looked) broken = !r.asked || !bar_wait(&sh.full[s], parity);
                looked = true;
                broken = __any_sync(0xffffffffu, broken);
                __syncwarp();
            };
            // ---- what the descriptor says (the same for all lanes) ----
            uint8_t st = BNK_PKT_OK, valid = 0;
            uint32_t body = 0, n_lo = 0, n_hi = 0, remote = 0;
            uint64_t ctr = 0;
            uint4 ka = make_uint4(0, 0, 0, 0), kb = ka;
            bool has_counter = !OPEN && slot < a.max_slots;
            auto load_keypair = [&] { // asked for together
                if (slot >= a.max_slots) return;
                const uint4 *const kp = reinterpret_cast<const uint4 *>(a.keys + (size_t)slot * 8);
                valid = a.valid[slot];
                ka = kp[0];
                kb = kp[1];
                if (!OPEN) remote = a.remote_index[slot];
            };
            if (OPEN) {
                if (!a.demux) load_keypair();
                arrived();
                const bool in_ring = (uint64_t)off + len <= a.ring_bytes, whole = in_ring && len >= BNK_WG_HEADER + BNK_WG_TAG;
                uint4 hdr = make_uint4(0, 0, 0, 0);
                if (in_stage) hdr = stage[0];
                if (a.demux) {
                    slot = 0; // descriptors refused below for other reasons
                    if (in_stage) slot = demux_index_warp(a.index_keys, a.index_vals, a.index_slots, hdr.y);
                    load_keypair();
                }
                if (broken) st = BNK_PKT_NOT_READ;
                else if ((off & 15u) || slot >= a.max_slots) st = slot == kSlotNoKeypair ? BNK_PKT_NO_KEYPAIR : BNK_PKT_BAD_DESC;
                else if (!valid) st = BNK_PKT_NO_KEYPAIR;
                else if (!in_ring) st = BNK_PKT_BAD_DESC;
                else if (!whole) st = BNK_PKT_MALFORMED;
                else if (!in_stage) st = BNK_PKT_BAD_DESC; // (longer than the host has said)
                else {
                    n_lo = hdr.z;
                    n_hi = hdr.w;
                    ctr = ((uint64_t)hdr.w << 32) | hdr.z;
                    has_counter = true;
                    if (hdr.x != 4u) st = BNK_PKT_MALFORMED;
                    body = len - (BNK_WG_HEADER + BNK_WG_TAG);
                }
            } else {
                ctr = a.behind_kernel ? a.counter[pkt] : r.counter[k];
                load_keypair();
                n_lo = (uint32_t)ctr;
                n_hi = (uint32_t)(ctr >> 32);
                body = wg_padded_len(len, a.mtu);
                if ((off & 15u) || slot >= a.max_slots) st = BNK_PKT_BAD_DESC;
                else if (!valid) st = BNK_PKT_NO_KEYPAIR;
                else if ((uint64_t)off + BNK_WG_HEADER + body + BNK_WG_TAG > a.ring_bytes || body < len || !in_stage) st = BNK_PKT_BAD_DESC;
                else if (ctr >= BNK_REJECT_AFTER_MESSAGES) st = BNK_PKT_COUNTER_EXHAUSTED;
            }
            FlowNote note;
            auto note_begin = [&] {
                if (NOTE && !broken && in_stage) note_head(note, a, stage, 1, len);
            };
            bool forged = false;
            if (st != BNK_PKT_OK) {
                if (NOTE) {
                    arrived();
                    note_begin();
                    note.place(a.ft);
                }
            } else {
                const uint32_t key[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
                const uint32_t blocks = ((body + 15u) >> 4) + 1u;
                uint32_t x[16], pad[4];
                chacha20_block<1>(x, key, lane, n_lo, n_hi); // lane 0 the one-time key, lane j the body's block j
                const P26 rr = one_time_key(x, pad);
                LanePower power;
                power.begin(rr);
                uint32_t steps = 32u - __clz((blocks + 3u) / 4u - 1u);
                if (!OPEN) {
#pragma unroll 1
                    for (; steps; steps--) power.step();
                    arrived();
                    note_begin();
                }
                if (!broken) {
                    if (!OPEN && len < body) { // WireGuard's padding: zeros behind the payload
                        if (lane < 16u && len + lane < body) reinterpret_cast<uint8_t *>(stage + 1)[len + lane] = 0;
                        __syncwarp();
                    }
                    P26 state = p26_zero();
                    forged = cipher_and_mac<OPEN>(stage + 1, body, body, true, x, rr, state, power, steps, pad, false, [&] {
                        if (NOTE) note.place(a.ft);
                    });
                    if (!OPEN && lane == 0) stage[0] = make_uint4(4u, remote, n_lo, n_hi);
                    __syncwarp();
                    if (OPEN && a.inner && !forged) {
                        const uint4 v = inner_head(a, stage, 1, body);
                        if (lane == n_inner) {
                            inner = v;
                            inner_of = pkt;
                        }
                        n_inner++;
                    }
                }
            }
            if (NOTE) note.count(a.ft);
            __syncwarp();
            if (lane == 0) {
                const bool good = st == BNK_PKT_OK && !broken && !forged;
                r.status[k] = st != BNK_PKT_OK ? st : broken ? BNK_PKT_NOT_READ : forged ? BNK_PKT_AUTH_FAIL : OPEN && body == 0 ? BNK_PKT_KEEPALIVE : BNK_PKT_OK;
                r.out_len[k] = !good ? 0u : OPEN ? body : BNK_WG_HEADER + body + BNK_WG_TAG;
                r.slot[k] = slot;
                r.counter[k] = ctr;
                r.has_counter[k] = has_counter;
                r.worked_on[k] = st == BNK_PKT_OK && !broken;
            }
        }
        bulk_fence_shared();
        __syncwarp();
        if (lane == 0) bar_arrive(&sh.over[s]);
        // The rules are asked while the link is busy, and nothing waits for the answer but the last checks: 10,100 mixed packets opened
        // with everything on 190 us, with the rules asked there 193, 16,160 259 and 262.
        if (OPEN && lane < n_inner) {
            if (a.judge && (inner.z & kInnerParses))
                inner.z |= kInnerJudged | (rules_allow(a.ft, inner_parsed(inner)) ? kInnerAllowed : 0u);
            a.inner[inner_of] = inner;
        }
        __syncwarp();
        if (++s == kStreamStages) {
            s = 0;
            parity ^= 1u;
        }
    }
}

// A CTA stays on its SM until the batch ends, and another call's packets should not have to wait for that.  A quarter of an SM, which has
// five of the 17 warps, has 16,384 registers: with 72 each (and a few in local memory) a warp of kernel 2 of up to 128 still fits beside
// them, with the 94 that the kernel would take it does not; and both have to want the same share of the SM for shared memory (see
// aead_kernels_init).  300 packets with own nonces beside other calls' batches sealed over and over, median and 99th of a hundred,
// as it was / so: 9000 x 64 B 55 and 61 us / 43 and 51, 16,000 x 64 B 89 and 96 / 63 and 85, 16,000 mixed 29 and 199 / 31 and 148,
// 40,000 mixed 49 and 427 / 52 and 178 (by packet or in pieces 43 and 69, 34 and 109, 33 and 117, 49 and 160).  The batches
// themselves take the same time.
constexpr int kStreamShare = 44; // of a hundred: 100 KB, which is what kernel 2's four CTAs get
template <bool OPEN, bool NOTE>
__global__ void __maxnreg__(72) aead_stream_kernel(const __grid_constant__ AeadArgs a) {
    static_assert(!(OPEN && NOTE), "flows are recorded on the seal side");
    let_next_kernel_start();
    __shared__ StreamShared sh;
    if (threadIdx.x < kStreamStages) {
        bar_init(&sh.ready[threadIdx.x]);
        bar_init(&sh.full[threadIdx.x]);
        bar_init(&sh.over[threadIdx.x], kStreamWorkers);
    }
    if (threadIdx.x == 0) sh.ended = false;
    bulk_fence_shared();
    __syncthreads();
    if (threadIdx.x < 32) { // what it reads is the host's
        stream_feed<OPEN>(a, sh);
    } else {
        wait_for_kernel_in_front();
        stream_work<OPEN, NOTE>(a, sh, (threadIdx.x >> 5) - 1u);
    }
    signal_done(a.done, NOTE && a.flow_report, [&] { flow_report(flow_ctl(a.ft), a.flow_report); });
}

// Below this many packets one-packet-per-thread leaves most of the GPU idle and its run time is that of one thread
// walking one packet (~39 us for 1420 B) whatever the batch size; one warp per packet takes ~13 us up to 2,400
// packets and then grows by ~14 us per 2,400 more.  Measured crossover on B200: between 6,000 and 7,000 packets.
#ifndef BNK_WPP_MAX_PACKETS
#define BNK_WPP_MAX_PACKETS 6144u
#endif

// Tiles and grid of a warp-per-packet launch.  Rings in device memory (n <= BNK_WPP_MAX_PACKETS): a warp per packet.
// Rings in host memory: the link is the bound (and packets that lie close together go through kernel 3, see in_stream in layout.h; the figures here
// are of 1472 bytes apart, as longer ones and ones further apart behave).  With a warp per packet all reads are asked for at once, end together and
// leave the writes for afterwards, so beyond kLinkWindow bytes a warp takes several packets: 1024 x 1420 B sealed by
// 32 to 96 CTAs 72 us, by 128 84, by 256 (a packet each) 92; 512 x 1420 46 against 54.  Small packets are bound by what
// a warp computes, and want more warps: 4096 x 300 B 104 us from 64 CTAs, 77 from 128 to 192, 92 from 512; 131,072 x 64 B
// 2.6 ms from 64, 1.16 from 256, 1.01 from 512.  Tiles of 2, 4 or 8 make descriptors and results one access.
// Packets on the device whose messages go to the host as well only store over the link, and all warps that fit help:
// 12,032 x 1420 B in 421 us by 64 CTAs, 395 by 128, 375 by 444 and more.
constexpr uint64_t kLinkWindow = 64u << 10, kLeastCtas = 64, kMostCtas = 512;
constexpr uint32_t kStoreCtas = 592, kEvenCtas = 96;
// The seal kernel hands out nonces for one packet per warp, counted over one tile of the whole batch: a batch of that size
// has to get a warp for every packet.
static_assert(kRankMax <= kLeastCtas * kWppWarps, "batches that hand out their own nonces run a packet per warp");
void wpp_grid(AeadArgs &a, uint32_t &ctas) {
    ctas = (a.n + kWppWarps - 1) / kWppWarps;
    a.tile = 1;
    if (!a.over_link || ctas <= kLeastCtas) return;
    const uint64_t per_packet = a.link_bytes / a.n + 1;
    if (!a.from_host) ctas = std::min(ctas, kStoreCtas);
    else ctas = (uint32_t)std::min<uint64_t>(ctas, std::min(std::max(kLinkWindow / per_packet, kLeastCtas), kMostCtas));
    while (a.tile < 8 && a.n > ctas * kWppWarps * a.tile) a.tile *= 2;
    // Warps that all take as many tiles end together: 9000 x 1420 B are 1125 tiles, five rounds for 64 CTAs, the last with 101 of its
    // 256 warps busy, and three for 94 (sealed 421 us and 394, opened 408 and 389); 15,000 are eight rounds and five (671 and 638, 660
    // and 627).  Where the last round is nearly full there is nothing to gain: 8000 (232 of 256 warps) 362 us, by 84 CTAs 361.  More
    // CTAs than kEvenCtas gain nothing more: 12,000 by 94 (four rounds) 515, by 128 (three) 514; 15,000 by 94 638, by 128 634.
    const uint32_t tiles = (a.n + a.tile - 1) / a.tile;
    if (a.from_host && tiles > ctas * kWppWarps) {
        const uint32_t rounds = (tiles + std::max(ctas, kEvenCtas) * kWppWarps - 1) / (std::max(ctas, kEvenCtas) * kWppWarps);
        ctas = (tiles + rounds * kWppWarps - 1) / (rounds * kWppWarps);
    }
}
template <bool OPEN, bool NOTE>
cudaError_t launch_wpp(const AeadArgs &a, uint32_t ctas, const HostDesc *h, cudaStream_t s) {
    // A launch that may start early costs the driver 2.7 us more when the stream's last kernel is just about to end, as it
    // is when a caller comes back right after its wait; only where a kernel of the same submit is in front does it pay.
    const bool early = a.behind_kernel;
    if (h == nullptr)
        return launch_kernel(early, aead_wpp_kernel<OPEN, NOTE, 0>, dim3(ctas), dim3(32 * kWppWarps), s, a, InlineDesc<0>{});
    const auto with = [&](auto d, auto kernel) {
        memcpy(d.off, h->off, a.n * sizeof(uint32_t));
        memcpy(d.len, h->len, a.n * sizeof(uint32_t));
        memcpy(d.slot, h->slot, a.n * sizeof(uint32_t));
        return launch_kernel(early, kernel, dim3(ctas), dim3(32 * kWppWarps), s, a, d);
    };
    // The cost of a launch grows with its parameters, 12 bytes a packet here: a quarter of a kilobyte, three quarters, two and
    // three kilobytes.  160 leaves a read of the upstream size (128) room for what a receive call brings beyond it.  With
    // room for 256 alone nine packets of 300 B took 57.7 us sealed and opened, 128 x 1420 B 24.2 sealed; with these 54.0
    // and 23.4.
    if (a.n <= 16) return with(InlineDesc<16>{}, aead_wpp_kernel<OPEN, NOTE, 16>);
    if (a.n <= 64) return with(InlineDesc<64>{}, aead_wpp_kernel<OPEN, NOTE, 64>);
    if (a.n <= 160) return with(InlineDesc<160>{}, aead_wpp_kernel<OPEN, NOTE, 160>);
    return with(InlineDesc<kRankMax>{}, aead_wpp_kernel<OPEN, NOTE, kRankMax>);
}

static_assert(kStreamPackets >= kRankMax, "it hands out no nonces itself");

template <bool OPEN>
cudaError_t launch_aead(AeadArgs a, cudaStream_t s, bnk_ctx *ctx) {
    if (a.n == 0) return cudaSuccess;
    if (a.stream) {
        const StreamGrid g = stream_grid(a.n, a.link_bytes);
        a.tile = g.tile;
        const dim3 grid(g.ctas), block(32 * kStreamWarps);
        const cudaError_t e = !OPEN && a.note ? launch_kernel(a.behind_kernel, aead_stream_kernel<OPEN, !OPEN>, grid, block, s, a)
                                              : launch_kernel(a.behind_kernel, aead_stream_kernel<OPEN, false>, grid, block, s, a);
        if (e != cudaSuccess) return e;
        ++ctx->launches;
        return cudaGetLastError();
    }
    const bool wpp = a.over_link || ctx->aead_mode == 2 || (ctx->aead_mode == 0 && a.n <= BNK_WPP_MAX_PACKETS);
    if (wpp) {
        uint32_t ctas;
        wpp_grid(a, ctas);
        // Up to kRankMax descriptors go with the launch: a read of them over the host link costs 1.4 us before the
        // first byte of a packet can be asked for.
        const HostDesc *const h = a.from_host && a.n <= kRankMax ? &a.host : nullptr;
        cudaError_t e = !OPEN && a.note ? launch_wpp<OPEN, !OPEN>(a, ctas, h, s) : launch_wpp<OPEN, false>(a, ctas, h, s);
        if (e != cudaSuccess) return e;
    } else {
        // one CTA per 128 packets; the hardware hands CTAs to SMs as slots free up, which measured faster
        // than persistent warps with an even static share of the packets
        const uint32_t ctas = (a.n + kThreads - 1) / kThreads;
        launch_kernel(a.n <= dependent_launch_up_to(), aead_kernel<OPEN>, dim3(ctas), dim3(kThreads), s, a);
    }
    ++ctx->launches;
    return cudaGetLastError();
}

} // namespace

cudaError_t aead_kernels_init() {
    const auto share = [](auto kernel) { return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, kStreamShare); };
    cudaError_t e = share(aead_stream_kernel<false, false>);
    if (e == cudaSuccess) e = share(aead_stream_kernel<false, true>);
    if (e == cudaSuccess) e = share(aead_stream_kernel<true, false>);
    return e;
}
cudaError_t launch_seal(const AeadArgs &a, cudaStream_t s, bnk_ctx *ctx) { return launch_aead<false>(a, s, ctx); }
cudaError_t launch_open(const AeadArgs &a, cudaStream_t s, bnk_ctx *ctx) { return launch_aead<true>(a, s, ctx); }
