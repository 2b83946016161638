// How a batch's packets lie in its ring, as far as a submit's way depends on it.
#pragma once

#include <stdint.h>

#include "scan.h"

constexpr uint32_t kMostRoom = 16 + 16 + 16; // header, padding and tag around a payload
constexpr uint32_t kDenseLongest = 1969;     // a message, with its padding, of one round in the kernels' terms
struct Layout {
    uint64_t bytes = 0;    // of the packets
    uint64_t end = 0;      // highest byte of one
    uint32_t joined = 0;   // packets that start where the one in front of them ends, or little behind it
    bool in_order = false; // they lie in the ring in order, each with its own room behind it
    bool dense = false;    // at most about a quarter of their stretch of it lies between them, and none is longer than kDenseLongest
};
// With `slack` bytes beside each packet's own.
inline Layout layout_of(const PacketScan &r, uint32_t n, uint32_t slack) {
    Layout l;
    l.bytes = r.sum + (uint64_t)n * slack;
    l.end = r.end;
    l.joined = r.joined;
    l.in_order = r.in_order;
    l.dense = n && r.longest <= kDenseLongest && 4 * (r.sum + (uint64_t)n * kMostRoom) >= 3 * (r.end - r.lowest);
    return l;
}

// Whether a batch in pinned memory is one for aead_stream_kernel, in which up to two copies of a CTA are on their way, each of
// packets that have been joined; otherwise it has a warp for each few packets, each packet a copy of its own ("by packet").
//
// Packets without gaps.  Below kStreamFrom bytes by packet is as fast: 1000 mixed packets (360 KB) sealed 29.5 us and 30.4, opened 34.3 and
// 35.3; 512 x 1420 B (730 KB) sealed 38.0 and 35.3.  An open works on a stage for longer, as nothing of it can be done beforehand, and of
// large packets few are at hand in a CTA: 1500 x 1000 B, whole path, 105.1 us and 106.7, 4096 x 700 B (2.9 MB) 152.0 and 154.4, 2000 x
// 1420 B (2.8 MB) 148.3 and 148.0, but 4096 x 1420 B opened 197 and 188, 12,000 518 and 500; small ones 9000 x 64 B 80 and 73.
// Sealed by packet and in the stream: 1024 x 1420 B 66 us and 61, 4096 201 and 183, 12,000 535 and 490, 9000 x 64 B 83 and 74, whole path
// 10,000 mixed 176 and 158; 2048 mixed packets (840 KB) are on the line: sealed 47 us, 45 to 50.
//
// Packets that do not all join (wide slots, another order than the ring's) make smaller copies.  9000 x 64 B, sealed / opened, by packet
// 73 / 80 us whatever their order; in the stream with none joined, as in slots of 128 bytes, 91 / 97, of 35 of a hundred 78 / 82, 50
// 73 / 80, 65 67 / 76, all 56 / 73.  None joined: 9000 x 200 B 103 / 113 and 105 / 110, x 300 B 116 / 123 and 120 / 127, x 1000 B
// 297 / 288 and 288 / 299, 4096 x 1300 B in slots of 1472 175 / 174 and 169 / 178, 12,000 x 1420 B 525 / 517 and 499 / 520; 30 of a hundred
// joined: 9000 x 1000 B 296 / 303 and 282 / 295, 12,000 x 1420 B 524 / 521 and 495 / 508.
// Of very many small packets the other way is pieces (see in_pieces), which copy what lies between them as well and of which each has its own
// start; the more packets, the less that counts.  None joined, in pieces and in the stream: 11,000 x 64 B 107 / 123 and 113 / 122, x 100 B 136 /
// 146 and 114 / 124; 15,000 x 200 B 202 / 217 and 169 / 185; 20,000 x 64 B 159 / 173 and 189 / 207, x 128 B 191 / 212 and 198 / 217, x 150 B 217 / 228 and
// 202 / 216, x 300 B in slots of 400 329 / 317 and 254 / 267; 40,000 x 100 B 324 / 338 and 370 / 392, x 150 B 384 / 401 and 395 / 416, x 200 B 432 / 450 and 412 /
// 439; 80,000 x 200 B 782 / 807 and 816 / 869, x 250 B 865 / 899 and 870 / 916, x 300 B 993 / 1009 and 909 / 944; 64 B of which half join, 20,000 146 / 161
// and 135 / 150, 40,000 250 / 262 and 257 / 285.  In no order it is by packet: 16,000 x 150 B 160 / 166 and 171 / 188, x 200 B 160 / 171 and 174 / 187, x 250 B
// 204 / 209 and 196 / 213, x 300 B 225 / 230 and 211 / 226.
// And of large ones beyond 24 MB, none joined: 20,000 of 1056 to 1408 B in slots of 1472 881 / 900 and 726 / 748, x 1420 B 891 / 910 and 819 / 848.
constexpr uint32_t kStreamPackets = 256, kManySmall = 10240, kSmallPacket = 512;
constexpr uint64_t kStreamFrom = 512u << 10, kStreamSmallFrom = 896u << 10, kStreamOpenFrom = 4u << 20, kStreamLarge = 24u << 20;
constexpr uint32_t kStreamCopy = 1000, kStreamOpenCopy = 1520, kStreamSmallCopy = 290; // bytes
constexpr uint32_t kStreamOrderedCopy = 120, kStreamOrderedPer = 400;                  // and a byte more for each so many packets
inline bool in_stream(const Layout &l, uint32_t n, bool open) {
    const bool small = l.bytes <= (uint64_t)kSmallPacket * n;
    if (!l.dense || n <= kStreamPackets || l.bytes < (open == small ? kStreamFrom : open ? kStreamOpenFrom : kStreamSmallFrom)) return false;
    const uint64_t copies = n - l.joined; // (or a few more)
    if (small) {
        const uint64_t least = l.in_order ? kStreamOrderedCopy + n / kStreamOrderedPer : kStreamSmallCopy;
        return 8ull * l.joined >= 5ull * n || (n >= kManySmall && l.bytes >= least * copies);
    }
    return l.end >= kStreamLarge || l.bytes >= (open ? kStreamOpenCopy : kStreamCopy) * copies;
}

// Tiles and grid of that kernel.  Large packets have as much outstanding as the link takes from 96 CTAs: 12,000 x 1420 B by 64 504 us, by 96
// 482, by 148 491.  With small packets more of them help, 9000 x 64 B sealed by 96 CTAs 71 us, by 113 57, by 141 52.  A CTA stays until
// the batch ends and leaves no room on its SM for another call's grouping kernel, so five SMs at the least are left.
// Tiles of 16 are worth a CTA each, smaller ones of 4 at the least spread a batch that has fewer than kStreamTiles of them.
constexpr uint32_t kStreamCtas = 96, kStreamCtasSmall = 143, kStreamTiles = 64;
struct StreamGrid {
    uint32_t tile, ctas;
};
inline StreamGrid stream_grid(uint32_t n, uint64_t bytes) {
    const uint32_t most = bytes <= (uint64_t)kSmallPacket * n ? kStreamCtasSmall : kStreamCtas;
    uint32_t tile = 16;
    while (tile > 4 && n < kStreamTiles * tile) tile /= 2;
    const uint32_t tiles = (n + tile - 1) / tile, rounds = (tiles + most - 1) / most;
    return StreamGrid{tile, (tiles + rounds - 1) / rounds};
}
