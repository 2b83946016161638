// One pass over a batch's descriptors before its copies are queued.
#pragma once

#include <stdint.h>

struct PacketScan {
    uint64_t end;  // highest off + len
    uint64_t sum;  // of the lengths
    uint32_t longest;
    uint32_t lowest; // off
    uint32_t joined; // packets that start where the one in front of them and `room` bytes behind it end, in whole pieces of
                     // 16 bytes, or kJoinGap behind that
    bool in_order; // every packet and `room` bytes behind it end where the next one starts, or before
};
constexpr uint32_t kJoinGap = 16;
__attribute__((visibility("hidden"))) PacketScan scan_packets(const uint32_t *off, const uint32_t *len, uint32_t n, uint32_t room);
