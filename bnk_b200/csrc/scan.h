// One pass over a batch's descriptors before its copies are queued.
#pragma once

#include <stdint.h>

struct PacketScan {
    uint64_t end;  // highest off + len
    uint64_t sum;  // of the lengths
    uint32_t longest;
    bool in_order; // every packet and `room` bytes behind it end where the next one starts, or before
};
__attribute__((visibility("hidden"))) PacketScan scan_packets(const uint32_t *off, const uint32_t *len, uint32_t n, uint32_t room);
