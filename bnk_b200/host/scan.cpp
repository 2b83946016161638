// The pass is on the way of every submit that copies: 131,072 descriptors took 140 us in scalar code, before the first
// byte of 190 MB could move.
#include "../csrc/scan.h"

namespace {

inline __attribute__((always_inline)) PacketScan scan(const uint32_t *off, const uint32_t *len, uint32_t n, uint32_t room) {
    PacketScan r{0, 0, 0, true};
    if (n == 0) return r;
    int64_t end = 0;
    uint64_t sum = 0, over = 0;
    uint32_t longest = 0;
    for (uint32_t i = 0; i + 1 < n; i++) {
        const int64_t e = (int64_t)off[i] + (int64_t)len[i];
        end = e > end ? e : end;
        sum += len[i];
        longest = len[i] > longest ? len[i] : longest;
        over |= (uint64_t)((int64_t)off[i + 1] - e - (int64_t)room); // negative: the top bit
    }
    const int64_t e = (int64_t)off[n - 1] + (int64_t)len[n - 1];
    r.end = (uint64_t)(e > end ? e : end);
    r.sum = sum + len[n - 1];
    r.longest = len[n - 1] > longest ? len[n - 1] : longest;
    r.in_order = !(over >> 63);
    return r;
}

#if defined(__x86_64__)
__attribute__((target("avx2"))) PacketScan scan_avx2(const uint32_t *off, const uint32_t *len, uint32_t n, uint32_t room) {
    return scan(off, len, n, room);
}
#endif

} // namespace

PacketScan scan_packets(const uint32_t *off, const uint32_t *len, uint32_t n, uint32_t room) {
#if defined(__x86_64__)
    static const bool wide = __builtin_cpu_supports("avx2");
    if (wide) return scan_avx2(off, len, n, room);
#endif
    return scan(off, len, n, room);
}
