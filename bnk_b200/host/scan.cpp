// The pass is on the way of every submit that copies: 131,072 descriptors took 140 us in scalar code, before the first
// byte of 190 MB could move, 63 in vectors of 64-bit sums and 48 in 32 bits, with more looked for.
#include "../csrc/scan.h"

#include <algorithm>

namespace {

struct Stretch { // of descriptors
    uint64_t end = 0, sum = 0;
    uint32_t longest = 0, lowest = ~0u, joined = 0;
    bool apart = true; // in_order
};
// All but the last one's distance from the one behind it.  In 32 bits; false: they do not hold it, as no ring's packets make them.
constexpr uint32_t kStretch = 1024, kLongestIn32 = (1u << 22) - 1, kEndIn32 = 0u - 64u;
inline __attribute__((always_inline)) bool scan_in_32(const uint32_t *off, const uint32_t *len, uint32_t n, uint32_t room, Stretch &s) {
    uint32_t end = 0, sum = 0, longest = 0, lowest = ~0u, joined = 0, wraps = 0, close = 0;
    for (uint32_t i = 0; i < n; i++) {
        const uint32_t e = off[i] + len[i], want = e + room, next = off[i + 1];
        end = e > end ? e : end;
        sum += len[i];
        longest = len[i] > longest ? len[i] : longest;
        lowest = off[i] < lowest ? off[i] : lowest;
        wraps |= e < off[i];
        close |= want > next;
        joined += ((next - ((want + 15u) & ~15u)) & ~kJoinGap) == 0u;
    }
    if (wraps || longest > kLongestIn32 || end >= kEndIn32) return false;
    s = Stretch{end, sum, longest, lowest, joined, !close};
    return true;
}
static_assert(kJoinGap == 16, "places are multiples of 16: at most kJoinGap is none, or one");
static_assert((uint64_t)kStretch * kLongestIn32 < 1ull << 32, "a stretch's sum");
void scan_in_64(const uint32_t *off, const uint32_t *len, uint32_t n, uint32_t room, Stretch &s) {
    s = Stretch{};
    for (uint32_t i = 0; i < n; i++) {
        const uint64_t e = (uint64_t)off[i] + len[i], want = e + room;
        s.end = std::max(s.end, e);
        s.sum += len[i];
        s.longest = std::max(s.longest, len[i]);
        s.lowest = std::min(s.lowest, off[i]);
        s.joined += ((off[i + 1] - ((want + 15u) & ~15ull)) & ~(uint64_t)kJoinGap) == 0u;
        s.apart &= want <= off[i + 1];
    }
}

inline __attribute__((always_inline)) PacketScan scan(const uint32_t *off, const uint32_t *len, uint32_t n, uint32_t room) {
    PacketScan r{0, 0, 0, ~0u, 0, true};
    if (n == 0) return r;
    r.end = (uint64_t)off[n - 1] + len[n - 1];
    r.sum = r.longest = len[n - 1];
    r.lowest = off[n - 1];
    for (uint32_t i = 0; i + 1 < n; i += kStretch) {
        const uint32_t many = n - 1 - i < kStretch ? n - 1 - i : kStretch;
        Stretch s;
        if (!scan_in_32(off + i, len + i, many, room, s)) scan_in_64(off + i, len + i, many, room, s);
        r.end = std::max(r.end, s.end);
        r.sum += s.sum;
        r.longest = std::max(r.longest, s.longest);
        r.lowest = std::min(r.lowest, s.lowest);
        r.joined += s.joined;
        r.in_order &= s.apart;
    }
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
