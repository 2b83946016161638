// C ABI of libbnkgpu.so (declared in include/bnk_gpu.h): contexts, device tables,
// pinned packet rings with device mirrors, and the submit/wait pipeline that strings
// host->device copies, the kernels and device->host copies on one CUDA stream per batch.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <thread>

#include "filter_device.cuh"
#include "layout.h"
#include "pieces.h"
#include "submit_order.h"

namespace {

thread_local std::string g_last_error; // for failures that have no context to hang on

int fail(bnk_ctx *ctx, int code, const char *what, cudaError_t e = cudaSuccess) {
    char buf[512];
    if (e != cudaSuccess)
        snprintf(buf, sizeof buf, "%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
    else
        snprintf(buf, sizeof buf, "%s", what);
    if (ctx) {
        std::lock_guard<std::mutex> g(ctx->mu);
        ctx->last_error = buf;
    }
    g_last_error = buf;
    return code;
}

#define CK(ctx, call)                                                  \
    do {                                                               \
        cudaError_t _e = (call);                                       \
        if (_e != cudaSuccess) return fail((ctx), BNK_ECUDA, #call, _e); \
    } while (0)

inline void cpu_relax() {
#if defined(__x86_64__) || defined(__i386__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
}

bool is_pow2(uint64_t v) { return v && !(v & (v - 1)); }

// Several zeroed arrays, the first at the beginning, in one allocation: a cudaMalloc or cudaHostAlloc costs tens to
// hundreds of microseconds however little it allocates, and a program pays that for every batch and context it makes.
class Slab {
  public:
    template <typename T>
    void add(T **p, size_t count) {
        parts_.push_back({reinterpret_cast<void **>(p), total_});
        total_ += (count * sizeof(T) + 255) & ~(size_t)255;
    }
    cudaError_t device() {
        void *base = nullptr;
        const cudaError_t e = cudaMalloc(&base, total_);
        if (e != cudaSuccess) return e;
        place(base);
        return cudaMemset(base, 0, total_);
    }
    cudaError_t pinned() {
        void *base = nullptr;
        const cudaError_t e = cudaHostAlloc(&base, total_, cudaHostAllocDefault);
        if (e != cudaSuccess) return e;
        place(base);
        memset(base, 0, total_);
        return cudaSuccess;
    }

  private:
    void place(void *base) {
        for (const auto &part : parts_) *part.first = static_cast<uint8_t *>(base) + part.second;
    }
    std::vector<std::pair<void **, size_t>> parts_;
    size_t total_ = 0;
};

// highest ring byte any of the first n packets can touch (input or output side); with `room` bytes of its own behind each
uint64_t ring_extent(const bnk_batch *b, uint32_t n, uint32_t slack, Layout *l = nullptr, uint32_t room = 0) {
    const PacketScan r = scan_packets(b->host.off, b->host.len, n, room);
    if (l) *l = layout_of(r, n, slack);
    const uint64_t ext = n ? (r.end + slack + 15) & ~15ull : 0;
    return ext > b->ring_bytes ? b->ring_bytes : ext;
}

int begin_submit(bnk_batch *b, uint32_t npkts, bool touches_host = true) {
    if (!b) return BNK_EINVAL;
    if (npkts > b->max_pkts) return fail(b->ctx, BNK_EINVAL, "npkts exceeds the batch capacity");
    if (b->in_flight && touches_host)
        return fail(b->ctx, BNK_EBUSY, "batch has work in flight; call bnk_wait first");
    CK(b->ctx, cudaSetDevice(b->ctx->device));
    return BNK_SUCCESS;
}

// Closes a submit on every path out of it: whatever was queued before an error is still on the batch's stream,
// so a later bnk_wait really waits for it before the host touches the ring.  (Completion is that of the stream:
// work on the side stream is always joined back before a submit returns, and no event is recorded per submit.)
struct SubmitScope {
    bnk_batch *b;
    std::shared_lock<std::shared_mutex> tables; // see bnk_ctx::submit_mu
    explicit SubmitScope(bnk_batch *batch) : b(batch), tables(batch->ctx->submit_mu) {
        b->stats_pending = b->done_watched = false;
        b->order.begins(b->stream);
    }
    ~SubmitScope() {
        b->in_flight = true;
        if (!b->counted) b->ctx->in_flight.fetch_add(1, std::memory_order_relaxed);
        b->counted = true;
    }
};
void submit_over(bnk_batch *b) { // waited for, or going away
    b->in_flight = false;
    launch_graph_give(b->graph);
    b->graph = nullptr;
    if (b->counted) b->ctx->in_flight.fetch_sub(1, std::memory_order_relaxed);
    b->counted = false;
    if (b->direct_counted) b->ctx->direct_in_flight.fetch_sub(b->direct_counted, std::memory_order_relaxed);
    b->direct_counted = 0;
}
// At most two other batches are in flight; more of them come from several threads.
constexpr int kFewOthers = 2;
bool few_in_flight(const bnk_batch *b) {
    return b->ctx->in_flight.load(std::memory_order_relaxed) - (b->counted ? 1 : 0) <= kFewOthers;
}
// Launches what a submit has gathered (launch.h), through a graph while few batches are in flight.
bool through_graph(const bnk_batch *b) { return b->ctx->launch_graphs && few_in_flight(b); }
cudaError_t send_launches(bnk_batch *b, Launches &all) {
    launch_graph_give(b->graph); // (of a submit that nobody waited for)
    b->graph = nullptr;
    const cudaError_t e = all.send(b->graph);
    if (b->graph) b->ctx->graph_launches.fetch_add(1, std::memory_order_relaxed);
    return e;
}
// For the kernel that is the submit's last piece of work: bnk_wait will watch for it.
Done watch_for(bnk_batch *b) {
    b->done_watched = true;
    return Done{b->d_ticket, b->h_done, ++b->done_seq};
}

// The counters of BNK_F_STATS: one launch behind the submit's last kernel, totals straight into pinned memory.
cudaError_t tally_if_asked(bnk_batch *b, uint32_t npkts, uint32_t flags, cudaStream_t s) {
    if (!(flags & BNK_F_STATS)) return cudaSuccess;
    b->stats_pending = true;
    return launch_tally(b, npkts, s);
}

// A batch whose results go back to the host need not be copied at all: the kernels read the caller's pinned ring and
// descriptors through the host link and write the results straight back (pinned memory has the same address on the
// device).  Copies either side of the kernels run one after the other, each at ~55 GB/s and ~8 us before it moves
// anything; a kernel that works on the pinned ring moves both directions at once.  While a HostAlias lives, the
// launchers see the host arrays where the device copies would be; the device copies fall behind (stale_pkts) until
// catch_up or an upload of as many packets.
// Measured with plain copies through SMs, 1440-byte pieces read and written in place, against upload, kernel and
// download in a row: 190 KB 17 us against 33, 1.6 MB 56 against 82, 6.4 MB 177 against 253, 24 MB 613 against 916,
// 190 MB 4.74 ms against 7.0.  Chunks of one batch over three streams, so that the copy engines run both ways, take
// 77 us at 1.6 MB, 234 at 6.4 MB, 680 at 24 MB and 4.55 ms at 190 MB: only far up they are the faster form.
// With several batches in flight the engines overlap the batches' copies with each other (48 GB/s each way together), so a
// large batch runs this way only if nothing else is in flight, or if all that run this way together stay below
// kDirectTogether bytes and at most two others are in flight: SMs move 28-35 GB/s each way over the link and the engines,
// kept busy by that many batches, 46-48.  Queue of 1024-packet batches, Gbit/s with up to fifteen others / two in place
// beyond 384 KB: 32 callers x 4 calls 195 / 255, 16 x 4 193 / 205, 16 x 2 (smaller batches) 182 / 170.
// A small batch always does.  Its copies are too small for the engines, and in-place kernels beside copied batches are
// slower than either alone.  128 x 1420 B a batch, threads x batches each in flight, Gbit/s with at most 16 in place / all
// (best of five to seven; a host that stalls halves single runs): 16 x 1 176 / 177, 12 x 2 118 / 187, 16 x 2 118 / 196, 8 x
// 4 121 / 199, 16 x 4 112 / 195, 32 x 2 97 / 160, 16 x 8 106 / 171, 32 x 4 93 / 148; 256 x 1420 B 16 x 2 146 / 222, 32 x 4 97 /
// 198; 128 x 300 B 16 x 2 40 / 95.
constexpr uint64_t kDirectTogether = 6ull << 20;
constexpr uint64_t kDirectSmall = 384u << 10;
constexpr int kDirectOthers = 2;
bool host_direct(bnk_batch *b, uint32_t npkts, uint32_t flags, uint64_t ext) {
    bnk_ctx *ctx = b->ctx;
    if (ctx->host_direct_bytes == 0 || npkts == 0 || (flags & (BNK_F_NO_H2D | BNK_F_NO_D2H | BNK_F_USE_OUT_LEN)) ||
        ext > ctx->host_direct_bytes)
        return false;
    const uint64_t together = ctx->direct_in_flight.load(std::memory_order_relaxed) - b->direct_counted;
    const int others = ctx->in_flight.load(std::memory_order_relaxed) - (b->counted ? 1 : 0);
    if (ext > kDirectSmall && others > 0 && (together + ext > kDirectTogether || others > kDirectOthers)) return false;
    ctx->direct_in_flight.fetch_add(ext - b->direct_counted, std::memory_order_relaxed);
    b->direct_counted = ext;
    return true;
}
// Calls that look at the first bytes of each packet only read them in place, however many there are and however close together:
// the link takes ~2.2 ns per head (65,536 of them 1472 bytes apart 156 us, 64 bytes apart 110: requests are lines), and a copy costs
// 6-8 us before it moves anything.
// Headers 48 bytes apart checked, copied first / in place: 2000 28.8 us / 17.0, 16,000 40.8 / 32, 80,000 121 / 108, 800,000 908 /
// 896; packets of 64 B noted and checked, 2000 76 / 36, 16,000 132 / 85; datagrams of 28 B classified, 5000 59 / 23, 50,000 178 /
// 117.  With other batches in flight as well, Mpackets/s copied / in place, threads x headers 48 bytes apart: 4 x 2000 159 / 344, 8 x
// 16,000 590 / 772, 8 x 200,000 808 / 913, 8 x 500,000 814 / 931, but 2 x 1,000,000 942 / 916.  (With a lane asking for both halves
// of a head, copying was ahead below 128 bytes a packet from 1024 packets on.)
// A program that goes on with such packets on the device (BNK_F_NO_H2D) then waits for their copy after all.  From the second time
// on they go up in front of the look at their heads: 2000 x 64 B checked and then sealed 68 us with the copy behind, 53 in front,
// 16,000 163 and 153, 300,000 2267 and 1922.
constexpr uint64_t kDense = 128;
constexpr uint32_t kHeadsFirst = 16384, kHeadsMost = 131072, kHeadSlack = 16; // see upload_heads
constexpr uint32_t kDenseFrom = 1024;
bool heads_are_dense(const bnk_batch *b, uint32_t npkts) {
    if (npkts <= kDenseFrom) return false;
    const auto end = [&](uint32_t i) { return (uint64_t)b->host.off[i] + b->host.len[i]; };
    if (!b->heads_go_up) return end(npkts - 1) < kDense * npkts; // (a guess will do, and a look at more is a microsecond)
    // Some seventy packets of a batch in any order come within an eighth of the extent; only if they leave a doubt are all of the
    // descriptors looked through.
    uint64_t seen = end(npkts - 1);
    for (uint32_t i = 0; i < npkts; i += npkts / 64) seen = std::max(seen, end(i));
    return seen * 8 < kDense * npkts * 7 || ring_extent(b, npkts, kHeadSlack) < kDense * npkts;
}
// By every submit, with its flags, in front of anything else.
void behind_heads(bnk_batch *b, uint32_t flags) {
    if (b->heads == Heads::in_place && (flags & BNK_F_NO_H2D)) b->heads_go_up = true;
    if (b->heads == Heads::copied && !(flags & BNK_F_NO_H2D)) b->heads_go_up = false;
    b->heads = Heads::none;
}
bool heads_direct(bnk_batch *b, uint32_t npkts, uint32_t flags) {
    const bool dense = heads_are_dense(b, npkts), direct = !(dense && b->heads_go_up) && host_direct(b, npkts, flags, 0);
    if (dense) b->heads = direct ? Heads::in_place : Heads::copied;
    return direct;
}
// Below ctx->pieces_from (24 MB) a kernel of a warp per packet on the pinned ring is as fast or faster, because the first piece up and the last
// one down have no company: 16,384 x 1420 B 710 us against 750, 32,768 1390 against 1330, 131,072 5.74 ms against 4.96.
// With small packets that kernel is bound by what its warps compute, ~7.5 ns a packet, and pieces win earlier: 8192 x
// 300 B 138 us against 144, 16,384 252 against 233, 131,072 x 64 B 990 against 600.
// Packets that lie close together go up and down by neighbours (see in_stream), and that kernel is ahead up to ctx->stream_pieces_from (64 MB); sealed, pieces /
// in place: 11,000 mixed 204 us and 161, 16,000 262 and 222, 30,000 449 and 400, 20,000 x 64 B 144 and 126, 40,000 x 300 B 508 and 483,
// 18,000 x 1420 B 815 and 741, 32,768 (48 MB) 1358 and 1315, 48,000 (71 MB) 1935 and 1916, 65,536 (96 MB) 2517 and 2595; opened 16,000 mixed
// 264 and 221, 32,768 x 1420 B 1385 and 1342, 65,536 2535 and 2597.  Of two in turn the second is copied while the first is in place, which
// is no slower than both in pieces or copied: 24,000 x 1420 B 833 us a batch and 838, 32,768 1115 and 1125, 30,000 mixed 340 and 338.
bool in_pieces(const bnk_batch *b, uint32_t n, uint32_t flags, uint64_t ext, const Layout &lay, bool open) {
    const bnk_ctx *const ctx = b->ctx;
    const bool stream = in_stream(lay, n, open) && ctx->aead_mode == 0 && ext <= ctx->host_direct_bytes;
    const uint64_t from = stream ? ctx->stream_pieces_from : ctx->pieces_from;
    if (n == 0) return false;
    if (ext < from && (stream || n < kManySmall || ext > (uint64_t)n * kSmallPacket || ext < from / 16)) return false;
    return lay.in_order && b->pieces.up && !(flags & (BNK_F_NO_H2D | BNK_F_NO_D2H | BNK_F_USE_OUT_LEN)) &&
           ctx->in_flight.load(std::memory_order_relaxed) == (b->counted ? 1 : 0);
}
AeadArgs piece_args(AeadArgs a, const Piece &p) {
    a.off += p.first;
    a.len += p.first;
    a.slot += p.first;
    a.counter += p.first;
    if (a.res[0].counter) a.res[0].counter += p.first;
    a.res[0].out_len += p.first;
    a.res[0].status += p.first;
    a.n = p.count;
    return a;
}

struct HostAlias {
    bnk_batch *b;
    DeviceBatch saved;
    bool on;
    HostAlias(bnk_batch *batch, bool enable, uint32_t n) : b(batch), saved(batch->dev), on(enable) {
        if (!on) return;
        DeviceBatch &d = b->dev;
        const bnk_batch_view &h = b->host;
        d.ring = h.ring;
        d.off = h.off;
        d.len = h.len;
        d.slot = h.slot;
        d.counter = h.counter;
        d.out_len = h.out_len;
        d.status = h.status;
        d.src_addr = h.src_addr;
        b->stale_pkts = std::max(b->stale_pkts, n);
    }
    ~HostAlias() {
        if (on) b->dev = saved;
    }
};

// Descriptor fields in slab order.  A run of fields moves as one copy when that is cheap (a batch that is mostly
// full, or a slab prefix of a few KB); otherwise each field moves its first n entries.
enum { D_OFF = 0, D_LEN, D_SLOT, D_COUNTER, D_OUT_LEN, D_STATUS };
const uint32_t kDescOff[7] = {0, 4, 8, 12, 20, 24, 25};   // bytes per entry before each field
cudaError_t desc_copy(bnk_batch *b, size_t n, int first, int last, bool to_device, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const size_t np = b->npad;
    const size_t lo = kDescOff[first] * np;
    const size_t hi = kDescOff[last] * np + (size_t)(kDescOff[last + 1] - kDescOff[last]) * n;
    const cudaMemcpyKind kind = to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    if (first == last || hi - lo <= 65536 || 2 * n >= np) {
        return to_device ? cudaMemcpyAsync(b->d_desc + lo, b->h_desc + lo, hi - lo, kind, s)
                         : cudaMemcpyAsync(b->h_desc + lo, b->d_desc + lo, hi - lo, kind, s);
    }
    for (int f = first; f <= last; f++) {
        const size_t at = kDescOff[f] * np, bytes = (size_t)(kDescOff[f + 1] - kDescOff[f]) * n;
        cudaError_t e = to_device ? cudaMemcpyAsync(b->d_desc + at, b->h_desc + at, bytes, kind, s)
                                  : cudaMemcpyAsync(b->h_desc + at, b->d_desc + at, bytes, kind, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// The ring and, when they travel together, the descriptors.
void ring_is_up(bnk_batch *b, uint64_t ext) {
    if (ext >= b->partial_to) b->partial_to = 0;
}
cudaError_t ring_up(bnk_batch *b, uint64_t ext, bool joint, cudaStream_t s) {
    ring_is_up(b, ext);
    if (joint) return cudaMemcpyAsync(b->d_desc, b->h_desc, b->desc_room + ext, cudaMemcpyHostToDevice, s);
    return ext ? cudaMemcpyAsync(b->dev.ring, b->host.ring, ext, cudaMemcpyHostToDevice, s) : cudaSuccess;
}
cudaError_t ring_down(bnk_batch *b, uint32_t n, uint64_t ext, bool joint, cudaStream_t s) {
    if (b->partial_to) { // what lies between the packets stays the host's
        const cudaError_t e = joint ? desc_copy(b, n, D_OFF, D_STATUS, false, s) : cudaSuccess;
        return e != cudaSuccess ? e : launch_packets_to_host(b, n, s);
    }
    if (joint) return cudaMemcpyAsync(b->h_desc, b->d_desc, b->desc_room + ext, cudaMemcpyDeviceToHost, s);
    return ext ? cudaMemcpyAsync(b->host.ring, b->dev.ring, ext, cudaMemcpyDeviceToHost, s) : cudaSuccess;
}

// Brings the device copies up to the host arrays where submits have run on those.  An upload of as many packets with all
// descriptor fields does the same.  One of those submits may still be in flight, in front on this stream (a submit that
// leaves the host arrays alone needs no wait in between): what is read here on the host, off[] and len[], no kernel writes.
cudaError_t catch_up(bnk_batch *b, cudaStream_t s) {
    const uint32_t n = b->stale_pkts;
    if (n == 0) return cudaSuccess;
    const uint64_t ext = ring_extent(b, n, kMostRoom);
    cudaError_t e = ring_up(b, ext, b->joint_copy, s);
    if (e == cudaSuccess && !b->joint_copy) e = desc_copy(b, n, D_OFF, D_STATUS, true, s);
    if (e == cudaSuccess && b->stale_src)
        e = cudaMemcpyAsync(b->dev.src_addr, b->host.src_addr, (size_t)b->stale_src * BNK_SRC_ADDR_STRIDE, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) b->stale_pkts = b->stale_src = 0;
    return e;
}
// In front of a submit's own upload of n packets, if it makes one: what that does not cover catches up first.  Not so when the
// results come down: the host arrays then hold all there is, and what is behind may stay so.  Returns in `all` whether the
// upload has to bring every descriptor field (and is then to be followed by caught_up).
cudaError_t catch_up_beside(bnk_batch *b, uint32_t n, bool uploads, bool results_down, cudaStream_t s, bool &all) {
    const bool covers = uploads && (results_down || (n >= b->stale_pkts && b->stale_src == 0));
    const cudaError_t e = covers ? cudaSuccess : catch_up(b, s);
    all = b->stale_pkts != 0;
    return e;
}
void caught_up(bnk_batch *b, uint32_t n) {
    if (n >= b->stale_pkts && b->stale_src == 0) b->stale_pkts = 0;
}

AeadArgs aead_args(bnk_batch *b, uint32_t n, bool open, const uint32_t *order) {
    bnk_ctx *ctx = b->ctx;
    AeadArgs a{};
    a.in = a.out = b->dev.ring;
    a.off = b->dev.off;
    a.len = b->dev.len;
    a.slot = b->dev.slot;
    a.counter = b->dev.counter;
    a.res[0] = AeadResults{b->dev.counter, b->dev.out_len, b->dev.status, nullptr};
    a.keys = open ? ctx->kt.recv_keys : ctx->kt.send_keys;
    a.remote_index = ctx->kt.remote_index;
    a.valid = ctx->kt.valid;
    a.order = order;
    a.n = n;
    a.mtu = ctx->cfg.mtu;
    a.max_slots = ctx->cfg.max_keypairs;
    a.ring_bytes = b->ring_bytes;
    return a;
}

} // namespace

int order_begin(bnk_batch *b, bnk_batch *behind) {
    b->behind = behind;
    if (!b->order.ev) CK(b->ctx, cudaEventCreateWithFlags(&b->order.ev, cudaEventDisableTiming));
    b->ordered = true;
    return BNK_SUCCESS;
}
void order_end(bnk_batch *b, int rc) {
    if (rc != BNK_SUCCESS && b->behind) SubmitOrder::failed_behind(b->behind->order);
    b->ordered = false;
    b->behind = nullptr;
}
void batch_set_direct_stream(bnk_batch *b, cudaStream_t s) { b->direct_stream = s; }
cudaError_t order_stream_create(bnk_ctx *ctx, cudaStream_t *s) {
    return cudaStreamCreateWithPriority(s, cudaStreamNonBlocking, ctx->prio_high);
}
// The submit's kernels come next, on the stream it has begun on ...
static cudaError_t order_kernels_begin(bnk_batch *b) {
    return b->ordered && b->behind ? b->order.follow(b->behind->order) : cudaSuccess;
}
// ... and these were the last of them; copies may follow.
static cudaError_t order_kernels_end(bnk_batch *b) { return b->ordered ? b->order.kernels_end() : cudaSuccess; }

extern "C" {

int bnk_abi_version(void) { return BNK_ABI_VERSION; }

const char *bnk_strerror(int code) {
    switch (code) {
    case BNK_SUCCESS: return "success";
    case BNK_EINVAL: return "invalid argument";
    case BNK_ENOMEM: return "out of memory";
    case BNK_ECUDA: return "CUDA error";
    case BNK_ETIMEDOUT: return "timed out";
    case BNK_EBUSY: return "batch busy";
    case BNK_EFULL: return "table full";
    default: return "unknown error";
    }
}

int bnk_device_count(void) {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) return fail(nullptr, BNK_ECUDA, "cudaGetDeviceCount", e);
    return n;
}

const char *bnk_last_error_string(bnk_ctx *ctx) {
    if (!ctx) return g_last_error.c_str();
    std::lock_guard<std::mutex> g(ctx->mu);
    g_last_error = ctx->last_error;
    return g_last_error.c_str();
}

int bnk_ctx_create(const bnk_cfg *cfg, bnk_ctx **out) {
    if (!cfg || !out || cfg->struct_size != sizeof(bnk_cfg)) return fail(nullptr, BNK_EINVAL, "bad bnk_cfg");
    if (cfg->max_keypairs == 0 || cfg->max_keypairs > (1u << 24)) return fail(nullptr, BNK_EINVAL, "max_keypairs out of range");
    if (!is_pow2(cfg->replay_ring_blocks) || cfg->replay_ring_blocks < 2 || cfg->replay_ring_blocks > 1024)
        return fail(nullptr, BNK_EINVAL, "replay_ring_blocks must be a power of two in 2..1024");
    if (cfg->flow_capacity && (!is_pow2(cfg->flow_capacity) || cfg->flow_capacity < 16))
        return fail(nullptr, BNK_EINVAL, "flow_capacity must be a power of two >= 16");
    *out = nullptr;
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess) return fail(nullptr, BNK_ECUDA, "no usable CUDA device (there is no CPU fallback)", e);
    if (cfg->device_id < 0 || cfg->device_id >= ndev) return fail(nullptr, BNK_EINVAL, "device_id out of range");
    CK(nullptr, cudaSetDevice(cfg->device_id));
    int major = 0, sms = 0, one_address = 0, maps_host = 0; // (the whole property record takes a millisecond to put together)
    CK(nullptr, cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, cfg->device_id));
    CK(nullptr, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, cfg->device_id));
    CK(nullptr, cudaDeviceGetAttribute(&one_address, cudaDevAttrUnifiedAddressing, cfg->device_id));
    CK(nullptr, cudaDeviceGetAttribute(&maps_host, cudaDevAttrCanMapHostMemory, cfg->device_id));
    if (major != 10) return fail(nullptr, BNK_ECUDA, "device is not sm_100: this library carries sm_100a code only");

    bnk_ctx *ctx = new (std::nothrow) bnk_ctx();
    if (!ctx) return fail(nullptr, BNK_ENOMEM, "host allocation failed");
    ctx->cfg = *cfg;
    ctx->device = cfg->device_id;
    ctx->sm_count = sms;
    ctx->launches = ctx->graph_launches = 0;
    ctx->aead_mode = 0;
    if (const char *m = getenv("BNK_AEAD_KERNEL")) // tuning and test aid: tpp | wpp
        ctx->aead_mode = !strcmp(m, "tpp") ? 1 : (!strcmp(m, "wpp") ? 2 : 0);
    ctx->host_direct_bytes = 512u << 20;
    if (const char *m = getenv("BNK_HOST_DIRECT_BYTES")) // largest ring extent served without copies; 0 = never
        ctx->host_direct_bytes = strtoull(m, nullptr, 0);
    if (!one_address || !maps_host) ctx->host_direct_bytes = 0; // pinned memory must have one address
    ctx->pieces_from = 24u << 20;
    ctx->stream_pieces_from = 64u << 20;
    if (const char *m = getenv("BNK_PIECES_FROM")) // tuning aid: ring extent from which a batch that is alone goes in pieces
        ctx->pieces_from = ctx->stream_pieces_from = strtoull(m, nullptr, 0);
    ctx->launch_graphs = true;
    if (const char *m = getenv("BNK_LAUNCH_GRAPHS")) // tuning and test aid: 0 = every launch by itself
        ctx->launch_graphs = strtoul(m, nullptr, 0) != 0;
    ctx->aead_side_stream_from = 1u << 18; // below, the seal/open launch is too short for the hand-over between streams to pay
    if (const char *m = getenv("BNK_AEAD_SIDE_STREAM_FROM")) // tuning aid: 0 = seal/open always on the batch's own stream
        ctx->aead_side_stream_from = (uint32_t)strtoul(m, nullptr, 0);
    ctx->prio_low = ctx->prio_high = 0;
    cudaDeviceGetStreamPriorityRange(&ctx->prio_low, &ctx->prio_high);
    ctx->kt = KeypairTables{};
    ctx->ft = FilterTables{};
    launch_graphs_context(ctx->device, true);
    const size_t k = cfg->max_keypairs;
    auto bail = [&](const char *what, cudaError_t err) {
        int rc = fail(nullptr, BNK_ECUDA, what, err);
        bnk_ctx_destroy(ctx);
        return rc;
    };
    if ((e = cudaStreamCreateWithPriority(&ctx->admin_stream, cudaStreamNonBlocking, ctx->prio_high)) != cudaSuccess) return bail("stream", e);
    if ((e = cudaEventCreate(&ctx->timer_start)) != cudaSuccess) return bail("event", e);
    if ((e = cudaEventCreateWithFlags(&ctx->ev_sweep, cudaEventDisableTiming)) != cudaSuccess) return bail("event", e);
    Slab tables;
    tables.add(&ctx->kt.send_keys, k * 8);
    tables.add(&ctx->kt.recv_keys, k * 8);
    tables.add(&ctx->kt.remote_index, k);
    tables.add(&ctx->kt.send_counter, k);
    tables.add(&ctx->kt.replay_last, k);
    tables.add(&ctx->kt.replay_next, k);
    tables.add(&ctx->kt.replay_ring, k * cfg->replay_ring_blocks);
    tables.add(&ctx->kt.allowed_ip, k);
    tables.add(&ctx->kt.valid, k);
    uint32_t islots = 16;
    while (islots < 2 * k) islots <<= 1;
    ctx->kt.index_slots = islots;
    ctx->index_keys_host.assign(islots, 0);
    ctx->index_vals_host.assign(islots, 0);
    ctx->index_live = ctx->index_dead = ctx->addr_live = ctx->addr_dead = 0;
    for (auto &h : ctx->flow_dead_hint) h = 0;
    ctx->flow_errors_seen = 0;
    tables.add(&ctx->kt.index_keys, (size_t)islots);
    tables.add(&ctx->kt.index_vals, (size_t)islots);
    ctx->kt.addr_slots = islots;
    ctx->addr_host.assign(islots, KeypairTables::AddrEntry{});
    tables.add(&ctx->kt.addr_tab, (size_t)islots);
    if ((e = tables.device()) != cudaSuccess) return bail("keypair tables", e);
    if ((e = group_kernels_init()) != cudaSuccess || (e = aead_kernels_init()) != cudaSuccess) return bail("kernel attributes", e);
    if ((e = filter_tables_alloc(ctx)) != cudaSuccess) return bail("filter tables", e);
    if ((e = cudaDeviceSynchronize()) != cudaSuccess) return bail("sync", e);
    *out = ctx;
    return BNK_SUCCESS;
}

int bnk_ctx_destroy(bnk_ctx *ctx) {
    if (!ctx) return BNK_EINVAL;
    cudaSetDevice(ctx->device);
    cudaDeviceSynchronize();
    launch_graphs_context(ctx->device, false);
    cudaFree(ctx->kt.send_keys); // all of the tables' arrays
    filter_tables_free(ctx);
    if (ctx->timer_start) cudaEventDestroy(ctx->timer_start);
    if (ctx->ev_sweep) cudaEventDestroy(ctx->ev_sweep);
    if (ctx->admin_stream) cudaStreamDestroy(ctx->admin_stream);
    delete ctx;
    return BNK_SUCCESS;
}

int bnk_ctx_synchronize(bnk_ctx *ctx) {
    if (!ctx) return BNK_EINVAL;
    CK(ctx, cudaSetDevice(ctx->device));
    CK(ctx, cudaDeviceSynchronize());
    return BNK_SUCCESS;
}

/* ---- keypairs ---- */
// cudaMemset returns before the memory is set, and the batches' streams do not wait for the default stream.
static int memsets_over(bnk_ctx *ctx) {
    CK(ctx, cudaStreamSynchronize(cudaStreamLegacy));
    return BNK_SUCCESS;
}
int bnk_keypair_set_many(bnk_ctx *ctx, uint32_t first_slot, uint32_t n, const uint8_t *send_keys,
                         const uint8_t *recv_keys, const uint32_t *remote_index) {
    if (!ctx || !send_keys || !recv_keys || !remote_index) return fail(ctx, BNK_EINVAL, "null argument");
    if ((uint64_t)first_slot + n > ctx->cfg.max_keypairs) return fail(ctx, BNK_EINVAL, "keypair slot out of range");
    if (n == 0) return BNK_SUCCESS;
    CK(ctx, cudaSetDevice(ctx->device));
    const uint32_t rb = ctx->cfg.replay_ring_blocks;
    CK(ctx, cudaMemcpy(ctx->kt.send_keys + (size_t)first_slot * 8, send_keys, (size_t)n * 32, cudaMemcpyHostToDevice));
    CK(ctx, cudaMemcpy(ctx->kt.recv_keys + (size_t)first_slot * 8, recv_keys, (size_t)n * 32, cudaMemcpyHostToDevice));
    CK(ctx, cudaMemcpy(ctx->kt.remote_index + first_slot, remote_index, (size_t)n * 4, cudaMemcpyHostToDevice));
    CK(ctx, cudaMemset(ctx->kt.send_counter + first_slot, 0, (size_t)n * sizeof(SendCounter)));
    CK(ctx, cudaMemset(ctx->kt.replay_last + first_slot, 0, (size_t)n * 8));
    CK(ctx, cudaMemset(ctx->kt.replay_ring + (size_t)first_slot * rb, 0, (size_t)n * rb * 8));
    CK(ctx, cudaMemset(ctx->kt.allowed_ip + first_slot, 0, (size_t)n * 4));
    CK(ctx, cudaMemset(ctx->kt.valid + first_slot, 1, (size_t)n));
    return memsets_over(ctx);
}

int bnk_keypair_set(bnk_ctx *ctx, uint32_t slot, const uint8_t send_key[32], const uint8_t recv_key[32],
                    uint32_t remote_index) {
    return bnk_keypair_set_many(ctx, slot, 1, send_key, recv_key, &remote_index);
}

static int index_drop_slot(bnk_ctx *ctx, uint32_t slot);

int bnk_keypair_clear(bnk_ctx *ctx, uint32_t slot) {
    static const uint8_t zeros[32] = {0};
    int rc = bnk_keypair_set(ctx, slot, zeros, zeros, 0);
    if (rc != BNK_SUCCESS) return rc;
    // no keys: seal and open refuse the slot with BNK_PKT_NO_KEYPAIR, and no receiver index leads to it any more
    CK(ctx, cudaMemset(ctx->kt.valid + slot, 0, 1));
    rc = memsets_over(ctx);
    return rc != BNK_SUCCESS ? rc : index_drop_slot(ctx, slot);
}

int bnk_send_counter_get(bnk_ctx *ctx, uint32_t slot, uint64_t *counter) {
    if (!ctx || !counter || slot >= ctx->cfg.max_keypairs) return fail(ctx, BNK_EINVAL, "bad slot");
    CK(ctx, cudaSetDevice(ctx->device));
    SendCounter c;
    CK(ctx, cudaMemcpy(&c, ctx->kt.send_counter + slot, sizeof c, cudaMemcpyDeviceToHost));
    *counter = c.e[c.e[0].seq >= c.e[1].seq ? 0 : 1].value;
    return BNK_SUCCESS;
}

int bnk_send_counter_set(bnk_ctx *ctx, uint32_t slot, uint64_t counter) {
    if (!ctx || slot >= ctx->cfg.max_keypairs) return fail(ctx, BNK_EINVAL, "bad slot");
    CK(ctx, cudaSetDevice(ctx->device));
    const SendCounter c{{{counter, 0}, {0, 0}}};
    CK(ctx, cudaMemcpy(ctx->kt.send_counter + slot, &c, sizeof c, cudaMemcpyHostToDevice));
    return BNK_SUCCESS;
}

int bnk_keypair_set_allowed_ip(bnk_ctx *ctx, uint32_t slot, uint32_t ipv4) {
    if (!ctx || slot >= ctx->cfg.max_keypairs) return fail(ctx, BNK_EINVAL, "bad slot");
    CK(ctx, cudaSetDevice(ctx->device));
    CK(ctx, cudaMemcpy(ctx->kt.allowed_ip + slot, &ipv4, 4, cudaMemcpyHostToDevice));
    return BNK_SUCCESS;
}

// The index table is edited in a host shadow and the touched entry is copied over: updates happen once per
// handshake, lookups once per packet.  A deleted entry keeps its slot as a tombstone so that probe chains stay
// intact; every handshake brings a new random index, so tombstones pile up, and once a quarter of the table is
// tombstones the table is rebuilt without them (otherwise a lookup of an unknown index, which anyone can send,
// would end up walking the whole table).
constexpr uint64_t kIndexLive = 1ull << 32, kIndexDead = 2ull << 32;
static int index_rebuild(bnk_ctx *ctx) {
    const uint32_t slots = ctx->kt.index_slots, mask = slots - 1;
    std::vector<uint64_t> keys(slots, 0);
    std::vector<uint32_t> vals(slots, 0);
    for (uint32_t i = 0; i < slots; i++) {
        const uint64_t k = ctx->index_keys_host[i];
        if ((k >> 32) != 1) continue;
        uint32_t h = index_hash((uint32_t)k) & mask;
        while (keys[h]) h = (h + 1) & mask;
        keys[h] = k;
        vals[h] = ctx->index_vals_host[i];
    }
    ctx->index_keys_host.swap(keys);
    ctx->index_vals_host.swap(vals);
    ctx->index_dead = 0;
    CK(ctx, cudaDeviceSynchronize()); // the whole table moves: not under a running lookup
    CK(ctx, cudaMemcpy(ctx->kt.index_vals, ctx->index_vals_host.data(), (size_t)slots * 4, cudaMemcpyHostToDevice));
    CK(ctx, cudaMemcpy(ctx->kt.index_keys, ctx->index_keys_host.data(), (size_t)slots * 8, cudaMemcpyHostToDevice));
    return BNK_SUCCESS;
}
static int index_update(bnk_ctx *ctx, uint32_t local_index, bool insert, uint32_t slot) {
    const uint64_t key = kIndexLive | local_index;
    std::vector<uint64_t> &keys = ctx->index_keys_host;
    const uint32_t mask = ctx->kt.index_slots - 1;
    uint32_t h = index_hash(local_index) & mask;
    int64_t spare = -1, at = -1;
    for (uint32_t probe = 0; probe <= mask; probe++) {
        if (keys[h] == key) {
            at = h;
            break;
        }
        if (keys[h] == kIndexDead && spare < 0) spare = h;
        if (keys[h] == 0) {
            if (spare < 0) spare = h;
            break;
        }
        h = (h + 1) & mask;
    }
    if (!insert) {
        if (at < 0) return BNK_SUCCESS;
        keys[at] = kIndexDead;
        ctx->index_live--;
        ctx->index_dead++;
        CK(ctx, cudaMemcpy(ctx->kt.index_keys + at, &kIndexDead, 8, cudaMemcpyHostToDevice));
        if (ctx->index_dead >= ctx->kt.index_slots / 4) return index_rebuild(ctx);
        return BNK_SUCCESS;
    }
    const bool fresh = at < 0;
    if (at < 0) at = spare;
    if (at < 0) return fail(ctx, BNK_EFULL, "receiver index table full");
    if (fresh) {
        if (keys[at] == kIndexDead) ctx->index_dead--;
        ctx->index_live++;
    }
    // value first, then the key that makes the entry visible
    ctx->index_vals_host[at] = slot;
    CK(ctx, cudaMemcpy(ctx->kt.index_vals + at, &slot, 4, cudaMemcpyHostToDevice));
    keys[at] = key;
    CK(ctx, cudaMemcpy(ctx->kt.index_keys + at, &key, 8, cudaMemcpyHostToDevice));
    return BNK_SUCCESS;
}
// bnk_keypair_clear: the indices that led to the slot lead nowhere now
static int index_drop_slot(bnk_ctx *ctx, uint32_t slot) {
    bool any = false;
    for (uint32_t i = 0; i < ctx->kt.index_slots; i++) {
        if ((ctx->index_keys_host[i] >> 32) != 1 || ctx->index_vals_host[i] != slot) continue;
        ctx->index_keys_host[i] = kIndexDead;
        ctx->index_live--;
        ctx->index_dead++;
        any = true;
        CK(ctx, cudaMemcpy(ctx->kt.index_keys + i, &kIndexDead, 8, cudaMemcpyHostToDevice));
    }
    if (any && ctx->index_dead >= ctx->kt.index_slots / 4) return index_rebuild(ctx);
    return BNK_SUCCESS;
}

int bnk_index_set(bnk_ctx *ctx, uint32_t local_index, uint32_t slot) {
    if (!ctx || slot >= ctx->cfg.max_keypairs) return fail(ctx, BNK_EINVAL, "bad slot");
    CK(ctx, cudaSetDevice(ctx->device));
    return index_update(ctx, local_index, true, slot);
}

int bnk_index_clear(bnk_ctx *ctx, uint32_t local_index) {
    if (!ctx) return BNK_EINVAL;
    CK(ctx, cudaSetDevice(ctx->device));
    return index_update(ctx, local_index, false, 0);
}

// byAddr: same host-shadow scheme as the receiver-index table, tombstones reclaimed the same way
constexpr uint32_t kAddrLive = 1u << 16, kAddrDead = 2u << 16;
static int addr_rebuild(bnk_ctx *ctx) {
    const uint32_t slots = ctx->kt.addr_slots, mask = slots - 1;
    std::vector<KeypairTables::AddrEntry> tab(slots, KeypairTables::AddrEntry{});
    for (const KeypairTables::AddrEntry &e : ctx->addr_host) {
        if (!(e.port & kAddrLive)) continue;
        uint32_t h = addr_hash(e.hi, e.lo, e.port & 0xffffu) & mask;
        while (tab[h].port) h = (h + 1) & mask;
        tab[h] = e;
    }
    ctx->addr_host.swap(tab);
    ctx->addr_dead = 0;
    CK(ctx, cudaDeviceSynchronize());
    CK(ctx, cudaMemcpy(ctx->kt.addr_tab, ctx->addr_host.data(), (size_t)slots * sizeof(KeypairTables::AddrEntry),
                       cudaMemcpyHostToDevice));
    return BNK_SUCCESS;
}
static int addr_update(bnk_ctx *ctx, const uint8_t addr[16], uint16_t port, bool insert, uint32_t peer) {
    uint64_t hi, lo;
    memcpy(&hi, addr, 8);
    memcpy(&lo, addr + 8, 8);
    const uint32_t live = (uint32_t)port | kAddrLive, dead = kAddrDead;
    std::vector<KeypairTables::AddrEntry> &tab = ctx->addr_host;
    const uint32_t mask = ctx->kt.addr_slots - 1;
    uint32_t h = addr_hash(hi, lo, port) & mask;
    int64_t spare = -1, at = -1;
    for (uint32_t probe = 0; probe <= mask; probe++) {
        const KeypairTables::AddrEntry &e = tab[h];
        if (e.port == live && e.hi == hi && e.lo == lo) {
            at = h;
            break;
        }
        if (e.port == dead && spare < 0) spare = h;
        if (e.port == 0) {
            if (spare < 0) spare = h;
            break;
        }
        h = (h + 1) & mask;
    }
    if (!insert) {
        if (at < 0) return BNK_SUCCESS;
        tab[at].port = dead;
        ctx->addr_live--;
        ctx->addr_dead++;
    } else {
        if (at < 0) {
            at = spare;
            if (at < 0) return fail(ctx, BNK_EFULL, "source address table full");
            if (tab[at].port == dead) ctx->addr_dead--;
            ctx->addr_live++;
        }
        tab[at] = KeypairTables::AddrEntry{hi, lo, live, peer, 0};
    }
    CK(ctx, cudaDeviceSynchronize()); // entries are 32 bytes: never rewrite one under a running kernel
    CK(ctx, cudaMemcpy(ctx->kt.addr_tab + at, &tab[at], sizeof tab[at], cudaMemcpyHostToDevice));
    if (!insert && ctx->addr_dead >= ctx->kt.addr_slots / 4) return addr_rebuild(ctx);
    return BNK_SUCCESS;
}

int bnk_addr_set(bnk_ctx *ctx, const uint8_t addr[16], uint16_t port, uint32_t peer_id) {
    if (!ctx || !addr) return BNK_EINVAL;
    CK(ctx, cudaSetDevice(ctx->device));
    return addr_update(ctx, addr, port, true, peer_id);
}

int bnk_addr_clear(bnk_ctx *ctx, const uint8_t addr[16], uint16_t port) {
    if (!ctx || !addr) return BNK_EINVAL;
    CK(ctx, cudaSetDevice(ctx->device));
    return addr_update(ctx, addr, port, false, 0);
}

int bnk_replay_export(bnk_ctx *ctx, uint32_t slot, uint64_t *last, uint64_t *ring) {
    if (!ctx || !last || !ring || slot >= ctx->cfg.max_keypairs) return fail(ctx, BNK_EINVAL, "bad slot");
    CK(ctx, cudaSetDevice(ctx->device));
    const uint32_t rb = ctx->cfg.replay_ring_blocks;
    CK(ctx, cudaMemcpy(last, ctx->kt.replay_last + slot, 8, cudaMemcpyDeviceToHost));
    CK(ctx, cudaMemcpy(ring, ctx->kt.replay_ring + (size_t)slot * rb, (size_t)rb * 8, cudaMemcpyDeviceToHost));
    return BNK_SUCCESS;
}

int bnk_replay_import(bnk_ctx *ctx, uint32_t slot, uint64_t last, const uint64_t *ring) {
    if (!ctx || !ring || slot >= ctx->cfg.max_keypairs) return fail(ctx, BNK_EINVAL, "bad slot");
    CK(ctx, cudaSetDevice(ctx->device));
    const uint32_t rb = ctx->cfg.replay_ring_blocks;
    CK(ctx, cudaMemcpy(ctx->kt.replay_last + slot, &last, 8, cudaMemcpyHostToDevice));
    CK(ctx, cudaMemcpy(ctx->kt.replay_ring + (size_t)slot * rb, ring, (size_t)rb * 8, cudaMemcpyHostToDevice));
    return BNK_SUCCESS;
}

/* ---- ACL ---- */
int bnk_acl_set(bnk_ctx *ctx, int enforce, const bnk_acl_tuple *tuples, size_t n) {
    if (!ctx || (n && !tuples)) return fail(ctx, BNK_EINVAL, "null tuples");
    if (ctx->cfg.max_acl_tuples && n > ctx->cfg.max_acl_tuples) return fail(ctx, BNK_EFULL, "more tuples than max_acl_tuples");
    CK(ctx, cudaSetDevice(ctx->device));
    const int rc = filter_acl_upload(ctx, enforce, tuples, n);
    if (rc != BNK_SUCCESS) return fail(ctx, rc, "rule table upload failed");
    return BNK_SUCCESS;
}

int bnk_flows_clear(bnk_ctx *ctx) {
    if (!ctx) return BNK_EINVAL;
    CK(ctx, cudaSetDevice(ctx->device));
    std::unique_lock<std::shared_mutex> tables(ctx->submit_mu);
    CK(ctx, cudaDeviceSynchronize());
    CK(ctx, filter_flows_clear(ctx, ctx->admin_stream));
    return BNK_SUCCESS;
}

int bnk_flows_count(bnk_ctx *ctx, uint64_t *live) {
    if (!ctx || !live) return BNK_EINVAL;
    CK(ctx, cudaSetDevice(ctx->device));
    CK(ctx, cudaDeviceSynchronize());
    unsigned long long v = 0;
    CK(ctx, cudaMemcpy(&v, ctx->ft.flow_live, sizeof v, cudaMemcpyDeviceToHost));
    *live = v;
    return BNK_SUCCESS;
}

int bnk_flows_export(bnk_ctx *ctx, bnk_flow_entry *out, size_t capacity, size_t *count) {
    if (!ctx || !count || (capacity && !out)) return BNK_EINVAL;
    CK(ctx, cudaSetDevice(ctx->device));
    std::unique_lock<std::shared_mutex> tables(ctx->submit_mu);
    CK(ctx, cudaDeviceSynchronize());
    const int rc = filter_flows_export(ctx, out, capacity, count);
    return rc == BNK_SUCCESS ? rc : fail(ctx, rc, "flow table export failed");
}

int bnk_flows_import(bnk_ctx *ctx, const bnk_flow_entry *entries, size_t n) {
    if (!ctx || (n && !entries)) return BNK_EINVAL;
    CK(ctx, cudaSetDevice(ctx->device));
    std::unique_lock<std::shared_mutex> tables(ctx->submit_mu);
    CK(ctx, cudaDeviceSynchronize());
    const int rc = filter_flows_import(ctx, entries, n);
    return rc == BNK_SUCCESS ? rc : fail(ctx, rc, rc == BNK_EFULL ? "flow table full" : "flow table import failed");
}

int bnk_table_stats_get(bnk_ctx *ctx, bnk_table_stats *out) {
    if (!ctx || !out) return BNK_EINVAL;
    CK(ctx, cudaSetDevice(ctx->device));
    CK(ctx, cudaDeviceSynchronize());
    memset(out, 0, sizeof *out);
    CK(ctx, filter_flow_stats(ctx, &out->flow_live, out->flow_used, out->flow_dead));
    out->flow_capacity = ctx->ft.flow_capacity;
    out->index_live = ctx->index_live;
    out->index_dead = ctx->index_dead;
    out->index_slots = ctx->kt.index_slots;
    out->addr_live = ctx->addr_live;
    out->addr_dead = ctx->addr_dead;
    out->addr_slots = ctx->kt.addr_slots;
    return BNK_SUCCESS;
}

/* ---- batches ---- */
int bnk_batch_destroy(bnk_batch *b) {
    if (!b) return BNK_EINVAL;
    cudaSetDevice(b->ctx->device);
    submit_over(b);
    b->ctx->flow_bounds.over(b->flow_work, nullptr);
    {
        std::unique_lock<std::shared_mutex> tables(b->ctx->submit_mu); // not while table maintenance walks the registry
        std::lock_guard<std::mutex> g(b->ctx->mu);
        std::vector<bnk_batch *> &all = b->ctx->batches;
        for (size_t i = 0; i < all.size(); i++)
            if (all[i] == b) {
                all.erase(all.begin() + i);
                break;
            }
    }
    if (b->stream) cudaStreamSynchronize(b->stream);
    if (b->direct_stream) cudaStreamSynchronize(b->direct_stream);
    for (cudaStream_t side : {b->aux_stream, b->aead_stream, b->pieces.up, b->pieces.down})
        if (side) cudaStreamSynchronize(side);
    cudaFreeHost(b->h_desc); // all of the pinned arrays
    cudaFree(b->d_desc);     // all of the device's
    if (b->k_begin) cudaEventDestroy(b->k_begin);
    if (b->k_end) cudaEventDestroy(b->k_end);
    if (b->a_begin) cudaEventDestroy(b->a_begin);
    if (b->a_end) cudaEventDestroy(b->a_end);
    if (b->t_end) cudaEventDestroy(b->t_end);
    if (b->order.ev) cudaEventDestroy(b->order.ev);
    if (b->pieces.ev_up) cudaEventDestroy(b->pieces.ev_up);
    if (b->pieces.ev_down) cudaEventDestroy(b->pieces.ev_down);
    if (b->pieces.up) cudaStreamDestroy(b->pieces.up);
    if (b->pieces.down) cudaStreamDestroy(b->pieces.down);
    if (b->ev_fork) cudaEventDestroy(b->ev_fork);
    if (b->ev_join) cudaEventDestroy(b->ev_join);
    if (b->ev_fence) cudaEventDestroy(b->ev_fence);
    if (b->ev_aead_go) cudaEventDestroy(b->ev_aead_go);
    if (b->ev_aead_done) cudaEventDestroy(b->ev_aead_done);
    if (b->aead_stream) cudaStreamDestroy(b->aead_stream);
    if (b->aux_stream) cudaStreamDestroy(b->aux_stream);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return BNK_SUCCESS;
}

int bnk_batch_create(bnk_ctx *ctx, uint32_t max_pkts, uint64_t ring_bytes, bnk_batch **out) {
    if (!ctx || !out || max_pkts == 0 || ring_bytes == 0) return fail(ctx, BNK_EINVAL, "bad batch size");
    if (ring_bytes > 0xffffffffull || (ring_bytes & 15)) return fail(ctx, BNK_EINVAL, "ring_bytes must be a multiple of 16 below 4 GiB");
    *out = nullptr;
    CK(ctx, cudaSetDevice(ctx->device));
    bnk_batch *b = new (std::nothrow) bnk_batch();
    if (!b) return fail(ctx, BNK_ENOMEM, "host allocation failed");
    memset(static_cast<void *>(b), 0, sizeof *b);
    b->ctx = ctx;
    b->max_pkts = max_pkts;
    b->ring_bytes = ring_bytes;
    const size_t n = max_pkts;
    cudaError_t e = cudaSuccess;
    // One slab per side: the descriptor arrays, then the ring.  A batch whose descriptor slab is small moves
    // descriptors and ring with one copy each way (joint_copy); otherwise the descriptor fields a call needs
    // move as one run or field by field (desc_copy).  What else the batch needs lies behind.
    b->npad = (max_pkts + 15u) & ~15u;
    const size_t np = b->npad;
    b->desc_room = (25 * np + 255) & ~(size_t)255;
    b->joint_copy = b->desc_room <= 64u * 1024;
    if (!b->joint_copy) b->desc_room = (b->desc_room + 4095) & ~(size_t)4095; // the ring then starts on a page: see Pieces
    DeviceBatch &d = b->dev;
    Slab pinned, device;
    pinned.add(&b->h_desc, b->desc_room + ring_bytes);
    pinned.add(&b->host.src_addr, n * BNK_SRC_ADDR_STRIDE);
    pinned.add(&b->h_gso, n);
    pinned.add(&b->h_flow, 1);
    pinned.add(&b->h_stats, 1);
    pinned.add(&b->h_done, 32);
    e = pinned.pinned();
    device.add(&b->d_desc, b->desc_room + ring_bytes);
    device.add(&d.src_addr, n * BNK_SRC_ADDR_STRIDE);
    device.add(&d.order, n);
    device.add(&d.order_tmp, n);
    device.add(&d.keys_tmp, 2 * n);
    device.add(&d.sorted_counter, n);
    device.add(&d.replay_state, n);
    device.add(&d.replay_hash, replay_hash_capacity(max_pkts));
    device.add(&d.replay_tile_head, (size_t)replay_scan_tiles(max_pkts) + 1);
    device.add(&d.replay_tile_max, replay_scan_tiles(max_pkts));
    device.add(&d.replay_tile_carry, replay_scan_tiles(max_pkts));
    device.add(&d.hist, (size_t)512 * group_sort_chunks(max_pkts)); // histogram columns + one row of totals
    device.add(&d.len_order, n);
    device.add(&d.inner, n);
    device.add(&d.counters32, 2048);
    device.add(&d.gso, n);
    device.add(&b->d_ticket, 32);
    device.add(&b->d_stats, 20);
    if (e == cudaSuccess) e = device.device();
    if (e == cudaSuccess) {
        auto fields = [&](uint8_t *p, auto &v) {
            v.ring = p + b->desc_room;
            v.off = reinterpret_cast<uint32_t *>(p);
            v.len = reinterpret_cast<uint32_t *>(p + 4 * np);
            v.slot = reinterpret_cast<uint32_t *>(p + 8 * np);
            v.counter = reinterpret_cast<uint64_t *>(p + 12 * np);
            v.out_len = reinterpret_cast<uint32_t *>(p + 20 * np);
            v.status = p + 24 * np;
        };
        fields(b->h_desc, b->host);
        fields(b->d_desc, d);
    }
    b->host.ring_bytes = ring_bytes;
    b->host.max_pkts = max_pkts;
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&b->stream, cudaStreamNonBlocking, ctx->prio_high);
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&b->aux_stream, cudaStreamNonBlocking, ctx->prio_high);
    if (e == cudaSuccess && ctx->aead_side_stream_from && max_pkts >= ctx->aead_side_stream_from && ctx->prio_low != ctx->prio_high) {
        e = cudaStreamCreateWithPriority(&b->aead_stream, cudaStreamNonBlocking, ctx->prio_low);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_aead_go, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_aead_done, cudaEventDisableTiming);
    }
    if (e == cudaSuccess && (ring_bytes >= ctx->pieces_from || max_pkts >= kManySmall)) {
        e = cudaStreamCreateWithPriority(&b->pieces.up, cudaStreamNonBlocking, ctx->prio_high);
        if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&b->pieces.down, cudaStreamNonBlocking, ctx->prio_high);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->pieces.ev_up, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->pieces.ev_down, cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_join, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_fence, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreate(&b->k_begin);
    if (e == cudaSuccess) e = cudaEventCreate(&b->k_end);
    if (e == cudaSuccess) e = cudaEventCreate(&b->t_end);
    if (e == cudaSuccess) e = cudaEventCreate(&b->a_begin);
    if (e == cudaSuccess) e = cudaEventCreate(&b->a_end);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        int rc = fail(ctx, e == cudaErrorMemoryAllocation ? BNK_ENOMEM : BNK_ECUDA, "batch allocation", e);
        bnk_batch_destroy(b);
        return rc;
    }
    {
        std::unique_lock<std::shared_mutex> tables(ctx->submit_mu);
        std::lock_guard<std::mutex> g(ctx->mu);
        ctx->batches.push_back(b);
    }
    *out = b;
    return BNK_SUCCESS;
}

int bnk_batch_view_get(bnk_batch *b, bnk_batch_view *out) {
    if (!b || !out) return BNK_EINVAL;
    *out = b->host;
    return BNK_SUCCESS;
}

int bnk_batch_upload(bnk_batch *b, uint32_t npkts) {
    int rc = begin_submit(b, npkts);
    if (rc) return rc;
    SubmitScope scope(b);
    bnk_ctx *ctx = b->ctx;
    const size_t n = npkts;
    bool all;
    CK(ctx, catch_up_beside(b, npkts, true, false, b->stream, all));
    const uint64_t ext = ring_extent(b, npkts, 64);
    CK(ctx, ring_up(b, ext, false, b->stream));
    if (n) {
        CK(ctx, desc_copy(b, n, D_OFF, all ? D_STATUS : D_COUNTER, true, b->stream));
    }
    caught_up(b, npkts);
    return BNK_SUCCESS;
}

int bnk_batch_download(bnk_batch *b, uint32_t npkts) {
    int rc = begin_submit(b, npkts);
    if (rc) return rc;
    SubmitScope scope(b);
    bnk_ctx *ctx = b->ctx;
    const size_t n = npkts;
    if (b->stale_pkts) return BNK_SUCCESS; // the last submit already left its results in the host arrays
    const uint64_t ext = ring_extent(b, npkts, 64);
    if (n) {
        CK(ctx, ring_down(b, npkts, ext, false, b->stream));
        CK(ctx, desc_copy(b, n, D_COUNTER, D_STATUS, false, b->stream));
    }
    return BNK_SUCCESS;
}

// A seal that works on the pinned ring and descriptors: one launch up to kRankMax packets, else one more in front of
// it for the counters, and one behind it when expired flows may have to be swept.  With `resident` the packets and
// descriptors are those on the device (BNK_F_NO_H2D), and the messages go to both rings as they are made: 17 MB of
// segments sealed and stored 0.38 ms, against 0.44 for seal and download in a row.
static int seal_direct(bnk_batch *b, uint32_t npkts, const Layout &lay, uint32_t flags, int64_t now_unix_ns, bool resident) {
    bnk_ctx *ctx = b->ctx;
    cudaStream_t s = b->direct_stream ? b->direct_stream : b->stream;
    b->order.begins(s);
    const bool timed = (flags & BNK_F_TIMED) != 0, stats = (flags & BNK_F_STATS) != 0;
    const bool assign = (flags & BNK_F_ASSIGN_COUNTERS) != 0;
    const bnk_batch_view &h = b->host;
    const DeviceBatch &d = b->dev;
    CK(ctx, order_kernels_begin(b));
    Launches all(s, !timed && !stats && through_graph(b));
    if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
    AeadArgs a = aead_args(b, npkts, false, nullptr);
    a.over_link = true;
    a.link_bytes = lay.bytes;
    a.out = h.ring;
    a.res[0] = AeadResults{assign ? h.counter : nullptr, h.out_len, h.status, nullptr};
    if (resident) {
        b->split_sealed = std::max(b->split_sealed, npkts);
        a.out2 = d.ring;
        a.res[1] = AeadResults{nullptr, d.out_len, d.status, nullptr}; // the counters are there
        if (!assign) a.res[0].counter = h.counter;
    } else {
        b->stale_pkts = std::max(b->stale_pkts, npkts);
        a.from_host = true;
        a.stream = ctx->aead_mode == 0 && in_stream(lay, npkts, false);
        a.host = HostDesc{h.off, h.len, h.slot};
        a.in = h.ring;
        a.off = h.off;
        a.len = h.len;
        a.slot = h.slot;
        a.counter = h.counter;
        if (stats) a.res[1] = AeadResults{nullptr, d.out_len, d.status, nullptr};
    }
    if (assign) {
        if (!resident && npkts <= kRankMax) {
            a.send_counter = ctx->kt.send_counter;
            a.seal_seq = ++ctx->seal_seq;
        } else {
            a.counter = d.counter;
            a.behind_kernel = true;
            CK(ctx, launch_assign_counters(b, npkts, a.slot, d.counter, s));
        }
    }
    const bool note = (flags & BNK_F_NOTE_OUTBOUND) && ctx->ft.enforce && ctx->ft.flow_capacity; // filter.go:192-194
    bool sweep = false;
    if (note) CK(ctx, flow_note_begins(b, npkts, now_unix_ns, s, sweep));
    const Done done = stats ? Done{} : watch_for(b);
    if (note) {
        a.note = true;
        a.now = now_unix_ns;
        a.ft = ctx->ft;
    }
    if (!sweep) {
        a.done = done;
        if (note && done.flag) {
            a.flow_report = b->h_flow;
            b->flow_reported = true;
        }
    }
    if (timed) CK(ctx, cudaEventRecord(b->a_begin, s));
    CK(ctx, launch_seal(a, s, ctx));
    if (timed) CK(ctx, cudaEventRecord(b->a_end, s));
    if (!sweep) CK(ctx, send_launches(b, all));
    else CK(ctx, all.stop()); // more than launches follow
    if (sweep) CK(ctx, launch_flow_sweep(b, now_unix_ns, done, s));
    else if (note && !done.flag) CK(ctx, launch_flow_report(b, s));
    if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
    b->kernel_timed = b->aead_timed = timed;
    CK(ctx, tally_if_asked(b, npkts, flags, s));
    return BNK_SUCCESS;
}

static int seal_pieces(bnk_batch *b, uint32_t npkts, uint64_t ext, uint32_t flags, int64_t now_unix_ns) {
    bnk_ctx *ctx = b->ctx;
    cudaStream_t s = b->stream;
    const bool timed = (flags & BNK_F_TIMED) != 0;
    Pieces pieces(b->host.off, b->host.len, npkts, kMostRoom, ext);
    PieceCopies copies(b->pieces, b->dev.ring, b->host.ring, s);
    Piece p;
    pieces.next(p); // the first is on its way while the kernels in front of the first seal are prepared
    CK(ctx, copies.up(p));
    CK(ctx, desc_copy(b, npkts, D_OFF, b->stale_pkts ? D_STATUS : (flags & BNK_F_ASSIGN_COUNTERS) ? D_SLOT : D_COUNTER, true, s));
    caught_up(b, npkts); // (more of them stay behind: the host arrays will hold this call's results as well)
    ring_is_up(b, ext);
    CK(ctx, order_kernels_begin(b));
    if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
    if (flags & BNK_F_ASSIGN_COUNTERS) CK(ctx, launch_assign_counters(b, npkts, b->dev.slot, b->dev.counter, s));
    AeadArgs a = aead_args(b, npkts, false, nullptr); // (length classes would only be those of a piece, and the link is the bound)
    a.res[0].counter = nullptr; // in place already
    a.behind_kernel = true;
    const bool note = (flags & BNK_F_NOTE_OUTBOUND) && ctx->ft.enforce && ctx->ft.flow_capacity; // filter.go:192-194
    bool sweep = false;
    if (note) CK(ctx, flow_note_begins(b, npkts, now_unix_ns, s, sweep));
    if (timed) CK(ctx, cudaEventRecord(b->a_begin, s));
    for (bool more = true; more;) {
        CK(ctx, copies.is_up());
        if (note) CK(ctx, launch_filter_note(b, p.first, p.count, now_unix_ns, Done{}, s));
        CK(ctx, launch_seal(piece_args(a, p), s, ctx));
        CK(ctx, copies.down(p));
        more = pieces.next(p);
        if (more) CK(ctx, copies.up(p));
    }
    if (timed) CK(ctx, cudaEventRecord(b->a_end, s));
    if (sweep) CK(ctx, launch_flow_sweep(b, now_unix_ns, Done{}, s));
    else if (note) CK(ctx, launch_flow_report(b, s));
    if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
    b->kernel_timed = b->aead_timed = timed;
    CK(ctx, tally_if_asked(b, npkts, flags, s));
    CK(ctx, order_kernels_end(b));
    CK(ctx, desc_copy(b, npkts, D_COUNTER, D_STATUS, false, s));
    CK(ctx, copies.join());
    return BNK_SUCCESS;
}

int bnk_seal_submit(bnk_batch *b, uint32_t npkts, uint32_t flags, int64_t now_unix_ns) {
    const bool device_only = (flags & BNK_F_NO_H2D) && (flags & BNK_F_NO_D2H);
    int rc = begin_submit(b, npkts, !device_only);
    if (rc) return rc;
    if (flags & BNK_F_NOTE_OUTBOUND) CK(b->ctx, filter_flows_maintain(b, b->stream));
    SubmitScope scope(b);
    behind_heads(b, flags);
    bnk_ctx *ctx = b->ctx;
    cudaStream_t s = b->stream;
    const bool timed = (flags & BNK_F_TIMED) != 0;
    const size_t n = npkts;
    Layout lay;
    const uint64_t ext = device_only ? 0 : ring_extent(b, npkts, kMostRoom, &lay, BNK_WG_HEADER + BNK_WG_TAG);
    if (in_pieces(b, npkts, flags, ext, lay, false)) return seal_pieces(b, npkts, ext, flags, now_unix_ns);
    if (ctx->aead_mode != 1) {
        if (host_direct(b, npkts, flags, ext)) return seal_direct(b, npkts, lay, flags, now_unix_ns, false);
        if (!b->stale_pkts && (flags & BNK_F_NO_H2D) && host_direct(b, npkts, flags & ~BNK_F_NO_H2D, ext))
            return seal_direct(b, npkts, lay, flags, now_unix_ns, true);
    }
    bool all;
    CK(ctx, catch_up_beside(b, npkts, !(flags & BNK_F_NO_H2D), !(flags & BNK_F_NO_D2H), s, all));
    if (!(flags & BNK_F_NO_H2D) && n) {
        CK(ctx, ring_up(b, ext, b->joint_copy, s));
        if (!b->joint_copy)
            CK(ctx, desc_copy(b, n, D_OFF, all ? D_STATUS : (flags & BNK_F_ASSIGN_COUNTERS) ? D_SLOT : D_COUNTER, true, s));
        caught_up(b, npkts);
    }
    CK(ctx, order_kernels_begin(b));
    if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
    if ((flags & BNK_F_NOTE_OUTBOUND) && n && ctx->ft.enforce && ctx->ft.flow_capacity) { // filter.go:192-194
        bool sweep;
        CK(ctx, flow_note_begins(b, npkts, now_unix_ns, s, sweep));
        CK(ctx, launch_filter_note(b, 0, npkts, now_unix_ns, Done{}, s));
        if (sweep) CK(ctx, launch_flow_sweep(b, now_unix_ns, Done{}, s));
        else CK(ctx, launch_flow_report(b, s));
    }
    const uint32_t *order = nullptr;
    const bool side_order = (flags & BNK_F_SORT_BY_LENGTH) && (flags & BNK_F_ASSIGN_COUNTERS) && npkts > 4096;
    if (side_order) { // the length classes need only len[]: they are built beside the grouping for the counters
        CK(ctx, cudaEventRecord(b->ev_fork, s));
        CK(ctx, cudaStreamWaitEvent(b->aux_stream, b->ev_fork, 0));
        CK(ctx, launch_length_order(b, npkts, b->dev.len, false, b->aux_stream));
        CK(ctx, cudaEventRecord(b->ev_join, b->aux_stream));
        order = b->dev.len_order;
    }
    if (flags & BNK_F_ASSIGN_COUNTERS) CK(ctx, launch_assign_counters(b, npkts, b->dev.slot, b->dev.counter, s));
    if (side_order) {
        CK(ctx, cudaStreamWaitEvent(s, b->ev_join, 0));
    } else if (flags & BNK_F_SORT_BY_LENGTH) {
        CK(ctx, launch_length_order(b, npkts, b->dev.len, false, s));
        order = b->dev.len_order;
    }
    AeadArgs a = aead_args(b, npkts, false, order);
    a.res[0].counter = nullptr; // in place already
    a.behind_kernel = true;
    const bool side = b->aead_stream && npkts >= ctx->aead_side_stream_from;
    cudaStream_t as = side ? b->aead_stream : s;
    if (side) {
        CK(ctx, cudaEventRecord(b->ev_aead_go, s));
        CK(ctx, cudaStreamWaitEvent(as, b->ev_aead_go, 0));
    }
    if (timed) CK(ctx, cudaEventRecord(b->a_begin, as));
    CK(ctx, launch_seal(a, as, ctx));
    b->split_sealed = std::max(b->split_sealed, npkts);
    if (timed) CK(ctx, cudaEventRecord(b->a_end, as));
    if (side) {
        CK(ctx, cudaEventRecord(b->ev_aead_done, as));
        CK(ctx, cudaStreamWaitEvent(s, b->ev_aead_done, 0));
    }
    if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
    b->kernel_timed = timed;
    b->aead_timed = timed;
    CK(ctx, tally_if_asked(b, npkts, flags, s));
    CK(ctx, order_kernels_end(b));
    if (!(flags & BNK_F_NO_D2H) && n) {
        if (b->joint_copy) {
            CK(ctx, ring_down(b, npkts, ext, true, s));
        } else {
            CK(ctx, ring_down(b, npkts, ext, false, s));
            CK(ctx, desc_copy(b, n, D_COUNTER, D_STATUS, false, s));
        }
    }
    return BNK_SUCCESS;
}

// An open that works on the pinned ring and descriptors.  What has to wait for the replay window (statuses, lengths)
// stays on the device until then, with the packets' inner headers, so that no later kernel goes back to the ring.
static int open_direct(bnk_batch *b, uint32_t npkts, const Layout &lay, uint32_t flags, int64_t now_unix_ns) {
    bnk_ctx *ctx = b->ctx;
    cudaStream_t s = b->direct_stream ? b->direct_stream : b->stream;
    b->order.begins(s);
    const bool timed = (flags & BNK_F_TIMED) != 0, stats = (flags & BNK_F_STATS) != 0;
    const bool replay = (flags & BNK_F_REPLAY) != 0, checks = (flags & (BNK_F_INNER_CHECK | BNK_F_CHECK_INBOUND)) != 0;
    const bnk_batch_view &h = b->host;
    b->stale_pkts = std::max(b->stale_pkts, npkts);
    const bool one_launch = npkts <= kGroupMax || !replay; // behind the open kernel
    CK(ctx, order_kernels_begin(b));
    Launches all(s, !timed && !stats && one_launch && through_graph(b));
    if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
    AeadArgs a = aead_args(b, npkts, true, nullptr);
    a.over_link = a.from_host = true;
    // With many batches in flight the link is the bound, and the headers' own requests take a share of it: 128 x 1420 B sealed and
    // opened, threads x batches, Gbit/s with the headers first / without: 8 x 2 177 / 181, 8 x 4 191 / 201, 16 x 4 200 / 214.
    a.header_first = few_in_flight(b);
    a.host = HostDesc{h.off, h.len, h.slot};
    a.link_bytes = lay.bytes;
    a.stream = ctx->aead_mode == 0 && in_stream(lay, npkts, true);
    a.in = a.out = h.ring;
    a.off = h.off;
    a.len = h.len;
    a.slot = h.slot;
    a.res[0] = AeadResults{h.counter, h.out_len, h.status, nullptr};
    if (flags & BNK_F_DEMUX_INDEX) {
        a.demux = true;
        a.index_keys = ctx->kt.index_keys;
        a.index_vals = ctx->kt.index_vals;
        a.index_slots = ctx->kt.index_slots;
        a.res[0].slot = h.slot;
    }
    const bool tail = replay || checks;
    if (tail) {
        a.res[0].out_len = nullptr;
        a.res[0].status = nullptr;
        a.res[1] = AeadResults{b->dev.counter, b->dev.out_len, b->dev.status, b->dev.slot};
        if (checks) a.inner = b->dev.inner;
        a.inner_cut = (flags & BNK_F_INNER_CHECK) != 0;
        a.ft = ctx->ft;
        a.judge = (flags & BNK_F_CHECK_INBOUND) && ctx->ft.enforce;
    } else if (stats) {
        a.res[1] = AeadResults{nullptr, b->dev.out_len, b->dev.status, nullptr};
    }
    // beyond one launch the replay window is a chain of kernels, and the results come back by copy
    const Done done = stats || !one_launch ? Done{} : watch_for(b);
    if (!tail) a.done = done;
    if (timed) CK(ctx, cudaEventRecord(b->a_begin, s));
    CK(ctx, launch_open(a, s, ctx));
    if (timed) CK(ctx, cudaEventRecord(b->a_end, s));
    if (tail) {
        VerdictArgs v{};
        v.ft = ctx->ft;
        v.inner = b->dev.inner;
        v.slot = b->dev.slot;
        v.allowed_ip = ctx->kt.allowed_ip;
        v.status = b->dev.status;
        v.out_len = b->dev.out_len;
        v.now = now_unix_ns;
        v.n = npkts;
        v.inner_check = (flags & BNK_F_INNER_CHECK) != 0;
        v.check_inbound = (flags & BNK_F_CHECK_INBOUND) != 0;
        if (v.check_inbound) CK(ctx, flow_check_begins(b, now_unix_ns, s));
        if (one_launch) {
            v.host_status = h.status;
            v.host_out_len = h.out_len;
            CK(ctx, launch_open_tail(b, npkts, replay, &v, done, s));
        } else {
            CK(ctx, launch_group_by_slot(b, npkts, s));
            CK(ctx, launch_replay(b, npkts, s));
            if (checks) CK(ctx, launch_verdict(ctx, v, Done{}, s));
        }
    }
    CK(ctx, send_launches(b, all));
    if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
    b->kernel_timed = b->aead_timed = timed;
    CK(ctx, tally_if_asked(b, npkts, flags, s));
    if (!one_launch) CK(ctx, desc_copy(b, npkts, D_OUT_LEN, D_STATUS, false, s));
    return BNK_SUCCESS;
}

static int open_pieces(bnk_batch *b, uint32_t npkts, uint64_t ext, uint32_t flags, int64_t now_unix_ns) {
    bnk_ctx *ctx = b->ctx;
    cudaStream_t s = b->stream;
    const bool timed = (flags & BNK_F_TIMED) != 0, demux = (flags & BNK_F_DEMUX_INDEX) != 0;
    Pieces pieces(b->host.off, b->host.len, npkts, 0, ext);
    PieceCopies copies(b->pieces, b->dev.ring, b->host.ring, s);
    Piece p;
    pieces.next(p);
    CK(ctx, copies.up(p));
    CK(ctx, desc_copy(b, npkts, D_OFF, b->stale_pkts ? D_STATUS : demux ? D_LEN : D_SLOT, true, s));
    caught_up(b, npkts);
    ring_is_up(b, ext);
    CK(ctx, order_kernels_begin(b));
    if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
    AeadArgs a = aead_args(b, npkts, true, nullptr);
    a.behind_kernel = true;
    const bool replay = (flags & BNK_F_REPLAY) != 0, one_launch = npkts <= kGroupMax;
    if (timed) CK(ctx, cudaEventRecord(b->a_begin, s));
    for (bool more = true; more;) {
        CK(ctx, copies.is_up());
        if (demux) CK(ctx, launch_demux_index(b, p.first, p.count, a.len, s));
        CK(ctx, launch_open(piece_args(a, p), s, ctx));
        CK(ctx, copies.down(p)); // the checks below say which plaintexts count, and change no byte of them
        more = pieces.next(p);
        if (more) CK(ctx, copies.up(p));
    }
    if (timed) CK(ctx, cudaEventRecord(b->a_end, s));
    if (replay && one_launch) {
        CK(ctx, launch_open_tail(b, npkts, true, nullptr, Done{}, s));
    } else if (replay) {
        CK(ctx, launch_group_by_slot(b, npkts, s));
        CK(ctx, launch_replay(b, npkts, s));
    }
    if (flags & BNK_F_INNER_CHECK) CK(ctx, launch_inner_check(b, npkts, s));
    if (flags & BNK_F_CHECK_INBOUND) {
        CK(ctx, flow_check_begins(b, now_unix_ns, s));
        CK(ctx, launch_filter_check(b, npkts, now_unix_ns, true, nullptr, Done{}, s));
    }
    if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
    b->kernel_timed = b->aead_timed = timed;
    CK(ctx, tally_if_asked(b, npkts, flags, s));
    CK(ctx, order_kernels_end(b));
    CK(ctx, desc_copy(b, npkts, demux ? D_SLOT : D_COUNTER, D_STATUS, false, s));
    CK(ctx, copies.join());
    return BNK_SUCCESS;
}

int bnk_open_submit(bnk_batch *b, uint32_t npkts, uint32_t flags, int64_t now_unix_ns) {
    const bool device_only = (flags & BNK_F_NO_H2D) && (flags & BNK_F_NO_D2H);
    int rc = begin_submit(b, npkts, !device_only);
    if (rc) return rc;
    SubmitScope scope(b);
    behind_heads(b, flags);
    bnk_ctx *ctx = b->ctx;
    cudaStream_t s = b->stream;
    const bool timed = (flags & BNK_F_TIMED) != 0;
    const size_t n = npkts;
    Layout lay;
    const uint64_t ext = device_only ? 0 : ring_extent(b, npkts, (flags & BNK_F_USE_OUT_LEN) || b->stale_pkts ? kMostRoom : 0, &lay);
    if (in_pieces(b, npkts, flags, ext, lay, true)) return open_pieces(b, npkts, ext, flags, now_unix_ns);
    if (ctx->aead_mode != 1 && host_direct(b, npkts, flags, ext)) return open_direct(b, npkts, lay, flags, now_unix_ns);
    // BNK_F_USE_OUT_LEN reads the lengths a seal left on the device: an upload beside it must not bring the
    // host's out_len along, so it moves the fields one by one instead of the whole slab.
    bool all;
    CK(ctx, catch_up_beside(b, npkts, !(flags & BNK_F_NO_H2D), !(flags & BNK_F_NO_D2H), s, all));
    if (!(flags & BNK_F_NO_H2D) && n) {
        const bool joint = b->joint_copy && (all || !(flags & BNK_F_USE_OUT_LEN));
        CK(ctx, ring_up(b, ext, joint, s));
        if (!joint) CK(ctx, desc_copy(b, n, D_OFF, all ? D_STATUS : (flags & BNK_F_DEMUX_INDEX) ? D_LEN : D_SLOT, true, s));
        caught_up(b, npkts);
    }
    CK(ctx, order_kernels_begin(b));
    if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
    const uint32_t *order = nullptr;
    AeadArgs oa = aead_args(b, npkts, true, nullptr);
    if (flags & BNK_F_USE_OUT_LEN) oa.len = b->dev.out_len;
    if (flags & BNK_F_DEMUX_INDEX) CK(ctx, launch_demux_index(b, 0, npkts, oa.len, s));
    if (flags & BNK_F_SORT_BY_LENGTH) {
        CK(ctx, launch_length_order(b, npkts, oa.len, true, s));
        order = b->dev.len_order;
    }
    oa.order = order;
    oa.behind_kernel = true;
    const bool replay = (flags & BNK_F_REPLAY) && n, one_launch = npkts <= kGroupMax;
    if (replay && !one_launch) {
        // grouping by keypair needs only the descriptors: it runs on the side stream beside the open kernel
        CK(ctx, cudaEventRecord(b->ev_fork, s));
        CK(ctx, cudaStreamWaitEvent(b->aux_stream, b->ev_fork, 0));
        CK(ctx, launch_group_by_slot(b, npkts, b->aux_stream));
        CK(ctx, cudaEventRecord(b->ev_join, b->aux_stream));
    }
    const bool side = b->aead_stream && npkts >= ctx->aead_side_stream_from;
    cudaStream_t as = side ? b->aead_stream : s;
    if (side) {
        CK(ctx, cudaEventRecord(b->ev_aead_go, s));
        CK(ctx, cudaStreamWaitEvent(as, b->ev_aead_go, 0));
    }
    if (timed) CK(ctx, cudaEventRecord(b->a_begin, as));
    CK(ctx, launch_open(oa, as, ctx));
    if (timed) CK(ctx, cudaEventRecord(b->a_end, as));
    if (side) {
        CK(ctx, cudaEventRecord(b->ev_aead_done, as));
        CK(ctx, cudaStreamWaitEvent(s, b->ev_aead_done, 0));
    }
    b->aead_timed = timed;
    if (replay && one_launch) {
        CK(ctx, launch_open_tail(b, npkts, true, nullptr, Done{}, s));
    } else if (replay) {
        CK(ctx, cudaStreamWaitEvent(s, b->ev_join, 0));
        CK(ctx, launch_replay(b, npkts, s));
    }
    if (flags & BNK_F_INNER_CHECK) CK(ctx, launch_inner_check(b, npkts, s));
    if (flags & BNK_F_CHECK_INBOUND) {
        CK(ctx, flow_check_begins(b, now_unix_ns, s));
        CK(ctx, launch_filter_check(b, npkts, now_unix_ns, true, nullptr, Done{}, s));
    }
    if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
    b->kernel_timed = timed;
    CK(ctx, tally_if_asked(b, npkts, flags, s));
    CK(ctx, order_kernels_end(b));
    if (!(flags & BNK_F_NO_D2H) && n) {
        if (b->joint_copy) {
            CK(ctx, ring_down(b, npkts, ext, true, s));
        } else {
            CK(ctx, ring_down(b, npkts, ext, false, s));
            CK(ctx, desc_copy(b, n, (flags & BNK_F_DEMUX_INDEX) ? D_SLOT : D_COUNTER, D_STATUS, false, s));
        }
    }
    return BNK_SUCCESS;
}

// What a call that looks at packet heads uploads when it does not work in place.  Descriptors first: how much of the ring
// is in use is known only after a pass over them, which a core does at ~20 GB/s out of memory, a third of a link's time
// with headers 48 bytes apart.  So each stretch of packets looked through sends up what it adds to the ring's extent
// while the next is looked through; pieces end on pages like those of a large batch.  (The highest byte only grows, so
// packets in any order are covered.)  900,000 headers checked 1337 us with the pass in front, 1023 so, of which the link
// needs 920 at 55 GB/s; 300,000 495 and 378, 30,000 69 and 58.
static int upload_heads(bnk_batch *b, uint32_t n, bool results_down, cudaStream_t s) {
    bnk_ctx *ctx = b->ctx;
    if (!results_down) CK(ctx, catch_up(b, s)); // (see catch_up_beside)
    CK(ctx, desc_copy(b, n, D_OFF, b->heads_go_up && results_down ? D_STATUS : D_LEN, true, s)); // (all that a catch-up would bring)
    uint64_t up = 0, ext = 0;
    for (uint32_t at = 0, k = kHeadsFirst; at < n; at += k, k = std::min(2 * k, kHeadsMost)) {
        k = std::min(k, n - at);
        const PacketScan r = scan_packets(b->host.off + at, b->host.len + at, k, 0);
        ext = std::max(ext, std::min<uint64_t>((r.end + kHeadSlack + 15) & ~15ull, b->ring_bytes));
        const uint64_t to = at + k < n ? ext & ~(kPage - 1) : ext;
        if (to > up) {
            CK(ctx, cudaMemcpyAsync(b->dev.ring + up, b->host.ring + up, to - up, cudaMemcpyHostToDevice, s));
            up = to;
        }
    }
    ring_is_up(b, up);
    return BNK_SUCCESS;
}

int bnk_filter_note_submit(bnk_batch *b, uint32_t npkts, uint32_t flags, int64_t now_unix_ns) {
    int rc = begin_submit(b, npkts);
    if (rc) return rc;
    CK(b->ctx, filter_flows_maintain(b, b->stream));
    SubmitScope scope(b);
    behind_heads(b, flags);
    bnk_ctx *ctx = b->ctx;
    cudaStream_t s = b->stream;
    const bool timed = (flags & BNK_F_TIMED) != 0;
    const bool upload = npkts && !(flags & BNK_F_NO_H2D);
    const bool direct = upload && heads_direct(b, npkts, flags);
    if (npkts && !upload) CK(ctx, catch_up(b, s));
    if (!direct && upload && (rc = upload_heads(b, npkts, true, s)) != BNK_SUCCESS) return rc;
    HostAlias alias(b, direct, npkts);
    if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
    const bool note = npkts && ctx->ft.enforce && ctx->ft.flow_capacity; // filter.go:192-194
    bool reported = false;
    if (note) {
        bool sweep;
        CK(ctx, flow_note_begins(b, npkts, now_unix_ns, s, sweep));
        const Done done = watch_for(b);
        Launches all(s, !timed && !sweep && through_graph(b));
        CK(ctx, launch_filter_note(b, 0, npkts, now_unix_ns, sweep ? Done{} : done, s));
        CK(ctx, send_launches(b, all));
        if (sweep) CK(ctx, launch_flow_sweep(b, now_unix_ns, done, s));
        reported = true;
    }
    if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
    b->kernel_timed = timed;
    if (!reported) CK(ctx, launch_flow_report(b, s));
    return BNK_SUCCESS;
}

int bnk_filter_check_submit(bnk_batch *b, uint32_t npkts, uint32_t flags, int64_t now_unix_ns) {
    int rc = begin_submit(b, npkts);
    if (rc) return rc;
    SubmitScope scope(b);
    behind_heads(b, flags);
    bnk_ctx *ctx = b->ctx;
    cudaStream_t s = b->stream;
    const bool timed = (flags & BNK_F_TIMED) != 0;
    const bool upload = npkts && !(flags & BNK_F_NO_H2D);
    const bool direct = upload && heads_direct(b, npkts, flags);
    if (npkts && !upload) CK(ctx, catch_up(b, s));
    if (!direct && upload && (rc = upload_heads(b, npkts, !(flags & BNK_F_NO_D2H), s)) != BNK_SUCCESS) return rc;
    HostAlias alias(b, direct, npkts);
    if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
    CK(ctx, flow_check_begins(b, now_unix_ns, s));
    const bool to_host = !(flags & BNK_F_NO_D2H);
    const Done done = to_host && npkts && !(flags & BNK_F_STATS) ? watch_for(b) : Done{};
    uint8_t *const host_status = to_host ? b->host.status : nullptr;
    if (direct) b->dev.status = alias.saved.status; // the kernel writes to both
    Launches all(s, !timed && through_graph(b));
    CK(ctx, launch_filter_check(b, npkts, now_unix_ns, false, host_status, done, s));
    CK(ctx, send_launches(b, all));
    if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
    b->kernel_timed = timed;
    CK(ctx, tally_if_asked(b, npkts, flags, s));
    return BNK_SUCCESS;
}

int bnk_classify_submit(bnk_batch *b, uint32_t npkts, uint32_t flags) {
    int rc = begin_submit(b, npkts);
    if (rc) return rc;
    SubmitScope scope(b);
    behind_heads(b, flags);
    bnk_ctx *ctx = b->ctx;
    cudaStream_t s = b->stream;
    const bool timed = (flags & BNK_F_TIMED) != 0;
    const size_t n = npkts;
    const bool upload = n && !(flags & BNK_F_NO_H2D);
    const bool direct = upload && heads_direct(b, npkts, flags);
    if (direct) b->stale_src = std::max(b->stale_src, npkts);
    if (npkts && !upload) CK(ctx, catch_up(b, s));
    if (!direct && upload) {
        if ((rc = upload_heads(b, npkts, !(flags & BNK_F_NO_D2H), s)) != BNK_SUCCESS) return rc;
        CK(ctx, cudaMemcpyAsync(b->dev.src_addr, b->host.src_addr, n * BNK_SRC_ADDR_STRIDE, cudaMemcpyHostToDevice, s));
    }
    HostAlias alias(b, direct, npkts);
    if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
    const Done done = direct && !(flags & BNK_F_STATS) ? watch_for(b) : Done{};
    Launches all(s, !timed && through_graph(b));
    CK(ctx, launch_classify(b, npkts, done, s));
    CK(ctx, send_launches(b, all));
    if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
    b->kernel_timed = timed;
    CK(ctx, tally_if_asked(b, npkts, flags, s));
    if (!direct && !(flags & BNK_F_NO_D2H) && n) {
        CK(ctx, cudaMemcpyAsync(b->host.slot, b->dev.slot, n * 4, cudaMemcpyDeviceToHost, s));
        CK(ctx, cudaMemcpyAsync(b->host.status, b->dev.status, n, cudaMemcpyDeviceToHost, s));
    }
    return BNK_SUCCESS;
}

constexpr uint32_t kPlainRuns = 16; // copies of plain packets between a split's segments
// Super-packets of up to kSplitInPlace bytes in all are read in place by the kernel that splits them: 120 segments of 1380 B
// split and sealed (two calls) 61.8 -> 47.4 us, 460 of 950 B 69.8 -> 57.3.  SMs read 48 GB/s over the link, the copy engine 55:
// 2400 of 1380 B (3.3 MB) 194.7 in place and 188.9 with a copy in front, 12,032 (17 MB) 768 and 733.  (In pieces, each split
// while the next comes up, 763: every piece costs the engine more than the split of all takes.)
// That kernel also brings up the packets that are no segments.  Up to kSplitWithPlain bytes with those it is ahead of their upload:
// two segments and 800 of 1420 B split 39 us and 53, 2500 (3.7 MB) 96 and 101, 5000 (7.3 MB) 170 and 168, 50,000 1506 and 1430;
// 40,000 of 64 B (4.5 MB, with 48 for each) 142 and 170.
constexpr uint64_t kSplitInPlace = 5ull << 19, kSplitWithPlain = 2 * kSplitInPlace;
int bnk_gso_split_submit(bnk_batch *b, const bnk_gso_super *supers, uint32_t n_super, uint32_t n_pkts,
                         uint32_t flags) {
    int rc = begin_submit(b, n_pkts, true); // the descriptor staging area is host memory in any case
    if (rc) return rc;
    SubmitScope scope(b);
    behind_heads(b, flags);
    bnk_ctx *ctx = b->ctx;
    cudaStream_t s = b->stream;
    const bool timed = (flags & BNK_F_TIMED) != 0;
    if (n_super > b->max_pkts || (n_super && !supers)) return fail(ctx, BNK_EINVAL, "bad super-packet list");
    const size_t n = n_pkts;
    const bool refresh = b->stale_pkts != 0;
    uint64_t ext = 0; // where the packets end, once they have been looked through
    CK(ctx, catch_up(b, s));
    if (!(flags & BNK_F_NO_H2D) && !refresh && gso_split_fits(supers, n_super, n_pkts, b->ring_bytes)) {
        uint64_t from = ~0ull, to = 0, sum = 0, segs = 0, of_segs = 0; // (bytes of segments, with their room)
        Layout all;
        for (uint32_t j = 0; j < n_super; j++) {
            from = std::min<uint64_t>(from, supers[j].src_off);
            to = std::max(to, (uint64_t)supers[j].src_off + supers[j].src_len);
            sum += supers[j].src_len;
            segs += supers[j].n_pkts;
            of_segs += supers[j].src_len - supers[j].hdr_len + supers[j].n_pkts * (uint64_t)(supers[j].hdr_len + kMostRoom);
        }
        from &= ~63ull;
        to = std::min<uint64_t>((to + 15) & ~15ull, b->ring_bytes);
        ext = ring_extent(b, n_pkts, kMostRoom, &all);
        const uint64_t over_link = sum + (segs < n_pkts && all.bytes > of_segs ? all.bytes - of_segs : 0);
        const bool in_place = sum <= kSplitInPlace && over_link <= kSplitWithPlain && host_direct(b, n_pkts, 0, over_link);
        if (in_place || (sum > kSplitInPlace && ctx->host_direct_bytes && segs == n_pkts && to - from <= 2 * sum + 65536)) {
            b->split_sealed = 0;
            b->partial_to = std::max({b->partial_to, ext, to});
            memcpy(b->h_gso, supers, (size_t)n_super * sizeof(bnk_gso_super));
            Launches all(s, in_place && !timed && through_graph(b));
            if (!in_place) { // the rest beside the copy
                CK(ctx, cudaEventRecord(b->ev_fork, s));
                CK(ctx, cudaStreamWaitEvent(b->aux_stream, b->ev_fork, 0));
                CK(ctx, cudaMemcpyAsync(b->dev.ring + from, b->host.ring + from, to - from, cudaMemcpyHostToDevice, s));
            }
            if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
            CK(ctx, launch_gso_prepare(b, n_super, n_pkts, in_place ? s : b->aux_stream));
            if (in_place) {
                CK(ctx, launch_gso_split_in_place(b, n_super, n_pkts, watch_for(b), s));
            } else {
                CK(ctx, cudaEventRecord(b->ev_join, b->aux_stream));
                CK(ctx, cudaStreamWaitEvent(s, b->ev_join, 0));
                CK(ctx, launch_gso_split_up(b, n_super, n_pkts, watch_for(b), s));
            }
            CK(ctx, send_launches(b, all));
            if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
            b->kernel_timed = timed;
            return BNK_SUCCESS;
        }
    }
    if (!(flags & BNK_F_NO_H2D) || refresh) {
        // The segments' slots are written on the device: of the ring only the super-packets have to go up, in one copy when
        // they lie close together, and the packets that are no super-packet's segments, each run of them in a copy of its
        // own.  (The whole ring goes up for a batch that is cut into many runs, whose plain packets are spread over most of
        // the ring, or whose super-packets are not in batch order.)
        uint64_t from = ~0ull, to = 0, sum = 0;
        if (ext == 0) ext = ring_extent(b, n_pkts, kMostRoom);
        struct {
            uint64_t at, to;
        } run[kPlainRuns];
        uint32_t runs = 0, next = 0; // packets below `next` are dealt with
        uint64_t plain_bytes = 0;
        bool whole = n_super == 0;
        auto plain_up_to = [&](uint32_t end) {
            if (next >= end || whole) return;
            uint64_t lo = ~0ull, hi = 0;
            for (uint32_t i = next; i < end; i++) {
                lo = std::min<uint64_t>(lo, b->host.off[i]);
                hi = std::max(hi, (uint64_t)b->host.off[i] + b->host.len[i] + 16 + 16 + 16);
            }
            lo &= ~63ull;
            hi = std::min<uint64_t>((hi + 15) & ~15ull, b->ring_bytes);
            if (lo >= hi) return;
            if (runs == kPlainRuns || (plain_bytes += hi - lo) > ext / 2) whole = true;
            else run[runs++] = {lo, hi};
        };
        for (uint32_t j = 0; j < n_super; j++) {
            const uint64_t at = supers[j].src_off, e = at + supers[j].src_len;
            if (e > b->ring_bytes) return fail(ctx, BNK_EINVAL, "super-packet lies outside the ring");
            if (at < from) from = at;
            if (e > to) to = e;
            sum += supers[j].src_len;
            if (supers[j].first_pkt < next) whole = true;
            plain_up_to(std::min(supers[j].first_pkt, n_pkts));
            next = (uint32_t)std::min<uint64_t>((uint64_t)supers[j].first_pkt + supers[j].n_pkts, n_pkts);
        }
        plain_up_to(n_pkts);
        from &= ~63ull;
        whole = whole || to - from > 2 * sum + 65536;
        b->split_sealed = 0;
        if (whole) {
            from = 0;
            if (to < ext) to = ext;
        }
        to = (to + 15) & ~15ull;
        if (to > b->ring_bytes) to = b->ring_bytes;
        if (whole) ring_is_up(b, to);
        else b->partial_to = std::max({b->partial_to, ext, to});
        if (to > from) CK(ctx, cudaMemcpyAsync(b->dev.ring + from, b->host.ring + from, to - from, cudaMemcpyHostToDevice, s));
        for (uint32_t k = 0; !whole && k < runs; k++)
            CK(ctx, cudaMemcpyAsync(b->dev.ring + run[k].at, b->host.ring + run[k].at, run[k].to - run[k].at, cudaMemcpyHostToDevice, s));
        if (n) CK(ctx, desc_copy(b, n, D_OFF, D_SLOT, true, s));
    }
    if (n_super) {
        memcpy(b->h_gso, supers, (size_t)n_super * sizeof(bnk_gso_super));
        CK(ctx, cudaMemcpyAsync(b->dev.gso, b->h_gso, (size_t)n_super * sizeof(bnk_gso_super), cudaMemcpyHostToDevice, s));
    }
    if (timed) CK(ctx, cudaEventRecord(b->k_begin, s));
    CK(ctx, launch_gso_split(b, n_super, n_pkts, s));
    if (timed) CK(ctx, cudaEventRecord(b->k_end, s));
    b->kernel_timed = timed;
    return BNK_SUCCESS;
}

// Watches the word that the submit's last kernel stores.  Like the driver's own wait it keeps the core; after
// ~200 us, or if the word does not come because the work failed, the driver's wait takes over.
static bool done_seen(bnk_batch *b, uint64_t timeout_ns) {
    if (!b->done_watched) return false;
    const volatile uint32_t *word = b->h_done;
    const uint64_t turns = timeout_ns / 64 < 4096 ? timeout_ns / 64 : 4096; // a turn is at least ~40 ns
    for (uint32_t i = 0; *word != b->done_seq; i++) {
        if (i >= turns) return false;
        cpu_relax();
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    return true;
}

int bnk_wait(bnk_batch *b, uint64_t timeout_ns) {
    if (!b) return BNK_EINVAL;
    if (!b->in_flight) return BNK_SUCCESS;
    bnk_ctx *ctx = b->ctx;
    if (!done_seen(b, timeout_ns)) {
        if (b->done_watched && timeout_ns == 0 && (++b->done_polls & 63u)) return BNK_ETIMEDOUT; // ask the driver now and then
        CK(ctx, cudaSetDevice(ctx->device));
        if (timeout_ns == UINT64_MAX) {
            CK(ctx, cudaStreamSynchronize(b->order.run));
        } else {
            const auto deadline = std::chrono::steady_clock::now() + std::chrono::nanoseconds(timeout_ns);
            for (;;) {
                cudaError_t e = cudaStreamQuery(b->order.run);
                if (e == cudaSuccess) break;
                if (e != cudaErrorNotReady) return fail(ctx, BNK_ECUDA, "cudaStreamQuery", e);
                if (std::chrono::steady_clock::now() >= deadline) return BNK_ETIMEDOUT;
                std::this_thread::yield();
            }
        }
    }
    submit_over(b);
    if (b->flow_work.on) ctx->flow_bounds.over(b->flow_work, b->flow_reported ? b->h_flow : nullptr);
    if (b->flow_reported) { // what the device said about the flow table after this batch: input of the next compaction
        b->flow_reported = false;
        for (int c = 0; c < 3; c++) ctx->flow_dead_hint[c] = b->h_flow->dead[c];
        int seen = ctx->flow_errors_seen.load();
        const int now_failed = b->h_flow->error;
        while (now_failed > seen && !ctx->flow_errors_seen.compare_exchange_weak(seen, now_failed)) {}
        if (now_failed > seen) return fail(ctx, BNK_EFULL, "flow table full: some outbound flows were not recorded");
    }
    return BNK_SUCCESS;
}

int bnk_batch_stats_get(bnk_batch *b, bnk_batch_stats *out) {
    if (!b || !out) return BNK_EINVAL;
    if (b->in_flight) return fail(b->ctx, BNK_EBUSY, "batch has work in flight; call bnk_wait first");
    if (!b->stats_pending) return fail(b->ctx, BNK_EINVAL, "the batch's last submit was not made with BNK_F_STATS");
    *out = *b->h_stats;
    return BNK_SUCCESS;
}

/* ---- stage timing ---- */
int bnk_batch_last_kernel_ms(bnk_batch *b, float *ms) {
    if (!b || !ms) return BNK_EINVAL;
    if (!b->kernel_timed) return fail(b->ctx, BNK_EINVAL, "no submit has been timed on this batch");
    CK(b->ctx, cudaSetDevice(b->ctx->device));
    CK(b->ctx, cudaEventSynchronize(b->k_end));
    CK(b->ctx, cudaEventElapsedTime(ms, b->k_begin, b->k_end));
    return BNK_SUCCESS;
}

int bnk_batch_last_aead_ms(bnk_batch *b, float *ms) {
    if (!b || !ms) return BNK_EINVAL;
    if (!b->aead_timed) return fail(b->ctx, BNK_EINVAL, "no seal/open has been submitted on this batch");
    CK(b->ctx, cudaSetDevice(b->ctx->device));
    CK(b->ctx, cudaEventSynchronize(b->a_end));
    CK(b->ctx, cudaEventElapsedTime(ms, b->a_begin, b->a_end));
    return BNK_SUCCESS;
}

int bnk_kernel_launch_count(bnk_ctx *ctx, uint64_t *count) {
    if (!ctx || !count) return BNK_EINVAL;
    *count = ctx->launches.load();
    return BNK_SUCCESS;
}

int bnk_graph_launch_count(bnk_ctx *ctx, uint64_t *count) {
    if (!ctx || !count) return BNK_EINVAL;
    *count = ctx->graph_launches.load();
    return BNK_SUCCESS;
}

} // extern "C"
