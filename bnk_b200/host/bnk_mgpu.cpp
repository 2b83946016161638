// Several GPUs behind one entry point: placement of peers by measured load and a dispatcher that routes mixed
// batches to per-GPU contexts (declared in include/bnk_gpu.h).  Host code only; every packet decision is made by
// the kernels behind bnk_seal_submit / bnk_open_submit of the GPU a packet is routed to.
//
// Why peers and nothing finer: the send counter hands out consecutive nonces per peer in batch order and the
// replay window is a sequential walk per peer, so a peer's packets must meet in one context; flows are keyed by
// the peer's tunnel address (one /32 per peer, internal/dataplane/engine.go:294 of the reference) and stay with
// it.  The rule table is read-only per packet and is replicated.  GPUs therefore never exchange packet data.
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <new>
#include <queue>
#include <string>
#include <thread>
#include <vector>

#include "../../include/bnk_gpu.h"
#include "../csrc/packet_copy.h"
#include "../csrc/submit_order.h"
#include "crew.h"

extern "C" int bnk_place_peers(const uint64_t *load, uint32_t n_peers, uint32_t n_gpus, uint32_t max_per_gpu,
                               uint32_t *gpu_of, uint32_t *slot_of, uint64_t *load_per_gpu) {
    if (!gpu_of || !slot_of || n_gpus == 0) return BNK_EINVAL;
    if ((uint64_t)n_gpus * max_per_gpu < n_peers) return BNK_EFULL;
    std::vector<uint32_t> order(n_peers);
    for (uint32_t p = 0; p < n_peers; p++) order[p] = p;
    if (load)
        std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return load[a] > load[b]; });
    // Longest processing time first.  Every peer weighs its load plus one, so that the many peers that carried
    // nothing in the measured period still spread evenly instead of piling onto the lightest GPU.
    struct Gpu {
        uint64_t weight;
        uint32_t count, id;
    };
    auto heavier = [](const Gpu &a, const Gpu &b) { // priority_queue keeps the largest on top: invert
        if (a.weight != b.weight) return a.weight > b.weight;
        if (a.count != b.count) return a.count > b.count;
        return a.id > b.id;
    };
    std::priority_queue<Gpu, std::vector<Gpu>, decltype(heavier)> heap(heavier);
    for (uint32_t g = 0; g < n_gpus; g++) heap.push(Gpu{0, 0, g});
    std::vector<uint64_t> carried(n_gpus, 0);
    for (uint32_t p : order) {
        Gpu g = heap.top();
        heap.pop();
        gpu_of[p] = g.id;
        slot_of[p] = g.count;
        const uint64_t l = load ? load[p] : 0;
        carried[g.id] += l;
        g.weight += l + 1;
        g.count++;
        if (g.count < max_per_gpu) heap.push(g); // a full GPU takes no more peers
    }
    if (load_per_gpu)
        for (uint32_t g = 0; g < n_gpus; g++) load_per_gpu[g] = carried[g];
    return BNK_SUCCESS;
}

namespace {

using namespace crew;

constexpr uint32_t kNoPeer = 0xffffffffu;

struct PeerInfo {
    bool set = false;
    uint32_t local_index = 0;
};

// Receiver index -> peer, looked up once per message of a batch: a flat table of index << 32 | peer + 1, linear probing,
// at most half full, deletions by moving the chain behind up.
class IndexTable {
  public:
    void Init(uint32_t peers) {
        uint64_t n = 16;
        while (n < 4ull * peers) n <<= 1;
        slots_.assign(n, 0);
    }
    uint32_t Find(uint32_t index) const { // kNoPeer when it is not there
        for (size_t h = At(index);; h = (h + 1) & (slots_.size() - 1)) {
            if (slots_[h] == 0) return kNoPeer;
            if ((uint32_t)(slots_[h] >> 32) == index) return (uint32_t)slots_[h] - 1;
        }
    }
    void Set(uint32_t index, uint32_t peer) { // not in the table
        size_t h = At(index);
        while (slots_[h]) h = (h + 1) & (slots_.size() - 1);
        slots_[h] = ((uint64_t)index << 32) | (peer + 1);
    }
    void Erase(uint32_t index) {
        const size_t mask = slots_.size() - 1;
        size_t h = At(index);
        while (slots_[h] && (uint32_t)(slots_[h] >> 32) != index) h = (h + 1) & mask;
        if (!slots_[h]) return;
        for (size_t q = (h + 1) & mask; slots_[q]; q = (q + 1) & mask) {
            const size_t home = At((uint32_t)(slots_[q] >> 32));
            if (((q - home) & mask) >= ((q - h) & mask)) { // its chain starts at or before the hole
                slots_[h] = slots_[q];
                h = q;
            }
        }
        slots_[h] = 0;
    }

  private:
    size_t At(uint32_t index) const { return (size_t)(index * 0x9e3779b1u ^ index >> 15) & (slots_.size() - 1); }
    std::vector<uint64_t> slots_;
};

} // namespace

struct bnk_mgpu {
    bnk_mgpu_cfg cfg;
    uint32_t slot_bytes;
    std::vector<bnk_ctx *> ctx;
    uint32_t piece; // packets per piece of a share
    std::vector<std::vector<bnk_batch *>> batch; // [gpu][Share::kSlots]
    std::vector<std::vector<bnk_batch_view>> view;
    std::vector<cudaStream_t> stream; // [gpu] of the pieces that stay in pinned memory
    std::vector<bnk_batch *> last; // [gpu] batch of the submit that the next one's kernels have to follow
    std::vector<std::unique_ptr<Worker>> worker;
    std::vector<std::unique_ptr<Crew>> helpers;
    std::vector<uint32_t> gpu_of, slot_of;
    std::vector<PeerInfo> peer;
    IndexTable peer_of_index; // receiver index -> peer
    std::vector<uint64_t> pkts_per_peer, bytes_per_peer, pkts_per_gpu;
    uint32_t peers_set = 0;
    std::mutex mu; // one call at a time: per-peer order is the order of the calls
    std::string last_error;
};

namespace {

int mfail(bnk_mgpu *m, int code, const std::string &what) {
    if (m) m->last_error = what;
    return code;
}

constexpr uint32_t kShareFrom = 2048; // packets; fewer are looked at sooner than a helper wakes up

// Runs f(first, last) over a call's n packets, with the helpers when there are many.
template <typename F>
void over_packets(bnk_mgpu *m, uint32_t n, F f) {
    if (n < kShareFrom) return f(0, n);
    Stretches all(n, f);
    m->helpers[0]->Do(all);
}

// Per-GPU lists of packet numbers in batch order (stable: a peer's packets keep their order), and what every peer carries.
// Returns the bytes.
uint64_t route(bnk_mgpu *m, const std::vector<uint32_t> &peer_of_pkt, const uint32_t *len, std::vector<std::vector<uint32_t>> &lists) {
    const uint32_t ng = (uint32_t)m->ctx.size(), n = (uint32_t)peer_of_pkt.size();
    lists.assign(ng, {});
    for (std::vector<uint32_t> &l : lists) l.reserve(n / ng + n / 8);
    uint64_t bytes = 0;
    for (uint32_t i = 0; i < n; i++) {
        const uint32_t p = peer_of_pkt[i];
        if (p == kNoPeer) continue;
        lists[m->gpu_of[p]].push_back(i);
        m->pkts_per_peer[p]++;
        m->bytes_per_peer[p] += len[i];
        bytes += len[i];
    }
    return bytes;
}

} // namespace

extern "C" {

const char *bnk_mgpu_last_error_string(bnk_mgpu *m) { return m ? m->last_error.c_str() : "null dispatcher"; }

int bnk_mgpu_destroy(bnk_mgpu *m) {
    if (!m) return BNK_EINVAL;
    m->worker.clear(); // joins the threads
    m->helpers.clear();
    for (std::vector<bnk_batch *> &of_gpu : m->batch)
        for (bnk_batch *b : of_gpu)
            if (b) bnk_batch_destroy(b);
    for (cudaStream_t s : m->stream)
        if (s) cudaStreamDestroy(s);
    for (bnk_ctx *c : m->ctx)
        if (c) bnk_ctx_destroy(c);
    delete m;
    return BNK_SUCCESS;
}

static int build(bnk_mgpu *m, const bnk_mgpu_cfg *cfg) {
    m->cfg = *cfg;
    m->cfg.devices = nullptr;
    m->slot_bytes = (16u + ((cfg->max_packet + 15u) & ~15u) + 16u + 15u) & ~15u;
    const uint32_t ng = cfg->n_devices;
    // A piece is about three megabytes of ring: the GPU then works ~100 us on it, and two of them may stay in pinned memory.
    m->piece = std::min(cfg->max_pkts_per_gpu, std::min(2048u, std::max(64u, (3u << 20) / m->slot_bytes)));
    const uint32_t cores = std::max(1u, std::thread::hardware_concurrency());
    const uint32_t n_helpers = std::min(8u, cores / ng > 1 ? cores / ng - 1 : 0u); // 24,576 x 1420 B sealed and opened: 4.9 ms with 4, 4.1 with 6, 3.8 with 8, 3.6 with 14
    m->ctx.assign(ng, nullptr);
    m->batch.assign(ng, std::vector<bnk_batch *>(Share::kSlots, nullptr));
    m->view.assign(ng, std::vector<bnk_batch_view>(Share::kSlots));
    m->stream.assign(ng, nullptr);
    m->last.assign(ng, nullptr);
    m->peer_of_index.Init(cfg->max_peers);
    m->pkts_per_gpu.assign(ng, 0);
    for (uint32_t g = 0; g < ng; g++) {
        bnk_cfg c = cfg->ctx;
        c.struct_size = sizeof c;
        c.device_id = cfg->devices[g];
        int rc = bnk_ctx_create(&c, &m->ctx[g]);
        if (rc == BNK_SUCCESS && order_stream_create(m->ctx[g], &m->stream[g]) != cudaSuccess) rc = BNK_ECUDA;
        for (uint32_t k = 0; k < Share::kSlots; k++) {
            if (rc == BNK_SUCCESS) rc = bnk_batch_create(m->ctx[g], m->piece, (uint64_t)m->piece * m->slot_bytes, &m->batch[g][k]);
            if (rc == BNK_SUCCESS) rc = bnk_batch_view_get(m->batch[g][k], &m->view[g][k]);
            if (rc == BNK_SUCCESS) batch_set_direct_stream(m->batch[g][k], m->stream[g]);
        }
        if (rc != BNK_SUCCESS) return rc;
        m->worker.push_back(std::make_unique<Worker>());
        m->helpers.push_back(std::make_unique<Crew>(n_helpers));
    }
    m->gpu_of.assign(cfg->max_peers, 0);
    m->slot_of.assign(cfg->max_peers, 0);
    m->peer.assign(cfg->max_peers, PeerInfo{});
    m->pkts_per_peer.assign(cfg->max_peers, 0);
    m->bytes_per_peer.assign(cfg->max_peers, 0);
    return bnk_place_peers(nullptr, cfg->max_peers, ng, cfg->ctx.max_keypairs, m->gpu_of.data(), m->slot_of.data(), nullptr);
}

int bnk_mgpu_create(const bnk_mgpu_cfg *cfg, bnk_mgpu **out) {
    if (!cfg || !out || cfg->struct_size != sizeof(bnk_mgpu_cfg) || cfg->n_devices == 0 || !cfg->devices ||
        cfg->max_pkts_per_gpu == 0 || cfg->max_peers == 0 || cfg->max_packet == 0)
        return BNK_EINVAL;
    *out = nullptr;
    if ((uint64_t)cfg->n_devices * cfg->ctx.max_keypairs < cfg->max_peers) return BNK_EINVAL;
    bnk_mgpu *m = new (std::nothrow) bnk_mgpu();
    if (!m) return BNK_ENOMEM;
    try {
        const int rc = build(m, cfg);
        if (rc == BNK_SUCCESS) *out = m;
        else bnk_mgpu_destroy(m);
        return rc;
    } catch (const std::exception &) { // no memory or no thread
        bnk_mgpu_destroy(m);
        return BNK_ENOMEM;
    }
}

bnk_ctx *bnk_mgpu_ctx(bnk_mgpu *m, uint32_t g) { return (m && g < m->ctx.size()) ? m->ctx[g] : nullptr; }

int bnk_mgpu_place(bnk_mgpu *m, const uint64_t *load) {
    if (!m) return BNK_EINVAL;
    std::lock_guard<std::mutex> g(m->mu);
    if (m->peers_set) return mfail(m, BNK_EBUSY, "peers are set: remove them before placing anew (a live peer moves with its next keypair)");
    return bnk_place_peers(load, m->cfg.max_peers, (uint32_t)m->ctx.size(), m->cfg.ctx.max_keypairs, m->gpu_of.data(),
                           m->slot_of.data(), nullptr);
}

int bnk_mgpu_locate(bnk_mgpu *m, uint32_t peer, uint32_t *gpu, uint32_t *slot) {
    if (!m || peer >= m->cfg.max_peers) return BNK_EINVAL;
    if (gpu) *gpu = m->gpu_of[peer];
    if (slot) *slot = m->slot_of[peer];
    return BNK_SUCCESS;
}

int bnk_mgpu_peer_clear(bnk_mgpu *m, uint32_t peer) {
    if (!m || peer >= m->cfg.max_peers) return BNK_EINVAL;
    std::lock_guard<std::mutex> g(m->mu);
    PeerInfo &pi = m->peer[peer];
    if (!pi.set) return BNK_SUCCESS;
    bnk_ctx *c = m->ctx[m->gpu_of[peer]];
    int rc = bnk_index_clear(c, pi.local_index);
    if (rc == BNK_SUCCESS) rc = bnk_keypair_clear(c, m->slot_of[peer]);
    if (rc != BNK_SUCCESS) return mfail(m, rc, bnk_last_error_string(c));
    m->peer_of_index.Erase(pi.local_index);
    pi.set = false;
    m->peers_set--;
    return BNK_SUCCESS;
}

int bnk_mgpu_peer_set(bnk_mgpu *m, uint32_t peer, const uint8_t send_key[32], const uint8_t recv_key[32],
                      uint32_t remote_index, uint32_t local_index, uint32_t allowed_ipv4) {
    if (!m || peer >= m->cfg.max_peers || !send_key || !recv_key) return BNK_EINVAL;
    int rc = bnk_mgpu_peer_clear(m, peer);
    if (rc != BNK_SUCCESS) return rc;
    std::lock_guard<std::mutex> g(m->mu);
    if (m->peer_of_index.Find(local_index) != kNoPeer) return mfail(m, BNK_EINVAL, "receiver index already belongs to another peer");
    bnk_ctx *c = m->ctx[m->gpu_of[peer]];
    const uint32_t slot = m->slot_of[peer];
    rc = bnk_keypair_set(c, slot, send_key, recv_key, remote_index);
    if (rc == BNK_SUCCESS) rc = bnk_keypair_set_allowed_ip(c, slot, allowed_ipv4);
    if (rc == BNK_SUCCESS) rc = bnk_index_set(c, local_index, slot);
    if (rc != BNK_SUCCESS) return mfail(m, rc, bnk_last_error_string(c));
    m->peer[peer].set = true;
    m->peer[peer].local_index = local_index;
    m->peer_of_index.Set(local_index, peer);
    m->peers_set++;
    return BNK_SUCCESS;
}

int bnk_mgpu_acl_set(bnk_mgpu *m, int enforce, const bnk_acl_tuple *tuples, size_t n) {
    if (!m) return BNK_EINVAL;
    for (bnk_ctx *c : m->ctx) {
        const int rc = bnk_acl_set(c, enforce, tuples, n);
        if (rc != BNK_SUCCESS) return mfail(m, rc, bnk_last_error_string(c));
    }
    return BNK_SUCCESS;
}

int bnk_mgpu_loads_get(bnk_mgpu *m, uint64_t *packets_per_peer, uint64_t *bytes_per_peer, uint64_t *packets_per_gpu,
                       int reset) {
    if (!m) return BNK_EINVAL;
    std::lock_guard<std::mutex> g(m->mu);
    if (packets_per_peer) memcpy(packets_per_peer, m->pkts_per_peer.data(), m->pkts_per_peer.size() * 8);
    if (bytes_per_peer) memcpy(bytes_per_peer, m->bytes_per_peer.data(), m->bytes_per_peer.size() * 8);
    if (packets_per_gpu) memcpy(packets_per_gpu, m->pkts_per_gpu.data(), m->pkts_per_gpu.size() * 8);
    if (reset) {
        std::fill(m->pkts_per_peer.begin(), m->pkts_per_peer.end(), 0);
        std::fill(m->bytes_per_peer.begin(), m->bytes_per_peer.end(), 0);
    }
    return BNK_SUCCESS;
}

// The two data calls share their shape: route, one share per GPU (fill a pinned ring, submit, wait, copy out, piece by
// piece), wait for all shares.  `in` and `out` move packet i of the call into and out of entry k of a batch; packet j is
// the next one (for entry k + 1).
using Mover = std::function<void(const bnk_batch_view &v, uint32_t k, uint32_t i, uint32_t j)>;
static int run_shares(bnk_mgpu *m, const std::vector<std::vector<uint32_t>> &lists, uint64_t bytes,
                      const Mover &in,
                      const std::function<int(bnk_batch *b, uint32_t cnt)> &submit,
                      const Mover &out) {
    const uint32_t ng = (uint32_t)m->ctx.size();
    int busy = 0;
    for (uint32_t g = 0; g < ng; g++) busy += !lists[g].empty();
    if (busy == 0) return BNK_SUCCESS;
    // The calling thread takes the last busy GPU itself: with one busy GPU (a small batch, a single-GPU box)
    // nothing is handed to another thread at all, and otherwise the caller works instead of sleeping.
    uint32_t own = 0;
    for (uint32_t g = 0; g < ng; g++)
        if (!lists[g].empty()) own = g;
    Latch latch(busy - 1);
    std::vector<int> rcs(ng, BNK_SUCCESS);
    auto work = [&](uint32_t g) {
        const std::vector<uint32_t> &l = lists[g];
        const uint32_t n = (uint32_t)l.size();
        m->last[g] = nullptr; // nothing is in flight between calls
        // Four pieces at least, of 256 packets at least: fewer leave nothing to overlap, smaller ones are all launch.
        Share s(n, std::min(m->piece, std::max(256u, (n + 3) / 4)));
        s.in = [&](uint32_t slot, uint32_t at, uint32_t first, uint32_t cnt) {
            for (uint32_t k = 0; k < cnt; k++) in(m->view[g][slot], at + k, l[first + k], l[first + std::min(k + 1, cnt - 1)]);
        };
        s.out = [&](uint32_t slot, uint32_t at, uint32_t first, uint32_t cnt) {
            for (uint32_t k = 0; k < cnt; k++) out(m->view[g][slot], at + k, l[first + k], l[first + std::min(k + 1, cnt - 1)]);
        };
        s.submit = [&](uint32_t slot, uint32_t, uint32_t cnt) {
            const int rc = submit_behind(m->batch[g][slot], m->last[g], [&] { return submit(m->batch[g][slot], cnt); });
            m->last[g] = m->batch[g][slot];
            return rc;
        };
        s.poll = [&](uint32_t slot) { return bnk_wait(m->batch[g][slot], 0); };
        // waking the helpers takes longer than copying half a megabyte
        rcs[g] = bytes / (uint32_t)busy < (512u << 10) ? s.Drive() : m->helpers[g]->Do(s);
    };
    auto job = [&](uint32_t g) {
        try {
            work(g);
        } catch (const std::exception &) { // no memory, before anything was submitted
            rcs[g] = BNK_ENOMEM;
        }
    };
    for (uint32_t g = 0; g < ng; g++) {
        if (lists[g].empty()) continue;
        m->pkts_per_gpu[g] += lists[g].size();
        if (g == own) continue;
        try {
            m->worker[g]->Post([&, g] {
                job(g);
                latch.Done();
            });
        } catch (const std::exception &) {
            rcs[g] = BNK_ENOMEM;
            latch.Done();
        }
    }
    job(own);
    latch.Wait();
    for (uint32_t g = 0; g < ng; g++)
        if (rcs[g] != BNK_SUCCESS) return mfail(m, rcs[g], bnk_last_error_string(m->ctx[g]));
    return BNK_SUCCESS;
}

int bnk_mgpu_seal(bnk_mgpu *m, const uint8_t *const *pkts, const uint32_t *len, const uint32_t *peer, uint32_t n,
                  uint32_t flags, int64_t now_unix_ns, uint8_t *const *out, uint32_t *out_len, uint64_t *counter,
                  uint8_t *status) try {
    if (!m || (n && (!pkts || !len || !peer || !out || !out_len || !status))) return BNK_EINVAL;
    std::lock_guard<std::mutex> guard(m->mu);
    std::vector<uint32_t> peer_of_pkt(n);
    over_packets(m, n, [&](uint32_t first, uint32_t last) {
        for (uint32_t i = first; i < last; i++) {
            const uint32_t p = peer[i];
            const bool known = p < m->cfg.max_peers && m->peer[p].set, fits = len[i] <= m->cfg.max_packet;
            peer_of_pkt[i] = known && fits ? p : kNoPeer;
            if (known && fits) continue;
            status[i] = known ? BNK_PKT_BAD_DESC : BNK_PKT_NO_KEYPAIR;
            out_len[i] = 0;
        }
    });
    std::vector<std::vector<uint32_t>> lists;
    const uint64_t bytes = route(m, peer_of_pkt, len, lists);
    const uint32_t f = (flags | BNK_F_ASSIGN_COUNTERS) & ~(BNK_F_NO_H2D | BNK_F_NO_D2H | BNK_F_USE_OUT_LEN);
    return run_shares(
        m, lists, bytes,
        [&](const bnk_batch_view &v, uint32_t k, uint32_t i, uint32_t j) {
            v.off[k] = k * m->slot_bytes;
            v.len[k] = len[i];
            v.slot[k] = m->slot_of[peer[i]];
            if (j != i) copy_comes_next(pkts[j], v.ring + (size_t)(k + 1) * m->slot_bytes + 16, len[j]);
            if (len[i]) memcpy(v.ring + (size_t)k * m->slot_bytes + 16, pkts[i], len[i]);
        },
        [&](bnk_batch *b, uint32_t cnt) { return bnk_seal_submit(b, cnt, f, now_unix_ns); },
        [&](const bnk_batch_view &v, uint32_t k, uint32_t i, uint32_t j) {
            status[i] = v.status[k];
            out_len[i] = v.out_len[k];
            if (counter) counter[i] = v.counter[k];
            if (j != i) copy_comes_next(v.ring + (size_t)(k + 1) * m->slot_bytes, out[j], v.out_len[k + 1]);
            if (v.out_len[k]) memcpy(out[i], v.ring + (size_t)k * m->slot_bytes, v.out_len[k]);
        });
} catch (const std::exception &) { // no memory
    return BNK_ENOMEM;
}

int bnk_mgpu_open(bnk_mgpu *m, const uint8_t *const *msgs, const uint32_t *len, uint32_t n, uint32_t flags,
                  int64_t now_unix_ns, uint8_t *const *out, uint32_t *out_len, uint64_t *counter, uint32_t *peer_out,
                  uint8_t *status) try {
    if (!m || (n && (!msgs || !len || !out || !out_len || !status))) return BNK_EINVAL;
    std::lock_guard<std::mutex> guard(m->mu);
    std::vector<uint32_t> peer_of_pkt(n, kNoPeer);
    // The headers lie in memory of the caller's, each a cache miss of its own: reading 24,576 of them on one thread, before
    // the helpers had anything to copy, made 1.94 ms out of the 1.65 that the call takes.
    constexpr uint32_t kPrefetch = 16;
    over_packets(m, n, [&](uint32_t first, uint32_t last) {
    for (uint32_t i = first; i < last; i++) {
        if (i + kPrefetch < last) __builtin_prefetch(msgs[i + kPrefetch]);
        out_len[i] = 0;
        if (peer_out) peer_out[i] = kNoPeer;
        if (len[i] < BNK_WG_HEADER + BNK_WG_TAG || (uint64_t)len[i] > (uint64_t)m->cfg.max_packet + 32u) {
            status[i] = BNK_PKT_MALFORMED;
            continue;
        }
        uint32_t type, index;
        memcpy(&type, msgs[i], 4);
        memcpy(&index, msgs[i] + 4, 4); // little-endian hosts only, like the rest of the library
        if (type != 4u) {
            status[i] = BNK_PKT_MALFORMED;
            continue;
        }
        const uint32_t p = m->peer_of_index.Find(index);
        if (p == kNoPeer) {
            status[i] = BNK_PKT_NO_KEYPAIR;
            continue;
        }
        peer_of_pkt[i] = p;
        if (peer_out) peer_out[i] = p;
    }
    });
    std::vector<std::vector<uint32_t>> lists;
    const uint64_t bytes = route(m, peer_of_pkt, len, lists);
    const uint32_t f = flags & ~(BNK_F_NO_H2D | BNK_F_NO_D2H | BNK_F_USE_OUT_LEN | BNK_F_DEMUX_INDEX);
    return run_shares(
        m, lists, bytes,
        [&](const bnk_batch_view &v, uint32_t k, uint32_t i, uint32_t j) {
            v.off[k] = k * m->slot_bytes;
            v.len[k] = len[i];
            v.slot[k] = m->slot_of[peer_of_pkt[i]];
            if (j != i) copy_comes_next(msgs[j], v.ring + (size_t)(k + 1) * m->slot_bytes, len[j]);
            memcpy(v.ring + (size_t)k * m->slot_bytes, msgs[i], len[i]);
        },
        [&](bnk_batch *b, uint32_t cnt) { return bnk_open_submit(b, cnt, f, now_unix_ns); },
        [&](const bnk_batch_view &v, uint32_t k, uint32_t i, uint32_t j) {
            // only what passed leaves the library: a replayed, filtered or otherwise refused packet yields no bytes
            const bool pass = v.status[k] == BNK_PKT_OK || v.status[k] == BNK_PKT_KEEPALIVE;
            status[i] = v.status[k];
            out_len[i] = pass ? v.out_len[k] : 0u;
            if (counter) counter[i] = v.counter[k];
            if (j != i) copy_comes_next(v.ring + (size_t)(k + 1) * m->slot_bytes, out[j], v.out_len[k + 1]);
            if (out_len[i]) memcpy(out[i], v.ring + (size_t)k * m->slot_bytes + 16, out_len[i]);
        });
} catch (const std::exception &) {
    return BNK_ENOMEM;
}

} // extern "C"
