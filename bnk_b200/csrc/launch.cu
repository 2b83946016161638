// Launches and their graphs (launch.h).
#include "launch.h"

#include <string.h>

#include <atomic>
#include <mutex>
#include <new>

namespace {

thread_local Launches *t_gathering = nullptr;

cudaError_t launch_now(const LaunchShape &k, void *const *args, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = k.grid;
    cfg.blockDim = k.block;
    cfg.dynamicSmemBytes = k.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (k.behind) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (k.cluster > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = k.cluster;
        attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
        cfg.numAttrs++;
    }
    return cudaLaunchKernelExC(&cfg, k.fn, const_cast<void **>(args));
}

} // namespace

// What a graph cannot change: its kernels, their clusters, whether the second is a dependent launch.
struct LaunchGraph {
    uint32_t n;
    const void *fn[2];
    uint32_t cluster[2];
    bool behind;
    bool taken;
    int device;
    cudaGraphExec_t exec;
    cudaGraph_t graph;
    cudaGraphNode_t node[2];
    bool is(const LaunchGraph &o) const {
        return n == o.n && fn[0] == o.fn[0] && fn[1] == o.fn[1] && cluster[0] == o.cluster[0] && cluster[1] == o.cluster[1] && behind == o.behind;
    }
};

namespace {

// The graphs of one device, used by all its contexts.  A graph belongs to one submit at a time, from its launch until that
// has been waited for.  One is made (50 us, 250 for two kernels, 100 KB) when its kernels are asked for the fourth time and
// none is free, so that a program that calls once or twice does not pay for it.  What is kept here is kept in place: a submit
// of a process without memory to spare goes launch by launch.
class GraphPool {
  public:
    LaunchGraph *take(const LaunchGraph &want) {
        std::lock_guard<std::mutex> g(mu_);
        for (uint32_t i = 0; i < made_n_; i++)
            if (!made_[i]->taken && made_[i]->is(want)) {
                made_[i]->taken = true;
                return made_[i];
            }
        if (made_n_ + making_ >= kMost) return nullptr;
        if (Asked *a = asked(want)) {
            if (++a->times < kFrom) return nullptr;
            making_++;
            return &make_;
        }
        if (asked_n_ < kMostAsked) asked_[asked_n_++] = {want, 1};
        return nullptr;
    }
    static bool to_be_made(const LaunchGraph *g) { return g == &make_; }
    void made(LaunchGraph *g) { // null: it could not be
        std::lock_guard<std::mutex> l(mu_);
        making_--;
        if (g) made_[made_n_++] = g;
    }
    void failed(const LaunchGraph &want) { // not again
        std::lock_guard<std::mutex> l(mu_);
        if (Asked *a = asked(want)) a->times = INT32_MIN;
    }
    void give(LaunchGraph *g) {
        std::lock_guard<std::mutex> l(mu_);
        g->taken = false;
    }
    void context(bool comes) {
        std::lock_guard<std::mutex> l(mu_);
        contexts_ += comes ? 1 : -1;
        if (contexts_ > 0) return;
        for (uint32_t i = 0; i < made_n_; i++) {
            cudaGraphExecDestroy(made_[i]->exec);
            cudaGraphDestroy(made_[i]->graph);
            delete made_[i];
        }
        made_n_ = asked_n_ = 0;
    }

  private:
    static constexpr uint32_t kMost = 48, kMostAsked = 4 * kMost;
    static constexpr int32_t kFrom = 4;
    struct Asked {
        LaunchGraph what;
        int32_t times;
    };
    Asked *asked(const LaunchGraph &want) {
        for (uint32_t i = 0; i < asked_n_; i++)
            if (asked_[i].what.is(want)) return &asked_[i];
        return nullptr;
    }
    static LaunchGraph make_; // "there is room for one more"
    std::mutex mu_;
    LaunchGraph *made_[kMost];
    Asked asked_[kMostAsked];
    uint32_t made_n_ = 0, asked_n_ = 0, making_ = 0;
    int contexts_ = 0;
};
LaunchGraph GraphPool::make_{};
// Made with a device's first context and never destroyed (the driver may be gone before); null if there was no memory for it.
constexpr int kDevices = 64;
std::atomic<GraphPool *> pools[kDevices];
GraphPool *pool_of(int device) { return device >= 0 && device < kDevices ? pools[device].load(std::memory_order_acquire) : nullptr; }

} // namespace

void launch_graphs_context(int device, bool comes) {
    if (comes && device >= 0 && device < kDevices && !pool_of(device)) {
        GraphPool *none = nullptr, *const made = new (std::nothrow) GraphPool;
        if (!pools[device].compare_exchange_strong(none, made)) delete made;
    }
    if (GraphPool *const p = pool_of(device)) p->context(comes);
}
void launch_graph_give(LaunchGraph *g) {
    if (g) pool_of(g->device)->give(g);
}

Launches::Launches(cudaStream_t s, bool gather) : s_(s), gathering_(gather), outer_(t_gathering) { t_gathering = this; }
Launches::~Launches() { t_gathering = outer_; }

bool Launches::add(const LaunchShape &shape, void *const *args, const uint32_t *sizes, uint32_t n) {
    if (!gathering_ || n_ == kMost || n > kArgs) return false;
    One &o = one_[n_];
    uint32_t at = 0;
    for (uint32_t i = 0; i < n; i++) {
        if (at + sizes[i] > kStore) return false;
        o.args[i] = o.store + at;
        memcpy(o.store + at, args[i], sizes[i]);
        at = (at + sizes[i] + 15u) & ~15u;
    }
    o.shape = shape;
    n_++;
    return true;
}

cudaError_t launch_any(const LaunchShape &shape, void *const *args, const uint32_t *sizes, uint32_t n, cudaStream_t s) {
    Launches *const l = t_gathering;
    if (l && l->s_ == s) {
        if (l->add(shape, args, sizes, n)) return cudaSuccess;
        const cudaError_t e = l->stop(); // in order
        if (e != cudaSuccess) return e;
    }
    return launch_now(shape, args, s);
}

static cudaKernelNodeParams node_params(const LaunchShape &k, void **args) {
    cudaKernelNodeParams p = {};
    p.func = const_cast<void *>(k.fn);
    p.gridDim = k.grid;
    p.blockDim = k.block;
    p.sharedMemBytes = k.smem;
    p.kernelParams = args;
    return p;
}
// A graph of the n gathered launches' kernels, made if need be.
LaunchGraph *Launches::graph(uint32_t n) {
    int device = 0;
    GraphPool *const p = n != 0 && cudaGetDevice(&device) == cudaSuccess ? pool_of(device) : nullptr;
    if (!p) return nullptr;
    GraphPool &pool = *p;
    LaunchGraph want{};
    want.n = n;
    for (uint32_t i = 0; i < n; i++) {
        want.fn[i] = one_[i].shape.fn;
        want.cluster[i] = one_[i].shape.cluster;
    }
    want.behind = n == 2 && one_[1].shape.behind; // (of the first: nothing is in front, or it is waited for)
    want.device = device;
    LaunchGraph *g = pool.take(want);
    if (!GraphPool::to_be_made(g)) return g;
    // Put together node by node: with a stream captured instead, cuCtxSynchronize of another thread (which a batch's creation
    // calls) crashed now and then.
    g = new (std::nothrow) LaunchGraph(want);
    int low = 0, high = 0; // the priority that batches' streams have
    cudaError_t e = g ? cudaDeviceGetStreamPriorityRange(&low, &high) : cudaErrorMemoryAllocation;
    if (e == cudaSuccess) e = cudaGraphCreate(&g->graph, 0);
    for (uint32_t i = 0; i < n && e == cudaSuccess; i++) {
        const cudaKernelNodeParams p = node_params(one_[i].shape, one_[i].args);
        e = cudaGraphAddKernelNode(&g->node[i], g->graph, nullptr, 0, &p);
        cudaLaunchAttributeValue v = {};
        v.priority = high;
        if (e == cudaSuccess) e = cudaGraphKernelNodeSetAttribute(g->node[i], cudaLaunchAttributePriority, &v);
        if (e == cudaSuccess && want.cluster[i] > 1) {
            v = {};
            v.clusterDim.x = want.cluster[i];
            v.clusterDim.y = v.clusterDim.z = 1;
            e = cudaGraphKernelNodeSetAttribute(g->node[i], cudaLaunchAttributeClusterDimension, &v);
        }
    }
    if (e == cudaSuccess && n == 2) {
        cudaGraphEdgeData edge = {};
        if (want.behind) {
            edge.type = cudaGraphDependencyTypeProgrammatic;
            edge.from_port = cudaGraphKernelNodePortProgrammatic;
        }
        e = cudaGraphAddDependencies_v2(g->graph, &g->node[0], &g->node[1], &edge, 1);
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&g->exec, g->graph, 0);
    if (e != cudaSuccess) {
        if (g && g->graph) cudaGraphDestroy(g->graph);
        delete g;
        g = nullptr;
        (void)cudaGetLastError();
        pool.failed(want);
    } else {
        g->taken = true;
    }
    pool.made(g);
    return g;
}

cudaError_t Launches::send(LaunchGraph *&taken) {
    LaunchGraph *const g = graph(n_);
    if (!g) return stop();
    cudaError_t e = cudaSuccess;
    for (uint32_t i = 0; i < n_ && e == cudaSuccess; i++) {
        const cudaKernelNodeParams p = node_params(one_[i].shape, one_[i].args);
        e = cudaGraphExecKernelNodeSetParams(g->exec, g->node[i], &p);
    }
    if (e == cudaSuccess) e = cudaGraphLaunch(g->exec, s_);
    if (e != cudaSuccess) {
        launch_graph_give(g);
        (void)cudaGetLastError();
        return stop();
    }
    taken = g;
    n_ = 0;
    gathering_ = false;
    return cudaSuccess;
}

cudaError_t Launches::stop() {
    const uint32_t n = n_;
    n_ = 0;
    gathering_ = false;
    cudaError_t e = cudaSuccess;
    for (uint32_t i = 0; i < n && e == cudaSuccess; i++) e = launch_now(one_[i].shape, one_[i].args, s_);
    return e;
}
