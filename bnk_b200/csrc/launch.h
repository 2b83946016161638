// How kernels are launched: one by one, or the one or two launches of a submit with one driver call.
//
// A launch of its own takes the driver 2.5 us, 4.3 when the caller comes back right after its last wait, and a submit of a
// few packets is little else.  An executable graph of the same kernel, whose grid and parameters are set anew each time,
// takes 1.3, and the kernel starts as much earlier (one thread, launch to pinned word: 7.1-8.8 us plain, 5.5-5.7; two kernels,
// the second a dependent launch: 9.1 and 6.6).  With several threads at it the two are alike or the graph is behind (8
// threads 9.9 and 10.0 us a round, 16 threads 10.1 and 10.9, but 4 threads 9.3 and 7.0), and a change of the kernel in such a graph
// costs what it saves (7.05 against 7.1).  So: few batches in flight, and a graph for every kernel or pair of kernels.
// Of a whole call, from submit to the end of the wait: 5 x 92 B sealed 15.0 us without and 14.4 with a graph, opened (two kernels)
// 20.9 and 17.2; 128 x 1420 B sealed 18.6 either way, opened 28.1 and 21.5.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

struct LaunchShape {
    const void *fn;
    dim3 grid, block;
    uint32_t smem, cluster; // dynamic shared memory; CTAs per cluster (1: none)
    bool behind;            // may be scheduled while the kernel in front is still running
};
__attribute__((visibility("hidden"))) cudaError_t launch_any(const LaunchShape &shape, void *const *args, const uint32_t *sizes, uint32_t n, cudaStream_t s);

template <typename T>
struct AsIs {
    using type = T;
};
template <typename... KArgs>
cudaError_t launch_shape(LaunchShape shape, void (*kernel)(KArgs...), cudaStream_t s, const typename AsIs<KArgs>::type &...args) {
    shape.fn = reinterpret_cast<const void *>(kernel);
    void *const at[] = {const_cast<void *>(static_cast<const void *>(&args))...};
    const uint32_t sizes[] = {(uint32_t)sizeof(KArgs)...};
    return launch_any(shape, at, sizes, sizeof...(KArgs), s);
}

struct LaunchGraph; // an executable graph that somebody has taken
// Gathers what its thread launches on a stream, from here to send() or its end (nothing but launches may be queued on the
// stream in between).
class __attribute__((visibility("hidden"))) Launches {
  public:
    Launches(cudaStream_t s, bool gather);
    ~Launches();
    Launches(const Launches &) = delete;
    // Launches what has been gathered, through a graph if there is one, and gathers no more.  The graph is left in `taken` and
    // has to be given back when the kernels are over.
    cudaError_t send(LaunchGraph *&taken);
    cudaError_t stop(); // the same without a graph

  private:
    friend cudaError_t launch_any(const LaunchShape &, void *const *, const uint32_t *, uint32_t, cudaStream_t);
    static constexpr uint32_t kMost = 2, kArgs = 16, kStore = 4096 + 16 * kArgs; // (kernels take up to 4 KB)
    struct One {
        LaunchShape shape;
        void *args[kArgs];
        alignas(16) uint8_t store[kStore];
    };
    LaunchGraph *graph(uint32_t n);
    bool add(const LaunchShape &shape, void *const *args, const uint32_t *sizes, uint32_t n);
    cudaStream_t s_;
    bool gathering_;
    uint32_t n_ = 0;
    Launches *outer_;
    One one_[kMost];
};
__attribute__((visibility("hidden"))) void launch_graph_give(LaunchGraph *g);
// Contexts of a device come and go: its graphs are destroyed with the last one.
__attribute__((visibility("hidden"))) void launch_graphs_context(int device, bool comes);
