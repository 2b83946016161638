"""Launches and their graphs (csrc/launch.cu) with a CUDA runtime that only keeps lists: who gets a graph and when, what is
launched, and that a process without memory, or a driver that refuses, gets its kernels launched one by one.  Host code only."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bnk_b200", "csrc")

RUNTIME = r"""
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>
enum cudaError_t { cudaSuccess, cudaErrorMemoryAllocation, cudaErrorUnknown };
struct dim3 { unsigned x, y, z; dim3(unsigned a = 1, unsigned b = 1, unsigned c = 1) : x(a), y(b), z(c) {} };
struct Launched { const void *fn; unsigned grid; int arg; const void *graph; };
struct Stream { std::vector<Launched> ran; };
typedef Stream *cudaStream_t;
enum cudaLaunchAttributeID { cudaLaunchAttributeProgrammaticStreamSerialization, cudaLaunchAttributeClusterDimension, cudaLaunchAttributePriority };
struct cudaLaunchAttributeValue { int programmaticStreamSerializationAllowed; struct { unsigned x, y, z; } clusterDim; int priority; };
struct cudaLaunchAttribute { cudaLaunchAttributeID id; cudaLaunchAttributeValue val; };
struct cudaLaunchConfig_t { dim3 gridDim, blockDim; size_t dynamicSmemBytes; cudaStream_t stream; cudaLaunchAttribute *attrs; unsigned numAttrs; };
struct cudaKernelNodeParams { void *func; dim3 gridDim, blockDim; unsigned sharedMemBytes; void **kernelParams, **extra; };
struct Node { const void *fn; unsigned grid; int arg; };
struct Graph { std::vector<Node *> nodes; };
struct Exec { std::vector<Node> nodes; Graph *of; };
typedef Node *cudaGraphNode_t;
typedef Graph *cudaGraph_t;
typedef Exec *cudaGraphExec_t;
enum { cudaGraphDependencyTypeProgrammatic = 1, cudaGraphKernelNodePortProgrammatic = 1 };
struct cudaGraphEdgeData { unsigned char from_port, to_port, type; };
inline int graphs = 0, execs = 0, refuse = 0; // refuse: 1 = instantiation fails, 2 = the launch of a graph does
inline Node node(const cudaKernelNodeParams *p) { return {p->func, p->gridDim.x, *static_cast<int *>(p->kernelParams[0])}; }
inline cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fn, void **args) {
    c->stream->ran.push_back({fn, c->gridDim.x, *static_cast<int *>(args[0]), nullptr});
    return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
inline cudaError_t cudaDeviceGetStreamPriorityRange(int *l, int *h) { *l = 0; *h = -5; return cudaSuccess; }
inline cudaError_t cudaGraphCreate(cudaGraph_t *g, unsigned) { *g = new Graph; graphs++; return cudaSuccess; }
inline cudaError_t cudaGraphDestroy(cudaGraph_t g) { for (Node *n : g->nodes) delete n; delete g; graphs--; return cudaSuccess; }
inline cudaError_t cudaGraphAddKernelNode(cudaGraphNode_t *n, cudaGraph_t g, const cudaGraphNode_t *, size_t, const cudaKernelNodeParams *p) {
    *n = new Node(node(p));
    g->nodes.push_back(*n);
    return cudaSuccess;
}
inline cudaError_t cudaGraphKernelNodeSetAttribute(cudaGraphNode_t, cudaLaunchAttributeID, const cudaLaunchAttributeValue *) { return cudaSuccess; }
inline cudaError_t cudaGraphAddDependencies_v2(cudaGraph_t, const cudaGraphNode_t *, const cudaGraphNode_t *, const cudaGraphEdgeData *, size_t) { return cudaSuccess; }
inline cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
    if (refuse == 1) return cudaErrorMemoryAllocation;
    *x = new Exec{{}, g};
    for (Node *n : g->nodes) (*x)->nodes.push_back(*n);
    execs++;
    return cudaSuccess;
}
inline cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete x; execs--; return cudaSuccess; }
inline cudaError_t cudaGraphExecKernelNodeSetParams(cudaGraphExec_t x, cudaGraphNode_t n, const cudaKernelNodeParams *p) {
    for (size_t i = 0; i < x->of->nodes.size(); i++) if (x->of->nodes[i] == n) x->nodes[i] = node(p);
    return cudaSuccess;
}
inline cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
    if (refuse == 2) return cudaErrorUnknown;
    for (const Node &n : x->nodes) s->ran.push_back({n.fn, n.grid, n.arg, x});
    return cudaSuccess;
}
"""
PROGRAM = r"""
#include "launch.cu"
#include <cstdio>
#include <cstdlib>
static bool no_memory = false; // (the lists above may go on)
static int allowed = 0;
void *operator new(size_t n) { if (no_memory && !allowed) throw std::bad_alloc(); return malloc(n); }
void *operator new(size_t n, const std::nothrow_t &) noexcept { return no_memory && !allowed ? nullptr : malloc(n); }
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }
template <int K> void kernel(int, int) {}
typedef void (*Kernel)(int, int);
template <size_t... K> static Kernel nth(size_t i, std::index_sequence<K...>) { static const Kernel all[] = {kernel<(int)K>...}; return all[i]; }
static Kernel k(size_t i) { return nth(i, std::make_index_sequence<300>()); }
#define WANT(c) do { if (!(c)) { printf("%d: " #c "\n", __LINE__); exit(1); } } while (0)
static int next_arg = 0;
// One submit of kernels a and, if b >= 0, b: both run, in order, with this submit's grid and argument.  Its graph, if it had one.
static LaunchGraph *submit(int a, int b = -1, bool gather = true) {
    static Stream s;
    { allowed++; s.ran.clear(); s.ran.reserve(8); allowed--; }
    const int arg = ++next_arg;
    LaunchGraph *g = nullptr;
    {
        Launches all(&s, gather);
        WANT(launch_shape(LaunchShape{nullptr, dim3(arg), dim3(32), 0, 1, false}, k(a), &s, arg, 0) == cudaSuccess);
        if (b >= 0) WANT(launch_shape(LaunchShape{nullptr, dim3(arg + 1), dim3(32), 0, 1, true}, k(b), &s, arg + 1, 0) == cudaSuccess);
        WANT(s.ran.empty() == gather);
        WANT(all.send(g) == cudaSuccess);
    }
    const size_t n = b >= 0 ? 2 : 1;
    WANT(s.ran.size() == n);
    for (size_t i = 0; i < n; i++) {
        const Launched &x = s.ran[i];
        WANT(x.fn == (const void *)k(i ? b : a) && x.arg == arg + (int)i && x.grid == (unsigned)x.arg && (x.graph != nullptr) == (g != nullptr));
    }
    return g;
}
static int passes(int a, int b = -1) { // of six submits, each waited for, how many went through a graph
    int through = 0;
    for (int i = 0; i < 6; i++) {
        LaunchGraph *const g = submit(a, b);
        through += g != nullptr;
        launch_graph_give(g);
    }
    return through;
}
int main(int, char **argv) {
    const char what = argv[1][0];
    if (what != 'n') launch_graphs_context(0, true);
    if (what == 'u') { // used from the fourth request on, one submit at a time, until the last context goes
        WANT(passes(0) == 3 && passes(0) == 6 && passes(0, 1) == 3 && passes(0, 2) == 3 && passes(1) == 3);
        WANT(submit(0, 1, false) == nullptr);
        LaunchGraph *held[3];
        for (auto &h : held) WANT((h = submit(0, 1)) != nullptr);
        WANT(held[0] != held[1] && held[1] != held[2] && held[0] != held[2]);
        launch_graphs_context(0, true);
        launch_graphs_context(0, false);
        LaunchGraph *const fourth = submit(0, 1);
        WANT(fourth && fourth != held[0] && fourth != held[1] && fourth != held[2]);
        launch_graph_give(held[1]);
        WANT(submit(0, 1) == held[1]);
        launch_graphs_context(0, false);
        WANT(graphs == 0 && execs == 0);
    } else if (what == 'b') { // bounded in number, and in what is remembered
        for (int i = 0; i < 300; i++) passes(i);
        WANT(execs == 48 && passes(0) == 6 && passes(299) == 0 && passes(60) == 0);
    } else if (what == 'm') { // no memory: as without graphs
        no_memory = true;
        for (int i = 0; i < 300; i++) WANT(passes(i) == 0 && passes(i, 0) == 0);
        WANT(graphs == 0);
    } else if (what == 'n') { // nor for the place they are kept in
        no_memory = true;
        launch_graphs_context(0, true);
        WANT(passes(0) == 0);
        launch_graphs_context(0, false);
    } else { // the driver refuses: kind by kind, and for the one launch
        refuse = 1;
        WANT(passes(0) == 0 && passes(0, 1) == 0 && graphs == 0);
        refuse = 0;
        WANT(passes(0) == 0 && passes(1) == 3);
        refuse = 2;
        WANT(passes(1) == 0);
        refuse = 0;
        WANT(passes(1) == 6);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("launch")
    (d / "cuda_runtime.h").write_text(RUNTIME)
    (d / "launch_test.cpp").write_text(PROGRAM)
    exe = str(d / "launch_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", "-I", str(d), "-I", CSRC, "-o", exe, str(d / "launch_test.cpp")], check=True)
    return exe


@pytest.mark.parametrize("what", ["used", "bounded", "memory", "no place", "refused"])
def test_launches_and_their_graphs(program, what):
    out = subprocess.run([program, what], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
