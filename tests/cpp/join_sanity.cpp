// The edges that the library's launches get in a captured stream: a launch
// that follows another of its stream alone may overlap that one's last wave
// (a programmatic edge); the first launch after the stream was joined with a
// second one waits for both in full, whatever the thread launched in between.
// The graphs are looked at and never run.
#include <cuda_runtime.h>

#include <cstdio>
#include <thread>
#include <vector>

#include "dsx.h"

namespace {

int failures = 0;

void check(bool ok, const char* what) {
    if (ok) return;
    std::printf("join_sanity: %s\n", what);
    ++failures;
}

// Edges into the nodes without a successor: how many, and how many of them
// are not full dependencies.
void last_edges(cudaGraph_t graph, int& edges, int& partial) {
    std::size_t n = 0, m = 0;
    check(cudaGraphGetEdges_v2(graph, nullptr, nullptr, nullptr, &n) == cudaSuccess, "edges");
    std::vector<cudaGraphNode_t> from(n), to(n);
    std::vector<cudaGraphEdgeData> data(n);
    m = n;
    check(cudaGraphGetEdges_v2(graph, from.data(), to.data(), data.data(), &m) == cudaSuccess, "edges");
    edges = partial = 0;
    for (std::size_t k = 0; k < n; ++k) {
        bool last = true;
        for (std::size_t j = 0; j < n; ++j) last = last && from[j] != to[k];
        if (!last) continue;
        ++edges;
        partial += data[k].type != cudaGraphDependencyTypeDefault || data[k].from_port != 0;
    }
}

}  // namespace

int main() {
    dsx_grid_desc d = {};
    d.nranks = 2;
    d.dims[0] = 2;
    d.dims[1] = d.dims[2] = 1;
    d.policy = DSX_MANUAL;
    for (int a = 0; a < 3; ++a) {
        d.upper[a] = 1.0;
        d.periodic[a] = 1;
    }
    d.halo_width = 0.1;
    d.dyn_interval = 1.0;
    d.dyn_threshold = 1.1;
    d.dyn_relaxation = 0.5;
    d.dyn_min_fraction = 0.1;
    dsx_grid* grid = nullptr;
    check(dsx_grid_create(&d, nullptr, 0, 64, 64, &grid) == DSX_OK, dsx_last_error());
    double* p = nullptr;
    int* out = nullptr;
    check(cudaMalloc(&p, 64 * sizeof(double)) == cudaSuccess, "malloc");
    check(cudaMalloc(&out, 64 * sizeof(int)) == cudaSuccess, "malloc");
    if (failures) return 1;
    cudaStream_t s, side, other;
    cudaEvent_t fork, join;
    cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking);
    cudaStreamCreateWithFlags(&other, cudaStreamNonBlocking);
    cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&join, cudaEventDisableTiming);
    auto launch = [&](cudaStream_t where) {
        check(dsx_grid_owner_rank(grid, p, p, p, 64, out, where) == DSX_OK, dsx_last_error());
    };
    // what runs between the join and the next launch on the joined stream
    const char* names[3] = {"nothing", "a launch on a second stream", "a launch by another thread"};
    for (int between = -1; between < 3; ++between) {
        cudaGraph_t g = nullptr;
        check(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess, "begin capture");
        launch(s);
        if (between >= 0) {
            cudaEventRecord(fork, s);
            cudaStreamWaitEvent(side, fork, 0);
            launch(side);
            launch(s);
            cudaEventRecord(join, side);
            cudaStreamWaitEvent(s, join, 0);
        }
        if (between == 1) launch(other);   // not part of the capture: it runs
        if (between == 2)
            std::thread([&] { launch(s); }).join();
        else
            launch(s);
        check(cudaStreamEndCapture(s, &g) == cudaSuccess, "end capture");
        int edges = 0, partial = 0;
        last_edges(g, edges, partial);
        std::printf("join_sanity: %s: %d edges into the last launch, %d of them partial\n",
                    between < 0 ? "no join" : names[between], edges, partial);
        if (between < 0) check(edges == 1 && partial == 1, "a launch along one stream waits in full");
        else check(edges == 2 && partial == 0, "the first launch after a join does not wait in full");
        cudaGraphDestroy(g);
    }
    cudaDeviceSynchronize();
    dsx_grid_destroy(grid);
    cudaFree(p);
    cudaFree(out);
    if (failures) return 1;
    std::printf("join_sanity: ok\n");
    return 0;
}
