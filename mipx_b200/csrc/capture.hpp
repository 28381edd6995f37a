// Capturing launches into an executable graph.
#pragma once

#include <cuda_runtime_api.h>

namespace pdlpx {

// begin(), launches(), end(), each returning an error code (E{}: none).  A capture
// that began is ended whatever the launches return, and the first error is the
// result: a launch that was refused is missing from the graph.
template <class E, class Begin, class Launches, class End>
E captured(Begin begin, Launches launches, End end) {
    E e = begin();
    if (e != E{}) return e;
    e = launches();
    const E f = end();
    return e != E{} ? e : f;
}

// Replaces `exec` by the graph of what `launches` (returns a cudaError_t) puts on the
// stream; null after an error, of which <<<>>> launches leave theirs as the last.
template <class Launches>
cudaError_t captureGraph(cudaStream_t s, cudaGraphExec_t& exec, Launches launches) {
    if (exec != nullptr) cudaGraphExecDestroy(exec);
    exec = nullptr;
    cudaGraph_t graph = nullptr;
    (void)cudaGetLastError();
    cudaError_t e = captured<cudaError_t>(
        [&] { return cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal); },
        [&] {
            const cudaError_t f = launches();
            const cudaError_t last = cudaGetLastError();
            return f != cudaSuccess ? f : last;
        },
        [&] { return cudaStreamEndCapture(s, &graph); });
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    if (graph != nullptr) cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
        exec = nullptr;
        (void)cudaGetLastError();
    }
    return e;
}

// Whether the blocks of a cooperative launch are all resident at once: what a grid
// whose blocks wait for one another needs.
inline bool residentAtOnce(int cooperative, int blocks_per_sm, int sms, int grid) {
    return cooperative != 0 && grid > 0 && static_cast<long long>(blocks_per_sm) * sms >= grid;
}
template <class... Args>
bool cooperativeFits(void (*kernel)(Args...), int device, int sms, int grid, int threads, int& blocks) {
    int coop = 0;
    blocks = 0;  // of the kernel that one SM holds
    const bool known = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) == cudaSuccess &&
                       cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                           &blocks, reinterpret_cast<const void*>(kernel), threads, 0) == cudaSuccess;
    if (!known) (void)cudaGetLastError();
    return known && residentAtOnce(coop, blocks, sms, grid);
}

}  // namespace pdlpx
