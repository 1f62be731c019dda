// Capture of a stretch of stream work into an instantiated graph.
#pragma once
#include <cuda_runtime_api.h>

namespace gelios {

// Captures what `enqueue` (true: everything was enqueued) puts on s, and on
// streams it forks to and joins back, into *exec.  The capture is ended
// whatever enqueue says: a stream left in capture would take every later
// launch into it.  False (and *exec null, no error pending) where there is no
// graph; nothing has run on s then, and the caller enqueues directly.
template <class F>
bool capture_graph(cudaStream_t s, cudaGraphExec_t* exec, F&& enqueue) {
    *exec = nullptr;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const bool ok = enqueue();
    cudaGraph_t graph = nullptr;
    const cudaError_t e = cudaStreamEndCapture(s, &graph);
    if (!ok || e != cudaSuccess || !graph || cudaGraphInstantiate(exec, graph, 0) != cudaSuccess) *exec = nullptr;
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    return *exec != nullptr;
}

}  // namespace gelios
