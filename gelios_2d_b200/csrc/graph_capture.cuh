// Capture of a stretch of stream work into an instantiated graph, and when
// that is worth its cost.
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

// Whether two steps of a moving-grid form run as one graph that is not there
// yet: `ahead` times in the rest of this call, `uses` times asked for before.
// Capturing it costs 560 us (MK2; MHD 100, five fluids 300, 8k cells) and a
// use saves 7 us against two one-step graphs (five fluids: 30 against direct
// launches), so a first call pays for it only where it replays it several
// times, and a program of short calls once it has missed it long enough.  us
// of the first call of a context of 8k cells, formed at once / one-step graphs
// or direct launches: MK2 4 steps 1418 / 1128, 6: 1412 / 1143, 8: 1408 / 1233,
// 9: 1258 / 1264, 20: 1837 / 1910; five fluids 8 steps 1597 / 1234, 10: 1544 /
// 1428, 20: 2432 / 2518; MHD 8: 1101 / 1119, 20: 1706 / 1880.
constexpr int kPairAhead = 4, kPairAheadDirect = 8, kPairUses = 64;
inline bool pair_graph_worth(bool direct_otherwise, int ahead, int uses) {
    return ahead >= (direct_otherwise ? kPairAheadDirect : kPairAhead) || uses >= kPairUses;
}
// The five-fluid form and the batched sweep launch a step's ten (six) kernels
// directly until a step graph has been asked for this often: capturing it costs
// 165 us (200 for the sweep's two branches) and saves 15.  (MK2 and MHD steps
// are longer chains on more streams: their graphs are captured at once.)
constexpr int kStepGraphUses = 16;

}  // namespace gelios
