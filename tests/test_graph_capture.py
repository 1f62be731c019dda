"""The library's capture helper against a stand-in for the CUDA runtime: the
capture is ended on every path, nothing is leaked and no error stays pending."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "gelios_2d_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "graph_capture.cuh"
static int capturing, graphs, fail_at, pending;
static char g_graph, g_exec;
static cudaError_t step(int at) {
    if (fail_at != at) return cudaSuccess;
    pending = 1;
    return cudaErrorUnknown;
}
extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    if (step(1) != cudaSuccess) return cudaErrorUnknown;
    capturing++;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    capturing--;
    *g = nullptr;
    if (step(3) != cudaSuccess) return cudaErrorUnknown;
    graphs++;
    *g = reinterpret_cast<cudaGraph_t>(&g_graph);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    *x = reinterpret_cast<cudaGraphExec_t>(&g_exec);
    return step(4);
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { graphs--; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { pending = 0; return cudaSuccess; }
}
int main() {
    int bad = 0;
    for (fail_at = 0; fail_at <= 4; fail_at++) {  // 2: the enqueued work itself
        cudaGraphExec_t x = reinterpret_cast<cudaGraphExec_t>(&g_graph);
        int in = 0;
        const bool ok = gelios::capture_graph(nullptr, &x, [&]() { in = capturing; return step(2) == cudaSuccess; });
        const bool want = fail_at == 0;
        if (ok != want || (x != nullptr) != want || capturing || graphs || pending || (fail_at != 1 && in != 1)) {
            std::printf("failure at %d: ok %d graph %d capturing %d graphs left %d pending %d\n", fail_at, ok, x != nullptr,
                        capturing, graphs, pending);
            bad++;
        }
    }
    return bad;
}
"""


def test_capture_is_ended_on_every_path(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = Path(nvcc).resolve().parent.parent / "include"
    if not (include / "cuda_runtime_api.h").exists():
        pytest.skip("CUDA headers not found")
    (tmp_path / "capture.cpp").write_text(PROGRAM)
    exe = tmp_path / "capture"
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", f"-I{include}", str(tmp_path / "capture.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
