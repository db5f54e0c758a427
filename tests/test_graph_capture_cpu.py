"""capture_graph leaves no graph behind when a launch or the capture fails: the header
compiled against stand-ins for the five CUDA calls that it makes."""
import subprocess
from pathlib import Path

from test_cabi_client import compiler

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <cstdio>
#include "graph_capture.h"
static cudaError_t begin_e, launch_e, end_e;
static int live, enqueued;
extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return begin_e; }
cudaError_t cudaGetLastError(void) { return launch_e; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    const bool made = end_e == cudaSuccess;
    *g = made ? (cudaGraph_t)&live : nullptr;
    live += made;
    return end_e;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { --live; return cudaSuccess; }
}
int main() {
    const cudaError_t ok = cudaSuccess, bad = cudaErrorInvalidValue, worse = cudaErrorUnknown;
    const cudaError_t cases[5][4] = {  // begin, launch, end; what comes back
        {ok, ok, ok, ok}, {bad, ok, ok, bad}, {ok, bad, ok, bad}, {ok, ok, bad, bad}, {ok, worse, bad, worse}};
    for (const auto& c : cases) {
        begin_e = c[0]; launch_e = c[1]; end_e = c[2];
        live = enqueued = 0;
        cudaGraph_t g = (cudaGraph_t)&enqueued;
        const cudaError_t e = sph::capture_graph(nullptr, [&] { ++enqueued; }, &g);
        std::printf("%d %d %d %d\n", e == c[3], live, g != nullptr, enqueued);
    }
}
"""


def test_no_graph_is_left(tmp_path):
    src, exe = tmp_path / "capture.cpp", tmp_path / "capture"
    src.write_text(PROGRAM)
    cuda = Path("/usr/local/cuda/include")
    r = subprocess.run([compiler("g++"), "-std=c++17", "-Wall", "-Werror", "-I", str(cuda), "-I",
                        str(ROOT / "sph2s_final_gb300" / "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout.split("\n")
    # right status, graphs alive, a graph returned, enqueued
    assert out[:5] == ["1 1 1 1", "1 0 0 0", "1 0 0 1", "1 0 0 1", "1 0 0 1"]
