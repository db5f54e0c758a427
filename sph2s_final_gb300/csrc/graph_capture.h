// graph_capture.h -- captures what a function enqueues on a stream as a CUDA graph.
#pragma once
#include <cuda_runtime.h>

namespace sph {

// On success *graph holds what enqueue() launched on st; on any failure, a launch's
// included, there is no graph left to destroy and *graph is NULL.
template <class F>
inline cudaError_t capture_graph(cudaStream_t st, F&& enqueue, cudaGraph_t* graph) {
    *graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    enqueue();
    const cudaError_t launch = cudaGetLastError();
    e = cudaStreamEndCapture(st, graph);
    if (launch != cudaSuccess) e = launch;
    if (e != cudaSuccess && *graph) {
        cudaGraphDestroy(*graph);
        *graph = nullptr;
    }
    return e;
}

}  // namespace sph
