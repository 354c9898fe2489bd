// Capture of a stream's launches into an executable graph that leaves nothing
// behind when it fails: neither a stream that still captures nor a graph.
#pragma once

#include <cuda_runtime_api.h>

namespace qb {

// Captures what `issue` launches on `stream` (other threads' work is not
// affected) and instantiates it.  An exception of `issue` is passed on.
template <class Issue>
cudaError_t capture_graph(cudaStream_t stream, Issue&& issue, cudaGraphExec_t* out) {
  cudaError_t e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return e;
  cudaGraph_t graph = nullptr;
  try {
    issue();
  } catch (...) {
    cudaStreamEndCapture(stream, &graph);
    if (graph) cudaGraphDestroy(graph);
    throw;
  }
  e = cudaStreamEndCapture(stream, &graph);
  if (e == cudaSuccess) e = cudaGraphInstantiate(out, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (e != cudaSuccess) *out = nullptr;
  return e;
}

// n graphs, issue(k) launching the k-th: all of them in out[0 .. n), or none
// (out all null) with the first error.
template <class Issue>
cudaError_t capture_graphs(cudaStream_t stream, int n, Issue&& issue, cudaGraphExec_t* out) {
  struct Undo {
    cudaGraphExec_t* out;
    int n, made = 0;
    ~Undo() {
      for (int k = 0; made < n && k < n; ++k) {
        if (out[k]) cudaGraphExecDestroy(out[k]);
        out[k] = nullptr;
      }
    }
  } undo{out, n};
  for (int k = 0; k < n; ++k) out[k] = nullptr;
  for (; undo.made < n; ++undo.made) {
    const int k = undo.made;
    const cudaError_t e = capture_graph(stream, [&] { issue(k); }, &out[k]);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace qb
