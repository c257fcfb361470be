// Capture and replay of a fixed sequence of launches: the CUDA calls and nothing else. A capture through torch would also
// put the device's default random generator into capture mode, in which every other thread that draws from it meanwhile
// gets an error; the sequences captured here draw nothing.
#include "common.cuh"

using namespace kwu;

static int graph_check(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return 0;
  cudaGetLastError();   // not sticky: the next launch must not report it
  set_last_error("%s: %s", what, cudaGetErrorString(e));
  return 11;
}

// A stream of its own: torch hands out the streams of a small pool in turn, so one of those may be in use by another thread,
// whose launches would end up in the capture.
KWU_API int kwu_stream_create(void** stream) {
  cudaStream_t s = nullptr;
  const int rc = graph_check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "stream_create");
  *stream = s;
  return rc;
}

KWU_API int kwu_stream_destroy(void* stream) {
  return graph_check(cudaStreamDestroy(reinterpret_cast<cudaStream_t>(stream)), "stream_destroy");
}

// Thread-local mode: other threads may go on allocating and synchronising.
KWU_API int kwu_capture_begin(void* stream) {
  return graph_check(cudaStreamBeginCapture(reinterpret_cast<cudaStream_t>(stream), cudaStreamCaptureModeThreadLocal), "capture_begin");
}

// Ends the capture on `stream`. exec: where the executable graph goes; null: what was captured is dropped.
KWU_API int kwu_capture_end(void* stream, void** exec) {
  cudaGraph_t graph = nullptr;
  int rc = graph_check(cudaStreamEndCapture(reinterpret_cast<cudaStream_t>(stream), &graph), "capture_end");
  if (rc == 0 && exec) {
    cudaGraphExec_t e = nullptr;
    rc = graph_check(cudaGraphInstantiate(&e, graph, 0), "graph_instantiate");
    *exec = e;
  }
  if (graph) cudaGraphDestroy(graph);
  return rc;
}

KWU_API int kwu_graph_launch(void* exec, void* stream) {
  return graph_check(cudaGraphLaunch(reinterpret_cast<cudaGraphExec_t>(exec), reinterpret_cast<cudaStream_t>(stream)), "graph_launch");
}

KWU_API int kwu_graph_destroy(void* exec) {
  return graph_check(cudaGraphExecDestroy(reinterpret_cast<cudaGraphExec_t>(exec)), "graph_destroy");
}
