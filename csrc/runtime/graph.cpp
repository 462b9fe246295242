// Capture and replay of launches as CUDA graphs (context_parallelism_b200/graphs.py).  torch.cuda.CUDAGraph puts the process's default
// random generator into a capturing state, in which torch.randn of every other thread raises; the calls recorded here draw nothing,
// and a capture begun here leaves the generator alone.
#include <cuda_runtime.h>

#include "../kernels/host_utils.h"

using namespace cpb;

// Only the calling thread is kept from what a capture does not allow: others may allocate and synchronise.
extern "C" int cpb_graph_begin(cudaStream_t stream) {
  CPB_CUDA_OK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
  return CPB_OK;
}

// Ends the capture; exec_out (a graph ready to launch) may be null: the capture is dropped.
extern "C" int cpb_graph_end(cudaStream_t stream, void** exec_out) {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaError_t e = cudaStreamEndCapture(stream, &graph);
  if (e == cudaSuccess && graph != nullptr && exec_out != nullptr) e = cudaGraphInstantiate(&exec, graph, 0);
  if (graph != nullptr) cudaGraphDestroy(graph);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();                                        // the next launch would report it as its own
    return set_error(CPB_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
  }
  if (exec_out != nullptr) *exec_out = exec;
  return CPB_OK;
}

extern "C" int cpb_graph_launch(void* exec, cudaStream_t stream, int device) {
  int current = 0;
  CPB_CUDA_OK(cudaGetDevice(&current));
  if (current != device) CPB_CUDA_OK(cudaSetDevice(device));
  const cudaError_t e = cudaGraphLaunch((cudaGraphExec_t)exec, stream);
  if (current != device) (void)cudaSetDevice(current);
  if (e != cudaSuccess) return set_error(CPB_ERR_CUDA, "graph launch: %s", cudaGetErrorString(e));
  return CPB_OK;
}

// The graph must not be running.
extern "C" int cpb_graph_free(void* exec) {
  CPB_CUDA_OK(cudaGraphExecDestroy((cudaGraphExec_t)exec));
  return CPB_OK;
}
