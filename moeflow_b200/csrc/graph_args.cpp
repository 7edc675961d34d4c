// Kernel nodes of a captured forward whose arguments change between replays.
//
// A serving step used to copy its inputs into the buffers the captured graph reads and its output out of the one it
// writes: three or four small stream operations around the replay, about 3 us each plus the gap in front of the graph.
// Instead the graph's first and last kernels are pointed at the caller's buffers (a host-side update of the executable
// graph, only when the pointers or the row count have changed).  That is done on an executable graph of its own, launched
// only behind such an update: the one that the owner of the capture replays keeps the arguments it was captured with.
#include <cuda_runtime.h>

#include "moeflow_b200.h"

extern "C" {

// The kernel node that the capture on `stream` added last.
int mf_capture_last_node(mf_stream_t stream, void** node_out) {
  if (!node_out) return -1;
  cudaStreamCaptureStatus status;
  const cudaGraphNode_t* deps = nullptr;
  const cudaGraphEdgeData* edges = nullptr;
  cudaGraph_t graph = nullptr;
  size_t n = 0;
  cudaError_t e = cudaStreamGetCaptureInfo_v3(static_cast<cudaStream_t>(stream), &status, nullptr, &graph, &deps, &edges, &n);
  if (e != cudaSuccess) return (int)e;
  if (status != cudaStreamCaptureStatusActive || n != 1) return -2;
  cudaGraphNodeType type;
  e = cudaGraphNodeGetType(deps[0], &type);
  if (e != cudaSuccess) return (int)e;
  if (type != cudaGraphNodeTypeKernel) return -3;
  *node_out = deps[0];
  return 0;
}

int mf_graph_instantiate(void* graph, mf_stream_t stream, void** exec_out) {
  if (!graph || !exec_out) return -1;
  cudaGraphExec_t exec = nullptr;
  cudaError_t e = cudaGraphInstantiate(&exec, static_cast<cudaGraph_t>(graph), 0);
  if (e != cudaSuccess) return (int)e;
  e = cudaGraphUpload(exec, static_cast<cudaStream_t>(stream));  // not at the first launch
  if (e != cudaSuccess) {
    cudaGraphExecDestroy(exec);
    return (int)e;
  }
  *exec_out = exec;
  return 0;
}

int mf_graph_launch(void* graph_exec, mf_stream_t stream) {
  if (!graph_exec) return -1;
  return (int)cudaGraphLaunch(static_cast<cudaGraphExec_t>(graph_exec), static_cast<cudaStream_t>(stream));
}

int mf_graph_destroy(void* graph_exec) {
  if (!graph_exec) return -1;
  return (int)cudaGraphExecDestroy(static_cast<cudaGraphExec_t>(graph_exec));
}

// Replaces the by-value arguments of a kernel node (one pointer per argument; same kernel, same launch shape) in an
// executable graph.  The graph that the node belongs to must still exist.
int mf_graph_set_args(void* graph_exec, void* node, void** args) {
  if (!graph_exec || !node || !args) return -1;
  cudaKernelNodeParams p = {};
  cudaError_t e = cudaGraphKernelNodeGetParams(static_cast<cudaGraphNode_t>(node), &p);
  if (e != cudaSuccess) return (int)e;
  p.kernelParams = args;
  p.extra = nullptr;
  return (int)cudaGraphExecKernelNodeSetParams(static_cast<cudaGraphExec_t>(graph_exec), static_cast<cudaGraphNode_t>(node), &p);
}

}  // extern "C"
