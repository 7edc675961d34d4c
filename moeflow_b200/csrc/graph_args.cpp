// Kernel nodes of a captured forward whose arguments change between replays.
//
// A serving step used to copy its inputs into the buffers the captured graph reads and its output out of the one it
// writes: three or four small stream operations around the replay, about 3 us each plus the gap in front of the graph.
// Instead the graph's first and last kernels are pointed at the caller's buffers (a host-side update of the executable
// graph, only when the pointers or the row count have changed).
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
