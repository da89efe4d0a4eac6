// A device-ended loop as a CUDA graph: a WHILE node whose body is made of the
// caller's launches and which a kernel of the body ends, so that no round of
// the loop waits for the host; and launches whose start overlaps the kernel before
// them, for loops of many short kernels.
#pragma once

#include <cuda_runtime.h>

#include <tuple>

namespace isdf_b200 {

// What the body's kernels get: with in_graph, end_loop() lets the running body be
// the last. max_rounds bounds the loop whatever else happens: the kernel that
// counts the rounds ends the loop beyond it.
struct LoopEnd {
  cudaGraphConditionalHandle handle;
  int in_graph;
  int max_rounds;
};

__device__ __forceinline__ void end_loop(const LoopEnd& le) {
  if (le.in_graph) cudaGraphSetConditional(le.handle, 0);
}

// Begins a kernel launched by launch_early (what no kernel of the loop writes may
// be read before): waits for the whole of
// the kernel before it and its writes, then lets the next kernel's blocks become
// resident (they wait here in turn). Every block passes here before it reads,
// writes or returns: a kernel that completed without waiting would let the next one
// run ahead of the one before it. What follows reads its state through plain
// pointers first, so that no read-only load moves above the wait.
__device__ __forceinline__ void after_previous() {
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
}

// Where a loop's launches go: onto a stream, or behind one another into a graph. (A
// graph is put together node by node, not captured: a capture on the caller's stream
// would take in what other threads launch there meanwhile.)
struct LoopQueue {
  cudaStream_t stream = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphNode_t last = nullptr;
  cudaError_t status = cudaSuccess;  // the first failure (of a graph; a stream's stay with the runtime)

  explicit LoopQueue(cudaStream_t s) : stream(s) {}
  explicit LoopQueue(cudaGraph_t g) : graph(g) {}
};

// Launches k, a kernel that begins with after_previous(), so that its blocks are
// set up while the kernel before it on the queue drains. An ordinary launch starts
// them only when that kernel has finished: about a microsecond on each kernel of a
// loop.
template <class... P, class... A>
void launch_early(void (*k)(P...), dim3 grid, dim3 block, size_t smem, LoopQueue& q,
                  const A&... args) {
  if (q.graph) {
    if (q.status != cudaSuccess) return;
    std::tuple<P...> values(static_cast<P>(args)...);
    void* params[sizeof...(P)];
    std::apply([&](auto&... v) { int i = 0; ((params[i++] = &v), ...); }, values);
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeKernel;
    np.kernel.func = reinterpret_cast<void*>(k);
    np.kernel.gridDim = grid;
    np.kernel.blockDim = block;
    np.kernel.sharedMemBytes = (unsigned)smem;
    np.kernel.kernelParams = params;
    cudaGraphEdgeData edge = {};
    edge.from_port = cudaGraphKernelNodePortProgrammatic;
    edge.type = cudaGraphDependencyTypeProgrammatic;
    cudaGraphNode_t node = nullptr;
    q.status = cudaGraphAddNode_v2(&node, q.graph, q.last ? &q.last : nullptr,
                                   q.last ? &edge : nullptr, q.last ? 1 : 0, &np);
    q.last = node;
    return;
  }
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = q.stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

struct LoopGraph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;  // null where the graph could not be made
  ~LoopGraph() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
  }

  // body(le, queue) launches one body of the loop on queue. Launches before it have
  // to be checked before it: errors that it meets are its own, and cleared (exec is
  // null then).
  template <class F>
  void build(int max_rounds, F body_launches) {
    LoopEnd le{0, 1, max_rounds};
    cudaGraphNodeParams np = {};
    cudaGraphNode_t node;
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    bool ok = cudaGraphCreate(&graph, 0) == cudaSuccess &&
              cudaGraphConditionalHandleCreate(&le.handle, graph, 1,
                                               cudaGraphCondAssignDefault) == cudaSuccess;
    if (ok) {
      np.conditional.handle = le.handle;
      ok = cudaGraphAddNode(&node, graph, nullptr, 0, &np) == cudaSuccess;
    }
    if (ok) {
      LoopQueue body(np.conditional.phGraph_out[0]);
      body_launches(le, body);
      ok = body.status == cudaSuccess;
    }
    if (!ok || cudaGraphInstantiate(&exec, graph, 0ull) != cudaSuccess) exec = nullptr;
    (void)cudaGetLastError();  // a refused step leaves an error to clear
  }
};

}  // namespace isdf_b200
