// Loops of many short kernels that a kernel of the loop ends: rounds go to the device
// a body's graph at a time, a little ahead of it, and the host watches their number
// and the end in mapped memory, so that neither waits for the other; and launches
// whose start overlaps the kernel before them.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <thread>
#include <tuple>

#include "errors.h"
#include "readback.h"

namespace isdf_b200 {

// What a loop's kernels tell the host, in mapped host memory: words[0] the rounds
// begun, words[1] whether the loop is over. nullptr: no one looks.
struct LoopSignal {
  int* words;
};

__device__ __forceinline__ void loop_round(const LoopSignal& sig, int rounds) {
  if (sig.words) *static_cast<volatile int*>(sig.words) = rounds;
}
__device__ __forceinline__ void loop_over(const LoopSignal& sig) {
  if (sig.words) *static_cast<volatile int*>(sig.words + 1) = 1;
}

// Begins a kernel launched by launch_early (what no kernel of the loop writes may
// be read before): waits for the whole of the kernel before it and its writes, then
// lets the next kernel's blocks become resident (they wait here in turn). Every block
// passes here before it reads, writes or returns: a kernel that completed without
// waiting would let the next one run ahead of the one before it. What a kernel of the
// loop writes is read through plain pointers: the block was resident while it was
// written, so that it is no read-only data.
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

// Runs a loop's rounds on a stream. A round in which the loop is over returns at once
// from each of its kernels, so a few too many do no harm.
//
// The rounds are launched as graphs of a body of them (a launch each would take the
// host longer than the GPU where the kernels are small), the first few directly, while
// the graph is made. A loop inside one graph, a WHILE node that a kernel ends, needs no
// host and runs as fast; but destroying such a graph waits for the whole device, so that
// a selection waited for every copy and every solve on other streams (75 ms behind a
// 4 GB copy; an ordinary graph's 0.2 ms does not), and with it the copy of the previous
// result to the host, which a pipeline of solves overlaps with the next one.
class Loop {
 public:
  explicit Loop(cudaStream_t s) : queue_(s) {
    progress_words(&host_, &sig_.words);
    if (host_) host_[0] = host_[1] = 0;
  }
  ~Loop() {
    // (no round may report once the words serve the next loop)
    (void)cudaStreamSynchronize(queue_.stream);
    if (exec_) cudaGraphExecDestroy(exec_);
    if (graph_) cudaGraphDestroy(graph_);
  }
  Loop(const Loop&) = delete;
  Loop& operator=(const Loop&) = delete;

  // Launches the first `rounds` rounds; round(queue, signal) launches one.
  template <class Round>
  int start(int rounds, Round round) {
    for (; launched_ < rounds; ++launched_) round(queue_, sig_);
    ISDF_CHECK_LAUNCH();
    return ISDF_OK;
  }

  // Launches the others, `per_body` at a time, until the loop is over or max_rounds
  // have been launched: the next body when no more than `slack` rounds are behind the
  // running one. stopped(&over) asks the device where no memory could be mapped.
  template <class Round, class Stopped>
  int finish(long long max_rounds, int per_body, int slack, Round round, Stopped stopped) {
    if (launched_ >= max_rounds || over()) return ISDF_OK;
    build(per_body, round);
    constexpr int kAskRounds = 8;
    long long idle = 0, ask = launched_ + kAskRounds;  // rounds known to have run; to ask at
    unsigned polls = 0;
    while (launched_ < max_rounds && !over()) {
      if (host_) {
        if (launched_ - std::max<long long>(idle, host_[0]) > slack) {
          // every so often, what the stream says: an error, or that nothing runs
          if ((++polls & 4095) == 0) {
            const cudaError_t e = cudaStreamQuery(queue_.stream);
            if (e == cudaSuccess) idle = launched_;
            else if (e != cudaErrorNotReady) ISDF_CUDA(e);
          }
          if ((polls & 63) == 0) std::this_thread::yield();
          continue;
        }
      } else if (launched_ >= ask) {
        bool done = false;
        ISDF_TRY(stopped(&done));
        if (done) break;
        ask = launched_ + kAskRounds;
      }
      if (exec_) ISDF_CUDA(cudaGraphLaunch(exec_, queue_.stream));
      else for (int i = 0; i < per_body; ++i) round(queue_, sig_);
      launched_ += per_body;
      ISDF_CHECK_LAUNCH();
    }
    return ISDF_OK;
  }

 private:
  bool over() const { return host_ && host_[1] != 0; }

  template <class Round>
  void build(int rounds, Round round) {
    bool ok = cudaGraphCreate(&graph_, 0) == cudaSuccess;
    if (ok) {
      LoopQueue body(graph_);
      for (int i = 0; i < rounds; ++i) round(body, sig_);
      ok = body.status == cudaSuccess;
    }
    if (!ok || cudaGraphInstantiate(&exec_, graph_, 0ull) != cudaSuccess) exec_ = nullptr;
    (void)cudaGetLastError();  // a refused step leaves an error to clear
  }

  LoopQueue queue_;
  LoopSignal sig_{nullptr};
  volatile int* host_ = nullptr;
  cudaGraph_t graph_ = nullptr;
  cudaGraphExec_t exec_ = nullptr;  // null where the graph could not be made
  long long launched_ = 0;          // rounds
};

}  // namespace isdf_b200
