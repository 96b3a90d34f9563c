// Host helpers shared by the large-problem entry points: the CUDA graph that runs the
// RK loop as a device-side WHILE node, and a small cache of its executables.
#pragma once

#include <cstdlib>

#include <cuda_runtime.h>

#include <cstring>
#include <mutex>
#include <vector>

namespace dqb {

// Executable graphs keyed by the bytes of the launch parameters (pointers and sizes):
// a repeated call with the same buffers reuses its executable.  An evicted executable may
// still be running, so it is parked with an event recorded on the stream it was last
// launched on and destroyed once that event has completed (checked without blocking on
// every later insert).
class GraphCache {
 public:
  struct Entry {
    std::vector<unsigned char> key;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t stream = nullptr;
  };
  struct Parked {
    cudaGraphExec_t exec;
    cudaEvent_t done;
  };

  cudaGraphExec_t find(const void* key, size_t len) {
    std::lock_guard<std::mutex> lock(mu_);
    for (auto& e : entries_)
      if (e.key.size() == len && std::memcmp(e.key.data(), key, len) == 0) return e.exec;
    return nullptr;
  }

  void insert(const void* key, size_t len, cudaGraphExec_t exec, cudaStream_t s) {
    std::lock_guard<std::mutex> lock(mu_);
    reap();
    if (entries_.size() >= kMax) {
      Entry& old = entries_.front();
      Parked p{old.exec, nullptr};
      if (cudaEventCreateWithFlags(&p.done, cudaEventDisableTiming) == cudaSuccess &&
          cudaEventRecord(p.done, old.stream) == cudaSuccess) {
        parked_.push_back(p);
      } else {  // no event: wait for the stream instead
        if (p.done) cudaEventDestroy(p.done);
        cudaStreamSynchronize(old.stream);
        cudaGraphExecDestroy(old.exec);
      }
      entries_.erase(entries_.begin());
    }
    Entry e;
    e.key.assign((const unsigned char*)key, (const unsigned char*)key + len);
    e.exec = exec;
    e.stream = s;
    entries_.push_back(std::move(e));
  }

  void touch(const void* key, size_t len, cudaStream_t s) {
    std::lock_guard<std::mutex> lock(mu_);
    for (auto& e : entries_)
      if (e.key.size() == len && std::memcmp(e.key.data(), key, len) == 0) e.stream = s;
  }

 private:
  void reap() {
    for (size_t i = 0; i < parked_.size();) {
      if (cudaEventQuery(parked_[i].done) == cudaSuccess) {
        cudaGraphExecDestroy(parked_[i].exec);
        cudaEventDestroy(parked_[i].done);
        parked_.erase(parked_.begin() + i);
      } else {
        ++i;
      }
    }
  }

  static constexpr size_t kMax = 64;
  std::mutex mu_;
  std::vector<Entry> entries_;
  std::vector<Parked> parked_;
};

// DQB_HOST_LOOP=1 in the environment (read once): run the RK loop from the host, one
// iteration per round trip, instead of as a graph WHILE node.  Same kernels, same
// results; it exists for profilers that cannot see kernels inside conditional graphs.
inline bool host_loop_requested() {
  static const bool on = [] {
    const char* v = std::getenv("DQB_HOST_LOOP");
    return v != nullptr && v[0] == '1';
  }();
  return on;
}

// Host-driven form of "WHILE (cond) { body }": `body(stream, 0, flag)` enqueues one
// iteration whose last kernel writes the condition to the device word `flag`; the call
// returns when it reads 0.  Synchronises `stream` once per iteration.
template <class Body>
cudaError_t run_host_loop(Body body, int* flag, cudaStream_t s) {
  for (;;) {
    body(s, cudaGraphConditionalHandle(0), flag);
    int more = 0;
    cudaError_t err = cudaMemcpyAsync(&more, flag, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err == cudaSuccess) err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    if (!more) return cudaSuccess;
  }
}

// Adds "WHILE (handle) { body }" to `g` after `dep` (or at its start): `body(stream, handle,
// nullptr)` enqueues one loop iteration on the capture stream `cap` and must end with a
// kernel that sets the condition.
template <class Body>
cudaError_t add_while_node(cudaGraph_t g, cudaGraphConditionalHandle handle, const cudaGraphNode_t* dep,
                           cudaStream_t cap, Body body, cudaGraphNode_t* node) {
  cudaGraphNodeParams p = {cudaGraphNodeTypeConditional};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = handle;
  p.conditional.type = cudaGraphCondTypeWhile;
  p.conditional.size = 1;
  cudaError_t err = cudaGraphAddNode(node, g, dep, dep ? 1 : 0, &p);
  if (err != cudaSuccess) return err;
  cudaGraph_t bodyg = p.conditional.phGraph_out[0];
  err = cudaStreamBeginCaptureToGraph(cap, bodyg, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
  if (err != cudaSuccess) return err;
  body(cap, handle, (int*)nullptr);
  err = cudaStreamEndCapture(cap, &bodyg);
  return err == cudaSuccess ? cudaGetLastError() : err;
}

// Build "WHILE (cond) { body }" (add_while_node).
template <class Body>
cudaError_t build_while_graph(Body body, cudaGraphExec_t* out) {
  cudaGraph_t g = nullptr;
  cudaError_t err = cudaGraphCreate(&g, 0);
  if (err != cudaSuccess) return err;
  cudaStream_t cap = nullptr;
  err = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
  if (err == cudaSuccess) {
    cudaGraphConditionalHandle handle;
    cudaGraphNode_t node;
    err = cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault);
    if (err == cudaSuccess) err = add_while_node(g, handle, nullptr, cap, body, &node);
    cudaStreamDestroy(cap);
  }
  if (err == cudaSuccess) err = cudaGraphInstantiate(out, g, 0);
  cudaGraphDestroy(g);
  return err;
}

// Conditions of the loops of build_choice_graph.
struct LoopHandles {
  static constexpr int kCount = 3;
  cudaGraphConditionalHandle h[kCount];
};

// Build "choose; WHILE (h[0]) { body(0) }; WHILE (h[1]) { body(1) }; ...": `choose(stream, handles)`
// enqueues one kernel that sets the conditions (all 0 before it), so that the launch runs
// one of the loops; `body(stream, handle, i)` enqueues an iteration of loop i.
template <class Choose, class Body>
cudaError_t build_choice_graph(Choose choose, Body body, cudaGraphExec_t* out) {
  cudaGraph_t g = nullptr;
  cudaError_t err = cudaGraphCreate(&g, 0);
  if (err != cudaSuccess) return err;
  cudaStream_t cap = nullptr;
  err = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
  if (err == cudaSuccess) {
    LoopHandles hs;
    cudaGraphNode_t node;
    size_t count = 1;
    for (int i = 0; i < LoopHandles::kCount && err == cudaSuccess; ++i)
      err = cudaGraphConditionalHandleCreate(&hs.h[i], g, 0, cudaGraphCondAssignDefault);
    if (err == cudaSuccess)
      err = cudaStreamBeginCaptureToGraph(cap, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    if (err == cudaSuccess) {
      choose(cap, hs);
      err = cudaStreamEndCapture(cap, &g);
      if (err == cudaSuccess) err = cudaGetLastError();
    }
    if (err == cudaSuccess) err = cudaGraphGetNodes(g, &node, &count);
    if (err == cudaSuccess && count != 1) err = cudaErrorUnknown;
    for (int i = 0; i < LoopHandles::kCount && err == cudaSuccess; ++i) {
      const cudaGraphNode_t before = node;
      err = add_while_node(
          g, hs.h[i], &before, cap,
          [&](cudaStream_t cs, cudaGraphConditionalHandle h, int*) { body(cs, h, i); }, &node);
    }
    cudaStreamDestroy(cap);
  }
  if (err == cudaSuccess) err = cudaGraphInstantiate(out, g, 0);
  cudaGraphDestroy(g);
  return err;
}

}  // namespace dqb
