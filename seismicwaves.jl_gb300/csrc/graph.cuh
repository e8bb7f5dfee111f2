// CUDA graphs of whole time loops, kept per simulation.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <utility>
#include <vector>

#include "internal.h"

namespace swgb {

// Runs `work` (device work on the context's stream: launches, memsets and
// device copies; no host synchronisation, no allocation) through a CUDA graph:
// captured on the second call with `key` (one-off calls run directly),
// replayed afterwards, at most 32 graphs per simulation, later keys directly.
// A time loop is thousands of short launches, which the host issues more
// slowly than small grids execute them.  Work runs directly while profiling
// (the events belong to single launches), when the caller's stream is itself
// being captured (the launches then join the caller's graph) and on the legacy
// default stream, on which CUDA lets no capture begin.
// `key` holds everything the captured launches depend on besides the device
// buffers; `gen` is bumped whenever one of those is (re)allocated.
struct GraphCache {
  long long gen = 0;
  std::map<std::vector<long long>, cudaGraphExec_t> graphs;
  std::map<std::vector<long long>, int> uses;  // calls per key

  GraphCache() = default;
  GraphCache(const GraphCache&) = delete;
  GraphCache& operator=(const GraphCache&) = delete;
  ~GraphCache() { drop(); }
  void drop() {
    for (auto& kv : graphs) cudaGraphExecDestroy(kv.second);
    graphs.clear();
    uses.clear();
  }

  template <typename Work>
  void run(sw_ctx* ctx, std::vector<long long> key, Work&& work) {
    cudaStream_t st = ctx->stream;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    check_cuda(cudaStreamIsCapturing(st, &cs), "cudaStreamIsCapturing");
    if (ctx->prof.on || cs != cudaStreamCaptureStatusNone || st == nullptr || st == cudaStreamLegacy) {
      work();
      return;
    }
    key.push_back(gen);
    auto it = graphs.find(key);
    if (it == graphs.end()) {
      if (uses.size() > 4096) uses.clear();
      if (++uses[key] < 2 || graphs.size() >= 32) {
        work();
        return;
      }
      check_cuda(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal), "begin stream capture");
      try {
        work();
      } catch (...) {
        cudaGraph_t g = nullptr;
        cudaStreamEndCapture(st, &g);
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
        throw;
      }
      cudaGraph_t g = nullptr;
      check_cuda(cudaStreamEndCapture(st, &g), "end stream capture");
      cudaGraphExec_t ex = nullptr;
      const cudaError_t e = cudaGraphInstantiate(&ex, g, 0);
      cudaGraphDestroy(g);
      check_cuda(e, "graph instantiate");
      it = graphs.emplace(key, ex).first;
    }
    check_cuda(cudaGraphLaunch(it->second, st), "graph launch");
  }
};

}  // namespace swgb
