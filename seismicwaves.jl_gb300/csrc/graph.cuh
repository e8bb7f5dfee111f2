// CUDA graphs of whole time loops, kept per simulation.
#pragma once

#include <cuda_runtime.h>

#include <limits>
#include <map>
#include <utility>
#include <vector>

#include "internal.h"

namespace swgb {

// Runs `work` (device work on the context's stream: launches, memsets and
// device copies; no host synchronisation, no allocation) through a CUDA graph:
// captured on the second call with `key` (one-off calls run directly) and
// replayed afterwards.  At most 32 graphs are held per simulation; a further
// key replaces the one that was left unused longest, if that is more than 256
// calls (a program that goes on to other shots or other output arrays would
// otherwise run directly for good; one that goes round more than 32 keys keeps
// 32 of them), and runs directly if not.
// A time loop is thousands of short launches, which the host issues more
// slowly than small grids execute them.  Work runs directly while profiling
// (the events belong to single launches), when the caller's stream is itself
// being captured (the launches then join the caller's graph) and on the legacy
// default stream, on which CUDA lets no capture begin.
// `key` holds everything the captured launches depend on besides the device
// buffers; `gen` is bumped whenever one of those is (re)allocated, which ends
// the use of every graph held.
struct GraphCache {
  struct Held {
    cudaGraphExec_t exec;
    long long last;  // the call that launched it last
  };
  static constexpr size_t MAX_HELD = 32;
  static constexpr long long UNUSED = 256;
  long long gen = 0;
  long long held_gen = 0, calls = 0;
  std::map<std::vector<long long>, Held> graphs;
  std::map<std::vector<long long>, int> uses;  // calls per key

  GraphCache() = default;
  GraphCache(const GraphCache&) = delete;
  GraphCache& operator=(const GraphCache&) = delete;
  ~GraphCache() { drop(); }
  void drop() {
    for (auto& kv : graphs) cudaGraphExecDestroy(kv.second.exec);
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
    ++calls;
    if (gen != held_gen) {
      if (!graphs.empty()) check_cuda(cudaStreamSynchronize(st), "graph release");
      drop();
      held_gen = gen;
    }
    auto it = graphs.find(key);
    if (it == graphs.end()) {
      if (uses.size() > 4096) uses.clear();
      if (++uses[key] < 2 || !make_room(st)) {
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
      if (e == cudaErrorMemoryAllocation) {  // no memory for the graph: this key goes on running directly
        cudaGetLastError();
        uses[key] = std::numeric_limits<int>::min();
        work();
        return;
      }
      check_cuda(e, "graph instantiate");
      it = graphs.emplace(key, Held{ex, 0}).first;
    }
    it->second.last = calls;
    check_cuda(cudaGraphLaunch(it->second.exec, st), "graph launch");
  }

 private:
  // Room for one more graph, by giving up one that the last UNUSED calls did not launch.
  bool make_room(cudaStream_t st) {
    if (graphs.size() < MAX_HELD) return true;
    auto old = graphs.begin();
    for (auto q = graphs.begin(); q != graphs.end(); ++q)
      if (q->second.last < old->second.last) old = q;
    if (calls - old->second.last <= UNUSED) return false;
    check_cuda(cudaStreamSynchronize(st), "graph release");
    cudaGraphExecDestroy(old->second.exec);
    uses.erase(old->first);
    graphs.erase(old);
    return true;
  }
};

}  // namespace swgb
