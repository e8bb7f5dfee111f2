"""GraphCache (csrc/graph.cuh) without a GPU: the header compiled against a stand-in for the CUDA calls it makes."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
BUILD = Path(__file__).resolve().parent / "_build"
CUDA = next((p for p in (Path("/usr/local/cuda/include"),) if (p / "cuda_runtime.h").exists()), None)

PROBE = r"""
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include "graph.cuh"

namespace {
bool capturing = false;
bool full = false;
long long made = 0, live = 0, launched = 0;
}
extern "C" {
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  if (s == nullptr || s == cudaStreamLegacy) return cudaErrorStreamCaptureUnsupported;
  capturing = true;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  capturing = false;
  *g = reinterpret_cast<cudaGraph_t>(1);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  if (full) return cudaErrorMemoryAllocation;
  *e = reinterpret_cast<cudaGraphExec_t>(++made);
  ++live;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { ++launched; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { --live; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
}
namespace swgb {
void check_cuda(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw std::runtime_error(what);
}
Profiler::~Profiler() {}
}  // namespace swgb

// argv: stream handle, then per call "key", "+" (a buffer was reallocated) or "!" (the device's memory is full from
// here on); prints per call whether the work ran directly (d), was captured (c) or replayed (r) or the call failed (x),
// then the number of graphs held
int main(int argc, char** argv) {
  sw_ctx ctx;
  ctx.stream = reinterpret_cast<cudaStream_t>(std::atoll(argv[1]));
  swgb::GraphCache cache;
  for (int k = 2; k < argc; ++k) {
    if (argv[k][0] == '+') {
      ++cache.gen;
      continue;
    }
    if (argv[k][0] == '!') {
      full = true;
      continue;
    }
    char how = 'r';
    try {
      cache.run(&ctx, {std::atoll(argv[k])}, [&] { how = capturing ? 'c' : 'd'; });
    } catch (const std::exception& e) {
      how = 'x';
    }
    std::putchar(how);
  }
  std::printf(" %lld\n", live);
  return 0;
}
"""


@pytest.fixture(scope="module")
def probe():
    cxx = shutil.which("g++")
    if cxx is None or CUDA is None:
        pytest.skip("no C++ compiler or CUDA headers")
    BUILD.mkdir(exist_ok=True)
    src, exe = BUILD / "graph_probe.cpp", BUILD / "graph_probe"
    src.write_text(PROBE)
    subprocess.run([cxx, "-std=c++17", "-I", str(CUDA), "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "seismicwaves.jl_gb300" / "csrc"), str(src), "-o", str(exe)], check=True)

    def run(stream, *calls):
        out = subprocess.run([str(exe), str(stream), *map(str, calls)], capture_output=True, text=True, check=True)
        how, held = out.stdout.split()
        return how, int(held)

    return run


def test_captured_on_the_second_call(probe):
    assert probe(64, 5, 5, 5, 6, 5, 6, 6) == ("dcrdrcr", 2)


@pytest.mark.parametrize("legacy", [0, 1])
def test_legacy_default_stream_runs_directly(probe, legacy):
    assert probe(legacy, 5, 5, 5, 5) == ("dddd", 0)


def test_graphs_of_freed_buffers_are_given_back(probe):
    assert probe(64, 5, 5, 6, 6, "+", 5, 5, 5) == ("dcdcdcr", 1)


def test_other_keys_take_over_from_unused_ones(probe):
    """32 graphs whose keys do not come back (other output arrays, say) make room for those in use."""
    old = [k for key in range(100, 132) for k in (key, key)]
    how, held = probe(64, *old, *[7] * 300)
    assert how[:64] == "dc" * 32 and held == 32
    late = how[64:]
    assert "c" in late and late == "d" * late.index("c") + "c" + "r" * (299 - late.index("c"))


def test_more_keys_than_graphs_in_turn(probe):
    """40 keys in turn: 32 are replayed throughout, the others run directly, none is captured twice."""
    how, held = probe(64, *list(range(40)) * 20)
    assert held == 32 and how.count("c") == 32 and how.count("r") == 32 * 18


def test_no_memory_for_a_graph(probe):
    assert probe(64, 5, 5, "!", 6, 6, 6, 5, 6) == ("dcdddrd", 1)
