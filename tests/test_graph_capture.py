"""The graph captures of the solver and the batch (quasar_b200/csrc/graph_capture.cuh)
against a fake CUDA runtime whose n-th call fails: no stream is left capturing,
no graph and no executable is left behind, and the handles are all made or all
null."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"

PROGRAM = r"""
#include "graph_capture.cuh"
#include <cstdio>
#include <stdexcept>
static int calls, fail_at, graphs, execs, capturing;
static bool failing() { return ++calls == fail_at; }
extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode m) {
  if (m != cudaStreamCaptureModeThreadLocal || capturing) return cudaErrorUnknown;
  if (failing()) return cudaErrorMemoryAllocation;
  capturing = 1;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  if (!capturing) return cudaErrorUnknown;
  capturing = 0;
  *g = nullptr;
  if (failing()) return cudaErrorStreamCaptureInvalidated;
  ++graphs;
  *g = reinterpret_cast<cudaGraph_t>(16);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  if (failing()) return cudaErrorMemoryAllocation;
  ++execs;
  *e = reinterpret_cast<cudaGraphExec_t>(32);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { --graphs; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { --execs; return cudaSuccess; }
}
int main() {
  const int n = 4;
  for (int throwing = 0; throwing < 2; ++throwing)
    for (fail_at = 1; fail_at <= 4 * n + 1; ++fail_at) {
      cudaGraphExec_t e[n];
      calls = 0;
      int issued = 0, thrown = 0;
      cudaError_t r = cudaSuccess;
      try {
        r = qb::capture_graphs(nullptr, n, [&](int k) {
          if (k != issued) std::puts("order");
          ++issued;
          if (throwing && failing()) throw std::runtime_error("launch");
        }, e);
      } catch (const std::runtime_error&) { thrown = 1; }
      const bool failed = fail_at <= (throwing ? 4 : 3) * n;
      bool any = false, all = true;
      for (auto h : e) { any = any || h; all = all && h; }
      if (capturing || graphs) std::printf("left capturing or a graph at %d\n", fail_at);
      if (failed != (thrown || r != cudaSuccess)) std::printf("result at %d\n", fail_at);
      if (failed ? any || execs : !all || execs != n) std::printf("handles at %d\n", fail_at);
      execs = 0;
    }
  std::puts("done");
}
"""


@pytest.mark.skipif(not (shutil.which("g++") and os.path.isdir(CUDA)), reason="no host compiler or CUDA headers")
def test_a_failed_capture_leaves_nothing_behind(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", "-I", CUDA, "-I",
                    os.path.join(ROOT, "quasar_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    assert out == "done\n", out


@pytest.mark.parametrize("name", ["mhd_solver.cu", "mhd_batch.cu"])
def test_every_capture_goes_through_it(name):
    with open(os.path.join(ROOT, "quasar_b200", "csrc", name)) as f:
        text = f.read()
    assert "capture_graphs(" in text
    assert "cudaStreamBeginCapture" not in text and "cudaGraphInstantiate" not in text


def test_a_step_gives_up_the_cached_limit_before_it_overwrites_it():
    """cfl_limit answers from the control block while its residual is cached; a
    step writes its own dt there, so the cache is dropped first, also when the
    launch that follows fails."""
    with open(os.path.join(ROOT, "quasar_b200", "csrc", "mhd_solver.cu")) as f:
        text = f.read()
    body = text[text.index("void MhdSolver2D::advance_positive("):text.index("void MhdSolver2D::controller(")]
    assert body.index("front_order_ = 0;") < body.index("&ctl_->dt, dt_host_")
