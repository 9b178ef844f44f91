"""Host logic of the gain-index check (no GPU): the pinned buffer it copies into
against a stand-in for the CUDA runtime whose copies land late.

A small program built with g++ from ``nsrno_b200/csrc/nsr_gain_check.cuh``
defines the handful of runtime calls the check makes: a copy is carried out when
its event or stream is waited for, and not before."""
import shutil
import subprocess
from pathlib import Path

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "nsr_gain_check.cuh"
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

struct Copy { void* dst; const void* src; size_t bytes; cudaStream_t st; };
static std::vector<Copy> pending;                      // copies that have not landed
static int live_buffers = 0;                           // pinned allocations
static std::vector<std::pair<cudaEvent_t, cudaStream_t>> events;
static bool fail_record = false;
static std::mutex guard;

static void land(cudaStream_t st) {
  std::vector<Copy> rest;
  for (const Copy& c : pending)
    if (c.st == st) std::memcpy(c.dst, c.src, c.bytes); else rest.push_back(c);
  pending.swap(rest);
}
extern "C" {
cudaError_t CUDARTAPI cudaHostAlloc(void** p, size_t n, unsigned) {
  std::lock_guard<std::mutex> l(guard);
  *p = std::malloc(n);
  ++live_buffers;
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFreeHost(void* p) {
  std::lock_guard<std::mutex> l(guard);
  for (const Copy& c : pending)
    if (c.dst == p) { std::printf("freed under a copy\n"); std::exit(1); }
  std::free(p);
  --live_buffers;
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  std::lock_guard<std::mutex> l(guard);
  pending.push_back({d, s, n, st});
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
  if (fail_record) return cudaErrorInvalidResourceHandle;
  std::lock_guard<std::mutex> l(guard);
  events.push_back({e, st});
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::mutex> l(guard);
  for (auto it = events.rbegin(); it != events.rend(); ++it)
    if (it->first == e) { land(it->second); break; }
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t st) {
  std::lock_guard<std::mutex> l(guard);
  land(st);
  return cudaSuccess;
}
}

int main(int argc, char** argv) {
  const int what = std::atoi(argv[1]);
  float params = 0.f;
  std::vector<int32_t> good(1500, 1), bad(1500, 1);
  bad[2] = 7;
  NsrLearned G = {&params, &params, good.data(), 4, 0}, B = {&params, &params, bad.data(), 4, 0};
  const cudaStream_t s1 = (cudaStream_t)8, s2 = (cudaStream_t)16;
  if (what == 0) {          // indices are looked at once they have landed
    GainCheck g, b;
    if (g.start(&G, 3, s1) || g.finish()) return 2;
    if (b.start(&B, 3, s1) || b.finish() != NSR_ERR_ARGUMENT) return 3;
    GainCheck n;
    if (n.start(&G, 0, s1) || n.finish()) return 4;
  } else if (what == 1) {   // a caller that gives up leaves no copy under way
    { GainCheck g; if (g.start(&B, 3, s1)) return 2; }
    if (!pending.empty()) { std::printf("copy outlives its check\n"); return 3; }
    GainCheck g;
    if (g.start(&G, 1200, s2) || g.finish()) return 4;
  } else if (what == 2) {   // nor does one whose event cannot be recorded
    fail_record = true;
    { GainCheck g; if (!g.start(&B, 3, s1)) return 2; }
    if (!pending.empty()) { std::printf("copy outlives its check\n"); return 3; }
  } else {                  // a thread gives its buffer back
    for (int k = 0; k < 5; ++k) {
      std::thread t([&] { GainCheck g; if (g.start(&G, 3, s1) || g.finish()) std::exit(5); });
      t.join();
    }
    if (live_buffers) { std::printf("%d buffers left behind\n", live_buffers); return 6; }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    gxx = shutil.which("g++")
    cuda = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parents[1] / "include"
    if not gxx or not (cuda / "cuda_runtime.h").exists():
        pytest.skip("g++ or the CUDA headers are not available")
    d = tmp_path_factory.mktemp("gaincheck")
    src, exe = d / "probe.cpp", d / "probe"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O1", f"-I{cuda}", f"-I{ROOT / 'include'}", f"-I{ROOT / 'nsrno_b200' / 'csrc'}",
                    str(src), "-o", str(exe), "-pthread"], check=True)
    return exe


@pytest.mark.parametrize("what", ["indices", "abandoned", "unrecorded", "thread"])
def test_gain_check(program, what):
    code = ["indices", "abandoned", "unrecorded", "thread"].index(what)
    run = subprocess.run([str(program), str(code)], capture_output=True, text=True)
    assert run.returncode == 0, (run.returncode, run.stdout)
