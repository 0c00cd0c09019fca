"""The host code that runs launches side by side (csrc/chains.h), compiled
here against fakes of the CUDA calls it makes: every one of them fails in
turn, and nothing may be left half made or an error go unseen."""
import os
import subprocess

from grim_b200.build import CSRC

CUDA_INCLUDE = "/usr/local/cuda/include"

FAKES = r"""
#include <cassert>
#include <cstdio>
#include "chains.h"
static int calls, failAt, live;  // the call to fail (-1: none), objects alive
static cudaError_t next() { return calls++ == failAt ? cudaErrorMemoryAllocation : cudaSuccess; }
static cudaStreamCaptureStatus status = cudaStreamCaptureStatusActive;
static std::vector<cudaGraphNode_t> now;
extern "C" {
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  const cudaError_t e = next();
  if (!e) *s = (cudaStream_t)(long)++live;
  return e;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* s, unsigned) {
  const cudaError_t e = next();
  if (!e) *s = (cudaEvent_t)(long)++live;
  return e;
}
// a capture: its dependency set is what the next launch depends on
cudaError_t cudaStreamGetCaptureInfo_v2(cudaStream_t, cudaStreamCaptureStatus* st, unsigned long long*, cudaGraph_t*,
                                        const cudaGraphNode_t** d, size_t* n) {
  const cudaError_t e = next();
  if (e) return e;
  *st = status;
  if (d) *d = now.data();
  if (n) *n = now.size();
  return e;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t* d, size_t n, unsigned) {
  const cudaError_t e = next();
  if (!e) now.assign(d, d + n);
  return e;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { live--; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { live--; return cudaSuccess; }
}
using namespace grim;
"""


def _run(tmp_path, main):
    src = tmp_path / "t.cpp"
    src.write_text(FAKES + main)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-g", "-D_GLIBCXX_ASSERTIONS", "-I", CSRC, "-I", CUDA_INCLUDE, str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_chains_are_made_whole_or_not_at_all(tmp_path):
    _run(tmp_path, r"""
int main() {
  std::vector<long long> work;
  std::vector<int> order;
  for (int p = 0; p < 40; p++) { work.push_back(1000 + 37 * p); order.insert(order.begin(), p); }
  for (int n : {1, 3, 40}) {
    work.resize(n, 5);
    std::vector<int> o;
    for (int p : order) if (p < n) o.push_back(p);
    const int streams = n < 16 ? n : 16;
    for (int f = 0; f < 2 * streams + 1; f++) {
      Chains c;
      calls = 0; failAt = f;
      assert(c.make(work, o, 16) == cudaErrorMemoryAllocation);
      // nothing made, nothing left behind, and the next step makes it
      assert(!c.made() && c.stream.empty() && c.join.empty() && !c.fork && live == 0);
      failAt = -1;
      assert(c.make(work, o, 16) == cudaSuccess && c.made());
      assert((int)c.stream.size() == streams && (int)c.join.size() == streams && c.fork && (int)c.of.size() == n);
      std::vector<long long> load(streams, 0);
      for (int p = 0; p < n; p++) { assert(c.of[p] >= 0 && c.of[p] < streams); load[c.of[p]] += work[p]; }
      long long lo = load[0], hi = load[0];
      for (long long l : load) { lo = std::min(lo, l); hi = std::max(hi, l); }
      assert(hi - lo <= *std::max_element(work.begin(), work.end()));
      c.release();
      assert(live == 0 && !c.made());
    }
    for (int p = n; p < 40; p++) work.push_back(1000 + 37 * p);
  }
}
""")


def test_a_fork_orders_its_branches_or_reports_the_failure(tmp_path):
    _run(tmp_path, r"""
static long node;
static std::vector<cudaGraphNode_t> launch() {  // a launch: its dependencies, and it is the next one's
  std::vector<cudaGraphNode_t> on = now;
  now.assign(1, (cudaGraphNode_t)(++node));
  return on;
}
int main() {
  for (int branches = 1; branches <= 4; branches++) {
    int total = 0;
    for (int f = -1; f < total || f < 0; f++) {
      node = 0;
      now.assign(1, (cudaGraphNode_t)(++node));
      const std::vector<cudaGraphNode_t> root = now;
      calls = 0; failAt = f;
      GraphFork fork(nullptr, true);
      std::vector<cudaGraphNode_t> tails;
      bool apart = true;
      for (int k = 0; k < branches; k++) {
        fork.branch();
        apart = apart && launch() == root;
        launch();
        tails.push_back(now[0]);
      }
      fork.join();
      if (f < 0) {
        assert(fork.error() == cudaSuccess && apart && now == tails);
        total = calls;
        assert(total > 2 * branches);
      } else {
        assert(fork.error() == cudaErrorMemoryAllocation);
      }
    }
  }
  failAt = -1;
  // not capturing: in order, no error
  status = cudaStreamCaptureStatusNone;
  GraphFork none(nullptr, true);
  none.branch(); none.branch(); none.join();
  assert(none.error() == cudaSuccess);
  // invalidated before or between the branches: reported
  status = cudaStreamCaptureStatusInvalidated;
  GraphFork bad(nullptr, true);
  bad.branch(); bad.join();
  assert(bad.error() != cudaSuccess);
  status = cudaStreamCaptureStatusActive;
  GraphFork late(nullptr, true);
  late.branch();
  status = cudaStreamCaptureStatusInvalidated;
  late.branch(); late.join();
  assert(late.error() != cudaSuccess);
  // off: not one call
  calls = 0;
  GraphFork off(nullptr, false);
  off.branch(); off.join();
  assert(calls == 0 && off.error() == cudaSuccess);
}
""")
