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
