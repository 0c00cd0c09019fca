// chains.h -- launches that run side by side: the branches of a captured
// graph and the streams of an eager batch step.  Host code; of CUDA it calls
// the runtime's stream, event and capture functions only.
#pragma once
#include <cuda_runtime_api.h>

#include <algorithm>
#include <vector>

namespace grim {

// Parallel branches of a graph being captured on one stream: each branch's
// first launch depends on what the fork's did, and what follows join()
// depends on every branch's last launches.  Works on the capture's
// dependency set directly, so a first step needs no side streams or events
// (making three streams and four events took 0.35 ms of a new handle's first
// pass).  Inactive (one stream, in order) when the stream is not capturing.
// These calls are all that orders the branches: after one has failed the
// capture may lack a dependency, and whoever ends it must drop the graph when
// error() is set.
class GraphFork {
 public:
  GraphFork(cudaStream_t s, bool on) : s_(s), on_(on) {
    if (on_) on_ = deps(root_);
  }
  void branch() {
    if (!on_) return;
    if (open_) deps(tails_);
    set(root_);
    open_ = true;
  }
  void join() {
    if (!on_ || !open_) return;
    deps(tails_);
    set(tails_);
    on_ = false;
  }
  cudaError_t error() const { return error_; }

 private:
  // adds the capture's dependency set to out; false when there is none to
  // branch (not capturing, or the query failed)
  bool deps(std::vector<cudaGraphNode_t>& out) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    const cudaGraphNode_t* d = nullptr;
    size_t n = 0;
    cudaError_t e = cudaStreamGetCaptureInfo_v2(s_, &st, nullptr, nullptr, &d, &n);
    if (e == cudaSuccess && (st == cudaStreamCaptureStatusInvalidated || (open_ && st != cudaStreamCaptureStatusActive)))
      e = cudaErrorStreamCaptureInvalidated;
    note(e);
    if (e != cudaSuccess || st != cudaStreamCaptureStatusActive) return false;
    out.insert(out.end(), d, d + n);
    return true;
  }
  void set(std::vector<cudaGraphNode_t>& nodes) {
    note(cudaStreamUpdateCaptureDependencies(s_, nodes.data(), nodes.size(), cudaStreamSetCaptureDependencies));
  }
  void note(cudaError_t e) {
    if (error_ == cudaSuccess) error_ = e;
  }
  cudaStream_t s_;
  bool on_, open_ = false;
  cudaError_t error_ = cudaSuccess;
  std::vector<cudaGraphNode_t> root_, tails_;
};

// Streams and events of a batch's chains, and which problem runs on which.
// make() fills all of it or nothing: a creation that fails leaves the set as
// it was, so that the next step makes it anew.
struct Chains {
  std::vector<cudaStream_t> stream;
  std::vector<cudaEvent_t> join;  // per stream
  cudaEvent_t fork = nullptr;
  std::vector<int> of;  // per problem

  bool made() const { return !of.empty(); }

  // the problems, in `order`, dealt to at most `most` streams so that each
  // carries about the same work
  cudaError_t make(const std::vector<long long>& work, const std::vector<int>& order, int most) {
    Chains c;
    cudaError_t e = c.create((int)std::min<size_t>(work.size(), (size_t)most));
    if (e != cudaSuccess) {
      c.release();
      return e;
    }
    std::vector<long long> load(c.stream.size(), 0);
    c.of.resize(work.size());
    for (int p : order) {
      const int k = (int)(std::min_element(load.begin(), load.end()) - load.begin());
      c.of[p] = k;
      load[k] += work[p];
    }
    std::swap(*this, c);
    c.release();
    return cudaSuccess;
  }

  void release() {
    for (cudaStream_t s : stream) cudaStreamDestroy(s);
    for (cudaEvent_t e : join) cudaEventDestroy(e);
    if (fork) cudaEventDestroy(fork);
    *this = Chains();
  }

 private:
  cudaError_t create(int n) {
    cudaError_t e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
    for (int k = 0; k < n && e == cudaSuccess; k++) {
      cudaStream_t s = nullptr;
      cudaEvent_t v = nullptr;
      e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
      if (e == cudaSuccess) {
        stream.push_back(s);
        e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
      }
      if (e == cudaSuccess) join.push_back(v);
    }
    return e;
  }
};

}  // namespace grim
