// chains.h -- launches that run side by side: the streams of an eager batch
// step.  Host code; of CUDA it calls the runtime's stream and event functions
// only.
#pragma once
#include <cuda_runtime_api.h>

#include <algorithm>
#include <vector>

namespace grim {

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
