// Streams for pieces of work side by side: forked from a stream, each piece on
// a side stream that starts after that stream's work so far, and joined to it
// again. Api names the calls (CudaForks below; host code only).
#pragma once
#include <cstddef>
#include <vector>

#include <cuda_runtime.h>

namespace icx {

struct CudaForks {
  static cudaError_t make_stream(cudaStream_t* s) { return cudaStreamCreateWithFlags(s, cudaStreamNonBlocking); }
  static cudaError_t make_event(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, cudaEventDisableTiming); }
  static void drop_stream(cudaStream_t s) { cudaStreamDestroy(s); }
  static void drop_event(cudaEvent_t e) { cudaEventDestroy(e); }
  static cudaError_t record(cudaEvent_t e, cudaStream_t s) { return cudaEventRecord(e, s); }
  static cudaError_t wait(cudaStream_t s, cudaEvent_t e) { return cudaStreamWaitEvent(s, e, 0); }
};

template <class Api>
class Forks {
  struct Side {
    cudaStream_t stream = nullptr;
    cudaEvent_t joined = nullptr;
  };
  std::vector<Side> side;
  cudaEvent_t forked = nullptr;

  // n side streams with their events: both of a pair or neither
  cudaError_t reserve(size_t n) {
    cudaError_t e = cudaSuccess;
    if (n > 0 && !forked && (e = Api::make_event(&forked)) != cudaSuccess) {
      forked = nullptr;
      return e;
    }
    while (side.size() < n) {
      Side s;
      if ((e = Api::make_stream(&s.stream)) != cudaSuccess) return e;
      if ((e = Api::make_event(&s.joined)) != cudaSuccess) {
        Api::drop_stream(s.stream);
        return e;
      }
      side.push_back(s);
    }
    return cudaSuccess;
  }

 public:
  Forks() = default;
  Forks(const Forks&) = delete;
  Forks& operator=(const Forks&) = delete;
  void release() {
    for (const Side& s : side) {
      Api::drop_stream(s.stream);
      Api::drop_event(s.joined);
    }
    side.clear();
    if (forked) Api::drop_event(forked);
    forked = nullptr;
  }

  // f(k, stream) for k < n: the pieces for which alone(k) holds on q, one after
  // the other (the last piece where it holds for none), the others on side
  // streams that q then waits for. Works the same under stream capture (fork
  // and join become edges of the graph).
  template <class A, class F>
  cudaError_t run(size_t n, cudaStream_t q, const A& alone, const F& f) {
    if (n == 0) return cudaSuccess;
    std::vector<size_t> aside, on_q;
    for (size_t k = 0; k < n; ++k) (alone(k) ? on_q : aside).push_back(k);
    if (on_q.empty()) {
      on_q.push_back(aside.back());
      aside.pop_back();
    }
    cudaError_t e = reserve(aside.size());
    if (e == cudaSuccess && !aside.empty()) e = Api::record(forked, q);
    size_t begun = 0;
    for (size_t k = 0; k < aside.size() && e == cudaSuccess; ++k) {
      if ((e = Api::wait(side[k].stream, forked)) != cudaSuccess) break;
      ++begun;
      e = f(aside[k], side[k].stream);
    }
    for (size_t k = 0; k < on_q.size() && e == cudaSuccess; ++k) e = f(on_q[k], q);
    // every stream begun is joined, also after an error
    for (size_t k = 0; k < begun; ++k) {
      cudaError_t j = Api::record(side[k].joined, side[k].stream);
      if (j == cudaSuccess) j = Api::wait(q, side[k].joined);
      if (e == cudaSuccess) e = j;
    }
    return e;
  }
};

}  // namespace icx
