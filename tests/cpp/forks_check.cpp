// icx::Forks over calls that only note what they were asked (no GPU, no CUDA
// runtime): streams and events are numbered as they are made, a chosen creation
// fails. Every check prints "FAIL ..." and the program returns 1 if one fails.
#include <cstdio>
#include <map>
#include <set>
#include <string>

#include "icx_forks.h"

static int n_made, fail_at, live;
static std::set<long> alive;
static std::map<cudaEvent_t, cudaStream_t> recorded;  // event -> the stream it marks
static std::map<cudaStream_t, std::set<cudaStream_t>> after;

struct Fake {
  template <class H>
  static cudaError_t make(H* h) {
    if (++n_made == fail_at) return cudaErrorMemoryAllocation;
    *h = reinterpret_cast<H>((long)(n_made + 100));
    alive.insert(n_made + 100);
    ++live;
    return cudaSuccess;
  }
  template <class H>
  static void drop(H h) {
    if (!alive.erase(reinterpret_cast<long>(h))) {
      std::printf("FAIL dropped twice or never made\n");
      fail_at = -1;
    }
    --live;
  }
  static bool known(const void* h) { return alive.count(reinterpret_cast<long>(h)) || h == nullptr; }
  static cudaError_t make_stream(cudaStream_t* s) { return make(s); }
  static cudaError_t make_event(cudaEvent_t* e) { return make(e); }
  static void drop_stream(cudaStream_t s) { drop(s); }
  static void drop_event(cudaEvent_t e) { drop(e); }
  static cudaError_t record(cudaEvent_t e, cudaStream_t s) {
    if (!e || !known(e) || !known(s)) return cudaErrorInvalidResourceHandle;
    recorded[e] = s;
    return cudaSuccess;
  }
  static cudaError_t wait(cudaStream_t s, cudaEvent_t e) {
    if (!e || !known(e) || !recorded.count(e)) return cudaErrorInvalidResourceHandle;
    after[s].insert(recorded[e]);
    return cudaSuccess;
  }
};

static int bad = 0;
#define CHECK(c)                                       \
  do {                                                 \
    if (!(c)) {                                        \
      std::printf("FAIL line %d: %s\n", __LINE__, #c); \
      bad = 1;                                         \
    }                                                  \
  } while (0)

int main() {
  const cudaStream_t q = nullptr;
  const auto none = [](size_t) { return false; };
  // each creation in turn fails; the call after it has all it needs
  for (int n = 1; n <= 4; ++n)
    for (int k = 1; k <= 2 * n; ++k) {
      icx::Forks<Fake> forks;
      n_made = 0;
      fail_at = k;
      const int calls = 2 * (n - 1) + (n > 1);
      std::set<cudaStream_t> used;
      auto f = [&](size_t, cudaStream_t t) {
        CHECK(used.insert(t).second);
        return cudaSuccess;
      };
      const cudaError_t e = forks.run(n, q, none, f);
      CHECK((e == cudaSuccess) == (k > calls));
      CHECK(e == cudaSuccess || used.empty());
      fail_at = 0;
      used.clear();
      after.clear();
      CHECK(forks.run(n, q, none, f) == cudaSuccess);
      CHECK((int)used.size() == n && used.count(q));
      for (cudaStream_t t : used)  // forked from q and joined to it
        if (t != q) CHECK(after[t].count(q) && after[q].count(t));
      forks.release();
      CHECK(live == 0);
    }
  // pieces that run alone: on q, in their order; the others have a side stream each
  for (unsigned mask = 1; mask < 32; ++mask) {
    icx::Forks<Fake> forks;
    after.clear();
    size_t last = 0;
    std::set<cudaStream_t> used;
    CHECK(forks.run(5, q, [&](size_t k) { return (mask >> k & 1) != 0; }, [&](size_t k, cudaStream_t t) {
      if (mask >> k & 1) {
        CHECK(t == q && last <= k);
        last = k;
      } else {
        CHECK(t != q && used.insert(t).second);
      }
      return cudaSuccess;
    }) == cudaSuccess);
    for (cudaStream_t t : used) CHECK(after[t].count(q) && after[q].count(t));
    forks.release();
  }
  // a piece that fails: the streams begun are joined all the same
  icx::Forks<Fake> forks;
  after.clear();
  std::set<cudaStream_t> used;
  CHECK(forks.run(4, q, none, [&](size_t k, cudaStream_t t) {
    used.insert(t);
    return k == 1 ? cudaErrorLaunchFailure : cudaSuccess;
  }) == cudaErrorLaunchFailure);
  CHECK(used.size() == 2);
  for (cudaStream_t t : used) CHECK(after[q].count(t));
  CHECK(forks.run(0, q, none, [&](size_t, cudaStream_t) { return cudaErrorUnknown; }) == cudaSuccess);
  forks.release();
  if (!bad) std::printf("ok\n");
  return bad;
}
