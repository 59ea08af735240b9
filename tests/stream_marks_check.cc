// Host checks of runtime/stream_mark.h over a CUDA runtime of a few lines: a stream is a count of the work enqueued on it, an
// event the count at which it was recorded.  Exits non-zero at the first check that fails.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>

#include "stream_mark.h"

struct CUstream_st { std::atomic<long> work{0}; long synchronised = -1; };
struct CUevent_st { long at = -1; };

static bool create_fails = false, record_fails = false;
static std::atomic<int> events{0};
static int waits = 0;

extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  if (create_fails) return cudaErrorMemoryAllocation;
  events++;
  *e = new CUevent_st();
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { events--; delete e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  if (record_fails) return cudaErrorLaunchFailure;
  e->at = s->work.load();
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t e, unsigned) { waits += e != nullptr; return e ? cudaSuccess : cudaErrorInvalidResourceHandle; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { s->synchronised = s->work.load(); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

#define CHECK(c)                                                          \
  do {                                                                    \
    if (!(c)) { fprintf(stderr, "line %d: %s\n", __LINE__, #c); exit(1); } \
  } while (0)

using namespace b2x;

int main() {
  {  // two executions record A, then B, and add B, then A: the list has to keep waiting for B
    MarkClock clock;
    CUstream_st s;
    MarkRef a, b;
    s.work = 1;
    CHECK(mark_stream(&clock, &s, &a) == cudaSuccess);
    s.work = 2;
    CHECK(mark_stream(&clock, &s, &b) == cudaSuccess);
    std::vector<MarkRef> list;
    add_mark(&list, b);
    add_mark(&list, a);
    CHECK(list.size() == 1 && list[0]->ev->at == 2);
    list.clear();
    add_mark(&list, a);
    add_mark(&list, b);
    CHECK(list.size() == 1 && list[0]->ev->at == 2);
  }
  {  // the same with threads: enqueue, mark, add
    MarkClock clock;
    CUstream_st s, other;
    std::mutex list_mu;
    std::vector<MarkRef> list;
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; t++)
      threads.emplace_back([&] {
        for (int i = 0; i < 2000; i++) {
          const long mine = ++s.work;
          MarkRef m;
          CHECK(mark_stream(&clock, &s, &m) == cudaSuccess && m->ev->at >= mine);
          std::lock_guard<std::mutex> lk(list_mu);
          add_mark(&list, m);
          CHECK(list.size() == 1 && list[0]->ev->at >= mine);
        }
      });
    for (auto& t : threads) t.join();
    CHECK(list[0]->ev->at == 16000);
    MarkRef m;
    CHECK(mark_stream(&clock, &other, &m) == cudaSuccess);
    add_mark(&list, m);
    CHECK(list.size() == 2);
  }
  {  // the wait on the mark's own stream is left out only for the plugin's streams
    MarkClock clock;
    CUstream_st s, t;
    MarkRef own, foreign;
    CHECK(mark_stream(&clock, &s, &own) == cudaSuccess && mark_stream(nullptr, &t, &foreign) == cudaSuccess);
    waits = 0;
    CHECK(wait_mark(&s, own) == cudaSuccess && waits == 0);
    CHECK(wait_mark(&t, own) == cudaSuccess && waits == 1);
    CHECK(wait_mark(&s, foreign) == cudaSuccess && waits == 2);
    CHECK(wait_mark(&t, foreign) == cudaSuccess && waits == 3);
    CHECK(wait_mark(&s, nullptr) == cudaSuccess && waits == 3);
    std::vector<MarkRef> list;
    add_mark(&list, foreign);
    MarkRef again;
    CHECK(mark_stream(nullptr, &t, &again) == cudaSuccess);
    add_mark(&list, again);
    CHECK(list.size() == 2);
  }
  for (bool* failure : {&create_fails, &record_fails}) {  // no event: the work is waited for, and an earlier mark is not given up
    MarkClock clock;
    CUstream_st s;
    MarkRef before, m;
    s.work = 3;
    CHECK(mark_stream(&clock, &s, &before) == cudaSuccess);
    std::vector<MarkRef> list{before};
    s.work = 4;
    *failure = true;
    CHECK(mark_stream(&clock, &s, &m) == cudaSuccess && !m && s.synchronised == 4);
    *failure = false;
    add_mark(&list, m);
    CHECK(list.size() == 1 && list[0] == before);
  }
  CHECK(events == 0);
  return 0;
}
