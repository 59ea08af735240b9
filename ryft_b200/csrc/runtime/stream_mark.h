// Points in a stream's work, and who has to wait for them.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <mutex>
#include <utility>
#include <vector>

namespace b2x {
// An event recorded once and never again, shared by everything that has to know when the stream has got there (the outputs
// of an execution, the views it read, its completion).  One event per execution instead of one per output, argument and
// completion: creating, recording and destroying them was a third of the execute call.
struct StreamMark {
  cudaEvent_t ev = nullptr;
  // The plugin's own stream that the mark lies on; null on a caller's.  Only the plugin's streams are told apart by their
  // handles: they live as long as the client, while a caller's handle can stand for another stream in another thread
  // (cudaStreamPerThread) or, once the stream has been destroyed, for a new one.
  cudaStream_t stream = nullptr;
  uint64_t order = 0;             // of two marks on one of the plugin's streams, the later one has the larger number
  StreamMark() = default;
  StreamMark(const StreamMark&) = delete;
  StreamMark& operator=(const StreamMark&) = delete;
  ~StreamMark() { if (ev) cudaEventDestroy(ev); }
};
using MarkRef = std::shared_ptr<StreamMark>;   // null: nothing to wait for

// Numbers the marks of a device's streams in the order in which they are recorded.
struct MarkClock {
  std::mutex mu;
  uint64_t last = 0;
};

// Records a mark behind the work that `stream` holds now (the stream's device must be current); `clock` is the device's for
// one of the plugin's streams and null for a caller's.  Where no event can be had, the work is waited for right here and the
// mark is null; an error means that the work itself has failed or cannot be waited for.
inline cudaError_t mark_stream(MarkClock* clock, cudaStream_t stream, MarkRef* out) {
  out->reset();
  MarkRef m = std::make_shared<StreamMark>();
  cudaError_t e = cudaEventCreateWithFlags(&m->ev, cudaEventDisableTiming);
  if (e != cudaSuccess) m->ev = nullptr;
  else if (clock) {
    std::lock_guard<std::mutex> lk(clock->mu);   // number and record together: two threads may be marking one stream
    m->stream = stream;
    m->order = ++clock->last;
    e = cudaEventRecord(m->ev, stream);
  } else {
    e = cudaEventRecord(m->ev, stream);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return cudaStreamSynchronize(stream);
  }
  *out = std::move(m);
  return cudaSuccess;
}

// Makes `stream` wait for a mark; nothing to do when the mark lies on the stream itself.
inline cudaError_t wait_mark(cudaStream_t stream, const MarkRef& m) {
  if (!m || (m->stream && m->stream == stream)) return cudaSuccess;
  return cudaStreamWaitEvent(stream, m->ev, 0);
}

// Remembers a reader.  The later of two marks of one stream covers the earlier one, whichever is added first (executions
// on two threads record their marks in one order and may add them in the other), so the list holds one per stream.
inline void add_mark(std::vector<MarkRef>* marks, MarkRef m) {
  if (!m) return;
  if (m->stream)
    for (auto& o : *marks)
      if (o->stream == m->stream) {
        if (o->order < m->order) o = std::move(m);
        return;
      }
  marks->push_back(std::move(m));
}
}  // namespace b2x
