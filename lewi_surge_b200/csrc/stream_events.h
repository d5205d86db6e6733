// Events that tie a side stream to the main one, a set per call.  A call records an event and lets the other stream wait for it in two steps;
// another host thread that recorded the same event in between would make the wait stand for that thread's stream.  So a call holds its set
// alone while it queues its work and gives it back as it returns: a wait has taken down what it waits for when cudaStreamWaitEvent
// returns, and the next call may record the events anew.
// Free sets are kept per device, at most kEventSetsKept of them (as many calls as queue at the same time need); those beyond are destroyed.
#pragma once

#include <cuda_runtime.h>

#include <mutex>

namespace lewi {

struct EventSet {
  cudaEvent_t fork, mid, join;
};

constexpr int kEventDevices = 64, kEventSetsKept = 16;

class EventLease {
 public:
  explicit EventLease(bool wanted) {
    if (!wanted || cudaGetDevice(&dev_) != cudaSuccess || dev_ < 0 || dev_ >= kEventDevices) return;
    {
      Pool& p = pool();
      std::lock_guard<std::mutex> hold(p.lock);
      if (p.n[dev_] > 0) {
        set_ = p.free[dev_][--p.n[dev_]];
        ok_ = true;
        return;
      }
    }
    cudaEvent_t* const made[3] = {&set_.fork, &set_.mid, &set_.join};
    for (int i = 0; i < 3; ++i) {
      if (cudaEventCreateWithFlags(made[i], cudaEventDisableTiming) != cudaSuccess) {
        while (i-- > 0) (void)cudaEventDestroy(*made[i]);
        return;
      }
    }
    ok_ = true;
  }
  ~EventLease() {
    if (!ok_) return;
    {
      Pool& p = pool();
      std::lock_guard<std::mutex> hold(p.lock);
      if (p.n[dev_] < kEventSetsKept) {
        p.free[dev_][p.n[dev_]++] = set_;
        return;
      }
    }
    (void)cudaEventDestroy(set_.fork);
    (void)cudaEventDestroy(set_.mid);
    (void)cudaEventDestroy(set_.join);
  }
  EventLease(const EventLease&) = delete;
  EventLease& operator=(const EventLease&) = delete;
  bool ok() const { return ok_; }
  const EventSet* operator->() const { return &set_; }

 private:
  struct Pool {
    std::mutex lock;
    EventSet free[kEventDevices][kEventSetsKept];
    int n[kEventDevices] = {0};
  };
  static Pool& pool() {
    static Pool* p = new Pool;   // (kept to the end of the process: calls may come from threads that outlive static objects)
    return *p;
  }
  EventSet set_{};
  int dev_ = -1;
  bool ok_ = false;
};

// `waiter` goes on only after what `from` holds so far.
inline bool stream_after(cudaEvent_t ev, cudaStream_t from, cudaStream_t waiter) {
  return cudaEventRecord(ev, from) == cudaSuccess && cudaStreamWaitEvent(waiter, ev, 0) == cudaSuccess;
}

}  // namespace lewi
