// rgf_inflight.h -- what the solver calls of a process have in flight on each
// GPU (host only, no CUDA).
//
// A call of few tasks may spread each over a cluster of CTAs, which shortens
// it but costs throughput (a cluster of 8 is about 3 times as fast as one
// CTA).  That pays on SMs that would idle, not on those that other contexts'
// calls fill, so every call puts its tasks up here while it runs and the
// launch geometry counts the others'.
#pragma once
#include <algorithm>
#include <cstdint>
#include <functional>
#include <list>
#include <mutex>
#include <vector>

namespace rgf {

class InFlight {
  struct Entry {
    int dev;
    const void* lane;   // calls of one stream follow one another
    int64_t tasks;
    void* done;         // asked whether the call is over; NULL: as long as the entry stands
  };
  std::mutex mu_;
  std::list<Entry> entries_;

 public:
  // A call's entry, taken down with the ticket.
  class Ticket {
    InFlight* board_ = nullptr;
    std::list<Entry>::iterator at_;

   public:
    Ticket() = default;
    Ticket(InFlight& b, int dev, const void* lane, int64_t tasks) : board_(&b) {
      std::lock_guard<std::mutex> l(b.mu_);
      at_ = b.entries_.insert(b.entries_.end(), Entry{dev, lane, tasks, nullptr});
    }
    Ticket(Ticket&& o) noexcept : board_(o.board_), at_(o.at_) { o.board_ = nullptr; }
    Ticket& operator=(Ticket&& o) noexcept {
      reset();
      board_ = o.board_;
      at_ = o.at_;
      o.board_ = nullptr;
      return *this;
    }
    ~Ticket() { reset(); }
    void reset() {
      if (!board_) return;
      std::lock_guard<std::mutex> l(board_->mu_);
      board_->entries_.erase(at_);
      board_ = nullptr;
    }
    // the call went on without its caller: it is over when `done` says so
    void until(void* done) {
      if (!board_) return;
      std::lock_guard<std::mutex> l(board_->mu_);
      at_->done = done;
    }
  };

  // Tasks of the calls that may run beside one on `lane`: the largest ones,
  // as many as the GPU takes from different streams at a time.
  int64_t others(int dev, const void* lane, int streams, const std::function<bool(void*)>& over) {
    std::vector<int64_t> t;
    {
      std::lock_guard<std::mutex> l(mu_);
      for (const Entry& e : entries_)
        if (e.dev == dev && e.lane != lane && !(e.done && over(e.done))) t.push_back(e.tasks);
    }
    std::sort(t.begin(), t.end(), std::greater<int64_t>());
    int64_t sum = 0;
    for (size_t i = 0; i < t.size() && (int)i < streams - 1; i++) sum += t[i];
    return sum;
  }
};

}  // namespace rgf
