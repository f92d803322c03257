// Which streams have work in flight that reads something, as far as the next
// writer has to know.
#pragma once

#include <atomic>

namespace krr {

// Streams by their ids, which a process never gives twice.  Readers call
// read(), a writer asks alone_on() and, when what was in flight before it has
// ended or is ordered before it, calls start_over().  Once a reader was
// captured into a graph, which may be launched on any stream at any time, no
// stream is alone any more.
class StreamUse {
  public:
    using Id = unsigned long long;

    void read(Id stream) {
        Id seen = kNone;
        if (!seen_.compare_exchange_strong(seen, stream) && seen != stream) seen_.store(kSeveral);
    }
    void read_captured() { captured_.store(true); }
    bool alone_on(Id stream) const {
        const Id seen = seen_.load();
        return !captured_.load() && (seen == kNone || seen == stream);
    }
    void start_over() { seen_.store(kNone); }

  private:
    static constexpr Id kNone = ~0ull, kSeveral = ~0ull - 1;
    std::atomic<Id> seen_{kNone};
    std::atomic<bool> captured_{false};
};

}  // namespace krr
