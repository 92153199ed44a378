// Counter pairs of the work queues (queue.cuh): who has which.  No CUDA in here.
#pragma once
#include <cstdint>
#include <mutex>

namespace fa {

// Two launches that run at the same time must not have the same pair: each would skip what the other has drawn.  Launches of a stream run
// one behind the other, so a stream has one pair, for good (a stream's id is not given to another one later, as its handle may be).  A launch
// that is captured into a graph may run beside any stream at any time: it has a pair to itself for as long as the graph lives.
// (Pairs in rotation, 64 of them, held only while fewer launches than that were under way, and a replayed graph keeps its pair over any number.)
// Tables of fixed size: nothing here throws, and one that stands in static memory needs neither a start nor an end.
template <int kStreams, int kCaptured> class QueueSlots {
 public:
  static constexpr int kPairs = kStreams + kCaptured;
  static constexpr int kNone = -1;    // no pair left that only this launch can have

  int of_stream(uint64_t id) {
    std::lock_guard<std::mutex> lock(mu_);
    uint32_t at = (uint32_t)((id * 0x9E3779B97F4A7C15u) >> 32) % kTable;
    for (; table_[at].pair != 0; at = (at + 1) % kTable)
      if (table_[at].id == id) return table_[at].pair - 1;
    if (streams_ == kStreams) return kNone;
    table_[at] = {id, ++streams_};
    return streams_ - 1;
  }
  int take() {
    std::lock_guard<std::mutex> lock(mu_);
    if (given_ > 0) return list_[--given_];
    return used_ == kCaptured ? kNone : kStreams + used_++;
  }
  void give(int i) {
    std::lock_guard<std::mutex> lock(mu_);
    list_[given_++] = i;
  }
  int taken() {
    std::lock_guard<std::mutex> lock(mu_);
    return used_ - given_;
  }

 private:
  static constexpr uint32_t kTable = 2 * kStreams;    // open addressing: at least half of it is free
  struct Entry {
    uint64_t id;
    int pair;                          // + 1; 0: free
  };
  std::mutex mu_;
  Entry table_[kTable] = {};
  int list_[kCaptured] = {};           // pairs given back
  int streams_ = 0, used_ = 0, given_ = 0;
};

}  // namespace fa
