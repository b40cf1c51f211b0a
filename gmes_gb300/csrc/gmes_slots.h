// Which barrier slot a cooperative launch meets at (host side; no CUDA here).
//
// The blocks of a one-launch kernel count their arrivals in a slot of device
// memory (gmes_barrier.cuh), and two launches that may run at the same time
// must not share one.  A direct launch takes its stream's slot: the launches of
// a stream run one after another.  A slot is dealt to another stream only when
// the last launch on it has left: launches are numbered per slot, and the
// kernel's last block writes its launch's number to done[slot].  A launch in a
// capture takes a slot that belongs to the graph until the graph, its copies and
// their launches are gone.  With every slot in use there is none to be had, and
// the caller takes the launches per half-step.
#pragma once

#include <cstdint>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace gmes {

class SlotPool {
 public:
  // Slots 0 .. streams - 1 for streams, the graphs after them for captures.
  SlotPool(int streams, int graphs, const volatile uint32_t* done)
      : done_(done), issued_(streams, 0), owner_(streams, 0) {
    for (int k = 0; k < graphs; ++k) graph_slots_.push_back(streams + graphs - 1 - k);
  }

  // The slot of the next launch on the stream of this id (one that no other
  // stream of the process ever has), and the launch's number; -1: none.
  int enter(unsigned long long stream, uint32_t* number) {
    std::lock_guard<std::mutex> lock(mutex_);
    const auto it = by_stream_.find(stream);
    int s = it != by_stream_.end() ? it->second : -1;
    const int n = (int)issued_.size();
    for (int k = 0; k < n && s < 0; ++k) {
      const int c = (hand_ + k) % n;
      if (issued_[c] != done_[c]) continue;  // its last launch is still to leave
      const auto old = by_stream_.find(owner_[c]);
      if (old != by_stream_.end() && old->second == c) by_stream_.erase(old);
      by_stream_[stream] = s = c;
      owner_[c] = stream;
      hand_ = c + 1;
    }
    if (s < 0) return -1;
    *number = ++issued_[s];
    return s;
  }

  int take_graph() {
    std::lock_guard<std::mutex> lock(mutex_);
    if (graph_slots_.empty()) return -1;
    const int s = graph_slots_.back();
    graph_slots_.pop_back();
    return s;
  }
  void give_graph(int slot) {
    std::lock_guard<std::mutex> lock(mutex_);
    graph_slots_.push_back(slot);
  }

 private:
  std::mutex mutex_;
  const volatile uint32_t* done_;
  std::vector<uint32_t> issued_;             // launches dealt, per slot
  std::vector<unsigned long long> owner_;    // stream that a slot was dealt to last
  std::unordered_map<unsigned long long, int> by_stream_;
  std::vector<int> graph_slots_;             // free ones
  int hand_ = 0;
};

}  // namespace gmes
