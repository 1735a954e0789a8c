// Where the last launch was one of calls that overlap: a kernel that lets what follows begin at its start and did not
// wait for the kernel before it (launch() in ccb_rt.cu). A kernel launched behind it with the programmatic attribute would
// wait for that one alone, while the call before it may still run, so the next launch there is a plain one. Host code
// without CUDA, shared with the CPU test.
#pragma once
#include <atomic>
#include <map>
#include <mutex>
#include <utility>

namespace ccb {

// What a launch goes to. `stream` is the number that CUDA gives a stream for good, not its handle: the default
// streams of all devices have one handle, the per-thread ones of all threads another, and a new stream can get the
// handle of one that is gone. `capture` is the capture's number, 0 outside of one.
struct LaunchPlace {
  int device;
  unsigned long long stream, capture;
};

// Kept for places that are never launched to again too, hence a bound, at which the oldest goes: a
// communicator has two such calls on the device at most, so only with as many streams under way at once would it still matter.
class OverlapNotes {
 public:
  static constexpr size_t kMost = 4096;
  // Nearly always false, and all that a launch looks at then.
  bool any() const { return count_.load(std::memory_order_acquire) != 0; }
  void note(const LaunchPlace& at) {
    std::lock_guard<std::mutex> hold(lock_);
    const Key key = key_of(at);
    auto known = ages_.find(key);
    if (known != ages_.end()) by_age_.erase(known->second);
    else if (ages_.size() >= kMost) {
      ages_.erase(by_age_.begin()->second);
      by_age_.erase(by_age_.begin());
    }
    ages_[key] = ++age_;
    by_age_[age_] = key;
    count_.store(ages_.size(), std::memory_order_release);
  }
  // Whether the next launch at this place has to be a plain one. On a stream that one settles it; a capture's streams
  // may depend on one another in any way, so there all launches from then on are plain.
  bool behind(const LaunchPlace& at) {
    std::lock_guard<std::mutex> hold(lock_);
    auto known = ages_.find(key_of(at));
    if (known == ages_.end()) return false;
    if (!at.capture) {
      by_age_.erase(known->second);
      ages_.erase(known);
      count_.store(ages_.size(), std::memory_order_release);
    }
    return true;
  }
  size_t kept() const { return count_.load(std::memory_order_acquire); }

 private:
  typedef std::pair<int, unsigned long long> Key;   // device and stream, or -1 and the capture
  static Key key_of(const LaunchPlace& at) { return at.capture ? Key(-1, at.capture) : Key(at.device, at.stream); }
  std::mutex lock_;
  std::map<Key, unsigned long long> ages_;
  std::map<unsigned long long, Key> by_age_;
  unsigned long long age_ = 0;
  std::atomic<size_t> count_{0};
};

}  // namespace ccb
