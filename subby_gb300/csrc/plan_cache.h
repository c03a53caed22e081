// Prepared plans by key, for the serving engine (server.cu; host code, one
// thread).  A plan is PINNED from the moment it is handed out until the run
// that uses it is over (or never started); a key may be pinned several times,
// by several jobs of one run.  The cache holds at most `capacity` plans that
// nothing pins, least recently used first out: pinned plans are never
// destroyed, so a run may hold more of them than the cache keeps.
#pragma once
#include <cstddef>
#include <cstdint>
#include <iterator>
#include <list>
#include <unordered_map>

namespace subby {

// Plan: a pointer type; Destroy: a callable on it.
template <class Plan, class Destroy>
class PlanCache {
 public:
  explicit PlanCache(Destroy destroy) : destroy_(destroy) {}
  size_t size() const { return plans_.size(); }

  // The plan of `key`, pinned and most recently used; nullptr when missing.
  Plan take(uint64_t key) {
    auto it = plans_.find(key);
    if (it == plans_.end()) return nullptr;
    lru_.splice(lru_.begin(), lru_, it->second.lru);
    it->second.pins += 1;
    return it->second.plan;
  }

  // A new plan (its key is missing), pinned and most recently used.
  void add(uint64_t key, Plan plan, size_t capacity) {
    lru_.push_front(key);
    plans_[key] = Entry{plan, 1, lru_.begin()};
    trim(capacity);
  }

  // One pin of `key` fewer; returns its plan.
  Plan drop(uint64_t key) {
    auto it = plans_.find(key);
    if (it == plans_.end() || it->second.pins < 1) return nullptr;
    it->second.pins -= 1;
    return it->second.plan;
  }

  bool pinned(uint64_t key) const {
    auto it = plans_.find(key);
    return it != plans_.end() && it->second.pins > 0;
  }

  // Destroys least recently used plans that nothing pins until `capacity`
  // plans are left.
  void trim(size_t capacity) {
    for (auto r = lru_.end(); plans_.size() > capacity && r != lru_.begin();) {
      --r;
      auto it = plans_.find(*r);
      if (it->second.pins > 0) continue;
      destroy_(it->second.plan);
      plans_.erase(it);
      r = lru_.erase(r);
    }
  }

  void clear() {
    for (auto &kv : plans_) destroy_(kv.second.plan);
    plans_.clear();
    lru_.clear();
  }

 private:
  struct Entry {
    Plan plan;
    int pins;
    std::list<uint64_t>::iterator lru;
  };
  std::unordered_map<uint64_t, Entry> plans_;
  std::list<uint64_t> lru_;   // most recently used first
  Destroy destroy_;
};

}  // namespace subby
