// Host memory for the final fields of an ensemble's requests.
#pragma once
#include <stddef.h>
#include <stdlib.h>
#include <map>
#include <mutex>

namespace mhit {

// A released request's buffers are kept for the next ones (up to kMost bytes,
// freed with the pool): a fresh one costs a page fault per 4 KB, half of a
// 96^3 request's download.
class HostPool {
 public:
  static constexpr size_t kMost = (size_t)512 << 20;
  double* take(size_t count) {
    {
      std::lock_guard<std::mutex> g(mu_);
      auto it = free_.find(count);
      if (it != free_.end()) {
        double* p = it->second;
        free_.erase(it);
        kept_ -= count * sizeof(double);
        return p;
      }
    }
    return static_cast<double*>(malloc(count * sizeof(double)));
  }
  void give(double* p, size_t count) {
    if (!p) return;
    {
      std::lock_guard<std::mutex> g(mu_);
      if (kept_ + count * sizeof(double) <= kMost) {
        try {
          free_.emplace(count, p);
          kept_ += count * sizeof(double);
          return;
        } catch (...) {  // no room for the entry: the buffer is freed
        }
      }
    }
    free(p);
  }
  HostPool() = default;
  HostPool(const HostPool&) = delete;
  HostPool& operator=(const HostPool&) = delete;
  ~HostPool() {
    for (auto& b : free_) free(b.second);
  }

 private:
  std::mutex mu_;
  std::multimap<size_t, double*> free_;
  size_t kept_ = 0;
};

// The final fields of one request: all of them, or none.  A buffer of the pool
// holds an earlier request's values until it is filled, so a field that
// could not be filled takes the others with it.
class ResultFields {
 public:
  // Takes nf buffers of `count` values and fills each with get(buffer, field).
  // Returns get's first error (or `nomem`); then no field is held.
  template <class Error, class Get> Error fill(HostPool* pool, int nf, size_t count, Error nomem, const Get& get) {
    drop();
    pool_ = pool;
    count_ = count;
    for (int f = 0; f < nf; ++f) {
      p_[f] = pool->take(count);
      const Error e = p_[f] ? get(p_[f], f) : nomem;
      if (e != Error()) {
        drop();
        return e;
      }
    }
    return Error();
  }
  void drop() {
    for (double*& p : p_) {
      if (p) pool_->give(p, count_);
      p = nullptr;
    }
  }
  bool held() const { return p_[0] != nullptr; }
  const double* field(int f) const { return p_[f]; }  // null: not kept
  size_t count() const { return count_; }

  ResultFields() = default;
  ResultFields(const ResultFields&) = delete;
  ResultFields& operator=(const ResultFields&) = delete;
  ~ResultFields() { drop(); }

 private:
  HostPool* pool_ = nullptr;
  double* p_[4] = {nullptr, nullptr, nullptr, nullptr};
  size_t count_ = 0;
};

}  // namespace mhit
