#pragma once
// A few host threads kept for the copies between callers' pageable memory and pinned
// staging: starting threads for every copy costs as much as copying megabytes. One
// pool serves one engine (one call at a time); its threads end with it.
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <functional>
#include <mutex>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

namespace rtg {

class HostPool {
 public:
  HostPool() = default;
  ~HostPool() {
    {
      std::lock_guard<std::mutex> g(m_);
      stop_ = true;
    }
    wake_.notify_all();
    for (auto& t : threads_) t.join();
  }
  HostPool(const HostPool&) = delete;
  HostPool& operator=(const HostPool&) = delete;

  // Runs f(0) .. f(n - 1), the caller taking part; returns when all have run. f must
  // not throw.
  void run(std::size_t n, const std::function<void(std::size_t)>& f) {
    if (n < 2) {
      if (n) f(0);
      return;
    }
    start();
    {
      std::lock_guard<std::mutex> g(m_);
      f_ = &f;
      n_ = n;
      next_.store(0, std::memory_order_relaxed);
      busy_ = threads_.size();
      ++round_;
    }
    wake_.notify_all();
    for (std::size_t k; (k = next_.fetch_add(1)) < n;) f(k);
    std::unique_lock<std::mutex> g(m_);
    idle_.wait(g, [&] { return busy_ == 0; });
  }

  // memcpy, split over the threads when it is worth waking them.
  void copy(void* dst, const void* src, std::size_t bytes) {
    constexpr std::size_t kPiece = std::size_t(1) << 17;
    if (bytes < 2 * kPiece) {
      std::memcpy(dst, src, bytes);
      return;
    }
    run((bytes + kPiece - 1) / kPiece, [=](std::size_t k) {
      const std::size_t at = k * kPiece;
      std::memcpy(static_cast<unsigned char*>(dst) + at, static_cast<const unsigned char*>(src) + at,
                  std::min(kPiece, bytes - at));
    });
  }

  // Writes a byte to every page of buffers that are about to be filled, when they are
  // large: fresh memory (an allocation that malloc maps anew each time) is then zeroed
  // by all threads at once, each in huge pages of its own. Left to the copies, which work
  // on a few megabytes at a time, two or three threads zero and the others wait (64 images,
  // 58 MB: 9.2 ms, with this 5.0).
  void touch(const std::vector<std::pair<void*, std::size_t>>& buffers) {
    constexpr std::uintptr_t kHuge = std::uintptr_t(1) << 21, kPage = 4096;
    std::size_t total = 0;
    for (const auto& b : buffers) total += b.second;
    if (total < (std::size_t(16) << 20)) return;
    std::vector<std::pair<std::uintptr_t, std::uintptr_t>> parts;
    for (const auto& b : buffers) {
      const std::uintptr_t end = reinterpret_cast<std::uintptr_t>(b.first) + b.second;
      for (std::uintptr_t at = reinterpret_cast<std::uintptr_t>(b.first); at < end;) {
        const std::uintptr_t next = std::min(end, (at | (kHuge - 1)) + 1);
        parts.emplace_back(at, next);
        at = next;
      }
    }
    run(parts.size(), [&parts](std::size_t k) {
      for (std::uintptr_t at = parts[k].first; at < parts[k].second; at = (at | (kPage - 1)) + 1)
        *reinterpret_cast<volatile unsigned char*>(at) = 0;
    });
  }

 private:
  void start() {
    if (!threads_.empty()) return;
    const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
    const unsigned workers = std::min(7u, cores > 1 ? cores - 1 : 0u);
    try {
      for (unsigned w = 0; w < workers; ++w) threads_.emplace_back([this] { work(); });
    } catch (const std::system_error&) {
      // No more threads to be had: those there are, or the caller alone, do the work.
    }
  }
  void work() {
    std::size_t seen = 0;
    std::unique_lock<std::mutex> g(m_);
    while (true) {
      wake_.wait(g, [&] { return stop_ || round_ != seen; });
      if (stop_) return;
      seen = round_;
      const std::function<void(std::size_t)>& f = *f_;
      const std::size_t n = n_;
      g.unlock();
      for (std::size_t k; (k = next_.fetch_add(1)) < n;) f(k);
      g.lock();
      if (--busy_ == 0) idle_.notify_one();
    }
  }

  std::vector<std::thread> threads_;
  std::mutex m_;
  std::condition_variable wake_, idle_;
  const std::function<void(std::size_t)>* f_ = nullptr;
  std::size_t n_ = 0, busy_ = 0, round_ = 0;
  std::atomic<std::size_t> next_{0};
  bool stop_ = false;
};

}  // namespace rtg
