// Host work over a few threads: memcpy / memcmp of large arrays, numbered pieces of a loop.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace mpsw {

// f(part, begin, end) over the bytes: four parts of at least 2 MB, or one
template <typename F>
inline void in_parts(size_t bytes, F &&f) {
  constexpr size_t kPart = (size_t)2 << 20;
  const int parts = (int)std::min<size_t>(4, bytes / kPart);
  if (parts < 2) {
    f(0, 0, bytes);
    return;
  }
  std::vector<std::thread> ts;
  const size_t step = (bytes / parts + 63) / 64 * 64;
  auto part = [&](int i) { f(i, i * step, i + 1 < parts ? (i + 1) * step : bytes); };
  int i = 1;
  try {
    ts.reserve(parts - 1);
    for (; i < parts; i++) ts.emplace_back(part, i);
  } catch (const std::exception &) {  // no more threads, or no memory for one: the rest here
  }
  for (; i < parts; i++) part(i);
  part(0);
  for (auto &t : ts) t.join();
}
inline void copy_bytes(void *dst, const void *src, size_t bytes) {
  in_parts(bytes, [=](int, size_t a, size_t b) { std::memcpy((char *)dst + a, (const char *)src + a, b - a); });
}
inline bool same_bytes(const void *x, const void *y, size_t bytes) {
  bool eq[4] = {true, true, true, true};
  in_parts(bytes, [&](int i, size_t a, size_t b) { eq[i] = !std::memcmp((const char *)x + a, (const char *)y + a, b - a); });
  return eq[0] && eq[1] && eq[2] && eq[3];
}

// f(0) .. f(n - 1), in any order over up to eight threads; the first exception of one is thrown on
template <typename F>
inline void in_turns(int n, F &&f) {
  std::atomic<int> next{0};
  std::exception_ptr err;
  std::mutex lock;
  auto work = [&] {
    for (int i; (i = next++) < n;) try {
        f(i);
      } catch (...) {
        std::lock_guard<std::mutex> g(lock);
        if (!err) err = std::current_exception();
      }
  };
  std::vector<std::thread> ts;
  const int extra = std::min(std::min(n, 8), (int)std::thread::hardware_concurrency()) - 1;
  try {
    ts.reserve(std::max(extra, 0));
    for (int i = 0; i < extra; i++) ts.emplace_back(work);
  } catch (const std::exception &) {  // no more threads, or no memory for one
  }
  work();
  for (auto &t : ts) t.join();
  if (err) std::rethrow_exception(err);
}

}  // namespace mpsw
