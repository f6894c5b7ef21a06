// Host run of numbered pieces over threads (compiled by tests/test_turns.py).
#include <atomic>
#include <cstdlib>
#include <new>
#include <stdexcept>

#include "mpsw_parts.h"

static std::atomic<int> g_left{-1};  // allocations until one fails (-1: none fails)

void *operator new(size_t n) {
  if (g_left >= 0 && g_left-- == 0) throw std::bad_alloc();
  if (void *p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

int main(int, char **argv) {
  const int n = std::atoi(argv[1]), bad = std::atoi(argv[3]);  // pieces; the one that throws (-1: none)
  std::atomic<int> ran[64] = {};
  bool thrown = false;
  g_left = std::atoi(argv[2]);
  try {
    mpsw::in_turns(n, [&](int i) {
      ran[i]++;
      if (i == bad) throw std::out_of_range("piece");
    });
  } catch (const std::out_of_range &) {
    thrown = true;
  }
  g_left = -1;
  for (int i = 0; i < 64; i++)
    if (ran[i] != (i < n)) return 1;
  return thrown == (bad >= 0) ? 0 : 2;
}
