// Host run of copies in parts (compiled by tests/test_parts.py): memory runs out at the n-th allocation.
#include <atomic>
#include <cstdlib>
#include <new>
#include <vector>

#include "mpsw_parts.h"

static std::atomic<int> g_left{-1};  // allocations until one fails (-1: none fails)

void *operator new(size_t n) {
  if (g_left >= 0 && g_left-- == 0) throw std::bad_alloc();
  if (void *p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

int main(int argc, char **argv) {
  const size_t n = (size_t)9 << 20;
  std::vector<char> a(n), b(n);
  for (size_t i = 0; i < n; i++) a[i] = (char)(i * 7 + i / 4096);
  g_left = std::atoi(argv[argc - 1]);
  mpsw::copy_bytes(b.data(), a.data(), n);
  g_left = -1;
  if (!mpsw::same_bytes(a.data(), b.data(), n)) return 1;
  b[n - 1]++;
  return mpsw::same_bytes(a.data(), b.data(), n) ? 2 : 0;
}
