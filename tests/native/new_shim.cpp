// Test helper, preloaded into a test's own process: the n-th operator new after
// arm_new(n) throws std::bad_alloc.  Test code only.
#include <atomic>
#include <cstdlib>
#include <new>

namespace {
std::atomic<long> left{0};

void *take(std::size_t n) {
  long l = left.load();
  while (l > 0 && !left.compare_exchange_weak(l, l - 1)) {
  }
  return l == 1 ? nullptr : std::malloc(n ? n : 1);
}
void *must(std::size_t n) {
  void *p = take(n);
  if (!p) throw std::bad_alloc();
  return p;
}
}  // namespace

extern "C" void arm_new(long n) { left.store(n); }
extern "C" long new_left(void) { return left.load(); }

void *operator new(std::size_t n) { return must(n); }
void *operator new[](std::size_t n) { return must(n); }
void *operator new(std::size_t n, const std::nothrow_t &) noexcept { return take(n); }
void *operator new[](std::size_t n, const std::nothrow_t &) noexcept { return take(n); }
void operator delete(void *p) noexcept { std::free(p); }
void operator delete[](void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }
void operator delete[](void *p, std::size_t) noexcept { std::free(p); }
