// Host loops of the upload and download paths over several threads.
//
// These loops read the caller's FP64 arrays once (16 bytes per complex element) and write FP32; one
// thread does that at a few GB/s, page faults of fresh buffers included, while the copy to the
// device runs at tens.  Threads are started per call: no pool outlives it.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdlib>
#include <exception>
#include <memory>
#include <new>
#include <thread>

namespace totem {

// f(lo, hi) over [0, n) in up to eight pieces of at least ``grain`` elements; f must not throw.
template <class F>
void host_parallel(size_t n, size_t grain, F&& f) {
  constexpr size_t kMost = 8;
  const size_t hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t parts = std::max<size_t>(1, std::min<size_t>({kMost, hw, n / std::max<size_t>(1, grain)}));
  const size_t step = (n + parts - 1) / parts;
  std::thread threads[kMost];  // (no container: nothing below may throw while one is running)
  size_t lo = step;            // the caller takes the first piece
  try {
    for (size_t i = 0; lo < n; lo += step, ++i) threads[i] = std::thread([&f, lo, hi = std::min(n, lo + step)] { f(lo, hi); });
  } catch (const std::exception&) {  // no more threads, or no memory for one: the rest here
    f(lo, n);
  }
  if (n > 0) f(0, std::min(n, step));
  for (std::thread& t : threads)
    if (t.joinable()) t.join();
}

// An uninitialised host array (std::vector would write it twice).
template <class T>
struct HostArray {
  explicit HostArray(size_t n) : p(static_cast<T*>(std::malloc(std::max<size_t>(n, 1) * sizeof(T)))) {
    if (!p) throw std::bad_alloc();
  }
  T* data() { return p.get(); }
  T& operator[](size_t i) { return p.get()[i]; }

 private:
  struct Free {
    void operator()(T* q) const { std::free(q); }
  };
  std::unique_ptr<T, Free> p;
};

}  // namespace totem
