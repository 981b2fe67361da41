// Host loops of the upload and download paths over several threads.
//
// These loops read the caller's FP64 arrays once (16 bytes per complex element) and write FP32; one
// thread does that at a few GB/s, page faults of fresh buffers included, while the copy to the
// device runs at tens.  Threads are started per call: no pool outlives it.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdlib>
#include <memory>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

namespace totem {

// f(lo, hi) over [0, n) in up to eight pieces of at least ``grain`` elements; f must not throw.
template <class F>
void host_parallel(size_t n, size_t grain, F&& f) {
  const size_t hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t parts = std::max<size_t>(1, std::min<size_t>({8, hw, n / std::max<size_t>(1, grain)}));
  const size_t step = (n + parts - 1) / parts;
  std::vector<std::thread> threads;
  threads.reserve(parts);
  size_t lo = step;  // the caller takes the first piece
  try {
    for (; lo < n; lo += step) threads.emplace_back([&f, lo, hi = std::min(n, lo + step)] { f(lo, hi); });
  } catch (const std::system_error&) {
    f(lo, n);  // no more threads to be had: the rest here
  }
  if (n > 0) f(0, std::min(n, step));
  for (std::thread& t : threads) t.join();
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
