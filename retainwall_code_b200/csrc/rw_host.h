// Host-side helpers of the engine that need no GPU.
#pragma once
#include <algorithm>
#include <cstddef>
#include <exception>
#include <thread>

namespace rw {

// Touches every page of a large destination from several host threads: the page faults of new
// memory otherwise run on the one thread that copies (a 35 MB array in 5 ms; 20 ms through a
// temporary vector on one thread).  An atomic or with zero: a write fault at once, and the
// contents stay, so a copy that then fails has not cost the caller what was there.
// Page-locked slots were slower to make (3 to 60 ms) than they saved, and populating on
// request (madvise) slower than the faults (122 MB in three arrays: 22 ms, 18 this way).
inline void touch_pages(void* dst, size_t bytes) {
  constexpr size_t kPage = 4096, kPerThread = 2u << 20, kThreads = 8;
  const size_t hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t of = std::min(bytes / kPerThread, std::min(hw, kThreads));
  auto part = [=](size_t w) {
    unsigned char* p = static_cast<unsigned char*>(dst);
    for (size_t k = bytes * w / of; k < bytes * (w + 1) / of; k += kPage) __atomic_fetch_or(p + k, 0, __ATOMIC_SEQ_CST);
  };
  std::thread th[kThreads];  // an array: a vector that fails to grow would destroy running threads
  size_t started = 1;
  try {
    for (; started < of; ++started) th[started] = std::thread(part, started);
  } catch (const std::exception&) {  // no thread or no memory: the copy meets the other pages itself
  }
  if (of) part(0);
  for (size_t w = 1; w < started; ++w) th[w].join();
}

// Bytes of the device buffer that exports are put together in: the widest array per particle
// (nine scalars) or the cells' begins whole, up to 8 MB (then in pieces of that; a piece costs
// a launch and a copy, so a small case in a large grid is not cut by its particle count).
inline size_t export_buffer_bytes(size_t np, size_t ncell, size_t scalar) {
  return std::min<size_t>(std::max(9 * scalar * np, sizeof(int) * ncell), 8u << 20);
}

}  // namespace rw
