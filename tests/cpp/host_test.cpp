// Checks of csrc/rw_host.h, one per command-line argument; prints what failed.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <string>

#include "rw_host.h"

// Allocations left before operator new fails (negative: it does not).
static std::atomic<int> g_left{-1};
void* operator new(size_t n) {
  if (g_left >= 0 && g_left.fetch_sub(1) <= 0) {
    g_left = 0;
    throw std::bad_alloc();
  }
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

// A destination's contents survive, whatever its alignment and whether its pages are mapped.
static bool contents() {
  const size_t big = (size_t)40 << 20;
  for (size_t bytes : {(size_t)0, (size_t)1, (size_t)4095, (size_t)3 << 20, big - 5})
    for (size_t shift : {0, 1, 4093}) {
      unsigned char* p = static_cast<unsigned char*>(std::malloc(big + 8192));
      for (size_t k = 0; k < big + 8192; ++k) p[k] = (unsigned char)(k * 2654435761u >> 7);
      rw::touch_pages(p + shift, bytes);
      for (size_t k = 0; k < big + 8192; ++k)
        if (p[k] != (unsigned char)(k * 2654435761u >> 7)) return false;
      std::free(p);
    }
  unsigned char* z = static_cast<unsigned char*>(std::calloc(big, 1));  // not mapped yet
  rw::touch_pages(z, big);
  for (size_t k = 0; k < big; ++k)
    if (z[k]) return false;
  std::free(z);
  return true;
}

// Host memory that runs out at any allocation ends neither the call nor the process.
static bool no_memory() {
  const size_t big = (size_t)40 << 20;
  unsigned char* p = static_cast<unsigned char*>(std::calloc(big, 1));
  for (int left = 0; left < 20; ++left) {
    g_left = left;
    rw::touch_pages(p, big);
    g_left = -1;
  }
  std::free(p);
  return true;
}

// Every array in the fewest pieces that 8 MB allow, also where cells outnumber particles.
static bool export_pieces() {
  for (size_t scalar : {4, 8})
    for (size_t np : {1, 1000, 60000, 2180000})
      for (size_t ncell : {1, 37404, 2000000, 30000000}) {
        const size_t buf = rw::export_buffer_bytes(np, ncell, scalar);
        if (buf > (8u << 20)) return false;
        for (size_t bytes : {9 * scalar * np, 6 * scalar * np, 4 * ncell}) {
          const size_t pieces = (bytes + buf - 1) / buf;
          if (pieces > (bytes + (8u << 20) - 1) / (8u << 20)) return false;
        }
      }
  return true;
}

int main(int argc, char** argv) {
  const std::string which = argc > 1 ? argv[1] : "";
  bool ok = false;
  if (which == "contents") ok = contents();
  if (which == "no_memory") ok = no_memory();
  if (which == "export_pieces") ok = export_pieces();
  if (!ok) std::printf("%s failed\n", which.c_str());
  return ok ? 0 : 1;
}
