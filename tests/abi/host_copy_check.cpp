// Checks of csrc/host_copy.h: every byte of a buffer belongs to one piece, whatever its size, and pieces that may not be handed
// over leave the destination alone; further threads enter before their first piece, and calls do without those that cannot be had.
#include "host_copy.h"

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

using namespace b200;

static int failures = 0;
#define CHECK(cond, ...) \
  do { if (!(cond)) { ++failures; std::printf("line %d: %s: ", __LINE__, #cond); std::printf(__VA_ARGS__); std::printf("\n"); } } while (0)

// Allocations of the main thread that still succeed (-1: all): what std::thread needs for its start-up state.
static thread_local int allocations_left = -1;
void* operator new(size_t n) {
  if (allocations_left == 0) throw std::bad_alloc();
  if (allocations_left > 0) --allocations_left;
  if (void* p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

static void check_cover(size_t n, int pieces) {
  const CopyPieces p(n, pieces);
  size_t at = 0;
  for (int i = 0; i < pieces; ++i) {
    CHECK(p.begin(i) == at, "%zu bytes, %d pieces, piece %d", n, pieces, i);
    at += p.size(i);
  }
  CHECK(at == n, "%zu bytes in %d pieces: %zu covered", n, pieces, at);
}

int main() {
  for (int pieces : {1, 4, 8})
    for (size_t pages : {0, 1, 7, 256, 2048})
      for (int extra = -9; extra <= 9; ++extra) {
        const long long n = (long long)pages * 4096 * pieces + extra;
        if (n >= 0) check_cover((size_t)n, pieces);
      }
  // logits of 63 / 33 / 17 sequences whose number of values is one above a multiple of 8192
  for (size_t n : {63 * (size_t)36799, 33 * (size_t)66529, 17 * (size_t)127217}) check_cover(4 * n, 8);

  for (size_t n : {(size_t)100, ((size_t)8 << 20) - 1, ((size_t)8 << 20) + 1, ((size_t)8 << 20) + 4 * 4096 + 3}) {
    std::vector<unsigned char> src(n), dst(n, 0);
    for (size_t i = 0; i < n; ++i) src[i] = (unsigned char)(1 + i % 251);
    parallel_memcpy(dst.data(), src.data(), n);
    CHECK(src == dst, "%zu bytes", n);
  }
  const size_t n = 8 * 4096 * 3 + 5;
  const std::vector<unsigned char> src(n, 7), untouched(n, 1);
  std::vector<unsigned char> dst;
  for (int nt : {1, 4}) {
    std::atomic<int> seen{0};
    dst.assign(n, 1);
    hand_over(dst.data(), src.data(), CopyPieces(n, 8), 8, nt, [] {}, [&](int) { ++seen; return true; });
    CHECK(dst == src && seen == 8, "%d threads, %d pieces asked for", nt, seen.load());
    dst.assign(n, 1);
    hand_over(dst.data(), src.data(), CopyPieces(n, 8), 8, nt, [] {}, [](int) { return false; });
    CHECK(dst == untouched, "%d threads, refused pieces", nt);
  }

  // every further thread enters once, before its first piece; the calling one does not
  static thread_local int entered = 0;
  std::atomic<int> threads{0}, early{0};
  const std::thread::id me = std::this_thread::get_id();
  dst.assign(n, 1);
  hand_over(dst.data(), src.data(), CopyPieces(n, 8), 8, 4, [&] { ++entered; ++threads; }, [&](int) {
    if (entered != (std::this_thread::get_id() == me ? 0 : 1)) ++early;
    return true;
  });
  CHECK(dst == src && threads == 3 && early == 0, "%d threads entered, %d pieces out of order", threads.load(), early.load());

  // no memory for the second or third thread: its pieces are handed over all the same, and nothing is thrown
  for (int left : {0, 1, 2}) {
    dst.assign(n, 1);
    allocations_left = left;
    hand_over(dst.data(), src.data(), CopyPieces(n, 8), 8, 4, [] {}, [](int) { return true; });
    allocations_left = -1;
    CHECK(dst == src, "%d allocations", left);
  }
  std::printf("%d failures\n", failures);
  return failures ? 1 : 0;
}
