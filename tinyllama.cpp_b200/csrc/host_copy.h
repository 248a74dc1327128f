// Copies of large host buffers, cut into pieces.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <system_error>
#include <thread>

namespace b200 {

// [0, bytes) as `pieces` runs of whole pages, the last ones shorter or empty: together they cover every byte, whatever the size.
struct CopyPieces {
  size_t bytes, per;
  CopyPieces(size_t n, int pieces) : bytes(n), per(((n + pieces - 1) / pieces + 4095) & ~(size_t)4095) {}
  size_t begin(int i) const { return std::min(bytes, per * i); }
  size_t size(int i) const { return begin(i + 1) - begin(i); }
};

inline void copy_piece(void* dst, const void* src, const CopyPieces& p, int i) {
  std::memcpy(static_cast<uint8_t*>(dst) + p.begin(i), static_cast<const uint8_t*>(src) + p.begin(i), p.size(i));
}

// memcpy split over a few threads: one thread moves 5-8 GB/s out of the page cache, which is less than the link takes.
inline void parallel_memcpy(void* dst, const void* src, size_t n) {
  const int nt = n >= ((size_t)8 << 20) ? 4 : 1;
  const CopyPieces p(n, nt);
  std::thread th[4];
  for (int i = 1; i < nt; ++i) th[i] = std::thread([=] { copy_piece(dst, src, p, i); });
  copy_piece(dst, src, p, 0);
  for (int i = 1; i < nt; ++i) th[i].join();
}

// Hands a buffer over piece by piece as it lands, on nt threads: piece i is copied once landed(i), which waits for it, says that
// it may be (false: the destination keeps what it held).
template <class Landed>
inline void hand_over(void* dst, const void* src, const CopyPieces& p, int pieces, int nt, Landed landed) {
  auto take = [&](int i) {
    if (landed(i)) copy_piece(dst, src, p, i);
  };
  std::thread th[8];
  for (int t = 1; t < nt; ++t) {
    try {
      th[t] = std::thread([&take, t, nt, pieces] { for (int i = t; i < pieces; i += nt) take(i); });
    } catch (const std::system_error&) {
      // no further thread to be had: its pieces are taken below
    }
  }
  for (int i = 0; i < pieces; ++i)
    if (i % nt == 0 || !th[i % nt].joinable()) take(i);
  for (int t = 1; t < nt; ++t)
    if (th[t].joinable()) th[t].join();
}

}  // namespace b200
