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

}  // namespace b200
