// Copies of large host buffers, cut into pieces.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstring>
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

// take(i) for every piece, on up to nt threads (this one included); enter() comes first on each further thread. Pieces of a
// thread that is not to be had (for whatever reason) are taken here, so that nothing leaves this function but its return.
template <class Enter, class Take>
inline void take_pieces(int pieces, int nt, Enter enter, Take take) {
  std::thread th[8];
  for (int t = 1; t < nt; ++t) {
    try {
      th[t] = std::thread([=, &enter, &take] {
        enter();
        for (int i = t; i < pieces; i += nt) take(i);
      });
    } catch (...) {
    }
  }
  for (int i = 0; i < pieces; ++i)
    if (i % nt == 0 || !th[i % nt].joinable()) take(i);
  for (int t = 1; t < nt; ++t)
    if (th[t].joinable()) th[t].join();
}

// memcpy split over a few threads: one thread moves 5-8 GB/s out of the page cache, which is less than the link takes.
inline void parallel_memcpy(void* dst, const void* src, size_t n) {
  const int nt = n >= ((size_t)8 << 20) ? 4 : 1;
  const CopyPieces p(n, nt);
  take_pieces(nt, nt, [] {}, [&](int i) { copy_piece(dst, src, p, i); });
}

// Hands a buffer over piece by piece as it lands, on nt threads: piece i is copied once landed(i), which waits for it, says that
// it may be (false: the destination keeps what it held).
template <class Enter, class Landed>
inline void hand_over(void* dst, const void* src, const CopyPieces& p, int pieces, int nt, Enter enter, Landed landed) {
  take_pieces(pieces, nt, enter, [&](int i) {
    if (landed(i)) copy_piece(dst, src, p, i);
  });
}

}  // namespace b200
