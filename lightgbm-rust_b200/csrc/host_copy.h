// Copies between the caller's pageable memory and the pinned staging buffers
// that the copy engine reads and writes.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstring>

namespace lgbm_b200 {

// dst[0, bytes) = src[0, bytes), split over the host's OpenMP threads in
// pieces of 128 KB (4 MB pieces left a 16 MB chunk to 4 of 16 threads); a
// copy of one piece stays in the calling thread, without the team's start.
inline void parallel_copy(void* dst, const void* src, size_t bytes) {
  constexpr size_t kPiece = (size_t)128 << 10;
  const int64_t pieces = (int64_t)((bytes + kPiece - 1) / kPiece);
#pragma omp parallel for schedule(static) if (pieces > 1)
  for (int64_t i = 0; i < pieces; ++i) {
    const size_t o = (size_t)i * kPiece;
    std::memcpy(static_cast<char*>(dst) + o, static_cast<const char*>(src) + o, std::min(kPiece, bytes - o));
  }
}

}  // namespace lgbm_b200
