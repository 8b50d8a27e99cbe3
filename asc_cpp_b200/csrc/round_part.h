// The part of a round of staged entries that belongs to one row (plain C++ too,
// so that it can be checked without a GPU).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define ASCB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define ASCB_HOST_DEVICE inline
#endif

namespace ascb {

// Entries [from, to) of the round [w, w + length) that lie in the row [b, e);
// none: from >= to.  Distances are bounded in 64 bits before they are narrowed:
// a row, and what stands between the rows of a warp, may have 2^31 entries.
struct RoundPart {
  int from, to;
};
ASCB_HOST_DEVICE RoundPart round_part(int64_t b, int64_t e, int64_t w, int length) {
  const int64_t from = b > w ? b - w : 0;
  const int64_t to = e > w ? e - w : 0;
  return {from < length ? static_cast<int>(from) : length,
          to < length ? static_cast<int>(to) : length};
}

}  // namespace ascb
