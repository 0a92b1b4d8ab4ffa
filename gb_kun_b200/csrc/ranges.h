// Ends of pieces of entry ranges.  Positions are int32 below 2^31 - 1, so
// beg + len can pass 2^31 where no entry does: these form no such sum.  Loops
// that step past the end of a range count in uint32, which does not wrap there.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define GBK_HD __host__ __device__ __forceinline__
#else
#define GBK_HD inline
#endif

namespace gbk {

// End of the piece of at most `len` entries that starts at beg in a range up to end (beg <= end).
GBK_HD int32_t piece_end(int32_t beg, int32_t len, int32_t end) { return end - beg > len ? beg + len : end; }

// Pieces of at most `len` entries that n entries make.
GBK_HD int32_t pieces_of(int32_t n, int32_t len) { return n > 0 ? (n - 1) / len + 1 : 0; }

// Whether positions up to 4,096 past the last of nnz entries are int32 too.
constexpr int32_t kLookAhead = 4096;
GBK_HD bool can_look_ahead(int64_t nnz) { return nnz <= INT32_MAX - kLookAhead; }

}  // namespace gbk
