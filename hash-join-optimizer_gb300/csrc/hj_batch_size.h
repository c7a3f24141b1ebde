// Sizes of the batch's hash tables (hj_batch.cu), the same on host and device.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#ifdef __CUDACC__
#define HJ_BATCH_HD __host__ __device__ __forceinline__
#else
#define HJ_BATCH_HD inline
#endif

namespace hj {

// Buckets (of four slots) per row in 65536ths, for a load of rows per slot within 0.25 .. 0.8.
inline uint32_t batch_buckets_q16(double load) {
    return uint32_t(std::lround(0.25 / std::min(0.8, std::max(0.25, load)) * 65536.0));
}

// Buckets of a piece of n rows: a fifth of its slots or more stays free.
HJ_BATCH_HD uint32_t batch_piece_buckets(uint32_t n, uint32_t q16) { return uint32_t((uint64_t(n) * q16) >> 16) + 1; }

// Buckets for two pieces of n rows in all, however the rows divide between them.
HJ_BATCH_HD uint32_t batch_pair_buckets(uint32_t n, uint32_t q16) { return batch_piece_buckets(n, q16) + 1; }

// Buckets for `pieces` pieces of `rows` rows in all, and the free bucket 0: no
// fewer than the pieces take however the rows divide among them.  In the
// pieces' own fixed point: with the exact quotient, pieces whose size it
// rounds up to a whole bucket took more than there were.
inline uint64_t batch_table_buckets(uint64_t rows, uint64_t pieces, uint32_t q16) {
    return uint64_t((static_cast<unsigned __int128>(rows) * q16) >> 16) + pieces + 1;
}

}  // namespace hj
