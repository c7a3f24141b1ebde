// Sizes of the batch's hash tables: whatever the load and the pieces' rows, a
// piece has more slots than rows and the memory holds every piece.  Exits 0.
#include <cstdio>

#include "hj_batch_size.h"

int main() {
    for (int pct = 1; pct <= 800; ++pct) {
        const double   load = pct / 100.0;
        const uint32_t q    = hj::batch_buckets_q16(load);
        for (uint32_t n = 0; n <= 16384; ++n) {
            const uint64_t piece = hj::batch_piece_buckets(n, q);
            if (4 * piece <= n) return std::printf("load %g: %u rows in %llu buckets\n", load, n, (unsigned long long)piece), 1;
            for (uint32_t a : {0u, 1u, n / 7, n / 3, n / 2, n})
                if (a <= n && hj::batch_piece_buckets(a, q) + hj::batch_piece_buckets(n - a, q) > hj::batch_pair_buckets(n, q))
                    return std::printf("load %g: %u and %u rows exceed their pair\n", load, a, n - a), 1;
            for (uint64_t pieces : {1ull, 2ull, 64ull, 763ull, 4096ull, 1ull << 22}) {
                const uint64_t have = hj::batch_table_buckets(n * pieces, pieces, q);  // bucket 0 is none of theirs
                // (a pair counts as two pieces)
                if (1 + hj::batch_pair_buckets(n, q) * pieces > hj::batch_table_buckets(n * pieces, 2 * pieces, q))
                    return std::printf("load %g: %llu pairs of %u rows\n", load, (unsigned long long)pieces, n), 1;
                if (1 + piece * pieces > have)
                    return std::printf("load %g: %llu pieces of %u rows take %llu buckets, there are %llu\n", load,
                                       (unsigned long long)pieces, n, (unsigned long long)(1 + piece * pieces),
                                       (unsigned long long)have), 1;
            }
        }
    }
    return 0;
}
