// Unchained hash-table build on the GPU.
//
// Semantics of UnchainedHash::finalize_build (include/unchained.h:155-217 of
// the reference): Fibonacci hash, directory of 2^b words (default b =
// log2(next_pow2(#tuples))), word = (first adjacency-array index << 16) |
// 16-bit Bloom tag (OR of bloom_mask over the bucket's tuples), sentinel word
// 2^b = #tuples << 16; the adjacency array holds the tuples grouped by bucket.
// The directory words are therefore bit-identical to UnchainedHash's for the
// same key multiset (only the order of tuples inside a bucket may differ).
//
// The reference's live table, PartitionedDirectoryHash
// (include/partitioned_directory_hash.h:86-198), builds the same kind of
// adjacency array on the host with per-thread slab buffers
// (include/slab_allocator.h) and three phases.  Here the slabs are replaced by
// a two-level MSD radix partition:
//   1. k_part_hist      histogram of the top R hash bits (R = b - 12), then
//   2. (its last block) partition offsets and per-partition chunk counts
//   3. k_part_scatter   (key, row) pairs scattered to their partition
// Partitions of at most kFuseMax tuples are then built by one block each
// (k_bucket_local); the larger ones (Zipf-heavy keys) take steps 4-7 as the
// phases of one kernel (k_bucket_big):
//   4. per 8192-tuple chunk: shared-memory bucket counts and Bloom tags over
//      the partition's 2^12 buckets
//   5. per partition: prefix sum -> directory words
//   6. per chunk: tuples to their final adjacency slots
//   7. flags buckets that hold more than one distinct key, then summaries
// Shared-memory histograms per chunk keep Zipf-heavy keys (one key can own
// millions of tuples) off global atomics: a chunk adds one atomic per
// non-empty bucket, and warp-aggregated shared atomics absorb duplicates.
#include <algorithm>

#include <cooperative_groups.h>

#include "hj_block.cuh"
#include "hj_common.cuh"
#include "hj_kernels.h"

namespace hj {
namespace {

constexpr int kLocalBits   = 12;  // buckets per partition = 2^12 (16 KB of shared counters)
constexpr int kMaxRadix    = 14;
constexpr int kThreads     = 512;
constexpr int kItems       = 16;
constexpr int kTile        = kThreads * kItems;  // rows per partition-scatter tile
constexpr int kChunk       = kTile;              // tuples per bucket chunk
// Partitions of at most kFuseMax tuples are built by one block each
// (k_bucket_local); the chunked kernels take the larger ones.
constexpr uint32_t kFuseMax = 12288;

struct Geo {
    uint32_t b;  // directory bits
    uint32_t R;  // partition bits
    uint32_t L;  // local bucket bits = b - R
};

__device__ __forceinline__ bool load_key(const KeyCol& kc, uint64_t i, int32_t& key) {
    if (i >= kc.n) return false;
    return int_get(kc.col, kc.rid ? uint64_t(__ldg(kc.rid + i)) : i, key);
}

// 2. Exclusive scans of partition sizes and chunk counts, by one block.  Only
//    the partitions k_bucket_local does not take are cut into chunks; each
//    chunk's partition is written to chunk_part, so that a block finds a
//    chunk's partition with one load.
struct Parts {
    uint32_t *cnt, *off, *cursor, *chunk_off, *chunk_part;
    unsigned long long* n_valid;  // [1]: blocks of k_part_hist that are done, [2..3]: k_bucket_big's tickets
};
__device__ __forceinline__ void part_offsets(const Parts& d, uint32_t P, uint32_t* sm) {
    uint32_t run_t = 0, run_c = 0;
    for (uint32_t base = 0; base < P; base += blockDim.x) {
        const uint32_t i  = base + threadIdx.x;
        const uint32_t c  = i < P ? __ldcg(d.cnt + i) : 0;  // (other blocks' atomics)
        const uint32_t ch = c > kFuseMax ? (c + kChunk - 1) / kChunk : 0u;
        uint32_t       tot_t, tot_c;
        const uint32_t et = block_exclusive_scan<uint32_t>(c, sm, &tot_t);
        const uint32_t ec = block_exclusive_scan<uint32_t>(ch, sm, &tot_c);
        if (i < P) {
            d.off[i]       = run_t + et;
            d.cursor[i]    = run_t + et;
            d.chunk_off[i] = run_c + ec;
            for (uint32_t q = 0; q < ch; ++q) d.chunk_part[run_c + ec + q] = i;
        }
        run_t += tot_t;
        run_c += tot_c;
    }
    if (threadIdx.x == 0) {
        d.off[P]       = run_t;
        d.chunk_off[P] = run_c;
    }
}

// 1. Partition histogram + count of valid keys; the block that is done last
//    makes the offsets (2).
__global__ void __launch_bounds__(kThreads) k_part_hist(KeyCol kc, uint32_t R, Parts d) {
    extern __shared__ uint32_t hist[];
    __shared__ uint32_t        sm[33];
    __shared__ bool            last;
    const uint32_t P = 1u << R;
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    uint32_t       mine = 0;
    constexpr int  kU   = 8;  // keys per thread loaded before any of them is counted
    const uint64_t step = uint64_t(gridDim.x) * blockDim.x * kU;
    for (uint64_t b0 = uint64_t(blockIdx.x) * blockDim.x * kU + threadIdx.x; b0 < kc.n; b0 += step) {
        int32_t key[kU];
        bool    ok[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) ok[u] = load_key(kc, b0 + uint64_t(u) * blockDim.x, key[u]);
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            if (ok[u]) {
                atomicAdd(hist + uint32_t(bucket_of(fib_hash(key[u]), R)), 1u);
                ++mine;
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x)
        if (hist[i]) atomicAdd(d.cnt + i, hist[i]);
    mine = warp_sum(mine);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(d.n_valid, (unsigned long long)mine);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(d.n_valid + 1, 1ull) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    part_offsets(d, P, sm);
}

// 3. Scatter (key, row) to partitions.  Each block owns a tile of kTile rows:
//    shared-memory counts give every item its rank in its partition within
//    the tile, one global atomic per (tile, non-empty partition) reserves the
//    partition's space, the items are placed partition by partition in shared
//    memory and then stored so that consecutive threads write consecutive
//    slots of a partition (runs instead of single 4-byte stores).
template <int kST>  // threads; a tile is kST * kItems rows
__global__ void __launch_bounds__(kST, 1024 / kST)
    k_part_scatter(KeyCol kc, uint32_t R, uint32_t* __restrict__ part_cursor,
                   int32_t* __restrict__ tkey, uint32_t* __restrict__ trow) {
    extern __shared__ uint32_t sh[];  // P counters / tile offsets, P global bases, staged items
    __shared__ uint32_t sm[33];
    const uint32_t P     = 1u << R;
    uint32_t*      off   = sh;                   // counts, then the tile's partition offsets
    uint32_t*      gbase = sh + P;               // global slot of each partition's first item
    int32_t*       sk    = reinterpret_cast<int32_t*>(sh + 2 * P);
    constexpr int  kT    = kST * kItems;
    uint32_t*      sr    = sh + 2 * P + kT;
    uint16_t*      sp    = reinterpret_cast<uint16_t*>(sh + 2 * P + 2 * kT);  // partition of each slot
    const uint64_t tile0 = uint64_t(blockIdx.x) * kT;
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) off[i] = 0;
    __syncthreads();
    int32_t  keys[kItems];
    uint32_t rank[kItems];
    uint32_t okmask = 0;
    // all of the thread's keys are loaded before any is counted
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint64_t i = tile0 + uint64_t(k) * kST + threadIdx.x;
        okmask |= uint32_t(load_key(kc, i, keys[k])) << k;
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const bool ok = (okmask >> k) & 1u;
        rank[k]       = ok ? atomicAdd(off + uint32_t(bucket_of(fib_hash(keys[k]), R)), 1u) : 0;
    }
    __syncthreads();
    // exclusive scan of the counts (thread t: partitions [t * per, (t + 1) * per))
    const uint32_t per = (P + kST - 1) / kST;
    uint32_t       run = 0;
    // the thread's reservations four at a time, all four in flight before any
    // result is stored
    for (uint32_t q0 = 0; q0 < per; q0 += 4) {
        uint32_t base[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t q = q0 + u, p = threadIdx.x * per + q;
            const uint32_t c = q < per && p < P ? off[p] : 0u;
            base[u]          = c ? atomicAdd(part_cursor + p, c) : 0u;
            run += c;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t q = q0 + u, p = threadIdx.x * per + q;
            if (q < per && p < P) gbase[p] = base[u];
        }
    }
    uint32_t       tot;
    const uint32_t ex = block_exclusive_scan<uint32_t>(run, sm, &tot);
    run               = ex;
    for (uint32_t q = 0; q < per; ++q) {
        const uint32_t p = threadIdx.x * per + q;
        if (p < P) {
            const uint32_t c = off[p];
            off[p]           = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        if ((okmask >> k) & 1u) {
            const uint32_t part = uint32_t(bucket_of(fib_hash(keys[k]), R));  // recomputed: fewer registers
            const uint32_t q    = off[part] + rank[k];
            sk[q]               = keys[k];
            sr[q]               = uint32_t(tile0 + uint64_t(k) * kST + threadIdx.x);
            sp[q]               = uint16_t(part);
        }
    }
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < tot; q += blockDim.x) {
        const uint32_t p   = sp[q];
        const uint32_t pos = gbase[p] + (q - off[p]);
        tkey[pos]          = sk[q];
        trow[pos]          = sr[q];
    }
}


__device__ __forceinline__ bool fused_part(const uint32_t* part_off, uint32_t part) {
    return part_off[part + 1] - part_off[part] <= kFuseMax;
}

// Locates chunk `cid`: its partition and tuple range.  Returns false past the end.
__device__ __forceinline__ bool chunk_range(uint32_t cid, const uint32_t* chunk_off, const uint32_t* chunk_part,
                                            const uint32_t* part_off, uint32_t P, uint32_t& part,
                                            uint32_t& s, uint32_t& e, bool& single) {
    if (cid >= chunk_off[P]) return false;
    part             = chunk_part[cid];
    const uint32_t k = cid - chunk_off[part];
    s                = part_off[part] + k * kChunk;
    e                = min(part_off[part + 1], s + kChunk);
    single           = chunk_off[part + 1] - chunk_off[part] == 1;
    return true;
}

// Shared counter addr[slot] += 1 for each active lane, returning the lane's
// old value.  Lanes of a warp that all carry one slot (a Zipf-heavy key fills
// whole chunks) need one atomic; otherwise each lane adds on its own.
__device__ __forceinline__ uint32_t bucket_add(uint32_t* addr, uint32_t slot, unsigned act) {
    const unsigned lane   = threadIdx.x & 31;
    const int      leader = __ffs(act) - 1;
    // uniform when every active lane carries the leader's slot (a shuffle and
    // a vote: cheaper than a match instruction)
    const bool uni = __all_sync(act, slot == __shfl_sync(act, slot, leader));
    if (uni) {
        uint32_t  base   = 0;
        if (int(lane) == leader) base = atomicAdd(addr + slot, uint32_t(__popc(act)));
        return __shfl_sync(act, base, leader) + __popc(act & ((1u << lane) - 1));
    }
    return atomicAdd(addr + slot, 1u);
}

// ---- partitions above kFuseMax tuples, in phases of one kernel (k_bucket_big) ----
// What a phase reads of an earlier one takes plain loads: other blocks of the
// same launch wrote it (no read-only loads), and a heavy key's warps all read
// the same words, which have to come from the L1 (from the L2, 16M tuples of
// one key: 525 -> 676 us).
// Most tuples of a build that takes these phases in one launch.  hj_table_build
// before (a launch a phase) / in one launch, us: distinct keys, which have
// nothing to do here, 300,000 78 / 51, 1M 88 / 61, 4M 151 / 132; one key only 4M
// 194 / 188; Zipf(1.1) keys 4M 212 / 208, but 6M 290 / 299 and 16M 569 / 589, where
// counting and comparing want more threads than the scatter's registers leave.
constexpr uint64_t kBigOne = 1u << 22;
struct Big {
    Geo             g;
    const uint32_t *chunk_off, *chunk_part, *part_off;
    const int32_t*  tkey;
    const uint32_t* trow;
    uint32_t *      cnt, *bloom;  // bucket counters (then cursors) and Bloom tags
    uint64_t*       dir;
    int32_t*        okey;
    uint32_t *      orow, *mixed;
    uint64_t*       summary;
    uint32_t*       ticket;  // the next chunk of each of the three chunk phases, zeroed
};

// Counters and Bloom tags of a partition cut into more than one chunk (its
// chunks add to them; a single chunk's are stored whole), and the mixed bits.
__device__ __forceinline__ void big_zero(const Big& d, uint32_t part) {
    const uint32_t nl = 1u << d.g.L;
    const uint64_t gb = uint64_t(part) << d.g.L;
    const bool     many = d.chunk_off[part + 1] - d.chunk_off[part] > 1;
    for (uint32_t i = threadIdx.x; i < nl; i += blockDim.x) {
        if (many) d.cnt[gb + i] = d.bloom[gb + i] = 0;
        if (nl >= 32 && i < nl / 32) d.mixed[(gb >> 5) + i] = 0;
    }
}

// 4. Per-chunk bucket counts and Bloom tags.
__device__ __forceinline__ void big_count(const Big& d, uint32_t cid, uint32_t* sh) {
    const Geo      g   = d.g;
    const uint32_t nl  = 1u << g.L;
    uint32_t*      cnt = sh;
    uint32_t*      blm = sh + nl;
    uint32_t       part, s, e;
    bool           single;
    if (!chunk_range(cid, d.chunk_off, d.chunk_part, d.part_off, 1u << g.R, part, s, e, single)) return;
    for (uint32_t i = threadIdx.x; i < 2 * nl; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    const uint32_t lmask = nl - 1;
    constexpr int  kU    = 8;  // keys per thread loaded before any of them is counted
    for (uint32_t b0 = s; b0 < e; b0 += kU * blockDim.x) {
        int32_t key[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const uint32_t j = b0 + uint32_t(u) * blockDim.x + threadIdx.x;
            key[u]           = j < e ? __ldg(d.tkey + j) : 0;
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const uint32_t j   = b0 + uint32_t(u) * blockDim.x + threadIdx.x;
            const bool     ok  = j < e;
            const unsigned act = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                const uint64_t h      = fib_hash(key[u]);
                const uint32_t local  = uint32_t(bucket_of(h, g.b)) & lmask;
                const int      leader = __ffs(act) - 1;
                bucket_add(cnt, local, act);
                // a warp of one heavy key ORs its tags once, not 32 times on one word
                if (__all_sync(act, local == __shfl_sync(act, local, leader))) {
                    const uint32_t all = __reduce_or_sync(act, bloom_mask(h));
                    if (int(threadIdx.x & 31) == leader) atomicOr(blm + local, all);
                } else {
                    atomicOr(blm + local, bloom_mask(h));
                }
            }
        }
    }
    __syncthreads();
    const uint64_t gb = uint64_t(part) << g.L;
    for (uint32_t i = threadIdx.x; i < nl; i += blockDim.x) {
        if (single) {
            d.cnt[gb + i]   = cnt[i];
            d.bloom[gb + i] = blm[i];
        } else if (cnt[i]) {
            atomicAdd(d.cnt + gb + i, cnt[i]);
            atomicOr(d.bloom + gb + i, blm[i]);
        }
    }}

// 5. Directory words of a partition; the counters become the scatter cursors.
__device__ __forceinline__ void big_dir(const Big& d, uint32_t part, uint32_t* sm) {
    const uint32_t nl  = 1u << d.g.L;
    const uint64_t gb  = uint64_t(part) << d.g.L;
    uint32_t       run = d.part_off[part];
    for (uint32_t base = 0; base < nl; base += blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t c = i < nl ? d.cnt[gb + i] : 0;
        uint32_t       tot;
        const uint32_t ex = block_exclusive_scan<uint32_t>(c, sm, &tot);
        if (i < nl) {
            const uint32_t start = run + ex;
            d.dir[gb + i]        = (uint64_t(start) << 16) | (d.bloom[gb + i] & 0xffffu);
            d.cnt[gb + i]        = start;
        }
        run += tot;
    }
}

// 6. Final scatter into bucket order.
__device__ __forceinline__ void big_scatter(const Big& d, uint32_t cid, uint32_t* sh) {
    const Geo      g  = d.g;
    const uint32_t nl = 1u << g.L;
    uint32_t       part, s, e;
    bool           single;
    if (!chunk_range(cid, d.chunk_off, d.chunk_part, d.part_off, 1u << g.R, part, s, e, single)) return;
    for (uint32_t i = threadIdx.x; i < nl; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    const uint32_t lmask = nl - 1;
    // the chunk's keys stay in registers between the count and the placing
    int32_t keys[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t j = s + uint32_t(k) * kThreads + threadIdx.x;
        keys[k]          = j < e ? __ldg(d.tkey + j) : 0;
        // the rows are stored after the counts: bring their lines into L1 now
        if (j < e) asm volatile("prefetch.global.L1 [%0];" ::"l"(d.trow + j));
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const bool     ok  = s + uint32_t(k) * kThreads + threadIdx.x < e;
        const unsigned act = __ballot_sync(0xffffffffu, ok);
        if (ok) bucket_add(sh, uint32_t(bucket_of(fib_hash(keys[k]), g.b)) & lmask, act);
    }
    __syncthreads();
    const uint64_t gb = uint64_t(part) << g.L;
    {
        // the thread's buckets (at most 2^kLocalBits / kThreads): every cursor
        // load or atomic issued before any result is stored
        constexpr int kPer = (1 << kLocalBits) / kThreads;
        uint32_t      c[kPer];
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t i = threadIdx.x + uint32_t(q) * kThreads;
            const uint32_t n = i < nl ? sh[i] : 0u;
            c[q]             = n == 0 ? 0u : (single ? d.cnt[gb + i] : atomicAdd(d.cnt + gb + i, n));
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t i = threadIdx.x + uint32_t(q) * kThreads;
            if (i < nl && sh[i]) sh[i] = c[q];
        }
    }
    __syncthreads();
    uint32_t rows[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t j = s + uint32_t(k) * kThreads + threadIdx.x;
        rows[k]          = j < e ? __ldg(d.trow + j) : 0u;
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const bool     ok  = s + uint32_t(k) * kThreads + threadIdx.x < e;
        const unsigned act = __ballot_sync(0xffffffffu, ok);
        if (ok) {
            const uint32_t pos = bucket_add(sh, uint32_t(bucket_of(fib_hash(keys[k]), g.b)) & lmask, act);
            d.okey[pos]        = keys[k];
            d.orow[pos]        = rows[k];
        }
    }
}

// 4-7 in one block for a partition of at most kFuseMax tuples: bucket counts
// and Bloom tags in shared memory, the directory words from one scan of the
// counts, then the tuples placed in bucket order in shared memory and stored
// with coalesced writes (scattered 4-byte stores would cost one L2 request
// each); the mixed bits come from neighbouring keys of the placed order.
// Larger partitions (Zipf-heavy keys) take the chunked kernels, which skip the
// partitions handled here.
constexpr int kLT = 1024;            // threads of k_bucket_local
constexpr int kLU = kFuseMax / kLT;  // tuples per thread of a partition it takes, at most
static_assert(kLU * kLT == int(kFuseMax), "a partition is one pass of the block");

__global__ void __launch_bounds__(kLT, 1)
    k_bucket_local(Geo g, const uint32_t* __restrict__ part_off, const int32_t* __restrict__ tkey,
                   const uint32_t* __restrict__ trow, uint64_t* __restrict__ dir, int32_t* __restrict__ okey,
                   uint32_t* __restrict__ orow, uint32_t* __restrict__ mixed, uint64_t* __restrict__ summary) {
    extern __shared__ uint32_t sh[];
    __shared__ uint32_t wsum[kLT / 32];
    const uint32_t nl    = 1u << g.L;
    const uint32_t lmask = nl - 1;
    const uint32_t P     = 1u << g.R;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nbw = (nl + 1) / 2, nmw = (nl + 31) / 32;
    uint32_t* cnt = sh;                 // nl: counts, then cursors
    uint32_t* blm = sh + nl;            // nbw words: two 16-bit Bloom tags each
    uint32_t* mix = sh + nl + nbw;      // nmw words of mixed bits
    int32_t*  sk  = reinterpret_cast<int32_t*>(mix + nmw);  // kFuseMax staged keys
    uint32_t* sr  = reinterpret_cast<uint32_t*>(sk + kFuseMax);        // and rows
    if (blockIdx.x == 0 && threadIdx.x == 0) dir[uint64_t(P) << g.L] = uint64_t(part_off[P]) << 16;
    for (uint32_t part = blockIdx.x; part < P; part += gridDim.x) {
        if (!fused_part(part_off, part)) continue;
        const uint32_t s = part_off[part], e = part_off[part + 1];
        const uint64_t gb = uint64_t(part) << g.L;
        for (uint32_t i = threadIdx.x; i < nl + nbw + nmw; i += blockDim.x) sh[i] = 0;
        __syncthreads();
        // the partition's keys, all loaded before any is counted (kLU per thread)
        int32_t key[kLU];
#pragma unroll
        for (int u = 0; u < kLU; ++u) {
            const uint32_t j = s + uint32_t(u) * kLT + threadIdx.x;
            key[u]           = j < e ? __ldg(tkey + j) : 0;
        }
        const int nu = int((e - s + kLT - 1) / kLT);  // passes of the block that hold tuples
        // counts and Bloom tags
#pragma unroll
        for (int u = 0; u < kLU; ++u) {
            if (u >= nu) break;
            const uint32_t j   = s + uint32_t(u) * kLT + threadIdx.x;
            const bool     ok  = j < e;
            const unsigned act = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                const uint64_t h     = fib_hash(key[u]);
                const uint32_t local = uint32_t(bucket_of(h, g.b)) & lmask;
                bucket_add(cnt, local, act);
                atomicOr(blm + (local >> 1), bloom_mask(h) << (16 * (local & 1)));
            }
        }
        // the rows are placed after the scan: their loads overlap it
        uint32_t row[kLU];
#pragma unroll
        for (int u = 0; u < kLU; ++u) {
            const uint32_t j = s + uint32_t(u) * kLT + threadIdx.x;
            row[u]           = j < e ? __ldg(trow + j) : 0u;
        }
        __syncthreads();
        // exclusive scan of the counts: warp w scans segments of 32 counts
        // (lane i reads count 32 q + i: no bank conflicts), then the warps' totals
        const uint32_t nseg = (nl + 31) / 32, per_w = (nseg + kLT / 32 - 1) / (kLT / 32);
        uint32_t       wrun = 0;
        for (uint32_t q = warp * per_w; q < min(nseg, (warp + 1) * per_w); ++q) {
            const uint32_t i = 32 * q + lane;
            const uint32_t c = i < nl ? cnt[i] : 0u;
            wrun += warp_sum(c);
        }
        if (lane == 0) wsum[warp] = wrun;
        __syncthreads();
        uint32_t base = s;
        for (uint32_t w = 0; w < warp; ++w) base += wsum[w];
        for (uint32_t q = warp * per_w; q < min(nseg, (warp + 1) * per_w); ++q) {
            const uint32_t i   = 32 * q + lane;
            const uint32_t c   = i < nl ? cnt[i] : 0u;
            const uint32_t inc = warp_inclusive_scan(c);
            if (i < nl) {
                const uint32_t start = base + inc - c;
                cnt[i]               = start;
                dir[gb + i]          = (uint64_t(start) << 16) | ((blm[i >> 1] >> (16 * (i & 1))) & 0xffffu);
            }
            base += __shfl_sync(0xffffffffu, inc, 31);
        }
        __syncthreads();
        // place the tuples in bucket order
#pragma unroll
        for (int u = 0; u < kLU; ++u) {
            if (u >= nu) break;
            const uint32_t j   = s + uint32_t(u) * kLT + threadIdx.x;
            const bool     ok  = j < e;
            const unsigned act = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                const uint32_t local = uint32_t(bucket_of(fib_hash(key[u]), g.b)) & lmask;
                const uint32_t q     = bucket_add(cnt, local, act) - s;
                sk[q]                = key[u];
                sr[q]                = row[u];
            }
        }
        __syncthreads();
        // coalesced stores; a bucket is mixed when two neighbours in it differ
        for (uint32_t q = threadIdx.x; q < e - s; q += blockDim.x) {
            const int32_t k = sk[q];
            okey[s + q]     = k;
            orow[s + q]     = sr[q];
            if (q > 0 && sk[q - 1] != k) {
                const uint32_t local = uint32_t(bucket_of(fib_hash(k), g.b)) & lmask;
                if ((uint32_t(bucket_of(fib_hash(sk[q - 1]), g.b)) & lmask) == local)
                    atomicOr(mix + (local >> 5), 1u << (local & 31));
            }
        }
        __syncthreads();
        // the partition's buckets are whole mixed words (2^L >= 32) or share one
        if (nl >= 32) {
            for (uint32_t i = threadIdx.x; i < nl / 32; i += blockDim.x) mixed[(gb >> 5) + i] = mix[i];
        } else if (threadIdx.x == 0 && mix[0]) {
            atomicOr(mixed + (gb >> 5), mix[0] << (gb & 31));
        }
        // bucket summaries: cnt[i] is now the end of bucket i, so bucket i
        // spans [end of bucket i - 1, cnt[i]); its first key is staged in sk
        for (uint32_t i = threadIdx.x; i < nl; i += blockDim.x) {
            const uint32_t b0  = i == 0 ? s : cnt[i - 1];
            const uint32_t len = cnt[i] - b0;
            summary[gb + i]    = len == 0 ? 0ull
                                          : make_summary(sk[b0 - s], (blm[i >> 1] >> (16 * (i & 1))) & 0xffffu, len,
                                                         (mix[i >> 5] >> (i & 31)) & 1u, sr[b0 - s]);
        }
        __syncthreads();
    }
}

// 7. mixed[p] bit set when bucket p holds two different keys.
__device__ __forceinline__ void big_mixed(const Big& d, uint32_t cid) {
    uint32_t part, s, e;
    bool     single;
    if (!chunk_range(cid, d.chunk_off, d.chunk_part, d.part_off, 1u << d.g.R, part, s, e, single)) return;
    // kMU tuples per thread at a time: keys, then directory words, then first keys
    constexpr int kMU = 8;
    for (uint32_t j0 = s + threadIdx.x; j0 < e; j0 += kMU * blockDim.x) {
        int32_t  k[kMU];
        uint32_t p[kMU], first[kMU];
#pragma unroll
        for (int u = 0; u < kMU; ++u) {
            const uint32_t j = j0 + u * blockDim.x;
            k[u]             = j < e ? d.okey[j] : 0;
        }
#pragma unroll
        for (int u = 0; u < kMU; ++u) {
            p[u]     = uint32_t(bucket_of(fib_hash(k[u]), d.g.b));
            first[u] = j0 + u * blockDim.x < e ? uint32_t(d.dir[p[u]] >> 16) : 0u;
        }
#pragma unroll
        for (int u = 0; u < kMU; ++u)
            if (j0 + u * blockDim.x < e && d.okey[first[u]] != k[u])
                atomicOr(d.mixed + (p[u] >> 5), 1u << (p[u] & 31));
    }
}

// Bucket summaries of a partition (those of the others come from k_bucket_local).
__device__ __forceinline__ void big_summary(const Big& d, uint32_t part) {
    const uint32_t nl = 1u << d.g.L;
    const uint64_t gb = uint64_t(part) << d.g.L;
    for (uint32_t i = threadIdx.x; i < nl; i += blockDim.x) {
        const uint64_t p   = gb + i;
        const uint64_t d0  = d.dir[p];
        const uint32_t b0  = uint32_t(d0 >> 16);
        const uint32_t len = uint32_t(d.dir[p + 1] >> 16) - b0;
        d.summary[p] = len == 0 ? 0ull
                                : make_summary(d.okey[b0], uint32_t(d0) & 0xffffu, len,
                                               (d.mixed[(p >> 5)] >> (p & 31)) & 1u,
                                               len == 1 ? d.orow[b0] : 0u);
    }
}

// 4-7 for the partitions that k_bucket_local leaves, after it: one cooperative
// launch (its blocks are resident together, so that they can wait for each
// other between the phases), which returns at once when there are none, as
// for most builds; six launches that found nothing to do took 1.6 us each on
// the GPU and some 2.7 us each on the host.
constexpr int kBigBlocks = 2;  // per SM
__global__ void __launch_bounds__(kThreads, kBigBlocks) k_bucket_big(Big d) {
    extern __shared__ uint32_t sh[];
    __shared__ uint32_t        sm[33];
    const uint32_t P = 1u << d.g.R, nc = d.chunk_off[P];
    if (nc == 0) return;
    const auto grid  = cooperative_groups::this_grid();
    auto       parts = [&](auto f) {
        for (uint32_t p = blockIdx.x; p < P; p += gridDim.x)
            if (!fused_part(d.part_off, p)) f(p);
    };
    // chunks go to whichever block is free: the first by its index, the others by tickets
    __shared__ uint32_t next;
    auto                chunks = [&](uint32_t* ticket, auto f) {
        for (uint32_t c = blockIdx.x; c < nc;) {
            f(c);
            __syncthreads();
            if (threadIdx.x == 0) next = gridDim.x + atomicAdd(ticket, 1u);
            __syncthreads();
            c = next;
        }
    };
    parts([&](uint32_t p) { big_zero(d, p); });
    grid.sync();
    chunks(d.ticket + 0, [&](uint32_t c) { big_count(d, c, sh); });
    grid.sync();
    parts([&](uint32_t p) { big_dir(d, p, sm); });
    grid.sync();
    chunks(d.ticket + 1, [&](uint32_t c) { big_scatter(d, c, sh); });
    grid.sync();
    chunks(d.ticket + 2, [&](uint32_t c) { big_mixed(d, c); });
    grid.sync();
    parts([&](uint32_t p) { big_summary(d, p); });
}

// The same phases as a launch each, with as many blocks as a phase has chunks
// or partitions and (but for the scatter) twice the threads on an SM.
template <int PHASE>
__global__ void __launch_bounds__(kThreads, PHASE == 3 ? 2 : 4) k_bucket_phase(Big d) {
    extern __shared__ uint32_t sh[];
    __shared__ uint32_t        sm[33];
    if (PHASE == 1) return big_count(d, blockIdx.x, sh);
    if (PHASE == 3) return big_scatter(d, blockIdx.x, sh);
    if (PHASE == 4) return big_mixed(d, blockIdx.x);
    if (fused_part(d.part_off, blockIdx.x)) return;
    if (PHASE == 0) big_zero(d, blockIdx.x);
    if (PHASE == 2) big_dir(d, blockIdx.x, sm);
    if (PHASE == 5) big_summary(d, blockIdx.x);
}

// Small builds in one launch: every block owns one partition of the directory
// and reads ALL keys, keeping those of its partition; the number of valid keys
// in lower partitions, counted on the way, is where its tuples start, so no
// histogram, offsets or scatter pass precedes it and nothing is cleared.  A
// partition of at most kDirectMax tuples is listed in shared memory and counted
// and placed from there; a larger one (a heavy key) reads the keys twice again.
// Every block reads the keys from L2, so the cost grows with keys x partitions.
constexpr int      kDT        = 1024;        // threads
constexpr uint32_t kDirectMax = 20480;       // listed tuples of a partition
constexpr int      kDU        = 8;           // keys per thread in flight

__host__ __device__ constexpr size_t direct_smem(uint32_t L) {
    return (size_t(1) << L) * 4 + (((size_t(1) << L) + 1) / 2) * 4 + (((size_t(1) << L) + 31) / 32) * 4 + 2 * size_t(kDirectMax) * 4;
}

__global__ void __launch_bounds__(kDT, 1)
    k_build_direct(KeyCol kc, Geo g, uint64_t* __restrict__ dir, int32_t* okey,
                   uint32_t* orow, uint32_t* __restrict__ mixed, uint64_t* __restrict__ summary) {
    extern __shared__ uint32_t sh[];
    __shared__ uint32_t wsum[kDT / 32], s_n, s_low;
    const uint32_t nl = 1u << g.L, lmask = nl - 1, part = blockIdx.x;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1;
    const uint32_t nbw = (nl + 1) / 2, nmw = (nl + 31) / 32;
    uint32_t* cnt = sh;             // nl: counts, then cursors
    uint32_t* blm = sh + nl;        // nbw words: two 16-bit Bloom tags each
    uint32_t* mix = sh + nl + nbw;  // nmw words of mixed bits
    int32_t*  sk  = reinterpret_cast<int32_t*>(mix + nmw);  // kDirectMax listed keys
    uint32_t* sr  = reinterpret_cast<uint32_t*>(sk + kDirectMax);  // and rows
    const uint64_t gb = uint64_t(part) << g.L;
    for (uint32_t i = threadIdx.x; i < nl + nbw + nmw; i += kDT) sh[i] = 0;
    if (threadIdx.x == 0) s_n = s_low = 0;
    __syncthreads();
    const uint32_t n = uint32_t(kc.n);
    // kDU keys of this thread from i0 on, and which of them are the partition's; lower partitions' are counted
    uint32_t low  = 0;
    auto     mine = [&](uint32_t i0, int32_t (&key)[kDU]) {
        uint32_t ok = 0, in = 0;
#pragma unroll
        for (int u = 0; u < kDU; ++u) ok |= uint32_t(load_key(kc, uint64_t(i0) + uint64_t(u) * kDT, key[u])) << u;
#pragma unroll
        for (int u = 0; u < kDU; ++u) {
            const uint32_t p    = g.R ? fib_hi(key[u]) >> (32 - g.R) : 0u;
            const bool     some = (ok >> u) & 1u;
            low += some && p < part;
            in |= uint32_t(some && p == part) << u;
        }
        return in;
    };
    auto bucket = [&](int32_t k) { return uint32_t(bucket_of(fib_hash(k), g.b)) & lmask; };
    // the Bloom tag of key k; a heavy key's is there already: a read, not an atomic on one word
    auto tag = [&](int32_t k) {
        const uint64_t h     = fib_hash(k);
        const uint32_t local = uint32_t(bucket_of(h, g.b)) & lmask;
        const uint32_t t     = bloom_mask(h) << (16 * (local & 1));
        if ((*reinterpret_cast<volatile uint32_t*>(blm + (local >> 1)) & t) != t) atomicOr(blm + (local >> 1), t);
    };
    // Of a warp's keys `in`, the ones equal to its first (in an unlisted
    // partition mostly the heavy key, counted by one atomic a warp): k0 and which they are.
    auto heavy = [&](uint32_t in, const int32_t (&k)[kDU], int32_t& k0) {
        const unsigned some = __ballot_sync(0xffffffffu, in != 0);
        int32_t        f    = 0;
#pragma unroll
        for (int u = kDU - 1; u >= 0; --u)
            if ((in >> u) & 1u) f = k[u];
        k0 = __shfl_sync(0xffffffffu, f, some ? __ffs(some) - 1 : 0);
        uint32_t eq = 0;
#pragma unroll
        for (int u = 0; u < kDU; ++u) eq |= uint32_t(((in >> u) & 1u) && k[u] == k0) << u;
        return eq;
    };
    for (uint32_t i0 = threadIdx.x; i0 - lane < n; i0 += kDT * kDU) {  // warp-uniform bound
        int32_t        key[kDU];
        const uint32_t in  = mine(i0, key);
        // list slots step by step, so that neighbouring lanes store to neighbouring slots
        uint32_t bal[kDU], tot = 0;
#pragma unroll
        for (int u = 0; u < kDU; ++u) {
            bal[u] = __ballot_sync(0xffffffffu, (in >> u) & 1u);
            tot += __popc(bal[u]);
        }
        if (tot == 0) continue;
        uint32_t q = 0;
        if (lane == 0) q = atomicAdd(&s_n, tot);
        q = __shfl_sync(0xffffffffu, q, 0);
#pragma unroll
        for (int u = 0; u < kDU; ++u) {
            const uint32_t at = q + __popc(bal[u] & lt);
            if (((in >> u) & 1u) && at < kDirectMax) {
                sk[at] = key[u];
                sr[at] = i0 + uint32_t(u) * kDT;
            }
            q += __popc(bal[u]);
        }
    }
    low = warp_sum(low);
    if (lane == 0 && low) atomicAdd(&s_low, low);
    __syncthreads();
    const uint32_t s = s_low, m = s_n;  // the partition's first slot and tuples
    const bool     listed = m <= kDirectMax;
    if (listed) {
        for (uint32_t q = threadIdx.x; q - lane < m; q += kDT) {
            const bool     ok  = q < m;
            const unsigned act = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                bucket_add(cnt, bucket(sk[q]), act);
                tag(sk[q]);
            }
        }
    } else {
        for (uint32_t i0 = threadIdx.x; i0 - lane < n; i0 += kDT * kDU) {
            int32_t        k[kDU];
            const uint32_t in = mine(i0, k);
            int32_t        k0;
            const uint32_t eq  = heavy(in, k, k0);
            const uint32_t tot = warp_sum(uint32_t(__popc(eq)));
            if (lane == 0 && tot) {
                atomicAdd(cnt + bucket(k0), tot);
                tag(k0);
            }
#pragma unroll
            for (int u = 0; u < kDU; ++u)
                if (((in & ~eq) >> u) & 1u) {
                    atomicAdd(cnt + bucket(k[u]), 1u);
                    tag(k[u]);
                }
        }
    }
    __syncthreads();
    // exclusive scan of the counts: warp w scans segments of 32 counts
    const uint32_t nseg = (nl + 31) / 32, per_w = (nseg + kDT / 32 - 1) / (kDT / 32);
    uint32_t       wrun = 0;
    for (uint32_t q = warp * per_w; q < min(nseg, (warp + 1) * per_w); ++q) {
        const uint32_t i = 32 * q + lane;
        wrun += warp_sum(i < nl ? cnt[i] : 0u);
    }
    if (lane == 0) wsum[warp] = wrun;
    __syncthreads();
    uint32_t base = s;
    for (uint32_t w = 0; w < warp; ++w) base += wsum[w];
    for (uint32_t q = warp * per_w; q < min(nseg, (warp + 1) * per_w); ++q) {
        const uint32_t i   = 32 * q + lane;
        const uint32_t c   = i < nl ? cnt[i] : 0u;
        const uint32_t inc = warp_inclusive_scan(c);
        if (i < nl) {
            const uint32_t start = base + inc - c;
            cnt[i]               = start;
            dir[gb + i]          = (uint64_t(start) << 16) | ((blm[i >> 1] >> (16 * (i & 1))) & 0xffffu);
        }
        base += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (gb + nl == (1ull << g.b) && threadIdx.x == 0) dir[gb + nl] = uint64_t(s + m) << 16;
    __syncthreads();
    if (listed) {
        for (uint32_t q = threadIdx.x; q - lane < m; q += kDT) {
            const bool     ok  = q < m;
            const unsigned act = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                const int32_t  k  = sk[q];
                const uint32_t to = bucket_add(cnt, bucket(k), act);
                okey[to]          = k;
                orow[to]          = sr[q];
            }
        }
    } else {
        for (uint32_t i0 = threadIdx.x; i0 - lane < n; i0 += kDT * kDU) {
            int32_t        k[kDU];
            const uint32_t in = mine(i0, k);
            int32_t        k0;
            const uint32_t eq = heavy(in, k, k0);
            uint32_t       bal[kDU], tot = 0, to = 0;
#pragma unroll
            for (int u = 0; u < kDU; ++u) {
                bal[u] = __ballot_sync(0xffffffffu, (eq >> u) & 1u);
                tot += __popc(bal[u]);
            }
            if (lane == 0 && tot) to = atomicAdd(cnt + bucket(k0), tot);
            to = __shfl_sync(0xffffffffu, to, 0);
#pragma unroll
            for (int u = 0; u < kDU; ++u) {
                if ((in >> u) & 1u) {
                    const uint32_t at = (eq >> u) & 1u ? to + __popc(bal[u] & lt) : atomicAdd(cnt + bucket(k[u]), 1u);
                    okey[at]          = k[u];
                    orow[at]          = i0 + uint32_t(u) * kDT;
                }
                to += __popc(bal[u]);
            }
        }
    }
    __syncthreads();
    // cnt[i] is now the end of bucket i.  A bucket is mixed when a tuple's key differs from its first tuple's.
    const int32_t* ks = okey + s;  // (this block's own stores)
    for (uint32_t q0 = threadIdx.x; q0 < m; q0 += kDT * kDU) {
        int32_t  k[kDU], first[kDU];
        uint32_t local[kDU];
#pragma unroll
        for (int u = 0; u < kDU; ++u) k[u] = q0 + u * kDT < m ? ks[q0 + u * kDT] : 0;
#pragma unroll
        for (int u = 0; u < kDU; ++u) {
            local[u] = bucket(k[u]);
            first[u] = q0 + u * kDT < m ? ks[(local[u] == 0 ? s : cnt[local[u] - 1]) - s] : k[u];
        }
#pragma unroll
        for (int u = 0; u < kDU; ++u)
            if (first[u] != k[u]) atomicOr(mix + (local[u] >> 5), 1u << (local[u] & 31));
    }
    __syncthreads();
    // the partition's buckets are whole mixed words (2^L >= 32), or all of the directory's
    for (uint32_t i = threadIdx.x; i < nmw; i += kDT) mixed[(gb >> 5) + i] = mix[i];
    for (uint32_t i = threadIdx.x; i < nl; i += kDT) {
        const uint32_t b0  = i == 0 ? s : cnt[i - 1];
        const uint32_t len = cnt[i] - b0;
        summary[gb + i]    = len == 0 ? 0ull
                                      : make_summary(ks[b0 - s], (blm[i >> 1] >> (16 * (i & 1))) & 0xffffu, len,
                                                     (mix[i >> 5] >> (i & 31)) & 1u, len == 1 ? orow[b0] : 0u);
    }
}

template <class K>
void prefer_shared(K kernel) {
    HJ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 int(cudaSharedmemCarveoutMaxShared)));
}

constexpr uint64_t kDirectPart = 2048;      // tuples of one of its partitions, about
constexpr uint32_t kDirectBits = 13;        // bucket bits of one, at most

void alloc_table(Table& t, uint32_t b, uint64_t nv, cudaStream_t st) {
    const uint64_t nb = 1ull << b;
    t.dir_bits        = b;
    t.n_tuples        = nv;
    t.dir             = dalloc_n<uint64_t>(nb + 1, st);
    t.keys            = dalloc_n<int32_t>(nv, st);
    t.rows            = dalloc_n<uint32_t>(nv, st);
    t.mixed           = dalloc_n<uint32_t>((nb + 31) / 32, st);
    t.summary         = dalloc_n<uint64_t>(nb, st);
}

template <class K>
void max_dynamic_smem(K kernel, size_t bytes) {
    HJ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
}

// Shared memory of k_bucket_local for 2^L buckets.
size_t local_smem(uint32_t L) {
    const size_t nl = size_t(1) << L;
    return (nl + (nl + 1) / 2 + (nl + 31) / 32 + 2 * size_t(kFuseMax)) * sizeof(uint32_t);
}

int grid_for(uint64_t work, int threads, int per_sm = 4) {
    const uint64_t want = (work + threads - 1) / threads;
    return int(std::min<uint64_t>(std::max<uint64_t>(want, 1), uint64_t(num_sms()) * per_sm));
}

}  // namespace

void build_table(const KeyCol& kc, int dir_bits, int radix_bits, Table& t, uint64_t* scratch_host,
                 cudaStream_t st, int64_t n_valid, int dir_cap_bits) {
    t = Table{};
    // Small builds whose tuples are counted already: one launch.  A partition
    // of about 2048 tuples a block, its buckets at most 2^kDirectBits, whole
    // words of mixed bits.  hj_table_build with and without it, us: 1,000 keys
    // 22 / 63, 16,000 28 / 76, 60,000 42 / 79 (device time 26 / 39), with Zipf
    // keys 50 / 91, with one key only 94 / 103.  At 131,072 keys distinct ones
    // still gain (60 / 80) but a heavy key's single block loses (170 / 104), so
    // the line is at 2^16.
    if (n_valid > 0 && uint64_t(n_valid) <= kDirectKeys && kc.n <= kDirectKeys && radix_bits < 0) {
        const uint32_t b = dir_bits >= 0 ? uint32_t(dir_bits)
                                         : std::min(uint32_t(std::max(0, dir_cap_bits)), ceil_log2(uint64_t(n_valid)));
        uint32_t R = uint64_t(n_valid) > kDirectPart ? ceil_log2((uint64_t(n_valid) + kDirectPart - 1) / kDirectPart) : 0;
        R          = std::max(R, b > kDirectBits ? b - kDirectBits : 0u);
        if (b >= 5) R = std::min(R, b - 5);
        else        R = 0;
        if (b - R <= kDirectBits && (1u << R) <= uint32_t(num_sms()) && (uint64_t(n_valid) >> R) <= 2 * kDirectMax) {
            const Geo g{b, R, b - R};
            alloc_table(t, b, uint64_t(n_valid), st);
            static OncePerDevice once;
            once([&] {
                HJ_CUDA(cudaFuncSetAttribute(k_build_direct, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             int(direct_smem(kDirectBits))));
                prefer_shared(k_build_direct);
            });
            k_build_direct<<<1u << R, kDT, direct_smem(g.L), st>>>(kc, g, t.dir, t.keys, t.rows, t.mixed, t.summary);
            HJ_LAUNCH_CHECK();
            return;
        }
    }
    const uint64_t n_upper = n_valid >= 0 ? uint64_t(n_valid) : kc.n;
    const uint32_t cap     = uint32_t(std::max(0, dir_cap_bits));
    const uint32_t b_upper = dir_bits >= 0 ? uint32_t(dir_bits)
                                           : std::min(cap, ceil_log2(std::max<uint64_t>(n_upper, 1)));
    // partition fan-out: the requested one, raised to what keeps a partition's
    // buckets within one shared-memory histogram (2^13) and capped at b
    const uint32_t R_min   = b_upper > kLocalBits ? b_upper - kLocalBits : 0;
    uint32_t       R       = radix_bits >= 0 ? std::max<uint32_t>(uint32_t(radix_bits), R_min) : R_min;
    R                      = std::min(R, b_upper);
    if (R > kMaxRadix) throw Error(HJ_ERR_INVALID, "build side too large for the radix partition");

    // dynamic shared memory up to the most that any geometry takes
    static OncePerDevice once;
    once([&] {
        prefer_shared(k_part_hist);
        prefer_shared(k_part_scatter<1024>);
        prefer_shared(k_part_scatter<kThreads>);
        prefer_shared(k_bucket_big);
        prefer_shared(k_bucket_phase<1>);
        prefer_shared(k_bucket_phase<3>);
        prefer_shared(k_bucket_local);
        max_dynamic_smem(k_part_hist, sizeof(uint32_t) << kMaxRadix);
        max_dynamic_smem(k_part_scatter<1024>, 200 * 1024);
        max_dynamic_smem(k_part_scatter<kThreads>, (8u << kMaxRadix) + size_t(kTile) * 10);
        max_dynamic_smem(k_bucket_local, local_smem(kLocalBits));
        max_dynamic_smem(k_bucket_big, 8u << kLocalBits);
    });
    // counters that start at zero in one piece: valid keys, finished blocks, partition sizes
    Parts d{};
    auto  free_parts = [&] {
        for (void* p : {(void*)d.n_valid, (void*)d.off, (void*)d.cursor, (void*)d.chunk_off, (void*)d.chunk_part})
            dfree(p, st);
    };
    // chunks of the partitions above kFuseMax tuples, at most
    const uint64_t n_most       = n_valid >= 0 ? uint64_t(n_valid) : kc.n;
    const uint64_t chunks_upper = (n_most + kChunk - 1) / kChunk + n_most / kFuseMax + 1;
    auto run_hist = [&](uint32_t r) {
        const uint32_t P = 1u << r;
        const size_t   z = 4 * sizeof(unsigned long long) + P * sizeof(uint32_t);
        d.n_valid        = reinterpret_cast<unsigned long long*>(dalloc_n<uint8_t>(z, st));
        d.cnt            = reinterpret_cast<uint32_t*>(d.n_valid + 4);
        d.off            = dalloc_n<uint32_t>(P + 1, st);
        d.cursor         = dalloc_n<uint32_t>(P, st);
        d.chunk_off      = dalloc_n<uint32_t>(P + 1, st);
        d.chunk_part     = dalloc_n<uint32_t>(chunks_upper, st);
        HJ_CUDA(cudaMemsetAsync(d.n_valid, 0, z, st));
        const size_t smem = P * sizeof(uint32_t);
        k_part_hist<<<grid_for(kc.n, kThreads), kThreads, smem, st>>>(kc, r, d);
        HJ_LAUNCH_CHECK();
        if (n_valid < 0) {
            readback(scratch_host, d.n_valid, sizeof(uint64_t), true, st);  // page-locked scratch
            HJ_CUDA(cudaStreamSynchronize(st));
        }
    };
    run_hist(R);
    const uint64_t nv = n_valid >= 0 ? uint64_t(n_valid) : scratch_host[0];
    if (nv == 0) {  // UnchainedHash with no tuples: no directory, every probe misses
        free_parts();
        return;
    }
    if (nv > 0xffffffffull) throw Error(HJ_ERR_INVALID, "more than 2^32 build tuples");
    const uint32_t b = dir_bits >= 0 ? uint32_t(dir_bits) : std::min(cap, ceil_log2(nv));
    if (R > b) {  // NULLs shrank the directory below the partition fan-out
        free_parts();
        R = b;
        run_hist(R);
    }
    if (b - R > kLocalBits) throw Error(HJ_ERR_INVALID, "radix_bits too small for the directory");
    const Geo      g{b, R, b - R};
    const uint32_t P = 1u << R;

    int32_t*  tkey = dalloc_n<int32_t>(nv, st);
    uint32_t* trow = dalloc_n<uint32_t>(nv, st);
    {
        // 16384-row tiles (runs of about 8 items per partition at 2048
        // partitions) when the shared memory allows, else 8192-row tiles
        auto smem_for = [&](size_t tile) { return (2 * size_t(P) + 2 * tile) * sizeof(uint32_t) + tile * sizeof(uint16_t); };
        const size_t big = smem_for(size_t(1024) * kItems);
        if (big <= 200 * 1024) {
            k_part_scatter<1024><<<div_up(kc.n, 1024 * kItems), 1024, big, st>>>(kc, R, d.cursor, tkey, trow);
        } else {
            const size_t smem = smem_for(kTile);
            k_part_scatter<kThreads><<<div_up(kc.n, kTile), kThreads, smem, st>>>(kc, R, d.cursor, tkey, trow);
        }
        HJ_LAUNCH_CHECK();
    }

    const uint64_t nb     = 1ull << b;
    alloc_table(t, b, nv, st);
    uint32_t* gcnt        = dalloc_n<uint32_t>(nb, st);
    uint32_t* gbloom      = dalloc_n<uint32_t>(nb, st);
    // partitions of less than a word of mixed bits share one
    if (g.L < 5) HJ_CUDA(cudaMemsetAsync(t.mixed, 0, ((nb + 31) / 32) * sizeof(uint32_t), st));
    k_bucket_local<<<std::min<uint32_t>(P, uint32_t(num_sms())), kLT, local_smem(g.L), st>>>(
        g, d.off, tkey, trow, t.dir, t.keys, t.rows, t.mixed, t.summary);
    HJ_LAUNCH_CHECK();
    if (nv > kFuseMax) {  // (else no partition is larger)
        Big          big{g, d.chunk_off, d.chunk_part, d.off, tkey, trow, gcnt, gbloom, t.dir, t.keys, t.rows, t.mixed, t.summary,
                         reinterpret_cast<uint32_t*>(d.n_valid + 2)};
        if (nv <= kBigOne) {
            void*          args[] = {&big};
            const uint64_t grid   = std::min<uint64_t>(std::max<uint64_t>(P, chunks_upper), kBigBlocks * uint64_t(num_sms()));
            HJ_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k_bucket_big), dim3(unsigned(grid)),
                                                dim3(kThreads), args, 8u << g.L, st));
            HJ_LAUNCH_CHECK();
        } else {
            const unsigned nc = unsigned((nv + kChunk - 1) / kChunk + nv / kFuseMax + 1);
            auto           go = [&](auto kernel, unsigned blocks, size_t smem) {
                kernel<<<blocks, kThreads, smem, st>>>(big);
                HJ_LAUNCH_CHECK();
            };
            go(k_bucket_phase<0>, P, 0);
            go(k_bucket_phase<1>, nc, 8u << g.L);
            go(k_bucket_phase<2>, P, 0);
            go(k_bucket_phase<3>, nc, 4u << g.L);
            go(k_bucket_phase<4>, nc, 0);
            go(k_bucket_phase<5>, P, 0);
        }
    }

    free_parts();
    for (void* p : {(void*)tkey, (void*)trow, (void*)gcnt, (void*)gbloom}) dfree(p, st);
}

void free_table(Table& t, cudaStream_t st) {
    for (void* p : {(void*)t.dir, (void*)t.keys, (void*)t.rows, (void*)t.mixed, (void*)t.summary})
        if (p) dfree(p, st);
    t = Table{};
}

}  // namespace hj
