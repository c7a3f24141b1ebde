// Batched execution of many independent joins (hj_batch_execute), and the
// synthetic instance generator the batched form is measured on
// (hj_batch_generate).
//
// An instance is a chain R0 x R1 x ... x Rm-1 of INT32 equi-joins on one key:
// R0 is probed against R1, the result against R2, and so on.  Every relation is
// (key, payload) with INT32 values and no NULLs.  An instance's result is
// summarised by its row count and an order-independent checksum: the sum mod
// 2^64, over its result rows, of a 64-bit fingerprint of key, payload0 ...
// payloadm-1 (fp_start / fp_add / fp_final below; the same on every path and
// in the oracle).
//
// Batched path: because every join of an instance is on the same key, the
// build relations (R1, R2, ...) are joined among themselves first -- radix
// partitioned together, one histogram, scan and scatter pass over all
// instances, then one block per partition -- into one hash table per
// instance, and R0 is streamed once against it; no intermediate is written.
// The kernels are persistent: grids sized to the resident capacity take work
// items in turn, so instances of very different sizes share the SMs evenly,
// and the whole batch runs without host synchronisation, captured and launched
// as one CUDA graph.  A partition too large for shared memory (heavy duplicate
// keys) flags its instance, which is then recomputed on the plain path.
//
// Plain path: the instances one at a time through the engine's regular
// radix-partitioned table build and two-pass probe (hj_build.cu, hj_probe.cu),
// with a host readback of each join's match count -- what a caller without
// batching runs.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "hj_batch_size.h"
#include "hj_block.cuh"
#include "hj_common.cuh"
#include "hj_kernels.h"

namespace hj {
namespace {


constexpr uint64_t kGold = 0x9e3779b97f4a7c15ull;

// splitmix64's output function (Steele, Lea, Flood 2014; constants as published by Vigna).
__host__ __device__ __forceinline__ uint64_t sm_fin(uint64_t x) {
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}
// Row fingerprint: a fold state over the row's values, one multiply per value
// (state' = (state ^ uint32(v)) * 0x9e3779b97f4a7c15, starting from the key
// xor 0x243f6a8885a308d3), finished by splitmix64's output function.  Joined
// rows carry the state; a result row contributes fp_final(state).
__host__ __device__ __forceinline__ uint64_t fp_add(uint64_t st, int32_t v) {
    return (st ^ uint64_t(uint32_t(v))) * kGold;
}
__host__ __device__ __forceinline__ uint64_t fp_start(int32_t key, int32_t payload0) {
    return fp_add((uint64_t(uint32_t(key)) ^ 0x243f6a8885a308d3ull) * kGold, payload0);
}
__host__ __device__ __forceinline__ uint64_t fp_final(uint64_t st) { return sm_fin(st); }

// ---- generator --------------------------------------------------------------
// Instance relations from (seed, instance, relation): key domain [0, 2b) with
// b = build rows; relation j >= 1 holds b distinct keys perm_j(0 .. b-1), where
// perm_j(x) = (x * 2654435761 + c_j) mod 2b is a bijection of [0, 2b)
// (2654435761 is a prime above 2b); the probe relation R0 draws each key from
// R1's keys with probability match_q24 / 2^24 and from the other half of the
// domain otherwise.  Payloads are uniform 32-bit values.
constexpr uint64_t kPermMul = 2654435761ull;

__host__ __device__ __forceinline__ uint64_t gen_base(uint64_t seed, uint32_t inst, uint32_t rel, uint32_t which) {
    return sm_fin(sm_fin(seed + kGold * (uint64_t(inst) + 1)) + 0xd1b54a32d192ed03ull * (uint64_t(rel) * 4 + which + 1));
}
__host__ __device__ __forceinline__ uint64_t gen_val(uint64_t base, uint64_t row) {
    return sm_fin(base + kGold * (row + 1));
}

__global__ void k_batch_generate(uint64_t seed, uint32_t inst, uint32_t rel, uint64_t b, uint32_t thr, uint64_t rows,
                                 int32_t* __restrict__ keys, int32_t* __restrict__ pay) {
    const uint64_t D      = 2 * b;
    const uint64_t bk     = gen_base(seed, inst, rel, 0);
    const uint64_t bp     = gen_base(seed, inst, rel, 1);
    const uint64_t bx     = gen_base(seed, inst, rel, 2);
    const uint64_t c      = gen_base(seed, inst, rel == 0 ? 1 : rel, 3) % D;
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t r = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; r < rows; r += stride) {
        uint64_t x = r;
        if (rel == 0) {
            const bool hit = (gen_val(bk, r) >> 40) < thr;
            x              = gen_val(bx, r) % b + (hit ? 0 : b);
        }
        keys[r] = int32_t((x * kPermMul + c) % D);
        pay[r]  = int32_t(uint32_t(gen_val(bp, r)));
    }
}

// ---- batched path -----------------------------------------------------------
// Every join of an instance is on the same key, so (R0 x R1) x R2 ... equals
// R0 x (R1 x R2 x ...), and the build relations are small beside R0 (a tenth
// in the synthetic workload).  They are partitioned and joined among
// themselves first, and R0 is then streamed once against the result:
//   1. row counts of the build relations per (relation, partition)  k_bpart_hist
//   2. exclusive scan -> partition offsets in one partitioned buffer
//   3. build rows into partition order                              k_bpart_scatter
//   4. per instance partition: R2, R3, ... become shared-memory
//      tables, R1's rows are looked up in them, and the rows whose
//      key is in all go to the partition's piece of table F, their
//      partners' payloads beside the slot                           k_bt_build
//   5. R0 rows looked up in F                                       k_bt_probe
//   6. R0 rows whose key repeats: their results enumerated          k_bt_enum
// Instance i gets p_i partition bits (about `part_rows` build rows per
// partition summed over its build relations); a row belongs to partition
// top_p_i(hash(key)).  A partition whose build rows exceed the shared-memory
// capacity (heavy duplicates) flags its instance, which is then recomputed on
// the plain path.
//
// F is read in place of a partitioned R0: random 32-byte reads of tables up to
// 64 MB (4M build rows) run at 292e9/s on a GB300 (one L2 sector per SM and cycle;
// 84e9/s at 256 MB, past the L2), and at 273e9 rows/s together with the stream of R0,
// where a partition of R0 beside the build relations (28 bytes a row in three
// passes) took 17 ps a row.  64 instances of 1k .. 4M build rows (364M R0
// rows): 5.5 ms with R0 partitioned, 3.5 ms so.  Tables built in place by
// atomics, without the partition, took 30 ps a build row to insert and 50 to
// reduce, against 7 to partition and 13 to build here.
constexpr int      kPT         = 512;   // threads of the partition and join blocks
constexpr uint32_t kPartItem   = 8192;  // rows per partition-pass work item
constexpr uint32_t kMaxPartBits = 11;
constexpr uint32_t kMaxRel     = 8;     // relations per instance

struct RelInst {  // one relation of one instance
    const int32_t* keys;
    const int32_t* pay;
    uint64_t       rows;
    uint64_t       item_base;  // first work item (build relations: of the partition passes, then R0s: of the probe)
    uint64_t       part_base;  // global partition id of partition 0 (R0s: of R1's, which their keys are looked up in)
    uint32_t       pbits;
    uint32_t       inst;
    uint32_t       irows;  // R0s: rows per work item
    uint32_t       nrel;
    uint32_t       fbase, flog;  // R0s: first word of the instance's filter; log2 of a partition's bits
};

// One work item of the probe, whole, so that a block waits for one load.
struct Item {
    const int32_t *k, *p;
    uint64_t       part_base;
    uint32_t       n, inst, pbits, nt;  // rows; instance; its partition bits and tables beside F
    uint32_t       fbase, flog;         // and its filter
};

struct InstInfo {
    uint64_t part_base;  // global partition id of (R1, partition 0); relation j, partition l: + (j - 1) * 2^pbits + l
    uint64_t ip_base;    // first instance partition (2^pbits of them)
    uint32_t nrel;
    uint32_t pbits;
    uint32_t fbase;      // first word of its filter (2^(pbits + flog - 5) of them)
    uint32_t flog;       // log2 of a partition's bits there
};

// Per-instance results and flags, cleared together.
struct InstOut {
    unsigned long long rows, sum;
    uint32_t           ovf;   // a partition too large for shared memory, or a row equal to kFree
    uint32_t           lists;  // its partitions with listed keys (k_bt_enum)
};

// A table in buckets of four (key, payload) slots, 32 bytes (one L2 sector,
// read by one 256-bit load).  A row goes to the first free slot from its home
// bucket on (linear probing over the piece's buckets); equal keys take a slot
// each.  A full bucket that rows went past has its last two slots in
// descending order, else ascending, so a lookup goes on only from those (5% of
// the buckets at half load; 14% are full).
// A piece is the part of a table that one instance partition's rows are in:
// its first bucket, and its buckets.  Pieces without rows are bucket 0, which is
// free.
// Keys that R2, R3, ... hold more than once, and keys with so many rows in R1 that
// they would fill runs of buckets which every lookup beside them walks, are not
// in F.  Their partition has a piece of listed keys for each of its relations: a
// slot a key, with the end of the key's list of payloads in place of a payload.
// The lists take the place of the partitioned rows, the last row of each with
// the list's length.  (A wave has fewer rows than 2^31, so an end is no kFree's.)
struct Piece {
    uint32_t first, nbk;  // nbk 0: no listed keys
};
// F is filled anew, without the keys of home buckets of more than kHeavy rows,
// when linear probing takes more than kSteps steps a row.  64 chains of 8,000
// build rows, 7,900 of one key, us: 410 (all of them in F: 10,044); of 16,000
// Zipf(0.8) rows 512 (1,235), Zipf(1.1) 562 (5,361).  kSteps at 1 gives up keys of 8
// rows each, which are as fast in F (497, 411); at 4 uniform keys of 16 rows stay
// (614, 525).
constexpr uint32_t kSteps = 2, kHeavy = 12;
// A filter of an instance's listed keys, for those who look for rows of them: two
// bits of a word a key, each partition with words of its own, at most as many as
// fit a block's shared memory (2^17 bits), and 8 to 16 bits a build row.  Few rows
// of other keys pass it, and what passes takes three dependent loads.
constexpr uint32_t kFilterPart = 13, kFilterAll = 17;

// A free slot.  A build row that is this very pair cannot be stored: its
// instance is left to the plain path.
constexpr uint64_t kFree = 0x8181818181818181ull;

__device__ __forceinline__ uint32_t part_of(int32_t k, uint32_t pbits) {
    return pbits ? fib_hi(k) >> (32 - pbits) : 0u;
}

// Largest i < n with key(i) <= t, for keys ascending in i (entries without
// work share their key with the next entry, so this is the owner of t).
template <class F>
__device__ __forceinline__ uint32_t owner(uint32_t n, uint64_t t, F key) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (key(mid) <= t) lo = mid;
        else               hi = mid;
    }
    return lo;
}

// The block's next work item from the queue (uniform across the block).
__device__ __forceinline__ uint64_t next_item(unsigned long long* q, unsigned long long* sh) {
    __syncthreads();
    if (threadIdx.x == 0) *sh = atomicAdd(q, 1ull);
    __syncthreads();
    return *sh;
}

// In-place scan of n shared-memory counters (exclusive or inclusive).  Warp w
// scans one contiguous slice 32 counters at a time (lane l touches counter
// i + l: no bank conflicts), then the slices are offset by the scanned slice
// totals.  `wsum` holds >= 32 words.  Every thread of the block must call it.
__device__ __forceinline__ void smem_scan(uint32_t* a, uint32_t n, bool inclusive, uint32_t* wsum) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t per  = ((n + 31) / 32 + nw - 1) / nw * 32;
    const uint32_t b = min(n, warp * per), e = min(n, b + per);
    uint32_t       carry = 0;
    for (uint32_t i = b; i < e; i += 32) {
        const uint32_t idx = i + lane;
        const uint32_t v   = idx < e ? a[idx] : 0u;
        const uint32_t inc = warp_inclusive_scan(v);
        if (idx < e) a[idx] = carry + (inclusive ? inc : inc - v);
        carry += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) wsum[warp] = carry;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < nw ? wsum[lane] : 0u;
        const uint32_t x = warp_inclusive_scan(w);
        if (lane < nw) wsum[lane] = x - w;
    }
    __syncthreads();
    const uint32_t off = wsum[warp];
    if (off)
        for (uint32_t i = b + lane; i < e; i += 32) a[i] += off;
    __syncthreads();
}

// Where the pieces go: buckets are handed out from a counter (the memory is
// sized for the rows of all build relations).
struct Tables {
    uint64_t* tab;
    uint32_t* side;      // `stride` words per slot: the payloads of an F slot's partners
    uint32_t* next;      // buckets handed out, from 1 on
    uint32_t* lists;     // zeroed; set when any partition has listed keys
    uint32_t  buckets;   // of the memory
    uint32_t  stride;
    uint32_t  slot_q16;  // buckets per row, in 65536ths
};

// 0. the relation of every partition-pass item, the probe's items and the
// instance of every instance partition, so that a block finds its work with one
// load instead of a binary search of dependent loads
__global__ void k_item_rel(const RelInst* __restrict__ R, uint32_t nr, uint64_t bitems, uint64_t items,
                           uint32_t* __restrict__ rmap, Item* __restrict__ imap, const InstInfo* __restrict__ I,
                           uint32_t n, uint64_t nip, uint32_t* __restrict__ pmap, Tables T) {
    if (blockIdx.x == 0 && threadIdx.x < 4) {  // bucket 0 stays free
        T.tab[threadIdx.x] = kFree;
        if (threadIdx.x == 0) *T.next = 1;
    }
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < items + nip; t += stride) {
        if (t >= items) {
            pmap[t - items] = owner(n, t - items, [&](uint32_t i) { return I[i].ip_base; });
            continue;
        }
        const uint32_t ri = owner(nr, t, [&](uint32_t i) { return R[i].item_base; });
        if (t < bitems) {
            rmap[t] = ri;
            continue;
        }
        const RelInst& r  = R[ri];
        const uint64_t r0 = (t - r.item_base) * r.irows;
        imap[t - bitems]  = Item{r.keys + r0, r.pay + r0, r.part_base, uint32_t(min(r.rows - r0, uint64_t(r.irows))),
                                r.inst, r.pbits, r.nrel - 2, r.fbase, r.flog};
    }
}

// 1. per (relation, partition) row counts
__global__ void __launch_bounds__(kPT)
    k_bpart_hist(const RelInst* __restrict__ R, const uint32_t* __restrict__ rmap, uint64_t items,
                 uint32_t* __restrict__ cnt) {
    // Items of equal size go to the blocks round robin (no queue, no barrier
    // per item).  The block's counts accumulate in shared memory over its items
    // of one relation and go to global memory when the relation changes (items
    // are numbered relation by relation), not once per item.
    extern __shared__ uint32_t hist[];
    uint32_t cur = ~0u;  // relation whose counts the shared histogram holds
    auto flush = [&]() {
        if (cur == ~0u) return;
        const RelInst& c = R[cur];
        for (uint32_t k = threadIdx.x; k < (1u << c.pbits); k += kPT)
            if (hist[k]) atomicAdd(cnt + c.part_base + k, hist[k]);
    };
    for (uint64_t t = blockIdx.x; t < items; t += gridDim.x) {
        const uint32_t ri = __ldg(rmap + t);
        const RelInst& s  = R[ri];
        const uint64_t r0 = (t - s.item_base) * kPartItem;
        const uint64_t r1 = min(s.rows, r0 + kPartItem);
        if (r0 >= r1) continue;
        if (s.pbits == 0) {
            if (threadIdx.x == 0) atomicAdd(cnt + s.part_base, uint32_t(r1 - r0));
            continue;
        }
        const uint32_t np2 = 1u << s.pbits;
        if (ri != cur) {
            __syncthreads();  // the last item's atomics are done
            flush();
            __syncthreads();
            for (uint32_t k = threadIdx.x; k < np2; k += kPT) hist[k] = 0;
            cur = ri;
            __syncthreads();
        }
        constexpr int kPer = kPartItem / kPT;
        int32_t       kv[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {  // all loads in flight before the atomics
            const uint64_t r = r0 + threadIdx.x + uint64_t(j) * kPT;
            if (r < r1) kv[j] = __ldg(s.keys + r);
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j)
            if (r0 + threadIdx.x + uint64_t(j) * kPT < r1) atomicAdd(&hist[part_of(kv[j], s.pbits)], 1u);
    }
    __syncthreads();
    flush();
}

// 4-byte global -> shared copy that completes asynchronously (cp.async);
// cp_async_wait_all waits for this thread's copies.
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// 3. rows into partition order.  Shared memory: the item's payloads in row
// order (copied asynchronously while the keys are ranked), its keys sorted by
// partition with each one's row in the item, then per partition its count,
// its first sorted row and its global base.
__global__ void __launch_bounds__(kPT, 2)
    k_bpart_scatter(const RelInst* __restrict__ R, const uint32_t* __restrict__ rmap, uint64_t items,
                    unsigned long long* q,
                    const uint64_t* __restrict__ off, uint32_t* __restrict__ fill, uint32_t pmax,
                    int2* __restrict__ okp) {
    extern __shared__ __align__(16) unsigned char smem[];
    int32_t*  spay  = reinterpret_cast<int32_t*>(smem);   // row order
    int32_t*  skey  = spay + kPartItem;                    // partition order
    uint32_t* hist  = reinterpret_cast<uint32_t*>(skey + kPartItem);
    uint32_t* loff  = hist + (1u << pmax);
    uint64_t* gbase = reinterpret_cast<uint64_t*>(loff + (1u << pmax));
    uint16_t* sidx  = reinterpret_cast<uint16_t*>(gbase + (1u << pmax));  // partition order: row in the item
    __shared__ unsigned long long sh;
    __shared__ uint32_t           wsum[32];
    constexpr int kPer = kPartItem / kPT;
    static_assert(kPartItem <= 65536, "row in the item fits 16 bits");
    for (uint64_t t = next_item(q, &sh); t < items; t = next_item(q, &sh)) {
        const RelInst& s  = R[__ldg(rmap + t)];
        const uint64_t r0 = (t - s.item_base) * kPartItem;
        const uint64_t r1 = min(s.rows, r0 + kPartItem);
        if (r0 >= r1) continue;
        const uint32_t pb  = s.pbits;
        const uint32_t np2 = 1u << pb;
        for (uint32_t k = threadIdx.x; k < np2; k += kPT) hist[k] = 0;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const uint32_t i = threadIdx.x + uint32_t(j) * kPT;
            if (r0 + i < r1) cp_async4(spay + i, s.pay + r0 + i);
        }
        __syncthreads();
        uint32_t pr[kPer];  // partition << 16 | rank in the partition
        int32_t  kv[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const uint64_t r = r0 + threadIdx.x + uint64_t(j) * kPT;
            if (r < r1) kv[j] = __ldg(s.keys + r);
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const uint64_t r = r0 + threadIdx.x + uint64_t(j) * kPT;
            if (r < r1) {
                const uint32_t k = part_of(kv[j], pb);
                pr[j]            = (k << 16) | atomicAdd(&hist[k], 1u);
            }
        }
        __syncthreads();
        // global ranges first (hist still holds the counts), then local offsets;
        // a thread's reservations four at a time, all four in flight before
        // any result is stored
        for (uint32_t k0 = threadIdx.x; k0 < np2; k0 += 4 * kPT) {
            uint64_t g[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t k = k0 + uint32_t(u) * kPT;
                const uint32_t c = k < np2 ? hist[k] : 0u;
                g[u]             = c ? off[s.part_base + k] + atomicAdd(fill + s.part_base + k, c) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t k = k0 + uint32_t(u) * kPT;
                if (k < np2 && hist[k]) gbase[k] = g[u];
            }
        }
        for (uint32_t k = threadIdx.x; k < np2; k += kPT) loff[k] = hist[k];
        __syncthreads();
        smem_scan(loff, np2, false, wsum);
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const uint32_t i = threadIdx.x + uint32_t(j) * kPT;
            if (r0 + i < r1) {
                const uint32_t pos = loff[pr[j] >> 16] + (pr[j] & 0xffffu);
                skey[pos]          = kv[j];
                sidx[pos]          = uint16_t(i);
            }
        }
        cp_async_wait_all();
        __syncthreads();
        const uint32_t m = uint32_t(r1 - r0);
        for (uint32_t j = threadIdx.x; j < m; j += kPT) {
            const int32_t  k   = skey[j];
            const uint32_t p   = part_of(k, pb);
            const uint64_t pos = gbase[p] + (j - loff[p]);
            okp[pos]           = make_int2(k, spay[sidx[j]]);
        }
        __syncthreads();  // the next item overwrites spay
    }
}

struct Slots {
    uint64_t s[4];
};
__device__ __forceinline__ Slots load_bucket(const uint64_t* tab, uint64_t b) {
    Slots r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(r.s[0]), "=l"(r.s[1]), "=l"(r.s[2]), "=l"(r.s[3])
                 : "l"(tab + 4 * b));
    return r;
}
// Home bucket of a key in a piece of nbk buckets: the first steps of
// MurmurHash3's 32-bit finaliser (Appleby), then the high product.  The
// partition's multiplicative hash will not do: keys in arithmetic progression
// can fall into few of its buckets, and linear probing then runs through them
// (64 chains of 1k .. 16k build rows: 148 us of probing, with this hash 41 us).
__device__ __forceinline__ uint32_t mix_of(int32_t k) {
    uint32_t h = uint32_t(k);
    h = (h ^ (h >> 16)) * 0x85ebca6bu;
    return (h ^ (h >> 13)) * 0xc2b2ae35u;
}
__device__ __forceinline__ uint32_t home_of(int32_t k, uint32_t nbk) { return __umulhi(mix_of(k), nbk); }
// A key's bits in a partition's 2^log bits of the filter, and the word that they are in.
__device__ __forceinline__ uint32_t filter_bits(int32_t k, uint32_t log, uint32_t& word) {
    const uint32_t h = mix_of(k);
    word             = (h >> 10) & ((1u << (log - 5)) - 1);
    return (1u << (h & 31)) | (1u << ((h >> 5) & 31));
}
__device__ __forceinline__ uint64_t slot_of(int32_t k, int32_t p) {
    return uint64_t(uint32_t(k)) | (uint64_t(uint32_t(p)) << 32);
}
__device__ __forceinline__ int32_t slot_key(uint64_t s) { return int32_t(uint32_t(s)); }
__device__ __forceinline__ int32_t slot_pay(uint64_t s) { return int32_t(uint32_t(s >> 32)); }
__device__ __forceinline__ bool goes_on(const Slots& s) { return s.s[2] >= s.s[3] && s.s[3] != kFree; }
__device__ __forceinline__ uint32_t next_bucket(uint32_t b, uint32_t nbk) { return b + 1 == nbk ? 0u : b + 1; }

__device__ __forceinline__ uint64_t part_rows(const uint64_t* off, uint64_t pid) { return off[pid + 1] - off[pid]; }

// 4. One block per instance partition.  Shared memory: rows of R2, R3, ...
// (keys, payloads; at most `cap` rows together), then per table its bucket
// bounds -- table j (relation j + 2) has 2^bits_j buckets after a gap word;
// after one inclusive scan over all tables' counts and the scatter, bucket b
// of table j holds tuples [S[ts_j + b + 1], S[ts_j + b + 2]) -- and the row
// counters of the piece that is being written.
// R1's rows are looked up twice: counted, so that the piece is as large as its
// rows need (tables of long chains shrink with every relation), then placed.
// Bound by the latency of its phases: two blocks an SM, each at another one.
// Listed keys take some 13 us more a block (8 chains of 1M rows, a hundredth
// repeated in R2: 428 us, without 248): each relation's table is made by atomics
// on its slots in L2, counts first, then the lists' starts, then the rows.
constexpr int kBuildT = 512;
__global__ void __launch_bounds__(kBuildT, 2)
    k_bt_build(const InstInfo* __restrict__ I, const uint32_t* __restrict__ pmap, uint64_t nip,
               const uint64_t* __restrict__ off, int2* kp, uint32_t cap, uint32_t scap, uint32_t fcap,
               uint32_t max_bits, uint32_t load_q8, Tables T, Piece* __restrict__ pieces, Piece* __restrict__ listed,
               uint32_t* __restrict__ filters, InstOut* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem[];
    int32_t*  skey = reinterpret_cast<int32_t*>(smem);
    int32_t*  spay = skey + cap;
    uint32_t* S    = reinterpret_cast<uint32_t*>(spay + cap);
    __shared__ uint32_t wsum[32];
    __shared__ uint32_t g_tb[kMaxRel], g_tn[kMaxRel], g_ts[kMaxRel], g_to[kMaxRel + 1], g_words, g_skip, g_cnt, g_nl,
        g_first, g_steps;
    __shared__ uint64_t g_src[kMaxRel];
    for (uint64_t e = blockIdx.x; e < nip; e += gridDim.x) {
        const uint32_t  ii  = pmap[e];
        const InstInfo& s   = I[ii];
        const uint32_t  pb  = s.pbits, nt = s.nrel - 2;
        const uint64_t  np2 = 1ull << pb, l = e - s.ip_base;
        const uint64_t  pid = s.part_base + l;
        __syncthreads();  // the last partition is done with shared memory
        if (threadIdx.x == 0) {
            uint64_t all   = part_rows(off, pid);
            bool     empty = all == 0;
            uint32_t nb    = 0;
            for (uint32_t j = 0; j < nt; ++j) {
                const uint64_t q = pid + (j + 1) * np2, rows = part_rows(off, q);
                all += rows;
                empty |= rows == 0;
                g_src[j] = off[q];
                g_tn[j]  = uint32_t(rows);
                g_to[j]  = nb;
                nb += g_tn[j];
                const uint32_t want = uint32_t((uint64_t(g_tn[j]) * 256 + load_q8 - 1) / load_q8);
                g_tb[j]             = min(max_bits, max(1u, want > 1 ? 32u - __clz(want - 1) : 1u));
            }
            uint32_t words = 0;
            for (;;) {  // shrink the largest tables until the bucket bounds fit
                uint32_t big = 0;
                words        = 0;
                for (uint32_t j = 0; j < nt; ++j) {
                    words += (1u << g_tb[j]) + 2;
                    if (g_tb[j] > g_tb[big]) big = j;
                }
                if (words <= scap || g_tb[big] == 1) break;
                --g_tb[big];
            }
            uint32_t w = 0;
            for (uint32_t j = 0; j < nt; ++j) {
                g_ts[j] = w;
                w += (1u << g_tb[j]) + 2;
            }
            g_words = words;
            // a partition too large for shared memory: the plain path redoes the instance
            const bool big = all > cap || words > scap;
            if (big && !empty) out[ii].ovf = 1;
            g_skip  = big || empty;
            g_cnt = g_nl = 0;
            pieces[pid]  = Piece{0, 1};
            listed[pid]  = Piece{0, 0};
        }
        __syncthreads();
        if (g_skip) continue;
        const uint32_t words = g_words, n1 = uint32_t(part_rows(off, pid));
        const int2*    r1    = kp + off[pid];
        // row counters of the piece being written, two to a word (a piece has less than 2^16 rows):
        // behind the tables, or in their place when there are none
        uint32_t*      fcnt  = nt ? S + scap : reinterpret_cast<uint32_t*>(smem);
        const uint32_t nbmax = nt ? fcap : 2 * (2 * cap + scap) + fcap;
        auto           count = [&](uint32_t b) { return (fcnt[b >> 1] >> (16 * (b & 1))) & 0xffffu; };
        auto bucket = [&](uint32_t j, int32_t k) { return (fib_hi(k) << pb) >> (32 - g_tb[j]); };
        // tables of R2, R3, ...
        for (uint32_t w = threadIdx.x; w < words; w += kBuildT) S[w] = 0;
        __syncthreads();
        // four rows per thread in flight per step, loads before the atomics
        constexpr uint32_t kBU = 4;
        for (uint32_t j = 0; j < nt; ++j) {
            const uint32_t tn = g_tn[j];
            const int2*    qj = kp + g_src[j];
            for (uint32_t r = threadIdx.x; r < tn; r += kBU * kBuildT) {
                int2 kv[kBU];
#pragma unroll
                for (uint32_t u = 0; u < kBU; ++u) kv[u] = r + u * kBuildT < tn ? __ldg(qj + r + u * kBuildT) : make_int2(0, 0);
#pragma unroll
                for (uint32_t u = 0; u < kBU; ++u)
                    if (r + u * kBuildT < tn) atomicAdd(&S[g_ts[j] + bucket(j, kv[u].x) + 1], 1u);
            }
        }
        __syncthreads();
        if (nt) smem_scan(S, words, true, wsum);
        for (uint32_t j = 0; j < nt; ++j) {
            const uint32_t tn = g_tn[j];
            const int2*    qj = kp + g_src[j];
            for (uint32_t r = threadIdx.x; r < tn; r += kBU * kBuildT) {
                int2 kv[kBU];
#pragma unroll
                for (uint32_t u = 0; u < kBU; ++u) kv[u] = r + u * kBuildT < tn ? __ldg(qj + r + u * kBuildT) : make_int2(0, 0);
#pragma unroll
                for (uint32_t u = 0; u < kBU; ++u)
                    if (r + u * kBuildT < tn) {
                        const uint32_t pos = atomicSub(&S[g_ts[j] + bucket(j, kv[u].x) + 1], 1u) - 1;
                        skey[pos]          = kv[u].x;
                        spay[pos]          = kv[u].y;
                    }
            }
        }
        __syncthreads();
        // rows of table j with key k: their number (0, 1, or 2 for more) and one of them
        auto lookup = [&](uint32_t j, int32_t k, uint32_t& one) {
            const uint32_t w = g_ts[j] + bucket(j, k), be = S[w + 2];
            uint32_t       c = 0;
            for (uint32_t y = S[w + 1]; y < be && c < 2; ++y)
                if (skey[y] == k) {
                    one = y;
                    ++c;
                }
            return c;
        };
        // R1 rows that are in every table, and the ones of them whose key a table
        // holds more than once: bits of this thread's rows, and how many
        static_assert((2u << 13) / kBuildT <= 32, "a bit for each of a thread's rows");
        uint32_t in_f = 0, in_l = 0;
        for (uint32_t r = threadIdx.x, i = 0; r < n1; r += kBuildT, ++i) {
            bool all = true, many = false;
            if (nt) {
                const int32_t k = __ldg(r1 + r).x;
                for (uint32_t j = 0; j < nt && all; ++j) {
                    uint32_t       y;
                    const uint32_t c = lookup(j, k, y);
                    all              = c > 0;
                    many |= c > 1;
                }
            }
            in_f |= uint32_t(all && !many) << i;
            in_l |= uint32_t(all && many) << i;
        }
        auto count_rows = [&](uint32_t bits, uint32_t* to) {
            const uint32_t c = warp_sum(uint32_t(__popc(bits)));
            if ((threadIdx.x & 31) == 0 && c) atomicAdd(to, c);
        };
        count_rows(in_f, &g_cnt);
        count_rows(in_l, &g_nl);
        __syncthreads();
        // Buckets from the table memory, at g_first (it is sized for all of them; were
        // it short, the instance would go to the plain path)
        auto reserve = [&](uint32_t nbk) {
            __syncthreads();
            if (threadIdx.x == 0) {
                g_first = atomicAdd(T.next, nbk);
                if (g_first > T.buckets || nbk > T.buckets - g_first) out[ii].ovf = g_skip = 1;
            }
            __syncthreads();
            return g_skip == 0;
        };
        // its slots emptied, and `words` counters beside it
        auto empty = [&](uint32_t first, uint32_t nbk, uint32_t* cnt, uint32_t words) {
            __syncthreads();
            for (uint32_t w = threadIdx.x; w < words; w += kBuildT) cnt[w] = 0;
            ulonglong2* to = reinterpret_cast<ulonglong2*>(T.tab + 4 * uint64_t(first));
            for (uint32_t b = threadIdx.x; b < 2 * nbk; b += kBuildT) to[b] = make_ulonglong2(kFree, kFree);
            __syncthreads();
        };
        auto buckets = [&](uint32_t n) { return min(nbmax, batch_piece_buckets(n, T.slot_q16)); };
        // f(bit, row, key, payload) for R1's rows in `bits`
        auto rows_of = [&](uint32_t bits, auto f) {
            for (; bits; bits &= bits - 1) {
                const uint32_t i = __ffs(bits) - 1, r = i * kBuildT + threadIdx.x;
                const int2     kv = __ldg(r1 + r);
                f(1u << i, r, kv.x, kv.y);
            }
        };
        auto add = [&](uint32_t b) {
            return (atomicAdd(fcnt + (b >> 1), 1u << (16 * (b & 1))) >> (16 * (b & 1))) & 0xffffu;
        };
        uint32_t nf = g_cnt, nl = g_nl, nbk = 0;
        if (nf + nl == 0) continue;
        // F's piece and behind it R1's listed keys, however the rows divide
        if (!reserve(batch_pair_buckets(nf + nl, T.slot_q16))) continue;
        const uint32_t first = g_first;
        // F: a slot a row (they fit: a fifth of the slots or more stays free)
        for (uint32_t limit = kSteps * nf; nf; limit = ~0u) {
            nbk = buckets(nf);
            if (threadIdx.x == 0) g_steps = 0;
            empty(first, nbk, fcnt, (nbk + 1) / 2);
            uint32_t steps = 0;  // past full buckets; in g_steps 8 at a time
            rows_of(in_f, [&](uint32_t, uint32_t, int32_t k, int32_t p) {
                if (*const_cast<volatile uint32_t*>(&g_steps) > limit) return;
                uint32_t b = home_of(k, nbk), r;
                while ((r = add(b)) >= 4) {
                    b = next_bucket(b, nbk);
                    if ((++steps & 7) == 0 && atomicAdd(&g_steps, 8u) >= limit) return;
                }
                const uint64_t slot = uint64_t(first + b) * 4 + r, v = slot_of(k, p);
                T.tab[slot] = v;
                if (v == kFree) out[ii].ovf = 1;
                for (uint32_t j = 0; j < nt; ++j) {
                    uint32_t y = 0;
                    lookup(j, k, y);
                    T.side[slot * T.stride + j] = uint32_t(spay[y]);
                }
            });
            steps = warp_sum(steps & 7);
            if ((threadIdx.x & 31) == 0 && steps) atomicAdd(&g_steps, steps);
            __syncthreads();
            if (limit == ~0u || g_steps <= limit) break;
            // the keys of heavy home buckets are listed, and F takes the others
            for (uint32_t b = threadIdx.x; b < (nbk + 1) / 2; b += kBuildT) fcnt[b] = 0;
            __syncthreads();
            rows_of(in_f, [&](uint32_t, uint32_t, int32_t k, int32_t) { add(home_of(k, nbk)); });
            __syncthreads();
            uint32_t heavy = 0;
            rows_of(in_f, [&](uint32_t bit, uint32_t, int32_t k, int32_t) {
                if (count(home_of(k, nbk)) > kHeavy) heavy |= bit;
            });
            in_f &= ~heavy;
            in_l |= heavy;
            count_rows(heavy, &g_nl);
            __syncthreads();
            nf -= g_nl - nl;
            nl = g_nl;
        }
        if (nf) {
            if (threadIdx.x == 0) pieces[pid] = Piece{first, nbk};
            // the order of each full bucket's last slots, and of their partners
            for (uint32_t b = threadIdx.x; b < nbk; b += kBuildT) {
                const uint32_t n = count(b);
                if (n < 4) continue;
                const uint64_t c = uint64_t(first + b) * 4 + 2;
                const uint64_t x = T.tab[c], y = T.tab[c + 1];
                if ((n > 4) == (x >= y)) continue;
                T.tab[c]     = y;
                T.tab[c + 1] = x;
                for (uint32_t j = 0; j < nt; ++j) {
                    const uint32_t w                  = T.side[c * T.stride + j];
                    T.side[c * T.stride + j]          = T.side[(c + 1) * T.stride + j];
                    T.side[(c + 1) * T.stride + j]    = w;
                }
            }
        } else {
            nbk = 0;
        }
        if (nl == 0) continue;
        // The listed keys.  R1's rows of them come to the others' in shared memory,
        // as the lists take the place of what has been read.
        __syncthreads();
        const uint32_t o1 = nt ? g_to[nt - 1] + g_tn[nt - 1] : 0u;
        const uint32_t flog   = s.flog;
        uint32_t*      filter = S + scap + (fcap + 1) / 2;
        for (uint32_t w = threadIdx.x; w < 1u << (flog - 5); w += kBuildT) filter[w] = 0;
        __syncthreads();
        rows_of(in_l, [&](uint32_t, uint32_t r, int32_t k, int32_t p) {
            skey[o1 + r]     = k;
            spay[o1 + r]     = p;
            uint32_t       w;
            const uint32_t m = filter_bits(k, flog, w);
            atomicOr(filter + w, m);
        });
        __syncthreads();
        for (uint32_t w = threadIdx.x; w < 1u << (flog - 5); w += kBuildT)
            filters[s.fbase + (uint32_t(l) << (flog - 5)) + w] = filter[w];
        if (threadIdx.x == 0) {
            atomicAdd(&out[ii].lists, 1u);
            *T.lists = 1;
        }
        const uint32_t  behind_f = first + nbk;
        uint32_t*       passed = S + scap;  // a bit a bucket: a key went past it
        const uint64_t* keys   = nullptr;   // R1's piece
        uint32_t        nbk1   = 0;
        // (this block's atomics and stores of a moment ago: past the L1)
        auto fresh = [&](const uint64_t* tab, uint32_t b) {
            Slots q;
#pragma unroll
            for (int i = 0; i < 4; ++i) q.s[i] = *const_cast<const volatile uint64_t*>(tab + 4 * b + i);
            return q;
        };
        auto slot_in = [&](const Slots& q, int32_t k) {
            int at = -1;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (q.s[i] != kFree && slot_key(q.s[i]) == k) at = i;
            return at;
        };
        for (uint32_t j = 0; j <= nt; ++j) {
            const uint32_t o = j ? g_to[j - 1] : o1;
            const uint32_t dst = uint32_t(j ? g_src[j - 1] : off[pid]);
            uint32_t       bits = in_l;
            if (j) {  // the rows whose key is listed
                bits = 0;
                for (uint32_t r = threadIdx.x, i = 0; r < g_tn[j - 1]; r += kBuildT, ++i) {
                    const int32_t  k = skey[o + r];
                    uint32_t       w;
                    const uint32_t m = filter_bits(k, flog, w);
                    if ((filter[w] & m) != m) continue;
                    for (uint32_t b = home_of(k, nbk1);; b = next_bucket(b, nbk1)) {
                        const Slots q    = fresh(keys, b);
                        const bool  here = slot_in(q, k) >= 0;
                        bits |= uint32_t(here) << i;
                        if (here || !goes_on(q)) break;
                    }
                }
                if (threadIdx.x == 0) g_nl = 0;
                __syncthreads();
                count_rows(bits, &g_nl);
            }
            auto each = [&](auto f) {
                for (uint32_t m = bits; m; m &= m - 1) {
                    const uint32_t r = o + (__ffs(m) - 1) * kBuildT + threadIdx.x;
                    f(skey[r], spay[r]);
                }
            };
            __syncthreads();
            const uint32_t nbk = buckets(g_nl);
            if (j && !reserve(nbk)) break;
            const uint32_t lf = j ? g_first : behind_f;
            if (threadIdx.x == 0) listed[pid + j * np2] = Piece{lf, nbk};
            empty(lf, nbk, passed, (nbk + 31) / 32);
            uint64_t* const tab = T.tab + 4 * uint64_t(lf);
            auto word = [&](uint64_t slot) { return reinterpret_cast<uint32_t*>(tab + slot) + 1; };
            // each key's slot, with the number of its rows
            each([&](int32_t k, int32_t) {
                for (uint32_t b = home_of(k, nbk);; b = next_bucket(b, nbk)) {
                    const Slots q  = fresh(tab, b);
                    int         at = -1;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (at >= 0) continue;
                        uint64_t v = q.s[i];
                        if (v == kFree) {
                            v = atomicCAS(reinterpret_cast<unsigned long long*>(tab + 4 * b + i), kFree, slot_of(k, 0));
                            if (v == kFree) v = slot_of(k, 0);
                        }
                        if (slot_key(v) == k) at = i;
                    }
                    if (at >= 0) {
                        atomicAdd(word(4 * b + at), 1u);
                        break;
                    }
                    atomicOr(passed + (b >> 5), 1u << (b & 31));
                }
            });
            __syncthreads();
            // the number becomes the list's start
            uint32_t at = dst;
            for (uint32_t b0 = 0; b0 < nbk; b0 += kBuildT) {
                const uint32_t b = b0 + threadIdx.x;
                uint32_t       c[4], sum = 0;
                Slots          q;
                if (b < nbk) q = fresh(tab, b);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    c[i] = b < nbk && q.s[i] != kFree ? uint32_t(slot_pay(q.s[i])) : 0u;
                    sum += c[i];
                }
                const uint32_t inc = warp_inclusive_scan(sum);
                if ((threadIdx.x & 31) == 31) wsum[threadIdx.x >> 5] = inc;
                __syncthreads();
                uint32_t x = at + inc - sum;
                for (uint32_t w = 0; w < kBuildT / 32; ++w) {
                    if (w < threadIdx.x >> 5) x += wsum[w];
                    at += wsum[w];
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!c[i]) continue;
                    *word(4 * b + i) = x;
                    x += c[i];
                    kp[x - 1].y = int32_t(c[i]);
                }
                __syncthreads();
            }
            // and, with the rows' payloads in place, its end
            each([&](int32_t k, int32_t p) {
                for (uint32_t b = home_of(k, nbk);; b = next_bucket(b, nbk)) {
                    const int at = slot_in(fresh(tab, b), k);
                    if (at < 0) continue;
                    kp[atomicAdd(word(4 * b + at), 1u)].x = p;
                    break;
                }
            });
            __syncthreads();
            for (uint32_t b = threadIdx.x; b < nbk; b += kBuildT) {
                const Slots q = fresh(tab, b);
                if (q.s[3] == kFree || ((passed[b >> 5] >> (b & 31)) & 1u) == (q.s[2] >= q.s[3])) continue;
                tab[4 * b + 2] = q.s[3];
                tab[4 * b + 3] = q.s[2];
            }
            __syncthreads();
            if (j == 0) {
                keys = tab;
                nbk1 = nbk;
            }
        }
    }
}

constexpr int kBT = 256;  // threads of the probe
constexpr int kU  = 2;    // rows per thread in flight

// Sums of the instance that a warp is at, added to its result when it comes to another.
struct Sums {
    unsigned long long rows = 0, sum = 0;
    uint32_t           cur  = ~0u;
    // every lane of the warp calls it
    __device__ __forceinline__ void at(uint32_t inst, InstOut* out) {
        if (inst == cur) return;
        if (cur != ~0u) {
            const unsigned long long tr = warp_sum(rows), ts = warp_sum(sum);
            if ((threadIdx.x & 31) == 0 && tr) {
                atomicAdd(&out[cur].rows, tr);
                atomicAdd(&out[cur].sum, ts);
            }
        }
        rows = sum = 0;
        cur        = inst;
    }
};

// 5. R0 rows against F.  kU rows a thread: keys and payloads of the next rows
// are on their way while the buckets of these are looked at.  Bound by its
// instructions and the L1's lines (about 155 a row of 32, 56% issue active, the
// L1 77% busy), not by where the table lies: 80M rows against a table of 1, 4, 16 or
// 64 MB 331, 337, 342, 361 us without a match, 477, 484, 482, 512 with one for half
// of the rows, 579, 586, 584, 595 with one each.  So the bucket reads allocate no
// L1 lines, two rows a thread fit 64 registers without spills, and what only some
// rows need is put off until a whole warp needs it: matches wait in the warp's queue
// until 32 of them are folded together, and rows that have to go on to a next bucket
// (one in twenty at half load, some in every warp) until 32 of them look together.  The instance's
// pieces are kept in shared memory (reads of them through L1 would cost as
// much as the buckets).  Each match of a key in F is a result row; listed keys are
// not in it.
constexpr uint32_t kQueue = 96;  // a step leaves at most 31 rows and adds at most 32 * kU
static_assert(31 + 32 * kU <= int(kQueue), "a step's rows fit the queues");
struct Queues {
    int4     hit[kQueue];  // key, payloads of R0 and R1, F slot
    int2     kp[kQueue];   // rows that go on, and the bucket they come from
    uint32_t b[kQueue];
};
__global__ void __launch_bounds__(kBT, 4)
    k_bt_probe(const Item* __restrict__ imap, uint64_t items, const uint64_t* __restrict__ tabs,
               const uint32_t* __restrict__ side, uint32_t stride, const Piece* __restrict__ pieces,
               InstOut* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem[];
    Piece* dir = reinterpret_cast<Piece*>(smem);  // the instance's pieces
    __shared__ __align__(16) Queues queues[kBT / 32];
    const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1;
    Queues&        Q    = queues[threadIdx.x >> 5];
    uint32_t       qn = 0, hn = 0;  // entries of the two (the same in every lane)
    Sums           acc;
    uint32_t       pb = 0, nt = 0;
    bool           skip = true;
    auto home = [&](int32_t k) {
        const Piece x = dir[part_of(k, pb)];
        return x.first + home_of(k, x.nbk);
    };
    // Matches folded into the sums, 32 at a time, until fewer than `keep` wait.
    auto fold = [&](uint32_t keep) {
        while (hn >= keep && hn) {
            __syncwarp();
            const uint32_t n = hn < 32 ? hn : 32;
            hn -= n;
            if (lane < n) {
                const int4 h  = Q.hit[hn + lane];
                uint64_t   fp = fp_add(fp_start(h.x, h.y), h.z);
                if (nt) {
                    const uint32_t* w = side + uint64_t(uint32_t(h.w)) * stride;
                    for (uint32_t j = 0; j < nt; ++j) fp = fp_add(fp, int32_t(__ldg(w + j)));
                }
                ++acc.rows;
                acc.sum += fp_final(fp);
            }
            __syncwarp();
        }
    };
    // Key k in its loaded bucket: its matches and the row itself to the queues.
    auto look = [&](bool on, int32_t k, int32_t p, uint32_t b, const Slots& q) {
        uint32_t m = 0;
        if (slot_key(q.s[0]) == k) m = 1;
        if (slot_key(q.s[1]) == k) m |= 2;
        if (slot_key(q.s[2]) == k) m |= 4;
        if (slot_key(q.s[3]) == k) m |= 8;
        if (k == slot_key(kFree)) {  // a free slot is no match
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (q.s[i] == kFree) m &= ~(1u << i);
        }
        if (!on) m = 0;
        for (unsigned bal; (bal = __ballot_sync(0xffffffffu, m != 0)) != 0;) {  // once, unless a key has several rows
            if (m) {
                const int32_t p1 = (m & 1) ? slot_pay(q.s[0]) : (m & 2) ? slot_pay(q.s[1]) : (m & 4) ? slot_pay(q.s[2])
                                                                                              : slot_pay(q.s[3]);
                Q.hit[hn + __popc(bal & lt)] = make_int4(k, p, p1, int32_t(b * 4 + __ffs(m) - 1));
                m &= m - 1;
            }
            hn += __popc(bal);
            if (hn > kQueue - 32) fold(32);
        }
        const bool     on2 = on && goes_on(q);
        const unsigned bal = __ballot_sync(0xffffffffu, on2);
        if (on2) {
            const uint32_t at = qn + __popc(bal & lt);
            Q.kp[at]          = make_int2(k, p);
            Q.b[at]           = b;
        }
        qn += __popc(bal);
    };
    // The rows that go on, at their next buckets, until fewer than `keep` wait.
    auto go_on = [&](uint32_t keep) {
        while (qn >= keep && qn) {
            __syncwarp();
            const uint32_t n  = qn < 32 ? qn : 32;
            const bool     on = lane < n;
            qn -= n;
            int2           kp = make_int2(0, 0);
            uint32_t       b  = 0;
            if (on) {
                kp            = Q.kp[qn + lane];
                b             = Q.b[qn + lane] + 1;
                const Piece x = dir[part_of(kp.x, pb)];
                if (b == x.first + x.nbk) b = x.first;
            }
            const Slots q = load_bucket(tabs, b);
            __syncwarp();
            look(on, kp.x, kp.y, b, q);
            fold(32);
        }
    };
    for (uint64_t t = blockIdx.x; t < items; t += gridDim.x) {
        const Item it = imap[t];
        if (it.inst != acc.cur) {
            go_on(0);
            fold(0);
            acc.at(it.inst, out);
            skip = out[it.inst].ovf;
            pb   = it.pbits;
            nt   = it.nt;
            __syncthreads();
            for (uint32_t x = threadIdx.x; x < (1u << pb); x += kBT) dir[x] = pieces[it.part_base + x];
            __syncthreads();
        }
        if (skip) continue;
        const int32_t *kk = it.k + threadIdx.x, *pp = it.p + threadIdx.x;
        int            left = int(it.n) - int(threadIdx.x);  // rows from this thread's next one on
        int32_t        nk[kU], np[kU];
        auto           fetch = [&]() {
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                nk[u] = np[u] = 0;
                if (left > u * kBT) {
                    nk[u] = __ldcs(kk + u * kBT);
                    np[u] = __ldcs(pp + u * kBT);
                }
            }
            kk += kU * kBT;
            pp += kU * kBT;
        };
        fetch();
        for (int steps = int((it.n + kU * kBT - 1) / (kU * kBT)); steps > 0; --steps) {
            int32_t  k[kU], p[kU];
            uint32_t b[kU];
            bool     on[kU];
            Slots    q[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                k[u]  = nk[u];
                p[u]  = np[u];
                on[u] = left > u * kBT;
                b[u]  = home(k[u]);
                q[u]  = load_bucket(tabs, b[u]);
            }
            left -= kU * kBT;
            fetch();
#pragma unroll
            for (int u = 0; u < kU; ++u) look(on[u], k[u], p[u], b[u], q[u]);
            go_on(32);
            fold(32);
        }
    }
    go_on(0);
    fold(0);
    acc.at(~0u, out);
}

// 6. The rows whose key is listed.  Their keys are looked for in the filter, kEU a
// lane in flight and the next ones on their way; those that it holds wait in the
// warp's queue until 32 of them are looked up in every relation, a lane each.  A
// row's results are the combinations of one payload a list.  The warp shares out those
// of its rows together: of a row with kMany of them by themselves, else by a
// search of the running sums.
// Bound by the scan of R0's keys where few are listed (500e9 rows/s, 57% issue
// active), so what a listed row needs is kept out of its registers (within them
// 360e9).  Results by the rows' own lanes instead: 64 chains of 16,000 rows, 16 a
// key, half of R0's rows with a partner 1,836 us, so 1,080.
constexpr int      kEU     = 8;
constexpr uint32_t kMany   = 64;
constexpr uint32_t kMaxTab = kMaxRel - 1;
struct EnumRows {
    int2     queue[32 * (kEU + 1)];  // key and row; a step leaves at most 31 and adds 32 * kEU
    uint64_t fp[32];                 // of the 32 rows: key and R0's payload folded
    uint32_t before[32];             // results of the rows before
    uint32_t start[kMaxTab][32], len[kMaxTab][32];
};
// What the rows of an instance are looked up in.
struct EnumOf {
    const uint64_t* tabs;
    const int2*     kp;
    const Piece*    listed;  // of R1's partition 0
    const int32_t*  pay;     // R0's payloads; the queue's rows count from here
    uint32_t        pb, nt;
};
// The results of the queue's n rows from q on.  (Not inlined: its registers would
// be the scan's.)
__device__ __noinline__ void enum_rows(EnumRows& W, const EnumOf& I, uint32_t q, uint32_t n, Sums& acc) {
    const unsigned lane = threadIdx.x & 31;
    const uint32_t nt   = I.nt;
    const int2*    kp   = I.kp;
    uint64_t       total = 0, sum = 0;
    uint32_t       done = 0;
    // a result: row r's combination c
    auto result = [&](uint32_t r, auto c) {
        uint32_t at[kMaxTab];
#pragma unroll
        for (int j = kMaxTab - 1; j > 0; --j) {
            if (j > int(nt)) continue;
            const uint32_t l = W.len[j][r];
            const auto     d = c / l;
            at[j] = uint32_t(c - d * l);
            c     = d;
        }
        at[0]       = uint32_t(c);
        uint64_t fp = W.fp[r];
#pragma unroll
        for (int j = 0; j < int(kMaxTab); ++j)
            if (j <= int(nt)) fp = fp_add(fp, __ldg(&kp[W.start[j][r] + at[j]].x));
        ++done;
        sum += fp_final(fp);
    };
    __syncwarp();
    if (lane < n) {
        const int2    r    = W.queue[q + lane];
        const int32_t p    = __ldcs(I.pay + uint32_t(r.y));
        const Piece*  part = I.listed + part_of(r.x, I.pb);
        total              = 1;
        for (uint32_t j = 0; j <= nt && total; ++j) {
            const Piece x   = part[uint64_t(j) << I.pb];
            uint32_t    end = 0, len = 0;
            for (uint32_t b = home_of(r.x, x.nbk);; b = next_bucket(b, x.nbk)) {
                const Slots s = load_bucket(I.tabs, uint64_t(x.first) + b);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (s.s[i] != kFree && slot_key(s.s[i]) == r.x) end = uint32_t(slot_pay(s.s[i]));
                if (end || !goes_on(s)) break;
            }
            if (end) len = uint32_t(__ldg(&kp[end - 1].y));
            W.start[j][lane] = end - len;
            W.len[j][lane]   = len;
            total *= len;
        }
        W.fp[lane] = fp_start(r.x, p);
    }
    const uint32_t few = total < kMany ? uint32_t(total) : 0u;
    const uint32_t inc = warp_inclusive_scan(few), all = __shfl_sync(0xffffffffu, inc, 31);
    W.before[lane]     = inc - few;
    __syncwarp();
    for (uint32_t i = lane; i < all; i += 32) {
        uint32_t r = 0;  // the last row with at most i results before it (one without results shares the next one's number)
#pragma unroll
        for (uint32_t d = 16; d; d >>= 1)
            if (W.before[r + d] <= i) r += d;
        result(r, i - W.before[r]);
    }
    for (unsigned big = __ballot_sync(0xffffffffu, total >= kMany); big; big &= big - 1) {
        const int      r = __ffs(big) - 1;
        const uint64_t t = __shfl_sync(0xffffffffu, total, r);
        if (nt == 0) {
            const uint64_t fp = W.fp[r];
            const int2*    l  = kp + W.start[0][r];
            for (uint32_t c = lane; c < t; c += 32, ++done) sum += fp_final(fp_add(fp, __ldg(&l[c].x)));
        } else if (t <= 0xffffffe0ull) {
            for (uint32_t c = lane; c < t; c += 32) result(uint32_t(r), c);
        } else {
            for (uint64_t c = lane; c < t; c += 32) result(uint32_t(r), c);
        }
    }
    acc.rows += done;
    acc.sum += sum;
    __syncwarp();
}

constexpr size_t kEnumSmem = sizeof(EnumRows) * (kBT / 32) + (size_t(1) << kFilterAll) / 8;
__global__ void __launch_bounds__(kBT, 3)
    k_bt_enum(const Item* __restrict__ imap, uint64_t items, const uint64_t* __restrict__ tabs,
              const int2* __restrict__ kp, const Piece* __restrict__ listed, const uint32_t* __restrict__ filters,
              const uint32_t* __restrict__ any, InstOut* __restrict__ out) {
    if (!*any) return;
    extern __shared__ __align__(16) unsigned char smem[];
    EnumRows&      W      = reinterpret_cast<EnumRows*>(smem)[threadIdx.x >> 5];
    uint32_t*      filter = reinterpret_cast<uint32_t*>(smem + sizeof(EnumRows) * (kBT / 32));  // the instance's
    const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1;
    uint32_t       qn   = 0, pb = 0, flog = 0;
    EnumOf         I{tabs, kp, listed, nullptr, 0, 0};
    Sums           acc;
    for (uint64_t t = blockIdx.x; t < items; t += gridDim.x) {
        const Item it = imap[t];
        if (out[it.inst].ovf || !out[it.inst].lists) continue;
        if (it.inst != acc.cur) {
            if (qn) enum_rows(W, I, 0, qn, acc);
            qn = 0;
            acc.at(it.inst, out);
            pb   = it.pbits;
            flog = it.flog;
            I    = EnumOf{tabs, kp, listed + it.part_base, it.p, pb, it.nt};
            __syncthreads();
            const uint32_t words = 1u << (pb + flog - 5);
            for (uint32_t w0 = threadIdx.x; w0 < words; w0 += 8 * kBT) {
                uint32_t v[8], on[8];
#pragma unroll
                for (uint32_t u = 0; u < 8; ++u) {  // (words of a partition without listed keys hold anything)
                    const uint32_t w = min(w0 + u * kBT, words - 1);
                    v[u]             = __ldg(filters + it.fbase + w);
                    on[u]            = __ldg(&I.listed[w >> (flog - 5)].nbk);
                }
#pragma unroll
                for (uint32_t u = 0; u < 8; ++u)
                    if (w0 + u * kBT < words) filter[w0 + u * kBT] = on[u] ? v[u] : 0u;
            }
            __syncthreads();
        }
        const uint32_t row = uint32_t(it.p - I.pay);
        int32_t        nk[kEU];
        uint32_t       x0    = threadIdx.x;
        auto           fetch = [&]() {
#pragma unroll
            for (int u = 0; u < kEU; ++u) nk[u] = x0 + u * kBT < it.n ? __ldcs(it.k + x0 + u * kBT) : 0;
        };
        fetch();
        while (x0 - lane < it.n) {
            int32_t        k[kEU];
            const uint32_t at = x0;
            uint32_t       on = 0;
#pragma unroll
            for (int u = 0; u < kEU; ++u) {
                k[u]             = nk[u];
                uint32_t       w;
                const uint32_t m = filter_bits(k[u], flog, w);
                const uint32_t f = filter[(part_of(k[u], pb) << (flog - 5)) + w];
                on |= uint32_t(x0 + u * kBT < it.n && (f & m) == m) << u;
            }
            x0 += kBT * kEU;
            fetch();
            if (!__any_sync(0xffffffffu, on != 0)) continue;
#pragma unroll
            for (int u = 0; u < kEU; ++u) {
                const unsigned bal = __ballot_sync(0xffffffffu, (on >> u) & 1u);
                if ((on >> u) & 1u) W.queue[qn + __popc(bal & lt)] = make_int2(k[u], int32_t(row + at + u * kBT));
                qn += __popc(bal);
            }
            while (qn >= 32) {
                qn -= 32;
                enum_rows(W, I, qn, 32, acc);
            }
        }
    }
    if (qn) enum_rows(W, I, 0, qn, acc);
    acc.at(~0u, out);
}

// ---- plain path helper --------------------------------------------------------
// (probe row, build row) pairs -> next (key, fold state) rows, or (okey null)
// the checksum of a last join.
__global__ void k_pairs_next(const uint32_t* __restrict__ prow, const uint32_t* __restrict__ brow, uint64_t n,
                             const int32_t* __restrict__ pkeys, const uint64_t* __restrict__ pfp,
                             const int32_t* __restrict__ ppay, const int32_t* __restrict__ bpay,
                             int32_t* __restrict__ okey, uint64_t* __restrict__ ofp, unsigned long long* __restrict__ sum) {
    unsigned long long acc    = 0;
    const uint64_t     stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint32_t p  = prow[i];
        const int32_t  k  = pkeys[p];
        const uint64_t fp = pfp ? pfp[p] : fp_start(k, ppay[p]);
        const uint64_t nf = fp_add(fp, bpay[brow[i]]);
        if (okey) {
            okey[i] = k;
            ofp[i]  = nf;
        } else {
            acc += fp_final(nf);
        }
    }
    if (!okey) {
        acc = warp_sum(acc);
        if ((threadIdx.x & 31) == 0 && acc) atomicAdd(sum, acc);
    }
}

uint32_t ceil_log2u(uint64_t x) {
    uint32_t b = 0;
    while (b < 63 && (1ull << b) < x) ++b;
    return b;
}

// Blocks of `kernel` that fit on the GPU at once with `smem` dynamic shared
// memory (the grid of a persistent launch); raises the kernel's dynamic
// shared-memory limit first.  Not capturable: called before a capture.
template <class K>
int resident_grid(K kernel, int threads, size_t smem) {
    HJ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    int per_sm = 0;
    HJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
    if (per_sm < 1) throw Error(HJ_ERR_INVALID, "batch: a kernel does not fit on an SM");
    return per_sm * num_sms();
}

}  // namespace

void launch_batch_generate(uint64_t seed, uint32_t instance, uint32_t relation, uint64_t build_rows,
                           uint32_t match_q24, uint64_t rows, int32_t* keys, int32_t* payload, cudaStream_t st) {
    if (build_rows == 0 || build_rows > (1ull << 30))
        throw Error(HJ_ERR_INVALID, "batch_generate: build rows must be in [1, 2^30]");
    if (relation > 0 && rows > build_rows)
        throw Error(HJ_ERR_INVALID, "batch_generate: a build relation has at most build_rows rows");
    if (match_q24 > (1u << 24)) throw Error(HJ_ERR_INVALID, "batch_generate: match rate above 2^24");
    if (rows == 0) return;
    if (!keys || !payload) throw Error(HJ_ERR_INVALID, "batch_generate: null output");
    const unsigned blocks = unsigned(std::min<uint64_t>(div_up(rows, 256), uint64_t(num_sms()) * 16));
    k_batch_generate<<<blocks, 256, 0, st>>>(seed, instance, relation, build_rows, match_q24, rows, keys, payload);
    HJ_LAUNCH_CHECK();
}

void BatchGraph::clear() {
    if (exec) cudaGraphExecDestroy(exec);
    exec = nullptr;
}

namespace {

// What the options give for partitions of ~T build rows (all build relations
// together): tables of up to 2T rows in shared memory, bucket bounds for
// 2^max_bits buckets; and in HBM the same load, kept where linear probing stays
// short, with a counter per bucket of a piece (a piece of `cap` rows always
// fits its counters).
struct Geometry {
    uint64_t T;
    uint32_t cap, max_bits, scap, load_q8, fcap;
    uint32_t slot_q16;  // buckets per row, in 65536ths
    size_t   build_smem;
};

Geometry geometry(const BatchOptions& o) {
    Geometry g;
    g.T        = 1ull << o.part_rows_log2;
    g.cap      = uint32_t(2 * g.T);
    g.max_bits = std::max<uint32_t>(1, ceil_log2u(uint64_t(std::ceil(double(g.T) / o.load))));
    g.scap     = (1u << g.max_bits) + 2 * kMaxRel;
    g.load_q8  = std::max<uint32_t>(1, uint32_t(std::lround(o.load * 256.0)));
    const size_t tables = size_t(g.cap) * 8 + size_t(g.scap) * 4;
    if (tables > 200 * 1024) throw Error(HJ_ERR_INVALID, "batch: partition tables exceed shared memory");
    g.slot_q16 = batch_buckets_q16(o.load);
    g.fcap     = uint32_t(std::min<uint64_t>(batch_piece_buckets(g.cap, g.slot_q16), (220 * 1024 - tables) / 2));
    g.build_smem = tables + size_t(g.fcap) * 2 + 4 + (1u << kFilterPart) / 8;
    return g;
}

// Build rows of an instance, all build relations together; 0 when any relation has none (no result rows).
uint64_t build_rows_of(const BatchInstance& b) {
    uint64_t nb = 0;
    for (size_t j = 0; j < b.rels.size(); ++j) {
        if (!b.rels[j].rows) return 0;
        if (j) nb += b.rels[j].rows;
    }
    return nb;
}

// Instances [i0, i1) of the batch; the ones in `idle` (without result rows, or
// left to the plain path) as if without rows.
void batch_wave(const std::vector<BatchInstance>& all, uint32_t i0, uint32_t i1, const std::vector<uint8_t>& idle,
                const BatchOptions& o, const Geometry& G, BatchGraph& graph, uint64_t* rows, uint64_t* sums,
                std::vector<uint32_t>& bad, cudaStream_t st) {
    const uint32_t n = i1 - i0;
    auto           rel_of = [&](uint32_t i, uint32_t j) {
        BatchRelation r = all[i0 + i].rels[j];
        if (idle[i0 + i]) r.rows = 0;
        return r;
    };
    const uint64_t T   = G.T;
    const uint32_t cap = G.cap, scap = G.scap, fcap = G.fcap, max_bits = G.max_bits, load_q8 = G.load_q8;
    const size_t   build_smem = G.build_smem;
    std::vector<RelInst>  hr;
    std::vector<InstInfo> hi(n);
    uint64_t pbase = 0, ipbase = 0, items = 0, build_rows = 0, fwords = 0;
    uint32_t pmax = 0, stride = 0;
    for (uint32_t i = 0; i < n; ++i) {
        const uint32_t nrel = uint32_t(all[i0 + i].rels.size());
        uint64_t       nb   = 0;
        for (uint32_t j = 1; j < nrel; ++j) nb += rel_of(i, j).rows;
        const uint32_t p = nb > T ? std::min(kMaxPartBits, ceil_log2u((nb + T - 1) / T)) : 0;
        InstInfo&      s = hi[i];
        pmax             = std::max(pmax, p);
        s.part_base      = pbase;
        s.ip_base        = ipbase;
        s.nrel           = nrel;
        s.pbits          = p;
        s.fbase          = uint32_t(fwords);
        s.flog           = std::min({kFilterPart, kFilterAll - p, std::max(5u, ceil_log2u(8 * std::max<uint64_t>(nb, 1)))});
        fwords += 1ull << (p + s.flog - 5);
        stride           = std::max(stride, s.nrel - 2);
        for (uint32_t j = 1; j < s.nrel; ++j) {
            const BatchRelation br = rel_of(i, j);
            hr.push_back({br.keys, br.payload, br.rows, items, pbase + (uint64_t(j - 1) << p), p, i, 0, 0, 0});
            items += (br.rows + kPartItem - 1) / kPartItem;
        }
        build_rows += nb;
        pbase += uint64_t(s.nrel - 1) << p;
        ipbase += 1ull << p;
    }
    // persistent grids (occupancy queries are not capturable: take them first)
    const size_t hist_smem = (size_t(1) << pmax) * 4;
    const size_t scat_smem = size_t(kPartItem) * 10 + (size_t(1) << pmax) * 16;
    const size_t prb_smem  = (size_t(1) << pmax) * sizeof(Piece);
    const int    g_hist    = resident_grid(k_bpart_hist, kPT, hist_smem);
    const int    g_scat    = resident_grid(k_bpart_scatter, kPT, scat_smem);
    const int    g_bld     = resident_grid(k_bt_build, kBuildT, build_smem);
    const int    g_prb     = resident_grid(k_bt_probe, kBT, prb_smem);
    const int    g_enm     = resident_grid(k_bt_enum, kBT, kEnumSmem);
    auto grid_for = [](int g, uint64_t work) { return unsigned(std::max<uint64_t>(1, std::min<uint64_t>(g, work))); };

    // R0s: an item is what one block has of its instance's rows when the grid
    // shares them twice over, so that blocks stay with an instance, within
    // 16 .. 64 steps of a block
    const uint64_t bitems = items;  // items of the build relations, then of the R0s
    constexpr uint64_t kStepRows = uint64_t(kBT) * kU;
    for (uint32_t i = 0; i < n; ++i) {
        const BatchRelation  br    = rel_of(i, 0);
        const uint64_t       steps = br.rows / (2 * uint64_t(g_prb) * kStepRows);
        const uint64_t       irows = std::min<uint64_t>(std::max<uint64_t>(steps, 16), 64) * kStepRows;
        hr.push_back({br.keys, br.payload, br.rows, items, hi[i].part_base, hi[i].pbits, i, uint32_t(irows), hi[i].nrel,
                      hi[i].fbase, hi[i].flog});
        items += (br.rows + irows - 1) / irows;
    }
    const uint32_t nr   = uint32_t(hr.size());
    const uint64_t nbkt = batch_table_buckets(build_rows, pbase + ipbase, G.slot_q16);

    std::vector<InstOut> ho(n);
    std::vector<void*>   owned;
    struct Release {
        std::vector<void*>& v;
        cudaStream_t        st;
        ~Release() {
            // the host arrays above are read and written by copies on the stream
            if (std::uncaught_exceptions()) cudaStreamSynchronize(st);
            for (void* p : v) dfree(p, st);
        }
    } release{owned, st};
    auto take = [&](size_t bytes) {
        void* p = dalloc(bytes + 16, st);
        owned.push_back(p);
        return p;
    };
    // results, counters and queues, cleared by one fill
    const size_t zero_bytes = n * sizeof(InstOut) + 4 * 8 + 2 * (pbase + 1) * 4;
    auto*        d_out      = static_cast<InstOut*>(take(zero_bytes));
    auto*        d_q        = reinterpret_cast<unsigned long long*>(d_out + n);
    auto*        cnt        = reinterpret_cast<uint32_t*>(d_q + 4);
    auto*        fill       = cnt + pbase + 1;
    // relations and instances, copied together
    std::vector<uint8_t> hd(nr * sizeof(RelInst) + n * sizeof(InstInfo));
    std::memcpy(hd.data(), hr.data(), nr * sizeof(RelInst));
    std::memcpy(hd.data() + nr * sizeof(RelInst), hi.data(), n * sizeof(InstInfo));
    auto* d_R    = static_cast<RelInst*>(take(hd.size()));
    auto* d_I    = reinterpret_cast<InstInfo*>(d_R + nr);
    auto* off    = static_cast<uint64_t*>(take((pbase + 2) * 8));
    auto* pieces = static_cast<Piece*>(take((pbase + 1) * sizeof(Piece)));
    auto* listed = static_cast<Piece*>(take((pbase + 1) * sizeof(Piece)));
    auto* filters = static_cast<uint32_t*>(take(fwords * 4));
    auto* tmp    = static_cast<uint64_t*>(take((scan_tmp_words(pbase) + 1) * 8));
    auto* pkp    = static_cast<int2*>(take(build_rows * 8));  // (key, payload) in partition order
    auto* rmap   = static_cast<uint32_t*>(take(bitems * 4));
    auto* imap   = static_cast<Item*>(take((items - bitems) * sizeof(Item)));
    auto* pmap   = static_cast<uint32_t*>(take(ipbase * 4));
    auto* tabs   = static_cast<uint64_t*>(take(nbkt * 32));
    auto* side   = static_cast<uint32_t*>(take(nbkt * 4 * stride * 4));
    HJ_CUDA(cudaMemcpyAsync(d_R, hd.data(), hd.size(), cudaMemcpyHostToDevice, st));

    Tables tb{tabs, side, reinterpret_cast<uint32_t*>(d_q + 2), reinterpret_cast<uint32_t*>(d_q + 3),
              uint32_t(nbkt), stride, G.slot_q16};

    auto enqueue = [&]() {
        HJ_CUDA(cudaMemsetAsync(d_out, 0, zero_bytes, st));
        if (!build_rows || items == bitems) return;  // no result rows
        k_item_rel<<<unsigned(std::min<uint64_t>(div_up(items + ipbase, 256), uint64_t(num_sms()) * 8)), 256, 0, st>>>(
            d_R, nr, bitems, items, rmap, imap, d_I, n, ipbase, pmap, tb);
        HJ_LAUNCH_CHECK();
        k_bpart_hist<<<grid_for(g_hist, bitems), kPT, hist_smem, st>>>(d_R, rmap, bitems, cnt);
        HJ_LAUNCH_CHECK();
        scan_exclusive_u32_to_u64_into(cnt, off, pbase, tmp, st);
        k_bpart_scatter<<<grid_for(g_scat, bitems), kPT, scat_smem, st>>>(d_R, rmap, bitems, d_q + 1, off, fill, pmax,
                                                                          pkp);
        HJ_LAUNCH_CHECK();
        k_bt_build<<<grid_for(g_bld, ipbase), kBuildT, build_smem, st>>>(d_I, pmap, ipbase, off, pkp, cap, scap, fcap,
                                                                         max_bits, load_q8, tb, pieces, listed, filters, d_out);
        HJ_LAUNCH_CHECK();
        k_bt_probe<<<grid_for(g_prb, items - bitems), kBT, prb_smem, st>>>(imap, items - bitems, tabs, side, stride,
                                                                           pieces, d_out);
        HJ_LAUNCH_CHECK();
        k_bt_enum<<<grid_for(g_enm, items - bitems), kBT, kEnumSmem, st>>>(imap, items - bitems, tabs, pkp, listed, filters,
                                                                           tb.lists, d_out);
        HJ_LAUNCH_CHECK();
    };
    if (o.graph) {
        cudaGraph_t g = nullptr;
        HJ_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        try {
            enqueue();
        } catch (...) {
            cudaStreamEndCapture(st, &g);
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            throw;
        }
        HJ_CUDA(cudaStreamEndCapture(st, &g));
        // the last call's executable graph takes this call's parameters when
        // its kernels are the same (10 us), else it is made anew (60 us)
        cudaError_t e = cudaSuccess;
        if (graph.exec) {
            cudaGraphExecUpdateResultInfo info;
            if (cudaGraphExecUpdate(graph.exec, g, &info) != cudaSuccess) {
                cudaGetLastError();
                graph.clear();
            }
        }
        if (!graph.exec) e = cudaGraphInstantiate(&graph.exec, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            graph.exec = nullptr;
            throw Error(HJ_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
        }
        HJ_CUDA(cudaGraphLaunch(graph.exec, st));
    } else {
        enqueue();
    }
    readback(ho.data(), d_out, n * sizeof(InstOut), o.host_write, st);
    HJ_CUDA(cudaStreamSynchronize(st));
    for (uint32_t i = 0; i < n; ++i) {
        rows[i0 + i] = ho[i].rows;
        sums[i0 + i] = ho[i].sum;
        if (ho[i].ovf) bad.push_back(i0 + i);
    }
}

}  // namespace

std::vector<uint32_t> batch_execute(const std::vector<BatchInstance>& B, const BatchOptions& o, BatchGraph& graph,
                                    std::vector<uint64_t>& rows, std::vector<uint64_t>& sums, cudaStream_t st) {
    const uint32_t n = uint32_t(B.size());
    rows.assign(n, 0);
    sums.assign(n, 0);
    if (n == 0) return {};
    if (!(o.load > 0.0 && o.load <= 8.0)) throw Error(HJ_ERR_INVALID, "batch: directory load out of range");
    if (o.part_rows_log2 < 8 || o.part_rows_log2 > 13)
        throw Error(HJ_ERR_INVALID, "batch: partition size must be 2^8 .. 2^13 build rows");
    for (const auto& b : B) {
        if (b.rels.size() < 2 || b.rels.size() > kMaxRel)
            throw Error(HJ_ERR_INVALID, "a batch instance needs 2 to 8 relations");
        for (const auto& r : b.rels) {
            if (r.rows > 0xffffffffull) throw Error(HJ_ERR_INVALID, "a batch relation has more than 2^32-1 rows");
            if (r.rows && (!r.keys || !r.payload)) throw Error(HJ_ERR_INVALID, "a batch relation lacks its columns");
        }
    }
    const Geometry        G = geometry(o);
    std::vector<uint8_t>  idle(n, 0);
    std::vector<uint32_t> bad;
    // Waves of instances whose tables stay within kWaveBytes, so that a large
    // batch takes no more memory than the inputs' own size and a slot's number
    // fits 32 bits.  An instance with more build rows than its partitions can
    // hold goes to the plain path at once; one with an empty relation has no
    // result rows, and its other relations take no memory.
    constexpr uint64_t kWaveBytes = 24ull << 30;
    for (uint32_t i0 = 0; i0 < n;) {
        uint64_t bytes = 0;
        uint32_t i1    = i0;
        for (; i1 < n; ++i1) {
            const uint64_t nb = build_rows_of(B[i1]);
            if (nb > (uint64_t(G.cap) << kMaxPartBits)) {
                bad.push_back(i1);
                idle[i1] = 1;
                continue;
            }
            idle[i1] = nb == 0;
            const uint64_t need = uint64_t(double(nb) * (G.slot_q16 / 65536.0 * (32 + 16 * (kMaxRel - 2)) + 8));
            if (i1 > i0 && bytes + need > kWaveBytes) break;
            bytes += need;
        }
        batch_wave(B, i0, i1, idle, o, G, graph, rows.data(), sums.data(), bad, st);
        i0 = i1;
    }
    return bad;
}

void plain_instance(const BatchInstance& b, const ProbeParams& prm, int dir_bits, int radix_bits, int dir_cap_bits,
                    uint64_t& rows, uint64_t& sum, cudaStream_t st) {
    rows = sum = 0;
    if (b.rels.size() < 2) throw Error(HJ_ERR_INVALID, "a batch instance needs at least two relations");
    std::vector<void*> owned;
    struct Release {
        std::vector<void*>& v;
        cudaStream_t        st;
        ~Release() {
            for (void* p : v) dfree(p, st);
        }
    } release{owned, st};
    auto take = [&](size_t bytes) {
        void* p = dalloc(bytes + 16, st);
        owned.push_back(p);
        return p;
    };
    auto*           d_sum = static_cast<unsigned long long*>(take(8));
    const int32_t*  pkeys = b.rels[0].keys;
    const int32_t*  ppay  = b.rels[0].payload;
    const uint64_t* pfp   = nullptr;
    uint64_t        np    = b.rels[0].rows;
    HJ_CUDA(cudaMemsetAsync(d_sum, 0, 8, st));
    for (size_t sg = 1; sg < b.rels.size() && np > 0; ++sg) {
        const BatchRelation& br   = b.rels[sg];
        const bool           last = sg + 1 == b.rels.size();
        if (br.rows == 0) break;
        IntCol bc;
        bc.plain = br.keys;
        IntCol pc;
        pc.plain = pkeys;
        const KeyCol pk{pc, nullptr, np};
        Table        t;
        build_table(KeyCol{bc, nullptr, br.rows}, dir_bits, radix_bits, t, prm.pinned, st, int64_t(br.rows),
                    dir_cap_bits);
        ProbePlan* pp    = nullptr;
        uint64_t   total = 0;
        RidOut     ro[2] = {{0, nullptr, nullptr}, {1, nullptr, nullptr}};
        try {
            // streams for one match a row, made before the count; others for more,
            // and where there is no room for them
            auto count = [&](bool ahead) {
                for (RidOut& o : ro) o.dst = ahead ? static_cast<uint32_t*>(take(np * 4)) : nullptr;
                total = probe_count(t, pk, prm, ro, ahead ? 2 : 0, &pp, st);
                if (ahead && total <= np) return;
                for (RidOut& o : ro) {
                    uint32_t* sized = static_cast<uint32_t*>(take(total * 4));
                    if (const uint64_t d = probe_direct(pp))
                        HJ_CUDA(cudaMemcpyAsync(sized, o.dst, d * 4, cudaMemcpyDeviceToDevice, st));
                    o.dst = sized;
                }
            };
            const size_t before = owned.size();
            try {
                count(true);
            } catch (const Error& e) {
                if (e.status != HJ_ERR_NOMEM) throw;
                probe_free(pp, st);
                pp = nullptr;
                for (; owned.size() > before; owned.pop_back()) dfree(owned.back(), st);
                count(false);
            }
            if (total) probe_write(t, pk, pp, ro, 2, st);
        } catch (...) {
            if (pp) probe_free(pp, st);
            free_table(t, st);
            throw;
        }
        probe_free(pp, st);
        free_table(t, st);
        int32_t*  nk = last ? nullptr : static_cast<int32_t*>(take(total * 4));
        uint64_t* nf = last ? nullptr : static_cast<uint64_t*>(take(total * 8));
        if (total) {
            k_pairs_next<<<unsigned(std::min<uint64_t>(div_up(total, 256), uint64_t(num_sms()) * 8)), 256, 0, st>>>(
                ro[0].dst, ro[1].dst, total, pkeys, pfp, ppay, br.payload, nk, nf, d_sum);
            HJ_LAUNCH_CHECK();
        }
        pkeys = nk;
        pfp   = nf;
        ppay  = nullptr;
        np    = total;
        if (last) rows = total;
    }
    readback(prm.pinned, d_sum, 8, true, st);  // page-locked scratch
    HJ_CUDA(cudaStreamSynchronize(st));
    sum = prm.pinned[0];
}

}  // namespace hj
