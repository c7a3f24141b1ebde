// Probe of the unchained table on the GPU.
//
// Semantics of UnchainedHash::probe (include/unchained.h:220-246 of the
// reference) applied to a column of probe keys, as the reference's probe
// workers do (src/execute.cpp:111-165): NULL keys never match (:127-129),
// Bloom early-reject on the bucket's tag, then every tuple of the bucket with
// an equal key is a match.
//
// Count pass, k_probe_tile for one tile of 1984 probe rows (one dense INT32
// page), whose matches keep their order, and k_probe_stream for more.  Per key
// the probe issues ONE global load, the bucket's 8-byte summary (first key, and
// the tuple's build row or Bloom tag, length and mixed flag; hj_common.cuh):
//   miss     empty bucket, or the Bloom tag rejects the key;
//   single   bucket of one tuple: its key decides, its build row is there;
//   uniform  bucket of one key (mixed flag clear): the key matches every tuple
//            of the bucket or none, decided by the first key; the hit is
//            (probe row, bucket, length from the summary) -- no further load;
//   mixed    bucket of several keys: the tuples of a bucket of at most
//            min(light_max, 31) are compared and the matching ones noted as a
//            mask over the bucket (one match: as its build row); larger buckets
//            go to a list counted by a warp or block per hit (k_mixed_count*).
// A match that is the only one of its probe row is written at once, its row
// ids straight to the output.  Other hits go to a list with their first output
// rows: ONE global 64-bit atomic a flush reserves both list slots (high word)
// and output rows (low word), so list order and output order agree and no
// device-wide prefix sum is needed (the reference's per-thread work-stealing
// counter becomes this reservation).  The listed matches follow the direct ones.
//
// Write pass.  k_write_uniform walks the OUTPUT positions in chunks of
// 32 x G per warp (G outputs per thread, option probe_group): a chunk's hits
// are located by the chunk map (k_chunk_first) and staged in the warp's own
// shared memory, a uniform hit's bucket start is read from its directory
// word, each thread finds its hit by binary search and reads build rows
// rows[start + k] consecutively, and writes its G row ids of every output
// stream as one 16-byte store (a warp covers 512 contiguous bytes).  Warps
// synchronise only with themselves.  Work is balanced by output rows, so one
// Zipf-heavy key with millions of tuples spreads over all SMs.
// Mixed hits follow the uniform ones.  Every match writes one row id per
// requested output stream, composed through the sides' row-id vectors (late
// materialisation).
#include <algorithm>
#include <type_traits>

#include "hj_block.cuh"
#include "hj_common.cuh"
#include "hj_kernels.h"

namespace hj {

namespace {

constexpr int      kPT        = 256;                    // threads of the stream kernel
constexpr uint32_t kTileRows  = uint32_t(kDenseRows);   // 1984 rows per tile (one page)
constexpr uint32_t kUncounted = 0xffffffffu;            // mixed hit still to be counted
constexpr uint32_t kMixedWarpMax = 4096;                // mixed buckets up to this size: one warp each

// L2 cache policy (createpolicy) for stores of lines written once and read
// back later in order (output row ids): they leave L2 first.
__device__ __forceinline__ uint64_t l2_evict_first() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// 16-byte stores with an L2 cache policy.
__device__ __forceinline__ void st_hint(uint4* p, uint4 v, uint64_t policy) {
    asm volatile("st.global.L2::cache_hint.v4.u32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z),
                 "r"(v.w), "l"(policy)
                 : "memory");
}
__host__ __device__ __forceinline__ uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }

enum KeySrc : int { kSrcPages = 0, kSrcPlain = 1, kSrcTagged = 2, kSrcGather = 3 };

struct ProbeTab {
    const uint64_t* dir;
    const uint64_t* sum;
    const int32_t*  keys;
    const uint32_t* rows;
    uint32_t        nb;  // buckets, a power of two
};

struct Lists {
    // staged hits, in output order: hit h owns output rows [off[h], off[h + 1])
    // (the last up to the staged total); mask 0: the whole bucket sp matches,
    // kRowHit: build row sp, else the tuples sp + i for the set bits i of mask
    uint32_t *u_row, *u_sp, *u_off, *u_mask;
    // entries of each list.  Past 2^32 staged matches (a result that is counted,
    // but never written) the low word of counter 0 carries into the number of
    // hits, and list slots up to one per carry lie behind the end: not stored
    uint32_t cap;
    uint32_t *m_row, *m_s, *m_e, *m_cnt;    // mixed hits: tuples [s, e) compared with m_key
    int32_t*  m_key;
    // 0 staged hits << 32 | staged matches mod 2^32, 1 mixed hits, 2 staged
    // matches, 3 mixed matches, 5 rows written directly, 6 blocks that are done
    unsigned long long* ctr;
};
constexpr int      kCtr    = 8;            // counters
constexpr uint32_t kRowHit = 0xffffffffu;  // no mask of a mixed bucket: one of its tuples differs

struct Outs {
    int    n;
    RidOut o[kMaxRidOut];
};

__device__ __forceinline__ void emit(const Outs& outs, uint64_t pos, uint32_t prow, uint32_t brow) {
#pragma unroll 4
    for (int i = 0; i < outs.n; ++i) {
        const RidOut& o = outs.o[i];
        const uint32_t x = o.side == 0 ? prow : brow;
        o.dst[pos]       = o.src ? __ldg(o.src + x) : x;
    }
}

// Key of row i of tile `tile`; false for NULL and past the end.
template <int SRC>
__device__ __forceinline__ bool tile_key(const KeyCol& pk, uint64_t tile, uint32_t i, int32_t& key) {
    const uint64_t r = tile * kTileRows + i;
    key              = 0;
    if (i >= kTileRows || r >= pk.n) return false;
    if (SRC == kSrcPages) {
        key = __ldcs(reinterpret_cast<const int32_t*>(pk.col.pages + tile * kPage + 4) + i);
        return true;
    } else if (SRC == kSrcPlain) {
        key = __ldcs(pk.col.plain + r);
        return bit_valid(pk.col.valid, r);
    } else if (SRC == kSrcTagged) {
        const uint64_t t = __ldcs(pk.col.tagged + r);
        key              = int32_t(uint32_t(t));
        return (t >> 62) == 1;
    } else {
        const uint64_t row = pk.rid ? uint64_t(__ldg(pk.rid + r)) : r;
        bool           ok  = int_get(pk.col, row, key);
        // a filtered scan read raw: rows failing its predicate never match
        if (pk.filt.n && ok) ok = filt_pass(pk.filt, row);
        return ok;
    }
}

// Bucket of a key (directories have at most 26 bits).
__device__ __forceinline__ uint32_t slot_of(const ProbeTab& T, int32_t key) { return __umulhi(fib_hi(key), T.nb); }

// The block that is done last hands the counters to the host and clears them
// for the next probe (not the mixed hits, which are still to be counted).
// Called by every thread after the block's last update of the counters.
__device__ __forceinline__ void hand_over(const Lists& Ls, unsigned long long* host_ctr) {
    if (!host_ctr || threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(Ls.ctr + 6, 1ull) != gridDim.x - 1) return;
    __threadfence();
    for (int q = 0; q < 6; ++q) {
        host_ctr[q] = atomicAdd(Ls.ctr + q, 0ull);
        if (q != 1) Ls.ctr[q] = 0;
    }
    Ls.ctr[6] = 0;
}

// Tuples of bucket p that equal key k, as a mask over the bucket, for a small
// mixed bucket with the high summary word hi; b0: its first tuple, row: the
// build row of a single match.
__device__ __forceinline__ uint32_t compare_mixed(const ProbeTab& T, int32_t k, uint32_t hi, uint32_t& b0, uint32_t& row) {
    const uint32_t bm = bloom_mask(fib_hash(k)), len = (hi >> 16) & kSumLenMax;
    uint32_t       mm = 0;
    b0 = row = 0;
    if ((hi & bm) != bm) return 0;
    b0 = uint32_t(__ldg(T.dir + slot_of(T, k)) >> 16);
    for (uint32_t q = 0; q < len; ++q) mm |= uint32_t(__ldg(T.keys + b0 + q) == k) << q;
    if (__popc(mm) == 1) row = __ldg(T.rows + b0 + __ffs(mm) - 1);
    return mm;
}

// A hit in a large mixed bucket: listed, to be counted later (rare: one atomic each).
__device__ __forceinline__ void list_mixed(const ProbeTab& T, const Lists& Ls, uint32_t row, int32_t k, uint32_t hi) {
    const uint32_t bm = bloom_mask(fib_hash(k)), p = slot_of(T, k);
    if ((hi & bm) != bm) return;
    const uint64_t q = atomicAdd(Ls.ctr + 1, 1ull);
    Ls.m_row[q]      = row;
    Ls.m_s[q]        = uint32_t(__ldg(T.dir + p) >> 16);
    Ls.m_e[q]        = uint32_t(__ldg(T.dir + p + 1) >> 16);
    Ls.m_key[q]      = k;
    Ls.m_cnt[q]      = kUncounted;
}

__device__ __forceinline__ uint32_t bucket_tuples(const ProbeTab& T, uint32_t p) {
    return uint32_t(__ldg(T.dir + p + 1) >> 16) - uint32_t(__ldg(T.dir + p) >> 16);
}

constexpr uint32_t kMaskTuples = 31;  // tuples of a small mixed bucket, at most

// Count pass of a probe column of one tile: one block, two rows a thread, so
// bound by the latency of its few dependent reads.  Matches keep an order (the
// tile's rows by (i / 32) % 8, then i / 256, then i % 32): a warp takes two
// runs of 32 rows that follow each other in it.  The block writes the counters
// itself.  8 rows a thread with a staged copy of the keys took 11-18 us.
constexpr int kTT = 1024;
template <int SRC>
__global__ void __launch_bounds__(kTT)
    k_probe_tile(ProbeTab T, KeyCol pk, int light_max, Lists Ls, Outs outs, unsigned long long* host_ctr) {
    constexpr uint32_t            kMany = 1u << 31;  // the warp has a hit that only the list can hold
    constexpr int                 kR    = 2;
    __shared__ uint32_t           s_wh[kTT / 32], s_wc[kTT / 32];
    __shared__ unsigned long long s_wx[kTT / 32];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1;
    const uint32_t small = min(uint32_t(light_max), kMaskTuples);
    // a hit: c matches; x = kRowHit: build row s, 0: bucket s, else the mask x over the tuples from s on
    uint32_t s[kR], x[kR], c[kR], row[kR], many = outs.n == 0;
    int32_t  k[kR];
    uint64_t w[kR];
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        row[u] = ((warp & 3) * kR + u) * 256 + (warp >> 2) * 32 + lane;
        w[u]   = tile_key<SRC>(pk, 0, row[u], k[u]) ? __ldg(T.sum + slot_of(T, k[u])) : 0ull;
    }
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        const int32_t  hi  = int32_t(uint32_t(w[u] >> 32));
        const uint32_t len = (uint32_t(hi) >> 16) & kSumLenMax;
        s[u] = x[u] = c[u] = 0;
        // a bucket of one key (hi > 0): its first key decides exactly (a
        // matching key's Bloom bits are always in the bucket's tag)
        if (hi > 0 && sum_head(w[u]) == k[u]) {
            if ((hi >> 30) == 1) {
                s[u] = uint32_t(hi) & 0x3fffffffu;
                x[u] = kRowHit;
                c[u] = 1;
            } else {
                s[u] = slot_of(T, k[u]);
                c[u] = len == kSumLenMax ? bucket_tuples(T, s[u]) : len;
                many |= 1;  // (also one tuple whose row does not fit the summary)
            }
        } else if (hi < 0 && len <= small) {
            uint32_t one;
            x[u] = compare_mixed(T, k[u], uint32_t(hi), s[u], one);
            c[u] = __popc(x[u]);
            many |= c[u] > 1;
            if (c[u] == 1) {
                s[u] = one;
                x[u] = kRowHit;
            }
        } else if (hi < 0) {
            list_mixed(T, Ls, row[u], k[u], uint32_t(hi));
        }
    }
    uint32_t nh = 0, slot[kR];
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        const unsigned bal = __ballot_sync(0xffffffffu, c[u] > 0);
        slot[u]            = nh + __popc(bal & lt);
        nh += __popc(bal);
    }
    many = __any_sync(0xffffffffu, many);
    if (lane == 0) s_wh[warp] = nh | (many ? kMany : 0u);
    __syncthreads();
    const uint32_t h  = s_wh[lane];
    const bool     direct = !__any_sync(0xffffffffu, h & kMany);
    const uint32_t hinc = warp_inclusive_scan(h & ~kMany), hs = __shfl_sync(0xffffffffu, hinc, 31);
    const uint32_t hw   = warp ? __shfl_sync(0xffffffffu, hinc, int(warp) - 1) : 0u;
    unsigned long long total = 0;
    if (direct) {
        for (int oi = 0; oi < outs.n; ++oi) {
            const RidOut o = outs.o[oi];
#pragma unroll
            for (int u = 0; u < kR; ++u)
                if (c[u]) {
                    const uint32_t v         = o.side == 0 ? row[u] : s[u];
                    o.dst[hw + slot[u]] = o.src ? __ldg(o.src + v) : v;
                }
        }
    } else {
        // first output rows from scans of the counts (32-bit prefix sums; the exact total beside them)
        const uint32_t i0 = warp_inclusive_scan(c[0]), t0 = __shfl_sync(0xffffffffu, i0, 31);
        const uint32_t i1 = warp_inclusive_scan(c[1]), t1 = __shfl_sync(0xffffffffu, i1, 31);
        const unsigned long long tx = warp_sum<unsigned long long>((unsigned long long)c[0] + c[1]);
        if (lane == 0) {
            s_wc[warp] = t0 + t1;
            s_wx[warp] = tx;
        }
        __syncthreads();
        const uint32_t cinc = warp_inclusive_scan(s_wc[lane]);
        const uint32_t cw   = warp ? __shfl_sync(0xffffffffu, cinc, int(warp) - 1) : 0u;
        total               = warp_sum(s_wx[lane]);
        const uint32_t oo[kR] = {cw + i0 - c[0], cw + t0 + i1 - c[1]};
#pragma unroll
        for (int u = 0; u < kR; ++u)
            if (c[u]) {
                const uint32_t q = hw + slot[u];
                Ls.u_row[q]      = row[u];
                Ls.u_sp[q]       = s[u];
                Ls.u_off[q]      = oo[u];
                Ls.u_mask[q]     = x[u];
            }
    }
    if (threadIdx.x == 0) {
        unsigned long long* to = host_ctr ? host_ctr : Ls.ctr;
        const unsigned long long mixed = atomicAdd(Ls.ctr + 1, 0ull);  // (the block's barriers are behind its listings)
        to[0] = direct ? 0ull : (uint64_t(hs) << 32) | uint32_t(total);
        to[1] = mixed;
        to[2] = total;
        to[3] = 0;
        to[5] = direct ? hs : 0u;
    }
}

// Count pass of a probe column of several tiles.  A warp works by itself, kSU
// rows a lane at a time, and puts off what only some rows need until a warp
// is full of it: hits wait in its queue until 256 go out together (single
// matches straight to the output, others to the list: one reservation each,
// coalesced stores), rows that met a small mixed bucket until 32 are compared,
// a lane each.  A block per tile with barriers and one reservation (as for a
// single tile, to keep its order) took 126 us for 10M keys against 1M, 70%
// matching; this 80.  Bound by the L1, whose random reads take a line each: the
// queues leave 92 KB of it at 256 hits; at 384 the same probe takes 140 us, at
// 128 (reservations twice as often) 103, with four rows a lane 253.
constexpr int      kSU   = 2;    // rows per lane in flight
constexpr uint32_t kQ     = 256;  // hits that a flush takes (reservations on one word run at 1.6e9/s in all)
constexpr uint32_t kQMore = 32 * kSU;  // what a step adds at most before the next flush
struct StreamQueues {
    // hits: probe row, s, and kRowHit, a mask, or kLen | tuples of bucket s
    uint32_t row[kQ + kQMore], s[kQ + kQMore], x[kQ + kQMore];
    uint32_t m_row[31 + kQMore + 1], m_hi[31 + kQMore + 1];
    int32_t  m_key[31 + kQMore + 1];  // rows that met a small mixed bucket: key and its summary's high word
};
constexpr uint32_t kLen = 1u << 31;

template <int SRC>
__global__ void __launch_bounds__(kPT, 4)
    k_probe_stream(ProbeTab T, KeyCol pk, int light_max, Lists Ls, uint64_t ntiles, Outs outs,
                   unsigned long long* host_ctr) {
    extern __shared__ __align__(128) uint8_t dyn[];
    const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1;
    StreamQueues&  Q    = reinterpret_cast<StreamQueues*>(dyn)[threadIdx.x >> 5];
    const uint32_t small = min(uint32_t(light_max), kMaskTuples);  // masks of 31 tuples leave kLen and kRowHit apart
    uint32_t       nq = 0, nm = 0;  // entries of the queues (the same in every lane)
    unsigned long long listed = 0;  // this lane's listed matches
    // The queue's last kQ hits out: matches of one build row each to the output
    // (to the list when there is none), the others to the list.
    auto flush = [&](uint32_t keep) {
        while (nq > keep) {
            __syncwarp();
            const uint32_t n = min(nq, kQ);
            nq -= n;
            const uint32_t *qr = Q.row + nq, *qs = Q.s + nq, *qx = Q.x + nq;
            auto one = [&](uint32_t e) { return outs.n != 0 && qx[e] == kRowHit; };
            uint32_t nd = 0, tot = 0;  // direct entries; listed matches
            for (uint32_t e = lane; e - lane < n; e += 32) {
                const bool     on = e < n, d = on && one(e);
                const uint32_t x  = on && !d ? qx[e] : 0u;
                nd += __popc(__ballot_sync(0xffffffffu, d));
                tot += x == kRowHit ? 1u : x & kLen ? x & ~kLen : uint32_t(__popc(x));
            }
            listed += tot;
            uint32_t           db = 0;
            unsigned long long lb = 0;
            if (nd < n) tot = warp_sum(tot);
            if (lane == 0) {
                if (nd) db = uint32_t(atomicAdd(Ls.ctr + 5, (unsigned long long)nd));
                if (nd < n) lb = atomicAdd(Ls.ctr + 0, (uint64_t(n - nd) << 32) + tot);
            }
            db = __shfl_sync(0xffffffffu, db, 0);
            if (nd == n) {
                for (int oi = 0; oi < outs.n; ++oi) {
                    const RidOut o = outs.o[oi];
                    const uint32_t* v = o.side == 0 ? qr : qs;
#pragma unroll 4
                    for (uint32_t e = lane; e < n; e += 32) o.dst[db + e] = o.src ? __ldg(o.src + v[e]) : v[e];
                }
                __syncwarp();
                continue;
            }
            lb = __shfl_sync(0xffffffffu, lb, 0);
            uint32_t li = uint32_t(lb >> 32), off = uint32_t(lb);
            for (uint32_t e = lane; e - lane < n; e += 32) {
                const bool     on = e < n, d = on && one(e);
                const unsigned bd = __ballot_sync(0xffffffffu, d), bl = __ballot_sync(0xffffffffu, on && !d);
                const uint32_t x  = on && !d ? qx[e] : 0u;
                const uint32_t c  = x == kRowHit ? 1u : x & kLen ? x & ~kLen : uint32_t(__popc(x));
                const uint32_t in = warp_inclusive_scan(c);
                if (d) {
                    for (int oi = 0; oi < outs.n; ++oi) {
                        const RidOut   o = outs.o[oi];
                        const uint32_t v = o.side == 0 ? qr[e] : qs[e];
                        o.dst[db + __popc(bd & lt)] = o.src ? __ldg(o.src + v) : v;
                    }
                } else if (const uint32_t h = li + __popc(bl & lt); on && h < Ls.cap) {
                    Ls.u_row[h]  = qr[e];
                    Ls.u_sp[h]   = qs[e];
                    Ls.u_off[h]  = off + in - c;
                    Ls.u_mask[h] = x != kRowHit && (x & kLen) ? 0u : x;
                }
                db += __popc(bd);
                li += __popc(bl);
                off += __shfl_sync(0xffffffffu, in, 31);
            }
            __syncwarp();
        }
    };
    // a lane's hit to the queue; every lane of the warp calls it
    auto push = [&](bool on, uint32_t row, uint32_t s, uint32_t x) {
        const unsigned bal = __ballot_sync(0xffffffffu, on);
        if (on) {
            const uint32_t q = nq + __popc(bal & lt);
            Q.row[q] = row;
            Q.s[q]   = s;
            Q.x[q]   = x;
        }
        nq += __popc(bal);
    };
    // rows that met a small mixed bucket: its tuples compared, the matching ones as a mask
    auto compare = [&](uint32_t keep) {
        while (nm > keep) {
            __syncwarp();
            const uint32_t n = min(nm, 32u);
            nm -= n;
            uint32_t mm = 0, row = 0, b0 = 0, one = 0;
            if (lane < n) {
                row = Q.m_row[nm + lane];
                mm  = compare_mixed(T, Q.m_key[nm + lane], Q.m_hi[nm + lane], b0, one);
            }
            __syncwarp();
            const bool single = __popc(mm) == 1;
            push(mm != 0, row, single ? one : b0, single ? kRowHit : mm);
            flush(kQ - 1);
        }
    };
    int32_t  nk[kSU];
    uint32_t nok = 0;  // keys of the next step, and which are valid
    auto     fetch = [&](uint64_t tile, uint32_t x0) {
        nok = 0;
#pragma unroll
        for (int u = 0; u < kSU; ++u)
            nok |= uint32_t(tile_key<SRC>(pk, tile, x0 + u * kPT + threadIdx.x, nk[u])) << u;
    };
    uint64_t tile = blockIdx.x;
    uint32_t x0   = 0;
    if (tile < ntiles) fetch(tile, 0);
    while (tile < ntiles) {
        int32_t        k[kSU];
        uint64_t       w[kSU];
        const uint32_t ok = nok;
        const uint32_t r0 = uint32_t(tile * kTileRows + x0 + threadIdx.x);
#pragma unroll
        for (int u = 0; u < kSU; ++u) {
            k[u] = nk[u];
            // through L1: with skewed probe keys the hot buckets' summaries stay there
            w[u] = (ok >> u) & 1u ? __ldg(T.sum + slot_of(T, k[u])) : 0ull;
        }
        x0 += kSU * kPT;
        if (x0 >= kTileRows) {
            x0 = 0;
            tile += gridDim.x;
        }
        if (tile < ntiles) fetch(tile, x0);
#pragma unroll
        for (int u = 0; u < kSU; ++u) {
            const int32_t  hi  = int32_t(uint32_t(w[u] >> 32));
            const uint32_t row = r0 + u * kPT, len = (uint32_t(hi) >> 16) & kSumLenMax;
            // a bucket of one key (hi > 0): its first key decides exactly (a
            // matching key's Bloom bits are always in the bucket's tag)
            const bool hit  = hi > 0 && sum_head(w[u]) == k[u];
            const bool one  = hit && (hi >> 30) == 1;
            const bool mix  = hi < 0 && len <= small;
            const bool rare = (hi < 0 && len > small) || (hit && !one && len == kSumLenMax);
            push(hit && !rare, row, one ? uint32_t(hi) & 0x3fffffffu : slot_of(T, k[u]), one ? kRowHit : kLen | len);
            if (__any_sync(0xffffffffu, hi < 0 || rare)) {
                const unsigned bal = __ballot_sync(0xffffffffu, mix);
                if (mix) {
                    const uint32_t q = nm + __popc(bal & lt);
                    Q.m_row[q]       = row;
                    Q.m_key[q]       = k[u];
                    Q.m_hi[q]        = uint32_t(hi);
                }
                nm += __popc(bal);
                if (rare) {
                    // a length beyond its field (listed at once), or a large mixed bucket
                    if (hi > 0) {
                        const uint32_t           p = slot_of(T, k[u]), n = bucket_tuples(T, p);
                        const unsigned long long base = atomicAdd(Ls.ctr + 0, (1ull << 32) + n);
                        const uint32_t           h    = uint32_t(base >> 32);
                        if (h < Ls.cap) {
                            Ls.u_row[h]  = row;
                            Ls.u_sp[h]   = p;
                            Ls.u_off[h]  = uint32_t(base);
                            Ls.u_mask[h] = 0;
                        }
                        listed += n;
                    } else {
                        list_mixed(T, Ls, row, k[u], uint32_t(hi));
                    }
                }
            }
        }
        flush(kQ - 1);
        compare(31);
    }
    compare(0);
    flush(0);
    listed = warp_sum(listed);
    if (lane == 0 && listed) atomicAdd(Ls.ctr + 2, listed);
    __syncthreads();
    hand_over(Ls, host_ctr);
}

// Mixed hits still uncounted: a warp each for buckets of up to kMixedWarpMax
// tuples, a block each above.
__global__ void __launch_bounds__(256) k_mixed_count_warp(ProbeTab T, Lists Ls) {
    const uint64_t n    = Ls.ctr[1];
    const unsigned lane = threadIdx.x & 31;
    const uint64_t gw   = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw   = (uint64_t(gridDim.x) * blockDim.x) >> 5;
    unsigned long long acc = 0;
    for (uint64_t q = gw; q < n; q += nw) {
        if (Ls.m_cnt[q] != kUncounted) continue;
        const uint32_t s = Ls.m_s[q], e = Ls.m_e[q];
        if (e - s > kMixedWarpMax) continue;
        const int32_t key = Ls.m_key[q];
        uint32_t      c   = 0;
        for (uint32_t i = s + lane; i < e; i += 32) c += __ldg(T.keys + i) == key;
        c = warp_sum(c);
        if (lane == 0) {
            Ls.m_cnt[q] = c;
            acc += c;
        }
    }
    if (lane == 0 && acc) atomicAdd(Ls.ctr + 3, acc);
}

__global__ void __launch_bounds__(512) k_mixed_count(ProbeTab T, Lists Ls) {
    __shared__ unsigned long long s_red[33];
    const uint64_t n   = Ls.ctr[1];
    uint64_t       acc = 0;
    for (uint64_t q = blockIdx.x; q < n; q += gridDim.x) {
        const uint32_t s = Ls.m_s[q], e = Ls.m_e[q];
        if (e - s <= kMixedWarpMax || Ls.m_cnt[q] != kUncounted) continue;
        const int32_t  key = Ls.m_key[q];
        unsigned long long c = 0;
        for (uint32_t k = s + threadIdx.x; k < e; k += blockDim.x) c += __ldg(T.keys + k) == key;
        unsigned long long tot;
        block_exclusive_scan<unsigned long long>(c, s_red, &tot);
        if (threadIdx.x == 0) {
            Ls.m_cnt[q] = uint32_t(tot);
            acc += tot;
        }
    }
    if (threadIdx.x == 0 && acc) atomicAdd(Ls.ctr + 3, (unsigned long long)acc);
}

// Largest h < n with off[h] <= x (off non-decreasing, off[0] = 0).
__device__ __forceinline__ uint64_t hit_of(const uint32_t* __restrict__ off, uint64_t n, uint64_t x) {
    uint64_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint64_t mid = (lo + hi) >> 1;
        if (__ldg(off + mid) <= x) lo = mid;
        else                       hi = mid;
    }
    return lo;
}

// chunk_first[c] = the uniform hit holding the first output position of chunk c.
// Chunk c is the positions from c * chunk - lead on, those below 0 absent.
__global__ void k_chunk_first(const uint32_t* __restrict__ off, uint64_t n_u, uint64_t nchunks, uint32_t chunk,
                              uint32_t lead, uint32_t* __restrict__ chunk_first) {
    const uint64_t c = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c < nchunks) chunk_first[c] = uint32_t(hit_of(off, n_u, c ? c * chunk - lead : 0));
}

// Outputs of one warp's chunk in k_write_uniform<G>, and the per-warp
// shared memory: the chunk's hits (at most chunk + 1: every hit holds at least
// one output, plus the hit that starts at the next chunk's first position):
// relative starts (chunk + 2), probe rows, tuple starts, unclamped relative
// starts and masks.
constexpr uint32_t warp_chunk(int G) { return 32u * uint32_t(G); }
constexpr size_t   write_uniform_smem(int G) { return 8 * 5 * (size_t(warp_chunk(G)) + 2) * sizeof(uint32_t); }

// Index of the k-th set bit of m (k < popcount(m)).
__device__ __forceinline__ uint32_t nth_bit(uint32_t m, uint32_t k) {
    for (uint32_t i = 0; i < k; ++i) m &= m - 1;
    return uint32_t(__ffs(m) - 1);
}

// G consecutive values to dst (16-byte aligned runs of 4 as vector stores).
template <int G>
__device__ __forceinline__ void store_run(uint32_t* dst, const uint32_t (&v)[G], bool vec, uint64_t pol) {
    if (G >= 4 && vec) {
#pragma unroll
        for (int i = 0; i < G; i += 4)
            st_hint(reinterpret_cast<uint4*>(dst + i), make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]), pol);
    } else if (G == 2 && vec) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(v[0], v[G > 1 ? 1 : 0]);
    } else {
#pragma unroll
        for (int i = 0; i < G; ++i) dst[i] = v[i];
    }
}

template <int G>
__global__ void __launch_bounds__(256, G <= 4 ? 6 : (G <= 8 ? 4 : 2))
    k_write_uniform(ProbeTab T, Lists Ls, uint64_t n_u, const uint32_t* __restrict__ chunk_first, uint64_t total,
                    uint32_t lead, Outs outs) {
    const uint32_t* __restrict__ off = Ls.u_off;
    constexpr uint32_t CH = warp_chunk(G);
    constexpr uint32_t NW = CH + 2;
    extern __shared__ __align__(16) uint32_t wsh[];
    const unsigned lane  = threadIdx.x & 31;
    uint32_t*      s_rel  = wsh + (threadIdx.x >> 5) * 5 * NW;  // hit starts relative to the chunk, clamped to [0, len]
    uint32_t*      s_pr   = s_rel + NW;                         // probe row of each hit
    uint32_t*      s_s    = s_pr + NW;                          // first tuple of each hit's bucket
    uint32_t*      s_orel = s_s + NW;                           // hit start - chunk start, mod 2^32
    uint32_t*      s_msk  = s_orel + NW;                        // match mask (0: every tuple)
    // vector stores need every stream 16-byte aligned at a chunk's start: `lead` words
    // before the first one's (the engine's streams start at the same word, behind
    // the rows that the count pass wrote).  6M rows behind one of them: 75 us with
    // single stores, 71 with vectors, and 72 behind none.
    bool vec = true;
    for (int oi = 0; oi < outs.n; ++oi)
        vec &= ((reinterpret_cast<uintptr_t>(outs.o[oi].dst) - 4 * lead) & 15) == 0;
    const uint64_t nchunks = (total + lead + CH - 1) / CH;
    const uint64_t nw      = (uint64_t(gridDim.x) * blockDim.x) >> 5;
    const uint64_t stream  = l2_evict_first();  // row ids are written once, read later in order
    for (uint64_t c = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; c < nchunks; c += nw) {
        const int64_t  o0  = int64_t(c * CH) - lead;
        const uint32_t len = uint32_t(umin64(CH, uint64_t(int64_t(total) - o0)));
        const uint32_t q_lo = c ? 0 : lead;  // the chunk's outputs are [q_lo, len)
        const uint64_t h0  = chunk_first ? __ldg(chunk_first + c) : hit_of(off, n_u, c ? o0 : 0);
        const uint64_t h1  = c + 1 < nchunks ? (chunk_first ? __ldg(chunk_first + c + 1) : hit_of(off, n_u, o0 + CH))
                                             : n_u - 1;
        const uint32_t nh  = uint32_t(h1 - h0) + 1;  // hits h0 .. h0 + nh - 1 cover the chunk
        if (nh == 1) {
            // the whole chunk inside one hit (the usual case for a Zipf-heavy
            // key): lane 0 reads the hit, every lane takes consecutive matches
            uint32_t orel = 0, m = 0, t0 = 0, prow = 0;
            if (lane == 0) {
                orel           = uint32_t(int64_t(__ldg(off + h0)) - o0);  // mod 2^32: the hit may start earlier
                m              = __ldg(Ls.u_mask + h0);
                const uint32_t sp = __ldg(Ls.u_sp + h0);
                prow           = __ldg(Ls.u_row + h0);
                t0             = m ? sp : uint32_t(__ldg(T.dir + sp) >> 16);
            }
            orel = __shfl_sync(0xffffffffu, orel, 0);
            m    = __shfl_sync(0xffffffffu, m, 0);
            t0   = __shfl_sync(0xffffffffu, t0, 0);
            prow = __shfl_sync(0xffffffffu, prow, 0);
            const uint32_t q0 = lane * G;
            if (q0 < len) {
                uint32_t brow[G];
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    const uint32_t idx = q0 + i - orel;  // match number within the hit
                    brow[i]            = q0 + i >= len || q0 + i < q_lo ? 0u
                                       : m == kRowHit ? t0 : __ldg(T.rows + t0 + (m ? nth_bit(m, idx) : idx));
                }
                const bool full = q0 >= q_lo && q0 + G <= len;
                for (int oi = 0; oi < outs.n; ++oi) {
                    const RidOut o = outs.o[oi];
                    uint32_t     v[G];
                    const uint32_t pv = o.side == 0 ? (o.src ? __ldg(o.src + prow) : prow) : 0u;
#pragma unroll
                    for (int i = 0; i < G; ++i)
                        v[i] = o.side == 0 ? pv : ((o.src && q0 + i < len) ? __ldg(o.src + brow[i]) : brow[i]);
                    uint32_t* dst = o.dst + (o0 + int64_t(q0));
                    if (full) {
                        store_run<G>(dst, v, vec, stream);
                    } else {
#pragma unroll
                        for (int i = 0; i < G; ++i)
                            if (q0 + i >= q_lo && q0 + i < len) dst[i] = v[i];
                    }
                }
            }
            continue;
        }
        for (uint32_t q = lane; q <= nh; q += 32) {
            const uint64_t hq  = h0 + q;
            const int64_t  o   = hq < n_u ? int64_t(__ldg(off + hq)) : int64_t(total);
            const uint64_t rel = o > o0 ? uint64_t(o - o0) : 0;
            s_rel[q]           = uint32_t(umin64(rel, len));
            if (q < nh) {
                const uint32_t m  = __ldg(Ls.u_mask + hq);
                const uint32_t sp = __ldg(Ls.u_sp + hq);
                s_pr[q]   = __ldg(Ls.u_row + hq);
                // a uniform hit names its bucket: the start is its directory word's
                s_s[q]    = m ? sp : uint32_t(__ldg(T.dir + sp) >> 16);
                s_orel[q] = uint32_t(o - o0);
                s_msk[q]  = m;
            }
        }
        __syncwarp();
        const uint32_t q0 = lane * G;
        if (q0 < len) {
            uint32_t prow[G], brow[G];
            uint32_t lo = 0, hi = nh;  // largest k with s_rel[k] <= q0
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (s_rel[mid] <= q0) lo = mid;
                else                  hi = mid;
            }
            uint32_t k = lo;
#pragma unroll
            for (int i = 0; i < G; ++i) {
                const uint32_t q = q0 + i;
                prow[i] = brow[i] = 0;
                if (q >= q_lo && q < len) {
                    while (s_rel[k + 1] <= q) ++k;
                    const uint32_t idx = q - s_orel[k];  // match number within the hit
                    const uint32_t m   = s_msk[k];
                    prow[i]            = s_pr[k];
                    brow[i]            = m == kRowHit ? s_s[k] : __ldg(T.rows + s_s[k] + (m ? nth_bit(m, idx) : idx));
                }
            }
            const bool full = q0 >= q_lo && q0 + G <= len;
            for (int oi = 0; oi < outs.n; ++oi) {
                const RidOut o = outs.o[oi];
                uint32_t     v[G];
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    const uint32_t x = o.side == 0 ? prow[i] : brow[i];
                    v[i]             = (o.src && q0 + i < len) ? __ldg(o.src + x) : x;
                }
                uint32_t* dst = o.dst + (o0 + int64_t(q0));
                if (full) {
                    store_run<G>(dst, v, vec, stream);
                } else {
#pragma unroll
                    for (int i = 0; i < G; ++i)
                        if (q0 + i >= q_lo && q0 + i < len) dst[i] = v[i];
                }
            }
        }
        __syncwarp();  // the next chunk's hits overwrite this warp's shared memory
    }
}

__global__ void __launch_bounds__(256)
    k_write_mixed_warp(ProbeTab T, Lists Ls, const uint64_t* __restrict__ mixed_off, uint64_t base_pos,
                       Outs outs) {
    const uint64_t n    = Ls.ctr[1];
    const unsigned lane = threadIdx.x & 31;
    const uint64_t gw   = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw   = (uint64_t(gridDim.x) * blockDim.x) >> 5;
    for (uint64_t q = gw; q < n; q += nw) {
        const uint32_t s = Ls.m_s[q], e = Ls.m_e[q];
        if (e - s > kMixedWarpMax) continue;
        const uint32_t prow = Ls.m_row[q];
        const int32_t  key  = Ls.m_key[q];
        uint64_t       pos  = base_pos + mixed_off[q];
        for (uint32_t b = s; b < e; b += 32) {
            const uint32_t k   = b + lane;
            const bool     m   = k < e && __ldg(T.keys + k) == key;
            const unsigned bal = __ballot_sync(0xffffffffu, m);
            if (m) emit(outs, pos + __popc(bal & ((1u << lane) - 1)), prow, __ldg(T.rows + k));
            pos += __popc(bal);
        }
    }
}

__global__ void __launch_bounds__(512)
    k_write_mixed(ProbeTab T, Lists Ls, const uint64_t* __restrict__ mixed_off, uint64_t base_pos,
                  Outs outs) {
    __shared__ uint32_t sm[33];
    const uint64_t n = Ls.ctr[1];
    for (uint64_t q = blockIdx.x; q < n; q += gridDim.x) {
        const uint32_t s = Ls.m_s[q], e = Ls.m_e[q], prow = Ls.m_row[q];
        if (e - s <= kMixedWarpMax) continue;  // done by k_write_mixed_warp
        const int32_t  key = Ls.m_key[q];
        uint64_t       pos = base_pos + mixed_off[q];
        for (uint32_t b = s; b < e; b += blockDim.x) {
            const uint32_t k = b + threadIdx.x;
            const bool     m = k < e && __ldg(T.keys + k) == key;
            uint32_t       tot;
            const uint32_t r = block_exclusive_scan<uint32_t>(m ? 1u : 0u, sm, &tot);
            if (m) emit(outs, pos + r, prow, __ldg(T.rows + k));
            pos += tot;
        }
    }
}

// More rows than row ids can number are refused before any is written.
void check_rows(uint64_t rows) {
    if (rows > 0xffffffffull) throw Error(HJ_ERR_INVALID, "join result exceeds 2^32 rows");
}

ProbeTab tab_of(const Table& t) { return ProbeTab{t.dir, t.summary, t.keys, t.rows, 1u << t.dir_bits}; }

// How the count kernels read a probe column's keys.
int key_source(const KeyCol& pk) {
    if (pk.rid || pk.filt.n) return kSrcGather;
    return pk.col.tagged ? kSrcTagged : pk.col.plain ? kSrcPlain : kSrcPages;
}

template <int SRC>
void launch_stream_src(const ProbeTab& T, const KeyCol& pk, int light_max, const Lists& L, const Outs& outs,
                       uint64_t* host_ctr, cudaStream_t st) {
    const uint64_t       ntiles = (pk.n + kTileRows - 1) / kTileRows;
    constexpr size_t     smem   = sizeof(StreamQueues) * (kPT / 32);
    static OncePerDevice    once;
    static std::atomic<int> resident{0};
    once([&] {
        int n = 0;
        HJ_CUDA(cudaFuncSetAttribute(k_probe_stream<SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        HJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_probe_stream<SRC>, kPT, smem));
        resident.store(n);
    });
    const uint64_t grid = std::min<uint64_t>(ntiles, uint64_t(num_sms()) * std::max(1, resident.load()));
    k_probe_stream<SRC><<<unsigned(grid), kPT, smem, st>>>(T, pk, light_max, L, ntiles, outs,
                                                           reinterpret_cast<unsigned long long*>(host_ctr));
    HJ_LAUNCH_CHECK();
}

// Count kernels over a probe column: uniform and mixed lists, counters in
// L.ctr; with outs, matches of one build row a probe row straight to the
// output (pk.n rows each); with host_ctr, the counters to the host and cleared.
void launch_count(const ProbeTab& T, const KeyCol& pk, int light_max, const Lists& L, const Outs& outs,
                  uint64_t* host_ctr, cudaStream_t st) {
    auto run = [&](auto src) {
        constexpr int S = decltype(src)::value;
        if (pk.n > kTileRows) return launch_stream_src<S>(T, pk, light_max, L, outs, host_ctr, st);
        k_probe_tile<S><<<1, kTT, 0, st>>>(T, pk, light_max, L, outs, reinterpret_cast<unsigned long long*>(host_ctr));
        HJ_LAUNCH_CHECK();
    };
    switch (key_source(pk)) {
    case kSrcPages: run(std::integral_constant<int, kSrcPages>{}); break;
    case kSrcPlain: run(std::integral_constant<int, kSrcPlain>{}); break;
    case kSrcTagged: run(std::integral_constant<int, kSrcTagged>{}); break;
    default: run(std::integral_constant<int, kSrcGather>{}); break;
    }
}

// After the counters were read back into host[0..4]: when the count pass
// listed large mixed buckets (host[1] > 0), counts their matches and reads
// their total back into host[3] (one more host wait; most tables have none).
void count_mixed(const ProbeTab& T, const Lists& L, uint64_t* host, cudaStream_t st) {
    if (host[1] == 0) return;
    k_mixed_count_warp<<<num_sms() * 4, 256, 0, st>>>(T, L);
    HJ_LAUNCH_CHECK();
    k_mixed_count<<<num_sms() * 2, 512, 0, st>>>(T, L);
    HJ_LAUNCH_CHECK();
    readback(host + 3, L.ctr + 3, sizeof(uint64_t), true, st);  // page-locked scratch
    HJ_CUDA(cudaStreamSynchronize(st));
}

// Outputs per thread of the uniform writer from option probe_group.
int writer_items(int group) {
    switch (group) {
    case 1: return 1;
    case 2: return 2;
    case 4: return 4;
    case 16:
    case 32: return 16;  // 32 would take 196 KB of shared memory per block
    default: return 8;
    }
}

// ---- build rows that a short probe side can meet ----------------------------
constexpr int      kRT       = 1024;  // threads
constexpr int      kRU       = 8;     // rows per lane in flight
constexpr uint32_t kRedBits  = 17;    // log2 of the bitmap's bits

// Two bits of the bitmap per key (1.4% of other keys have both set at
// kReduceKeys keys, 0.1% at 1984).  MurmurHash3's finaliser, not the
// directory's hash: what passes by chance would else lie in the buckets of the
// keys it was taken for, and those would become large mixed ones.
__device__ __forceinline__ uint32_t red_hash(int32_t k) {
    uint32_t h = uint32_t(k);
    h = (h ^ (h >> 16)) * 0x85ebca6bu;
    h = (h ^ (h >> 13)) * 0xc2b2ae35u;
    return h ^ (h >> 16);
}
__device__ __forceinline__ uint32_t red_bit(uint32_t h, int i) {
    return i ? h & ((1u << kRedBits) - 1) : h >> (32 - kRedBits);
}

// Each block makes the bitmap of the probe keys for itself (they come from the
// L2; a launch less), then streams the build keys once, which bounds it for a
// large build side; for a small one its launch and the host's wait do.  A warp
// reserves once per 256 rows that hold a survivor (reservations on one word run
// at 1.6e9/s).  The join of 10M rows with 1,984: 325 -> 106 us.
template <int SRC>
__global__ void __launch_bounds__(kRT, 2)
    k_reduce(KeyCol b, KeyCol p, Outs outs, unsigned long long* __restrict__ ctr, unsigned long long* host_ctr) {
    __shared__ uint32_t bits[1u << (kRedBits - 5)];
    const unsigned      lane = threadIdx.x & 31, lt = (1u << lane) - 1;
    for (uint32_t i = threadIdx.x; i < (1u << (kRedBits - 5)); i += kRT) bits[i] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < p.n; i += kRT) {
        int32_t k;
        if (tile_key<kSrcGather>(p, i / kTileRows, i % kTileRows, k)) {
            const uint32_t h = red_hash(k);
            for (int q = 0; q < 2; ++q) atomicOr(bits + (red_bit(h, q) >> 5), 1u << (red_bit(h, q) & 31));
        }
    }
    __syncthreads();
    const uint64_t step = uint64_t(gridDim.x) * kRT * kRU;
    for (uint64_t w0 = (uint64_t(blockIdx.x) * (kRT / 32) + (threadIdx.x >> 5)) * (32 * kRU); w0 < b.n; w0 += step) {
        uint64_t r[kRU];
        int32_t  k[kRU];
        uint32_t in = 0;
#pragma unroll
        for (int u = 0; u < kRU; ++u) {
            const uint64_t i = w0 + u * 32 + lane;
            r[u]             = i;
            if (SRC == kSrcGather && i < b.n && b.rid) r[u] = __ldg(b.rid + i);
        }
#pragma unroll
        for (int u = 0; u < kRU; ++u) {
            bool ok = w0 + u * 32 + lane < b.n;
            k[u]    = 0;
            if (ok) {
                if (SRC == kSrcPlain) {
                    k[u] = __ldcs(b.col.plain + r[u]);
                    ok   = bit_valid(b.col.valid, r[u]);
                } else if (SRC == kSrcTagged) {
                    const uint64_t t = __ldcs(b.col.tagged + r[u]);
                    k[u]             = int32_t(uint32_t(t));
                    ok               = (t >> 62) == 1;
                } else {
                    ok = int_get(b.col, r[u], k[u]);
                }
            }
            in |= uint32_t(ok) << u;
        }
        uint32_t n = 0;
        unsigned bal[kRU];
#pragma unroll
        for (int u = 0; u < kRU; ++u) {
            const uint32_t h = red_hash(k[u]), x = red_bit(h, 0), y = red_bit(h, 1);
            bool           s = ((in >> u) & 1u) && ((bits[x >> 5] >> (x & 31)) & 1u);
            if (s) s = (bits[y >> 5] >> (y & 31)) & 1u;
            bal[u] = __ballot_sync(0xffffffffu, s);
            n += __popc(bal[u]);
        }
        if (n == 0) continue;
        uint32_t pos = 0;
        if (lane == 0) pos = uint32_t(atomicAdd(ctr, (unsigned long long)n));
        pos = __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
        for (int u = 0; u < kRU; ++u) {
            if ((bal[u] >> lane) & 1u)
                emit(outs, pos + __popc(bal[u] & lt), 0, uint32_t(w0 + u * 32 + lane));
            pos += __popc(bal[u]);
        }
    }
    // the last block hands the count over and clears it
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(ctr + 6, 1ull) != gridDim.x - 1) return;
    __threadfence();
    host_ctr[0] = atomicAdd(ctr, 0ull);
    ctr[0]      = 0;
    ctr[6]      = 0;
}

// Words between the 16-byte boundary before the first stream's start and that start.
uint32_t stream_lead(const Outs& outs) { return uint32_t(reinterpret_cast<uintptr_t>(outs.o[0].dst) >> 2) & 3; }

template <int G>
void launch_uniform_g(const ProbeTab& T, const Lists& L, uint64_t n_u, const uint32_t* chunk_first, uint64_t total,
                      const Outs& outs, cudaStream_t st) {
    const size_t smem = write_uniform_smem(G);
    static OncePerDevice    once;
    static std::atomic<int> resident{0};
    once([&] {
        int n = 0;
        HJ_CUDA(cudaFuncSetAttribute(k_write_uniform<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        HJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_write_uniform<G>, 256, smem));
        resident.store(n);
    });
    const int per_sm = resident.load();
    const uint32_t lead    = stream_lead(outs);
    const uint64_t nchunks = (total + lead + warp_chunk(G) - 1) / warp_chunk(G);
    const uint64_t grid    = std::max<uint64_t>(1, std::min<uint64_t>((nchunks + 7) / 8, uint64_t(num_sms()) * std::max(1, per_sm)));
    k_write_uniform<G><<<unsigned(grid), 256, smem, st>>>(T, L, n_u, chunk_first, total, lead, outs);
    HJ_LAUNCH_CHECK();
}

// The staged hits' matches (total of them, < 2^32) into the output streams.
void launch_uniform(int G, const ProbeTab& T, const Lists& L, uint64_t n_u, const uint32_t* chunk_first,
                    uint64_t total, const Outs& outs, cudaStream_t st) {
    switch (G) {
    case 1: launch_uniform_g<1>(T, L, n_u, chunk_first, total, outs, st); break;
    case 2: launch_uniform_g<2>(T, L, n_u, chunk_first, total, outs, st); break;
    case 4: launch_uniform_g<4>(T, L, n_u, chunk_first, total, outs, st); break;
    case 16: launch_uniform_g<16>(T, L, n_u, chunk_first, total, outs, st); break;
    default: launch_uniform_g<8>(T, L, n_u, chunk_first, total, outs, st); break;
    }
}

void launch_mixed_writers(const ProbeTab& T, const Lists& L, const uint64_t* mixed_off, uint64_t base_pos,
                          const Outs& outs, cudaStream_t st) {
    k_write_mixed_warp<<<num_sms() * 8, 256, 0, st>>>(T, L, mixed_off, base_pos, outs);
    HJ_LAUNCH_CHECK();
    k_write_mixed<<<num_sms() * 2, 512, 0, st>>>(T, L, mixed_off, base_pos, outs);
    HJ_LAUNCH_CHECK();
}

}  // namespace

struct ProbePlan {
    Lists     ls{};
    uint64_t  n_u = 0, n_m = 0, tot_u = 0, tot_m = 0, tot_d = 0;
    uint64_t* host    = nullptr;  // pinned readback of the counters (owned by the caller)
    int       group   = 8;
};

uint64_t probe_count(const Table& t, const KeyCol& pk, const ProbeParams& prm, const RidOut* ro, int nout,
                     ProbePlan** out, cudaStream_t st) {
    if (nout > kMaxRidOut) throw Error(HJ_ERR_INVALID, "too many output row-id streams");
    auto* pp  = new ProbePlan();
    *out      = pp;
    pp->group = prm.group;
    if (t.n_tuples == 0 || pk.n == 0) return 0;
    if (pk.n > 0xffffffffull) throw Error(HJ_ERR_INVALID, "more than 2^32 probe rows");
    const uint64_t n = pk.n;
    Lists& L         = pp->ls;
    L.u_row = dalloc_n<uint32_t>(n, st);
    L.u_sp  = dalloc_n<uint32_t>(n, st);
    L.u_off = dalloc_n<uint32_t>(n, st);
    L.u_mask = dalloc_n<uint32_t>(n, st);
    L.m_row = dalloc_n<uint32_t>(n, st);
    L.m_s   = dalloc_n<uint32_t>(n, st);
    L.m_e   = dalloc_n<uint32_t>(n, st);
    L.m_cnt = dalloc_n<uint32_t>(n, st);
    L.m_key = dalloc_n<int32_t>(n, st);
    L.cap   = uint32_t(n);
    L.ctr   = reinterpret_cast<unsigned long long*>(prm.counters);
    Outs outs{};
    outs.n = nout;
    for (int i = 0; i < nout; ++i) outs.o[i] = ro[i];
    pp->host = prm.pinned;
    launch_count(tab_of(t), pk, prm.light_max, L, outs, pp->host, st);
    if (prm.after_count) prm.after_count();
    HJ_CUDA(cudaStreamSynchronize(st));
    pp->n_m = pp->host[1];  // probe_free clears their counters
    count_mixed(tab_of(t), L, pp->host, st);
    pp->n_u   = pp->host[0] >> 32;
    pp->tot_u = pp->host[2];
    pp->tot_m = pp->host[3];
    pp->tot_d = pp->host[5];
    return pp->tot_d + pp->tot_u + pp->tot_m;
}

uint64_t reduce_build(const KeyCol& b, const KeyCol& p, const ProbeParams& prm, const RidOut* ro, int nout,
                      cudaStream_t st) {
    if (nout > kMaxRidOut) throw Error(HJ_ERR_INVALID, "too many output row-id streams");
    if (p.n > kReduceKeys || b.n > 0xffffffffull) throw Error(HJ_ERR_INVALID, "reduce_build: too many rows");
    if (b.n == 0 || p.n == 0) return 0;
    Outs outs{};
    outs.n = nout;
    for (int i = 0; i < nout; ++i) outs.o[i] = RidOut{1, ro[i].src, ro[i].dst};
    auto*          ctr  = reinterpret_cast<unsigned long long*>(prm.counters);
    auto*          host = reinterpret_cast<unsigned long long*>(prm.pinned);
    const unsigned grid = unsigned(std::min<uint64_t>(div_up(b.n, kRT * kRU), uint64_t(num_sms()) * 2));
    if (!b.rid && b.col.tagged)     k_reduce<kSrcTagged><<<grid, kRT, 0, st>>>(b, p, outs, ctr, host);
    else if (!b.rid && b.col.plain) k_reduce<kSrcPlain><<<grid, kRT, 0, st>>>(b, p, outs, ctr, host);
    else                            k_reduce<kSrcGather><<<grid, kRT, 0, st>>>(b, p, outs, ctr, host);
    HJ_LAUNCH_CHECK();
    HJ_CUDA(cudaStreamSynchronize(st));
    return prm.pinned[0];
}

uint64_t probe_direct(const ProbePlan* pp) { return pp->tot_d; }

namespace {
// 16 bytes a load, four in flight; an unaligned destination by words, as the last
// ones.  Blocks with an odd index copy b.  Bound by HBM: 7M pairs in 13.6 us, which
// two device copies took 26 for.
__global__ void __launch_bounds__(256)
    k_copy_pairs(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint32_t* __restrict__ da,
                 uint32_t* __restrict__ db, uint64_t n) {
    const uint32_t* s    = blockIdx.x & 1 ? b : a;
    uint32_t*       d    = blockIdx.x & 1 ? db : da;
    const uint64_t  t    = uint64_t(blockIdx.x >> 1) * blockDim.x + threadIdx.x, nt = uint64_t(gridDim.x >> 1) * blockDim.x;
    // (the sources are whole allocations, so 16-byte aligned)
    if (reinterpret_cast<uintptr_t>(d) & 15) {
        for (uint64_t i = t; i < n; i += nt) d[i] = __ldcs(s + i);
        return;
    }
    const uint4*   s4 = reinterpret_cast<const uint4*>(s);
    uint4*         d4 = reinterpret_cast<uint4*>(d);
    const uint64_t n4 = n / 4;
    for (uint64_t i = t; i < n4; i += 4 * nt) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * nt < n4) v[u] = __ldcs(s4 + i + u * nt);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * nt < n4) d4[i + u * nt] = v[u];
    }
    for (uint64_t i = 4 * n4 + t; i < n; i += nt) d[i] = s[i];
}
}  // namespace

void copy_pairs(const uint32_t* a, const uint32_t* b, uint32_t* da, uint32_t* db, uint64_t n, cudaStream_t st) {
    if (n == 0) return;
    const uint64_t half = std::min<uint64_t>(div_up(n, 256 * 16), uint64_t(num_sms()) * 4);
    k_copy_pairs<<<unsigned(2 * half), 256, 0, st>>>(a, b, da, db, n);
    HJ_LAUNCH_CHECK();
}

void probe_write(const Table& t, const KeyCol& pk, ProbePlan* pp, const RidOut* ro, int nout,
                 cudaStream_t st) {
    (void)pk;
    if (nout > kMaxRidOut) throw Error(HJ_ERR_INVALID, "too many output row-id streams");
    if (nout == 0) return;
    check_rows(pp->tot_d + pp->tot_u);
    Outs outs{};
    outs.n = nout;
    for (int i = 0; i < nout; ++i) {
        outs.o[i] = ro[i];
        outs.o[i].dst += pp->tot_d;  // the directly written rows come first
    }
    const ProbeTab T = tab_of(t);
    Lists&         L = pp->ls;
    if (pp->n_u) {
        const int      G       = writer_items(pp->group);
        const uint64_t chunk   = warp_chunk(G);
        const uint32_t lead    = stream_lead(outs);
        const uint64_t nchunks = (pp->tot_u + lead + chunk - 1) / chunk;
        uint32_t*      cfirst  = dalloc_n<uint32_t>(nchunks + 1, st);
        k_chunk_first<<<div_up(nchunks, 256), 256, 0, st>>>(L.u_off, pp->n_u, nchunks, uint32_t(chunk), lead, cfirst);
        HJ_LAUNCH_CHECK();
        launch_uniform(G, T, L, pp->n_u, cfirst, pp->tot_u, outs, st);
        dfree(cfirst, st);
    }
    if (pp->n_m) {
        uint64_t* off = dalloc_n<uint64_t>(pp->n_m + 1, st);
        scan_exclusive_u32_to_u64(L.m_cnt, off, pp->n_m, st);
        launch_mixed_writers(T, L, off, pp->tot_u, outs, st);
        dfree(off, st);
    }
}

namespace {

// Bump carve-out of 256-byte-aligned pieces from a caller-owned buffer.
struct Carve {
    uint8_t* p;
    size_t   used = 0;
    template <class T>
    T* take(uint64_t n) {
        T* r = reinterpret_cast<T*>(p + used);
        used += (n * sizeof(T) + 255) & ~size_t(255);
        return r;
    }
};

}  // namespace

size_t probe_scratch_bytes(uint64_t n) {
    const uint64_t tmp = scan_tmp_words(n) + 1;
    return 256 + 9 * ((4 * n + 255) & ~uint64_t(255)) + ((8 * (n + 1) + 255) & ~uint64_t(255))
         + ((8 * tmp + 255) & ~uint64_t(255));
}

int probe_into_scratch(const Table& t, const KeyCol& pk, const ProbeParams& prm, uint8_t* scratch,
                       size_t scratch_bytes, uint32_t* out_probe, uint32_t* out_build, uint64_t capacity,
                       uint64_t* num_matches, cudaStream_t st) {
    *num_matches = 0;
    if (t.n_tuples == 0 || pk.n == 0) return HJ_OK;
    const uint64_t n = pk.n;
    if (probe_scratch_bytes(n) > scratch_bytes) throw Error(HJ_ERR_INVALID, "probe scratch too small");
    Lists     L{};
    uint64_t *m_off, *tmp;
    Carve     c{scratch};
    L.ctr   = c.take<unsigned long long>(kCtr);
    L.u_row = c.take<uint32_t>(n);
    L.u_sp  = c.take<uint32_t>(n);
    L.u_off = c.take<uint32_t>(n);
    L.u_mask = c.take<uint32_t>(n);
    L.m_row = c.take<uint32_t>(n);
    L.m_s   = c.take<uint32_t>(n);
    L.m_e   = c.take<uint32_t>(n);
    L.m_cnt = c.take<uint32_t>(n);
    L.m_key = c.take<int32_t>(n);
    L.cap   = uint32_t(n);
    m_off   = c.take<uint64_t>(n + 1);
    tmp     = c.take<uint64_t>(scan_tmp_words(n) + 1);
    // the scratch keeps the previous call's contents: the counters restart at zero
    HJ_CUDA(cudaMemsetAsync(L.ctr, 0, 8 * sizeof(unsigned long long), st));
    const ProbeTab T = tab_of(t);
    launch_count(T, pk, prm.light_max, L, Outs{}, nullptr, st);
    uint64_t* h = prm.pinned;
    readback(h, L.ctr, 5 * sizeof(uint64_t), true, st);  // page-locked scratch
    HJ_CUDA(cudaStreamSynchronize(st));
    count_mixed(T, L, h, st);
    const uint64_t n_u = h[0] >> 32, n_m = h[1], tot_u = h[2], total = h[2] + h[3];
    *num_matches = total;
    if (total > capacity) return HJ_ERR_CAPACITY;
    if (total == 0) return HJ_OK;
    check_rows(tot_u);
    Outs outs{};
    outs.n    = 2;
    outs.o[0] = RidOut{0, nullptr, out_probe};
    outs.o[1] = RidOut{1, nullptr, out_build};
    if (n_u) {
        // no chunk map (its size would follow the match count): each chunk
        // finds its first hit by binary search
        launch_uniform(writer_items(prm.group), T, L, n_u, nullptr, tot_u, outs, st);
    }
    if (n_m) {
        scan_exclusive_u32_to_u64_into(L.m_cnt, m_off, n_m, tmp, st);
        launch_mixed_writers(T, L, m_off, tot_u, outs, st);
    }
    return HJ_OK;
}

void probe_free(ProbePlan* pp, cudaStream_t st) {
    if (!pp) return;
    Lists& L = pp->ls;
    if (pp->n_m) cudaMemsetAsync(L.ctr, 0, kCtr * sizeof(unsigned long long), st);
    for (void* p : {(void*)L.u_row, (void*)L.u_sp, (void*)L.u_off, (void*)L.u_mask, (void*)L.m_row, (void*)L.m_s, (void*)L.m_e,
                    (void*)L.m_cnt, (void*)L.m_key})
        if (p) dfree(p, st);
    delete pp;
}

}  // namespace hj
