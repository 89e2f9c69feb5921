// Sparse row closure: a transitive-closure-shaped SCC whose rows stay small.
//
// Shape, as for the dense evaluator: R(z, x) :- R_delta(y, x), S_full(y, z) with S fixed
// (tests/transitive_closure.cpp:60-68 of parallel-RA).  Row x of R evolves on its own, as a
// breadth-first search over S, and a tuple can only repeat a tuple of its own row.  The
// iteration loop finds that out with one random 16-byte claim per candidate in a table of
// all tuples, a candidate stream and a select pass; here a warp runs the whole search of
// kSpRows neighbouring rows by itself, with a Bloom filter of the tuples it has in shared
// memory (a hit is checked against the warp's queue, or against an exact table once that costs
// more), and no tuple is looked up anywhere else.  The few tiles that are too much for a warp are
// searched again by a CTA each.
//
// The log is the loop's, ids included.  When the initial delta is grouped by x (ascending; the
// host path checks it), every later delta of the loop is too: candidates follow the
// order of their outer rows and the first occurrence wins.  So delta k is, x after x, the
// tuples of distance k in the order in which row x's search finds them, and the position of
// a tuple is the tuples of earlier deltas + those of the same delta in earlier tiles +
// its rank in its tile.
//
//   sparse_adj / sparse_bounds  edge ranges and targets in 8 + 4 bytes; each tile's share of
//                        the initial delta, and whether it is grouped by x
//   sparse_search        tiles of kSpRows rows, one warp each: the search, its queue copied to the
//                        arena, new tuples per level counted per block of tiles
//   sparse_big           the same for the tiles that were too much for a warp, one CTA each
//   sparse_scan          per level: blocks' first positions, level totals
//   sparse_place         keys and ids of every tile's tuples at their positions in the log
//
// Declined (nothing written; the loop runs the SCC), as early as can be told: a tile of more
// tuples or candidates than a CTA takes (kSpBigQueue, kSpBigTry), or about to grow past them
// (sparse_grows); more than kSpBig tiles for CTAs, or more large ones than the search pays for
// (SparseArgs::large); more than kSpLevels levels; an initial delta that is not grouped by x;
// scratch that does not fit.
#pragma once
#include "ra_iter.cuh"

namespace ra {

constexpr int kSpShift = 4;
constexpr int kSpRows = 1 << kSpShift;   // rows of a tile
// Tuples of a tile that a warp's own queue holds.  (6,144: a tile of 6,125 in a graph of 2^20 values, whose
// filter hits in every level, took its warp 1.7 ms, 0.9 and a CTA 0.3 so.)
constexpr u32 kSpQueue = 4096;
constexpr u32 kSpBuckets = 1024;         // buckets of four slots of a warp's exact table,
constexpr u32 kSpTable = 3584;           // and the tuples it holds
constexpr u32 kSpTry = 2048;             // candidates of a tile, besides two per tuple, that a warp
constexpr u32 kSpTryMost = 16384;        // takes when there are no other tiles left, and when there are;
constexpr u32 kSpTryOnce = 4096;         // of 32 of its tuples
constexpr u32 kSpBigQueue = 32768;       // ... and a CTA's, in shared memory
constexpr u32 kSpBigTry = 262144;
constexpr u32 kSpBigSlots = 40960;       // slots of a CTA's exact table, beside it
constexpr int kSpBigThreads = 1024;
constexpr u32 kSpBig = 512;              // tiles searched by a CTA; with those handed over early
constexpr u32 kSpBigMost = 8192;         // (by the warps that run at the end, fewer than this)
constexpr u32 kSpLevels = 1024;          // levels of a tile
constexpr int kSpBlockShift = 8;         // tiles of a block (positions are scanned per block)
constexpr int kSpWarps = 8;              // warps of a CTA
constexpr int kSpCtas = 5;               // CTAs per SM
constexpr u32 kSpBloom = 1024;           // 32-bit words of a warp's filter
constexpr u32 kSpRing = 128;             // the queue's last entries, in shared memory
constexpr int kSpScan = 16;              // loads of a lane in flight while a queue is scanned (a round)
constexpr int kSpMany = 8;               // keys of a step to look for from which a table is asked instead,
constexpr u32 kSpScans = 16;             // after so many rounds of the tile, and one for 8 of its tuples
constexpr u32 kSpExact = 1u << 30;
constexpr u32 kSpLook = 2048;            // tuples of a large tile; candidates from which a warp looks
constexpr u32 kSpLookStep = 512;         // around, every so many of them

constexpr u32 kSpNone = 0xffffu;        // an empty slot of a CTA's table, of a warp's
constexpr u32 kSpFree = 0xffffffffu;

constexpr u32 kSpOrder = 1;      // the initial delta is not grouped by x
constexpr u32 kSpWide = 2;       // a tile outgrew its queue or its levels, or too many go to CTAs
constexpr u32 kSpArena = 4;      // the arena is too small (the counters say how much is needed)

// Counters, a cache line each: every tile adds to four of them, and reads the flags.  (In one line with
// the flags the search of n = 2^22 took 2.4 ms instead of 2.2, with more code then.)
constexpr u32 kSpTaken = 0;       // tiles taken
constexpr u32 kSpArenaN = 16;     // arena entries
constexpr u32 kSpLevelN = 32;     // level entries
constexpr u32 kSpTried = 48;      // candidates
constexpr u32 kSpBigN = 64;       // tiles for a CTA
constexpr u32 kSpBigTaken = 80;   // of these taken
constexpr u32 kSpLargeN = 96;     // large tiles
constexpr u32 kSpCtrWords = 112;

struct SparseArgs {
    u64 n;                // values
    int bits;
    u32 tiles, blocks;
    const u64* delta;     // R's initial delta: keys (y << bits) | x, grouped by x
    u64 n_delta;
    u64* first;           // tiles + 1: first delta row of each tile
    u64* adj;             // per value y: (first edge << 24) | edges
    u32* target;          // per edge: z
    u32* queue;           // per warp: kSpQueue entries
    u16* warp_lv;         // per warp: kSpLevels level starts
    u32* table;           // per warp: 4 * kSpBuckets tuples (kSpFree: none)
    u32* big_tile;        // tiles that were too much for a warp, kSpBigMost at most
    u32 large;            // large tiles that the search goes on with
    u32* arena;           // new tuples of the tiles, (row in tile << bits) | z, in search order
    u64 arena_cap;
    u32* levels;          // per tile: first entry of each level (levels + 1 values)
    u64 levels_cap;
    u64* tile_at;         // per tile: its first arena entry
    u64* tile_lv;         // per tile: its first entry of `levels`
    u32* tile_nlv;        // per tile: levels
    u32* block_lv;        // [block][level] new tuples, then the block's first position within the level
    u64* level_total;     // per level: new tuples
    u64* ctr;             // counters, at the words above
    u32* flags;
};

// Edge ranges and targets of S (rows sorted by (y, z)).
__global__ void __launch_bounds__(kThreads) sparse_adj_kernel(SparseArgs a, const u64* __restrict__ csr,
                                                              const u64* __restrict__ keys, u64 sn)
{
    const u64 mask = (1ull << a.bits) - 1;
    for (u64 i = (u64)blockIdx.x * kThreads + threadIdx.x; i < max(a.n, sn); i += (u64)gridDim.x * kThreads) {
        if (i < a.n) {
            const u64 s = csr[i], c = csr[i + 1] - s;
            a.adj[i] = (s << 24) | c;
            if (c >> 24) atomicOr(a.flags, kSpWide);
        }
        if (i < sn) a.target[i] = (u32)(keys[i] & mask);
    }
}

// First delta row of every tile, by search (a thread that fills in the tiles between two rows takes
// 60 us for the 16,000 that a few rows leave without any); the delta must be grouped by x, ascending.
__global__ void __launch_bounds__(kThreads) sparse_bounds_kernel(SparseArgs a)
{
    const u64 mask = (1ull << a.bits) - 1;
    const u64 t0 = (u64)blockIdx.x * kThreads + threadIdx.x, step = (u64)gridDim.x * kThreads;
    for (u64 i = t0; i + 1 < a.n_delta; i += step)
        if ((a.delta[i] & mask) > (a.delta[i + 1] & mask)) atomicOr(a.flags, kSpOrder);
    for (u64 t = t0; t <= a.tiles; t += step) {
        u64 lo = 0, hi = a.n_delta;
        while (lo < hi) {
            const u64 m = (lo + hi) >> 1;
            if ((a.delta[m] & mask) >> kSpShift < t) lo = m + 1;
            else hi = m;
        }
        a.first[t] = lo;
    }
}

// MurmurHash3's 32-bit finaliser.
__device__ __forceinline__ u32 sparse_hash(u32 k)
{
    k ^= k >> 16;
    k *= 0x85ebca6bu;
    k ^= k >> 13;
    k *= 0xc2b2ae35u;
    return k ^ (k >> 16);
}

// Three bits of a filter word (bits 12 up choose them; the word is h % kSpBloom).
__device__ __forceinline__ u32 sparse_bits(u32 h)
{
    return 1u << ((h >> 12) & 31) | 1u << ((h >> 17) & 31) | 1u << ((h >> 22) & 31);
}

// A warp's exact table of tuples of its queue: buckets of four slots, read as one; a tuple is in
// the first bucket from its hash's on that had a free slot.  Does it hold `key`?  (Scanning the queue
// for each repeated candidate is quadratic: 4,375 cliques of 16 values took 2.5 ms, 0.50 with the
// table; 300 rows that lead by 100 hubs to 300 values each, 976 ms.  A filter's false hits are
// few per step and cheaper to scan for: with the table for all, the search of n = 2^22 took 2.9 ms.)
__device__ __forceinline__ bool sparse_in_table(const u32* table, u32 key)
{
    u32 h = sparse_hash(key) % kSpBuckets;
    for (u32 probe = 0; probe < kSpBuckets; probe++) {
        const uint4 v = __ldcg((const uint4*)table + h);
        if (v.x == key || v.y == key || v.z == key || v.w == key) return true;
        if (v.w == kSpFree) return false;   // slots are taken in order
        h = (h + 1) % kSpBuckets;
    }
    return false;
}

// Puts entries [from, to) of the queue in (from == 0: into an empty table), by the warp.
__device__ __forceinline__ void sparse_fill(u32* table, const u32* q, u32 from, u32 to)
{
    const u32 lane = threadIdx.x & 31;
    if (from == 0)
        for (u32 i = lane; i < kSpBuckets; i += 32)
            __stcg((uint4*)table + i, make_uint4(kSpFree, kSpFree, kSpFree, kSpFree));
    __syncwarp();
#pragma unroll 1
    for (u32 i = from + lane; i < to; i += 32) {
        const u32 e = __ldcg(&q[i]);
        u32 at = sparse_hash(e) % kSpBuckets * 4;   // the first free slot from there on
        for (u32 probe = 0; probe < 4 * kSpBuckets && atomicCAS(&table[at], kSpFree, e) != kSpFree; probe++)
            at = (at + 1) % (4 * kSpBuckets);
    }
    __syncwarp();
}

// Is a large tile about to grow much further?  A quarter of its tuples are of the level it is
// finding ([f1, qn) of the queue) or, if those are still few, of the one before ([f0, f1)), and they
// lead to half as many again: a tree's root or a giant component.  (A hub's leaves lead
// nowhere, a subcritical graph's tuples to fewer.)  The closure of a tree of 200,000 nodes, 0.90 ms by
// the loop: 8.1 ms when its root's tile went on to the end of a queue, 1.07 so.
__device__ __forceinline__ bool sparse_grows(const SparseArgs& a, const u32* q, u32 f0, u32 f1, u32 qn, u32 zmask)
{
    if (4 * (qn - f1) >= qn) f0 = f1, f1 = qn;
    const u32 wide = f1 - f0;
    if (4 * wide < qn) return false;
    u32 next = 0;   // a few thousand of at most 2^24
#pragma unroll 2
    for (u32 i = f0 + (threadIdx.x & 31); i < f1; i += 32)
        next += min((u32)__ldg(&a.adj[__ldcg(&q[i]) & zmask]) & 0xffffffu, 1u << 16);
    next = __reduce_add_sync(0xffffffffu, next);
    return 2 * next >= 3 * wide;
}

// A warp looks around in the middle of a tile of many candidates: does the search end (one large
// tile too many, this one about to grow, given up elsewhere), or the tile's (too many candidates for a
// warp: to a CTA; many when no other tiles are left: to a CTA while these have few)?  What a search that
// is given up costs, with 70,000 values, on top of the loop: out-degree 1.05, 8.6 -> 0.1 of 10.2 ms.
// The code that is seldom reached is kept small: as much again slowed the search by a tenth.
constexpr u32 kSpEndWide = 1, kSpEndBig = 2, kSpEndEarly = 3;
__device__ __forceinline__ u32 sparse_look(const SparseArgs& a, const u32* q, u32 f0, u32 f1, u32 qn, u32 nlv,
                                        u32 tried, u32 tot)
{
    if (tried < kSpLook) return 0;
    const bool first = qn >= kSpLook && qn < kSpLook + kSpLookStep;   // about once per large tile
    u32 stop = 0, alone = 0;
    if ((threadIdx.x & 31) == 0) {
        stop = *((volatile u32*)a.flags) & ~kSpArena;
        if (first && atomicAdd((unsigned long long*)&a.ctr[kSpLargeN], 1ull) >= a.large) stop = 1;
        alone = tried > kSpTry + 2 * qn && *((volatile u64*)&a.ctr[kSpTaken]) >= a.tiles &&
                *((volatile u64*)&a.ctr[kSpBigN]) < kSpBig;
    }
    if (__shfl_sync(0xffffffffu, stop, 0)) return kSpEndWide;
    if (first && nlv && sparse_grows(a, q, f0, f1, qn, (u32)((1ull << a.bits) - 1))) return kSpEndWide;
    if (tot > kSpTryOnce || tried > kSpTryMost + 2 * qn) return kSpEndBig;
    return __shfl_sync(0xffffffffu, alone, 0) ? kSpEndEarly : 0;
}

// Where a tile's fresh_n new tuples and nlv + 1 level starts go; is there room; and the level starts lv(k)
// (lv(nlv) == fresh_n), by `threads` threads, of which `t` is one.
__device__ __forceinline__ void sparse_reserve(const SparseArgs& a, u32 fresh_n, u32 nlv, u64* at, u64* lat)
{
    *at = atomicAdd((unsigned long long*)&a.ctr[kSpArenaN], (unsigned long long)fresh_n);
    *lat = atomicAdd((unsigned long long*)&a.ctr[kSpLevelN], (unsigned long long)(nlv + 1));
}

__device__ __forceinline__ bool sparse_room(const SparseArgs& a, u32 tile, u32 fresh_n, u32 nlv, u64 at, u64 lat, u32 t)
{
    if (at + fresh_n > a.arena_cap || lat + nlv + 1 > a.levels_cap) {
        if (t == 0) atomicOr(a.flags, kSpArena);   // the other tiles go on: their sizes are wanted
        return false;
    }
    if (t == 0) {
        a.tile_at[tile] = at;
        a.tile_lv[tile] = lat;
        a.tile_nlv[tile] = nlv;
    }
    return true;
}

template <typename Level>
__device__ __forceinline__ void sparse_put_levels(const SparseArgs& a, u32 tile, u32 nlv, u64 lat, u32 t, u32 threads,
                                                  Level lv)
{
    u32* blk = a.block_lv + (u64)(tile >> kSpBlockShift) * kSpLevels;
    for (u32 k = t; k <= nlv; k += threads) {
        const u32 s = lv(k);
        a.levels[lat + k] = s;
        if (k < nlv) atomicAdd(&blk[k], lv(k + 1) - s);
    }
}

// One warp: tiles from the counter, each tile's search to its end.  Bound by the latency of
// a level's chain -- queue entry (shared memory while the level is narrow) -> edge range ->
// target, two L2 round trips -- and by its instructions; kSpWarps * kSpCtas warps per SM overlap.
// Measured on n = 2^22, out-degree 0.95 (76M new tuples): 1.93 ms, where the loop's joins,
// selects and tail kernel take 8.6 ms and clearing its seen set 1.2 ms.  Tiles of 8, 16 and 32 rows
// with 40 to 48 warps per SM: 3.2, 2.0 and 2.1 ms; 32-bit filter words per warp 512 and 1,024:
// 2.6 and 2.0 ms (a hit scans the queue, so full filters cost the largest tiles most).
__global__ void __launch_bounds__(kSpWarps * 32, kSpCtas) sparse_search_kernel(SparseArgs a)
{
    __shared__ u32 s_bloom[kSpWarps][kSpBloom];
    __shared__ u32 s_ring[kSpWarps][kSpRing];
    __shared__ uint2 s_own[kSpWarps][32];   // entries with edges: first edge - first candidate, row bits
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    u32* bloom = s_bloom[warp];
    u32* ring = s_ring[warp];
    uint2* own = s_own[warp];
    const u64 gw = (u64)blockIdx.x * kSpWarps + warp;
    u32* q = a.queue + gw * kSpQueue;
    u32* table = a.table + gw * 4 * kSpBuckets;
    u16* lv = a.warp_lv + gw * kSpLevels;   // first new tuple of each level
    const u32 zmask = (u32)((1ull << a.bits) - 1);
    for (;;) {
        u32 tile = 0;
        if (lane == 0)
            tile = (*((volatile u32*)a.flags) & ~kSpArena) ? a.tiles : (u32)atomicAdd((unsigned long long*)&a.ctr[kSpTaken], 1ull);
        tile = __shfl_sync(0xffffffffu, tile, 0);
        if (tile >= a.tiles) break;
        const u64 d0 = a.first[tile], d1 = a.first[tile + 1];
        const u32 n0 = (u32)min(d1 - d0, (u64)kSpBigQueue + 1);
        if (lane == 0) a.tile_nlv[tile] = 0;
        if (n0 == 0) continue;
        // why the search ends, or the tile's by this warp
        u32 end = n0 <= kSpQueue ? 0 : n0 <= kSpBigQueue ? kSpEndBig : kSpEndWide;
        for (u32 i = lane; i < kSpBloom; i += 32) bloom[i] = 0;
        __syncwarp();
        for (u32 i = lane; i < n0 && !end; i += 32) {   // level 0: the initial delta
            const u64 k = a.delta[d0 + i];
            const u32 e = ((u32)(k & (kSpRows - 1)) << a.bits) | (u32)((k >> a.bits) & zmask);
            __stcg(&q[i], e);
            if (n0 - i <= kSpRing) ring[i % kSpRing] = e;
            const u32 h = sparse_hash(e);
            atomicOr(&bloom[h % kSpBloom], sparse_bits(h));
        }
        u32 f0 = 0, qn = n0, nlv = 0;
        u32 scans = 0;          // rounds of loads that checks against the queue took; then
                                // kSpExact + the entries of the queue that are in the warp's table
        u32 tried = 0;          // candidates
        __syncwarp();
        while (!end) {
            const u32 f1 = qn;
            for (u32 b = f0; b < f1; b += 32) {
                u32 e = 0, deg = 0, st = 0;
                if (b + lane < f1) {
                    e = qn - b <= kSpRing ? ring[(b + lane) % kSpRing] : __ldcg(&q[b + lane]);
                    const u64 r = __ldg(&a.adj[e & zmask]);
                    deg = (u32)(r & 0xffffffu);
                    st = (u32)(r >> 24);
                }
                u32 incl = deg;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const u32 t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                const u32 tot = __shfl_sync(0xffffffffu, incl, 31);
                if (tot == 0) continue;
                tried += tot;
                if ((tried ^ (tried - tot)) >= kSpLookStep) {   // past a multiple of it
                    end = sparse_look(a, q, f0, f1, qn, nlv, tried, tot);
                    if (end) break;
                }
                const u32 ex = incl - deg;
                const u32 has = __ballot_sync(0xffffffffu, deg != 0);
                if (deg) own[__popc(has & lanemask_lt())] = make_uint2(st - ex, e & ~zmask);
                __syncwarp();
                for (u32 j0 = 0; j0 < tot; j0 += 32) {
                    // candidate j0 + lane: its entry is the last of those with edges that starts at or before it
                    const u32 j = j0 + lane;
                    const u32 starts = __reduce_or_sync(0xffffffffu, deg && ex >= j0 && ex < j0 + 32 ? 1u << (ex - j0) : 0u);
                    const u32 before = j0 ? __popc(__ballot_sync(0xffffffffu, deg && ex < j0)) : 0u;
                    u32 key = 0xffffffffu - lane;
                    bool fresh = j < tot, maybe = false;
                    if (fresh) {
                        const uint2 w = own[before + __popc(starts & (lanemask_lt() | 1u << lane)) - 1];
                        key = w.y | __ldg(&a.target[w.x + j]);
                        const u32 h = sparse_hash(key), bm = sparse_bits(h);
                        maybe = (atomicOr(&bloom[h % kSpBloom], bm) & bm) == bm;
                    }
                    if (__any_sync(0xffffffffu, maybe)) {
                        // in the filter before, or from an equal candidate of this step: the first of
                        // equal ones stays, unless the queue holds it
                        if (__match_any_sync(0xffffffffu, key) & lanemask_lt()) fresh = false;
                        u32 m = __ballot_sync(0xffffffffu, maybe && fresh);
                        if (__popc(m) >= kSpMany) {   // many, and again and again: a table pays
                            if (scans < kSpExact) scans += __popc(m) * (1 + qn / (32 * kSpScan));
                            if (scans > kSpScans + qn / 8) {
                                if (qn > kSpTable) {
                                    end = kSpEndBig;
                                    break;
                                }
                                const u32 from = scans < kSpExact ? 0 : scans - kSpExact;
                                if (from < qn) sparse_fill(table, q, from, qn);
                                scans = kSpExact + qn;
                                if (maybe && fresh && sparse_in_table(table, key)) fresh = false;
                                m = 0;
                            }
                        }
                        for (; m; m &= m - 1) {
                            const int src = __ffs(m) - 1;
                            const u32 k = __shfl_sync(0xffffffffu, key, src);
                            bool found = false;
                            for (u32 t = 0; t < qn && !found; t += 32 * kSpScan) {
                                bool hit = false;
#pragma unroll
                                for (int u = 0; u < kSpScan; u++) {
                                    const u32 i = t + u * 32 + lane;
                                    hit |= i < qn && __ldcg(&q[i]) == k;
                                }
                                found = __any_sync(0xffffffffu, hit);
                            }
                            if (lane == src && found) fresh = false;
                        }
                        __syncwarp();
                    }
                    const u32 nm = __ballot_sync(0xffffffffu, fresh);
                    if (qn + __popc(nm) > kSpQueue) {
                        end = kSpEndBig;
                        break;
                    }
                    if (fresh) {
                        const u32 i = qn + __popc(nm & lanemask_lt());
                        __stcg(&q[i], key);
                        ring[i % kSpRing] = key;
                    }
                    qn += __popc(nm);
                    __syncwarp();
                }
                if (end) break;
            }
            if (nlv + 2 > kSpLevels) end = kSpEndWide;
            if (end) break;
            if (qn == f1) break;
            if (lane == 0) __stcg(&lv[nlv], (u16)(f1 - n0));
            nlv++;
            f0 = f1;
        }
        if (end) {
            if (lane == 0) {   // to a CTA, if these do not have too many
                const u64 at = end == kSpEndWide ? kSpBigMost : atomicAdd((unsigned long long*)&a.ctr[kSpBigN], 1ull);
                if (at < (end == kSpEndBig ? kSpBig : kSpBigMost)) a.big_tile[at] = tile;
                else atomicOr(a.flags, kSpWide);
            }
            continue;
        }
        if (lane == 0 && tried) atomicAdd((unsigned long long*)&a.ctr[kSpTried], (unsigned long long)tried);
        const u32 fresh_n = qn - n0;
        if (fresh_n == 0) continue;
        if (lane == 0) __stcg(&lv[nlv], (u16)fresh_n);
        __syncwarp();
        u64 at = 0, lat = 0;
        if (lane == 0) sparse_reserve(a, fresh_n, nlv, &at, &lat);
        at = __shfl_sync(0xffffffffu, at, 0);
        lat = __shfl_sync(0xffffffffu, lat, 0);
        if (!sparse_room(a, tile, fresh_n, nlv, at, lat, lane)) continue;
        for (u32 i0 = lane; i0 < fresh_n; i0 += 128) {   // four entries of a lane in flight
            u32 e[4];
#pragma unroll
            for (int u = 0; u < 4; u++) e[u] = i0 + u * 32 < fresh_n ? __ldcg(&q[n0 + i0 + u * 32]) : 0u;
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (i0 + u * 32 < fresh_n) a.arena[at + i0 + u * 32] = e[u];
        }
        sparse_put_levels(a, tile, nlv, lat, lane, 32, [&](u32 k) { return (u32)__ldcg(&lv[k]); });
        __syncwarp();
    }
}

// One CTA: tiles that outgrew a warp's queue, searched from their start with the queue and an
// exact table in shared memory, kSpBigThreads candidates at a time.  Equal candidates of one step meet
// in a slot of the table, which keeps the first of them (kSpPending | its thread) until it has its
// place in the queue.  Bound by the step's chain, an L2 round trip or two and four barriers; a level
// of a narrow tile takes 2.2 us.  A warp with its queue and an exact table in L2 took 7 ms for
// 32,768 tuples; n = 70,000, out-degree 1.0 (292 such tiles, given up for their number): 6.1 ms, now 1.8.
constexpr u32 kSpPending = 0x8000u;
static_assert(kSpBigQueue <= kSpPending && kSpBigThreads <= (int)(kSpNone - kSpPending), "a slot's two meanings");
static_assert(kSpBigSlots > kSpBigQueue + kSpBigThreads, "a probe meets an empty slot");
constexpr u64 kSpBigSmem = 4ull * kSpBigQueue + 2ull * kSpBigSlots;

__global__ void __launch_bounds__(kSpBigThreads, 1) sparse_big_kernel(SparseArgs a)
{
    extern __shared__ __align__(16) u32 b_queue[];
    __shared__ u32 s_pre[kSpBigThreads];   // entries of a batch: candidates before it,
    __shared__ u32 s_at[kSpBigThreads];    // its first edge less these
    __shared__ u32 s_key[kSpBigThreads];   // candidates of a step
    __shared__ u32 s_warp[32];
    __shared__ u16 s_lv[kSpLevels];        // first new tuple of each level
    __shared__ u32 s_tile;
    __shared__ u64 s_place[2];
    u32* q = b_queue;
    u16* table = (u16*)(q + kSpBigQueue);
    const u32 t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const u32 zmask = (u32)((1ull << a.bits) - 1);
    u64 cands = 0;
    // exclusive sums over the block, and the total
    auto block_scan = [&](u32 v, u32* total) {
        u32 incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (u32)o) incl += x;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        u32 w = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 x = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= (u32)o) w += x;
        }
        *total = __shfl_sync(0xffffffffu, w, 31);
        const u32 before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31);
        return incl - v + (warp ? before : 0u);
    };
    for (;;) {
        if (t == 0) {
            const u64 n = min(*((volatile u64*)&a.ctr[kSpBigN]), (u64)kSpBigMost);
            const u64 i = (*((volatile u32*)a.flags) & ~kSpArena) ? n : atomicAdd((unsigned long long*)&a.ctr[kSpBigTaken], 1ull);
            s_tile = i < n ? a.big_tile[i] : a.tiles;
        }
        __syncthreads();
        const u32 tile = s_tile;
        if (tile >= a.tiles) break;
        const u64 d0 = a.first[tile];
        const u32 n0 = (u32)(a.first[tile + 1] - d0);   // at most kSpBigQueue
        for (u32 i = t; i < kSpBigSlots / 2; i += kSpBigThreads) ((u32*)table)[i] = ~0u;
        __syncthreads();
        for (u32 i = t; i < n0; i += kSpBigThreads) {   // level 0: the initial delta
            const u64 k = a.delta[d0 + i];
            const u32 e = ((u32)(k & (kSpRows - 1)) << a.bits) | (u32)((k >> a.bits) & zmask);
            q[i] = e;
            for (u32 h = sparse_hash(e) % kSpBigSlots, probe = 0; probe < kSpBigSlots; probe++) {
                if (atomicCAS(&table[h], (u16)kSpNone, (u16)i) == kSpNone) break;   // a repeated tuple twice
                h = h + 1 == kSpBigSlots ? 0 : h + 1;
            }
        }
        __syncthreads();
        u32 f0 = 0, qn = n0, nlv = 0;
        u32 tried = 0;
        bool wide = false;
        for (;;) {
            const u32 f1 = qn;
            for (u32 b = f0; b < f1 && !wide; b += kSpBigThreads) {
                u32 deg = 0, st = 0;
                if (b + t < f1) {
                    const u64 r = __ldg(&a.adj[q[b + t] & zmask]);
                    deg = (u32)(r & 0xffffffu);
                    st = (u32)(r >> 24);
                }
                u32 tot;
                if (__syncthreads_or(deg >> 21)) {   // sums stay below 2^32
                    wide = true;
                    break;
                }
                const u32 pre = block_scan(deg, &tot);
                if (tot > kSpBigTry - tried) {   // uniform
                    wide = true;
                    break;
                }
                s_pre[t] = pre;
                s_at[t] = st - pre;
                tried += tot;
                __syncthreads();
                for (u32 j0 = 0; j0 < tot && !wide; j0 += kSpBigThreads) {
                    // candidate j0 + t: its entry is the last that starts at or before it
                    const u32 j = j0 + t;
                    u32 key = 0, slot = kSpBigSlots;
                    if (j < tot) {
                        u32 at = 0;
#pragma unroll
                        for (u32 h = kSpBigThreads / 2; h; h >>= 1)
                            if (s_pre[at + h] <= j) at += h;
                        key = (q[b + at] & ~zmask) | __ldg(&a.target[s_at[at] + j]);
                    }
                    s_key[t] = key;
                    __syncthreads();
                    if (j < tot) {
                        const u16 own = (u16)(kSpPending | t);
                        for (u32 h = sparse_hash(key) % kSpBigSlots, probe = 0; probe < kSpBigSlots; probe++) {
                            u32 v = *((volatile u16*)&table[h]);
                            if (v == kSpNone) {
                                v = atomicCAS(&table[h], (u16)kSpNone, own);
                                if (v == kSpNone) {
                                    slot = h;
                                    break;
                                }
                            }
                            if ((v & kSpPending ? s_key[v & (kSpPending - 1)] : q[v]) == key) {
                                // known, or the same as another candidate: the first of them stays
                                if (v & kSpPending) slot = h;
                                while ((v & kSpPending) && v > own) {
                                    const u32 seen = atomicCAS(&table[h], (u16)v, own);
                                    if (seen == v) break;
                                    v = seen;
                                }
                                break;
                            }
                            h = h + 1 == kSpBigSlots ? 0 : h + 1;
                        }
                    }
                    __syncthreads();
                    const bool fresh = slot < kSpBigSlots && *((volatile u16*)&table[slot]) == (kSpPending | t);
                    u32 won;
                    const u32 i = qn + block_scan(fresh, &won);
                    if (qn + won > kSpBigQueue) {
                        wide = true;   // uniform
                        break;
                    }
                    if (fresh) {
                        q[i] = key;
                        table[slot] = (u16)i;
                    }
                    qn += won;
                    __syncthreads();
                }
            }
            if (!wide && t == 0 && nlv < kSpLevels) s_lv[nlv] = (u16)(f1 - n0);
            if (wide || nlv + 2 > kSpLevels ||
                (nlv % 16 == 15 && __syncthreads_or(t == 0 && (*((volatile u32*)a.flags) & ~kSpArena)))) {
                wide = true;
                break;
            }
            if (qn == f1) break;
            nlv++;
            f0 = f1;
        }
        if (wide) {
            if (t == 0) atomicOr(a.flags, kSpWide);
            break;
        }
        cands += tried;
        const u32 fresh_n = qn - n0;
        if (fresh_n == 0) continue;
        if (t == 0) {
            s_lv[nlv] = (u16)fresh_n;
            sparse_reserve(a, fresh_n, nlv, &s_place[0], &s_place[1]);
        }
        __syncthreads();
        const u64 at = s_place[0], lat = s_place[1];
        if (sparse_room(a, tile, fresh_n, nlv, at, lat, t)) {
            for (u32 i = t; i < fresh_n; i += kSpBigThreads) a.arena[at + i] = q[n0 + i];
            sparse_put_levels(a, tile, nlv, lat, t, kSpBigThreads, [&](u32 k) { return (u32)s_lv[k]; });
        }
        __syncthreads();
    }
    if (t == 0 && cands) atomicAdd((unsigned long long*)&a.ctr[kSpTried], (unsigned long long)cands);
}

// Per level (one warp each): the blocks' counts to first positions, and the level's total.
__global__ void __launch_bounds__(kThreads) sparse_scan_kernel(SparseArgs a)
{
    const int lane = threadIdx.x & 31;
    const u32 level = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (level >= kSpLevels) return;
    u32 run = 0;
    for (u32 b = 0; b < a.blocks; b += 32) {
        u32* p = a.block_lv + (u64)(b + lane) * kSpLevels + level;
        const u32 c = b + lane < a.blocks ? *p : 0u;
        u32 incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (b + lane < a.blocks) *p = run + incl - c;
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) a.level_total[level] = run;
}

// Per block of tiles: each tile's level starts become its first positions within the level
// (a thread per level walks the block's tiles).
__global__ void __launch_bounds__(kThreads) sparse_offsets_kernel(SparseArgs a, u32* __restrict__ pos)
{
    constexpr int kTiles = 1 << kSpBlockShift;
    __shared__ u64 s_lv[kTiles];
    __shared__ u32 s_n[kTiles];
    __shared__ u32 s_max;
    const u32 t0 = blockIdx.x << kSpBlockShift;
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    for (u32 i = threadIdx.x; i < kTiles; i += kThreads) {
        const u32 n = t0 + i < a.tiles ? a.tile_nlv[t0 + i] : 0;
        s_n[i] = n;
        s_lv[i] = n ? a.tile_lv[t0 + i] : 0;
        if (n) atomicMax(&s_max, n);
    }
    __syncthreads();
    for (u32 k = threadIdx.x; k < s_max; k += kThreads) {
        u32 run = a.block_lv[(u64)blockIdx.x * kSpLevels + k];
        for (u32 i0 = 0; i0 < kTiles; i0 += 8) {
            u32 c[8];
#pragma unroll
            for (int u = 0; u < 8; u++)
                c[u] = k < s_n[i0 + u] ? a.levels[s_lv[i0 + u] + k + 1] - a.levels[s_lv[i0 + u] + k] : 0u;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (k < s_n[i0 + u]) pos[s_lv[i0 + u] + k] = run;
                run += c[u];
            }
        }
    }
}

// A tile's new tuples to the log (one warp per tile): entry i of level k goes to row
// base[k] + pos + (i - the level's first entry).  Neighbouring tiles write neighbouring runs
// of each level.  Bound by the chain tile -> level starts -> entries -> stores, so the next
// tile's start and four entries of a lane are loaded ahead; at sizes beyond L2 by DRAM writes to
// as many places as there are levels, so only the keys go there; ids follow the rows and are
// written row after row.  n = 2^22, 1.5 GB: 1.06 ms with ids beside their keys, 0.78 so.
__global__ void __launch_bounds__(kThreads) sparse_place_kernel(SparseArgs a, const u32* __restrict__ pos,
                                                                const u64* __restrict__ base,
                                                                u64* __restrict__ keys_out, u64* __restrict__ ids_out,
                                                                u64 rows, u64 id0)
{
    constexpr int kAhead = 4;
    const int lane = threadIdx.x & 31;
    const u32 zmask = (u32)((1ull << a.bits) - 1);
    const u32 warps = gridDim.x * kWarps;
    const u32* __restrict__ levels = a.levels;
    const u32* __restrict__ arena = a.arena;
    u32 tile = blockIdx.x * kWarps + (threadIdx.x >> 5);
    u32 nlv = tile < a.tiles ? a.tile_nlv[tile] : 0;
    u64 lat = nlv ? a.tile_lv[tile] : 0, at = nlv ? a.tile_at[tile] : 0;
    u32 start = levels[lat + min((u32)lane, nlv)];
    while (tile < a.tiles) {
        const u32 next = tile + warps;
        const u32 nlv_next = next < a.tiles ? a.tile_nlv[next] : 0;
        const u64 x0 = (u64)tile << kSpShift;
        for (u32 k0 = 0; k0 < nlv; k0 += 32) {   // 32 levels at a time, lane l's level k0 + l
            const u32 k = k0 + lane;
            if (k0) start = levels[lat + min(k, nlv)];
            const u64 to = k < nlv ? base[k] + pos[lat + k] : 0;
            const u32 i1 = levels[lat + min(k0 + 32, nlv)];
            for (u32 i = __shfl_sync(0xffffffffu, start, 0); i < i1; i += 32 * kAhead) {
                u32 e[kAhead];
#pragma unroll
                for (int u = 0; u < kAhead; u++) {
                    const u32 j = i + u * 32 + lane;
                    e[u] = j < i1 ? arena[at + j] : 0u;
                }
#pragma unroll
                for (int u = 0; u < kAhead; u++) {
                    const u32 j = i + u * 32 + lane;
                    if (i + u * 32 >= i1) break;   // uniform
                    u32 l = 0;   // the last level that starts at or before the entry
#pragma unroll
                    for (int h = 16; h; h >>= 1)
                        if (__shfl_sync(0xffffffffu, start, l + h) <= j) l += h;
                    const u64 row = __shfl_sync(0xffffffffu, to, l) + (j - __shfl_sync(0xffffffffu, start, l));
                    if (j < i1) keys_out[row] = ((u64)(e[u] & zmask) << a.bits) | (x0 + (e[u] >> a.bits));
                }
            }
        }
        tile = next;
        nlv = nlv_next;
        lat = nlv ? a.tile_lv[tile] : 0;
        at = nlv ? a.tile_at[tile] : 0;
        start = levels[lat + min((u32)lane, nlv)];
    }
    for (u64 r = (u64)blockIdx.x * kThreads + threadIdx.x; r < rows; r += (u64)gridDim.x * kThreads) ids_out[r] = id0 + r;
}

}  // namespace ra
