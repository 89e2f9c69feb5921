// Sparse row closure: a transitive-closure-shaped SCC whose rows stay small.
//
// Shape, as for the dense evaluator: R(z, x) :- R_delta(y, x), S_full(y, z) with S fixed
// (tests/transitive_closure.cpp:60-68 of parallel-RA).  Row x of R evolves on its own, as a
// breadth-first search over S, and a tuple can only repeat a tuple of its own row.  The
// iteration loop finds that out with one random 16-byte claim per candidate in a table of
// all tuples, a candidate stream and a select pass; here a warp runs the whole search of
// kSpRows neighbouring rows by itself, with a Bloom filter of the tuples it has in shared memory
// (a hit is checked against the warp's queue, or the exact table of a large tile), and no tuple is looked up anywhere else.
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
//   sparse_scan          per level: blocks' first positions, level totals
//   sparse_place         keys and ids of every tile's tuples at their positions in the log
//
// Declined (nothing written; the loop runs the SCC): a tile of more than kSpBigQueue tuples, or
// more than kSpBig tiles of more than kSpQueue, more than kSpLevels levels, an initial delta that is not grouped by x, scratch that
// does not fit.
#pragma once
#include "ra_iter.cuh"

namespace ra {

constexpr int kSpShift = 4;
constexpr int kSpRows = 1 << kSpShift;   // rows of a tile
constexpr u32 kSpQueue = 4096;            // tuples of a tile that a warp's own queue holds
constexpr u32 kSpBigQueue = 32768;       // ... and one of the kSpBig large queues, with an exact table
constexpr u32 kSpBigSlots = 2 * kSpBigQueue;
constexpr u32 kSpBig = 512;
constexpr u32 kSpLevels = 1024;          // levels of a tile
constexpr int kSpBlockShift = 8;         // tiles of a block (positions are scanned per block)
constexpr int kSpWarps = 8;              // warps of a CTA
constexpr int kSpCtas = 5;             // CTAs per SM
constexpr u32 kSpBloom = 1024;            // 32-bit words of a warp's filter
constexpr u32 kSpRing = 128;             // the queue's last entries, in shared memory
constexpr int kSpScan = 16;              // loads of a lane in flight while a queue is scanned

constexpr u32 kSpOrder = 1;      // the initial delta is not grouped by x
constexpr u32 kSpWide = 2;       // a tile outgrew its queue or its levels
constexpr u32 kSpArena = 4;      // the arena is too small (the counters say how much is needed)

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
    u32* big_queue;       // big: kSpBigQueue entries each
    u16* big_table;       // big: kSpBigSlots queue indices each (0xffff: empty)
    u32 big;
    u32* arena;           // new tuples of the tiles, (row in tile << bits) | z, in search order
    u64 arena_cap;
    u32* levels;          // per tile: first entry of each level (levels + 1 values)
    u64 levels_cap;
    u64* tile_at;         // per tile: its first arena entry
    u64* tile_lv;         // per tile: its first entry of `levels`
    u32* tile_nlv;        // per tile: levels
    u32* block_lv;        // [block][level] new tuples, then the block's first position within the level
    u64* level_total;     // per level: new tuples
    u64* ctr;             // [0] tiles taken, [1] arena entries, [2] level entries, [3] candidates, [4] large queues taken
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

// First delta row of every tile; the delta must be grouped by x, ascending.
__global__ void __launch_bounds__(kThreads) sparse_bounds_kernel(SparseArgs a)
{
    const u64 mask = (1ull << a.bits) - 1;
    for (u64 i = (u64)blockIdx.x * kThreads + threadIdx.x; i <= a.n_delta; i += (u64)gridDim.x * kThreads) {
        const u64 x = i < a.n_delta ? a.delta[i] & mask : a.n;
        const u64 before = i ? a.delta[i - 1] & mask : 0;
        if (i && before > x) atomicOr(a.flags, kSpOrder);
        const u64 t0 = i ? (before >> kSpShift) + 1 : 0, t1 = i < a.n_delta ? x >> kSpShift : a.tiles;
        for (u64 t = t0; t <= t1 && t <= a.tiles; t++) a.first[t] = i;
    }
}

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

// Is `key` one of the queue's entries (exact table: linear probing, entries are queue indices)?
__device__ __forceinline__ bool sparse_in_table(const u16* table, const u32* q, u32 key)
{
    for (u32 h = sparse_hash(key) % kSpBigSlots, probe = 0; probe < kSpBigSlots; h = (h + 1) % kSpBigSlots, probe++) {
        const u32 v = __ldcg(&table[h]);
        if (v == 0xffffu) return false;
        if (__ldcg(&q[v]) == key) return true;
    }
    return false;
}

__device__ __forceinline__ void sparse_table_insert(u16* table, u32 key, u32 at)
{
    // at most kSpBigQueue entries in twice as many slots: an empty one is met
    for (u32 h = sparse_hash(key) % kSpBigSlots, probe = 0; probe < kSpBigSlots; h = (h + 1) % kSpBigSlots, probe++)
        if (atomicCAS(&table[h], (u16)0xffff, (u16)at) == 0xffff) return;
}

// One warp: tiles from the counter, each tile's search to its end.  Bound by the latency of
// a level's chain -- queue entry (shared memory while the level is narrow) -> edge range ->
// target, two L2 round trips -- and by its instructions; kSpWarps * kSpCtas warps per SM overlap.
// Measured on n = 2^22, out-degree 0.95 (76M new tuples): 1.94 ms, where the loop's joins,
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
    u16* lv = a.warp_lv + gw * kSpLevels;   // first new tuple of each level
    const u32 zmask = (u32)((1ull << a.bits) - 1);
    u64 cands = 0;
    for (;;) {
        u32 tile = 0;
        if (lane == 0)
            tile = (*((volatile u32*)a.flags) & ~kSpArena) ? a.tiles : (u32)atomicAdd((unsigned long long*)&a.ctr[0], 1ull);
        tile = __shfl_sync(0xffffffffu, tile, 0);
        if (tile >= a.tiles) break;
        const u64 d0 = a.first[tile], d1 = a.first[tile + 1];
        const u32 n0 = (u32)min(d1 - d0, (u64)kSpBigQueue + 1);
        if (lane == 0) a.tile_nlv[tile] = 0;
        if (n0 == 0) continue;
        u32* q = a.queue + gw * kSpQueue;
        u32 cap = kSpQueue;
        u16* table = nullptr;   // exact membership of a tile that outgrew kSpQueue
        // to a large queue with an empty exact table, if one is left
        auto go_big = [&]() {
            u32 slot = kSpBig;
            if (lane == 0 && !table) slot = (u32)atomicAdd((unsigned long long*)&a.ctr[4], 1ull);
            slot = __shfl_sync(0xffffffffu, slot, 0);
            if (table || slot >= a.big) return false;
            table = a.big_table + (u64)slot * kSpBigSlots;
            for (u32 i = lane; i < kSpBigSlots / 8; i += 32)
                __stcg((uint4*)table + i, make_uint4(~0u, ~0u, ~0u, ~0u));
            q = a.big_queue + (u64)slot * kSpBigQueue;
            cap = kSpBigQueue;
            __syncwarp();
            return true;
        };
        if (n0 > cap && (n0 > kSpBigQueue || !go_big())) {
            if (lane == 0) atomicOr(a.flags, kSpWide);
            break;
        }
        for (u32 i = lane; i < kSpBloom; i += 32) bloom[i] = 0;
        __syncwarp();
        for (u32 i = lane; i < n0; i += 32) {   // level 0: the initial delta
            const u64 k = a.delta[d0 + i];
            const u32 e = ((u32)(k & (kSpRows - 1)) << a.bits) | (u32)((k >> a.bits) & zmask);
            __stcg(&q[i], e);
            if (table) sparse_table_insert(table, e, i);
            if (n0 - i <= kSpRing) ring[i % kSpRing] = e;
            const u32 h = sparse_hash(e);
            atomicOr(&bloom[h % kSpBloom], sparse_bits(h));
        }
        u32 f0 = 0, qn = n0, nlv = 0;
        bool wide = false;
        __syncwarp();
        for (;;) {
            const u32 f1 = qn;
            for (u32 b = f0; b < f1 && !wide; b += 32) {
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
                cands += tot;
                const u32 ex = incl - deg;
                const u32 has = __ballot_sync(0xffffffffu, deg != 0);
                if (deg) own[__popc(has & lanemask_lt())] = make_uint2(st - ex, e & ~zmask);
                __syncwarp();
                for (u32 j0 = 0; j0 < tot && !wide; j0 += 32) {
                    // candidate j0 + lane: its entry is the last of those with edges that starts at or before it
                    const u32 j = j0 + lane;
                    const u32 starts = __reduce_or_sync(0xffffffffu, deg && ex >= j0 && ex < j0 + 32 ? 1u << (ex - j0) : 0u);
                    const u32 before = j0 ? __popc(__ballot_sync(0xffffffffu, deg && ex < j0)) : 0u;
                    u32 key = 0xffffffffu - lane, word = 0, bm = 0;
                    bool fresh = j < tot, maybe = false;
                    if (fresh) {
                        const uint2 w = own[before + __popc(starts & (lanemask_lt() | 1u << lane)) - 1];
                        key = w.y | __ldg(&a.target[w.x + j]);
                        const u32 h = sparse_hash(key);
                        word = h % kSpBloom;
                        bm = sparse_bits(h);
                        maybe = (atomicOr(&bloom[word], bm) & bm) == bm;
                    }
                    if (__any_sync(0xffffffffu, maybe)) {
                        // in the filter before, or from an equal candidate of this step: the first of
                        // equal ones stays, unless the queue holds it
                        if (__match_any_sync(0xffffffffu, key) & lanemask_lt()) fresh = false;
                        u32 m = __ballot_sync(0xffffffffu, maybe && fresh);
                        if (table) {
                            if (maybe && fresh && sparse_in_table(table, q, key)) fresh = false;
                            m = 0;
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
                    if (qn + __popc(nm) > cap) {
                        const u32* small = q;
                        if (!go_big()) {
                            wide = true;
                            break;
                        }
                        for (u32 i = lane; i < qn; i += 32) {
                            const u32 k = __ldcg(&small[i]);
                            __stcg(&q[i], k);
                            sparse_table_insert(table, k, i);
                        }
                        __syncwarp();
                    }
                    if (fresh) {
                        const u32 i = qn + __popc(nm & lanemask_lt());
                        __stcg(&q[i], key);
                        ring[i % kSpRing] = key;
                        if (table) sparse_table_insert(table, key, i);
                    }
                    qn += __popc(nm);
                    __syncwarp();
                }
            }
            if (wide || nlv + 2 > kSpLevels) {
                wide = true;
                break;
            }
            if (qn == f1) break;
            if (lane == 0) __stcg(&lv[nlv], (u16)(f1 - n0));
            nlv++;
            f0 = f1;
        }
        if (wide) {
            if (lane == 0) atomicOr(a.flags, kSpWide);
            break;
        }
        const u32 fresh_n = qn - n0;
        if (fresh_n == 0) continue;
        if (lane == 0) __stcg(&lv[nlv], (u16)fresh_n);
        __syncwarp();
        u64 at = 0, lat = 0;
        if (lane == 0) {
            at = atomicAdd((unsigned long long*)&a.ctr[1], (unsigned long long)fresh_n);
            lat = atomicAdd((unsigned long long*)&a.ctr[2], (unsigned long long)(nlv + 1));
        }
        at = __shfl_sync(0xffffffffu, at, 0);
        lat = __shfl_sync(0xffffffffu, lat, 0);
        if (at + fresh_n > a.arena_cap || lat + nlv + 1 > a.levels_cap) {
            if (lane == 0) atomicOr(a.flags, kSpArena);   // the other tiles go on: their sizes are wanted
            continue;
        }
        if (lane == 0) {
            a.tile_at[tile] = at;
            a.tile_lv[tile] = lat;
            a.tile_nlv[tile] = nlv;
        }
        for (u32 i0 = lane; i0 < fresh_n; i0 += 128) {   // four entries of a lane in flight
            u32 e[4];
#pragma unroll
            for (int u = 0; u < 4; u++) e[u] = i0 + u * 32 < fresh_n ? __ldcg(&q[n0 + i0 + u * 32]) : 0u;
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (i0 + u * 32 < fresh_n) a.arena[at + i0 + u * 32] = e[u];
        }
        u32* blk = a.block_lv + (u64)(tile >> kSpBlockShift) * kSpLevels;
        for (u32 k = lane; k <= nlv; k += 32) {
            const u32 s = __ldcg(&lv[k]);
            a.levels[lat + k] = s;
            if (k < nlv) atomicAdd(&blk[k], (u32)__ldcg(&lv[k + 1]) - s);
        }
        __syncwarp();
    }
    if (lane == 0 && cands) atomicAdd((unsigned long long*)&a.ctr[3], (unsigned long long)cands);
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
