// Dense row-closure evaluation of a transitive-closure-shaped SCC.
//
// Shape: one recursive rule  R(z, x) :- R_delta(y, x), S_full(y, z)  with R and
// S binary, S fixed for the SCC, the join on column 0 of both, and the
// output keeping the outer row's column 1 -- the rule of
// tests/transitive_closure.cpp:60-68 of parallel-RA.  Row x of R (the tuples
// (., x)) then evolves on its own: iteration k adds to row x exactly
//     { z : y in delta_k(x), (y, z) in S } \ known(x),
// so every row's sequence of deltas is a breadth-first search over S from
// row x's initial delta, and iteration k of the semi-naive loop is level k of
// all rows' searches.  The evaluator keeps one bit matrix per instance (row x:
// one bit per value of x's instance) and runs each row's whole search in
// shared memory -- a CTA per 32 rows with a bit per row and value (up to kMsMaxN
// values), or a CTA per row, for the known tuples, the frontier and the next
// level -- adding every level's new-tuple count to the per-iteration (and
// per-instance) totals.  The result is the same set of
// tuples, iteration by iteration, as the hash-set path produces; only the
// order in which the new tuples enter the log differs (row by row, values
// ascending).
#pragma once
#include "ra_iter.cuh"

namespace ra {

// One instance's bit matrix: `n` rows (its values, from `base`), each `words`
// u32 words long (bit c of row r: tuple (base + c, base + r) is known), rows
// contiguous from word `word_off`.
struct DenseInst {
    u64 base;
    u64 n;
    u64 words;
    u64 word_off;
};

constexpr u32 kDenseFlagLevels = 1;   // a row went deeper than the level arrays hold
constexpr u32 kDenseFlagRange = 2;    // a value outside its row's instance range
constexpr u64 kDenseMaxN = 65536;     // values per instance (3 rows of bits in shared memory)
// not an edge: the self-loop of an instance's value 0, which never adds a tuple (its target
// is known as soon as its source is on a frontier)
constexpr u32 kNoEdge = 0;

struct DenseArgs {
    const DenseInst* inst;       // n_inst entries (1 without instances)
    const u64* inst_base;        // n_inst + 1 ascending bases for instance_of, or null (one instance)
    u32 n_inst;
    u64 rows;                    // rows 0 .. rows-1 are the values of the union
    u32* known;                  // known tuples; after the closure pass: the new ones
    u32* delta0;                 // the SCC's initial delta (the same matrix when R's full version is empty)
    int bits;                    // packed column width
    const u64* s_keys;           // S full rows, sorted
    const u64* s_csr;            // S rows with column 0 == v: [s_csr[v], s_csr[v + 1])
    uint4* s_rec;                // per value: its first seven edges' targets (DenseRec)
    u32* s_edge;                 // per S row: its columns minus its instance's base, column 0 in the upper half
    u64* row_new;                // per row: new tuples
    u64* level_total;            // per iteration: new tuples
    u64* inst_level;             // [iteration][instance] new tuples, or null
    u64 level_cap;
    u64* counters;               // [0], [2..4], [7] chunks taken (per kernel shape), [1] join candidates (S rows visited),
                                 // [5] 1 + the first key found outside its instance, [6] its relation (1: R, 2: S)
    u32* flags;
};

// S rows of value y (the edges a search visits when it reaches y)
__device__ __forceinline__ u64 row_edges(const DenseArgs& a, u64 y)
{
    return y < a.rows ? a.s_csr[y + 1] - a.s_csr[y] : 0;
}

__device__ __forceinline__ u32 dense_instance(const DenseArgs& a, u64 v)
{
    return a.inst_base ? instance_of(a.inst_base, a.n_inst, v) : 0u;
}

// A key with a value outside its row's instance: flag the run, keep the first such key.
__device__ __forceinline__ void dense_range_error(const DenseArgs& a, u64 key, u64 which)
{
    atomicOr(a.flags, kDenseFlagRange);
    if (atomicCAS((unsigned long long*)&a.counters[5], 0ull, (unsigned long long)(key + 1)) == 0ull)
        atomicExch((unsigned long long*)&a.counters[6], (unsigned long long)which);
}

// Bits of R's stored tuples: all of them into `known`, the delta region's also into `delta0`.
__global__ void __launch_bounds__(kThreads) dense_load_kernel(DenseArgs a, const u64* __restrict__ keys,
                                                              u64 n_full, u64 n_total)
{
    for (u64 i = (u64)blockIdx.x * kThreads + threadIdx.x; i < n_total; i += (u64)gridDim.x * kThreads) {
        const u64 k = keys[i];
        const u64 y = column_of(k, 2, 0, a.bits), x = column_of(k, 2, 1, a.bits);
        const u32 inst = dense_instance(a, x);
        const DenseInst d = a.inst[inst];
        const u64 r = x - d.base, c = y - d.base;   // unsigned: values below the base wrap high
        if (r >= d.n || c >= d.n) {
            dense_range_error(a, k, 1);
            continue;
        }
        const u64 w = d.word_off + r * d.words + (c >> 5);
        const u32 bit = 1u << (c & 31);
        atomicOr(&a.known[w], bit);
        if (i >= n_full && a.delta0 != a.known) atomicOr(&a.delta0[w], bit);
    }
}

// S's rows as instance-local pairs, once per SCC (the searches' inner loops then read
// 4 bytes per edge); a row with a value outside its instance is stored as kNoEdge (the
// run fails).
__global__ void __launch_bounds__(kThreads) dense_local_kernel(DenseArgs a, u64 n)
{
    for (u64 j = (u64)blockIdx.x * kThreads + threadIdx.x; j < n; j += (u64)gridDim.x * kThreads) {
        const u64 k = a.s_keys[j];
        const u64 y = column_of(k, 2, 0, a.bits), z = column_of(k, 2, 1, a.bits);
        const DenseInst d = a.inst[dense_instance(a, y)];
        const u64 zl = z - d.base;
        if (zl >= d.n || y - d.base >= d.n) {
            a.s_edge[j] = kNoEdge;
            dense_range_error(a, k, 2);
        } else {
            a.s_edge[j] = (u32)((y - d.base) << 16 | zl);
        }
    }
}

// A value's edges in one 16-byte word: u16 number of edges, then the local targets of up to
// seven (more edges: kRecMany, and the search reads the edge list).  A search step then makes
// one L2 round trip for a value, where edge range and edges make two.
constexpr u32 kRecEdges = 7, kRecMany = 0xffffu;

__global__ void __launch_bounds__(kThreads) dense_rec_kernel(DenseArgs a)
{
    for (u64 v = (u64)blockIdx.x * kThreads + threadIdx.x; v < a.rows; v += (u64)gridDim.x * kThreads) {
        const u64 s = a.s_csr[v], c = a.s_csr[v + 1] - s;
        u32 w[4] = {0, 0, 0, 0};
        if (c > kRecEdges) {
            w[0] = kRecMany;
        } else {
            w[0] = (u32)c;
            for (u32 k = 0; k < (u32)c; k++) w[(k + 1) >> 1] |= (a.s_edge[s + k] & 0xffffu) << (((k + 1) & 1) * 16);
        }
        a.s_rec[v] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Work unit of the searches: `count` consecutive rows of one instance.
struct DenseChunk {
    u64 first_row;
    u32 inst;
    u32 count;
};

constexpr int kDenseLevels = 64;      // levels counted in shared memory per chunk (deeper ones directly)

// A level's new-tuple count of a row: into the chunk's shared counters, or
// (beyond kDenseLevels) straight into the per-iteration totals.
__device__ __forceinline__ void dense_count_level(const DenseArgs& a, u64* lvl, u64 level, u32 inst, u64 cnt)
{
    if (level < (u64)kDenseLevels) {
        lvl[level] += cnt;
    } else if (level < a.level_cap) {
        atomicAdd((unsigned long long*)&a.level_total[level], (unsigned long long)cnt);
        if (a.inst_level)
            atomicAdd((unsigned long long*)&a.inst_level[level * a.n_inst + inst], (unsigned long long)cnt);
    } else {
        atomicOr(a.flags, kDenseFlagLevels);
    }
}

__device__ __forceinline__ void dense_flush_levels(const DenseArgs& a, u64* lvl, u32 inst, int from, int step)
{
    for (int i = from; i < kDenseLevels; i += step) {
        const u64 v = lvl[i];
        if (!v) continue;
        lvl[i] = 0;
        if ((u64)i < a.level_cap) {
            atomicAdd((unsigned long long*)&a.level_total[i], (unsigned long long)v);
            if (a.inst_level) atomicAdd((unsigned long long*)&a.inst_level[(u64)i * a.n_inst + inst], (unsigned long long)v);
        } else {
            atomicOr(a.flags, kDenseFlagLevels);
        }
    }
}

// Rows of instances with more than kMsMaxN values: one CTA per row, chunks taken from
// a device counter; the row's whole search in shared memory.  Dynamic shared memory:
// 3 * wmax u32.
__global__ void __launch_bounds__(kThreads) dense_closure_kernel(DenseArgs a, u32 wmax, const DenseChunk* __restrict__ chunks,
                                                                 u64 n_chunks, u64* __restrict__ chunk_ctr)
{
    extern __shared__ u32 dsm[];
    u32* known = dsm;
    u32* frontier = dsm + wmax;
    u32* next = dsm + 2 * wmax;
    __shared__ u64 s_chunk;
    __shared__ u64 red[kWarps + 1];
    __shared__ u64 lvl[kDenseLevels];
    for (int i = threadIdx.x; i < kDenseLevels; i += kThreads) lvl[i] = 0;
    u64 relax = 0;
    for (;;) {
        if (threadIdx.x == 0) s_chunk = atomicAdd((unsigned long long*)chunk_ctr, 1ull);
        __syncthreads();
        const u64 c = s_chunk;
        if (c >= n_chunks) break;
        const DenseChunk ch = chunks[c];
        const DenseInst d = a.inst[ch.inst];
        const u32 W = (u32)d.words;
        for (u32 k = 0; k < ch.count; k++) {
            const u64 row = ch.first_row + k;
            u32* krow = a.known + d.word_off + (row - d.base) * d.words;
            const u32* drow = a.delta0 + d.word_off + (row - d.base) * d.words;
            bool any = false;
            for (u32 w = threadIdx.x; w < W; w += kThreads) {
                const u32 f = drow[w];
                frontier[w] = f;
                known[w] = krow[w];
                next[w] = 0;
                any |= f != 0;
            }
            if (!__syncthreads_or(any)) continue;   // uniform: no initial delta in this row
            u64 level = 0, total = 0;
            for (;;) {
                for (u32 w = threadIdx.x; w < W; w += kThreads) {
                    u32 f = frontier[w];
                    if (!f) continue;
                    frontier[w] = 0;
                    while (f) {
                        const u32 b = __ffs(f) - 1;
                        f &= f - 1;
                        const u64 y = d.base + (u64)w * 32 + b;
                        const u64 s = a.s_csr[y], e = a.s_csr[y + 1];
                        relax += e - s;
                        for (u64 j = s; j < e; j++) {
                            const u32 z = a.s_edge[j] & 0xffffu;
                            const u32 bit = 1u << (z & 31);
                            if (!(known[z >> 5] & bit)) atomicOr(&next[z >> 5], bit);
                        }
                    }
                }
                __syncthreads();
                u64 cnt = 0;
                for (u32 w = threadIdx.x; w < W; w += kThreads) {
                    const u32 nw = next[w] & ~known[w];
                    next[w] = 0;
                    known[w] |= nw;
                    frontier[w] = nw;
                    cnt += __popc(nw);
                }
                cnt = block_reduce_sum(cnt, red);   // synchronises the block
                if (cnt == 0) break;
                if (threadIdx.x == 0) dense_count_level(a, lvl, level, ch.inst, cnt);
                total += cnt;
                level++;
            }
            // the row's new tuples replace its known bits in global memory
            for (u32 w = threadIdx.x; w < W; w += kThreads) krow[w] = known[w] & ~krow[w];
            if (threadIdx.x == 0) a.row_new[row] = total;
            __syncthreads();
        }
        dense_flush_levels(a, lvl, ch.inst, threadIdx.x, kThreads);
        __syncthreads();
    }
    relax = block_reduce_sum(relax, red);
    if (threadIdx.x == 0 && relax) atomicAdd((unsigned long long*)&a.counters[1], (unsigned long long)relax);
}

// 32 x 32 bit transpose across a warp: bit r of lane l's result is bit l of lane r's word.
__device__ __forceinline__ u32 warp_transpose32(u32 x)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 16, k = 0; j; j >>= 1, k++) {
        const u32 m = k == 0 ? 0x0000ffffu : k == 1 ? 0x00ff00ffu : k == 2 ? 0x0f0f0f0fu : k == 3 ? 0x33333333u : 0x55555555u;
        const u32 y = __shfl_xor_sync(0xffffffffu, x, j);
        x = (lane & j) ? ((x & ~m) | ((y & ~m) >> j)) : ((x & m) | ((y & m) << j));
    }
    return x;
}

// The two queues of a block: entries in shared memory (`near` of each), the rest of a long
// queue in global memory.
struct MsQueue {
    u16* near;
    u16* far;
    u32 nnear, nmax;
    __device__ __forceinline__ u16& at(u32 side, u32 i) const
    {
        return i < nnear ? near[side * nnear + i] : far[(u64)side * nmax + i];
    }
};

// z to the end of queue `side`; called by the lanes that have one (any subset of a warp).
__device__ __forceinline__ void queue_push(const MsQueue& q, u32 side, u32* qn, u32 z)
{
    const u32 m = __activemask();
    const u32 before = __popc(m & lanemask_lt());
    u32 at = 0;
    if (before == 0) at = atomicAdd(qn, (u32)__popc(m));
    at = __shfl_sync(m, at, __ffs(m) - 1);
    q.at(side, at + before) = (u16)z;
}

constexpr int kMsRows = 32;           // rows searched together: one bit each of a value's words
constexpr u64 kMsMaxN = 18944;        // values per instance: three words of each fit an SM's shared memory
constexpr u32 kMsSmemQueueN = 13824;  // ... with both queues beside them; above, kMsNear entries of each are
constexpr u32 kMsNear = 1024;
constexpr int kMsWords = 4;           // neighbouring words of a row a lane loads at a time

// Rows of instances of at most kMsMaxN values: 32 rows of one instance at a time by one
// CTA, their breadth-first searches run together.  Value z has one word each of known,
// frontier and next bits, bit r for the group's row r; a level visits every value of the
// frontier once for all the rows that reached it in that level, where a search per row
// visits it once for each row: in a dense closure (n = 14,336, out-degree 2, 26 levels) 32
// rows meet each value in 7 levels.  A level with a wide frontier (1/kMsSweep of the
// values) sweeps the instance's edge list, every lane an edge -- each warp's frontier words
// are neighbours in shared memory, and no lane waits for another's longer list; a
// narrow one follows the queue of its values (its edge ranges and edges are a chain of L2
// round trips: with 1/8, 1/16, 1/32 and 1/64 of the values as the line between the two, a wave
// of 64 graphs ran its fixed point in 7.13, 6.98, 6.91 and 6.80 ms, and always queueing took
// 11.5).  Bound by instruction issue and shared-memory conflicts of the random known / next
// words.  Measured against one warp or CTA per row: n = 16,384, out-degree 2, 3.52 -> 0.97 ms;
// n = 2,000, 0.24 -> 0.09 ms; the wave's searches 10.0 -> 4.9 ms.
// A narrow level costs one L2 round trip (DenseRec) and two barriers: with edge range, edges and
// queue each read from L2, and a place in the queue taken for each edge, it took 2.9 us, 2.0 now (n =
// 16,384, out-degree 1.1, 152 levels:
// 1.74 -> 1.21 ms).  Where searches are short, the rows' matrix words bound it: a lane takes neighbouring
// words of its row (they share a sector), and a word with no new tuples is not written (n = 16,384,
// out-degree 0.3: 232 -> 153 us; 2.0: 820 -> 779).
// Dynamic shared memory: 3 * nmax u32, then the queues: 2 * (gqueue ? kMsNear : nmax) u16.
constexpr u32 kMsSweep = 64;
template <int T>
__global__ void __launch_bounds__(T) dense_ms_kernel(DenseArgs a, u32 nmax, u16* __restrict__ gqueue,
                                                     const DenseChunk* __restrict__ chunks, u64 n_chunks,
                                                     u64* __restrict__ chunk_ctr)
{
    extern __shared__ u32 dsm[];
    u32* known = dsm;
    u32* front = dsm + nmax;
    u32* next = dsm + 2 * (u64)nmax;
    const MsQueue queue{(u16*)(dsm + 3 * (u64)nmax), gqueue + (gqueue ? (u64)blockIdx.x * 2 * nmax : 0),
                        gqueue ? kMsNear : nmax, nmax};
    __shared__ u64 s_chunk;
    __shared__ u32 s_qn[2];
    __shared__ u32 s_lvl[kDenseLevels];   // a chunk's counts stay below 32 * kMsMaxN
    __shared__ u32 s_row[kMsRows];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    u64 relax = 0;
    for (;;) {
        if (threadIdx.x == 0) {
            s_chunk = atomicAdd((unsigned long long*)chunk_ctr, 1ull);
            s_qn[0] = s_qn[1] = 0;
        }
        for (int i = threadIdx.x; i < kDenseLevels; i += T) s_lvl[i] = 0;
        if (threadIdx.x < kMsRows) s_row[threadIdx.x] = 0;
        __syncthreads();
        const u64 c = s_chunk;
        if (c >= n_chunks) break;
        const DenseChunk ch = chunks[c];
        const DenseInst d = a.inst[ch.inst];
        const u32 W = (u32)d.words;
        const u64 w0 = d.word_off + (ch.first_row - d.base) * d.words;
        u32* krow = a.known + w0 + (u64)lane * d.words;      // lane r: row r of the group
        const u32* drow = a.delta0 + w0 + (u64)lane * d.words;
        const bool own = lane < (int)ch.count;
        const u32 n = (u32)d.n;
        const u64 e0 = a.s_csr[d.base], e1 = a.s_csr[min(d.base + d.n, a.rows)];   // the instance's edges
        for (u32 w0 = warp * kMsWords; w0 < W; w0 += kMsWords * T / 32) {
            u32 kw[kMsWords], fw[kMsWords];   // the rows' words, in flight together
#pragma unroll
            for (int u = 0; u < kMsWords; u++) {
                const u32 w = w0 + u;
                kw[u] = own && w < W ? krow[w] : 0u;
                fw[u] = drow != krow && own && w < W ? drow[w] : kw[u];
            }
#pragma unroll
            for (int u = 0; u < kMsWords; u++) {
                const u32 w = w0 + u;
                if (w >= W) break;   // uniform
                const u32 k = warp_transpose32(kw[u]), f = drow == krow ? k : warp_transpose32(fw[u]);
                const u32 z = w * 32 + lane;
                known[z] = k;
                front[z] = f;
                next[z] = 0;
                if (f) queue_push(queue, 0, &s_qn[0], z);
                if (z < n) relax += row_edges(a, d.base + z) * (u64)(long long)(__popc(f) - __popc(k));
            }
        }
        __syncthreads();
        u32 cur = 0, qn = s_qn[0];
        bool queued = true;   // queue `cur` lists the frontier's values
        for (u64 level = 0; qn; level++) {
            u32 cnt = 0;
            if (qn >= n / kMsSweep) {
                queued = false;
                for (u64 j = (e0 & ~3ull) + 4 * threadIdx.x; j < e1; j += 4 * T) {
                    u32 edge[4];
                    *(uint4*)edge = *(const uint4*)(a.s_edge + j);
                    if (j < e0 || j + 4 > e1) {   // another instance's edges
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            if (j + k < e0 || j + k >= e1) edge[k] = kNoEdge;
                    }
                    u32 fr[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) fr[k] = front[edge[k] >> 16];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        if (!fr[k]) continue;
                        const u32 z = edge[k] & 0xffffu;
                        const u32 nb = fr[k] & ~known[z];
                        if (nb) atomicOr(&next[z], nb);
                    }
                }
                __syncthreads();
                u32 some = 0;   // values of the new frontier
                for (u32 z = 4 * threadIdx.x; z < W * 32; z += 4 * T) {
                    const uint4 f = *(const uint4*)(next + z);
                    *(uint4*)(front + z) = f;
                    if (!(f.x | f.y | f.z | f.w)) continue;
                    *(uint4*)(next + z) = make_uint4(0, 0, 0, 0);
                    uint4 k = *(const uint4*)(known + z);
                    k.x |= f.x;
                    k.y |= f.y;
                    k.z |= f.z;
                    k.w |= f.w;
                    *(uint4*)(known + z) = k;
                    cnt += __popc(f.x) + __popc(f.y) + __popc(f.z) + __popc(f.w);
                    some += (f.x != 0) + (f.y != 0) + (f.z != 0) + (f.w != 0);
                }
                some = __reduce_add_sync(0xffffffffu, some);
                if (lane == 0 && some) atomicAdd(&s_qn[cur ^ 1], some);
            } else {
                if (!queued) {   // a sweep counted the frontier's values: list them
                    __syncthreads();   // every thread has read the count
                    if (threadIdx.x == 0) s_qn[cur] = 0;
                    __syncthreads();
                    for (u32 z = threadIdx.x; z < W * 32; z += T)
                        if (front[z]) queue_push(queue, cur, &s_qn[cur], z);
                    queued = true;
                    __syncthreads();
                }
                for (u32 i = threadIdx.x; i < qn; i += T) {
                    const u32 y = queue.at(cur, i);
                    const u32 f = front[y];
                    front[y] = 0;
                    const uint4 r = d.base + y < a.rows ? a.s_rec[d.base + y] : make_uint4(0, 0, 0, 0);
                    const u32 c = r.x & 0xffffu;
                    if (c != kRecMany) {
                        // all edges' words, then their ORs, then one place in the queue for the values first reached
                        const u32 w[4] = {r.x, r.y, r.z, r.w};
                        u32 nb[kRecEdges], first = 0;
#pragma unroll
                        for (u32 k = 0; k < kRecEdges; k++)
                            nb[k] = k < c ? f & ~known[(w[(k + 1) >> 1] >> (((k + 1) & 1) * 16)) & 0xffffu] : 0u;
#pragma unroll
                        for (u32 k = 0; k < kRecEdges; k++)
                            if (nb[k] && atomicOr(&next[(w[(k + 1) >> 1] >> (((k + 1) & 1) * 16)) & 0xffffu], nb[k]) == 0)
                                first |= 1u << k;
                        if (first) {
                            u32 at = atomicAdd(&s_qn[cur ^ 1], (u32)__popc(first));
#pragma unroll
                            for (u32 k = 0; k < kRecEdges; k++)
                                if (first >> k & 1)
                                    queue.at(cur ^ 1, at++) = (u16)(w[(k + 1) >> 1] >> (((k + 1) & 1) * 16));
                        }
                    } else {
                        const u64 s = a.s_csr[d.base + y], e = a.s_csr[d.base + y + 1];
                        for (u64 j = s; j < e; j++) {
                            const u32 z = a.s_edge[j] & 0xffffu;
                            const u32 nb = f & ~known[z];
                            if (nb && atomicOr(&next[z], nb) == 0) queue_push(queue, cur ^ 1, &s_qn[cur ^ 1], z);
                        }
                    }
                }
                __syncthreads();
                const u32 qnew = s_qn[cur ^ 1];
                for (u32 i = threadIdx.x; i < qnew; i += T) {
                    const u32 z = queue.at(cur ^ 1, i);
                    const u32 f = next[z];
                    next[z] = 0;
                    known[z] |= f;
                    front[z] = f;
                    cnt += __popc(f);
                }
            }
            cnt = __reduce_add_sync(0xffffffffu, cnt);
            if (lane == 0 && cnt) {
                if (level < (u64)kDenseLevels) {
                    atomicAdd(&s_lvl[level], cnt);
                } else if (level < a.level_cap) {
                    atomicAdd((unsigned long long*)&a.level_total[level], (unsigned long long)cnt);
                    if (a.inst_level)
                        atomicAdd((unsigned long long*)&a.inst_level[level * a.n_inst + ch.inst],
                                  (unsigned long long)cnt);
                } else {
                    atomicOr(a.flags, kDenseFlagLevels);
                }
            }
            if (threadIdx.x == 0) s_qn[cur] = 0;
            __syncthreads();
            cur ^= 1;
            qn = s_qn[cur];
        }
        // the rows' new tuples replace their known bits in global memory
        u32 rcnt = 0;
        for (u32 w0 = warp * kMsWords; w0 < W; w0 += kMsWords * T / 32) {
            u32 old[kMsWords];
#pragma unroll
            for (int u = 0; u < kMsWords; u++) {
                const u32 w = w0 + u;
                old[u] = own && w < W ? krow[w] : 0u;
            }
#pragma unroll
            for (int u = 0; u < kMsWords; u++) {
                const u32 w = w0 + u;
                if (w >= W) break;
                const u32 z = w * 32 + lane;
                const u32 kz = known[z];
                const u32 nw = warp_transpose32(kz) & ~old[u];
                if (z < n) relax += row_edges(a, d.base + z) * (u64)__popc(kz);
                if (own && nw != old[u]) krow[w] = nw;
                if (own) rcnt += __popc(nw);
            }
        }
        if (rcnt) atomicAdd(&s_row[lane], rcnt);
        __syncthreads();
        if (threadIdx.x < ch.count) a.row_new[ch.first_row + threadIdx.x] = s_row[threadIdx.x];
        for (int i = threadIdx.x; i < kDenseLevels; i += T) {
            const u32 v = s_lvl[i];
            if (!v) continue;
            if ((u64)i < a.level_cap) {
                atomicAdd((unsigned long long*)&a.level_total[i], (unsigned long long)v);
                if (a.inst_level)
                    atomicAdd((unsigned long long*)&a.inst_level[(u64)i * a.n_inst + ch.inst], (unsigned long long)v);
            } else {
                atomicOr(a.flags, kDenseFlagLevels);
            }
        }
        __syncthreads();
    }
    for (int o = 16; o > 0; o >>= 1) relax += __shfl_xor_sync(0xffffffffu, relax, o);
    if (lane == 0 && relax) atomicAdd((unsigned long long*)&a.counters[1], (unsigned long long)relax);
}

// New tuples of each row into the log: row by row (values ascending), within a
// row by column-0 value ascending; key (z, x), id tag_word | (id_base + position).
// One warp per row, 32 words at a time (emit_words): consecutive lanes write consecutive
// rows of the log (coalesced).
__global__ void __launch_bounds__(kThreads) dense_emit_kernel(DenseArgs a, const u64* __restrict__ row_off,
                                                              u64* __restrict__ keys_out, u64* __restrict__ ids_out,
                                                              u64 tag_word, u64 id_base)
{
    const int lane = threadIdx.x & 31;
    const u64 warps = (u64)gridDim.x * (kThreads / 32);
    for (u64 row = (u64)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); row < a.rows; row += warps) {
        if (a.row_new[row] == 0) continue;   // uniform per warp
        const DenseInst d = a.inst[dense_instance(a, row)];
        const u32* nrow = a.known + d.word_off + (row - d.base) * d.words;
        const u32 W = (u32)d.words;
        u64 pos = row_off[row];
        for (u32 g = 0; g < W; g += 32) {
            const u32 word = (g + lane < W) ? nrow[g + lane] : 0u;
            pos += emit_words(word, [&](u32 t, u32 bit) {
                keys_out[pos + t] = ((d.base + (u64)g * 32 + bit) << a.bits) | row;
                ids_out[pos + t] = tag_word | (id_base + pos + t);
            });
        }
    }
}

}  // namespace ra
