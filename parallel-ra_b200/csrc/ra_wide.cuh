// Wide tuples: programs whose tuples do not pack into one 63-bit key (arity x
// value bits > 63, e.g. the slog-generated analyses whose columns hold intern
// ids) or whose join keys exceed the CSR index.  A relation version is an array
// of rows of arity + 1 u64 (data columns, then the id) in trie order --
// lexicographic over all columns, the order in which the reference's tries
// enumerate tuples (src/relation/shmap_relation_exp.cpp:77-112).
//
// Operations are index sorts with a row comparator (bitonic networks over rows held in
// shared memory; merge passes by binary-searched ranks for larger inputs), hash
// grouping of candidates, prefix binary
// searches (join ranges on the first jcc columns; membership on the data
// columns), and rank merges of sorted arrays.  All integer; with the small deltas
// of the generated analyses, latency-bound.
#pragma once

#include "ra_iter.cuh"

namespace ra {

constexpr int kWideMaxCols = 64;     // arity + 1 columns at most
constexpr int kWideMaxSegs = 32;     // rules writing one relation within an SCC

// Lexicographic compare of two rows over their first `ncmp` columns: -1, 0, 1.  Four
// columns at a time: their loads overlap.
__device__ __forceinline__ int wide_cmp(const u64* __restrict__ a, const u64* __restrict__ b, int ncmp)
{
    int c = 0;
    for (; c + 4 <= ncmp; c += 4) {
        u64 x[4], y[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            x[k] = a[c + k];
            y[k] = b[c + k];
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (x[k] != y[k]) return x[k] < y[k] ? -1 : 1;
    }
    for (; c < ncmp; c++) {
        const u64 x = a[c], y = b[c];
        if (x != y) return x < y ? -1 : 1;
    }
    return 0;
}

// Strict total order on row indices: the first `ncmp` columns, then the index.
__device__ __forceinline__ bool wide_before(const u64* __restrict__ rows, int W, int ncmp, u64 i, u64 j)
{
    const int c = wide_cmp(rows + i * W, rows + j * W, ncmp);
    return c < 0 || (c == 0 && i < j);
}

// Sort of a block's rows, held in shared memory column after column (s[c * n + i]), by
// (first ncmp columns, index) into idx; n <= blockDim.x = kWideBlockSort, the whole block calls it.
// The rows of the generated analyses agree on many leading columns and differ by small
// offsets in the others, so the columns in which some rows differ are packed, each in the bits
// of its range, into one 64-bit key as far as they go: a comparison is that key's, then the
// remaining columns', then the index.  The bitonic network keeps an element per thread,
// exchanges over less than a warp by shuffle and the others through shared memory: 10 block
// barriers of 45 stages for 512 rows.  Bound by those stages' chain.
constexpr u32 kWideBlockSort = 1024;     // rows a block sorts in shared memory
constexpr u64 kWideSmem = 160u << 10;    // shared memory for its rows
struct WideSortSmem {
    u64 lo[kWideMaxCols], hi[kWideMaxCols];   // least and largest value of a column
    u64 key[kWideBlockSort];                  // exchange of the network's elements
    u32 idx[kWideBlockSort];
    unsigned char cols[kWideMaxCols];         // columns with more than one value
    unsigned char bits[kWideMaxCols];         // bits of their ranges
    int ncols;
};

__device__ __forceinline__ void wide_block_sort(WideSortSmem& S, const u64* s, u32 n, int ncmp)
{
    const u32 t = threadIdx.x, lane = t & 31;
    for (int c = t >> 5; c < ncmp; c += blockDim.x >> 5) {   // a warp per column
        u64 lo = ~0ull, hi = 0;
        for (u32 i = lane; i < n; i += 32) {
            const u64 v = s[(u32)c * n + i];
            lo = min(lo, v);
            hi = max(hi, v);
        }
        for (int d = 16; d > 0; d >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, d));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d));
        }
        if (lane == 0) {
            S.lo[c] = lo;
            S.hi[c] = hi;
        }
    }
    __syncthreads();
    if (t < 32) {   // the columns that vary, in order
        int m = 0;
        for (int c0 = 0; c0 < ncmp; c0 += 32) {
            const int c = c0 + (int)lane;
            const bool vary = c < ncmp && S.lo[c] != S.hi[c];
            const u32 mask = __ballot_sync(0xffffffffu, vary);
            if (vary) {
                const int q = m + __popc(mask & lanemask_lt());
                S.cols[q] = (unsigned char)c;
                S.bits[q] = (unsigned char)(64 - __clzll((long long)(S.hi[c] - S.lo[c])));
            }
            m += __popc(mask);
        }
        if (lane == 0) S.ncols = m;
    }
    __syncthreads();
    u32 P = 32;
    while (P < n) P <<= 1;
    const int ncols = S.ncols;
    int nkey = 0;   // columns the key holds
    u64 key = 0;
    u32 id = t;     // from n on: padding, last
    for (int used = 0; nkey < ncols && used + S.bits[nkey] <= 64; nkey++) {
        const int c = S.cols[nkey];
        used += S.bits[nkey];
        if (t < n) key |= (s[(u32)c * n + t] - S.lo[c]) << (64 - used);
    }
    auto before = [&](u64 ka, u32 a, u64 kb, u32 b) {
        if (a >= n || b >= n) return a < b;   // padding last
        if (ka != kb) return ka < kb;
        for (int q = nkey; q < ncols; q++) {
            const u32 at = S.cols[q] * n;
            const u64 x = s[at + a], y = s[at + b];
            if (x != y) return x < y;
        }
        return a < b;
    };
    for (u32 k = 2; k <= P; k <<= 1) {
        for (u32 j = k >> 1; j > 0; j >>= 1) {
            u64 pk = 0;
            u32 pi = 0;
            if (j >= 32) {
                if (t < P) {
                    S.key[t] = key;
                    S.idx[t] = id;
                }
                __syncthreads();
                if (t < P) {
                    pk = S.key[t ^ j];
                    pi = S.idx[t ^ j];
                }
                __syncthreads();
            } else if (t < P) {   // whole warps
                pk = __shfl_xor_sync(0xffffffffu, key, j);
                pi = __shfl_xor_sync(0xffffffffu, id, j);
            }
            if (t < P) {
                const bool keep_least = ((t & j) == 0) == ((t & k) == 0);
                if (before(pk, pi, key, id) == keep_least) {
                    key = pk;
                    id = pi;
                }
            }
        }
    }
    __syncthreads();
    if (t < n) S.idx[t] = id;
    __syncthreads();
}

// Rows of a tile of the larger sorts: a tile's rows fit kWideSmem.
__host__ __device__ __forceinline__ u32 wide_tile_rows(int W)
{
    return W <= 20 ? kWideBlockSort : W <= 40 ? kWideBlockSort / 2 : kWideBlockSort / 4;
}
static_assert(20 * kWideBlockSort * 8 <= kWideSmem && kWideMaxCols * (kWideBlockSort / 4) * 8 <= kWideSmem,
              "a tile's rows fit");

// Tile sort: indices [b * tile, ...) of `n` rows, block b.  Dynamic shared memory: the rows of
// a tile.  1,024 rows of 10 columns took 144 us with 256 threads and two cached columns, 25 us now.
__global__ void __launch_bounds__(kWideBlockSort) wide_tile_sort_kernel(const u64* __restrict__ rows, int W, int ncmp,
                                                                        u64 n, u32 tile, u64* __restrict__ idx)
{
    extern __shared__ u64 w_cols[];
    __shared__ WideSortSmem S;
    const u64 base = (u64)blockIdx.x * tile;
    const u32 m = (u32)min((u64)tile, n - base);
    const u64* r0 = rows + base * (u64)W;
    for (u32 e = threadIdx.x; e < m * (u32)W; e += blockDim.x) {
        const u32 i = e / (u32)W, c = e - i * (u32)W;
        w_cols[c * m + i] = r0[e];
    }
    __syncthreads();
    wide_block_sort(S, w_cols, m, ncmp);
    if (threadIdx.x < m) idx[base + threadIdx.x] = base + S.idx[threadIdx.x];
}

// Exclusive scan of at most kThreads * kWideScanPer values by one block; the
// total into *total (device memory: no host round trip).
constexpr int kWideScanPer = 16;

// The scan itself: get(i) for i < n, put(i, exclusive sum); returns the total.  A thread takes
// as few consecutive values as cover n (each is a dependent read).
template <typename Get, typename Put>
__device__ __forceinline__ u64 wide_block_scan(u64 n, u64* sm, Get get, Put put)
{
    const u64 per = (n + kThreads - 1) / kThreads, b = min(n, threadIdx.x * per), e = min(n, b + per);
    u64 loc = 0;
    for (u64 i = b; i < e; i++) loc += get(i);
    u64 agg;
    u64 ex = block_exclusive_scan(loc, sm, &agg);
    for (u64 i = b; i < e; i++) {
        put(i, ex);
        if (i + 1 < e) ex += get(i);
    }
    return agg;
}

template <typename T>
__global__ void __launch_bounds__(kThreads) wide_scan_small_kernel(const T* __restrict__ in, u64 n,
                                                                   u64* __restrict__ out, u64* __restrict__ total)
{
    __shared__ u64 sm[kWarps + 1];
    const u64 agg = wide_block_scan(n, sm, [&](u64 i) { return (u64)in[i]; }, [&](u64 i, u64 v) { out[i] = v; });
    if (threadIdx.x == 0) *total = agg;
}

// One merge pass: sorted runs of length L in `in`, pairs merged into `out`.  An
// element's output position is its offset in its run plus its rank in the
// partner run (the order is strict, so the ranks of both runs interleave exactly).
__global__ void __launch_bounds__(kThreads) wide_merge_pass_kernel(const u64* __restrict__ rows, int W, int ncmp,
                                                                   u64 n, u64 L, const u64* __restrict__ in,
                                                                   u64* __restrict__ out)
{
    for (u64 p = (u64)blockIdx.x * kThreads + threadIdx.x; p < n; p += (u64)gridDim.x * kThreads) {
        const u64 start = (p / (2 * L)) * 2 * L;
        const u64 mid = min(start + L, n), end = min(start + 2 * L, n);
        const u64 v = in[p];
        const bool left = p < mid;
        u64 a = left ? mid : start, b = left ? end : mid;
        const u64 lo = a;
        while (a < b) {
            const u64 m = (a + b) >> 1;
            if (wide_before(rows, W, ncmp, in[m], v)) a = m + 1;
            else b = m;
        }
        out[start + (p - (left ? start : mid)) + (a - lo)] = v;
    }
}

// out row k = rows[idx[k]] (W columns), one thread per column value.
__global__ void __launch_bounds__(kThreads) wide_gather_kernel(const u64* __restrict__ rows, int W,
                                                               const u64* __restrict__ idx, u64 n,
                                                               u64* __restrict__ out)
{
    const u64 total = n * (u64)W;
    for (u64 e = (u64)blockIdx.x * kThreads + threadIdx.x; e < total; e += (u64)gridDim.x * kThreads) {
        const u64 k = e / (u64)W, c = e - k * (u64)W;
        out[e] = rows[idx[k] * (u64)W + c];
    }
}

// First row of `sorted` (n rows of Ws columns) whose first `ncmp` columns are not
// below `key`'s.
__device__ __forceinline__ u64 wide_lower_bound(const u64* __restrict__ sorted, int Ws, u64 n,
                                                const u64* __restrict__ key, int ncmp)
{
    u64 a = 0, b = n;
    while (a < b) {
        const u64 m = (a + b) >> 1;
        if (wide_cmp(sorted + m * (u64)Ws, key, ncmp) < 0) a = m + 1;
        else b = m;
    }
    return a;
}

__device__ __forceinline__ u64 wide_upper_bound(const u64* __restrict__ sorted, int Ws, u64 n,
                                                const u64* __restrict__ key, int ncmp)
{
    u64 a = 0, b = n;
    while (a < b) {
        const u64 m = (a + b) >> 1;
        if (wide_cmp(sorted + m * (u64)Ws, key, ncmp) <= 0) a = m + 1;
        else b = m;
    }
    return a;
}

// wide_lower_bound / wide_upper_bound by a warp: 32 rows of the range are compared at a time,
// so 2.8 million rows take 5 rounds where one thread takes 22 dependent reads.  Worth its
// 30-fold reads while the searches do not fill the GPU (kWideWarpSearch).
template <bool kUpper>
__device__ __forceinline__ u64 wide_bound_warp(const u64* __restrict__ sorted, int Ws, u64 n,
                                               const u64* __restrict__ key, int ncmp)
{
    const u32 lane = threadIdx.x & 31;
    u64 lo = 0, hi = n;   // the bound is in [lo, hi]
    while (hi - lo > 32) {
        const u64 at = lo + (hi - lo) * (lane + 1) / 33;   // ascending, below hi
        const int c = wide_cmp(sorted + at * (u64)Ws, key, ncmp);
        const u32 below = __popc(__ballot_sync(0xffffffffu, kUpper ? c <= 0 : c < 0));
        const u64 last = __shfl_sync(0xffffffffu, at, below ? below - 1 : 0);
        const u64 next = __shfl_sync(0xffffffffu, at, below & 31);
        if (below) lo = last + 1;
        if (below < 32) hi = next;
    }
    bool in = lo + lane < hi;
    if (in) {
        const int c = wide_cmp(sorted + (lo + lane) * (u64)Ws, key, ncmp);
        in = kUpper ? c <= 0 : c < 0;
    }
    return lo + __popc(__ballot_sync(0xffffffffu, in));
}
// Searches of a launch up to which a warp each is faster than a thread each (a GPU of 148 SMs
// holds 9,472 warps).
constexpr u64 kWideWarpSearch = 16384;

// Does `sorted` hold a row whose first `ncmp` columns equal `key`'s
// (relation::find_in_full / find_in_delta, balanced_hash_relation.cpp:1015-1035)?
template <bool kWarp>
__device__ __forceinline__ bool wide_has_prefix(const u64* __restrict__ sorted, int Ws, u64 n,
                                                const u64* __restrict__ key, int ncmp)
{
    if (!n) return false;
    const u64 i = kWarp ? wide_bound_warp<false>(sorted, Ws, n, key, ncmp) : wide_lower_bound(sorted, Ws, n, key, ncmp);
    return i < n && wide_cmp(sorted + i * (u64)Ws, key, ncmp) == 0;
}

// Output column j of a rule = column src[j] of the concatenation
// (in0 row ++ in1 row[jcc..]) for a join (as_all_to_allv_{left,right}_join_buffer_helper,
// shmap_relation_exp.cpp:335-349, 403-417), or of the input row for a copy.
struct WideProj {
    int n;        // output columns
    int left;     // join: the outer rows are in0's (LEFT) or in1's (RIGHT)
    int W0, W1;   // join: in0 and in1 row widths (arity + 1)
    int jcc;
    int src[kWideMaxCols];
};

// Up to kWideMaxSegs segments of a relation's candidate buffer, one per rule
// writing it, with the id base of each (the tag's intern counter when the rule runs).
struct WideSegs {
    int n;
    u64 start[kWideMaxSegs + 1];   // candidate positions; start[n] = total
    u64 win_base[kWideMaxSegs];    // winners before the segment
    u64 id_base[kWideMaxSegs];     // (tag << 46) | counter of the segment's first winner
};

// New tuples into newt rows (arity + 1 columns) in position order; a join or
// copy winner gets the next id of its rule's segment, an acopy candidate
// carries its own last column.
__global__ void __launch_bounds__(kThreads) wide_newt_kernel(const u64* __restrict__ cand, int cw, u64 n,
                                                             const u32* __restrict__ win, const u64* __restrict__ wpos,
                                                             WideSegs sg, int W, u64* __restrict__ newt)
{
    for (u64 c = (u64)blockIdx.x * kThreads + threadIdx.x; c < n; c += (u64)gridDim.x * kThreads) {
        if (!win[c]) continue;
        int q = 0;
        while (q + 1 < sg.n && c >= sg.start[q + 1]) q++;
        const u64 at = wpos[c];
        const u64* src = cand + c * (u64)cw;
        u64* dst = newt + at * (u64)W;
        for (int j = 0; j < cw; j++) dst[j] = src[j];
        if (cw < W) dst[W - 1] = sg.id_base[q] + (at - sg.win_base[q]);
    }
}

// Rows equal (all columns) to their predecessor, in a sorted array.
__global__ void __launch_bounds__(kThreads) wide_dup_kernel(const u64* __restrict__ rows, int W, u64 n,
                                                            u32* __restrict__ keep, u32* __restrict__ any_dup)
{
    for (u64 k = (u64)blockIdx.x * kThreads + threadIdx.x; k < n; k += (u64)gridDim.x * kThreads) {
        const bool dup = k > 0 && wide_cmp(rows + (k - 1) * (u64)W, rows + k * (u64)W, W) == 0;
        keep[k] = dup ? 0u : 1u;
        if (dup) atomicOr(any_dup, 1u);
    }
}

// Kept rows to their scanned positions.
__global__ void __launch_bounds__(kThreads) wide_compact_kernel(const u64* __restrict__ rows, int W, u64 n,
                                                                const u32* __restrict__ keep,
                                                                const u64* __restrict__ pos, u64* __restrict__ out)
{
    for (u64 k = (u64)blockIdx.x * kThreads + threadIdx.x; k < n; k += (u64)gridDim.x * kThreads) {
        if (!keep[k]) continue;
        const u64* src = rows + k * (u64)W;
        u64* dst = out + pos[k] * (u64)W;
        for (int j = 0; j < W; j++) dst[j] = src[j];
    }
}

// Exclusive-scanned winner counts at each segment's start (the total past the
// end), i.e. the winners before each rule's candidates.
__global__ void wide_pick_kernel(const u64* __restrict__ scanned, u64 n, const u64* __restrict__ total,
                                 WideSegs sg, u64* __restrict__ out)
{
    const int q = threadIdx.x;
    if (q <= sg.n) out[q] = sg.start[q] < n ? scanned[sg.start[q]] : *total;
}

// ---------------------------------------------------------------------------
// Batched launches: one kernel per phase of an iteration for all of its small
// rules or relations (one block each, or one flattened index space), with the
// work list passed as a kernel parameter (no host-to-device copy).  Most
// iterations of a generated analysis move a few hundred tuples, so launches,
// not bytes, set their cost.
// ---------------------------------------------------------------------------
constexpr int kWideJobs = 64;          // work items per batched launch
constexpr u32 kWideBlockScan = kThreads * kWideScanPer;   // rows a block counts and scans
constexpr int kWideWideBlock = 1024;   // threads of the per-relation sort kernels (no block scan)

// 64-bit hash of a row's first n columns (grouping key of the winner sorts).
__device__ __forceinline__ u64 wide_row_hash(const u64* __restrict__ row, int n)
{
    u64 h = 0x243f6a8885a308d3ull;
    for (int c = 0; c < n; c++) h = mix64(h ^ (row[c] + 0x9e3779b97f4a7c15ull * (u64)(c + 1)));
    return h;
}

// Phase 1a: every job's rows in one flattened index space: a join's range of inner rows
// sharing the outer row's first jcc columns (trie order; all of them when jcc is 0 --
// parallel_join::local_join, src/RA/parallel_join.cpp:157-230), or a copy_filter's pass
// flag.  kWarp: a warp per row.
struct WideCountJob {
    const u64* outer;
    const u64* inner;
    u64 no, ni, first;       // first flattened index of this job
    u64* lo;       // join: first match per outer row
    u64* cnt;      // join: matches per outer row
    u64* off;      // join: scanned counts; filter: scanned flags
    u32* keep;     // filter: pass flags
    u64* total;
    int Wo, Wi, jcc, pred;   // pred < 0: a join
};
struct WideCountBatch {
    int n;
    u64 total;
    WideCountJob job[kWideJobs];
};

// The job of flattened index g: the last whose first index is at most g.
template <typename Batch>
__device__ __forceinline__ int wide_job_of(const Batch& b, u64 g)
{
    int r = 0, hi = b.n;
    while (hi - r > 1) {
        const int m = (r + hi) >> 1;
        if (b.job[m].first <= g) r = m;
        else hi = m;
    }
    return r;
}

template <bool kWarp>
__global__ void __launch_bounds__(kThreads) wide_range_batch_kernel(const __grid_constant__ WideCountBatch b)
{
    const u64 id = (u64)blockIdx.x * kThreads + threadIdx.x;
    const u64 stride = (u64)gridDim.x * kThreads >> (kWarp ? 5 : 0);
    for (u64 g = kWarp ? id >> 5 : id; g < b.total; g += stride) {
        const WideCountJob& j = b.job[wide_job_of(b, g)];
        const u64 o = g - j.first;
        const u64* row = j.outer + o * (u64)j.Wo;
        if (j.pred >= 0) {
            j.keep[o] = eval_pred(j.pred, row[0], j.Wo > 1 ? row[1] : 0) ? 1u : 0u;
            continue;
        }
        u64 a = 0, e = j.ni;
        if (j.jcc && kWarp) {
            a = wide_bound_warp<false>(j.inner, j.Wi, j.ni, row, j.jcc);
            e = a + wide_bound_warp<true>(j.inner + a * (u64)j.Wi, j.Wi, j.ni - a, row, j.jcc);
        } else if (j.jcc) {
            a = wide_lower_bound(j.inner, j.Wi, j.ni, row, j.jcc);
            e = wide_upper_bound(j.inner, j.Wi, j.ni, row, j.jcc);
        }
        j.lo[o] = a;
        j.cnt[o] = e - a;
    }
}

// Phase 1b: per job of at most kWideBlockScan rows, one block scans the counts (or flags);
// the total into *total.
__global__ void __launch_bounds__(kThreads) wide_count_scan_kernel(const __grid_constant__ WideCountBatch b)
{
    __shared__ u64 sm[kWarps + 1];
    const WideCountJob& j = b.job[blockIdx.x];
    if (j.no > kWideBlockScan) return;   // scanned by the whole grid
    const u64 agg = wide_block_scan(j.no, sm, [&](u64 o) { return j.pred < 0 ? j.cnt[o] : (u64)j.keep[o]; },
                                    [&](u64 o, u64 v) { j.off[o] = v; });
    if (threadIdx.x == 0) *j.total = agg;
}

// Phase 2: every rule's candidates in one flattened index space.
struct WideExpandJob {
    const u64* outer;   // join: outer rows; copy: input rows
    const u64* inner;
    const u64* lo;
    const u64* off;     // join: scanned counts; filter: scanned pass flags (null for a plain copy)
    u64* dst;
    u64 no;
    u64 first;          // first flattened index of this job
    int Wi;             // copy: input width
    int n, left, W0, W1, jcc, kind;   // kind 0: join, 1: copy
    unsigned char src[kWideMaxCols];
};
struct WideExpandBatch {
    int n;
    u64 total;
    WideExpandJob job[kWideJobs];
};

__global__ void __launch_bounds__(kThreads) wide_expand_batch_kernel(const __grid_constant__ WideExpandBatch b)
{
    for (u64 g = (u64)blockIdx.x * kThreads + threadIdx.x; g < b.total; g += (u64)gridDim.x * kThreads) {
        const WideExpandJob& j = b.job[wide_job_of(b, g)];
        const u64 c = g - j.first;
        u64* dst = j.dst + c * (u64)j.n;
        if (j.kind == 0) {
            u64 a = 0, e = j.no;
            while (a < e) {
                const u64 m = (a + e) >> 1;
                if (j.off[m] <= c) a = m + 1;
                else e = m;
            }
            const u64 o = a - 1, u = j.lo[o] + (c - j.off[o]);
            const int Wo = j.left ? j.W0 : j.W1, Wi = j.left ? j.W1 : j.W0;
            const u64* ro = j.outer + o * (u64)Wo;
            const u64* ri = j.inner + u * (u64)Wi;
            const u64* r0 = j.left ? ro : ri;
            const u64* r1 = j.left ? ri : ro;
            for (int k = 0; k < j.n; k++) {
                const int x = j.src[k];
                dst[k] = x < j.W0 ? r0[x] : r1[j.jcc + (x - j.W0)];
            }
        } else {
            u64 rin = c;
            if (j.off) {   // the c-th kept row: the last row whose scanned flag is <= c
                u64 a = 0, e = j.no;
                while (a < e) {
                    const u64 m = (a + e) >> 1;
                    if (j.off[m] <= c) a = m + 1;
                    else e = m;
                }
                rin = a - 1;
            }
            const u64* row = j.outer + rin * (u64)j.Wi;
            for (int k = 0; k < j.n; k++) dst[k] = row[j.src[k]];
        }
    }
}

// Phase 3a: flags the first candidate of each group of equal ones (the group's first
// occurrence).  Per relation of at most kWideBlockSort candidates, one block puts them into
// a hash table in shared memory: a slot keeps its group's smallest position.  Grouping needs
// no order, so there is nothing to sort; rows are compared when their 64-bit hashes agree.
// Measured against sorting by hash: 12.5 -> 4.2 us per launch on cfa-4-4-64.
struct WideHeadJob {
    const u64* cand;
    u32* flag;
    u64 n;
    int cw;
};
struct WideHeadBatch {
    int n;
    WideHeadJob job[kWideJobs];
};

constexpr u32 kWideNone = 0xffffffffu;

__global__ void __launch_bounds__(kWideWideBlock) wide_heads_batch_kernel(const __grid_constant__ WideHeadBatch b)
{
    __shared__ u64 s_hash[kWideBlockSort];
    __shared__ u32 s_slot[2 * kWideBlockSort];
    const WideHeadJob& j = b.job[blockIdx.x];
    u32 slots = 64;
    while (slots < 2 * (u32)j.n) slots <<= 1;
    for (u32 t = threadIdx.x; t < slots; t += blockDim.x) s_slot[t] = kWideNone;
    for (u32 c = threadIdx.x; c < j.n; c += blockDim.x) s_hash[c] = wide_row_hash(j.cand + c * (u64)j.cw, j.cw);
    __syncthreads();
    const u32 c = threadIdx.x;   // kWideWideBlock == kWideBlockSort: one candidate per thread
    u32 at = 0;
    if (c < j.n) {
        const u64 h = s_hash[c];
        for (at = (u32)h & (slots - 1);; at = (at + 1) & (slots - 1)) {   // at least half the slots stay empty
            const u32 cur = atomicCAS(&s_slot[at], kWideNone, c);
            if (cur == kWideNone) break;
            if (s_hash[cur] == h && wide_cmp(j.cand + cur * (u64)j.cw, j.cand + c * (u64)j.cw, j.cw) == 0) {
                atomicMin(&s_slot[at], c);   // still one of the group
                break;
            }
        }
    }
    __syncthreads();
    if (c < j.n) j.flag[c] = s_slot[at] == c ? 1u : 0u;
}
static_assert(kWideWideBlock == (int)kWideBlockSort, "a thread per candidate");

// The same for a larger relation, over the whole grid: hashes (and an empty table), then the
// groups, then the flags.  T: u32, or u64 where positions or slots need it.
template <typename T>
__global__ void __launch_bounds__(kThreads) wide_heads_hash_kernel(const u64* __restrict__ cand, int cw, u64 n,
                                                                   u64* __restrict__ hash, T* __restrict__ slot,
                                                                   u64 slots)
{
    for (u64 i = (u64)blockIdx.x * kThreads + threadIdx.x; i < slots; i += (u64)gridDim.x * kThreads) {
        slot[i] = (T)~0ull;
        if (i < n) hash[i] = wide_row_hash(cand + i * (u64)cw, cw);
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) wide_heads_group_kernel(const u64* __restrict__ cand, int cw, u64 n,
                                                                    const u64* __restrict__ hash,
                                                                    T* __restrict__ slot, u64 slots,
                                                                    T* __restrict__ at_out)
{
    const T none = (T)~0ull;
    for (u64 c = (u64)blockIdx.x * kThreads + threadIdx.x; c < n; c += (u64)gridDim.x * kThreads) {
        const u64 h = hash[c];
        u64 at = __umul64hi(h, slots);
        for (;; at = at + 1 == slots ? 0 : at + 1) {   // twice as many slots as candidates
            const T cur = atomicCAS(&slot[at], none, (T)c);
            if (cur == none) break;
            if (hash[cur] == h && wide_cmp(cand + cur * (u64)cw, cand + c * (u64)cw, cw) == 0) {
                atomicMin(&slot[at], (T)c);
                break;
            }
        }
        at_out[c] = (T)at;
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) wide_heads_flag_kernel(u64 n, const T* __restrict__ slot,
                                                                   const T* __restrict__ at,
                                                                   u32* __restrict__ flag)
{
    for (u64 c = (u64)blockIdx.x * kThreads + threadIdx.x; c < n; c += (u64)gridDim.x * kThreads)
        flag[c] = slot[at[c]] == (T)c ? 1u : 0u;
}

// Phase 3b: a head loses when full or delta holds its data columns (all columns
// for acopy targets); one warp (kWarp) or thread per candidate of every relation.
struct WideMemberJob {
    const u64* cand;
    const u64* full;
    const u64* delta;
    u32* flag;
    u64 n, nf, nd, first;
    int cw, W;
};
struct WideMemberBatch {
    int n;
    u64 total;
    WideMemberJob job[kWideJobs];
};

template <bool kWarp>
__global__ void __launch_bounds__(kThreads) wide_member_batch_kernel(const __grid_constant__ WideMemberBatch b)
{
    const u64 id = (u64)blockIdx.x * kThreads + threadIdx.x;
    const u64 stride = (u64)gridDim.x * kThreads >> (kWarp ? 5 : 0);
    for (u64 g = kWarp ? id >> 5 : id; g < b.total; g += stride) {
        const WideMemberJob& j = b.job[wide_job_of(b, g)];
        const u64 c = g - j.first;
        if (!j.flag[c]) continue;
        const u64* row = j.cand + c * (u64)j.cw;
        if (wide_has_prefix<kWarp>(j.full, j.W, j.nf, row, j.cw) ||
            wide_has_prefix<kWarp>(j.delta, j.W, j.nd, row, j.cw))
            j.flag[c] = 0u;
    }
}

// Phase 3c: per relation of at most kWideBlockScan candidates, one block scans
// the winner flags into positions and picks each rule segment's winners-before
// count (and the total at picks[kWideMaxSegs + 1]).
struct WideScanJob {
    const u32* flag;
    u64* pos;
    u64* picks;
    u64 n;
    int seg0, nseg;
};
struct WideScanBatch {
    int n;
    WideScanJob job[kWideJobs];
    u64 seg_start[2 * kWideJobs];
};

__global__ void __launch_bounds__(kThreads) wide_scan_pick_batch_kernel(const __grid_constant__ WideScanBatch b)
{
    __shared__ u64 sm[kWarps + 1];
    const WideScanJob& j = b.job[blockIdx.x];
    const u64 agg = wide_block_scan(j.n, sm, [&](u64 i) { return (u64)j.flag[i]; },
                                    [&](u64 i, u64 v) { j.pos[i] = v; });
    __syncthreads();   // positions visible to the picking threads
    if ((int)threadIdx.x <= j.nseg) {
        const u64 st = threadIdx.x < (u32)j.nseg ? b.seg_start[j.seg0 + threadIdx.x] : j.n;
        j.picks[threadIdx.x] = st < j.n ? j.pos[st] : agg;
    }
    if (threadIdx.x == 0) j.picks[kWideMaxSegs + 1] = agg;
}

// Phase 5: per relation of at most kWideBlockSort new tuples whose rows fit kWideSmem, one
// block collects the newt rows (ids per rule segment) in shared memory, sorts them into trie
// order there and writes them to the relation's newt.  Dynamic shared memory: the largest
// job's rows.  Measured against rows in global memory and two cached columns: 34 -> 15 us per
// launch on cfa-4-4-64 (about 480 rows of up to 24 columns), 14.5 -> 8 on worstcase-110-terms-4-m.
struct WideNewtJob {
    const u64* cand;
    const u32* flag;
    const u64* pos;
    u64* newt;
    u64 n, winners;
    int cw, W, seg0, nseg;
};
struct WideNewtBatch {
    int n;
    WideNewtJob job[kWideJobs];
    u64 seg_start[2 * kWideJobs];
    u64 win_base[2 * kWideJobs];
    u64 id_base[2 * kWideJobs];
};

__global__ void __launch_bounds__(kWideWideBlock) wide_newt_batch_kernel(const __grid_constant__ WideNewtBatch b)
{
    extern __shared__ u64 w_cols[];
    __shared__ WideSortSmem S;
    const WideNewtJob& j = b.job[blockIdx.x];
    const u32 n = (u32)j.winners, W = (u32)j.W, cw = (u32)j.cw;
    if (j.n * cw <= 64 * (u64)kWideWideBlock) {
        for (u32 e = threadIdx.x; e < (u32)j.n * cw; e += blockDim.x) {   // a thread per value
            const u32 c = e / cw;
            if (j.flag[c]) w_cols[(e - c * cw) * n + (u32)j.pos[c]] = j.cand[e];
        }
    } else {   // many candidates for the winners: a warp looks at 32 flags and copies the winners' rows
        const u32 lane = threadIdx.x & 31;
        for (u64 c0 = threadIdx.x & ~31u; c0 < j.n; c0 += blockDim.x)
            for (u32 m = __ballot_sync(0xffffffffu, c0 + lane < j.n && j.flag[c0 + lane]); m; m &= m - 1) {
                const u64 c = c0 + __ffs(m) - 1;
                const u32 at = (u32)j.pos[c];
                for (u32 k = lane; k < cw; k += 32) w_cols[k * n + at] = j.cand[c * cw + k];
            }
    }
    if (cw < W)
        for (u64 c = threadIdx.x; c < j.n; c += blockDim.x) {
            if (!j.flag[c]) continue;
            int q = 0;
            while (q + 1 < j.nseg && c >= b.seg_start[j.seg0 + q + 1]) q++;
            const u64 at = j.pos[c];
            w_cols[(W - 1) * n + (u32)at] = b.id_base[j.seg0 + q] + (at - b.win_base[j.seg0 + q]);
        }
    __syncthreads();
    wide_block_sort(S, w_cols, n, j.W);
    for (u32 e = threadIdx.x; e < n * W; e += blockDim.x) {
        const u32 k = e / W, c = e - k * W;
        j.newt[e] = w_cols[c * n + S.idx[k]];
    }
}

// Phase 6: full + delta of every relation of the SCC.  First every delta row's place in
// the merge (a row of full goes before equal rows of delta, so duplicates land next to each
// other), a warp or thread per row in one flattened index space; then the rows, by tiles of
// kWideMergeTile values of the output: a tile that no delta row falls into is one shifted copy,
// the others find each row's side among the tile's delta places.  Bound by reading and
// writing full: consecutive threads move consecutive values, where a thread per row moved
// strided ones and searched for every row of full as well.  Measured on
// worstcase-110-terms-4-m (full up to 2.8M rows of 11 columns): 152 -> 83 ms over 4,312 merges.
struct WideMergeJob {
    const u64* full;
    const u64* delta;
    u64* out;
    u64* pos;        // per delta row: its row in out
    u64 nf, nd;
    u64 first;       // delta rows of the earlier jobs
    u64 tile0;       // tiles of the earlier jobs
    int W;
};
struct WideMergeBatch {
    int n;
    u64 total;       // delta rows
    u64 tiles;
    WideMergeJob job[kWideJobs];
};
constexpr u32 kWideMergeTile = 2048;

template <bool kWarp>
__global__ void __launch_bounds__(kThreads) wide_merge_rank_kernel(const __grid_constant__ WideMergeBatch b)
{
    const u64 id = (u64)blockIdx.x * kThreads + threadIdx.x;
    const u64 stride = (u64)gridDim.x * kThreads >> (kWarp ? 5 : 0);
    for (u64 g = kWarp ? id >> 5 : id; g < b.total; g += stride) {
        const WideMergeJob& j = b.job[wide_job_of(b, g)];
        const u64 d = g - j.first;
        const u64* row = j.delta + d * (u64)j.W;
        const u64 r = kWarp ? wide_bound_warp<true>(j.full, j.W, j.nf, row, j.W)
                            : wide_upper_bound(j.full, j.W, j.nf, row, j.W);
        j.pos[d] = r + d;
    }
}

__global__ void __launch_bounds__(kThreads) wide_merge_copy_kernel(const __grid_constant__ WideMergeBatch b)
{
    __shared__ u64 s_pos[kWideMergeTile + 1];   // delta places of the tile (a row has at least one value)
    __shared__ u64 s_d[2];
    for (u64 t = blockIdx.x; t < b.tiles; t += gridDim.x) {
        int r = 0, hi = b.n;
        while (hi - r > 1) {
            const int m = (r + hi) >> 1;
            if (b.job[m].tile0 <= t) r = m;
            else hi = m;
        }
        const WideMergeJob& j = b.job[r];
        const u32 W = (u32)j.W;
        const u64 e0 = (t - j.tile0) * kWideMergeTile, e1 = min(e0 + kWideMergeTile, (j.nf + j.nd) * W);
        const u64 p0 = e0 / W, p1 = (e1 - 1) / W;      // rows of the tile
        if (threadIdx.x < 64) {   // delta rows before the tile and up to its end: a warp each, places ascend
            const u64 p = threadIdx.x < 32 ? p0 : p1 + 1;
            const u64 d = wide_bound_warp<false>(j.pos, 1, j.nd, &p, 1);
            if ((threadIdx.x & 31) == 0) s_d[threadIdx.x >> 5] = d;
        }
        __syncthreads();
        const u64 d0 = s_d[0], d1 = s_d[1];
        const u64* full = j.full - d0 * W;             // row p of out is full's row p - (delta rows before it)
        if (d0 == d1) {
#pragma unroll
            for (u32 k = 0; k < kWideMergeTile / kThreads; k++) {
                const u64 e = e0 + k * kThreads + threadIdx.x;
                if (e < e1) j.out[e] = full[e];
            }
        } else {
            const u32 nd = (u32)(d1 - d0);
            for (u32 i = threadIdx.x; i < nd; i += kThreads) s_pos[i] = j.pos[d0 + i];
            __syncthreads();
            for (u64 e = e0 + threadIdx.x; e < e1; e += kThreads) {
                const u64 p = e / W;
                u32 lo = 0, up = nd;   // delta rows of the tile before row p
                while (lo < up) {
                    const u32 m = (lo + up) >> 1;
                    if (s_pos[m] < p) lo = m + 1;
                    else up = m;
                }
                j.out[e] = lo < nd && s_pos[lo] == p ? j.delta[(d0 + lo) * W + (e - p * W)] : full[e - (u64)lo * W];
            }
        }
        __syncthreads();
    }
}

// Count and digest of a relation's rows, data columns only (no instances).
__global__ void __launch_bounds__(kThreads) wide_summary_kernel(const u64* __restrict__ rows, int W, u64 n,
                                                                u64* __restrict__ acc)
{
    u64 d = 0;
    for (u64 k = (u64)blockIdx.x * kThreads + threadIdx.x; k < n; k += (u64)gridDim.x * kThreads)
        d += tuple_digest(rows + k * (u64)W, W - 1);
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if ((threadIdx.x & 31) == 0 && d) atomicAdd((unsigned long long*)&acc[1], (unsigned long long)d);
}

}  // namespace ra
