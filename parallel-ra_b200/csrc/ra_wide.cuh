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

// Lexicographic compare of two rows over their first `ncmp` columns: -1, 0, 1.
__device__ __forceinline__ int wide_cmp(const u64* __restrict__ a, const u64* __restrict__ b, int ncmp)
{
    for (int c = 0; c < ncmp; c++) {
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
template <typename T>
__global__ void __launch_bounds__(kThreads) wide_scan_small_kernel(const T* __restrict__ in, u64 n,
                                                                   u64* __restrict__ out, u64* __restrict__ total)
{
    __shared__ u64 sm[kWarps + 1];
    const u64 base = (u64)threadIdx.x * kWideScanPer;
    u64 loc = 0;
    for (int k = 0; k < kWideScanPer; k++)
        if (base + k < n) loc += (u64)in[base + k];
    u64 agg;
    u64 ex = block_exclusive_scan(loc, sm, &agg);
    for (int k = 0; k < kWideScanPer; k++)
        if (base + k < n) {
            out[base + k] = ex;
            ex += (u64)in[base + k];
        }
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

// Does `sorted` hold a row whose first `ncmp` columns equal `key`'s
// (relation::find_in_full / find_in_delta, balanced_hash_relation.cpp:1015-1035)?
__device__ __forceinline__ bool wide_has_prefix(const u64* __restrict__ sorted, int Ws, u64 n,
                                                const u64* __restrict__ key, int ncmp)
{
    if (!n) return false;
    const u64 i = wide_lower_bound(sorted, Ws, n, key, ncmp);
    return i < n && wide_cmp(sorted + i * (u64)Ws, key, ncmp) == 0;
}

// Join ranges: per outer row, the inner rows (trie order) sharing its first jcc
// columns -- all of them when jcc is 0 (parallel_join::local_join,
// src/RA/parallel_join.cpp:157-230).
__global__ void __launch_bounds__(kThreads) wide_join_count_kernel(const u64* __restrict__ outer, int Wo, u64 no,
                                                                   const u64* __restrict__ inner, int Wi, u64 ni,
                                                                   int jcc, u64* __restrict__ lo, u64* __restrict__ cnt)
{
    for (u64 o = (u64)blockIdx.x * kThreads + threadIdx.x; o < no; o += (u64)gridDim.x * kThreads) {
        const u64* key = outer + o * (u64)Wo;
        const u64 a = jcc ? wide_lower_bound(inner, Wi, ni, key, jcc) : 0;
        const u64 b = jcc ? wide_upper_bound(inner, Wi, ni, key, jcc) : ni;
        lo[o] = a;
        cnt[o] = b - a;
    }
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

// copy_filter's predicate on columns 0 and 1 of each input row.
__global__ void __launch_bounds__(kThreads) wide_filter_kernel(const u64* __restrict__ in, int Wi, u64 n, int pred,
                                                               u32* __restrict__ keep)
{
    for (u64 r = (u64)blockIdx.x * kThreads + threadIdx.x; r < n; r += (u64)gridDim.x * kThreads) {
        const u64* row = in + r * (u64)Wi;
        keep[r] = eval_pred(pred, row[0], Wi > 1 ? row[1] : 0) ? 1u : 0u;
    }
}

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

// Rank merge of two sorted arrays of W-column rows: a row of A goes before equal
// rows of B, so duplicates land next to each other.
__global__ void __launch_bounds__(kThreads) wide_merge_rows_kernel(const u64* __restrict__ A, u64 na,
                                                                   const u64* __restrict__ B, u64 nb, int W,
                                                                   u64* __restrict__ out)
{
    const u64 n = na + nb;
    for (u64 p = (u64)blockIdx.x * kThreads + threadIdx.x; p < n; p += (u64)gridDim.x * kThreads) {
        const bool fromA = p < na;
        const u64 i = fromA ? p : p - na;
        const u64* row = fromA ? A + i * (u64)W : B + i * (u64)W;
        const u64 r = fromA ? wide_lower_bound(B, W, nb, row, W) : wide_upper_bound(A, W, na, row, W);
        u64* dst = out + (i + r) * (u64)W;
        for (int j = 0; j < W; j++) dst[j] = row[j];
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

// Phase 1: per job, a join's range counts and their exclusive scan, or a
// copy_filter's pass flags and their scan; the total into *total.
struct WideCountJob {
    const u64* outer;
    const u64* inner;
    u64 no, ni;
    u64* lo;       // join: first match per outer row
    u64* cnt;      // join: matches per outer row
    u64* off;      // join: scanned counts; filter: scanned flags
    u32* keep;     // filter: pass flags
    u64* total;
    int Wo, Wi, jcc, pred;   // pred < 0: a join
};
struct WideCountBatch {
    int n;
    WideCountJob job[kWideJobs];
};

__global__ void __launch_bounds__(kThreads) wide_count_batch_kernel(const __grid_constant__ WideCountBatch b)
{
    __shared__ u64 sm[kWarps + 1];
    const WideCountJob& j = b.job[blockIdx.x];
    // the searches, one row per thread (their latencies overlap)
    for (u64 o = threadIdx.x; o < j.no; o += blockDim.x) {
        const u64* row = j.outer + o * (u64)j.Wo;
        if (j.pred < 0) {
            const u64 a = j.jcc ? wide_lower_bound(j.inner, j.Wi, j.ni, row, j.jcc) : 0;
            const u64 e = j.jcc ? wide_upper_bound(j.inner, j.Wi, j.ni, row, j.jcc) : j.ni;
            j.lo[o] = a;
            j.cnt[o] = e - a;
        } else {
            j.keep[o] = eval_pred(j.pred, row[0], j.Wo > 1 ? row[1] : 0) ? 1u : 0u;
        }
    }
    __syncthreads();
    // the scan, contiguous rows per thread
    const u64 base = (u64)threadIdx.x * kWideScanPer;
    u64 loc = 0;
    for (int k = 0; k < kWideScanPer; k++) {
        const u64 o = base + k;
        if (o >= j.no) break;
        loc += j.pred < 0 ? j.cnt[o] : (u64)j.keep[o];
    }
    u64 agg;
    u64 ex = block_exclusive_scan(loc, sm, &agg);
    for (int k = 0; k < kWideScanPer; k++) {
        const u64 o = base + k;
        if (o >= j.no) break;
        j.off[o] = ex;
        ex += j.pred < 0 ? j.cnt[o] : (u64)j.keep[o];
    }
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
        int r = 0, hi = b.n;   // last job whose first index is <= g
        while (hi - r > 1) {
            const int m = (r + hi) >> 1;
            if (b.job[m].first <= g) r = m;
            else hi = m;
        }
        const WideExpandJob& j = b.job[r];
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
// for acopy targets); one thread per candidate of every relation.
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

__global__ void __launch_bounds__(kThreads) wide_member_batch_kernel(const __grid_constant__ WideMemberBatch b)
{
    for (u64 g = (u64)blockIdx.x * kThreads + threadIdx.x; g < b.total; g += (u64)gridDim.x * kThreads) {
        int r = 0, hi = b.n;
        while (hi - r > 1) {
            const int m = (r + hi) >> 1;
            if (b.job[m].first <= g) r = m;
            else hi = m;
        }
        const WideMemberJob& j = b.job[r];
        const u64 c = g - j.first;
        if (!j.flag[c]) continue;
        const u64* row = j.cand + c * (u64)j.cw;
        if (wide_has_prefix(j.full, j.W, j.nf, row, j.cw) || wide_has_prefix(j.delta, j.W, j.nd, row, j.cw))
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
    const u64 base = (u64)threadIdx.x * kWideScanPer;
    u64 loc = 0;
    for (int k = 0; k < kWideScanPer; k++)
        if (base + k < j.n) loc += j.flag[base + k];
    u64 agg;
    u64 ex = block_exclusive_scan(loc, sm, &agg);
    for (int k = 0; k < kWideScanPer; k++)
        if (base + k < j.n) {
            j.pos[base + k] = ex;
            ex += j.flag[base + k];
        }
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

// Phase 6: full + delta of every relation of the SCC, one flattened index space.
struct WideMergeJob {
    const u64* full;
    const u64* delta;
    u64* out;
    u64 nf, nd, first;
    int W;
};
struct WideMergeBatch {
    int n;
    u64 total;
    WideMergeJob job[kWideJobs];
};

__global__ void __launch_bounds__(kThreads) wide_merge_batch_kernel(const __grid_constant__ WideMergeBatch b)
{
    for (u64 g = (u64)blockIdx.x * kThreads + threadIdx.x; g < b.total; g += (u64)gridDim.x * kThreads) {
        int r = 0, hi = b.n;
        while (hi - r > 1) {
            const int m = (r + hi) >> 1;
            if (b.job[m].first <= g) r = m;
            else hi = m;
        }
        const WideMergeJob& j = b.job[r];
        const u64 p = g - j.first;
        const bool fromA = p < j.nf;
        const u64 i = fromA ? p : p - j.nf;
        const u64* row = fromA ? j.full + i * (u64)j.W : j.delta + i * (u64)j.W;
        const u64 rk = fromA ? wide_lower_bound(j.delta, j.W, j.nd, row, j.W) : wide_upper_bound(j.full, j.W, j.nf, row, j.W);
        u64* dst = j.out + (i + rk) * (u64)j.W;
        for (int k = 0; k < j.W; k++) dst[k] = row[k];
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
