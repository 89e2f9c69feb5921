// Device-driven fixed-point iteration: every size lives in an IterCtl block in
// device memory, so one iteration is a fixed sequence of launches that can be
// captured once into a CUDA graph and replayed by a conditional WHILE node
// until the delta is empty (RAM::check_for_fixed_point's MPI_Allreduce,
// src/RAM/RA_tasks.cpp:1072-1085, becomes a device flag).
//
// Per iteration, for an SCC whose rules read the DELTA of its relations and
// inputs that do not change while it runs (e.g. the FULL of a loaded relation):
//   join_fused     per tile of outer (delta) rows: match counts from the inner
//                  CSR, single-pass decoupled look-back scan of the counts, then
//                  the tile's candidates expanded in place (merge-path over the
//                  tile's rows, so a row is spread over all the block's warps;
//                  a row of more than kHeavyRow matches goes to every block of
//                  the launch as work items), written to the candidate stream and
//                  claimed in the output relation's seen set (first occurrence =
//                  least stream position) -- count, scan and write in one launch
//   copy_claim     (copy / copy_filter rules) one candidate per input row
//   select         per candidate: winner test, ordered compaction (look-back)
//                  straight into the relation's log, intern ids; the last tile
//                  of the last rule runs the iteration end: region bump,
//                  history, intern counters, graph condition
//   join_bitmap, bitmap_select  the same two steps for output relations whose seen
//                  set is a bitmap: a claim is one reduction, the log follows the rows
//   (reference id order only) digit histograms in select, radix launches over the
//   new delta (by buckets of the top digit, or onesweep LSD passes), then a separate
//   iteration-end launch
// An iteration that finds a buffer too small stops before select writes
// anything; claims made so far are idempotent, so the host grows the buffer
// and replays the same iteration (same epoch, same stream positions).
#pragma once
#include "ra_kernels.cuh"

namespace ra {

constexpr int kMaxSccRels = 8;
constexpr int kMaxSccRules = 8;
constexpr int kMaxTagSlots = 8;
constexpr int kMaxPasses = 8;
constexpr int kTileSlots = 128;
constexpr int kTailMaxRules = 2;   // join rules of an SCC the tail kernel (ra_tail.cuh) runs
// a bank of launch counters: kTileSlots tile counters, then 3 heavy-row counters per rule
constexpr int kBankWords = kTileSlots + 3 * kMaxSccRules;

// flags
constexpr u32 kFlagOverflow = 1u;   // a buffer is too small: replay the iteration after growing it
constexpr u32 kFlagTimeout = 2u;    // a bounded look-back wait gave up (fatal)
constexpr u32 kFlagProbe = 4u;      // a seen-set probe gave up (table too full): grow, replay
constexpr u32 kFlagGrow = 8u;       // iteration done; the seen set needs room before the next one
constexpr u32 kFlagRange = 16u;     // a tuple whose columns lie in different instances (fatal)
constexpr u32 kFlagStatus = 32u;    // a launch has more tiles than the look-back status array (fatal)
constexpr u64 kMaxProbe = 4096;

struct IterCtl {
    u64 full_n[kMaxSccRels], delta_n[kMaxSccRels], seen_n[kMaxSccRels];
    u64 cand_n[kMaxSccRules], cand_base[kMaxSccRules], win_n[kMaxSccRules];
    u64 intern[kMaxTagSlots];
    u64 iteration;          // iterations run in this SCC
    u64 epoch;              // seen-set epoch of the running iteration (>= 1)
    u64 batch_pos;
    u64 hist_n;             // (sum_delta, sum_full) pairs recorded
    u64 new_tuples, candidates, outer_rows;
    u64 runs[kMaxSccRels];  // non-empty deltas moved into full (sorted runs added)
    u64 t_start;                    // %globaltimer when the SCC started (ns)
    u64 time_cap;                   // entries of the per-iteration end-time buffer
    u32 tile_ctr[2 * kBankWords];   // two banks: iteration k uses bank k & 1
    u32 exit_ctr;                   // blocks of the running select launch that have finished
    u32 flags;
    u32 done;
    // persistent SCC kernel (ra_persist.cuh): heavy-row work items of the running
    // iteration, and the grid barrier with the values its last arriver publishes
    u32 heavy_ctr;                  // items taken
    u64 heavy_n;                    // items pushed
    u64 ns_claims, ns_heavy, ns_select;   // device time of the phases of the persistent kernel (ns)
    u64 t_phase;                    // %globaltimer at the last barrier release (or kernel start)
    u64 tail_iters;                 // iterations run by the tail kernel (ra_tail.cuh)
    u64 tail_off;                   // the tail kernel declined a skewed iteration: no more tail in this SCC run
    // joins into bitmap relations (join_bitmap_kernel): a launch's candidates so far and its
    // blocks that have finished; whether claims look at the seen bits first
    u64 bit_cand[kMaxSccRules];
    u32 bit_exit[kMaxSccRules];
    u64 bit_filter;
    u64 last_delta, last_full, last_time;   // the latest history entry and iteration end time
    u32 bar_count;                  // blocks arrived at the running barrier
    u32 bar_gen;                    // barrier generation (bumped on release)
    u32 bar_flags;                  // flags / done / heavy_n as the last arriver saw them
    u32 bar_done;
    u64 bar_heavy;
    u64 heavy_items;                // heavy-row work items pushed in this SCC (both paths)
    u64 sort_hist[kMaxSccRels][kMaxPasses][kRadix];
};

// static description of one SCC's iteration, passed by value to the kernels
struct SccPlan {
    int n_rels, n_rules;
    int rule_out[kMaxSccRules];          // output relation slot
    int rule_tag[kMaxSccRules];          // tag slot of the output relation
    int rule_is_join[kMaxSccRules];
    int rule_in_slot[kMaxSccRules];      // copy input: relation slot (DELTA region) or -1 for fixed rows
    u64 rule_in_static_n[kMaxSccRules];  // copy input: rows of a fixed input
    u64 rel_tag_word[kMaxSccRels];       // (tag << 46)
    u64 cand_cap;                        // candidate buffer capacity (all rules of one iteration)
    u64 stage_cap;                       // per-relation staging capacity
    u64 log_cap[kMaxSccRels];
    u64 seen_limit[kMaxSccRels];         // keys a seen set may hold
    u64 hist_cap;                        // history pairs
    u64 batch_size;
    u64 iter_limit;
    int fixpoint;
};

// Rows a rule reads: the DELTA region of an SCC relation (slot >= 0, sizes from
// the control block) or a fixed array (slot < 0: a FULL or DELTA no rule of the
// SCC changes).
struct RowsRef {
    const u64* keys;
    int slot;
    u64 static_n;
};

__device__ __forceinline__ u64 rows_n(const IterCtl* c, const RowsRef& r)
{
    return r.slot >= 0 ? c->delta_n[r.slot] : r.static_n;
}
__device__ __forceinline__ const u64* rows_ptr(const IterCtl* c, const RowsRef& r)
{
    return r.slot >= 0 ? r.keys + c->full_n[r.slot] : r.keys;
}

// ---------------------------------------------------------------------------
// decoupled look-back status words: [tag:24 | flag:2 | value:38]
// ---------------------------------------------------------------------------
constexpr u64 kStAgg = 1, kStIncl = 2;
constexpr int kValBits = 38;
constexpr u64 kValMask = (1ull << kValBits) - 1;
// polls before a look-back wait gives up (about a second of L2 round trips); a
// predecessor tile is always resident and running, so a legitimate wait is far shorter
constexpr u64 kSpinLimit = 1ull << 22;

__device__ __forceinline__ u64 st_pack(u32 tag, u64 flag, u64 v)
{
    return ((u64)(tag & 0xffffffu) << 40) | (flag << kValBits) | (v & kValMask);
}
__device__ __forceinline__ u32 st_tag(u64 s) { return (u32)(s >> 40); }
__device__ __forceinline__ u64 st_flag(u64 s) { return (s >> kValBits) & 3; }
__device__ __forceinline__ u64 st_val(u64 s) { return s & kValMask; }

__device__ __forceinline__ void st_publish(u64* p, u64 w)
{
    __threadfence();
    atomicExch((unsigned long long*)p, (unsigned long long)w);
}

__device__ __forceinline__ u64 st_read(const u64* p) { return *((volatile const u64*)p); }

// Exclusive prefix of tile `tile`'s aggregate `agg` over all earlier tiles.
// Called by one thread.  Bounded: gives up after kSpinLimit polls (flag set).
__device__ u64 lookback_one(u64* status, u32 tile, u64 agg, u32 tag, u32* flags, u64 limit = kSpinLimit)
{
    if (tile == 0) {
        st_publish(&status[0], st_pack(tag, kStIncl, agg));
        return 0;
    }
    st_publish(&status[tile], st_pack(tag, kStAgg, agg));
    u64 excl = 0;
    long t = (long)tile - 1;
    u64 spins = 0;
    while (t >= 0) {
        u64 s = st_read(&status[t]);
        if (st_tag(s) != (tag & 0xffffffu) || st_flag(s) == 0) {
            if (++spins > limit) {
                atomicOr(flags, kFlagTimeout);
                break;
            }
            continue;
        }
        excl += st_val(s);
        if (st_flag(s) == kStIncl) break;
        t--;
    }
    st_publish(&status[tile], st_pack(tag, kStIncl, excl + agg));
    return excl;
}

// Warp-cooperative look-back (all 32 lanes of one warp): each round reads the
// 32 nearest unresolved predecessors at once.  Returns the exclusive prefix on
// every lane.  Bounded like lookback_one.
__device__ u64 lookback_warp(u64* status, u32 tile, u64 agg, u32 tag, u32* flags)
{
    const int lane = threadIdx.x & 31;
    const u32 tg = tag & 0xffffffu;
    if (tile == 0) {
        if (lane == 0) st_publish(&status[0], st_pack(tag, kStIncl, agg));
        return 0;
    }
    if (lane == 0) st_publish(&status[tile], st_pack(tag, kStAgg, agg));
    u64 excl = 0;
    long base = (long)tile - 1;
    u64 spins = 0;
    for (;;) {
        const long t = base - lane;
        u64 s = 0;
        bool ready = true, incl = true;
        if (t >= 0) {
            s = st_read(&status[t]);
            ready = st_tag(s) == tg && st_flag(s) != 0;
            incl = ready && st_flag(s) == kStIncl;
        }
        const u32 inclmask = __ballot_sync(0xffffffffu, incl);
        const u32 notready = __ballot_sync(0xffffffffu, !ready);
        const int first = inclmask ? __ffs(inclmask) - 1 : 32;
        const u32 needed = first >= 31 ? 0xffffffffu : ((2u << first) - 1);
        if (notready & needed) {
            if (++spins > kSpinLimit) {
                if (lane == 0) atomicOr(flags, kFlagTimeout);
                break;
            }
            continue;
        }
        u64 v = (lane <= first && t >= 0) ? st_val(s) : 0;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        excl += v;
        if (first < 32) break;
        base -= 32;
    }
    if (lane == 0) st_publish(&status[tile], st_pack(tag, kStIncl, excl + agg));
    return excl;
}

// Failure-path self-test: tile 1 of a look-back whose tile 0 never publishes.
// The wait must give up after `limit` polls and set kFlagTimeout.
__global__ void lookback_selftest_kernel(u64* status, u32* flags, u64 limit)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) lookback_one(status, 1, 1, 7, flags, limit);
}

__device__ __forceinline__ u32 iter_tag(const IterCtl* c, int slot)
{
    return (u32)(((c->iteration + 1) << 7) | (u64)slot);
}

__device__ __forceinline__ u32* tile_counter(IterCtl* c, int slot)
{
    return &c->tile_ctr[(c->iteration & 1) * kBankWords + slot];
}

// first index i in [0, n) with a[i] > x (n if none)
template <typename T>
__device__ __forceinline__ u64 upper_bound_dev(const T* a, u64 n, u64 x)
{
    u64 lo = 0, hi = n;
    while (lo < hi) {
        u64 mid = (lo + hi) >> 1;
        if ((u64)a[mid] <= x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// candidates of rules before `rule` in this iteration's stream
__device__ __forceinline__ u64 stream_base(const IterCtl* c, int rule)
{
    u64 b = 0;
    for (int q = 0; q < rule; q++) b += c->cand_n[q];
    return b;
}

// ---------------------------------------------------------------------------
// first-occurrence claims: one 16-byte CAS per probed slot.  An empty slot
// becomes {k, mine}; a slot holding k keeps the smaller tag (older tuples carry
// smaller tags: 0, or an earlier epoch).  Every candidate that is not the first
// occurrence of a new tuple ends up marked in `loser` (indexed by stream
// position, value = epoch): it marks itself when the key is older or holds a
// smaller position, and marks the position it displaces when it lowers the
// tag.  select then needs no access to the seen set.  kClaimBatch independent
// claims are issued back to back: two per thread, so that the join kernel fits
// 31 registers and a full SM of threads (measured on tc-er22: 12.03 ms per step
// against 12.55 with four per thread at 64 registers and 4 CTAs per SM).
// ---------------------------------------------------------------------------
constexpr int kClaimBatch = 2;
constexpr u64 kPosMask = (1ull << 40) - 1;

struct LoserMarks {
    u32* mark;      // per stream position (minus `base`)
    u32 epoch;      // marks of this iteration (older values mean "not a loser now")
    u64 epoch_tag;  // epoch << 40: tags below it belong to tuples from earlier iterations
    u64 base;       // stream position of mark[0] (a slice of outer rows starts there; else 0)
};

__device__ __forceinline__ void claim_rest(Slot* __restrict__ t, u64 cap, u64 k, u64 mine, u64 h, Slot cur,
                                           const LoserMarks& lm, u32* flags)
{
    const Slot empty{kEmpty, ~0ull};
    const Slot mineslot{k, mine};
    for (u64 probe = 0; probe < kMaxProbe; probe++) {
        if (slot_eq(cur, empty)) return;   // we inserted it
        if (cur.key == k) {
            for (;;) {
                if (cur.tag == mine) return;     // our own claim from an attempt being replayed
                if (cur.tag < mine) {            // older tuple, or an earlier position this iteration
                    lm.mark[(mine & kPosMask) - lm.base] = lm.epoch;
                    return;
                }
                const Slot prev = atomicCAS(&t[h], cur, mineslot);
                if (slot_eq(prev, cur)) {      // we took the slot from a later position
                    lm.mark[(cur.tag & kPosMask) - lm.base] = lm.epoch;   // a later position: same slice
                    return;
                }
                cur = prev;
            }
        }
        h = slot_next(h, cap);
        cur = atomicCAS(&t[h], empty, mineslot);
    }
    atomicOr(flags, kFlagProbe);
}

// N claims of one thread, issued back to back (N from the caller's arrays, so a
// caller's batch size and this loop cannot disagree)
template <int N>
__device__ __forceinline__ void claim_batch(Slot* __restrict__ t, u64 cap, const u64 (&key)[N], const u64 (&mine)[N],
                                            const bool (&valid)[N], const LoserMarks& lm, u32* flags)
{
    const Slot empty{kEmpty, ~0ull};
    Slot cur[N];
    u64 h[N];
#pragma unroll
    for (int k = 0; k < N; k++) {
        h[k] = slot_start(key[k], cap);
        if (valid[k]) cur[k] = atomicCAS(&t[h[k]], empty, Slot{key[k], mine[k]});
    }
#pragma unroll
    for (int k = 0; k < N; k++)
        if (valid[k]) claim_rest(t, cap, key[k], mine[k], h[k], cur[k], lm, flags);
}

__device__ __forceinline__ LoserMarks loser_marks(const IterCtl* c, u32* mark)
{
    return LoserMarks{mark, (u32)c->epoch, c->epoch << 40, 0};
}

// ---------------------------------------------------------------------------
// Bitmap seen set of a binary relation over a small value domain (at most
// 65,536 values): bit c1 of row c0 is set for every tuple (c0, c1) the relation
// holds.  A claim is one OR, nothing read back, on a word of `fresh`, a table a fraction
// of the size of the hash set; `dirty[c0]` marks rows holding some.  bitmap_select_kernel
// takes the tuples not yet in `seen` from it, adds them there and emits them in key
// order.  No candidate stream and no loser marks: the set of new tuples is the same as
// the hash-set path's, and their order (sorted) does not depend on which duplicate
// claimed first.  In an iteration after one whose candidates were mostly known
// (IterCtl::bit_filter: fewer than 3/4 new) claims read `seen` first and leave known tuples
// out, which costs a read per claim and saves the select's.
// ---------------------------------------------------------------------------
struct BitSeen {
    u32* seen;      // null: the relation uses its hash seen set
    u32* fresh;
    u8* dirty;
    u32 words;      // u32 words per row (one matrix: no instances)
    u32 n;          // rows (values)
    // with instances, one matrix per instance: row v's first word, the base value and
    // the words of its instance's rows, the instance itself (null without instances)
    const u64* row_word;
    const u32* row_base;
    const u32* row_words;
    const u32* row_inst;
};

__device__ __forceinline__ u64 bit_word(const BitSeen& b, u64 c0, u64 c1)
{
    return b.row_word ? b.row_word[c0] + ((c1 - b.row_base[c0]) >> 5) : c0 * b.words + (c1 >> 5);
}
__device__ __forceinline__ u32 bit_of(const BitSeen& b, u64 c0, u64 c1)
{
    return 1u << ((b.row_word ? c1 - b.row_base[c0] : c1) & 31);
}

// With instances, is (c0, c1) inside c0's instance matrix?
__device__ __forceinline__ bool bit_in_range(const BitSeen& b, u64 c0, u64 c1)
{
    return !b.row_word || ((c1 - b.row_base[c0]) >> 5) < b.row_words[c0];
}

// The bits `m` of word w of row c0.  A row's first claims mark it dirty.
__device__ __forceinline__ void bit_claim_word(const BitSeen& b, u64 c0, u64 w, u32 m, bool filter)
{
    if (filter) m &= ~*((volatile u32*)&b.seen[w]);
    if (!m) return;
    atomicOr(&b.fresh[w], m);
    if (!*((volatile u8*)&b.dirty[c0])) b.dirty[c0] = 1;
}

__device__ __forceinline__ void bit_claim(const BitSeen& b, u64 key, int bits, IterCtl* ctl)
{
    const u64 c0 = key >> bits, c1 = key & ((1ull << bits) - 1);
    if (!bit_in_range(b, c0, c1)) {
        atomicOr(&ctl->flags, kFlagRange);
        return;
    }
    bit_claim_word(b, c0, bit_word(b, c0, c1), bit_of(b, c0, c1), ctl->bit_filter != 0);
}

// Bits of a relation's stored tuples (its full and delta regions).
__global__ void __launch_bounds__(kThreads) bitmap_build_kernel(BitSeen b, const u64* __restrict__ keys, u64 n,
                                                                int bits, u32* __restrict__ err)
{
    for (u64 i = (u64)blockIdx.x * kThreads + threadIdx.x; i < n; i += (u64)gridDim.x * kThreads) {
        const u64 k = keys[i];
        const u64 c0 = k >> bits, c1 = k & ((1ull << bits) - 1);
        if (!bit_in_range(b, c0, c1)) {
            *err = 1u;
            continue;
        }
        atomicOr(&b.seen[bit_word(b, c0, c1)], bit_of(b, c0, c1));
    }
}

// ---------------------------------------------------------------------------
// join_fused: count + look-back scan + expansion + claim, one launch per rule
// ---------------------------------------------------------------------------
#ifndef RA_JOIN_ROWS_PER_THREAD
#define RA_JOIN_ROWS_PER_THREAD 2
#endif
#ifndef RA_JOIN_MIN_BLOCKS
#define RA_JOIN_MIN_BLOCKS 8   // 31 registers: 8 CTAs (2,048 threads) per SM hide the claims' latency
#endif
#ifndef RA_SELECT_IPT
#define RA_SELECT_IPT 4
#endif
#ifndef RA_SELECT_MIN_BLOCKS
#define RA_SELECT_MIN_BLOCKS 4
#endif
constexpr int kJRowsPerThread = RA_JOIN_ROWS_PER_THREAD;
constexpr int kJRows = kThreads * kJRowsPerThread;   // outer rows per tile

// One slice of a rule's outer rows (an iteration whose candidates exceed the
// candidate buffer runs in slices): rows [lo, lo + rows) of the rule's input,
// their candidates at buffer index 0.., stream positions from `pos`.
struct JoinSlice {
    u64 lo, rows, pos;
    int on;
};

// Skewed keys.  An outer row with more than kHeavyRow matches is not expanded
// by its tile's block: it keeps its stream positions, and the tile pushes it as
// work items of kHeavyPiece candidates that every warp of the grid takes from a
// shared list once all tiles have been scanned.
constexpr u64 kHeavyRow = 4096;
constexpr u64 kHeavyPiece = 2048;

// One heavy row's slice of candidates: stream positions [pos, pos + count).
struct __align__(16) HeavyItem {
    u64 pos;     // stream position of the first candidate (relative to the launch's first)
    u64 key;     // the outer row
    u64 start;   // its first inner row of the slice
    u32 count;
    u32 rule;
};
static_assert(sizeof(HeavyItem) == 32, "HeavyItem is read as two 16-byte words");

__device__ __forceinline__ u32 ldcg_u32(const u32* p) { return __ldcg(p); }
__device__ __forceinline__ HeavyItem ldcg_item(const HeavyItem* p)
{
    const ulonglong2 a = __ldcg((const ulonglong2*)p), b = __ldcg((const ulonglong2*)p + 1);
    HeavyItem h;
    h.pos = a.x;
    h.key = a.y;
    h.start = b.x;
    h.count = (u32)b.y;
    h.rule = (u32)(b.y >> 32);
    return h;
}

// Per-rule counters of the heavy-row list, banked with the tile counters.
enum HeavyWord { kHvItems = 0, kHvScanned = 1, kHvTaken = 2 };
__device__ __forceinline__ u32* heavy_counter(IterCtl* c, int rule, int w)
{
    return &c->tile_ctr[(c->iteration & 1) * kBankWords + kTileSlots + 3 * rule + w];
}

// Shared memory of one join block.
struct JoinSmem {
    u64 ex[kJRows + 1];   // exclusive prefix of match counts inside the tile
    u32 lx[kJRows + 1];   // the same over the rows this block expands (kSplit: heavy rows count 0)
    u64 start[kJRows];    // first inner row of each outer row
    u64 key[kJRows];      // outer keys
    u64 sm[kWarps + 1];
    u32 tile;
    u64 prefix, hbase, hn;
};

// The tiles of one join launch (bitmap relations: only kSplit; join_bitmap_kernel runs
// their other joins).  kSplit: the inner CSR has rows longer than
// kHeavyRow, so a tile's heavy rows go to the shared list and every block
// expands that list after the tiles; without it the code is the plain tile loop.
template <bool kSplit>
__device__ __forceinline__ void join_tiles(JoinSmem& S, IterCtl* __restrict__ ctl, int rule, const u64* __restrict__ outer,
                                           u64 n, int outer_shift, const u64* __restrict__ csr,
                                           const u64* __restrict__ inner, const Projection& pj, int bits,
                                           u64* __restrict__ cand, u64 cand_cap, Slot* __restrict__ seen,
                                           u64 seen_cap, u32* __restrict__ loser, u64* __restrict__ status,
                                           int tile_slot, const BitSeen& bs, const JoinSlice& sl,
                                           HeavyItem* __restrict__ heavy, u64 heavy_cap)
{
    const u64 ntiles = (n + kJRows - 1) / kJRows;
    if (!kSplit && blockIdx.x >= ntiles) return;
    const u64 cbase = sl.on ? 0 : stream_base(ctl, rule);   // buffer index of the first candidate
    const u64 tag_base = (ctl->epoch << 40) | (sl.on ? sl.pos : cbase);
    const u32 tag = iter_tag(ctl, tile_slot);
    u32* ctr = tile_counter(ctl, tile_slot);
    LoserMarks lm = loser_marks(ctl, loser);
    lm.base = sl.on ? sl.pos : 0;
    if (kSplit && threadIdx.x == 0) {   // heavy items of the earlier rules of this iteration come first
        u64 b = 0;
        for (int r = 0; r < rule; r++) b += *heavy_counter(ctl, r, kHvItems);
        S.hbase = b;
    }
    for (;;) {
        // (kSplit) a block beyond the tiles that sees every tile taken needs no atomic
        if (threadIdx.x == 0)
            S.tile = (kSplit && blockIdx.x >= ntiles && ldcg_u32(ctr) >= (u32)ntiles) ? (u32)ntiles
                                                                                     : atomicAdd(ctr, 1u);
        __syncthreads();
        const u64 tile = S.tile;
        __syncthreads();
        if (tile >= ntiles) break;
        const u64 r0 = tile * kJRows;
        u64 cnt[kJRowsPerThread];
        u64 local = 0;   // kSplit: (all matches << 24) | matches of the rows expanded here
#pragma unroll
        for (int k = 0; k < kJRowsPerThread; k++) {
            const int li = threadIdx.x * kJRowsPerThread + k;
            const u64 i = r0 + li;
            cnt[k] = 0;
            if (i < n) {
                const u64 key = outer[i];
                const u64 j = key >> outer_shift;
                const u64 s = csr[j];
                cnt[k] = csr[j + 1] - s;
                S.start[li] = s;
                S.key[li] = key;
            }
            local += kSplit ? ((cnt[k] << 24) | (cnt[k] > kHeavyRow ? 0 : cnt[k])) : cnt[k];
        }
        u64 aggp;
        u64 ex = block_exclusive_scan(local, S.sm, &aggp);
        bool mine_heavy = false;
#pragma unroll
        for (int k = 0; k < kJRowsPerThread; k++) {
            const int li = threadIdx.x * kJRowsPerThread + k;
            if (kSplit) {
                S.ex[li] = ex >> 24;
                S.lx[li] = (u32)(ex & 0xffffffu);
                ex += (cnt[k] << 24) | (cnt[k] > kHeavyRow ? 0 : cnt[k]);
                mine_heavy |= cnt[k] > kHeavyRow;
            } else {
                S.ex[li] = ex;
                ex += cnt[k];
            }
        }
        const u64 agg = kSplit ? aggp >> 24 : aggp, lagg = kSplit ? aggp & 0xffffffu : aggp;
        if (threadIdx.x == 0) {
            S.ex[kJRows] = agg;
            if (kSplit) S.lx[kJRows] = (u32)lagg;
        }
        if (threadIdx.x < 32) {
            const u64 pre = lookback_warp(status, (u32)tile, agg, tag, &ctl->flags);
            if (threadIdx.x == 0) S.prefix = pre;
        }
        __syncthreads();
        const u64 prefix = S.prefix;
        if (tile == ntiles - 1 && threadIdx.x == 0) {
            ctl->cand_n[rule] = prefix + agg;
            ctl->outer_rows += n;
        }
        const bool room = (kSplit && bs.seen) || cbase + prefix + agg <= cand_cap;
        if (!room && threadIdx.x == 0) atomicOr(&ctl->flags, kFlagOverflow);
        if (kSplit) {
            if (room && mine_heavy) {
#pragma unroll
                for (int k = 0; k < kJRowsPerThread; k++) {
                    if (cnt[k] <= kHeavyRow) continue;
                    const int li = threadIdx.x * kJRowsPerThread + k;
                    const u64 pieces = (cnt[k] + kHeavyPiece - 1) / kHeavyPiece;
                    const u64 at = S.hbase + atomicAdd(heavy_counter(ctl, rule, kHvItems), (u32)pieces);
                    if (at + pieces > heavy_cap) {
                        atomicOr(&ctl->flags, kFlagOverflow);
                        continue;
                    }
                    const u64 p0 = prefix + S.ex[li];
                    for (u64 pc = 0; pc < pieces; pc++) {
                        const u64 off = pc * kHeavyPiece;
                        heavy[at + pc] = HeavyItem{p0 + off, S.key[li], S.start[li] + off,
                                                   (u32)min(kHeavyPiece, cnt[k] - off), (u32)rule};
                    }
                    atomicAdd((unsigned long long*)&ctl->heavy_items, (unsigned long long)pieces);
                }
                __threadfence();
            }
            __syncthreads();
            if (threadIdx.x == 0) atomicAdd(heavy_counter(ctl, rule, kHvScanned), 1u);
        }
        if (room) {
            // the tile's candidates expanded here: position prefix + ex[row] + rank
            const u64 nr = min((u64)kJRows, n - r0);
            for (u64 j0 = 0; j0 < lagg; j0 += (u64)kThreads * kClaimBatch) {
                u64 key[kClaimBatch], mine[kClaimBatch];
                bool valid[kClaimBatch];
                u64 ik[kClaimBatch];
                u64 at[kClaimBatch];
                int rr[kClaimBatch];
#pragma unroll
                for (int k = 0; k < kClaimBatch; k++) {
                    const u64 j = j0 + threadIdx.x + (u64)k * kThreads;
                    valid[k] = j < lagg;
                    rr[k] = 0;
                    at[k] = 0;
                    ik[k] = 0;
                    if (valid[k]) {
                        u64 rank;
                        if (!kSplit || lagg == agg) {   // no heavy row in the tile: j is the position
                            rr[k] = (int)upper_bound_dev(S.ex, nr, j) - 1;
                            rank = j - S.ex[rr[k]];
                            at[k] = prefix + j;
                        } else {
                            rr[k] = (int)upper_bound_dev(S.lx, nr, j) - 1;
                            rank = j - S.lx[rr[k]];
                            at[k] = prefix + S.ex[rr[k]] + rank;
                        }
                        ik[k] = inner[S.start[rr[k]] + rank];
                    }
                }
#pragma unroll
                for (int k = 0; k < kClaimBatch; k++) {
                    key[k] = valid[k] ? project(pj, S.key[rr[k]], ik[k], bits) : 0;
                    mine[k] = tag_base + at[k];
                    if (valid[k] && !(kSplit && bs.seen)) cand[cbase + at[k]] = key[k];
                }
                // never taken without kSplit, but compiled: where this branch was left out, the claims of
                // repeated candidates took longer (a closure of 145 grids of 30 x 30 values, half of
                // its candidates repeated: 5.37 ms of iterations against 4.80)
                if (bs.seen) {
#pragma unroll
                    for (int k = 0; k < kClaimBatch; k++)
                        if (valid[k]) bit_claim(bs, key[k], bits, ctl);
                } else {
                    claim_batch(seen, seen_cap, key, mine, valid, lm, &ctl->flags);
                }
            }
        }
        __syncthreads();
    }
    if (!kSplit) return;
    // Heavy rows.  This block saw every tile taken, each by a running block that
    // scans (and pushes) its tile before expanding it, so the wait ends once the
    // last tile's look-back has; bounded all the same.
    if (threadIdx.x == 0) {
        u64 spins = 0;
        const u32* scanned = heavy_counter(ctl, rule, kHvScanned);
        while (ldcg_u32(scanned) < (u32)ntiles) {
            if (++spins > kSpinLimit) {
                atomicOr(&ctl->flags, kFlagTimeout);
                break;
            }
            __nanosleep(64);
        }
        __threadfence();
        // a push that found the list full reserved items it never wrote: the
        // iteration is replayed with more room, so nothing is taken
        const u64 items = ldcg_u32(heavy_counter(ctl, rule, kHvItems));
        const bool bad = spins > kSpinLimit || (ldcg_u32(&ctl->flags) & (kFlagOverflow | kFlagTimeout)) ||
                         S.hbase + items > heavy_cap;
        S.hn = bad ? 0 : items;
    }
    __syncthreads();
    const u64 hn = S.hn;
    if (hn == 0) return;
    const int lane = threadIdx.x & 31;
    u32* taken = heavy_counter(ctl, rule, kHvTaken);
    for (;;) {
        u32 it = 0;
        if (lane == 0) it = atomicAdd(taken, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= hn) break;
        const HeavyItem h = ldcg_item(&heavy[S.hbase + it]);
        for (u32 t0 = 0; t0 < h.count; t0 += 32 * kClaimBatch) {
            u64 key[kClaimBatch], mine[kClaimBatch], ik[kClaimBatch];
            bool valid[kClaimBatch];
#pragma unroll
            for (int b = 0; b < kClaimBatch; b++) {
                const u32 t = t0 + (u32)b * 32 + lane;
                valid[b] = t < h.count;
                ik[b] = valid[b] ? inner[h.start + t] : 0;
            }
#pragma unroll
            for (int b = 0; b < kClaimBatch; b++) {
                const u64 at = h.pos + t0 + (u64)b * 32 + lane;
                key[b] = valid[b] ? project(pj, h.key, ik[b], bits) : 0;
                mine[b] = tag_base + at;
                if (valid[b] && !bs.seen) cand[cbase + at] = key[b];
            }
            if (bs.seen) {
#pragma unroll
                for (int b = 0; b < kClaimBatch; b++)
                    if (valid[b]) bit_claim(bs, key[b], bits, ctl);
            } else {
                claim_batch(seen, seen_cap, key, mine, valid, lm, &ctl->flags);
            }
        }
    }
}

// One join rule's launch.  kSplit (the host's choice: the inner CSR has a row
// longer than kHeavyRow) adds the heavy-row list; otherwise the plain tile loop.
template <bool kSplit>
__global__ void __launch_bounds__(kThreads, RA_JOIN_MIN_BLOCKS) join_fused_kernel(IterCtl* __restrict__ ctl, int rule, RowsRef outer_ref,
                                                              int outer_shift, const u64* __restrict__ csr,
                                                              const u64* __restrict__ inner, Projection pj, int bits,
                                                              u64* __restrict__ cand, u64 cand_cap,
                                                              Slot* __restrict__ seen, u64 seen_cap,
                                                              u32* __restrict__ loser, u64* __restrict__ status,
                                                              u64 status_cap, int tile_slot, BitSeen bs, JoinSlice sl,
                                                              HeavyItem* __restrict__ heavy, u64 heavy_cap)
{
    __shared__ JoinSmem S;
    if (ctl->flags || ctl->done) return;   // done: the tail kernel reached the fixed point
    const u64 n = sl.on ? sl.rows : rows_n(ctl, outer_ref);
    const u64* outer = rows_ptr(ctl, outer_ref) + (sl.on ? sl.lo : 0);
    if (n == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl->cand_n[rule] = 0;
        return;
    }
    const u64 ntiles = (n + kJRows - 1) / kJRows;
    if (ntiles > status_cap) {   // the host sizes status for the largest outer input: never taken
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&ctl->flags, kFlagStatus);
        return;
    }
    join_tiles<kSplit>(S, ctl, rule, outer, n, outer_shift, csr, inner, pj, bits, cand, cand_cap, seen, seen_cap,
                       loser, status, tile_slot, bs, sl, heavy, heavy_cap);
}

// A join rule into a bitmap relation whose inner CSR has no row longer than kHeavyRow.
// The bitmap needs no stream positions, so there is no scan, no look-back and no search for a
// candidate's row: a thread takes whole outer rows (kBitRows at a time, their loads in
// flight together) and walks their matches, ORing the bits of one word of a row together
// before it claims them -- siblings' values are neighbours; rows of more than kBitLong
// matches are walked by the warp.  Bound by the rate of ORs on random sectors in L2.
// Measured on a tree of 2^15 nodes against the tile loop (556M candidates): 17.2 -> 4.1 ms.
constexpr int kBitRows = 4;
constexpr u32 kBitLong = 16;

__global__ void __launch_bounds__(kThreads) join_bitmap_kernel(IterCtl* __restrict__ ctl, int rule, RowsRef outer_ref,
                                                               int outer_shift, const u64* __restrict__ csr,
                                                               const u64* __restrict__ inner, Projection pj, int bits,
                                                               BitSeen bs)
{
    __shared__ u64 sm[kWarps + 1];
    if (ctl->flags || ctl->done) return;
    const u64 n = rows_n(ctl, outer_ref);
    const u64 step = (u64)gridDim.x * kThreads * kBitRows;
    // blocks past the rows take no part (a thousand arrivals at one counter cost 2 us)
    const u32 parting = (u32)max((u64)1, min((u64)gridDim.x, (n + kThreads * kBitRows - 1) / (kThreads * kBitRows)));
    if (blockIdx.x >= parting) return;
    const u64* outer = rows_ptr(ctl, outer_ref);
    const bool filter = ctl->bit_filter != 0;
    const u64 mask = (1ull << bits) - 1;
    const bool in0 = pj.side[0] != 0, in1 = pj.side[1] != 0;   // output column from the inner row
    const int sh0 = ((in0 ? pj.inner_arity : pj.outer_arity) - 1 - pj.col[0]) * bits;
    const int sh1 = ((in1 ? pj.inner_arity : pj.outer_arity) - 1 - pj.col[1]) * bits;
    const int lane = threadIdx.x & 31;
    u64 total = 0;
    for (u64 base = (u64)blockIdx.x * kThreads * kBitRows; base < n; base += step) {   // block-uniform
        u64 key[kBitRows], s[kBitRows];
        u32 c[kBitRows];
#pragma unroll
        for (int k = 0; k < kBitRows; k++) {
            const u64 i = base + (u64)k * kThreads + threadIdx.x;
            key[k] = i < n ? outer[i] : ~0ull;
        }
#pragma unroll
        for (int k = 0; k < kBitRows; k++) {
            const u64 j = key[k] >> outer_shift;
            s[k] = c[k] = 0;
            if (key[k] != ~0ull) {
                s[k] = csr[j];
                c[k] = (u32)(csr[j + 1] - s[k]);
            }
            total += c[k];
        }
#pragma unroll
        for (int k = 0; k < kBitRows; k++) {
            const u64 o0 = (key[k] >> sh0) & mask, o1 = (key[k] >> sh1) & mask;
            if (c[k] && c[k] <= kBitLong) {
                u64 pw = 0, pr = 0;   // the word being collected, its row
                u32 pm = 0;
                for (u32 t = 0; t < c[k]; t++) {
                    const u64 ik = inner[s[k] + t];
                    const u64 c0 = in0 ? (ik >> sh0) & mask : o0, c1 = in1 ? (ik >> sh1) & mask : o1;
                    if (!bit_in_range(bs, c0, c1)) {
                        atomicOr(&ctl->flags, kFlagRange);
                        continue;
                    }
                    const u64 w = bit_word(bs, c0, c1);
                    if (pm && w != pw) {
                        bit_claim_word(bs, pr, pw, pm, filter);
                        pm = 0;
                    }
                    pw = w;
                    pr = c0;
                    pm |= bit_of(bs, c0, c1);
                }
                if (pm) bit_claim_word(bs, pr, pw, pm, filter);
            }
            for (u32 big = __ballot_sync(0xffffffffu, c[k] > kBitLong); big; big &= big - 1) {
                const int src = __ffs(big) - 1;
                const u64 ok = __shfl_sync(0xffffffffu, key[k], src), os = __shfl_sync(0xffffffffu, s[k], src);
                const u32 oc = __shfl_sync(0xffffffffu, c[k], src);
                for (u32 t = lane; t < oc; t += 32) {
                    const u64 ik = inner[os + t];
                    const u64 c0 = ((in0 ? ik : ok) >> sh0) & mask, c1 = ((in1 ? ik : ok) >> sh1) & mask;
                    if (bit_in_range(bs, c0, c1))
                        bit_claim_word(bs, c0, bit_word(bs, c0, c1), bit_of(bs, c0, c1), filter);
                    else
                        atomicOr(&ctl->flags, kFlagRange);
                }
            }
        }
    }
    total = block_reduce_sum(total, sm);
    if (threadIdx.x == 0) {
        if (total) atomicAdd((unsigned long long*)&ctl->bit_cand[rule], (unsigned long long)total);
        __threadfence();
        if (atomicAdd(&ctl->bit_exit[rule], 1u) == parting - 1) {   // the launch's last block
            __threadfence();
            ctl->cand_n[rule] = __ldcg((unsigned long long*)&ctl->bit_cand[rule]);
            ctl->bit_cand[rule] = 0;
            ctl->bit_exit[rule] = 0;
            ctl->outer_rows += n;
        }
    }
}

// Candidates of every tile of kJRows outer rows (the host cuts an iteration
// whose candidates exceed the candidate buffer into slices of whole tiles).
__global__ void __launch_bounds__(kThreads) join_tile_counts_kernel(const IterCtl* __restrict__ ctl, RowsRef outer_ref,
                                                                    int outer_shift, const u64* __restrict__ csr,
                                                                    u64* __restrict__ tile_cnt)
{
    __shared__ u64 sm[kWarps + 1];
    const u64 n = rows_n(ctl, outer_ref);
    const u64* outer = rows_ptr(ctl, outer_ref);
    const u64 ntiles = (n + kJRows - 1) / kJRows;
    for (u64 t = blockIdx.x; t < ntiles; t += gridDim.x) {
        u64 c = 0;
        for (u64 i = t * kJRows + threadIdx.x; i < min(n, (t + 1) * kJRows); i += kThreads) {
            const u64 j = outer[i] >> outer_shift;
            c += csr[j + 1] - csr[j];
        }
        const u64 tot = block_reduce_sum(c, sm);
        if (threadIdx.x == 0) tile_cnt[t] = tot;
    }
}

// copy / copy_filter: one candidate per input row, stream position = row index
__global__ void __launch_bounds__(kThreads) copy_claim_kernel(IterCtl* __restrict__ ctl, SccPlan plan, int rule,
                                                              RowsRef in_ref, Projection pj, int bits, int pred,
                                                              u64* __restrict__ cand, u64 cand_cap,
                                                              Slot* __restrict__ seen, u64 seen_cap,
                                                              u32* __restrict__ loser, BitSeen bs)
{
    if (ctl->flags || ctl->done) return;
    const u64 c = rows_n(ctl, in_ref);
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->cand_n[rule] = c;
    if (c == 0) return;
    const u64 cbase = stream_base(ctl, rule);
    if (!bs.seen && cbase + c > cand_cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&ctl->flags, kFlagOverflow);
        return;
    }
    const u64* in = rows_ptr(ctl, in_ref);
    const u64 tag_base = (ctl->epoch << 40) | cbase;
    const LoserMarks lm = loser_marks(ctl, loser);
    u64* out = cand + cbase;
    const u64 stride = (u64)gridDim.x * kThreads * kClaimBatch;
    for (u64 p0 = (u64)blockIdx.x * kThreads * kClaimBatch; p0 < c; p0 += stride) {
        u64 key[kClaimBatch], mine[kClaimBatch];
        bool valid[kClaimBatch];
#pragma unroll
        for (int k = 0; k < kClaimBatch; k++) {
            const u64 p = p0 + threadIdx.x + (u64)k * kThreads;
            valid[k] = false;
            key[k] = 0;
            mine[k] = tag_base + p;
            if (p < c) {
                const u64 kk = in[p];
                bool keep = true;
                if (pred != 0) {
                    u64 a = column_of(kk, pj.outer_arity, 0, bits);
                    u64 b = pj.outer_arity > 1 ? column_of(kk, pj.outer_arity, 1, bits) : 0;
                    keep = eval_pred(pred, a, b);
                }
                key[k] = keep ? project(pj, kk, 0, bits) : kEmpty;
                if (!bs.seen) out[p] = key[k];
                valid[k] = keep;
            }
        }
        if (bs.seen) {
#pragma unroll
            for (int k = 0; k < kClaimBatch; k++)
                if (valid[k]) bit_claim(bs, key[k], bits, ctl);
        } else if (seen) {   // else the candidates are known to be new and different
            claim_batch(seen, seen_cap, key, mine, valid, lm, &ctl->flags);
        }
    }
    (void)plan;
}

// ---------------------------------------------------------------------------
// end of an iteration (one thread): semi-naive swap on the counters, history,
// intern counters, next bank of tile counters, graph condition.
// ---------------------------------------------------------------------------
struct SccRelMap {
    int n_rules_in[kMaxSccRels];
    int rules_in[kMaxSccRels][kMaxSccRules];
};

__device__ __forceinline__ u64 global_ns()
{
    u64 t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// history holds plan.hist_cap (sum_delta, sum_full) pairs, then time_cap
// per-iteration end times (%globaltimer, ns)
__device__ void end_of_iteration(IterCtl* __restrict__ ctl, const SccPlan& plan, const SccRelMap& rm,
                                 u64* __restrict__ history, cudaGraphConditionalHandle cond, int use_cond)
{
    bool cont = false;
    const bool records = !plan.fixpoint || ctl->batch_pos + 1 >= plan.batch_size;
    if (ctl->flags == 0 && records && ctl->hist_n >= plan.hist_cap) atomicOr(&ctl->flags, kFlagOverflow);
    if (ctl->flags == 0) {
        u64 sum_delta = 0, sum_full = 0, added = 0;
        bool grow = false;
        for (int s = 0; s < plan.n_rels; s++) {
            u64 nn = 0, in = 0;
            for (int q = 0; q < rm.n_rules_in[s]; q++) {
                nn += ctl->win_n[rm.rules_in[s][q]];
                in += ctl->cand_n[rm.rules_in[s][q]];
            }
            // relation::insert_delta_in_full + local_insert_in_delta
            if (ctl->delta_n[s]) ctl->runs[s]++;
            ctl->full_n[s] += ctl->delta_n[s];
            ctl->delta_n[s] = nn;
            ctl->seen_n[s] += nn;
            added += nn;
            sum_delta += ctl->delta_n[s];
            sum_full += ctl->full_n[s];
            if (rm.n_rules_in[s] && ctl->seen_n[s] + 2 * in > plan.seen_limit[s]) grow = true;
        }
        u64 tag_add[kMaxTagSlots] = {0};
        for (int r = 0; r < plan.n_rules; r++) tag_add[plan.rule_tag[r]] += ctl->win_n[r];
        for (int t = 0; t < kMaxTagSlots; t++) ctl->intern[t] += tag_add[t];
        u64 cands = 0;
        for (int r = 0; r < plan.n_rules; r++) cands += ctl->cand_n[r];
        ctl->candidates += cands;
        ctl->new_tuples += added;
        ctl->bit_filter = 4 * added < 3 * cands;
        ctl->last_time = global_ns();
        if (ctl->iteration < ctl->time_cap) history[2 * plan.hist_cap + ctl->iteration] = ctl->last_time;
        ctl->iteration++;
        ctl->epoch++;
        ctl->batch_pos++;
        cont = true;
        if (records) {
            ctl->batch_pos = 0;
            history[2 * ctl->hist_n] = ctl->last_delta = sum_delta;
            history[2 * ctl->hist_n + 1] = ctl->last_full = sum_full;
            ctl->hist_n++;
            cont = plan.fixpoint && sum_delta != 0;
        }
        if (ctl->iteration >= plan.iter_limit) cont = false;
        ctl->done = cont ? 0u : 1u;
        if (cont && grow) {
            atomicOr(&ctl->flags, kFlagGrow);
            cont = false;
        }
        // the next iteration's bank of tile counters (used last by the previous iteration)
        for (int i = 0; i < kBankWords; i++) ctl->tile_ctr[(ctl->iteration & 1) * kBankWords + i] = 0;
        ctl->heavy_n = 0;
        ctl->heavy_ctr = 0;
    }
    if (use_cond) cudaGraphSetConditional(cond, cont ? 1u : 0u);
}

// The iteration end by one block, on a copy of the control block in shared memory (`buf`,
// kEndWords u64): some fifty dependent reads and writes of one thread cost as many L2 round
// trips in place, 5 to 8 us; here two, to fetch the block and to put it back.  Called by
// every thread of the launch's last block, when no other block touches the control block
// any more; tail, when given, decides on the result whether the loop stops for the tail
// kernel.
constexpr int kEndWords = (int)(offsetof(IterCtl, bar_count) / 8);
template <typename Tail>
__device__ __forceinline__ void end_of_iteration_block(IterCtl* __restrict__ ctl, u64* buf, const SccPlan& plan,
                                                       const SccRelMap& rm, u64* __restrict__ history,
                                                       cudaGraphConditionalHandle cond, int use_cond, Tail tail)
{
    u64* g = (u64*)ctl;
    for (int i = threadIdx.x; i < kEndWords; i += kThreads) buf[i] = __ldcg(&g[i]);
    __syncthreads();
    if (threadIdx.x == 0) {
        IterCtl* L = (IterCtl*)buf;
        L->exit_ctr = 0;   // the launch is over
        end_of_iteration(L, plan, rm, history, cond, use_cond);
        if (use_cond && tail(L)) cudaGraphSetConditional(cond, 0u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kEndWords; i += kThreads) __stcg(&g[i], buf[i]);
}

// The last of `parting` blocks to get here (after its writes); uniform over the block.
__device__ __forceinline__ bool last_block(IterCtl* __restrict__ ctl, u32 parting)
{
    __shared__ u32 s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&ctl->exit_ctr, 1u) == parting - 1;
        if (s_last) {
            __threadfence();
            atomicExch(&ctl->exit_ctr, 0u);
        }
    }
    __syncthreads();
    return s_last != 0;
}

// ---------------------------------------------------------------------------
// select: winners in candidate order -> the relation's log (emission ids) or
// its staging rows (reference ids, sorted afterwards)
// ---------------------------------------------------------------------------
constexpr int kSelIpt = RA_SELECT_IPT;
constexpr int kSelTile = kThreads * kSelIpt;

struct SelectArgs {
    int rule;
    int last;                 // last rule of the iteration: runs the iteration end
    u64* dst_keys;            // log (to_log) or staging rows
    u64* dst_ids;
    int to_log;
    int passes;               // digit histograms to accumulate (reference ids)
    int last_shift;           // shift of the last of them
    u64 stage_cap;
    // a slice of the rule's outer rows: candidates at buffer index 0; `appended` winners of
    // this iteration already in the relation's log (earlier rules and slices), `id_appended`
    // already numbered under the rule's tag; the iteration end runs after the last slice
    int sliced;
    u64 appended, id_appended;
    // instance accounting (batched programs): instance i owns values [inst_base[i], inst_base[i+1])
    const u64* inst_base;     // n_inst + 1 entries, or null
    u32 n_inst;
    int inst_shift;           // bit offset of column 0 in the output relation's key
    u64* inst_new;            // [iteration][instance] counts of new tuples
    u64 inst_iter_cap;
    // the tail kernel (ra_tail.cuh) follows the graph's WHILE loop: the iteration end
    // stops the loop when every join rule's next outer delta has at most tail_rows rows
    int tail_on;
    int tail_nslots;
    int tail_slot[kTailMaxRules];
    u64 tail_rows;
};

// Does the next iteration go to the tail kernel?  (After the iteration end: not
// done, no flag, every join rule's next delta small.)
__device__ __forceinline__ bool tail_next(const IterCtl* c, const SelectArgs& a)
{
    bool small = c->flags == 0 && c->done == 0 && c->tail_off == 0;
    for (int i = 0; i < a.tail_nslots; i++) small = small && c->delta_n[a.tail_slot[i]] <= a.tail_rows;
    return small;
}

// instance owning value v (inst_base sorted, n + 1 entries)
__device__ __forceinline__ u32 instance_of(const u64* __restrict__ base, u32 n, u64 v)
{
    u32 lo = 0, hi = n;   // base[lo] <= v < base[hi]
    while (hi - lo > 1) {
        const u32 mid = (lo + hi) >> 1;
        if (__ldg(&base[mid]) <= v) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Per-row tables of the instances' bit matrices: row v of instance i (values
// base[i] .. min(base[i + 1], rows) - 1, words w_i = ceil(n_i / 32) per row) starts at
// word inst_word[i] + (v - base[i]) * w_i.  `base` holds n_inst + 1 entries (a sentinel last).
__global__ void __launch_bounds__(kThreads) bitmap_tables_kernel(const u64* __restrict__ base, u32 n_inst,
                                                                 const u64* __restrict__ inst_word, u64 rows,
                                                                 u64* __restrict__ row_word, u32* __restrict__ row_base,
                                                                 u32* __restrict__ row_words, u32* __restrict__ row_inst)
{
    for (u64 v = (u64)blockIdx.x * kThreads + threadIdx.x; v < rows; v += (u64)gridDim.x * kThreads) {
        const u32 i = instance_of(base, n_inst, v);
        const u64 b = base[i], e = min(base[i + 1], rows), w = v < b ? 0 : (e - b + 31) / 32;
        // a value below the first instance has no words: every tuple on its row is out of range
        row_word[v] = v < b ? 0 : inst_word[i] + (v - b) * w;
        row_base[v] = (u32)b;
        row_words[v] = (u32)w;
        row_inst[v] = i;
    }
}

__global__ void __launch_bounds__(kThreads, RA_SELECT_MIN_BLOCKS) select_kernel(IterCtl* __restrict__ ctl,
                                                          // read in place from the parameter space (indexed by rule / relation)
                                                          const __grid_constant__ SccPlan plan,
                                                          const __grid_constant__ SccRelMap rm,
                                                          const __grid_constant__ SelectArgs a, const u64* __restrict__ cand,
                                                          const u32* __restrict__ loser,
                                                          u64* __restrict__ status, int tile_slot,
                                                          u64* __restrict__ history, cudaGraphConditionalHandle cond,
                                                          int use_cond)
{
    static_assert(kSelIpt == 4, "select loads a thread's candidates as 2 x 16 bytes and its marks as 16 bytes");
    __shared__ u64 sm[kWarps + 1];
    __shared__ u32 s_tile;
    __shared__ u64 s_prefix;
    __shared__ u32 s_hist[kMaxPasses][kRadix];
    __shared__ u64 s_win[kSelTile];   // the tile's winners, compacted, for coalesced stores
    if (ctl->done) return;   // the tail kernel reached the fixed point in this body
    const int rule = a.rule;
    const u64 c = ctl->cand_n[rule];
    const int out = plan.rule_out[rule], tslot = plan.rule_tag[rule];
    bool active = ctl->flags == 0;
    if (active) {
        // Room for every candidate of every rule of the iteration, checked by every select
        // before any write, so that an iteration either writes all its winners or none
        // (a replay then never counts a winner twice).  The new delta lands in the log
        // either way (directly, or via staging + sort).
        bool over = a.inst_base && ctl->iteration >= a.inst_iter_cap;
        if (a.sliced) {
            const int s = plan.rule_out[rule];
            over = over || ctl->full_n[s] + ctl->delta_n[s] + a.appended + ctl->cand_n[rule] > plan.log_cap[s];
        } else {
            for (int s = 0; s < plan.n_rels; s++) {
                u64 incoming = 0;
                for (int q = 0; q < rm.n_rules_in[s]; q++) incoming += ctl->cand_n[rm.rules_in[s][q]];
                if (!incoming) continue;
                over = over || ctl->full_n[s] + ctl->delta_n[s] + incoming > plan.log_cap[s] ||
                       (!a.to_log && incoming > a.stage_cap);
            }
        }
        if (over) {
            if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&ctl->flags, kFlagOverflow);
            active = false;
        }
    }
    if (c == 0 && blockIdx.x == 0 && threadIdx.x == 0) ctl->win_n[rule] = 0;
    const u64 ntiles = (c + kSelTile - 1) / kSelTile;
    if (active && c > 0 && blockIdx.x < ntiles) {
        // destination offset and intern base: winners of earlier rules into the same relation / tag
        u64 dst_off = 0, id_ctr = ctl->intern[tslot];
        if (a.sliced) {
            dst_off = a.appended;
            id_ctr += a.id_appended;
        } else {
            for (int q = 0; q < rule; q++) {
                if (plan.rule_out[q] == out) dst_off += ctl->win_n[q];
                if (plan.rule_tag[q] == tslot) id_ctr += ctl->win_n[q];
            }
        }
        u64* dk = a.dst_keys;
        u64* dv = a.dst_ids;
        if (a.to_log) dst_off += ctl->full_n[out] + ctl->delta_n[out];
        const u64 tag_word = plan.rel_tag_word[out];
        const u64 cbase = a.sliced ? 0 : stream_base(ctl, rule);
        const u32 ep = (u32)ctl->epoch;
        const u64* in = cand + cbase;
        const bool aligned = (cbase & 3) == 0;   // 16-byte vector loads of candidates and marks
        const u32 tag = iter_tag(ctl, tile_slot);
        u32* ctr = tile_counter(ctl, tile_slot);
        for (int i = threadIdx.x; i < a.passes * kRadix; i += kThreads) (&s_hist[0][0])[i] = 0;
        for (;;) {
            if (threadIdx.x == 0) s_tile = atomicAdd(ctr, 1u);
            __syncthreads();
            const u64 tile = s_tile;
            __syncthreads();
            if (tile >= ntiles) break;
            const u64 base = tile * kSelTile + (u64)threadIdx.x * kSelIpt;
            u64 key[kSelIpt];
            u32 mk[kSelIpt];
            if (aligned && base + kSelIpt <= c) {
                // a thread's 4 candidates and their marks in three 16-byte loads
                const ulonglong2 k01 = *(const ulonglong2*)(in + base), k23 = *(const ulonglong2*)(in + base + 2);
                const uint4 m = *(const uint4*)(loser + cbase + base);
                key[0] = k01.x; key[1] = k01.y; key[2] = k23.x; key[3] = k23.y;
                mk[0] = m.x; mk[1] = m.y; mk[2] = m.z; mk[3] = m.w;
            } else {
#pragma unroll
                for (int k = 0; k < kSelIpt; k++) {
                    const bool v = base + k < c;
                    key[k] = v ? in[base + k] : kEmpty;
                    mk[k] = v ? loser[cbase + base + k] : ep;
                }
            }
            u32 win = 0;
#pragma unroll
            for (int k = 0; k < kSelIpt; k++) {
                if (key[k] == kEmpty || mk[k] == ep) key[k] = kEmpty;
                else win++;
            }
            u64 agg;
            const u64 ex = block_exclusive_scan((u64)win, sm, &agg);
            if (threadIdx.x < 32) {
                const u64 pre = lookback_warp(status, (u32)tile, agg, tag, &ctl->flags);
                if (threadIdx.x == 0) s_prefix = pre;
            }
            {   // compacted into shared memory meanwhile
                u64 e = ex;
#pragma unroll
                for (int k = 0; k < kSelIpt; k++)
                    if (key[k] != kEmpty) s_win[e++] = key[k];
            }
            __syncthreads();
            const u64 pre = s_prefix;
            // the tile's winners: log rows dst_off + pre + i, consecutive threads, consecutive rows
            for (u32 i = threadIdx.x; i < agg; i += kThreads) {
                const u64 kk = s_win[i];
                const u64 r = pre + i;
                dk[dst_off + r] = kk;
                dv[dst_off + r] = tag_word | (id_ctr + r);
                for (int ps = 0; ps < a.passes; ps++)
                    atomicAdd(&s_hist[ps][(kk >> min(ps * kRadixBits, a.last_shift)) & (kRadix - 1)], 1u);
            }
            if (a.inst_base) {
                u64* row = a.inst_new + ctl->iteration * a.n_inst;
                for (u32 i0 = 0; i0 < agg; i0 += kThreads) {   // warp-uniform trip count
                    const u32 i = i0 + threadIdx.x;
                    const bool v = i < agg;
                    const u32 inst = v ? instance_of(a.inst_base, a.n_inst, s_win[i] >> a.inst_shift)
                                       : (0x80000000u | (u32)threadIdx.x);
                    const u32 peers = __match_any_sync(0xffffffffu, inst);
                    if (v && (peers & lanemask_lt()) == 0) atomicAdd(&row[inst], (u64)__popc(peers));
                }
            }
            if (tile == ntiles - 1 && threadIdx.x == 0) ctl->win_n[rule] = s_prefix + agg;
            __syncthreads();
        }
        if (a.passes) {
            __syncthreads();
            for (int i = threadIdx.x; i < a.passes * kRadix; i += kThreads) {
                const u32 v = (&s_hist[0][0])[i];
                if (v) atomicAdd(&ctl->sort_hist[out][i / kRadix][i % kRadix], (u64)v);
            }
        }
    }
    // the last block to finish runs the iteration end (after every write of this launch);
    // blocks past the last tile never write, so only min(grid, tiles) blocks take part
    const u32 parting = (u32)min((u64)gridDim.x, (active && c > 0) ? ntiles : (u64)1);
    if (blockIdx.x >= parting) return;
    static_assert(kEndWords <= kSelTile, "s_win holds the control block");
    if (last_block(ctl, parting) && a.last)
        end_of_iteration_block(ctl, s_win, plan, rm, history, cond, use_cond,
                               [&](const IterCtl* c) { return a.tail_on && tail_next(c, a); });
}

// ---------------------------------------------------------------------------
// radix launches over a relation's staged rows
// ---------------------------------------------------------------------------
constexpr int kSortIpt = 8;
constexpr int kSortTile = kThreads * kSortIpt;

// ---------------------------------------------------------------------------
// bitmap_select: the new tuples of a bitmap relation (all rules into it at
// once) into its log, in key order, a warp per row (or a few narrow rows).  A row's words
// are read kBitBatch to a lane, so a row of 1,024 words costs four round trips, and only its
// 32-word groups with new tuples are read again to be written out (emit_words).  Bound by
// those round trips and the look-back of each tile; the log's 16 bytes per tuple are a third of
// its time.  Measured on a tree of 2^15 nodes, together with the `seen` update that the
// claims made before: 5.2 -> 3.7 ms.
// Takes part in the iteration like select_kernel: the same capacity check before any
// write, the same exit counter, the iteration end when it is the iteration's last launch.
// ---------------------------------------------------------------------------
constexpr int kBitSelRows = 16;  // rows a warp takes at most
constexpr int kBitBatch = 8;

struct BitSelectArgs {
    int rel;          // output relation slot
    int first_rule;   // the relation's first rule: credited with all its new tuples
    int last;         // this launch ends the iteration
    u64* dst_keys;
    u64* dst_ids;
    BitSeen bs;
    int rows_per_warp;   // of a tile (a tile's look-back then serves that many rows per warp)
    int bits;         // packed column width
    u64* inst_new;    // [iteration][instance] new tuples (with instances), else null
    u32 n_inst;
    u64 inst_iter_cap;
};

__global__ void __launch_bounds__(kThreads) bitmap_select_kernel(IterCtl* __restrict__ ctl,
                                                                 const __grid_constant__ SccPlan plan,
                                                                 const __grid_constant__ SccRelMap rm,
                                                                 const __grid_constant__ BitSelectArgs a, u64* __restrict__ status,
                                                                 u64 status_cap, int tile_slot, u64* __restrict__ history,
                                                                 cudaGraphConditionalHandle cond, int use_cond)
{
    __shared__ u64 sm[kWarps + 1];
    __shared__ u64 s_cnt[kWarps];
    __shared__ u32 s_tile;
    __shared__ u64 s_prefix;
    __shared__ u32 s_rows[kWarps][kBitSelRows];     // new tuples of a warp's rows
    __shared__ u64 s_groups[kWarps][kBitSelRows];   // and their groups
    __shared__ u64 s_end[kEndWords];
    const int out = a.rel, tslot = plan.rule_tag[a.first_rule];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u64 rows = a.bs.n;
    const int rpw = a.rows_per_warp;
    const u64 ntiles = (rows + kWarps * rpw - 1) / (kWarps * rpw);
    bool active = ctl->flags == 0;
    if (active && ntiles > status_cap) {   // never taken: status is sized for the rows
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&ctl->flags, kFlagStatus);
        active = false;
    }
    if (active) {
        // select_kernel's check: room for every candidate of the iteration
        bool over = a.inst_new && ctl->iteration >= a.inst_iter_cap;
        for (int s = 0; s < plan.n_rels; s++) {
            u64 incoming = 0;
            for (int q = 0; q < rm.n_rules_in[s]; q++) incoming += ctl->cand_n[rm.rules_in[s][q]];
            if (incoming && ctl->full_n[s] + ctl->delta_n[s] + incoming > plan.log_cap[s]) over = true;
        }
        if (over) {
            if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&ctl->flags, kFlagOverflow);
            active = false;
        }
    }
    if (active && blockIdx.x < ntiles) {
        u64 dst_off = ctl->full_n[out] + ctl->delta_n[out], id_ctr = ctl->intern[tslot];
        for (int q = 0; q < a.first_rule; q++)
            if (plan.rule_tag[q] == tslot) id_ctr += ctl->win_n[q];
        const u64 tag_word = plan.rel_tag_word[out];
        const u32 tag = iter_tag(ctl, tile_slot);
        u32* ctr = tile_counter(ctl, tile_slot);
        for (;;) {
            if (threadIdx.x == 0) s_tile = atomicAdd(ctr, 1u);
            __syncthreads();
            const u64 tile = s_tile;
            __syncthreads();
            if (tile >= ntiles) break;
            const u64 row0 = (tile * kWarps + warp) * rpw;
            // the rows' new tuples: fresh bits not yet seen; known ones leave `fresh` here
            u32 mine = 0;
            const u32 dirty = __ballot_sync(0xffffffffu, lane < rpw && row0 + lane < rows && a.bs.dirty[row0 + lane]);
            for (u32 dm = dirty; dm; dm &= dm - 1) {
                const int r = __ffs(dm) - 1;
                const u64 row = row0 + r;
                u32 cnt = 0;
                u64 groups = 0;   // 32-word groups of the row that hold some (2,048 words at most)
                const u64 W = a.bs.row_word ? a.bs.row_words[row] : a.bs.words;
                const u64 f0 = a.bs.row_word ? a.bs.row_word[row] : row * W;
                for (u64 g = 0; g < W; g += 32 * kBitBatch) {   // kBitBatch words of a lane in flight
                    u32 f[kBitBatch], sw[kBitBatch], some = 0;
#pragma unroll
                    for (int q = 0; q < kBitBatch; q++) {
                        const u64 w = g + q * 32 + lane;
                        f[q] = w < W ? a.bs.fresh[f0 + w] : 0u;
                        some |= f[q];
                    }
                    if (!__any_sync(0xffffffffu, some != 0)) continue;
#pragma unroll
                    for (int q = 0; q < kBitBatch; q++) sw[q] = f[q] ? a.bs.seen[f0 + g + q * 32 + lane] : 0u;
#pragma unroll
                    for (int q = 0; q < kBitBatch; q++) {
                        const u64 w = f0 + g + q * 32 + lane;
                        const u32 nw = f[q] & ~sw[q];
                        if (nw) a.bs.seen[w] = sw[q] | nw;
                        if (nw != f[q]) a.bs.fresh[w] = nw;
                        if (__any_sync(0xffffffffu, nw != 0)) groups |= 1ull << ((g >> 5) + q);
                        cnt += __popc(nw);
                    }
                }
                cnt = __reduce_add_sync(0xffffffffu, cnt);
                mine += cnt;
                if (lane == 0) {
                    s_rows[warp][r] = cnt;
                    s_groups[warp][r] = groups;
                }
            }
            if (lane == 0) s_cnt[warp] = mine;
            __syncthreads();
            u64 agg;
            const u64 ex = block_exclusive_scan(threadIdx.x < kWarps ? s_cnt[threadIdx.x] : 0, sm, &agg);
            __syncthreads();
            if (threadIdx.x < kWarps) s_cnt[threadIdx.x] = ex;   // warp offsets inside the tile
            if (threadIdx.x < 32) {
                const u64 pre = lookback_warp(status, (u32)tile, agg, tag, &ctl->flags);
                if (threadIdx.x == 0) s_prefix = pre;
            }
            __syncthreads();
            __syncwarp();
            u64 pos = s_prefix + s_cnt[warp];
            for (u32 dm = dirty; dm; dm &= dm - 1) {
                const int r = __ffs(dm) - 1;
                const u64 row = row0 + r;
                const u64 W = a.bs.row_word ? a.bs.row_words[row] : a.bs.words;
                const u64 vbase = a.bs.row_word ? a.bs.row_base[row] : 0;
                u32* frow = a.bs.fresh + (a.bs.row_word ? a.bs.row_word[row] : row * W);
                u64 gm = s_groups[warp][r];
                u64 g = gm ? (u64)(__ffsll((long long)gm) - 1) * 32 : 0;
                u32 ahead = (gm && g + lane < W) ? frow[g + lane] : 0u;
                while (gm) {
                    const u32 word = ahead;
                    const u64 g_now = g;
                    gm &= gm - 1;
                    if (gm) {   // the next group's words, on their way meanwhile
                        g = (u64)(__ffsll((long long)gm) - 1) * 32;
                        ahead = g + lane < W ? frow[g + lane] : 0u;
                    }
                    if (word) frow[g_now + lane] = 0u;
                    pos += emit_words(word, [&](u32 t, u32 bit) {
                        a.dst_keys[dst_off + pos + t] = (row << a.bits) | (vbase + g_now * 32 + bit);
                        a.dst_ids[dst_off + pos + t] = tag_word | (id_ctr + pos + t);
                    });
                }
                if (lane == 0) {
                    a.bs.dirty[row] = 0;
                    if (a.inst_new && s_rows[warp][r])
                        atomicAdd((unsigned long long*)&a.inst_new[ctl->iteration * a.n_inst + a.bs.row_inst[row]],
                                  (unsigned long long)s_rows[warp][r]);
                }
            }
            if (tile == ntiles - 1 && threadIdx.x == 0) {
                ctl->win_n[a.first_rule] = s_prefix + agg;
                for (int q = 0; q < rm.n_rules_in[out]; q++)
                    if (rm.rules_in[out][q] != a.first_rule) ctl->win_n[rm.rules_in[out][q]] = 0;
            }
            __syncthreads();
        }
    }
    const u32 parting = (u32)min((u64)gridDim.x, active ? ntiles : (u64)1);
    if (blockIdx.x >= parting) return;
    if (last_block(ctl, parting) && a.last)
        end_of_iteration_block(ctl, s_end, plan, rm, history, cond, use_cond, [](const IterCtl*) { return false; });
}

struct SortPassArgs {
    int rel;                  // relation slot
    int pass, shift;
    const u64* src_k;
    const u64* src_v;
    u64* dst_k;               // when dst_log: the log base (rows go to base + full_n + delta_n)
    u64* dst_v;
    int dst_log;
    u64 log_cap;              // rows the relation's log holds
    int buckets;              // the relation sorts in two launches when sort_fits
    int last_pass, last_shift;   // the top digit's pass and shift
    u64* log_k;               // the log base, for the second of those launches
    u64* log_v;
    int n_rules_in;           // rules writing this relation
    int rules_in[kMaxSccRules];
};

// The tiles of one onesweep LSD radix pass: (k, v) rows from src to dst, stably by digit
// (k >> shift) & 255, given the digits' counts over all n rows.  Tiles are taken from tile_ctr; a
// tile ranks its rows by warp matches, looks back over the earlier tiles for each digit's
// position and writes each digit's run together.
struct SortSmem {
    u64 gstart[kRadix];         // global start of each digit (exclusive scan of the counts)
    u64 out[kRadix];            // output position of each digit's run in this tile
    u32 loc[kRadix];            // tile-local start of each digit's run
    u32 wcnt[kWarps][kRadix];   // per-warp digit counts, then per-warp bases
    u64 k[kSortTile];           // the tile, in digit order
    u64 v[kSortTile];
    u64 sm[kWarps + 1];
    u32 tile;
};

// Ranks the tn rows held by the block (kk, thread order of sort_tiles) by digit: rk[r] counts the
// row's equals before it in its warp, S.loc[d] is digit d's first place and S.wcnt[w][d] the
// warp's share before it.  S.wcnt is zero and synchronised on entry.  Returns the count of
// digit threadIdx.x.
__device__ __forceinline__ u32 sort_rank(SortSmem& S, const u64 (&kk)[kSortIpt], u32 (&rk)[kSortIpt], u32 tn, int shift)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int r = 0; r < kSortIpt; r++) {
        const u32 li = (u32)(warp * 32 * kSortIpt + r * 32 + lane);
        const bool valid = li < tn;
        const int d = valid ? (int)((kk[r] >> shift) & (kRadix - 1)) : (kRadix + lane);
        const u32 peers = __match_any_sync(0xffffffffu, d);
        const u32 before = __popc(peers & lanemask_lt());
        const u32 prior = valid ? S.wcnt[warp][d] : 0;
        __syncwarp();
        if (valid && before == 0) S.wcnt[warp][d] = prior + __popc(peers);
        __syncwarp();
        rk[r] = prior + before;
    }
    __syncthreads();
    // digit totals of the tile -> tile-local run starts; per-warp bases inside each run
    const int d = threadIdx.x;   // kThreads == kRadix
    u32 run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        const u32 c = S.wcnt[w][d];
        S.wcnt[w][d] = run;
        run += c;
    }
    u64 tot;
    S.loc[d] = (u32)block_exclusive_scan((u64)run, S.sm, &tot);
    return run;
}

// Places the ranked rows in shared memory in digit order (stable).  S.loc and S.wcnt synchronised.
__device__ __forceinline__ void sort_put(SortSmem& S, const u64 (&kk)[kSortIpt], const u64 (&vv)[kSortIpt],
                                         const u32 (&rk)[kSortIpt], u32 tn, int shift)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int r = 0; r < kSortIpt; r++) {
        const u32 li = (u32)(warp * 32 * kSortIpt + r * 32 + lane);
        if (li >= tn) continue;
        const int dd = (int)((kk[r] >> shift) & (kRadix - 1));
        const u32 pos = S.loc[dd] + S.wcnt[warp][dd] + rk[r];
        S.k[pos] = kk[r];
        S.v[pos] = vv[r];
    }
}

template <typename Timeout>
__device__ __forceinline__ void sort_tiles(SortSmem& S, const u64* __restrict__ src_k, const u64* __restrict__ src_v,
                                           u64* __restrict__ dk, u64* __restrict__ dv, u64 n, int shift,
                                           const u64* __restrict__ counts, u32* __restrict__ tile_ctr,
                                           u64* __restrict__ status, u32 tag, u64 limit, Timeout timeout)
{
    const u64 ntiles = (n + kSortTile - 1) / kSortTile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        u64 tot;
        S.gstart[threadIdx.x] = block_exclusive_scan(counts[threadIdx.x], S.sm, &tot);
    }
    for (;;) {
        if (threadIdx.x == 0) S.tile = atomicAdd(tile_ctr, 1u);
        for (int i = threadIdx.x; i < kWarps * kRadix; i += kThreads) (&S.wcnt[0][0])[i] = 0;
        __syncthreads();
        const u64 tile = S.tile;
        if (tile >= ntiles) break;
        const u64 t0 = tile * kSortTile;
        const u32 tn = (u32)min((u64)kSortTile, n - t0);
        // warp w owns items [w*32*IPT, (w+1)*32*IPT) of the tile, round-major = index order
        u64 kk[kSortIpt], vv[kSortIpt];
        u32 rk[kSortIpt];
#pragma unroll
        for (int r = 0; r < kSortIpt; r++) {   // every load of the tile in flight before the ranking rounds
            const u32 li = (u32)(warp * 32 * kSortIpt + r * 32 + lane);
            kk[r] = li < tn ? src_k[t0 + li] : 0;
            vv[r] = li < tn ? src_v[t0 + li] : 0;
        }
        const int d = threadIdx.x;   // kThreads == kRadix
        const u32 run = sort_rank(S, kk, rk, tn, shift);
        // look-back for this digit across tiles (one thread per digit)
        u64* st = status + tile * kRadix + d;
        u64 excl = 0;
        if (tile == 0) {
            st_publish(st, st_pack(tag, kStIncl, run));
        } else {
            st_publish(st, st_pack(tag, kStAgg, run));
            long t = (long)tile - 1;
            u64 spins = 0;
            while (t >= 0) {
                const u64 sv = st_read(status + (u64)t * kRadix + d);
                if (st_tag(sv) != (tag & 0xffffffu) || st_flag(sv) == 0 || limit == 0) {
                    if (++spins > limit) {
                        timeout();
                        break;
                    }
                    continue;
                }
                excl += st_val(sv);
                if (st_flag(sv) == kStIncl) break;
                t--;
            }
            st_publish(st, st_pack(tag, kStIncl, excl + run));
        }
        S.out[d] = S.gstart[d] + excl;
        __syncthreads();
        sort_put(S, kk, vv, rk, tn, shift);
        __syncthreads();
        // each digit's run is contiguous in the output: coalesced writes
        for (u32 q = threadIdx.x; q < tn; q += kThreads) {
            const u64 k = S.k[q];
            const int dd = (int)((k >> shift) & (kRadix - 1));
            const u64 pos = S.out[dd] + (q - S.loc[dd]);
            dk[pos] = k;
            dv[pos] = S.v[q];
        }
        __syncthreads();
    }
}

// The rows of the top digits' buckets (from `src`, bucket after bucket) to dk / dv in key order: a
// block per bucket, by comparing each row with all others (up to kSortCompare rows: one pass, a
// few compares per row and cycle) or digit by digit in shared memory.
constexpr u32 kSortCompare = 512;
__device__ __forceinline__ void sort_buckets(SortSmem& S, const u64* __restrict__ src_k, const u64* __restrict__ src_v,
                                             u64* __restrict__ dk, u64* __restrict__ dv, u32 count, int top_shift)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u64 tot;
    S.gstart[threadIdx.x] = block_exclusive_scan((u64)count, S.sm, &tot);
    S.out[threadIdx.x] = count;
    __syncthreads();
    for (int b = blockIdx.x; b < kRadix; b += gridDim.x) {
        const u32 tn = (u32)S.out[b];   // at most kSortTile (sort_fits)
        const u64 at = S.gstart[b];
        if (tn == 0) continue;
        if (tn <= kSortCompare) {
            constexpr int kOwn = kSortCompare / kThreads;
            u64 k[kOwn], v[kOwn];
            u32 less[kOwn];
#pragma unroll
            for (int e = 0; e < kOwn; e++) {
                const u32 i = threadIdx.x + e * kThreads;
                k[e] = i < tn ? src_k[at + i] : ~0ull;
                v[e] = i < tn ? src_v[at + i] : 0;
                S.k[i] = k[e];
                less[e] = 0;
            }
            __syncthreads();
            if (warp * 32 < tn)
                for (u32 j = 0; j < tn; j++) {
                    const u64 o = S.k[j];
#pragma unroll
                    for (int e = 0; e < kOwn; e++)
                        less[e] += o < k[e] || (o == k[e] && j < threadIdx.x + e * kThreads);
                }
#pragma unroll
            for (int e = 0; e < kOwn; e++)
                if (threadIdx.x + e * kThreads < tn) {
                    dk[at + less[e]] = k[e];
                    dv[at + less[e]] = v[e];
                }
        } else {
            u64 kk[kSortIpt], vv[kSortIpt];
            u32 rk[kSortIpt];
            for (int shift = 0; shift < top_shift; shift += kRadixBits) {
#pragma unroll
                for (int r = 0; r < kSortIpt; r++) {
                    const u32 li = (u32)(warp * 32 * kSortIpt + r * 32 + lane);
                    kk[r] = li < tn ? (shift ? S.k[li] : src_k[at + li]) : 0;
                    vv[r] = li < tn ? (shift ? S.v[li] : src_v[at + li]) : 0;
                }
                for (int i = threadIdx.x; i < kWarps * kRadix; i += kThreads) (&S.wcnt[0][0])[i] = 0;
                __syncthreads();
                sort_rank(S, kk, rk, tn, shift);
                __syncthreads();
                sort_put(S, kk, vv, rk, tn, shift);
                __syncthreads();
            }
            for (u32 q = threadIdx.x; q < tn; q += kThreads) {
                dk[at + q] = S.k[q];
                dv[at + q] = S.v[q];
            }
        }
        __syncthreads();
    }
}

// One launch of a new delta's sort (reference id order).  By digits, lowest first, a launch per
// digit; when no top digit has more than kSortTile rows, the first launch instead parts the rows
// by their top digit, the second sorts every bucket in shared memory into the log, and the others
// return at once.  Bound by each launch's chain of round trips (a few thousand to a hundred
// thousand rows).  Transitive closure of 100,003 values and 95,000 edges, 78 deltas of 34-bit keys:
// 5.89 -> 4.11 ms for the fixed point against five digit launches each.
__global__ void __launch_bounds__(kThreads) sort_pass_kernel(IterCtl* __restrict__ ctl,
                                                             const __grid_constant__ SortPassArgs a,
                                                             u64* __restrict__ status, int tile_slot)
{
    __shared__ SortSmem S;
    const u32 top = a.buckets ? (u32)min(ctl->sort_hist[a.rel][a.last_pass][threadIdx.x], (u64)kSortTile + 1) : 0u;
    if (ctl->flags) return;
    u64 n = 0;
    for (int q = 0; q < a.n_rules_in; q++) n += ctl->win_n[a.rules_in[q]];
    if (n == 0) return;
    const u64 ntiles = (n + kSortTile - 1) / kSortTile;
    if (blockIdx.x >= max(ntiles, (u64)(a.buckets && a.pass == 1 ? kRadix : 0))) return;
    u64* dk = a.dst_k;
    u64* dv = a.dst_v;
    const bool fits = a.buckets && !__syncthreads_or(top > kSortTile);
    if (fits && a.pass > 1) return;
    if (fits && a.pass == 1) {
        const u64 o = ctl->full_n[a.rel] + ctl->delta_n[a.rel];
        if (o + n > a.log_cap) {   // as below
            if (threadIdx.x == 0) atomicOr(&ctl->flags, kFlagOverflow);
            return;
        }
        sort_buckets(S, a.src_k, a.src_v, a.log_k + o, a.log_v + o, top, a.last_shift);
        return;
    }
    if (blockIdx.x >= ntiles) return;
    const int pass = fits ? a.last_pass : a.pass;
    if (a.dst_log) {
        const u64 o = ctl->full_n[a.rel] + ctl->delta_n[a.rel];
        if (o + n > a.log_cap) {   // select checks this first; never write past the log
            if (threadIdx.x == 0) atomicOr(&ctl->flags, kFlagOverflow);
            return;
        }
        dk += o;
        dv += o;
    }
    sort_tiles(S, a.src_k, a.src_v, dk, dv, n, fits ? a.last_shift : a.shift, ctl->sort_hist[a.rel][pass],
               tile_counter(ctl, tile_slot),
               status, iter_tag(ctl, tile_slot), kSpinLimit, [&] { atomicOr(&ctl->flags, kFlagTimeout); });
}

// A whole array's radix sort (loading, sorted views): every pass's digit counts in one read,
// then a pass per digit.  Bound by the tiles' look-backs (128 MB per pass at 4M rows in 85 us).
// Against counting, scanning (three launches) and scattering per pass: 4M rows of 44 bits 675 ->
// 525 us in 7 launches instead of 30; 1.4M rows of 34 bits, 250 -> 240.
__global__ void __launch_bounds__(kThreads) sort_counts_kernel(const u64* __restrict__ keys, u64 n, int lo, int passes,
                                                               u64* __restrict__ counts)
{
    __shared__ u32 s[8][kRadix];   // a block's share stays below 2^32
    for (int i = threadIdx.x; i < passes * kRadix; i += kThreads) (&s[0][0])[i] = 0;
    __syncthreads();
    constexpr int kAhead = 4;
    const u64 step = (u64)gridDim.x * kThreads * kAhead;
    for (u64 i0 = (u64)blockIdx.x * kThreads * kAhead + threadIdx.x; i0 < n; i0 += step) {
        u64 k[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; u++) k[u] = i0 + u * kThreads < n ? keys[i0 + u * kThreads] : 0;
#pragma unroll
        for (int u = 0; u < kAhead; u++)
            if (i0 + u * kThreads < n)
                for (int p = 0; p < passes; p++) atomicAdd(&s[p][(k[u] >> (lo + p * kRadixBits)) & (kRadix - 1)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * kRadix; i += kThreads) {
        const u32 c = (&s[0][0])[i];
        if (c) atomicAdd((unsigned long long*)&counts[i], (unsigned long long)c);
    }
}

// A look-back that gives up (after `limit` polls) tells the host, and the sort's later passes: a
// pass that lacks some of its prefixes writes within the array, but leaves rows of other digits than
// were counted, which the next pass would place beyond it.
__global__ void __launch_bounds__(kThreads) sort_array_kernel(const u64* __restrict__ src_k, const u64* __restrict__ src_v,
                                                              u64* __restrict__ dk, u64* __restrict__ dv, u64 n,
                                                              int shift, const u64* __restrict__ counts,
                                                              u32* __restrict__ tile_ctr, u64* __restrict__ status,
                                                              u32 tag, u64 limit, u64* gave_up, u64* host_timeout)
{
    __shared__ SortSmem S;
    if (__syncthreads_or(threadIdx.x == 0 && *(volatile u64*)gave_up)) return;
    sort_tiles(S, src_k, src_v, dk, dv, n, shift, counts, tile_ctr, status, tag, limit, [&] {
        *(volatile u64*)gave_up = 1;
        *(volatile u64*)host_timeout = 1;
    });
}

__global__ void scc_start_kernel(IterCtl* __restrict__ ctl) { ctl->t_start = global_ns(); }

// Order-independent digest of a tuple's data columns: depends only on the
// column values (not on the packing width), so runs with different widths agree.
__device__ __forceinline__ u64 digest_start(int arity) { return 0x9e3779b97f4a7c15ull * (u64)arity; }
__device__ __forceinline__ u64 digest_column(u64 h, u64 value, int c)
{
    return mix64(h ^ (value + 0x632be59bd9b4e019ull * (u64)(c + 1)));
}
__device__ __forceinline__ u64 tuple_digest(const u64* cols, int arity)
{
    u64 h = digest_start(arity);
    for (int c = 0; c < arity; c++) h = digest_column(h, cols[c], c);
    return h;
}

// Per-instance count and digest (sum of tuple digests, values rebased to the
// instance) of packed rows.  Each warp walks a contiguous segment of rows
// (coalesced, kSummaryBatch loads of a lane in flight), every lane keeps a running
// (count, digest) for the instance of its last rows and flushes it when the instance
// changes; relation logs hold each instance's rows in long runs, so flushes are rare, a
// row inside the current instance's value range skips the search over the bases, and a
// warp whose lanes end on one instance adds up before its last flush.  Up to
// kSummarySmemInst instances accumulate in shared memory first.  The hash of column 0 is
// kept while the column repeats (logs in key order).  ARITY > 0 fixes the arity at compile
// time (columns in registers); 0 reads `arity`.  Bound by the 64-bit multiplies of the
// digests: 326M + 223M rows of a tree of 2^15 nodes in 1.1 ms (4.4 GB, 4.0 TB/s) against 1.8
// with one load of a lane in flight; a few hundred rows in 5 us against 16-20.
constexpr u32 kSummarySmemInst = 1024;
constexpr int kSummaryRowsPerLane = 16;
constexpr int kSummaryBatch = 8;

template <int ARITY>
__global__ void __launch_bounds__(kThreads) instance_summary_kernel(
    const u64* __restrict__ keys, u64 n, int arity_rt, int bits, const u64* __restrict__ base, u32 n_inst,
    u64* __restrict__ counts, u64* __restrict__ digests)
{
    const int arity = ARITY > 0 ? ARITY : arity_rt;
    constexpr int kCols = ARITY > 0 ? ARITY : kMaxArity;
    __shared__ u64 s_cnt[kSummarySmemInst];
    __shared__ u64 s_dig[kSummarySmemInst];
    const u32 m = base ? n_inst : 1;
    const bool in_smem = m <= kSummarySmemInst;
    if (in_smem)
        for (u32 i = threadIdx.x; i < m; i += blockDim.x) s_cnt[i] = s_dig[i] = 0;
    __syncthreads();
    u32 cur = 0xffffffffu;
    u64 cur_lo = 1, cur_hi = 0;   // value range of instance `cur` (empty: no instance yet)
    u64 c = 0, dsum = 0;
    u64 col0 = ~0ull, h0 = 0;     // column 0 of the last row (values are below 2^63), its hash
    auto flush = [&]() {
        if (!c) return;
        u64* ca = in_smem ? &s_cnt[cur] : &counts[cur];
        u64* da = in_smem ? &s_dig[cur] : &digests[cur];
        atomicAdd((unsigned long long*)ca, (unsigned long long)c);
        atomicAdd((unsigned long long*)da, (unsigned long long)dsum);
        c = 0;
        dsum = 0;
    };
    const int lane = threadIdx.x & 31;
    const u64 seg = 32ull * kSummaryRowsPerLane;
    const u64 warps = (u64)gridDim.x * (blockDim.x >> 5);
    for (u64 w = (u64)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w * seg < n; w += warps) {
        for (int j = 0; j < kSummaryRowsPerLane; j += kSummaryBatch) {
            u64 k[kSummaryBatch];
#pragma unroll
            for (int b = 0; b < kSummaryBatch; b++) {
                const u64 i = w * seg + (u64)(j + b) * 32 + lane;
                k[b] = i < n ? keys[i] : kEmpty;
            }
#pragma unroll
            for (int b = 0; b < kSummaryBatch; b++) {
                if (k[b] == kEmpty) continue;
                u64 cols[kCols];
#pragma unroll
                for (int q = 0; q < kCols; q++)
                    if (q < arity) cols[q] = column_of(k[b], arity, q, bits);
                if (cols[0] != col0) {
                    if (!(cols[0] >= cur_lo && cols[0] < cur_hi)) {
                        const u32 inst = base ? instance_of(base, n_inst, cols[0]) : 0;
                        if (inst != cur) {
                            flush();
                            cur = inst;
                        }
                        cur_lo = base ? __ldg(&base[inst]) : 0;
                        cur_hi = base ? __ldg(&base[inst + 1]) : ~0ull;
                    }
                    col0 = cols[0];
                    h0 = digest_column(digest_start(arity), col0 - cur_lo, 0);
                }
                u64 h = h0;
#pragma unroll
                for (int q = 1; q < kCols; q++)
                    if (q < arity) h = digest_column(h, cols[q] - cur_lo, q);
                c++;
                dsum += h;
            }
        }
    }
    const u32 mine = c ? cur : 0xffffffffu, one = __reduce_min_sync(0xffffffffu, mine);
    if (__all_sync(0xffffffffu, mine == one || !c)) {   // the warp's rows are of one instance (or none)
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            c += __shfl_xor_sync(0xffffffffu, c, d);
            dsum += __shfl_xor_sync(0xffffffffu, dsum, d);
        }
        cur = one;
        if (lane) c = 0;
    }
    flush();
    if (!in_smem) return;
    __syncthreads();
    for (u32 i = threadIdx.x; i < m; i += blockDim.x)
        if (s_cnt[i]) {
            atomicAdd((unsigned long long*)&counts[i], (unsigned long long)s_cnt[i]);
            atomicAdd((unsigned long long*)&digests[i], (unsigned long long)s_dig[i]);
        }
}

// ---------------------------------------------------------------------------
// iteration end as its own launch (reference id order: after the sort passes)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) iter_end_kernel(IterCtl* __restrict__ ctl,
                                                            const __grid_constant__ SccPlan plan,
                                                            const __grid_constant__ SccRelMap rm,
                                                            u64* __restrict__ history, cudaGraphConditionalHandle cond,
                                                            int use_cond)
{
    __shared__ u64 s_end[kEndWords];
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < (u64)kMaxSccRels * kMaxPasses * kRadix;
         i += (u64)gridDim.x * blockDim.x)
        (&ctl->sort_hist[0][0][0])[i] = 0;
    if (blockIdx.x == 0)
        end_of_iteration_block(ctl, s_end, plan, rm, history, cond, use_cond, [](const IterCtl*) { return false; });
}

}  // namespace ra
