// wavefront.cu - seed_kernels 2 to 4: the seed/extend search as rounds of
// data-parallel passes over the whole batch (fm_seed_extend_kernel,
// fq2bam-meth/src/linear_gpu_fm.mojo:1156-1837, with the candidate order
// and exactness argument of seed_core.cuh).
//
// Round k covers right endpoints [resume, resume + width) of every read
// still active (width w0 in round 0, w after it):
//   search   per (read, endpoint): duplicate prediction, backward search, SA
//            rows -> candidate loci appended to a batch-wide locus list (one
//            atomic per warp);
//   eval     one thread per (locus, shift): the shift's candidates (full
//            compare, soft-clip retry, deletion probe) and an atomicMin of
//            the best key per read, packed with the locus' list index;
//   finalize one thread per active read: the new best (its fields are
//            recomputed from the winning locus and shift), the nm == 0 stop,
//            the exact nm == 1 early stop, the next round's active list.
// Every candidate of a round comes after the best of the rounds before it
// in the reference's order, so pruning against that best and taking the
// minimum key over the round gives the reference's hit.  A read whose loci
// do not fit the list is left out of its round (its memo and best roll
// back) and starts the next one from the same endpoint, or where the list is
// far too short goes to the stage-2 warp kernel, which also finishes the reads
// still active after the last round.
#include <cuda_runtime.h>

#include "ma_device.cuh"
#include "ma_internal.h"
#include "seed_core.cuh"

namespace ma {

int launch_stage2_pending(const DevIndex& ix, const DevReads& R, const DevParams& P, const DevOut& out,
                          uint64_t* key, uint64_t* memo, uint8_t* memo_n, uint16_t* resume, uint32_t* pending,
                          uint32_t* counters, int blocks, int level, int first_wave, unsigned long long* tally,
                          cudaStream_t st);

namespace {

// counters[]
constexpr int C_ACTIVE = 0;    // reads active in the current round
constexpr int C_NEXT = 1;      // reads appended to the next round's list
constexpr int C_LOCI = 32;     // loci appended in the current round: a u64 in counters[32..33]
constexpr int C_ROUNDS = 3;    // read-rounds processed (tally)
constexpr int C_HANDOFF = 8;   // [8] reads for stage 2, [9] its work cursor
constexpr int C_SEARCH = 64;   // deals of the round's items and loci beyond the
constexpr int C_EVAL = 96;     // warps' first ones: u64 each
constexpr int N_COUNTERS = 128;  // what whole grids add to lies 128 bytes apart

// Round keys: nm << (27 + ib) | ordinal << ib | locus index, ib bits of
// index: what the largest nm of the call leaves of the 64 bits, at most 31.
constexpr uint64_t MAX_LOCI = (1ull << 31) - 1;  // list capacity limit (indices fit 31 bits)

constexpr uint32_t DEAD_LOCUS = 0xFFFFFFFFu;  // WLocus.read of a slot without a locus
constexpr int PREDICT_MEMO = 4;  // memo loci a duplicate prediction checks besides the best

// One candidate locus of a round (32 bytes: two per 64-B line).
struct WLocus {
    int64_t b0;
    uint64_t uk;         // first SA row of the seed's interval
    uint32_t read, ord_row;
    int32_t rev;         // strand
    uint16_t us;         // seed start
    uint16_t e_dl;       // right endpoint (bits 0-10) | (ul - uk) << 11
    __device__ int e() const { return e_dl & 0x7FF; }
    __device__ uint64_t ul() const { return uk + (e_dl >> 11); }
};
static_assert(sizeof(WLocus) == 32, "WLocus is 32 bytes");

struct Wave {
    uint32_t* counters;
    uint64_t* best_key;   // nm << 27 | ordinal of the best so far, ~0 = none
    uint64_t* round_key;  // this round's minimum, packed with the locus index
    uint64_t* memo;       // [n][MEMO1] loci evaluated (b0 * 2 + strand)
    uint8_t* memo_n;      // memo entries valid at the start of the round
    uint32_t* memo_next;  // memo entries claimed during the round
    uint16_t* resume;     // first right endpoint of the read's next round
    uint8_t* overflow;    // the read's loci did not fit the list this round
    int64_t* best_tag;    // locus of the best hit, -1 = none
    uint32_t* active[2];  // ping-pong lists of active reads
    uint32_t* pending;    // reads handed to stage 2
    WLocus* loci;
    uint64_t locus_cap;
    int idx_bits;  // locus-index bits of the round keys
};

size_t align256(size_t b) { return (b + 255) & ~static_cast<size_t>(255); }

// The round's locus count (64-bit: the rows a round asks for can exceed 2^32).
__device__ __forceinline__ unsigned long long* loci_count(const Wave& w) {
    return reinterpret_cast<unsigned long long*>(w.counters + C_LOCI);
}

// The round's items or loci in groups of 32, dealt to the warps a few groups at
// a time: a warp's first ones by its place in the grid, later ones from a
// counter, asked for ahead.  Dealt by place alone, the warps whose groups held
// the long searches and the repeats kept the rest waiting (eval ran with 40 %
// of an SM's warps on average where 50 % fit).  A warp that is to come back
// more than DEALS times takes several groups at once and the counters lie in
// lines of their own: one group at a time, in the line of the loci's count,
// the 4 M additions for 2 M reads' items took 12 ms on some cards.  Loci of
// one read lie together, so eval takes two groups at most.  2 M uneven reads:
// search 8.2 -> 7.3 ms, eval 6.6 -> 6.0 (6.45 with up to 8 groups); 800 k reads
// of 250 bases 2.04 -> 1.95 and 1.47 -> 1.47.
constexpr uint32_t DEALS = 4, SEARCH_DEAL = 8, EVAL_DEAL = 2;
struct Groups {
    unsigned long long* counter;
    uint64_t base, ticket;  // base: first item of the group in hand
    uint32_t per, left;     // groups of a deal; of this one from the group in hand on
    __device__ __forceinline__ Groups(uint32_t* counters, int c, uint64_t n_items, uint32_t most)
        : counter(reinterpret_cast<unsigned long long*>(counters + c)), ticket(0) {
        const uint64_t threads = static_cast<uint64_t>(gridDim.x) * blockDim.x;
        per = 1;
        while (per < most && 2 * per * DEALS * threads <= n_items) per *= 2;
        left = per;
        base = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + (threadIdx.x & ~31u)) * per;
    }
    // The group in hand, one of the round's, is taken up (an empty round asks
    // for nothing) ...
    __device__ __forceinline__ void take() {
        if (--left == 0 && (threadIdx.x & 31) == 0) ticket = atomicAdd(counter, 1ull);
    }
    // ... and worked through: the following one.
    __device__ __forceinline__ void next() {
        if (left) {
            base += 32;
        } else {
            left = per;
            base = 32 * per * (__shfl_sync(0xFFFFFFFFu, ticket, 0) + gridDim.x * (blockDim.x >> 5));
        }
    }
};

// Carves the scratch; returns the bytes used (layout only when p != null).
size_t wave_layout(char* p, int64_t n_seq, uint64_t locus_cap, Wave* w) {
    const size_t n = static_cast<size_t>(n_seq);
    size_t o = 0;
    auto take = [&](size_t bytes) {
        char* q = p ? p + o : nullptr;
        o += align256(bytes);
        return q;
    };
    Wave v{};
    v.counters = reinterpret_cast<uint32_t*>(take(N_COUNTERS * 4));
    v.best_key = reinterpret_cast<uint64_t*>(take(n * 8));
    v.round_key = reinterpret_cast<uint64_t*>(take(n * 8));
    v.memo = reinterpret_cast<uint64_t*>(take(n * 8 * MEMO1));
    v.memo_n = reinterpret_cast<uint8_t*>(take(n));
    v.memo_next = reinterpret_cast<uint32_t*>(take(n * 4));
    v.resume = reinterpret_cast<uint16_t*>(take(n * 2));
    v.overflow = reinterpret_cast<uint8_t*>(take(n));
    v.best_tag = reinterpret_cast<int64_t*>(take(n * 8));
    v.active[0] = reinterpret_cast<uint32_t*>(take(n * 4));
    v.active[1] = reinterpret_cast<uint32_t*>(take(n * 4));
    v.pending = reinterpret_cast<uint32_t*>(take(n * 4));
    v.loci = reinterpret_cast<WLocus*>(take(locus_cap * sizeof(WLocus)));
    v.locus_cap = locus_cap;
    if (w) *w = v;
    return o;
}

uint64_t locus_capacity(uint64_t entries) {
    if (entries < 1024) entries = 1024;
    return entries < MAX_LOCI ? entries : MAX_LOCI;
}

__global__ void __launch_bounds__(256) wf_init_kernel(Wave w, DevOut out, const uint32_t* __restrict__ lens,
                                                      int64_t n_seq) {
    const int64_t r = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (r == 0) {
        for (int i = 0; i < N_COUNTERS; ++i) w.counters[i] = 0;
        w.counters[C_ACTIVE] = static_cast<uint32_t>(n_seq);
    }
    if (r >= n_seq) return;
    w.best_key[r] = ~0ull;
    w.round_key[r] = ~0ull;
    w.memo_n[r] = 0;
    w.memo_next[r] = 0;
    w.resume[r] = 0;
    w.overflow[r] = 0;
    w.best_tag[r] = -1;
    w.active[0][r] = static_cast<uint32_t>(r);
    Best none;
    none.key = ~0ull;
    none.crid = -1;
    none.uk = none.ul = 0;
    none.us = none.e = -1;
    write_hit(out, r, none, static_cast<int>(lens[r]));
}

// Moves the next round's active count into place (one thread).
__global__ void wf_round_begin_kernel(Wave w) {
    w.counters[C_ACTIVE] = w.counters[C_NEXT];
    w.counters[C_NEXT] = 0;
    *loci_count(w) = 0;
    for (int i = 0; i < 2; ++i) w.counters[C_SEARCH + i] = w.counters[C_EVAL + i] = 0;
}

// A read's memo (MEMO1 loci, 64 bytes), all of it in flight at once; entries
// from n on are not valid.
struct MemoRow {
    ulonglong2 v[MEMO1 / 2];
    __device__ __forceinline__ MemoRow(const Wave& w, uint32_t r) {
        const ulonglong2* p = reinterpret_cast<const ulonglong2*>(w.memo + static_cast<uint64_t>(r) * MEMO1);
#pragma unroll
        for (int i = 0; i < MEMO1 / 2; ++i) v[i] = p[i];
    }
    __device__ __forceinline__ bool holds(uint64_t tag, int n) const {
        bool found = false;
#pragma unroll
        for (int i = 0; i < MEMO1 / 2; ++i) found |= (2 * i < n && v[i].x == tag) || (2 * i + 1 < n && v[i].y == tag);
        return found;
    }
};

// Search: the round's items are (active read, endpoint) pairs.  Most end at
// their table lookup, the others step back one base at a time for anything
// from one to a hundred steps, and each seed found has 1 to 16 rows: a thread
// that took an item through all three would leave most of its warp waiting
// (12.6 lanes of 32 active per instruction).  So each warp keeps two lists in
// shared memory and every pass runs with its lanes full:
//   lookup  32 items, one per lane: duplicate prediction and the table steps;
//           searches that go on are pushed on the warp's list of searches;
//   step    32 searches from that list, one per lane, one backward step at a
//           time; a lane whose search ends takes the next one.  With the list
//           empty, items left and fewer than STEP_MIN lanes busy, the busy
//           ones are put back until further lookups have filled the list;
//   rows    the SA rows of the seeds found, one per lane, once more than
//           SEED_STAGE - 32 seeds wait (or nothing else is left): one list
//           slot per row (one atomic per pass); rows that give no new locus
//           leave their slot dead.
// Which pass finds a seed does not change the round's result: the eval keys
// carry the candidate order.
// 2 M uneven reads on 250 Mbp (62 M lookups, 56 M steps, 103 M rows): 7.3 ms;
// with a thread per item through all three the pass took a quarter longer.
// Bound by the latency of the gathers.
constexpr int SEARCH_WARPS = 8;   // 256 threads
constexpr int SEARCH_LIST = 64;   // searches under way per warp
constexpr int SEED_STAGE = 64;    // seeds waiting per warp
constexpr int STEP_MIN = 20;

struct SearchLists {
    // a search: k | s << 35 | e << 45, rows - 1 | last << 35 (SeedSearch's, plus one),
    // last_k | endpoint index << 35, read
    uint64_t a[SEARCH_LIST], b[SEARCH_LIST], c[SEARCH_LIST];
    uint32_t read[SEARCH_LIST];
    // a seed: its first row, read, staged rows up to and including it, then
    // start | right endpoint << 16 and endpoint index | read length << 16
    uint64_t seed_k[SEED_STAGE];
    uint32_t seed_read[SEED_STAGE], rows_end[SEED_STAGE], s_e[SEED_STAGE], ei_len[SEED_STAGE];
};
static_assert(SEARCH_WARPS * sizeof(SearchLists) <= 32768, "six blocks per SM leave room for the L1 cache");

// Words of read r for the backward steps (qlen is not needed there).
__device__ __forceinline__ ReadView step_view(const DevReads& R, uint32_t r) {
    const uint64_t* b = R.packed + static_cast<uint64_t>(r) * 4 * static_cast<uint64_t>(R.words);
    ReadView v;
    v.fwd = b;
    v.rc = nullptr;
    v.nf = b + 2 * R.words;
    v.nr = nullptr;
    v.qlen = 0;
    return v;
}

template <bool S, int MINB>
__global__ void __launch_bounds__(256, MINB) wf_search_kernel(DevIndex ix, DevReads R, DevParams P, Wave w,
                                                        const uint32_t* __restrict__ act, int width,
                                                        unsigned long long* __restrict__ tally_out) {
    __shared__ SearchLists s_lists[SEARCH_WARPS];
    constexpr unsigned FULL = 0xFFFFFFFFu;
    constexpr uint64_t MASK35 = (1ull << 35) - 1;
    Tally t{};
    const uint64_t n_items = static_cast<uint64_t>(w.counters[C_ACTIVE]) * static_cast<uint64_t>(width);
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1;
    const bool can_predict = ix.summary && ix.kmer3_k > 0 && ix.kmer3_k <= P.seed_len;
    SearchLists& q = s_lists[threadIdx.x >> 5];
    Groups groups(w.counters, C_SEARCH, n_items, SEARCH_DEAL);
    int n_search = 0, n_seeds = 0;  // entries of the lists (warp-uniform)
    uint32_t n_rows = 0;
    // pushes the seeds of the lanes that found one
    auto push_seeds = [&](const Seed& sd, uint32_t r, int e, int ei) {
        const unsigned fb = __ballot_sync(FULL, sd.found);
        if (!fb) return;
        const uint32_t rows = sd.found ? static_cast<uint32_t>(sd.l - sd.k + 1) : 0u;
        uint32_t incl = rows;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += v;
        }
        if (sd.found) {
            const int i = n_seeds + __popc(fb & lt_mask);
            q.seed_k[i] = sd.k;
            q.seed_read[i] = r;
            q.rows_end[i] = n_rows + incl;
            q.s_e[i] = static_cast<uint32_t>(sd.s) | static_cast<uint32_t>(e) << 16;
            q.ei_len[i] = static_cast<uint32_t>(ei) | __ldg(R.lens + r) << 16;
        }
        n_seeds += __popc(fb);
        n_rows += __shfl_sync(FULL, incl, 31);
    };
    // pushes the searches of the lanes that are `on`
    auto push_search = [&](bool on, const SeedSearch& c, uint32_t r, int e, int ei) {
        const unsigned ob = __ballot_sync(FULL, on);
        if (on) {
            const int i = n_search + __popc(ob & lt_mask);
            q.a[i] = c.k | static_cast<uint64_t>(c.s) << 35 | static_cast<uint64_t>(e) << 45;
            q.b[i] = (c.l - c.k) | static_cast<uint64_t>(c.last + 1) << 35;
            q.c[i] = c.last_k | static_cast<uint64_t>(ei) << 35;
            q.read[i] = r;
        }
        n_search += __popc(ob);
    };
    for (;;) {
        const bool more = groups.base < n_items;
        const bool look = more && n_search <= SEARCH_LIST - 32;
        if (n_seeds > SEED_STAGE - 32 || (!more && n_search == 0)) {
            // ---- rows ----
            if (n_seeds == 0) break;
            __syncwarp();
            unsigned long long wbase = 0;
            if (lane == 0) wbase = atomicAdd(loci_count(w), static_cast<unsigned long long>(n_rows));
            wbase = __shfl_sync(FULL, wbase, 0);
            for (uint32_t idx = lane; idx < n_rows; idx += 32) {
                int lo = 0, hi = n_seeds - 1;  // first seed whose rows_end exceeds idx
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (q.rows_end[mid] > idx) hi = mid;
                    else lo = mid + 1;
                }
                const uint32_t first = lo ? q.rows_end[lo - 1] : 0u;
                const uint32_t r = q.seed_read[lo];
                const uint64_t slot = static_cast<uint64_t>(wbase) + idx;
                if (slot >= w.locus_cap) {
                    w.overflow[r] = 1;
                    continue;
                }
                const MemoRow memo(w, r);  // in flight together with the SA row
                const int n_memo = w.memo_n[r];
                const uint64_t k = q.seed_k[lo], sa_pos = sa_at(ix, k + (idx - first));
                if constexpr (S) t.sa_loads++;
                const uint32_t s_e = q.s_e[lo], ei_len = q.ei_len[lo];
                const int s = static_cast<int>(s_e & 0xFFFF), e = static_cast<int>(s_e >> 16);
                const int qlen = static_cast<int>(ei_len >> 16);
                WLocus L;
                int64_t b0;
                int rev;
                if (!locus_of_row(ix, sa_pos, s, e, qlen, b0, rev) ||
                    memo.holds(static_cast<uint64_t>(b0 * 2 + rev), n_memo)) {
                    w.loci[slot].read = DEAD_LOCUS;
                    continue;
                }
                L.b0 = b0;
                L.uk = k;
                L.read = r;
                L.ord_row = ((ei_len & 0xFFFF) * 16 + (idx - first)) * ADJ_SPAN;
                L.us = static_cast<uint16_t>(s);
                L.e_dl = static_cast<uint16_t>(e | ((q.rows_end[lo] - first - 1) << 11));
                L.rev = rev;
                w.loci[slot] = L;
                if constexpr (S) tally_locus(t, b0, clamps_for(P, qlen).adj_cap, qlen);
                const uint32_t m = atomicAdd(&w.memo_next[r], 1u);
                if (m < static_cast<uint32_t>(MEMO1)) w.memo[static_cast<uint64_t>(r) * MEMO1 + m] = static_cast<uint64_t>(b0 * 2 + rev);
            }
            __syncwarp();
            n_seeds = 0;
            n_rows = 0;
        } else if (look) {
            // ---- lookup ----
            const uint64_t item = groups.base + lane;
            groups.take();
            Seed sd{0, 0, -1, false};
            SeedSearch c{};
            bool go_on = false;
            uint32_t r = 0;
            int ei = 0, e = 0;
            if (item < n_items) {
                const uint64_t a = item < (1ull << 32) ? static_cast<uint32_t>(item) / static_cast<uint32_t>(width)
                                                       : item / static_cast<uint64_t>(width);
                const int j = static_cast<int>(item - a * static_cast<uint64_t>(width));
                r = act[a];
                const ReadView rd = read_view(R, r);
                ei = static_cast<int>(w.resume[r]) + j;
                if (ei < endpoint_count(P, rd.qlen)) {
                    e = P.seed_len - 1 + ei * P.seed_stride;
                    // a read with no hit yet gains little from predicting its
                    // rejected loci again: only reads with a best try the memo
                    const int64_t best_tag = w.best_tag[r];
                    bool dup = false;
                    if (can_predict && best_tag != -1) {
                        const int n_memo = w.memo_n[r];
                        dup = predicted_duplicate<S>(ix, rd, e, P, best_tag, w.memo + static_cast<uint64_t>(r) * MEMO1,
                                                     n_memo < PREDICT_MEMO ? n_memo : PREDICT_MEMO, t);
                    }
                    if constexpr (S) t.skipped += dup;
                    if (!dup) go_on = search_start<S>(ix, rd, e, P, c, sd, t);
                }
            }
            push_search(go_on, c, r, e, ei);
            push_seeds(sd, r, e, ei);
            groups.next();
            __syncwarp();
        } else {
            // ---- step ----
            bool busy = false;
            SeedSearch c{};
            uint32_t r = 0;
            int ei = 0, e = 0;
            for (;;) {
                // idle lanes take searches from the end of the list
                const unsigned idle = __ballot_sync(FULL, !busy);
                const int rank = __popc(idle & lt_mask);
                if (!busy && rank < n_search) {
                    const int i = n_search - 1 - rank;
                    const uint64_t a = q.a[i], b = q.b[i], d = q.c[i];
                    c.k = a & MASK35;
                    c.l = c.k + (b & MASK35);
                    c.last_k = d & MASK35;
                    c.s = static_cast<int>(a >> 35) & 0x3FF;
                    c.last = static_cast<int>(b >> 35) - 1;
                    e = static_cast<int>(a >> 45);
                    ei = static_cast<int>(d >> 35);
                    r = q.read[i];
                    busy = true;
                }
                n_search -= min(n_search, __popc(idle));
                const int n_busy = __popc(__ballot_sync(FULL, busy));
                if (n_busy == 0) break;
                if (n_seeds > SEED_STAGE - 32 || (n_search == 0 && more && n_busy < STEP_MIN)) {
                    __syncwarp();
                    push_search(busy, c, r, e, ei);
                    break;
                }
                Seed sd{0, 0, -1, false};
                if (busy) busy = search_next<S>(ix, step_view(R, r), e, P, c, sd, t);
                push_seeds(sd, r, e, ei);
            }
            __syncwarp();
        }
    }
    flush_tally<S>(t, tally_out);
}

// Eval: one thread per locus filters its shifts (live_shifts); what is left
// goes through the parts of a shift (seed_core.cuh) in lists of the warp, in
// shared memory, each part run with 32 entries, one per lane: the core
// compare of the live shifts (a fraction of a shift per locus at genome
// scale), the full compare of those that pass, the deletion probe's bound of
// those that need it and its offsets where the bound allows one.  With the parts run one after the other by the lane that had
// the shift, the rare long ones kept the warp at 16 lanes of 32.  Candidates
// are pruned against the read's best from earlier rounds; the round's minimum
// key per read is an atomicMin of (nm, ordinal, locus index) packed in 64 bits.
// 102 M loci, 31 M live shifts of 2 M uneven reads: 6.0 ms; with a lane for all
// parts of a shift the pass took a fifth longer.
constexpr int EVAL_THREADS = 256;
constexpr int SHIFT_LIST = 64;  // entries per list and warp: locus index << 5 | shift
enum : int { L_CORE = 0, L_FULL = SHIFT_FULL, L_DELETION = SHIFT_DELETION, L_OFFSETS = SHIFT_OFFSETS };

// The largest nm that can still matter for read r.
__device__ __forceinline__ int prune_of(const Wave& w, uint32_t r) {
    const uint64_t bn = w.best_key[r] >> ORD_SHIFT;
    return bn < (1u << 20) ? static_cast<int>(bn) : (1 << 20);
}

template <bool S, int MINB>
__global__ void __launch_bounds__(EVAL_THREADS, MINB) wf_eval_kernel(DevIndex ix, DevReads R, DevParams P, Wave w,
                                                               unsigned long long* __restrict__ tally_out) {
    __shared__ uint64_t s_list[EVAL_THREADS / 32][4][SHIFT_LIST];
    constexpr unsigned FULL = 0xFFFFFFFFu;
    Tally t{};
    uint64_t n_loci = *loci_count(w);
    if (n_loci > w.locus_cap) n_loci = w.locus_cap;
    const int adj_cap = clamps_for(P, 1 << 20).adj_cap;  // read-independent
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1;
    uint64_t(*list)[SHIFT_LIST] = s_list[threadIdx.x >> 5];
    int n[4] = {0, 0, 0, 0};  // entries of each list (warp-uniform)
    uint32_t rem = 0, li = 0;  // the lane's locus and its live shifts not yet listed
    Groups groups(w.counters, C_EVAL, n_loci, EVAL_DEAL);
    for (;;) {
        const bool have = groups.base < n_loci, pending = __any_sync(FULL, rem != 0);
        // a full list first, the last part's before the others; then the shifts
        // waiting, the next loci, and in the end what the lists still hold
        int part = -1;
        if (n[L_OFFSETS] >= 32) part = L_OFFSETS;
        else if (n[L_DELETION] >= 32) part = L_DELETION;
        else if (n[L_FULL] >= 32) part = L_FULL;
        else if (n[L_CORE] >= 32) part = L_CORE;
        else if (!pending && !have) part = n[L_CORE] ? L_CORE : n[L_FULL] ? L_FULL : n[L_DELETION] ? L_DELETION : L_OFFSETS;
        if (part >= 0) {
            const int count = part == L_CORE ? n[L_CORE] : part == L_FULL ? n[L_FULL]
                              : part == L_DELETION ? n[L_DELETION] : n[L_OFFSETS];
            if (count == 0) break;
            __syncwarp();
            const int from = count > 32 ? count - 32 : 0;  // the last 32 entries
            const bool on = lane < count - from;
            const uint64_t v = on ? list[part][from + lane] : 0;
            if (part == L_CORE) n[L_CORE] = from;
            else if (part == L_FULL) n[L_FULL] = from;
            else if (part == L_DELETION) n[L_DELETION] = from;
            else n[L_OFFSETS] = from;
            int left = SHIFT_DEAD;
            if (on) {
                const uint32_t i = static_cast<uint32_t>(v >> 5);
                const WLocus L = w.loci[i];
                const ReadView rd = read_view(R, L.read);
                const Clamps cl = clamps_for(P, rd.qlen);
                const Shift c{L.b0, L.rev, static_cast<int>(v & 31) - adj_cap, cl.budget, cl.clip_cap,
                              prune_of(w, L.read), L.ord_row, L.uk, L.ul(), L.us, L.e()};
                if (part == L_CORE) {
                    left = shift_core<S>(ix, rd, c, t);
                } else if (part == L_DELETION) {
                    left = shift_deletion<S>(ix, rd, c, t);
                } else {
                    Best lb;
                    lb.key = ~0ull;
                    if (part == L_FULL) left = shift_full<S>(ix, rd, c, lb, t);
                    else shift_offsets<S>(ix, rd, c, lb, t);
                    if (lb.key != ~0ull) {
                        const uint64_t nm = lb.key >> ORD_SHIFT, ord = lb.key & ((1ull << ORD_SHIFT) - 1);
                        atomicMin(reinterpret_cast<unsigned long long*>(w.round_key + L.read),
                                  static_cast<unsigned long long>((nm << (ORD_SHIFT + w.idx_bits)) | (ord << w.idx_bits) | i));
                    }
                }
            }
            __syncwarp();
#pragma unroll
            for (int k = L_FULL; k <= L_OFFSETS; ++k) {
                const unsigned kb = __ballot_sync(FULL, left == k);
                if (left == k) list[k][n[k] + __popc(kb & lt_mask)] = v;
                n[k] += __popc(kb);
            }
        } else if (pending) {
            // as many live shifts as fit (lanes in order)
            const int k = __popc(rem);
            int incl = k;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += v;
            }
            int at = n[L_CORE] + incl - k;
            while (rem && at < SHIFT_LIST) {
                list[L_CORE][at++] = static_cast<uint64_t>(li) << 5 | static_cast<uint32_t>(__ffs(rem) - 1);
                rem &= rem - 1;
            }
            const int total = n[L_CORE] + __shfl_sync(FULL, incl, 31);
            n[L_CORE] = total < SHIFT_LIST ? total : SHIFT_LIST;
        } else {
            li = static_cast<uint32_t>(groups.base) + lane;
            groups.take();
            if (li < n_loci) {
                const WLocus L = w.loci[li];
                if (L.read != DEAD_LOCUS && !w.overflow[L.read]) {
                    const ReadView rd = read_view(R, L.read);
                    const Clamps cl = clamps_for(P, rd.qlen);
                    rem = live_shifts<S>(ix, rd, L.b0, L.rev, adj_cap, cl.budget, cl.clip_cap, prune_of(w, L.read), t);
                }
            }
            groups.next();
        }
    }
    flush_tally<S>(t, tally_out);
}

// Finalize: one thread per active read (warp-uniform loop for the list
// appends).  last_round: reads with endpoints left go to stage 2.
template <bool S>
__global__ void __launch_bounds__(256, 4) wf_finalize_kernel(DevIndex ix, DevReads R, DevParams P, DevOut out, Wave w,
                                                          const uint32_t* __restrict__ act,
                                                          uint32_t* __restrict__ next, int width, int last_round,
                                                          int* __restrict__ err,
                                                          unsigned long long* __restrict__ tally_out) {
    Tally t{};
    const uint32_t n_act = w.counters[C_ACTIVE];
    const int lane = threadIdx.x & 31;
    const uint32_t stride = gridDim.x * blockDim.x;
    // Reads that the list had no room for wait for the next round when it held
    // two thirds of what the round asked for.  With less room most reads would
    // wait, and their searches run again round after round: 400 k pairs 2x150 with
    // 1, 2 or (rounds of 32 endpoints) 4 entries per read 9.3, 6.6 and 5.3 ms,
    // 18.4, 11.9 and 6.8 when all wait.  With nearly enough stage 2 takes longer:
    // 3.3 and 3.7 ms with 3 entries and with 4 (2 endpoints in the first round),
    // 3.5 and 5.4 when none waits.
    const bool wait = !last_round && 2 * *loci_count(w) <= 3 * w.locus_cap;
    if constexpr (S) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&w.counters[C_ROUNDS], n_act);
    }
    for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n_act; base += stride) {
        const uint32_t a = base + lane;
        bool to_next = false, to_stage2 = false;
        int64_t r = 0;
        if (a < n_act) {
            r = act[a];
            const ReadView rd = read_view(R, r);
            const int qlen = rd.qlen;
            const Clamps cl = clamps_for(P, qlen);
            const int n_end = endpoint_count(P, qlen);
            if (w.overflow[r]) {
                // left out of this round: roll back; the next round takes the
                // same endpoints up again, or stage 2 does
                w.overflow[r] = 0;
                w.memo_next[r] = w.memo_n[r];
                if (!wait) to_stage2 = true;
                else to_next = true;
            } else {
                const uint32_t mn = w.memo_next[r];
                w.memo_n[r] = static_cast<uint8_t>(mn < static_cast<uint32_t>(MEMO1) ? mn : MEMO1);
                const uint64_t rk = w.round_key[r];
                const uint64_t old = w.best_key[r];
                bool stop = false;
                const uint64_t rkey = rk >> w.idx_bits;  // nm << ORD_SHIFT | ordinal, the best-key format
                if (rk != ~0ull && rkey < old) {
                    // the new best: recompute its fields from the winning locus and shift
                    const WLocus L = w.loci[rk & ((1ull << w.idx_bits) - 1)];
                    const uint32_t ord = static_cast<uint32_t>(rkey & ((1ull << ORD_SHIFT) - 1));
                    const int adj = static_cast<int>(ord / KIND_SPAN) - static_cast<int>(L.ord_row) - 12;
                    const uint64_t bn = old >> ORD_SHIFT;
                    const int prune = bn < (1u << 20) ? static_cast<int>(bn) : (1 << 20);
                    Best lb;
                    const Shift c{L.b0, L.rev, adj, cl.budget, cl.clip_cap, prune, L.ord_row, L.uk, L.ul(), L.us, L.e()};
                    if (!shift_candidate<S>(ix, rd, c, rkey, lb, t)) {
                        atomicExch(err, 3);  // the recomputed candidate must be the round's minimum
                    } else {
                        write_hit(out, r, lb, qlen);
                        w.best_key[r] = lb.key;
                        w.best_tag[r] = L.b0 * 2 + L.rev;
                        const uint64_t nm = lb.key >> ORD_SHIFT;
                        if (nm == 0) {
                            stop = true;
                        } else if (nm <= 2 && full_compare_key(lb.key)) {
                            const int64_t bstart = static_cast<int64_t>(__ldg(ix.coff + lb.crid)) + lb.pos - lb.sl;
                            stop = better_hit_impossible<S>(ix, rd, bstart, (lb.flag & 16) ? 1 : 0, cl.clip_cap,
                                                            static_cast<int>(nm), t);
                        }
                    }
                }
                w.round_key[r] = ~0ull;
                const int nxt = static_cast<int>(w.resume[r]) + width;
                if (!stop && nxt < n_end) {
                    w.resume[r] = static_cast<uint16_t>(nxt);
                    if (last_round) to_stage2 = true;
                    else to_next = true;
                }
            }
        }
        const unsigned bn = __ballot_sync(0xFFFFFFFFu, to_next);
        if (bn) {
            uint32_t b = 0;
            if (lane == 0) b = atomicAdd(&w.counters[C_NEXT], static_cast<uint32_t>(__popc(bn)));
            b = __shfl_sync(0xFFFFFFFFu, b, 0);
            if (to_next) next[b + __popc(bn & ((1u << lane) - 1))] = static_cast<uint32_t>(r);
        }
        const unsigned bs = __ballot_sync(0xFFFFFFFFu, to_stage2);
        if (bs) {
            uint32_t b = 0;
            if (lane == 0) b = atomicAdd(&w.counters[C_HANDOFF], static_cast<uint32_t>(__popc(bs)));
            b = __shfl_sync(0xFFFFFFFFu, b, 0);
            if (to_stage2) w.pending[b + __popc(bs & ((1u << lane) - 1))] = static_cast<uint32_t>(r);
        }
    }
    flush_tally<S>(t, tally_out);
}

// See wave_plan below.
constexpr int64_t WAVE_ONE = 131072, WAVE_ITEMS = 4 << 20, WAVE_LOCI = 2 << 20, WAVE_LOCI_MOST = 16 << 20;

int endpoint_count_host(const DevParams& P, int qlen) {
    return qlen >= P.seed_len ? (qlen - P.seed_len) / P.seed_stride + 1 : 0;
}

template <typename K>
int grid_blocks(K kernel, int sm_count) {
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, 256, 0);
    if (nb < 1) nb = 1;
    return nb * sm_count;
}

// Register budget of the search / eval kernels (result-neutral): blocks of
// 256 threads asked per SM (1 = the compiler's choice).
template <bool S, int MS, int ME>
int launch_rounds(const DevIndex& ix, const DevReads& R, const DevParams& P, const DevOut& out, const Wave& w,
                  int max_len, int w0, int wn, int max_rounds, int growth, int sm_count, int* d_err,
                  unsigned long long* tally, WaveTimer* timer, cudaStream_t st) {
    const int n_end_max = endpoint_count_host(P, max_len);
    // round widths: w0, then wn (doubling from the third round with growth)
    int widths[1100];
    int rounds = 0, covered = 0;
    for (int width = w0; covered < n_end_max || rounds == 0; ++rounds) {
        widths[rounds] = width;
        covered += width;
        if (rounds == 0) width = wn;
        else if (growth && width < 4096) width *= 2;
    }
    // a large batch gets one more round for the reads that had to wait for list
    // space (10 us when there are none): a warp each would take longer
    if (R.n_seq > WAVE_ONE && rounds > 1) {
        widths[rounds] = widths[rounds - 1];
        ++rounds;
    }
    if (max_rounds > 0 && rounds > max_rounds) rounds = max_rounds;
    static const int g_search = grid_blocks(wf_search_kernel<S, MS>, sm_count);
    static const int g_eval = grid_blocks(wf_eval_kernel<S, ME>, sm_count);  // EVAL_THREADS = 256
    static const int g_fin = grid_blocks(wf_finalize_kernel<S>, sm_count);
    const unsigned init_blocks = static_cast<unsigned>((R.n_seq + 255) / 256);
    wf_init_kernel<<<init_blocks ? init_blocks : 1, 256, 0, st>>>(w, out, R.lens, R.n_seq);
    int launches = 1;
    for (int k = 0; k < rounds; ++k) {
        const int width = widths[k];
        const uint32_t* act = w.active[k & 1];
        uint32_t* nxt = w.active[(k + 1) & 1];
        if (k > 0) {
            wf_round_begin_kernel<<<1, 1, 0, st>>>(w);
            ++launches;
        }
        const bool timed = timer && k < WaveTimer::MAX_ROUNDS;
        if (timed) cudaEventRecord(timer->e[3 * k], st);
        wf_search_kernel<S, MS><<<g_search, 256, 0, st>>>(ix, R, P, w, act, width, tally);
        if (timed) cudaEventRecord(timer->e[3 * k + 1], st);
        wf_eval_kernel<S, ME><<<g_eval, 256, 0, st>>>(ix, R, P, w, tally);
        if (timed) cudaEventRecord(timer->e[3 * k + 2], st);
        wf_finalize_kernel<S><<<g_fin, 256, 0, st>>>(ix, R, P, out, w, act, nxt, width, k == rounds - 1, d_err,
                                                     tally);
        launches += 3;
    }
    if (timer) {
        const int timed = rounds < WaveTimer::MAX_ROUNDS ? rounds : WaveTimer::MAX_ROUNDS;
        cudaEventRecord(timer->e[3 * timed], st);
        timer->recorded = timed;
        timer->complete = rounds <= WaveTimer::MAX_ROUNDS;
    }
    return launches;
}

}  // namespace

size_t wavefront_scratch_bytes(int64_t n_seq, uint64_t loci) {
    return wave_layout(nullptr, n_seq, locus_capacity(loci), nullptr);
}

// The plan that takes a tuning as it is.
WavePlan wave_plan_asked(const ma_tuning& asked, int64_t n_seq) {
    return WavePlan{asked, static_cast<uint64_t>(asked.wave_loci_per_read) * static_cast<uint64_t>(n_seq)};
}

// The round widths and the locus list of a call under the default tuning,
// fitted to its size; any other tuning is taken as it is.  A round costs the
// latency of its longest search whatever its width, narrow rounds save the
// searches of reads that a hit ends or predicts: a batch that does not fill
// the GPU is better off with few wide ones.  Kernel time of all rounds, 2x150
// pairs on 250 Mbp:
//   32 pairs     5 rounds (1, 8, 16, 32, 64 endpoints) 0.27 ms, one round 0.09
//   2 k pairs    5 rounds 0.74 ms, two rounds (2, the rest) 0.31
//   16 k pairs   1.03 and 0.51 ms
//   400 k 2x250  4.6 (8 endpoints, doubling) and 5.2 ms (16 endpoints)
// So a batch of up to WAVE_ONE items (reads x endpoints) takes one round, and
// a later round covers up to WAVE_ITEMS items.  Wide rounds need longer locus
// lists: 256 entries per read up to 2 M entries (64 MB) in all, 8 up to 16 M (512
// MB): 800 k reads of 250 bases take 4.3 ms with 8 entries and 4.9 with 4, whose
// list fills up.  The list never gets shorter as the reads of a call grow in
// number, so that a call with fewer reads than one before it finds its scratch
// there: it allocates nothing, and no captured graph is dropped for it.
WavePlan wave_plan(const ma_tuning& asked, int64_t n_seq, int max_len, const DevParams& P) {
    WavePlan plan = wave_plan_asked(asked, n_seq);
    ma_tuning& t = plan.tuning;
    if (t.stage1_endpoints != 1 || t.wave_endpoints != 8 || t.wave_loci_per_read != 4 || t.wave_max_rounds != 0 ||
        t.wave_growth != 1 || n_seq < 1)
        return plan;
    const int64_t n_end = endpoint_count_host(P, max_len);
    if (n_seq * n_end <= WAVE_ONE) {
        t.stage1_endpoints = static_cast<int32_t>(n_end > 1 ? n_end : 1);
    } else if (WAVE_ITEMS / n_seq > t.wave_endpoints) {
        t.stage1_endpoints = 2;
        t.wave_endpoints = static_cast<int32_t>(WAVE_ITEMS / n_seq < n_end ? WAVE_ITEMS / n_seq : n_end);
    }
    const auto at_most = [](int64_t a, int64_t b) { return static_cast<uint64_t>(a < b ? a : b); };
    for (const uint64_t c : {at_most(256 * n_seq, WAVE_LOCI), at_most(8 * n_seq, WAVE_LOCI_MOST)})
        if (c > plan.loci) plan.loci = c;
    return plan;
}

// The wavefront form; `scratch` holds wavefront_scratch_bytes(n_seq,
// plan.loci) bytes, d_err is the batch's error word.  Returns the number of
// kernel launches.
int launch_seed_wavefront(const DevIndex& ix, const DevReads& R, const DevParams& P, const DevOut& out, int max_len,
                          const WavePlan& plan, int stage2_blocks, void* scratch, int sm_count, int* d_err,
                          unsigned long long* d_tally, WaveTimer* timer, cudaStream_t st) {
    const ma_tuning& t = plan.tuning;
    Wave w;
    wave_layout(static_cast<char*>(scratch), R.n_seq, locus_capacity(plan.loci), &w);
    // an accepted candidate has nm <= its read's budget <= max(2, max_diff)
    // (and <= 512): the round keys give the rest to the locus index
    const int max_nm = P.max_diff < 2 ? 2 : (P.max_diff > 512 ? 512 : P.max_diff);
    int nm_bits = 1;
    while ((1 << nm_bits) <= max_nm) ++nm_bits;
    w.idx_bits = 64 - ORD_SHIFT - nm_bits < 31 ? 64 - ORD_SHIFT - nm_bits : 31;
    if (w.locus_cap > (1ull << w.idx_bits) - 1) w.locus_cap = (1ull << w.idx_bits) - 1;
    const int w0 = t.stage1_endpoints > 0 ? t.stage1_endpoints : 1;
    const int wn = t.wave_endpoints > 0 ? t.wave_endpoints : 1;
    int launches = 0;
    const int mr = t.wave_max_rounds, gr = t.wave_growth;
    if (d_tally)
        launches = launch_rounds<true, 1, 1>(ix, R, P, out, w, max_len, w0, wn, mr, gr, sm_count, d_err, d_tally, timer, st);
    else if (t.reg_level == 1)
        launches = launch_rounds<false, 5, 4>(ix, R, P, out, w, max_len, w0, wn, mr, gr, sm_count, d_err, nullptr, timer, st);
    else if (t.reg_level == 2)
        launches = launch_rounds<false, 6, 5>(ix, R, P, out, w, max_len, w0, wn, mr, gr, sm_count, d_err, nullptr, timer, st);
    else
        launches = launch_rounds<false, 1, 1>(ix, R, P, out, w, max_len, w0, wn, mr, gr, sm_count, d_err, nullptr, timer, st);
    // reads that overflowed the locus list or outlived the rounds (their
    // tallies in the second half of the tally array, their time between
    // the timer's stage-2 events)
    if (timer) cudaEventRecord(timer->s2[0], st);
    launches += launch_stage2_pending(ix, R, P, out, w.best_key, w.memo, w.memo_n, w.resume, w.pending,
                                      w.counters + C_HANDOFF, stage2_blocks, t.reg_level, 32,
                                      d_tally ? d_tally + TALLY_N : nullptr, st);
    if (timer) cudaEventRecord(timer->s2[1], st);
    return launches;
}

}  // namespace ma
