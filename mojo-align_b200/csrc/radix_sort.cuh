// radix_sort.cuh - stable LSD radix sort of (u64 key, u32 value) pairs on
// the device, digits of up to 8 bits, for the coordinate and duplicate-key
// orders of sort_markdup.cu.
//
// A pass over digit d is three kernels:
//   rs_hist     one block per tile of TILE keys: the tile's digit counts,
//               stored digit-major (count[d][tile]);
//   rs_scan     one block per digit: exclusive prefix of count[d][*] over the
//               tiles, and the digit's total;
//   rs_scatter  one block per tile: the digit bases (exclusive scan of the
//               totals), each key's rank among the tile's keys of its digit
//               (in tile order), then key and value to
//               base[d] + prefix[d][tile] + rank.
// Ranks follow the input order, so every pass is stable and the whole sort
// gives the order of a stable sort by the full key (ties by input position),
// the order of the reference's own 8-bit LSD radix.
//
// A pass sorts by up to 8 of the bits that decide an order.  A bit that is
// the same in every key decides nothing, and neither does one that equals
// the next higher bit in every key: where two keys differ in it they differ
// in that one first.  rs_bits ORs key ^ key[0] and key ^ (key >> 1) over the
// input, and rs_plan (one thread) deals the bits that are left to passes, up
// to four runs of bits in a digit (8 neighbouring bits hold no more, so 8
// passes always do).  Coordinate and duplicate keys, whose unplaced records
// have all upper bits set, take 5 passes instead of 8.  rs_plan also lays
// out each pass's source and destination so that the last one writes the
// caller's output buffers (or rs_copy copies the input there when there is
// none).  The plan lives in device memory: nothing waits on the host, and a
// stream capture of the sort is a plain kernel sequence.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace ma {
namespace radix {

constexpr int THREADS = 256;
constexpr int ROUNDS = 16;                 // keys per thread
constexpr int TILE = THREADS * ROUNDS;     // 4096 keys per tile
constexpr int WARPS = THREADS / 32;
constexpr int PASSES = 8;                  // 64-bit keys, 8 or more of their bits a pass

// A digit: for each of its runs of key bits, the shift that brings the run
// to its place in the digit and the mask of that place.
struct Digit {
    uint32_t shift[4];
    uint32_t mask[4];

    __device__ __forceinline__ uint32_t of(uint64_t key) const {
        uint32_t d = (static_cast<uint32_t>(key >> shift[0]) & mask[0]) |
                     (static_cast<uint32_t>(key >> shift[1]) & mask[1]);
        if (mask[2])
            d |= (static_cast<uint32_t>(key >> shift[2]) & mask[2]) |
                 (static_cast<uint32_t>(key >> shift[3]) & mask[3]);
        return d;
    }
};

struct Plan {
    const uint64_t* src_k[PASSES];
    const uint32_t* src_v[PASSES];
    uint64_t* dst_k[PASSES];
    uint32_t* dst_v[PASSES];
    Digit digit[PASSES];
    int passes;  // 0: no bit varies, the input is copied to the output
};

// bits[0]: the bits that vary; bits[1]: those that differ from the next
// higher one in some key.
__global__ void rs_bits(const uint64_t* __restrict__ keys, uint64_t n, unsigned long long* __restrict__ bits) {
    const uint64_t k0 = keys[0];
    uint64_t v = 0, e = 0;
#pragma unroll 4
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(THREADS) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * THREADS) {
        const uint64_t k = keys[i];
        v |= k ^ k0;
        e |= k ^ (k >> 1);
    }
    for (int o = 16; o > 0; o >>= 1) {
        v |= __shfl_xor_sync(0xFFFFFFFFu, v, o);
        e |= __shfl_xor_sync(0xFFFFFFFFu, e, o);
    }
    __shared__ uint64_t s_v[WARPS], s_e[WARPS];
    if ((threadIdx.x & 31) == 0) {
        s_v[threadIdx.x >> 5] = v;
        s_e[threadIdx.x >> 5] = e;
    }
    __syncthreads();
    if (threadIdx.x < 2) {  // one atomic a block: they meet at one address
        const uint64_t* s = threadIdx.x ? s_e : s_v;
        uint64_t all = 0;
        for (int k = 0; k < WARPS; ++k) all |= s[k];
        if (all) atomicOr(&bits[threadIdx.x], static_cast<unsigned long long>(all));
    }
}

// Pass p reads the input or the previous pass's output; the passes alternate
// between `tmp` and `out` so that the last one writes `out`.
__global__ void rs_plan(const unsigned long long* __restrict__ bits, const uint64_t* in_k, const uint32_t* in_v,
                        uint64_t* out_k, uint32_t* out_v, uint64_t* tmp_k, uint32_t* tmp_v, Plan* plan) {
    uint64_t need = bits[0] & (bits[1] | 1ull << 63);
    int n = 0;
    for (; need && n < PASSES; ++n) {
        Digit d{};
        int width = 0;
        for (int run = 0; run < 4 && need && width < 8; ++run) {
            const int b = __ffsll(static_cast<long long>(need)) - 1;
            const uint64_t up = ~(need >> b);  // its lowest set bit ends the run
            int w = up ? __ffsll(static_cast<long long>(up)) - 1 : 64;
            if (w > 8 - width) w = 8 - width;
            d.shift[run] = static_cast<uint32_t>(b - width);  // at least `width` bits lie below b
            d.mask[run] = ((1u << w) - 1u) << width;
            need &= ~(((1ull << w) - 1ull) << b);
            width += w;
        }
        plan->digit[n] = d;
    }
    plan->passes = n;
    for (int p = 0; p < n; ++p) {
        // an odd number of passes to go (this one included) writes the output
        const bool out = ((n - p) & 1) != 0;
        plan->src_k[p] = p == 0 ? in_k : out ? tmp_k : out_k;
        plan->src_v[p] = p == 0 ? in_v : out ? tmp_v : out_v;
        plan->dst_k[p] = out ? out_k : tmp_k;
        plan->dst_v[p] = out ? out_v : tmp_v;
    }
}

__global__ void rs_copy(const Plan* __restrict__ plan, const uint64_t* __restrict__ in_k,
                        const uint32_t* __restrict__ in_v, uint64_t* __restrict__ out_k, uint32_t* __restrict__ out_v,
                        uint64_t n) {
    if (plan->passes) return;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(THREADS) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * THREADS) {
        out_k[i] = in_k[i];
        out_v[i] = in_v ? in_v[i] : static_cast<uint32_t>(i);
    }
}

__global__ void __launch_bounds__(THREADS) rs_hist(const Plan* __restrict__ plan, int p, uint64_t n,
                                                  uint32_t n_tiles, uint32_t* __restrict__ count) {
    if (p >= plan->passes) return;
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t* keys = plan->src_k[p];
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * TILE;
    const Digit digit = plan->digit[p];
    uint32_t d[ROUNDS];  // every load is in flight before the first count
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) {
        const uint64_t i = base + static_cast<uint64_t>(j) * THREADS + threadIdx.x;
        d[j] = i < n ? digit.of(keys[i]) : 256;
    }
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j)
        if (d[j] < 256) atomicAdd(&h[d[j]], 1u);
    __syncthreads();
    count[static_cast<uint64_t>(threadIdx.x) * n_tiles + blockIdx.x] = h[threadIdx.x];
}

// One block per digit: count[d][*] becomes its exclusive prefix over the
// tiles; total[d] the digit's count.
__global__ void __launch_bounds__(THREADS) rs_scan(const Plan* __restrict__ plan, int p, uint32_t n_tiles,
                                                  uint32_t* __restrict__ count, uint64_t* __restrict__ total) {
    if (p >= plan->passes) return;
    __shared__ uint64_t part[THREADS];
    uint32_t* c = count + static_cast<uint64_t>(blockIdx.x) * n_tiles;
    const uint32_t per = (n_tiles + THREADS - 1) / THREADS;
    const uint32_t a = threadIdx.x * per;
    const uint32_t b = a + per < n_tiles ? a + per : n_tiles;
    uint64_t s = 0;
    for (uint32_t i = a; i < b; ++i) s += c[i];
    part[threadIdx.x] = s;
    __syncthreads();
    for (int o = 1; o < THREADS; o <<= 1) {  // inclusive scan of the parts
        const uint64_t v = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    uint64_t run = part[threadIdx.x] - s;
    for (uint32_t i = a; i < b; ++i) {
        const uint32_t v = c[i];
        c[i] = static_cast<uint32_t>(run);  // a tile prefix stays below n <= 2^32
        run += v;
    }
    if (threadIdx.x == THREADS - 1) total[blockIdx.x] = part[THREADS - 1];
}

// Exclusive prefix of v over the block's threads; `part` is shared, one
// value a warp.
template <class T>
__device__ __forceinline__ T block_exclusive(T v, T* part) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) part[w] = x;
    __syncthreads();
    T before = 0;
    for (int k = 0; k < w; ++k) before += part[k];
    return before + x - v;
}

// Bound by the issue of the ranking (about 130 instructions for 32 keys) and
// the waits on shared memory between its steps.  A warp takes ROUNDS * 32
// consecutive keys, all loaded at once, and ranks them 32 at a time against
// its own counters, with no barrier between the rounds; the lanes of equal
// digit come from eight ballots.  The tile is then put in digit order in
// shared memory, so that neighbouring threads store to neighbouring
// addresses.  A pass over 4 M pairs takes 30 us (3.2 TB/s); with counters
// that the block's warps share, a barrier a round and each key stored from
// where it was read, 44.  __match_any_sync for the ballots takes 32, half
// the keys a thread at twice the threads 33.
__global__ void __launch_bounds__(THREADS, 3) rs_scatter(const Plan* __restrict__ plan, int p, uint64_t n,
                                                        uint32_t n_tiles, const uint32_t* __restrict__ count,
                                                        const uint64_t* __restrict__ total) {
    if (p >= plan->passes) return;
    __shared__ uint64_t s_key[TILE];          // the tile in digit order: keys, then values
    __shared__ uint16_t s_cnt[WARPS][256];  // per warp: keys of digit d so far, then those of the warps before
    __shared__ uint64_t s_base[256];          // output index of tile position 0, were the tile all digit d
    __shared__ uint32_t s_start[256];         // tile position of the first key of digit d
    __shared__ uint64_t s_part[WARPS];
    __shared__ uint32_t s_part32[WARPS];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const uint64_t* sk = plan->src_k[p];
    const uint32_t* sv = plan->src_v[p];
    uint64_t* dk = plan->dst_k[p];
    uint32_t* dv = plan->dst_v[p];
    const Digit digit = plan->digit[p];
    const uint64_t tile0 = static_cast<uint64_t>(blockIdx.x) * TILE;
    const int here = static_cast<int>(n - tile0 < TILE ? n - tile0 : TILE);
    const int first = w * (32 * ROUNDS) + lane;  // tile position of the lane's first key
    uint64_t key[ROUNDS];
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) {
        const int i = first + 32 * j;
        key[j] = i < here ? sk[tile0 + i] : ~0ull;  // past the end: the last digit, after every key of the tile
    }
    for (int k = lane; k < 256; k += 32) s_cnt[w][k] = 0;
    __syncwarp();
    const unsigned lt = (1u << lane) - 1u;
    uint32_t rank[ROUNDS / 2];  // two 16-bit ranks each
    uint32_t dg[ROUNDS / 4];    // four digits each
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) {
        const uint32_t d = digit.of(key[j]);
        if (j & 3) dg[j / 4] |= d << (8 * (j & 3));
        else dg[j / 4] = d;
        unsigned peers = 0xFFFFFFFFu;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const bool bit = (d >> b) & 1u;
            const unsigned m = __ballot_sync(0xFFFFFFFFu, bit);
            peers &= bit ? m : ~m;
        }
        const uint32_t before = s_cnt[w][d];
        const uint32_t in_warp = __popc(peers & lt);
        __syncwarp();
        if (in_warp == 0) s_cnt[w][d] = static_cast<uint16_t>(before + __popc(peers));
        __syncwarp();
        const uint32_t r = before + in_warp;
        if (j & 1) rank[j / 2] |= r << 16;
        else rank[j / 2] = r;
    }
    __syncthreads();
    {  // thread t: digit t
        uint32_t run = 0;
#pragma unroll
        for (int k = 0; k < WARPS; ++k) {
            const uint32_t c = s_cnt[k][t];
            s_cnt[k][t] = static_cast<uint16_t>(run);
            run += c;
        }
        const uint32_t start = block_exclusive(run, s_part32);
        const uint64_t digit0 = block_exclusive(total[t], s_part);
        s_start[t] = start;
        s_base[t] = digit0 + count[static_cast<uint64_t>(t) * n_tiles + blockIdx.x] - start;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) {
        const uint32_t d = (dg[j / 4] >> (8 * (j & 3))) & 0xFFu;
        const uint32_t pos = s_start[d] + s_cnt[w][d] + ((rank[j / 2] >> (16 * (j & 1))) & 0xFFFFu);
        s_key[pos] = key[j];
        if (j & 1) rank[j / 2] = (rank[j / 2] & 0xFFFFu) | pos << 16;
        else rank[j / 2] = (rank[j / 2] & 0xFFFF0000u) | pos;
    }
    uint32_t val[ROUNDS];
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) {
        const int i = first + 32 * j;
        val[j] = i >= here ? 0u : sv ? sv[tile0 + i] : static_cast<uint32_t>(tile0 + i);
    }
    __syncthreads();
    uint32_t to[ROUNDS];  // output index of tile position t + THREADS * j
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) {
        const int i = t + THREADS * j;
        to[j] = 0xFFFFFFFFu;
        if (i < here) {
            const uint64_t k = s_key[i];
            const uint64_t o = s_base[digit.of(k)] + i;
            if (o < n) {  // always true; the check keeps a wrong count from writing past the end
                dk[o] = k;
                to[j] = static_cast<uint32_t>(o);
            }
        }
    }
    __syncthreads();
    uint32_t* s_val = reinterpret_cast<uint32_t*>(s_key);
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) s_val[(rank[j / 2] >> (16 * (j & 1))) & 0xFFFFu] = val[j];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j)
        if (to[j] < n) dv[to[j]] = s_val[t + THREADS * j];
}

inline uint32_t tiles_for(uint64_t n) { return static_cast<uint32_t>((n + TILE - 1) / TILE); }

// Device scratch of a sort of n pairs.
inline size_t scratch_bytes(uint64_t n) {
    auto a256 = [](size_t b) { return (b + 255) & ~static_cast<size_t>(255); };
    const uint64_t nt = tiles_for(n ? n : 1);
    return a256(n * 8) + a256(n * 4) + a256(256 * nt * 4) + a256(256 * 8) + a256(sizeof(Plan)) + a256(16);
}

// Sorts (in_k, in_v) into (out_k, out_v); n >= 1, below 2^32.  A null in_v
// stands for 0, 1, .., n - 1.  Returns the kernels enqueued.
inline int sort_pairs(const uint64_t* in_k, const uint32_t* in_v, uint64_t* out_k, uint32_t* out_v, uint64_t n,
                      void* scratch, int sm_count, cudaStream_t st) {
    auto a256 = [](size_t b) { return (b + 255) & ~static_cast<size_t>(255); };
    const uint32_t nt = tiles_for(n);
    uint8_t* s = static_cast<uint8_t*>(scratch);
    uint64_t* tmp_k = reinterpret_cast<uint64_t*>(s);
    s += a256(n * 8);
    uint32_t* tmp_v = reinterpret_cast<uint32_t*>(s);
    s += a256(n * 4);
    uint32_t* count = reinterpret_cast<uint32_t*>(s);
    s += a256(256 * static_cast<size_t>(nt) * 4);
    uint64_t* total = reinterpret_cast<uint64_t*>(s);
    s += a256(256 * 8);
    Plan* plan = reinterpret_cast<Plan*>(s);
    s += a256(sizeof(Plan));
    unsigned long long* bits = reinterpret_cast<unsigned long long*>(s);
    cudaMemsetAsync(bits, 0, 16, st);
    const unsigned grid = static_cast<unsigned>(sm_count > 0 ? sm_count * 8 : 1184);
    rs_bits<<<grid, THREADS, 0, st>>>(in_k, n, bits);
    rs_plan<<<1, 1, 0, st>>>(bits, in_k, in_v, out_k, out_v, tmp_k, tmp_v, plan);
    rs_copy<<<grid, THREADS, 0, st>>>(plan, in_k, in_v, out_k, out_v, n);
    for (int p = 0; p < PASSES; ++p) {
        rs_hist<<<nt, THREADS, 0, st>>>(plan, p, n, nt, count);
        rs_scan<<<256, THREADS, 0, st>>>(plan, p, nt, count, total);
        rs_scatter<<<nt, THREADS, 0, st>>>(plan, p, n, nt, count, total);
    }
    return 3 + 3 * PASSES;
}

}  // namespace radix
}  // namespace ma
