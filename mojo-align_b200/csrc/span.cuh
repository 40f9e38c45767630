// span.cuh - device helpers of the kernels that write byte records of any
// length one after the other (BAM records, SAM lines): eight-byte windows of
// unaligned source spans, and a warp's shared-memory stage of its output.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace ma {
namespace span {

// Bytes 8i .. 8i+7 of a span of n bytes, in order or (rev) of the span read
// backwards: the aligned words that cover them, loaded where they hold a byte
// of the span, and then the bytes as two words (what lies outside the span is
// undefined).
struct Span8 {
    uint32_t w0, w1, w2;
};

__device__ __forceinline__ Span8 span8_load(const uint8_t* src, uint32_t n, uint32_t i, bool rev) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(src);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
    const uint32_t lead = static_cast<uint32_t>(a & 3), nw = (lead + n + 3) >> 2;
    const uint32_t k = rev ? ((lead + n) >> 2) - 2 - 2 * i : 2 * i;  // first word; wraps below the span's start
    w += static_cast<int32_t>(k);
    Span8 s;
    s.w0 = k < nw ? __ldg(w) : 0;
    s.w1 = k + 1 < nw ? __ldg(w + 1) : 0;
    s.w2 = k + 2 < nw ? __ldg(w + 2) : 0;
    return s;
}

__device__ __forceinline__ uint2 span8_bytes(const Span8& s, const uint8_t* src, uint32_t n, bool rev) {
    const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src));
    const uint32_t sh = ((rev ? lead + n : lead) & 3) * 8;
    const uint32_t lo = __funnelshift_r(s.w0, s.w1, sh), hi = __funnelshift_r(s.w1, s.w2, sh);
    return rev ? make_uint2(__byte_perm(hi, 0, 0x0123), __byte_perm(lo, 0, 0x0123)) : make_uint2(lo, hi);
}

// The first n (1 .. 4) bytes of v at p.
__device__ __forceinline__ void put_bytes(uint8_t* p, uint32_t v, uint32_t n) {
    p[0] = static_cast<uint8_t>(v);
    if (n > 1) p[1] = static_cast<uint8_t>(v >> 8);
    if (n > 2) p[2] = static_cast<uint8_t>(v >> 16);
    if (n > 3) p[3] = static_cast<uint8_t>(v >> 24);
}

// Stores stage[from, to) (stage[0] stands for the 16-byte aligned address
// g): 16-byte stores, byte stores where a block is not whole.
__device__ __forceinline__ void store_stage(uint8_t* g, const uint8_t* stage, uint32_t from, uint32_t to,
                                            uint32_t lane) {
    const uint32_t a = (from + 15) & ~15u, e = to & ~15u;
    for (uint32_t i = a + 16 * lane; i < e; i += 512)
        *reinterpret_cast<uint4*>(g + i) = *reinterpret_cast<const uint4*>(stage + i);
    if (a > from) {  // the first block is not whole
        const uint32_t i = from + lane;
        if (i < min(a, to)) g[i] = stage[i];
    }
    if (to > e && e >= a) {  // the last one
        const uint32_t i = e + lane;
        if (i < to) g[i] = stage[i];
    }
}

// The warp writes `count` records (record k: the size in lane k's `bytes`)
// one after the other from the address g on.  write(dst, k), called once per
// record in order, puts record k at dst: in the warp's stage (STAGE + 16
// bytes of shared memory, 16-byte aligned), which stands for the output at
// its 16-byte phase and is stored in 16-byte blocks when the next record does
// not fit, or in place in the output when the record is longer than the stage.
template <uint32_t STAGE, typename F>
__device__ __forceinline__ void staged_run(uint8_t* g, uint8_t* stage, uint32_t bytes, uint32_t count, uint32_t lane,
                                           F&& write) {
    constexpr unsigned FULL = 0xffffffffu;
    uint32_t from = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(g) & 15);  // the stage's first own byte
    uint32_t fill = from;
    g -= from;
    for (uint32_t k = 0; k < count; ++k) {
        const uint32_t n = __shfl_sync(FULL, bytes, k);
        if (fill + n > STAGE || fill + n < n) {
            __syncwarp();
            // the whole blocks; what is left of the last one moves to the front
            const uint32_t e = fill & ~15u;
            if (e > from) {
                store_stage(g, stage, from, e, lane);
                const uint8_t v = lane < fill - e ? stage[e + lane] : 0;
                __syncwarp();
                if (lane < fill - e) stage[lane] = v;
                __syncwarp();
                g += e;
                fill -= e;
                from = 0;
            }
            if (fill + n > STAGE || fill + n < n) {  // longer than the stage
                store_stage(g, stage, from, fill, lane);
                write(g + fill, k);
                __syncwarp();
                g += fill + static_cast<uint64_t>(n);
                from = fill = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(g) & 15);
                g -= from;
                continue;
            }
        }
        write(stage + fill, k);
        fill += n;
    }
    __syncwarp();
    if (fill > from) store_stage(g, stage, from, fill, lane);
    __syncwarp();
}

}  // namespace span
}  // namespace ma
