// bgzf_inflate.cu - BGZF members inflated on the device (bgzf_inflate.cuh), one
// CTA per member, a grid-stride loop over the members, and one warp per member
// for those that the CTAs leave.
//
// A deflate stream is serial: where a code starts is known once the codes
// before it are read.  But a decoder that starts in mid-stream falls into step
// with the true codes after a few of them, so a block is read by all threads
// at once:
//   sync     thread i decodes from bit 224 i of the block on to bit
//            224 (i + 1), keeping where it ended; a thread whose
//            neighbour ended elsewhere than it began starts again from there,
//            until nothing changes.  The first threads' starts are then exact
//            by induction, and the block ends in the first of them that met
//            the end-of-block code;
//   place    a block scan of the bytes each thread's codes produce;
//   write    each thread decodes once more and writes a 16-bit cell where a
//            code's output starts: 0xff00 | byte, or the position it copies from
//            (BGZF pieces have at most 0xff00 bytes, so positions and bytes do
//            not meet), and a bit that tells the starts;
//   resolve  strips of 3968 bytes in order: each byte gets its own cell from
//            the code it belongs to and follows positions until it meets a
//            byte; those before the strip are bytes already, so only chains
//            inside the strip take more than one step.  The bytes go to the
//            output from here;
//   CRC-32   66 bytes per thread, counted from the member's end (zero bytes
//            in front leave a CRC register of zero as it is), combined in GF(2).
// A second kernel, one warp per member (left_kernel: lane 0 decodes the stream
// code by code, inflate.cuh, the warp writes its bytes), takes what the first
// leaves: members that this form does not hold (more than 0xff00 bytes, as some
// writers fill them, or many blocks), members with anything invalid in them (it
// gives their status), and those that many warps finish sooner than the CTAs
// (Cost, Rounds).
// Every code's reads stay in the staged input and every cell in the member:
// sizes are checked before they are used.
// Bound by latency: per member of 65280 bytes of FASTQ the sync rounds take
// about 80 k cycles (segments of equal code lengths fall into step late), the
// write pass 25 k, the resolve 54 k, the CRC 11 k; the next member's header and
// tables (82 k by one warp) are read meanwhile.  128 MB in 1961 members (zlib
// level 6): 1.42 ms, 1.45 with one literal per table entry; segments of 96 bits
// 1.87, of 160 or 288 bits 1.46 and 1.49 ms, 3 to 5 checkpoints per segment that
// stop a second decode early 1.74 ms; all members in left_kernel 6.2 ms.
#include <string>

#include "bgzf_inflate.cuh"
#include "ma_internal.h"

namespace ma {
namespace {

constexpr int THREADS = 992;              // that work on a member; one more warp reads the next member's header
constexpr int WARPS = THREADS / 32;
constexpr int CTA_THREADS = THREADS + 32;
constexpr int LEFT_WARPS = 4;             // per block of left_kernel
constexpr uint32_t S_LEFT = 0xffffffffu;  // the status of a member that is left to it
constexpr uint32_t CRC_POLY = 0xEDB88320u;

struct __align__(16) WarpSmem {
    inflate::Tables t;
    inflate::Tok tok[inflate::BATCH_TOKENS];
    uint8_t lit[inflate::BATCH_LITERALS];
    uint32_t lane_crc[32];
    int ntok, status, done;
    uint32_t o0;
};

// a * b mod P in the reflected CRC-32 representation (bit 31 = x^0)
__device__ __forceinline__ uint32_t gf2_mul(uint32_t a, uint32_t b) {
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) {
        if (a & (0x80000000u >> i)) r ^= b;
        b = (b & 1u) ? (b >> 1) ^ CRC_POLY : b >> 1;
    }
    return r;
}

// x^k mod P
__device__ uint32_t gf2_xpow(uint64_t k) {
    uint32_t r = 0x80000000u, b = 0x40000000u;
    while (k) {
        if (k & 1) r = gf2_mul(r, b);
        b = gf2_mul(b, b);
        k >>= 1;
    }
    return r;
}

// CRC-32 of out[0, n) by the warp: lane l folds bytes [l*seg, (l+1)*seg)
// from a zero register; the parts are shifted by the bytes after them and
// added; the initial all-ones register and the final inversion are added
// last.  Lane 0 returns it.
__device__ uint32_t warp_crc(const uint8_t* out, uint32_t n, const uint32_t* crc_tab, WarpSmem& S, int lane) {
    const uint32_t seg = (n + 31) / 32;
    const uint32_t a = min(n, static_cast<uint32_t>(lane) * seg), b = min(n, a + seg);
    uint32_t c = 0;
    for (uint32_t i = a; i < b; ++i) c = (c >> 8) ^ crc_tab[(c ^ out[i]) & 255u];
    S.lane_crc[lane] = c;
    __syncwarp();
    uint32_t r = 0;
    if (lane == 0 && n) {
        const uint32_t x_seg = gf2_xpow(8ull * seg);
        for (int l = 0; l < 32; ++l) {
            const uint32_t la = min(n, static_cast<uint32_t>(l) * seg), lb = min(n, la + seg);
            if (lb > la) r = gf2_mul(r, lb - la == seg ? x_seg : gf2_xpow(8ull * (lb - la))) ^ S.lane_crc[l];
        }
    }
    if (lane == 0) r = r ^ gf2_mul(0xffffffffu, gf2_xpow(8ull * n)) ^ 0xffffffffu;
    __syncwarp();
    return r;
}

// Member m by the warp, its spans checked; returns its status (valid in lane 0).
__device__ uint32_t warp_member(const bgzf_inflate::Job& j, uint32_t m, WarpSmem& S, const uint32_t* crc_tab,
                                int lane) {
    const uint8_t* in = j.in + j.src_off[m];
    uint8_t* out = j.out + j.dst_off[m];
    const uint32_t isz = j.isize[m];
    inflate::Stream st;  // lane 0's decoder state
    if (lane == 0) inflate::stream_init(st, in, j.src_len[m], isz);
    for (;;) {
        if (lane == 0) {
            S.o0 = st.o;
            S.ntok = inflate::decode_tokens(st, S.t, S.tok, inflate::BATCH_TOKENS, S.lit, inflate::BATCH_LITERALS);
            S.status = st.status;
            S.done = st.finished || st.status != inflate::OK;
        }
        __syncwarp();
        const int ntok = S.ntok;
        uint32_t o = S.o0;
        for (int i = 0; i < ntok; ++i) {
            const inflate::Tok k = S.tok[i];
            if (k.dist == inflate::TOK_LITERAL) {
                for (uint32_t x = lane; x < k.len; x += 32) out[o + x] = S.lit[k.src + x];
            } else if (k.dist == inflate::TOK_STORED) {
                for (uint32_t x = lane; x < k.len; x += 32) out[o + x] = in[k.src + x];
            } else {
                for (uint32_t x = lane; x < k.len; x += 32) out[o + x] = out[o - k.dist + x % k.dist];
            }
            o += k.len;
            __syncwarp();
        }
        const bool done = S.done;
        __syncwarp();
        if (done) break;
    }
    const int status = S.status;
    if (status != inflate::OK) return static_cast<uint32_t>(status);
    // the decoder stopped at the final block: the bytes written are its output
    uint32_t got = 0;
    if (lane == 0) got = st.o;
    got = __shfl_sync(0xFFFFFFFFu, got, 0);
    if (got != isz) return bgzf_inflate::S_SIZE;
    const uint32_t c = warp_crc(out, got, crc_tab, S, lane);
    return c == j.crc[m] ? 0u : bgzf_inflate::S_CRC;
}

// The members that the CTAs left.
__global__ void __launch_bounds__(LEFT_WARPS * 32) left_kernel(bgzf_inflate::Job j) {
    __shared__ WarpSmem smem[LEFT_WARPS];
    __shared__ uint32_t crc_tab[256];
    bgzf_inflate::crc_table(crc_tab, static_cast<int>(threadIdx.x), LEFT_WARPS * 32);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t n_warps = static_cast<uint64_t>(gridDim.x) * LEFT_WARPS;
    for (uint64_t m = static_cast<uint64_t>(blockIdx.x) * LEFT_WARPS + warp; m < j.n; m += n_warps) {
        if (j.status[m] != S_LEFT) continue;
        __syncwarp();
        const uint32_t s = warp_member(j, static_cast<uint32_t>(m), smem[warp], crc_tab, lane);
        if (lane == 0) j.status[m] = s;
        __syncwarp();
    }
}

constexpr uint32_t MAX_BYTES = 0xff00;   // output bytes of a member in cells
constexpr uint32_t SEG_WORDS = 7;        // bits per thread: an odd number of words, so the threads' reads spread over the banks
constexpr uint32_t SEG_BITS = 32 * SEG_WORDS;
constexpr uint32_t IN_WORDS = THREADS * SEG_WORDS + 8;  // 8: the first bits' offset, a code and the words read ahead
constexpr uint32_t HEAD_WORDS = 160;     // a block's header: at most 17 + 57 + 316 * 14 bits
constexpr int LIT_BITS = 12, DIST_BITS = 10;  // longer codes are rare enough that few warps meet one
constexpr int MAX_BLOCKS = 64;
constexpr uint32_t CRC_BYTES = 66;       // per thread: 33 words apart in the cells, one bank each
static_assert(THREADS * CRC_BYTES >= MAX_BYTES, "the CRC covers a member");
constexpr int STRIP = 4 * THREADS;

// Decoding table entries: bits 0-3 code length, 4-5 kind, 6-9 extra bits,
// 16-31 value (the length's or distance's base).  Of a literal: 7-10 its code
// length, 16-23 the byte; where the table's bits hold another literal after it
// bit 6 is set, 24-31 are that byte, and 0-3 the length of both codes.
enum : uint32_t { K_LITERAL = 0, K_COPY = 1, K_END = 2, K_OTHER = 3 };  // K_OTHER: longer than the table's bits, or no code

// The canonical codes of an alphabet: of length l, `count` codes from `first`
// on, their symbols from symbol[index] on.
struct Canon {
    uint32_t count[16], first[16], index[16];
    uint16_t symbol[inflate::NLIT];
};

// A block's header and the tables of its codes.
struct Head {
    uint32_t lit[1 << LIT_BITS], dist[1 << DIST_BITS];
    Canon cl, cd;
    uint8_t lens[inflate::NLIT + inflate::NDIST];
    uint32_t in[HEAD_WORDS + 2];
    uint32_t pos;   // bit of the stream after the header
    uint32_t type, last, nlit, ndist, ok;
    uint32_t flat;  // all but an eighth of the literal codes are of one length
};

struct __align__(16) Smem {
    uint16_t cell[MAX_BYTES];
    Head head[2];  // the member's, and the next one's
    uint32_t in[IN_WORDS];
    uint32_t starts[(MAX_BYTES + 31) / 32];  // a code's output (or a piece of it) starts at this byte
    uint32_t crc[4][256];
    uint32_t xpow[10];  // x^(8 CRC_BYTES 2^k)
    uint32_t end[THREADS];
    uint32_t part[32];
    uint32_t carry_at, carry_cell;  // the code that a strip begins in
    uint32_t first_flag;
    uint32_t mine[CTA_THREADS / 32];  // which of the CTA's next members it takes
    uint32_t stopped;                 // it takes no more of them
    unsigned long long cta_ns, warp_ns;  // of those that warps are faster at: in the CTA all, in a warp the slowest
};

// Barriers of the THREADS that work on a member (the header warp takes none).
__device__ __forceinline__ void work_sync() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }
__device__ __forceinline__ bool work_or(bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"(static_cast<uint32_t>(v)), "n"(THREADS)
        : "memory");
    return r != 0;
}

// Words [0, words) of `to`: the stream's bytes from `base` (a multiple of 4)
// on, zero past its end.
__device__ void stage_input(uint32_t* to, uint32_t words, const uint8_t* in, uint32_t n, uint32_t base, uint32_t t,
                            uint32_t threads) {
    const uintptr_t a0 = reinterpret_cast<uintptr_t>(in) + base, end = reinterpret_cast<uintptr_t>(in) + n;
    const uint32_t sh = static_cast<uint32_t>(a0 & 3) * 8;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(a0 & ~uintptr_t(3));
    for (uint32_t i = t; i < words; i += threads) {
        const uint32_t at = base + 4 * i;  // below 2^27 + 2^15
        uint32_t v = 0;
        if (at < n) {
            const uint32_t lo = __ldg(w + i);
            const uint32_t hi = sh && reinterpret_cast<uintptr_t>(w + i + 1) < end ? __ldg(w + i + 1) : 0;
            v = __funnelshift_r(lo, hi, sh);
            if (n - at < 4) v &= (1u << (8 * (n - at))) - 1;
        }
        to[i] = v;
    }
}

// The 64 bits of the staged input from bit pos on, as two words.
struct Window {
    uint32_t lo, hi;
    __device__ __forceinline__ Window(const uint32_t* in, uint32_t pos) {
        const uint32_t* w = in + (pos >> 5);
        const uint32_t a = w[0], b = w[1], c = w[2], sh = pos & 31;
        lo = __funnelshift_r(a, b, sh);
        hi = __funnelshift_r(b, c, sh);
    }
    __device__ __forceinline__ uint32_t from(uint32_t k) const { return __funnelshift_r(lo, hi, k); }  // k < 32
};

__device__ __forceinline__ uint32_t low_bits(uint32_t v, uint32_t k) { return v & ((1u << k) - 1); }  // k < 32

// Canonical codes of lens[0, n) by a warp; false when zlib rejects the set
// (inflate::build's rules; kind as there).
__device__ bool canon_build(Canon& c, const uint8_t* lens, int n, int kind, int lane) {
    if (lane < 16) c.count[lane] = 0;
    __syncwarp();
    for (int s = lane; s < n; s += 32) atomicAdd(&c.count[lens[s]], 1u);
    __syncwarp();
    int left = 1, max_len = 0;
    uint32_t first = 0, index = 0;
    bool ok = true;
    for (int l = 1; l <= 15; ++l) {
        const uint32_t k = c.count[l];
        left = 2 * left - static_cast<int>(k);
        if (left < 0) ok = false;
        if (k) max_len = l;
        if (lane == 0) {
            c.first[l] = first;
            c.index[l] = index;
        }
        first = (first + k) << 1;
        index += k;
        if (!ok) break;
    }
    if (!ok || (left > 0 && index > 0 && (kind == 0 || max_len != 1))) return false;
    __syncwarp();
    for (int b = 0; b < n; b += 32) {  // symbols of a length in order; index[] moves past them
        const int s = b + lane;
        const uint32_t l = s < n ? lens[s] : 0;
        const uint32_t peers = __match_any_sync(0xffffffffu, l);
        const uint32_t at = l ? c.index[l] + __popc(peers & ((1u << lane) - 1)) : 0;
        if (l) c.symbol[at] = static_cast<uint16_t>(s);
        __syncwarp();
        if (l && lane == 31 - __clz(peers)) c.index[l] = at + 1;
        __syncwarp();
    }
    if (lane >= 1 && lane < 16) c.index[lane] -= c.count[lane];
    __syncwarp();
    return true;
}

// Symbol of the code at the head of the 15 bits v (first bit on top), of at
// least `from` and at most `to` bits; -1: none.
__device__ __forceinline__ int canon_find(const Canon& c, uint32_t v, int from, int to, uint32_t& bits) {
    for (int l = from; l <= to; ++l) {
        const uint32_t off = (v >> (15 - l)) - c.first[l];
        if (off < c.count[l]) {
            bits = l;
            return c.symbol[c.index[l] + off];
        }
    }
    return -1;
}

__device__ __forceinline__ uint32_t lit_entry(int sym, uint32_t bits) {
    if (sym < 0 || sym > 285) return K_OTHER << 4;
    if (sym < 256) return bits | bits << 7 | static_cast<uint32_t>(sym) << 16;
    if (sym == 256) return bits | K_END << 4;
    const int i = sym - 257;
    return bits | K_COPY << 4 | static_cast<uint32_t>(inflate::len_extra(i)) << 6 | inflate::len_base(i) << 16;
}

__device__ __forceinline__ uint32_t dist_entry(int sym, uint32_t bits) {
    if (sym < 0 || sym > 29) return K_OTHER << 4;
    return bits | static_cast<uint32_t>(inflate::dist_extra(sym)) << 6 | inflate::dist_base(sym) << 16;
}

// The code of an alphabet at the head of the bits v: its table entry, or for
// a code longer than the table's bits the same from the canonical codes.
template <int BITS, typename F>
__device__ __forceinline__ uint32_t entry_at(uint32_t v, const uint32_t* table, const Canon& c, F entry) {
    uint32_t e = table[low_bits(v, BITS)];
    if (((e >> 4) & 3) == K_OTHER) {
        uint32_t bits = 0;
        const int sym = canon_find(c, __brev(v) >> 17, BITS + 1, 15, bits);
        e = entry(sym, bits);
    }
    return e;
}

enum : uint32_t { F_NONE = 0, F_END = 1, F_BAD = 2 };

// Decodes the codes that start in bits [pos, limit) of the staged input, in
// the lanes that are `on`; called by whole warps, whose lanes step from code to
// code together (left to themselves, lanes on literals and lanes on copies
// part for good and the warp runs them one by one).  Returns how it ended
// (F_END: `end` is past the end-of-block code; F_BAD: no code, past bit n_bits,
// or WRITE a distance that reaches before the output); o moves past the bytes
// they produce.  WRITE: a cell (byte, or the position copied from) and a bit in
// S.starts where each one's output starts.
template <bool WRITE>
__device__ __forceinline__ uint32_t decode_bits(Smem& S, const Head& H, bool on, uint32_t pos, uint32_t limit,
                                                uint32_t n_bits, uint32_t& end, uint32_t& o) {
    uint32_t flag = pos < n_bits ? F_NONE : F_BAD;
    bool go = on && flag == F_NONE && pos < limit;
    while (__any_sync(0xffffffffu, go)) {
        if (go) {
            const Window w(S.in, pos);
            const uint32_t e = entry_at<LIT_BITS>(w.lo, H.lit, H.cl, lit_entry);
            const uint32_t kind = (e >> 4) & 3;
            uint32_t used = e & 15, v = 0xff00u | ((e >> 16) & 0xff), len = 1, dist = 1;
            bool two = false;
            if (kind == K_LITERAL) {
                // a second literal that starts past the limit is the next
                // segment's: where a segment ends must not depend on how its
                // literals fall into pairs, or starts would take longer to settle
                const uint32_t b1 = (e >> 7) & 15;
                two = (e & 64) && pos + b1 < limit;
                if (two) len = 2;
                else used = b1;
            } else if (kind == K_COPY) {
                const uint32_t eb = (e >> 6) & 15;
                len = (e >> 16) + low_bits(w.lo >> used, eb);
                used += eb;  // at most 20
                const uint32_t x = w.from(used);
                const uint32_t d = entry_at<DIST_BITS>(x, H.dist, H.cd, dist_entry);
                const uint32_t db = d & 15, deb = (d >> 6) & 15;  // at most 28 bits
                dist = (d >> 16) + low_bits(x >> db, deb);
                used += db + deb;
                if (((d >> 4) & 3) == K_OTHER || (WRITE && dist > o)) flag = F_BAD;
                v = o - dist;
            } else {
                flag = kind == K_END ? F_END : F_BAD;
            }
            pos += used;
            if (flag == F_NONE) {
                if (WRITE && two) {
                    S.cell[o] = static_cast<uint16_t>(v);
                    S.cell[o + 1] = static_cast<uint16_t>(0xff00u | (e >> 24));
                    atomicOr(S.starts + (o >> 5), 3u << (o & 31));
                    if ((o & 31) == 31) atomicOr(S.starts + (o >> 5) + 1, 1u);
                } else if (WRITE) {
                    // a copy that overlaps itself in pieces of dist, 2 dist,
                    // 4 dist ... bytes, each of which copies from v on, where
                    // the pieces before it have put as many
                    for (;;) {
                        S.cell[o] = static_cast<uint16_t>(v);
                        atomicOr(S.starts + (o >> 5), 1u << (o & 31));
                        if (len <= dist) break;
                        o += dist;
                        len -= dist;
                        dist *= 2;
                    }
                }
                o += len;
            }
            go = flag == F_NONE && pos < limit;
        }
    }
    end = pos;
    return flag;
}

// The decoding table of an alphabet by `threads` threads: entry brev(v) for
// the BITS bits v (first bit on top).  In the order of v the codes come in
// canonical order, so a thread looks up its first v and walks on.
template <int BITS, typename F>
__device__ __forceinline__ void fill_table(uint32_t* table, const Canon& c, uint32_t t, uint32_t threads, F entry) {
    const uint32_t per = ((1u << BITS) + threads - 1) / threads;
    uint32_t v = t * per, upto = 0, e = K_OTHER << 4;
    for (uint32_t k = 0; k < per && v < (1u << BITS); ++k, ++v) {
        if (v >= upto) {
            uint32_t bits = 0;
            const int sym = canon_find(c, v << (15 - BITS), 1, BITS, bits);
            e = entry(sym, bits);
            upto = sym < 0 ? v + 1 : ((v >> (BITS - bits)) + 1) << (BITS - bits);
        }
        table[__brev(v) >> (32 - BITS)] = e;
    }
}

// Exclusive prefix of v over the THREADS; `total` the sum.
__device__ __forceinline__ uint32_t block_scan(Smem& S, uint32_t v, uint32_t t, uint32_t& total) {
    const uint32_t lane = t & 31, warp = t >> 5;
    uint32_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) S.part[warp] = incl;
    work_sync();
    uint32_t before = 0, sum = 0;
    for (uint32_t w = 0; w < WARPS; ++w) {
        if (w < warp) before += S.part[w];
        sum += S.part[w];
    }
    work_sync();
    total = sum;
    return before + incl - v;
}

// The header of the block at bit `pos` of the stream and, for a compressed
// block, its canonical codes, by one warp.  H.ok 0: anything invalid.
__device__ void read_head(Head& H, const uint8_t* in, uint32_t n, uint32_t pos, int lane) {
    const uint32_t base = (pos >> 3) & ~3u, p0 = pos - 8 * base;
    stage_input(H.in, HEAD_WORDS + 2, in, n, base, static_cast<uint32_t>(lane), 32);
    __syncwarp();
    const Window w(H.in, p0);
    const uint32_t type = low_bits(w.lo >> 1, 2);
    uint32_t nlit = inflate::NLIT, ndist = inflate::NDIST, at = p0 + 3;
    bool ok = type != 3;
    if (type == 1) {
        for (int v = lane; v < inflate::NLIT; v += 32) H.lens[v] = v < 144 ? 8 : v < 256 ? 9 : v < 280 ? 7 : 8;
        H.lens[inflate::NLIT + lane] = 5;
    } else if (type == 2) {
        nlit = low_bits(w.lo >> 3, 5) + 257;
        ndist = low_bits(w.lo >> 8, 5) + 1;
        at = p0 + 17 + 3 * (low_bits(w.lo >> 13, 4) + 4);
        ok = nlit <= 286 && ndist <= 30;
        if (lane < 19) {
            // the lane-th length in the order 16, 17, 18, 0, 8, 7, 9, 6, 10, ...
            const uint32_t b = p0 + 17 + 3 * lane;
            const int sym = lane < 3 ? 16 + lane : lane == 3 ? 0 : (lane & 1) ? 8 - ((lane - 3) >> 1) : 8 + ((lane - 4) >> 1);
            H.lens[sym] = b < at ? static_cast<uint8_t>(Window(H.in, b).lo & 7) : 0;
        }
        __syncwarp();
        // the code-length codes, their 7-bit table in the distance table's place
        ok = ok && canon_build(H.cd, H.lens, 19, 0, lane);
        if (ok) {
            for (int i = lane; i < 128; i += 32) {
                uint32_t bits = 0;
                const int sym = canon_find(H.cd, __brev(static_cast<uint32_t>(i)) >> 17, 1, 7, bits);
                H.dist[i] = sym < 0 ? K_OTHER << 4 : bits | static_cast<uint32_t>(sym) << 16;
            }
        }
        __syncwarp();
        if (ok && lane == 0) {
            const uint32_t total = nlit + ndist;
            uint32_t i = 0, prev = 0;
            while (ok && i < total) {
                const uint32_t v = __funnelshift_r(H.in[at >> 5], H.in[(at >> 5) + 1], at & 31);
                const uint32_t e = H.dist[v & 127], sym = e >> 16, x = v >> (e & 15);
                at += e & 15;
                uint32_t rep = 1;
                if (sym < 16) {
                    prev = sym;
                    ok = e != K_OTHER << 4;
                } else {
                    const uint32_t eb = sym == 16 ? 2 : sym == 17 ? 3 : 7;
                    rep = (sym == 18 ? 11 : 3) + low_bits(x, eb);
                    at += eb;
                    if (sym != 16) prev = 0;
                    ok = !(sym == 16 && i == 0) && i + rep <= total;
                }
                if (ok)
                    for (uint32_t k = 0; k < rep; ++k) H.lens[i + k] = static_cast<uint8_t>(prev);
                i += rep;
            }
            ok = ok && H.lens[256] != 0;  // an end-of-block code
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        at = __shfl_sync(0xffffffffu, at, 0);
    }
    __syncwarp();
    if (ok && type != 0) {
        ok = canon_build(H.cl, H.lens, static_cast<int>(nlit), 1, lane);
        ok = ok && canon_build(H.cd, H.lens + nlit, static_cast<int>(ndist), 1, lane);
    }
    const uint32_t of_length = ok && type == 2 && lane >= 1 && lane < 16 ? H.cl.count[lane] << (15 - lane) : 0;
    const uint32_t flat = __any_sync(0xffffffffu, of_length > (7u << 12));
    if (lane == 0) {
        H.flat = flat;
        H.pos = 8 * base + at;
        H.type = type;
        H.last = w.lo & 1;
        H.ok = ok;
    }
    __syncwarp();
}

// The tables of H by `threads` threads that `sync` waits for.  The entries of
// two literals come from the single ones in place: one that is paired already
// still tells its first literal.
template <typename F>
__device__ __forceinline__ void fill_tables(Head& H, uint32_t t, uint32_t threads, F sync) {
    if (!H.ok || H.type == 0) return;
    fill_table<LIT_BITS>(H.lit, H.cl, t, threads, lit_entry);
    fill_table<DIST_BITS>(H.dist, H.cd, t, threads, dist_entry);
    sync();
    volatile uint32_t* lit = H.lit;
    for (uint32_t i = t; i < (1u << LIT_BITS); i += threads) {
        const uint32_t e = lit[i], b1 = (e >> 7) & 15;
        if (((e >> 4) & 3) != K_LITERAL) continue;
        const uint32_t d = lit[i >> b1], b2 = (d >> 7) & 15;
        if (((d >> 4) & 3) == K_LITERAL && b1 + b2 <= LIT_BITS)
            lit[i] = (b1 + b2) | 64u | b1 << 7 | (e & 0xff0000u) | (d & 0xff0000u) << 8;
    }
}

// Whether member m's spans lie in their buffers.
__device__ __forceinline__ bool member_spans(const bgzf_inflate::Job& j, uint32_t m) {
    const uint64_t so = j.src_off[m], sl = j.src_len[m], dof = j.dst_off[m], isz = j.isize[m];
    return !(so > j.in_bytes || sl > j.in_bytes - so || dof > j.out_bytes || isz > j.out_bytes - dof);
}

// What a member takes, in nanoseconds by the kind of its first block (fitted to
// members of 512 .. 65280 bytes: FASTQ at level 6, zeros, base-64 text, fixed
// codes, whose segments fall into step late, and stored noise).
struct Cost {
    uint64_t cta;   // a CTA, which has the SM to itself
    uint64_t warp;  // a warp, alone
    uint64_t sm;    // one more on an SM whose 64 warps are at work
};

__device__ __forceinline__ Cost member_cost(const bgzf_inflate::Job& j, uint32_t m) {
    const uint64_t isz = j.isize[m], src = j.src_len[m];
    const uint32_t type = j.in[j.src_off[m]] >> 1 & 3;
    if (type == 0) return Cost{17000 + isz * 3 / 4, 10000 + isz * 8, 4000 + isz * 9 / 16};
    return Cost{type == 1 ? 45000 + src * 45 : 50000 + isz * 9 / 10, 130000 + src * 260 + isz * 6, 9000 + src * 17 + isz / 2};
}

// Whether a CTA can take member m; its spans are checked.
__device__ __forceinline__ bool cta_holds(const bgzf_inflate::Job& j, uint32_t m) {
    return j.isize[m] >= 4 && j.isize[m] <= MAX_BYTES && j.src_len[m] >= 1 && j.src_len[m] <= (1u << 26);
}

// A CTA decodes a large member up to 40 times as fast as a warp, but 148 members
// are in CTAs at a time and 9472 in warps, and a small member's time is the CTA's
// own.  So a CTA leaves those of its members that an SM's warps are faster at
// (Cost), when they would take the CTAs longer than the slowest of them takes a
// warp, and the second kernel's start.  16000 members of 512 bytes of FASTQ: 1.5 ms in
// warps, 5.3 in CTAs; 2368 of 4096 bytes 0.82 and 0.95, of 16384 bytes 2.5 and
// 1.15.  8000 members of 65280 bytes of zeros 2.1 and 6.8 ms, of stored noise 2.2
// and 3.5, 2000 of FASTQ in fixed codes 9.8 and 18.3.  One member of 600 bytes
// among 1960 of 65280 stays with its CTA: in a warp it would add 0.2 ms to 1.4.
constexpr uint64_t LEFT_START = 15000;

// Codes that fall into step late, beyond four turns of the CTAs: there a member
// whose literal codes are all but an eighth of one length (base-64, hexadecimal
// text; FASTQ's are up to 0.8) is left, and so is one whose sync rounds go past
// USUAL (FASTQ takes 3 to 12) and what is left of the CTA's SPARE.  A CTA that
// left one leaves its later ones too: beside it in other warps they cost nothing.
// 2000 members of base-64 text take 17 ms in warps, up to 51 in CTAs (850 rounds).
struct Rounds {
    static constexpr int USUAL = 32, SPARE = 64;
    bool limited, out;  // out: the CTA leaves the rest
    int over;           // spent beyond USUAL
    __device__ __forceinline__ int limit() const { return limited ? USUAL + max(0, SPARE - over) : THREADS + 1; }
};

// Member m by THREADS threads, from its first block's header H on; returns its
// status (valid in thread 0), S_LEFT: nothing written.
__device__ uint32_t cta_member(const bgzf_inflate::Job& j, uint32_t m, Smem& S, Head& H, uint32_t t, Rounds& rounds) {
    const uint8_t* in = j.in + j.src_off[m];
    uint8_t* out = j.out + j.dst_off[m];
    const uint32_t n = j.src_len[m], isz = j.isize[m], lane = t & 31, warp = t >> 5;
    if (rounds.limited && H.flat) {
        rounds.out = true;
        return S_LEFT;
    }
    for (uint32_t i = t; i < (MAX_BYTES + 31) / 32; i += THREADS) S.starts[i] = 0;
    work_sync();
    uint32_t made = 0;  // bytes whose cells are written
    for (int blocks = 0;; ++blocks) {
        if (!H.ok || blocks == MAX_BLOCKS) return S_LEFT;
        const bool last = H.last;
        uint32_t pos = H.pos;  // bit of the stream
        if (H.type == 0) {
            const uint32_t p = (pos + 7) >> 3;  // LEN, NLEN, the bytes
            if (p + 4 > n) return S_LEFT;
            const uint32_t len = in[p] | in[p + 1] << 8, nlen = in[p + 2] | in[p + 3] << 8;
            if (len != (~nlen & 0xffffu) || len > n - p - 4 || len > isz - made) return S_LEFT;
            for (uint32_t i = t; i < len; i += THREADS) {
                S.cell[made + i] = static_cast<uint16_t>(0xff00u | in[p + 4 + i]);
                atomicOr(S.starts + ((made + i) >> 5), 1u << ((made + i) & 31));
            }
            made += len;
            pos = 8 * (p + 4 + len);
        } else {
            // the block's codes, THREADS segments at a time
            for (bool ended = false; !ended;) {
                if (pos >= 8 * n) return S_LEFT;
                const uint32_t base = (pos >> 3) & ~3u, at = pos - 8 * base;  // `at`: bit of the staged input
                stage_input(S.in, IN_WORDS, in, n, base, t, THREADS);
                work_sync();
                const uint32_t n_bits = 8 * (n - base);
                const uint32_t limit = at + (t + 1) * SEG_BITS;
                uint32_t start = at + t * SEG_BITS, end = 0, bytes = 0;
                uint32_t flag = decode_bits<false>(S, H, true, start, limit, n_bits, end, bytes);
                uint32_t f = THREADS;  // the first thread that met an end or no code
                bool settled = false;  // after at most one round per thread, if it may spend them
                int round = 0;
                for (const int most = rounds.limit(); round < most && !settled; ++round) {
                    if (t == 0) S.first_flag = THREADS - 1;
                    S.end[t] = end;
                    work_sync();
                    if (flag != F_NONE) atomicMin(&S.first_flag, t);
                    work_sync();
                    f = S.first_flag;
                    const uint32_t from = t && t <= f ? S.end[t - 1] : at;
                    const bool again = t && t <= f && from != start;
                    if (again) start = from;
                    uint32_t e2, b2 = 0;
                    const uint32_t f2 = decode_bits<false>(S, H, again, start, limit, n_bits, e2, b2);
                    if (again) {
                        end = e2;
                        bytes = b2;
                        flag = f2;
                    }
                    settled = !work_or(again);
                }
                rounds.over += max(0, round - Rounds::USUAL);
                if (!settled) rounds.out = rounds.limited;
                if (t > f) bytes = 0;
                const bool bad = work_or(t == f && flag == F_BAD);
                ended = work_or(t == f && flag == F_END);
                if (bad || !settled) return S_LEFT;
                uint32_t total;
                uint32_t o = made + block_scan(S, bytes, t, total);
                const uint32_t reached = S.end[f];
                if (reached > n_bits || total > isz - made) return S_LEFT;
                const uint32_t f2 = decode_bits<true>(S, H, t <= f, start, limit, n_bits, end, o);
                if (work_or(t <= f && f2 == F_BAD)) return S_LEFT;
                made += total;
                pos = 8 * base + reached;
            }
        }
        if (last) break;
        if (pos >= 8 * n) return S_LEFT;
        work_sync();  // the block's tables are done with
        if (warp == 0) read_head(H, in, n, pos, static_cast<int>(lane));
        work_sync();
        fill_tables(H, t, THREADS, [] { work_sync(); });
        work_sync();
    }
    if (made != isz) return S_LEFT;
    work_sync();
    // resolve, a strip at a time, four bytes per thread
    volatile uint16_t* cell = S.cell;
    volatile uint64_t* cell4 = reinterpret_cast<volatile uint64_t*>(S.cell);
    const bool aligned = (reinterpret_cast<uintptr_t>(out) & 3) == 0;
    if (t == 0) S.carry_at = S.carry_cell = 0;
    for (uint32_t strip = 0; strip < isz; strip += STRIP) {
        const uint32_t q = strip + 4 * t;
        uint32_t c[4] = {0xff00u, 0xff00u, 0xff00u, 0xff00u}, from = 0, cf = 0;
        work_sync();  // carry, and the last strip's bytes
        if (q < isz) {
            // the code that makes the first byte: the last start at or before
            // it, in the strip or (carry) before it; the next bytes follow on
            uint32_t w = q >> 5;
            const uint32_t word = S.starts[w], four = word >> (q & 31);
            if (!(four & 1)) {
                uint32_t m = word & ((1u << (q & 31)) - 1);
                while (!m && 32 * w > strip) m = S.starts[--w];
                from = m ? 32 * w + 31 - __clz(m) : S.carry_at;
                cf = m ? cell[from] : S.carry_cell;
            }
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                if (four >> k & 1) {
                    from = q + k;
                    cf = cell[from];
                }
                c[k] = cf < MAX_BYTES ? cf + (q + k - from) : cf;
            }
        }
        work_sync();  // all starts' cells are read
        auto put = [&] {
            cell4[q >> 2] = c[0] | c[1] << 16 | static_cast<uint64_t>(c[2] | c[3] << 16) << 32;
        };
        if (q < isz) put();  // MAX_BYTES is a multiple of 4
        if (t == THREADS - 1) {  // its last byte is the strip's last
            S.carry_at = from;
            S.carry_cell = cf;
        }
        work_sync();
        // four chains at once; the cells take each position they come to,
        // which shortens the chains that go through them
        while (c[0] < MAX_BYTES || c[1] < MAX_BYTES || c[2] < MAX_BYTES || c[3] < MAX_BYTES) {
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                if (c[k] < MAX_BYTES) c[k] = cell[c[k]];
            put();
        }
        const uint32_t v = (c[0] & 0xff) | (c[1] & 0xff) << 8 | (c[2] & 0xff) << 16 | c[3] << 24;
        if (aligned && q + 4 <= isz) {
            *reinterpret_cast<uint32_t*>(out + q) = v;
        } else {
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                if (q + k < isz) out[q + k] = static_cast<uint8_t>(v >> (8 * k));
        }
    }
    work_sync();
    // CRC-32; the all-ones start of the register is that of the first four
    // bytes inverted
    uint32_t c = 0;
    {
        const uint32_t q0 = isz - (THREADS - t) * CRC_BYTES;  // wraps below 0: zero bytes
        auto byte = [&](uint32_t q) { return q < isz ? (cell[q] & 0xffu) ^ (q < 4 ? 0xffu : 0u) : 0u; };
        for (uint32_t i = 0; i + 4 <= CRC_BYTES; i += 4) {
            const uint32_t q = q0 + i;
            c ^= byte(q) | byte(q + 1) << 8 | byte(q + 2) << 16 | byte(q + 3) << 24;
            c = S.crc[3][c & 255] ^ S.crc[2][(c >> 8) & 255] ^ S.crc[1][(c >> 16) & 255] ^ S.crc[0][c >> 24];
        }
        for (uint32_t i = CRC_BYTES & ~3u; i < CRC_BYTES; ++i) c = (c >> 8) ^ S.crc[0][(c ^ byte(q0 + i)) & 255];
    }
    for (int k = 0; k < 5; ++k) c = gf2_mul(c, S.xpow[k]) ^ __shfl_down_sync(0xffffffffu, c, 1 << k);
    if (lane == 0) S.part[warp] = c;
    work_sync();
    if (warp == 0) {
        // the member's bytes lie in the last WARPS parts
        c = lane ? S.part[lane - 1] : 0;
        for (int k = 0; k < 5; ++k) c = gf2_mul(c, S.xpow[5 + k]) ^ __shfl_down_sync(0xffffffffu, c, 1 << k);
    }
    return ~c == j.crc[m] ? 0u : bgzf_inflate::S_CRC;
}

__global__ void __launch_bounds__(CTA_THREADS, 1) bgzf_inflate_kernel(bgzf_inflate::Job j) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    Smem& S = *reinterpret_cast<Smem*>(smem_raw);
    const uint32_t t = threadIdx.x;
    bool tables = false;
    auto make_tables = [&] {  // for the first member that the CTA takes
        bgzf_inflate::crc_table(S.crc[0], static_cast<int>(t), CTA_THREADS);
        if (t == 0) {
            uint32_t x = gf2_xpow(8ull * CRC_BYTES);
            for (int k = 0; k < 10; ++k) {
                S.xpow[k] = x;
                x = gf2_mul(x, x);
            }
        }
        __syncthreads();
        if (t < 256) {
            uint32_t c = S.crc[0][t];
            for (int k = 1; k < 4; ++k) {
                c = (c >> 8) ^ S.crc[0][c & 255];
                S.crc[k][t] = c;
            }
        }
        tables = true;
    };
    if (t == 0) S.stopped = 0;
    Rounds rounds{j.n > 4 * static_cast<uint64_t>(gridDim.x), false, 0};
    // the CTA's members are blockIdx.x + i * gridDim.x; which of the next
    // CTA_THREADS it takes is looked up for all of them at once
    for (uint64_t base = 0; blockIdx.x + base * gridDim.x < j.n; base += CTA_THREADS) {
        auto member = [&](int i) { return static_cast<uint32_t>(blockIdx.x + (base + i) * gridDim.x); };
        const bool any = blockIdx.x + (base + t) * gridDim.x < j.n;
        const uint64_t n = j.n, turns = (n + gridDim.x - 1) / gridDim.x, here = (n - blockIdx.x + gridDim.x - 1) / gridDim.x;
        const uint32_t m0 = member(static_cast<int>(t));
        const bool spans = any && member_spans(j, m0), holds = spans && cta_holds(j, m0);
        bool slower = false;
        if (t == 0) S.cta_ns = S.warp_ns = 0;
        __syncthreads();
        if (holds) {
            const Cost c = member_cost(j, m0);
            slower = c.cta > c.sm;
            if (slower) {
                atomicAdd(&S.cta_ns, static_cast<unsigned long long>(c.cta));
                atomicMax(&S.warp_ns, static_cast<unsigned long long>(c.warp));
            }
        }
        __syncthreads();
        // CTAs of one member more or less than others are to decide alike
        const bool leave = S.cta_ns * turns > (S.warp_ns + LEFT_START) * here;
        const bool take = holds && !(slower && leave);
        if (any && !take) j.status[m0] = spans ? S_LEFT : bgzf_inflate::S_SPAN;
        const uint32_t word = __ballot_sync(0xffffffffu, take);
        if ((t & 31) == 0) S.mine[t >> 5] = word;
        __syncthreads();
        auto after = [&](int i) {  // the first one taken after i, -1: none
            for (int w = ++i >> 5; w < CTA_THREADS / 32; ++w, i = 0) {
                const uint32_t x = S.mine[w] >> (i & 31) << (i & 31);
                if (x) return 32 * w + __ffs(static_cast<int>(x)) - 1;
            }
            return -1;
        };
        // the last warp reads the next member's first header while the others
        // work on this one
        auto header_of = [&](int i, Head& H) {
            if (i < 0 || S.stopped) return;
            const uint32_t m = member(i);
            read_head(H, j.in + j.src_off[m], j.src_len[m], 0, static_cast<int>(t - THREADS));
            fill_tables(H, t - THREADS, 32, [] { __syncwarp(); });
        };
        int i = after(-1);
        if (i >= 0 && !tables) make_tables();
        if (t >= THREADS) header_of(i, S.head[0]);
        __syncthreads();
        for (uint32_t which = 0; i >= 0; which ^= 1) {
            const int next = after(i);
            if (t >= THREADS) {
                header_of(next, S.head[which ^ 1]);
            } else {
                const uint32_t m = member(i);
                const uint32_t status = S.stopped ? S_LEFT : cta_member(j, m, S, S.head[which], t, rounds);
                if (t == 0) j.status[m] = status;
            }
            __syncthreads();
            if (t == 0 && rounds.out) S.stopped = 1;
            __syncthreads();
            i = next;
        }
    }
}

void check_launch(cudaError_t e, const char* what) {
    if (e != cudaSuccess) fail(MA_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

}  // namespace

int bgzf_inflate_enqueue(const bgzf_inflate::Job& j, int sm_count, cudaStream_t st) {
    if (!j.n) return 0;
    const uint32_t sms = static_cast<uint32_t>(sm_count > 0 ? sm_count : 148);
    check_launch(cudaFuncSetAttribute(bgzf_inflate_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(sizeof(Smem))),
                 "inflate smem");
    bgzf_inflate_kernel<<<j.n < sms ? j.n : sms, CTA_THREADS, sizeof(Smem), st>>>(j);
    check_launch(cudaGetLastError(), "bgzf_inflate_kernel");
    const uint32_t want = (j.n + LEFT_WARPS - 1) / LEFT_WARPS;
    left_kernel<<<want < sms * 16 ? want : sms * 16, LEFT_WARPS * 32, 0, st>>>(j);
    check_launch(cudaGetLastError(), "left_kernel");
    return 2;
}

}  // namespace ma
