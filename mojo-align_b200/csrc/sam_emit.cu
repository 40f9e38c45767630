// sam_emit.cu - SAM text lines of one mapped batch on the device.
//
// Replaces the per-record host loop of map_fastq_fm_gpu's SAM path
// (fq2bam-meth/src/linear_gpu_fm.mojo:2787-2836), which builds a LinearHit
// per read with _hit_from_fm (L987-1025), pairs mates with pair_hits
// (fq2bam-meth/src/linear_extend.mojo:263-294), formats each line with
// hit_to_sam_line (L297-320) + the RG tag (_sam_with_rg_fm, L80-81) and
// writes it.  Here the lines of a whole batch are built in HBM in three
// passes:
//   1. sam_layout_kernel (one thread per line): its hit and the pair
//      fields, the line's byte length and a compact record of its fields,
//      names' bytes >= 0x80 counted (each becomes U+FFFD), SEQ / QUAL
//      checked for strict UTF-8, mapped records and error bits;
//   2. a device scan of the lengths (line end offsets);
//   3. sam_write_kernel (a warp per run of lines): one lane formats a line's
//      fields FLAG .. TLEN, then the warp assembles the lines in a
//      shared-memory stage at the destination's 16-byte phase (name, the
//      formatted fields, SEQ reverse-complemented on flag 16, QUAL and the RG
//      tag from aligned word loads) and stores it in 16-byte blocks; lines
//      longer than the stage are built in place.
#include <cub/device/device_scan.cuh>

#include <string>

#include "ma_internal.h"
#include "sam_emit.h"
#include "span.cuh"

namespace ma {
namespace {

constexpr int THREADS = 256;
constexpr unsigned FULL = 0xffffffffu;
constexpr int WRITE_WARPS = 4;
constexpr uint32_t STAGE = 2048;  // bytes of output a warp gathers before it stores them
constexpr uint32_t SLOT = 100;    // formatted fields of a line; an odd number of words, so lanes' slots spread over the banks

enum : unsigned { E_OVER = 1, E_UTF8 = 2, E_RID = 4, E_SPAN = 8 };
enum : uint8_t { K_NAME = 0, K_STAR = 1, K_EQ = 2 };

void check_launch(cudaError_t e, const char* what) {
    if (e != cudaSuccess) fail(MA_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

size_t align256(size_t n) { return (n + 255) & ~static_cast<size_t>(255); }

// One record's SAM fields before and after pairing (LinearHit,
// linear_extend.mojo:11-48).
struct Hit {
    int64_t flag, pos1, mapq, pnext, tlen, sl, m, sr;
    uint64_t contig_off, rnext_off;
    uint32_t contig_len, rnext_len;
    uint32_t canon;
    uint8_t contig_kind, rnext_kind;
    bool mapped;  // placed by _hit_from_fm (CIGAR and strand apply)
    bool star;    // RNAME "*": unplaced, or a canonical name "*"
};

// _hit_from_fm: unplaced when rid < 0 or no base is left between the clips.
__device__ Hit hit_of(const SamDev& d, uint64_t r, unsigned& err) {
    Hit h{};
    h.rnext_kind = K_STAR;
    h.rnext_len = 1;
    const int32_t rid = d.rid[r];
    const int64_t m = static_cast<int64_t>(d.seq_len[r]) - d.sl[r] - d.sr[r];
    bool ok = rid >= 0 && m >= 1;
    if (rid >= 0 && static_cast<uint32_t>(rid) >= d.n_contigs) {
        err |= E_RID;
        ok = false;
    }
    uint64_t co = 0;
    uint32_t cl = 0;
    if (ok) {
        co = d.cname_off[rid];
        cl = d.cname_len[rid];
        if (co > d.names_bytes || cl > d.names_bytes - co) {
            err |= E_SPAN;
            ok = false;
        }
    }
    if (!ok) {
        h.star = true;
        h.flag = 4;
        h.contig_kind = K_STAR;
        h.contig_len = 1;
        return h;
    }
    h.mapped = true;
    h.flag = d.flag[r];
    h.pos1 = static_cast<int64_t>(d.pos[r]) + 1;
    h.mapq = d.mapq[r];
    h.sl = d.sl[r];
    h.sr = d.sr[r];
    h.m = m;
    h.contig_kind = K_NAME;
    h.contig_off = co;
    h.contig_len = cl;
    h.canon = d.canon[rid];
    h.star = cl == 1 && d.names[co] == '*';
    return h;
}

// pair_hits (linear_extend.mojo:263-294) from the side of one mate: R1 sits
// in lane 2i, R2 in lane 2i + 1; seq_len = len(SEQ) of this lane's read.
__device__ __forceinline__ void pair_up(Hit& h, uint32_t seq_len, bool second) {
    const bool mstar = __shfl_xor_sync(FULL, static_cast<int>(h.star), 1) != 0;
    const uint32_t mcanon = __shfl_xor_sync(FULL, h.canon, 1), mlen = __shfl_xor_sync(FULL, h.contig_len, 1);
    const uint32_t mseq = __shfl_xor_sync(FULL, seq_len, 1);
    const int64_t mpos1 = __shfl_xor_sync(FULL, h.pos1, 1);
    const uint64_t moff = __shfl_xor_sync(FULL, h.contig_off, 1);
    h.flag |= second ? 1 | 128 : 1 | 64;
    if (!h.star && !mstar && h.canon == mcanon) {
        h.flag |= 2;
        h.rnext_kind = K_EQ;
        h.pnext = mpos1;
        int64_t t = mpos1 - h.pos1;
        if (t < 0) t = -t;
        t += second ? seq_len : mseq;  // len(SEQ of R2)
        h.tlen = second ? -t : t;
        return;
    }
    if (mstar) {
        h.flag |= 8;
    } else {
        h.rnext_kind = K_NAME;
        h.rnext_off = moff;
        h.rnext_len = mlen;
        h.pnext = mpos1;
    }
}

// Decimal digits of u: comparisons against powers of ten below 2^32, a
// division loop above.
__device__ __forceinline__ uint32_t ndig(uint64_t u) {
    if (u >> 32) {
        uint32_t k = 10;
        u /= 10000000000ull;
        while (u) {
            u /= 10;
            ++k;
        }
        return k;
    }
    const uint32_t v = static_cast<uint32_t>(u);
    return 1 + (v >= 10u) + (v >= 100u) + (v >= 1000u) + (v >= 10000u) + (v >= 100000u) + (v >= 1000000u) +
           (v >= 10000000u) + (v >= 100000000u) + (v >= 1000000000u);
}

__device__ __forceinline__ uint64_t mag(int64_t v) {
    return v < 0 ? uint64_t(0) - static_cast<uint64_t>(v) : static_cast<uint64_t>(v);
}

__device__ __forceinline__ uint32_t sdig(int64_t v) { return (v < 0) + ndig(mag(v)); }

// Strict UTF-8 (RFC 3629): no overlong forms, surrogates or code points
// above U+10FFFF.
__device__ bool utf8_ok(const uint8_t* p, uint64_t n) {
    uint64_t i = 0;
    while (i < n) {
        const uint8_t c = p[i];
        if (c < 0x80) {
            ++i;
            continue;
        }
        int k;
        uint8_t lo = 0x80, hi = 0xbf;
        if (c >= 0xc2 && c <= 0xdf) {
            k = 1;
        } else if (c >= 0xe0 && c <= 0xef) {
            k = 2;
            if (c == 0xe0) lo = 0xa0;
            if (c == 0xed) hi = 0x9f;
        } else if (c >= 0xf0 && c <= 0xf4) {
            k = 3;
            if (c == 0xf0) lo = 0x90;
            if (c == 0xf4) hi = 0x8f;
        } else {
            return false;
        }
        if (n - i - 1 < static_cast<uint64_t>(k)) return false;
        if (p[i + 1] < lo || p[i + 1] > hi) return false;
        for (int j = 2; j <= k; ++j)
            if (p[i + j] < 0x80 || p[i + j] > 0xbf) return false;
        i += k + 1;
    }
    return true;
}

__device__ __forceinline__ bool span_ok(uint64_t off, uint32_t len, uint64_t n) { return off <= n && len <= n - off; }

__device__ __forceinline__ bool spans_ok(const SamDev& d, uint64_t r) {
    return span_ok(d.name_off[r], d.name_len[r], d.arena_bytes) && span_ok(d.seq_off[r], d.seq_len[r], d.arena_bytes) &&
           span_ok(d.qual_off[r], d.qual_len[r], d.arena_bytes);
}

// What the write pass needs of a line, resolved once by the layout pass.
struct LineRec {
    int64_t flag, pos1, pnext, tlen;
    uint64_t contig_off, rnext_off;
    uint32_t mapq, sl, sr, m;
    uint32_t contig_len, rnext_len;
    uint8_t contig_kind, rnext_kind, mapped, widen;
    uint32_t pad;
};
static_assert(sizeof(LineRec) == 80, "line record layout");

__device__ __forceinline__ uint32_t clip_dig(uint32_t n) { return n ? ndig(n) + 1 : 0; }

// Length of a line's formatted fields, from the tab after the name to the
// one before SEQ.
__device__ __forceinline__ uint64_t fields_len(const LineRec& h) {
    const uint32_t cig = h.mapped ? clip_dig(h.sl) + ndig(h.m) + 1 + clip_dig(h.sr) : 1;
    return 9ull + sdig(h.flag) + h.contig_len + sdig(h.pos1) + ndig(h.mapq) + cig + h.rnext_len + sdig(h.pnext) +
           sdig(h.tlen);
}

// Bytes >= 0x80 in p[0, n), from the aligned 16-byte blocks that cover the
// span (their bytes outside the span lie in the same block as one inside).
__device__ __forceinline__ uint32_t count_high(const uint8_t* p, uint32_t n) {
    if (!n) return 0;
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), e = a + n;
    uint32_t c = 0;
    for (uintptr_t q = a & ~uintptr_t(15); q < e; q += 16) {
        const uint4 v = *reinterpret_cast<const uint4*>(q);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint32_t m = w[k] & 0x80808080u;
            if (m) {
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const uintptr_t x = q + 4 * k + b;
                    if (x < a || x >= e) m &= ~(0x80u << (8 * b));
                }
                c += __popc(m);
            }
        }
    }
    return c;
}

// This lane's part of the 16-byte blocks that cover [lo, hi) (at most 1009
// bytes), ORed: the bit 0x80 of some byte tells a byte >= 0x80.
__device__ __forceinline__ uint32_t covered_or(const uint8_t* lo, const uint8_t* hi, uint32_t lane) {
    const uintptr_t e = lo < hi ? reinterpret_cast<uintptr_t>(hi) : 0;
    const uintptr_t q = (reinterpret_cast<uintptr_t>(lo) & ~uintptr_t(15)) + 16 * lane;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    const uint4 v = q < e ? __ldg(reinterpret_cast<const uint4*>(q)) : zero;
    const uint4 w = q + 512 < e ? __ldg(reinterpret_cast<const uint4*>(q + 512)) : zero;
    return (v.x | v.y | v.z | v.w | w.x | w.y | w.z | w.w) & 0x80808080u;
}

// One thread per line: its hit, the pairing (by shuffle), its length and
// record; the SEQ / QUAL UTF-8 check; mapped records and error bits gathered
// per block.  The warp looks through each record's bytes together (the stretch
// from its first span to the end of its last one, up to HIGH_SPAN bytes):
// without a byte >= 0x80 there no name widens and SEQ and QUAL are valid,
// otherwise the record's own thread checks its spans.  1 M records of 356
// bytes: 137 us; with a thread per pair that walked the pair's bytes 222.
constexpr uint64_t HIGH_SPAN = 1008;
constexpr int HIGH_UNROLL = 4;  // records whose bytes are on their way at once

__global__ void __launch_bounds__(THREADS, 4) sam_layout_kernel(SamDev d, uint64_t n_lines, uint32_t* line_len,
                                                                LineRec* recs) {
    __shared__ unsigned long long blk_mapped;
    __shared__ unsigned blk_err;
    if (threadIdx.x == 0) {
        blk_mapped = 0;
        blk_err = 0;
    }
    __syncthreads();
    unsigned err = 0;
    uint32_t mapped = 0;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * THREADS;
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t base = static_cast<uint64_t>(blockIdx.x) * THREADS + (threadIdx.x & ~31u); base < n_lines;
         base += stride) {
        const uint64_t L = base + lane;
        const uint64_t r = d.paired ? (L >> 1) + (L & 1) * d.n1 : L;
        const bool mine = L < n_lines;
        const bool spans = mine && spans_ok(d, r);
        uint64_t lo = 0, hi = 0;
        if (spans) {
            const uint64_t a = d.name_off[r], b = d.seq_off[r], c = d.qual_off[r];
            lo = min(a, min(b, c));
            hi = max(a + d.name_len[r], max(b + d.seq_len[r], c + d.qual_len[r]));
            if (hi - lo > HIGH_SPAN) hi = lo;
        }
        uint32_t seen = 0;  // bit k: lane k's record holds a byte >= 0x80
        for (int k = 0; k < 32; k += HIGH_UNROLL) {
            uint32_t v[HIGH_UNROLL];
#pragma unroll
            for (int j = 0; j < HIGH_UNROLL; ++j)
                v[j] = covered_or(d.arena + __shfl_sync(FULL, lo, k + j), d.arena + __shfl_sync(FULL, hi, k + j), lane);
#pragma unroll
            for (int j = 0; j < HIGH_UNROLL; ++j) seen |= (__any_sync(FULL, v[j] != 0) ? 1u : 0u) << (k + j);
        }
        const bool clean = hi > lo && !((seen >> lane) & 1u);
        Hit h{};
        h.star = true;
        const uint32_t n_sq = mine ? d.seq_len[r] : 0;
        if (mine) h = hit_of(d, r, err);
        if (d.paired) pair_up(h, n_sq, L & 1);
        if (!mine) continue;
        if (!spans) {
            err |= E_SPAN;
            line_len[L] = 0;
            continue;
        }
        const uint32_t n_nm = d.name_len[r], n_ql = d.qual_len[r];
        uint32_t high = 0;
        if (!clean) {
            const uint8_t* sq = d.arena + d.seq_off[r];
            const uint8_t* ql = d.arena + d.qual_off[r];
            high = count_high(d.arena + d.name_off[r], n_nm);
            if ((count_high(sq, n_sq) || count_high(ql, n_ql)) && !(utf8_ok(sq, n_sq) && utf8_ok(ql, n_ql)))
                err |= E_UTF8;
        }
        LineRec rc;
        rc.flag = h.flag;
        rc.pos1 = h.pos1;
        rc.pnext = h.pnext;
        rc.tlen = h.tlen;
        rc.contig_off = h.contig_off;
        rc.rnext_off = h.rnext_off;
        rc.mapq = static_cast<uint32_t>(h.mapq);
        rc.sl = static_cast<uint32_t>(h.sl);
        rc.sr = static_cast<uint32_t>(h.sr);
        rc.m = static_cast<uint32_t>(h.mapped ? h.m : 0);
        rc.contig_len = h.contig_len;
        rc.rnext_len = h.rnext_len;
        rc.contig_kind = h.contig_kind;
        rc.rnext_kind = h.rnext_kind;
        rc.mapped = h.mapped;
        rc.widen = high != 0;
        rc.pad = 0;
        const uint64_t len = n_nm + 2ull * high + fields_len(rc) + n_sq + 1 + n_ql + 6 + d.rg_n + 1;
        if (len > 0xffffffffull) err |= E_OVER;
        line_len[L] = static_cast<uint32_t>(len);
        mapped += !h.star;
        recs[L] = rc;
    }
    for (int o = 16; o > 0; o >>= 1) {
        err |= __shfl_xor_sync(FULL, err, o);
        mapped += __shfl_xor_sync(FULL, mapped, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (mapped) atomicAdd(&blk_mapped, static_cast<unsigned long long>(mapped));
        if (err) atomicOr(&blk_err, err);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (blk_mapped) atomicAdd(&d.status[1], blk_mapped);
        if (blk_err) atomicOr(&d.status[2], static_cast<unsigned long long>(blk_err));
    }
}

// The decimal text of v at o (k = sdig(v) bytes); 32-bit divisions while
// the value fits.
__device__ __forceinline__ void put_int(uint8_t* o, int64_t v, uint32_t k) {
    uint64_t u = mag(v);
    uint32_t j = k;
    while (u >> 32) {
        o[--j] = static_cast<uint8_t>('0' + u % 10);
        u /= 10;
    }
    uint32_t x = static_cast<uint32_t>(u);
    do {
        o[--j] = static_cast<uint8_t>('0' + x % 10);
        x /= 10;
    } while (x);
    if (v < 0) o[0] = '-';
}

// Where in a line's formatted fields its contig names begin, or belong when
// they are left out of them, and the fields' end.
struct Cuts {
    uint32_t rname, rnext, end;
};

// \t FLAG \t RNAME \t POS \t MAPQ \t CIGAR \t RNEXT \t PNEXT \t TLEN \t at o (one
// lane); fields_len(h) bytes, or with `names` false those without the contig
// names (at most 99: nine tabs, two "*" or "=", and the numbers).
__device__ __forceinline__ Cuts put_fields(uint8_t* o, const SamDev& d, const LineRec& h, bool names) {
    uint8_t* const first = o;
    Cuts cuts;
    auto contig = [&](uint8_t kind, uint64_t off, uint32_t len) {
        if (kind != K_NAME) {
            *o++ = kind == K_EQ ? '=' : '*';
        } else if (names) {
            for (uint32_t j = 0; j < len; ++j) o[j] = __ldg(d.names + off + j);
            o += len;
        }
    };
    auto num = [&](int64_t v, uint8_t after) {
        const uint32_t k = sdig(v);
        put_int(o, v, k);
        o[k] = after;
        o += k + 1;
    };
    *o++ = '\t';
    num(h.flag, '\t');
    cuts.rname = static_cast<uint32_t>(o - first);
    contig(h.contig_kind, h.contig_off, h.contig_len);
    *o++ = '\t';
    num(h.pos1, '\t');
    num(h.mapq, '\t');
    if (h.mapped) {
        if (h.sl) num(h.sl, 'S');
        num(h.m, 'M');
        if (h.sr) num(h.sr, 'S');
    } else {
        *o++ = '*';
    }
    *o++ = '\t';
    cuts.rnext = static_cast<uint32_t>(o - first);
    contig(h.rnext_kind, h.rnext_off, h.rnext_len);
    *o++ = '\t';
    num(h.pnext, '\t');
    num(h.tlen, '\t');
    cuts.end = static_cast<uint32_t>(o - first);
    return cuts;
}

// The reverse strand's bases of four read backwards: A<->T, C<->G, any other
// byte N.  Bits 1-2 of a letter tell A, C, T and G apart; the letter they
// stand for is compared with the byte to find the others.
__device__ __forceinline__ uint32_t complement4(uint32_t x) {
    const uint32_t i = (x >> 1) & 0x03030303u;
    const uint32_t sel = __byte_perm(i | (i >> 4), 0, 0x4420);  // one nibble per base
    const uint32_t d = __byte_perm(0x47544341u, 0, sel) ^ x;
    const uint32_t other = (((((d & 0x7f7f7f7fu) + 0x7f7f7f7fu) | d) >> 7) & 0x01010101u) * 255u;
    return (__byte_perm(0x43414754u, 0, sel) & ~other) | (0x4e4e4e4eu & other);
}

__device__ __forceinline__ uint8_t tail_byte(const SamDev& d, uint32_t j) {
    if (j < 6) return "\tRG:Z:"[j];
    return j < 6 + d.rg_n ? d.rg[j - 6] : '\n';
}

// What the warp needs of a line to write its bytes, filled in by one lane.
struct __align__(16) LinePlan {
    const uint8_t *name, *seq, *qual;
    uint32_t n_nm, n_sq, n_ql;
    uint32_t fields;  // bytes of the formatted fields in the line's slot, 0: put_head
    uint32_t rc;
    // put_head's: the name holds bytes >= 0x80, bytes in the slot, and where
    // the contig names that are not in it belong (NONE: they are)
    uint8_t widen, slot, at_rname, at_rnext;
};
constexpr uint32_t NONE = 255;
static_assert(sizeof(LinePlan) == 48, "line plan layout");

// A lane's share of a line's source bytes: two name bytes, eight bases and
// eight qualities; for lines of up to 64 name bytes and 256 bases that is all
// of them.
struct LineRaw {
    uint32_t n0, n1;
    span::Span8 seq, qual;
};

__device__ __forceinline__ void load_raw(LineRaw& x, const LinePlan& q, uint32_t lane) {
    x.n0 = lane < q.n_nm ? __ldg(q.name + lane) : 0;
    x.n1 = lane + 32 < q.n_nm ? __ldg(q.name + lane + 32) : 0;
    x.seq = span::span8_load(q.seq, q.n_sq, lane, q.rc);
    x.qual = span::span8_load(q.qual, q.n_ql, lane, false);
}

// The bytes of a line after its fields, by the warp: SEQ, tab, QUAL and the
// RG tag; tail: this lane's byte of the tag.
__device__ __forceinline__ void put_rest(uint8_t* o, const SamDev& d, const LinePlan& q, const LineRaw& x,
                                         uint32_t tail, uint32_t lane) {
    const uint32_t n_sq = q.n_sq, n_ql = q.n_ql;
    const bool rc = q.rc;
    for (uint32_t i = lane; 8 * i < n_sq; i += 32) {
        const uint32_t left = n_sq - 8 * i;
        uint2 v = span::span8_bytes(i < 32 ? x.seq : span::span8_load(q.seq, n_sq, i, rc), q.seq, n_sq, rc);
        if (rc) v = make_uint2(complement4(v.x), complement4(v.y));
        span::put_bytes(o + 8 * i, v.x, min(4u, left));
        if (left > 4) span::put_bytes(o + 8 * i + 4, v.y, min(4u, left - 4));
    }
    if (lane == 0) o[n_sq] = '\t';
    uint8_t* oq = o + n_sq + 1;
    for (uint32_t i = lane; 8 * i < n_ql; i += 32) {
        const uint32_t left = n_ql - 8 * i;
        const uint2 v = span::span8_bytes(i < 32 ? x.qual : span::span8_load(q.qual, n_ql, i, false), q.qual, n_ql, false);
        span::put_bytes(oq + 8 * i, v.x, min(4u, left));
        if (left > 4) span::put_bytes(oq + 8 * i + 4, v.y, min(4u, left - 4));
    }
    uint8_t* ot = oq + n_ql;
    const uint32_t n_tail = 7 + d.rg_n;
    if (lane < n_tail) ot[lane] = static_cast<uint8_t>(tail);
    if (n_tail > 32)
        for (uint32_t j = 32 + lane; j < n_tail; j += 32) ot[j] = tail_byte(d, j);
}

// The name and fields of a line whose name has bytes >= 0x80 (each becomes
// U+FFFD) or whose contig names are not in its slot; returns their bytes.
__device__ __noinline__ uint64_t put_head(uint8_t* o, const SamDev& d, const LinePlan& q, const LineRec& h,
                                          const uint8_t* slot, uint32_t lane) {
    const uint32_t n_nm = q.n_nm;
    uint64_t w = 0;
    for (uint32_t b = 0; b < n_nm; b += 32) {
        const uint32_t i = b + lane;
        const uint8_t c = i < n_nm ? q.name[i] : 0;
        const uint32_t wd = i < n_nm ? (c >= 0x80 ? 3u : 1u) : 0u;
        uint32_t ex = lane, all = min(32u, n_nm - b);
        if (q.widen) {
            uint32_t incl = wd;
            for (int s = 1; s < 32; s <<= 1) {
                const uint32_t v = __shfl_up_sync(FULL, incl, s);
                if (lane >= s) incl += v;
            }
            ex = incl - wd;
            all = __shfl_sync(FULL, incl, 31);
        }
        if (wd == 1) {
            o[w + ex] = c;
        } else if (wd == 3) {
            o[w + ex] = 0xef;
            o[w + ex + 1] = 0xbf;
            o[w + ex + 2] = 0xbd;
        }
        w += all;
    }
    o += w;
    const uint32_t a = q.at_rname, b = q.at_rnext, n = q.slot;
    const uint32_t n1 = a != NONE && h.contig_kind == K_NAME ? h.contig_len : 0;
    const uint32_t n2 = b != NONE && h.rnext_kind == K_NAME ? h.rnext_len : 0;
    const uint8_t *name1 = d.names + h.contig_off, *name2 = d.names + h.rnext_off;
    for (uint32_t i = lane; i < n; i += 32) o[i + (i >= a ? n1 : 0) + (i >= b ? n2 : 0)] = slot[i];
    for (uint32_t i = lane; i < n1; i += 32) o[a + i] = __ldg(name1 + i);
    for (uint32_t i = lane; i < n2; i += 32) o[b + n1 + i] = __ldg(name2 + i);
    return w + n + n1 + n2;
}

// A warp takes `per` consecutive lines.  One lane per line formats its
// fields into a slot of shared memory (all 32 lanes busy); the warp then puts
// the lines together one after the other in its stage and stores it in
// 16-byte blocks when the next line does not fit.  Contig names that do not
// fit the slot are left out of it and put in their places by the warp: 200 k
// lines with names of 80 bytes take 0.28 ms, 0.75 with the lane copying them
// byte by byte (0.18 with names of 20).
// Bound by instruction issue: 1 M lines of 388 B take 0.43 ms with 64 registers
// (eight blocks an SM), 0.49 with the 80 that the compiler would take; with each
// line's fields formatted by its warp, eight lanes busy, and byte-wise copies it
// was 2.04 ms.
__global__ void __launch_bounds__(WRITE_WARPS * 32, 8) sam_write_kernel(SamDev d, uint64_t n_lines, const uint64_t* ends,
                                                                    const LineRec* recs, uint32_t per) {
    __shared__ __align__(16) uint8_t s_stage[WRITE_WARPS][STAGE + 16];
    __shared__ LinePlan s_plan[WRITE_WARPS][32];
    __shared__ uint8_t s_slot[WRITE_WARPS][32][SLOT];
    const uint64_t total = ends[n_lines - 1];
    const bool over = total > d.cap;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        d.status[0] = total;
        if (over) atomicOr(&d.status[2], static_cast<unsigned long long>(E_OVER));
    }
    // error bits of the layout pass (the overflow bit above only repeats
    // `over`)
    if (over || *static_cast<volatile unsigned long long*>(&d.status[2]) != 0) return;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    LinePlan* plan = s_plan[warp];
    uint8_t(*slot)[SLOT] = s_slot[warp];
    const uint32_t tail = lane < 7 + d.rg_n ? tail_byte(d, lane) : 0;
    const uint64_t n_warps = static_cast<uint64_t>(gridDim.x) * WRITE_WARPS;
    for (uint64_t base = (static_cast<uint64_t>(blockIdx.x) * WRITE_WARPS + warp) * per; base < n_lines;
         base += n_warps * per) {
        const uint64_t L = base + lane;
        uint64_t start = 0;
        uint32_t bytes = 0;
        if (lane < per && L < n_lines) {
            const LineRec h = recs[L];
            const uint64_t r = d.paired ? (L >> 1) + (L & 1) * d.n1 : L;
            start = L ? ends[L - 1] : 0;
            bytes = static_cast<uint32_t>(ends[L] - start);
            LinePlan q;
            q.name = d.arena + d.name_off[r];
            q.seq = d.arena + d.seq_off[r];
            q.qual = d.arena + d.qual_off[r];
            q.n_nm = d.name_len[r];
            q.n_sq = d.seq_len[r];
            q.n_ql = d.qual_len[r];
            q.rc = h.mapped && (h.flag & 16);
            const uint64_t f = fields_len(h);
            const bool names = f <= SLOT;  // the contig names fit the slot too
            const Cuts cuts = put_fields(slot[lane], d, h, names);
            q.fields = names && !h.widen ? static_cast<uint32_t>(f) : 0;
            q.widen = h.widen;
            q.slot = static_cast<uint8_t>(cuts.end);
            q.at_rname = static_cast<uint8_t>(names ? NONE : cuts.rname);
            q.at_rnext = static_cast<uint8_t>(names ? NONE : cuts.rnext);
            plan[lane] = q;
        }
        __syncwarp();
        const uint32_t count = static_cast<uint32_t>(n_lines - base < per ? n_lines - base : per);
        LineRaw next;
        load_raw(next, plan[0], lane);
        span::staged_run<STAGE>(d.sam + __shfl_sync(FULL, start, 0), s_stage[warp], bytes, count, lane,
                                [&](uint8_t* o, uint32_t k) {
                                    const LineRaw x = next;  // the next line's bytes are on their way
                                    const LinePlan& q = plan[k];
                                    if (k + 1 < count) load_raw(next, plan[k + 1], lane);
                                    const uint32_t n_nm = q.n_nm, fields = q.fields;
                                    if (!fields) {
                                        o += put_head(o, d, q, recs[base + k], slot[k], lane);
                                    } else {
                                        if (lane < n_nm) o[lane] = static_cast<uint8_t>(x.n0);
                                        if (lane + 32 < n_nm) o[lane + 32] = static_cast<uint8_t>(x.n1);
                                        if (n_nm > 64)
                                            for (uint32_t i = 64 + lane; i < n_nm; i += 32) o[i] = __ldg(q.name + i);
                                        o += n_nm;
                                        for (uint32_t i = lane; i < fields; i += 32) o[i] = slot[k][i];
                                        o += fields;
                                    }
                                    put_rest(o, d, q, x, tail, lane);
                                });
    }
}

}  // namespace

size_t sam_scratch_bytes(uint64_t n_lines) {
    size_t t = 0;
    cub::DeviceScan::InclusiveSum(nullptr, t, static_cast<const uint32_t*>(nullptr), static_cast<uint64_t*>(nullptr),
                                  static_cast<int64_t>(n_lines ? n_lines : 1));
    return align256(n_lines * 4) + align256(n_lines * 8) + align256(n_lines * sizeof(LineRec)) + align256(t);
}

int enqueue_sam(const SamDev& d, void* scratch, size_t scratch_bytes, int sm_count, cudaStream_t st) {
    const uint64_t n_lines = static_cast<uint64_t>(d.n1) * (d.paired ? 2 : 1);
    if (!n_lines) return 0;
    uint8_t* s = static_cast<uint8_t*>(scratch);
    uint32_t* line_len = reinterpret_cast<uint32_t*>(s);
    s += align256(n_lines * 4);
    uint64_t* ends = reinterpret_cast<uint64_t*>(s);
    s += align256(n_lines * 8);
    LineRec* recs = reinterpret_cast<LineRec*>(s);
    s += align256(n_lines * sizeof(LineRec));
    void* temp = s;
    size_t tb = scratch_bytes - static_cast<size_t>(s - static_cast<uint8_t*>(scratch));
    const uint64_t sms = static_cast<uint64_t>(sm_count > 0 ? sm_count : 148);
    const uint64_t g1w = (n_lines + THREADS - 1) / THREADS, g1c = sms * 8;
    sam_layout_kernel<<<static_cast<unsigned>(g1w < g1c ? g1w : g1c), THREADS, 0, st>>>(d, n_lines, line_len, recs);
    check_launch(cudaGetLastError(), "sam_layout_kernel");
    check_launch(cub::DeviceScan::InclusiveSum(temp, tb, static_cast<const uint32_t*>(line_len), ends,
                                               static_cast<int64_t>(n_lines), st),
                 "sam scan");
    // 32 lines a warp where that still gives every SM 32 warps, fewer (down to
    // 4) for a small batch: its lines spread over more warps
    uint32_t per = 32;
    while (per > 4 && (n_lines + per - 1) / per < sms * 32) per /= 2;
    const uint64_t g2w = (n_lines + WRITE_WARPS * per - 1) / (WRITE_WARPS * per), g2c = sms * 16;
    sam_write_kernel<<<static_cast<unsigned>(g2w < g2c ? g2w : g2c), WRITE_WARPS * 32, 0, st>>>(d, n_lines, ends, recs,
                                                                                             per);
    check_launch(cudaGetLastError(), "sam_write_kernel");
    return 4;
}

}  // namespace ma
