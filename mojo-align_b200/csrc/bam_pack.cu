// bam_pack.cu - BAM records of one mapped batch, packed on the device.
//
// Replaces the host loop _emit_bam_from_batch / _pack_bam_aln
// (fq2bam-meth/src/linear_gpu_fm.mojo:497-666, 669-984).  The reference
// packs records one after another into a host buffer; here the layout is
// split from the bytes so every record is written in parallel at the same
// offset the serial loop would give it:
//   1. bam_layout_kernel   one thread per read (single-end) or pair: flags,
//                          mate fields and the record sizes, plus every
//                          sort/markdup metadata entry except `rec`.
//   2. an inclusive scan of the record sizes (CUB) -> end offsets.
//   3. bam_records_kernel  a warp per run of records: one lane works out a
//                          record's fields, then the warp assembles the
//                          records in a shared-memory stage placed at the
//                          destination's 16-byte phase and stores it in
//                          16-byte blocks (byte stores at the run's two
//                          ragged ends).  Records too long for the stage
//                          are assembled in place in HBM.
// All byte-order, clamping and truncation rules are the reference's; every
// integer is formed in 64-bit arithmetic and truncated where the reference
// stores 32 bits.
#include <cub/device/device_scan.cuh>

#include <string>

#include "bam_pack.h"
#include "ma_internal.h"
#include "span.cuh"

namespace ma {
namespace {

using span::put_bytes;
using span::Span8;
using span::span8_bytes;
using span::span8_load;

constexpr int LAYOUT_THREADS = 256;
constexpr int REC_WARPS = 4;
constexpr uint32_t REC_STAGE = 3072;  // bytes of output a warp gathers before it stores them

// Per-record fields after the mate logic of _emit_bam_from_batch.
struct BamRec {
    int64_t flag, tid, pos, mapq, sl, sr, nm, qlen, ntid, npos, tlen;
    uint64_t name_off, orig_off, qual_off;
    uint32_t name_len, qual_len;
    bool has_qual;  // qualities exist and their length equals qlen
    bool bad;       // an arena span lies outside the arena
};

// One read's own fields; `mate_bit` is 64 for R1 and 128 for R2
// (L756-768, L838-848).
__device__ __forceinline__ void load_read(const BamDev& b, uint64_t r, int64_t mate_bit, BamRec& o) {
    const int64_t rid = b.rid[r];
    o.pos = b.pos[r];
    o.mapq = b.mapq[r];
    o.flag = static_cast<int64_t>(b.flag[r]) | 1 | mate_bit;
    o.sl = b.sl[r];
    o.sr = b.sr[r];
    o.nm = b.nm[r];
    o.tid = -1;
    if (rid >= 0 && rid < b.n_tid) o.tid = b.rid_to_tid[rid];
    else o.flag |= 4;
    o.qlen = b.orig_len[r];
    o.name_off = b.name_off[r];
    o.name_len = b.name_len[r];
    o.orig_off = b.orig_off[r];
    o.ntid = o.npos = -1;
    o.tlen = 0;
    o.bad = o.name_off + o.name_len > b.arena_bytes || o.orig_off + static_cast<uint64_t>(o.qlen) > b.arena_bytes;
    o.has_qual = false;
    o.qual_off = 0;
    o.qual_len = 0;
    if (b.qual_off) {
        o.qual_off = b.qual_off[r];
        o.qual_len = b.qual_len[r];
        o.has_qual = static_cast<int64_t>(o.qual_len) == o.qlen;
        if (o.has_qual && o.qual_off + o.qual_len > b.arena_bytes) o.bad = true;
    }
    if (o.bad) o.has_qual = false;
}

// Mate flags, mate fields and TLEN of a pair (L849-874).
__device__ __forceinline__ void pair_up(BamRec& a, BamRec& c) {
    if (a.tid < 0) c.flag |= 8;
    if (c.tid < 0) a.flag |= 8;
    if (a.tid >= 0 && c.tid >= 0 && a.tid == c.tid) {
        a.flag |= 2;
        c.flag |= 2;
        a.ntid = a.tid;
        c.ntid = c.tid;
        a.npos = c.pos;
        c.npos = a.pos;
        int64_t tl = c.pos - a.pos;
        if (tl < 0) tl = -tl;
        tl += c.qlen;
        a.tlen = a.pos <= c.pos ? tl : -tl;
        c.tlen = -a.tlen;
    } else {
        if (a.tid >= 0) {
            c.ntid = a.tid;
            c.npos = a.pos;
        }
        if (c.tid >= 0) {
            a.ntid = c.tid;
            a.npos = c.pos;
        }
    }
}

// Loads unit u (a read, or pair u) into r[0] (and r[1]).
__device__ __forceinline__ void load_unit(const BamDev& b, uint64_t u, BamRec* r) {
    load_read(b, u, 64, r[0]);
    if (b.paired) {
        load_read(b, static_cast<uint64_t>(b.n1) + u, 128, r[1]);
        pair_up(r[0], r[1]);
    }
}

// Clip clamping of _pack_bam_aln (L521-530) and _unclipped5 (L371-386).
__device__ __forceinline__ void clamp_clips(const BamRec& r, int64_t& sl, int64_t& sr, int64_t& mid) {
    sl = r.sl < 0 ? 0 : r.sl;
    sr = r.sr < 0 ? 0 : r.sr;
    if (sl + sr >= r.qlen) sl = sr = 0;
    mid = r.qlen - sl - sr;
}

__device__ __forceinline__ bool placed(const BamRec& r) { return r.tid >= 0 && (r.flag & 4) == 0; }

__device__ __forceinline__ int64_t n_cigar_of(const BamRec& r) {
    int64_t sl, sr, mid;
    clamp_clips(r, sl, sr, mid);
    return placed(r) ? (sl > 0) + (mid > 0) + (sr > 0) : 0;
}

// Bytes of the record including its block_size word (L545-546).
__device__ __forceinline__ uint64_t record_bytes(const BamRec& r, uint32_t rg_n) {
    const int64_t block = 32 + (static_cast<int64_t>(r.name_len) + 1) + 4 * n_cigar_of(r) + (r.qlen + 1) / 2 +
                          r.qlen + (3 + static_cast<int64_t>(rg_n) + 1 + 4);
    return static_cast<uint64_t>(4 + block);
}

__device__ __forceinline__ int64_t unclipped5(const BamRec& r) {
    if ((r.flag & 4) != 0 || r.qlen <= 0) return 0;
    int64_t sl, sr, mid;
    clamp_clips(r, sl, sr, mid);
    return (r.flag & 16) ? r.pos + mid + sl - 1 : r.pos - sl;
}

__device__ __forceinline__ uint64_t coord_key(int64_t tid, int64_t pos, uint64_t orig) {
    if (tid < 0) return (0xffffffffull << 32) | (orig & 0xffffffffull);
    return (static_cast<uint64_t>(tid) << 32) | static_cast<uint64_t>(pos < 0 ? 0 : pos);
}

__device__ __forceinline__ uint64_t pack_end(const BamRec& r) {
    const uint64_t t = r.tid >= 0 ? static_cast<uint64_t>(r.tid + 1) : 0;
    int64_t u = unclipped5(r) + 1073741824;
    if (u < 0) u = 0;
    return (t << 48) | (static_cast<uint64_t>((r.flag >> 4) & 1) << 47) |
           (static_cast<uint64_t>(u) & 140737488355327ull);
}

__device__ __forceinline__ int64_t clamp255(int64_t v) { return v < 0 ? 0 : (v > 255 ? 255 : v); }

// Metadata and sizes, one thread per unit (L799-822, L928-982).
__global__ void __launch_bounds__(LAYOUT_THREADS) bam_layout_kernel(BamDev b, uint64_t* rec_bytes) {
    const uint64_t n_units = b.n1;
    const uint64_t u = static_cast<uint64_t>(blockIdx.x) * LAYOUT_THREADS + threadIdx.x;
    unsigned mapped = 0;
    unsigned bad = 0;
    if (u < n_units) {
        BamRec r[2];
        load_unit(b, u, r);
        if (!b.paired) {
            const uint64_t t = b.n_reads + u, m = t - b.meta_origin;
            b.coord[m] = coord_key(r[0].tid, r[0].pos, t);
            if (r[0].tid >= 0) {
                b.dhi[m] = pack_end(r[0]);
                b.dlo[m] = 0;
            } else {
                b.dhi[m] = ~0ull;
                b.dlo[m] = t;
            }
            const uint64_t n = record_bytes(r[0], b.rg_n);
            rec_bytes[u] = n;
            b.len[m] = static_cast<uint32_t>(n);
            b.score[m] = static_cast<uint32_t>((r[0].mapq << 8) | (255 - clamp255(r[0].nm)));
            b.pair[m] = static_cast<uint32_t>(b.n_total + t);
            mapped = r[0].tid >= 0;
            bad = r[0].bad;
        } else {
            const uint64_t i1 = b.n_reads + 2 * u, i2 = i1 + 1;
            const uint32_t pid = static_cast<uint32_t>((b.n_total + i1) / 2);
            const uint32_t pscore =
                static_cast<uint32_t>(((r[0].mapq + r[1].mapq) << 8) | (255 - clamp255(r[0].nm + r[1].nm)));
            uint64_t dhi = ~0ull, dlo = i1;
            if (r[0].tid >= 0 || r[1].tid >= 0) {
                const uint64_t e1 = pack_end(r[0]), e2 = pack_end(r[1]);
                if (r[0].tid < 0) {
                    dhi = e2;
                    dlo = 0;
                } else if (r[1].tid < 0) {
                    dhi = e1;
                    dlo = 0;
                } else {
                    dhi = e1 <= e2 ? e1 : e2;
                    dlo = e1 <= e2 ? e2 : e1;
                }
            }
            const uint64_t n1b = record_bytes(r[0], b.rg_n), n2b = record_bytes(r[1], b.rg_n);
            rec_bytes[2 * u] = n1b;
            rec_bytes[2 * u + 1] = n2b;
            const uint64_t m1 = i1 - b.meta_origin, m2 = m1 + 1;
            b.coord[m1] = coord_key(r[0].tid, r[0].pos, i1);
            b.coord[m2] = coord_key(r[1].tid, r[1].pos, i2);
            b.dhi[m1] = b.dhi[m2] = dhi;
            b.dlo[m1] = b.dlo[m2] = dlo;
            b.len[m1] = static_cast<uint32_t>(n1b);
            b.len[m2] = static_cast<uint32_t>(n2b);
            b.score[m1] = b.score[m2] = pscore;
            b.pair[m1] = b.pair[m2] = pid;
            mapped = (r[0].tid >= 0) + (r[1].tid >= 0);
            bad = r[0].bad + r[1].bad;
        }
    }
    // one atomic per warp for each counter
    for (int o = 16; o > 0; o >>= 1) {
        mapped += __shfl_xor_sync(0xffffffffu, mapped, o);
        bad += __shfl_xor_sync(0xffffffffu, bad, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (mapped) atomicAdd(&b.status[1], static_cast<unsigned long long>(mapped));
        if (bad) atomicAdd(&b.status[2], static_cast<unsigned long long>(bad));
    }
}

__device__ __forceinline__ int64_t reg2bin(int64_t beg, int64_t end) {
    if (end <= beg) end = beg + 1;
    --end;
    if ((beg >> 14) == (end >> 14)) return 4681 + (beg >> 14);
    if ((beg >> 17) == (end >> 17)) return 585 + (beg >> 17);
    if ((beg >> 20) == (end >> 20)) return 73 + (beg >> 20);
    if ((beg >> 23) == (end >> 23)) return 9 + (beg >> 23);
    if ((beg >> 26) == (end >> 26)) return 1 + (beg >> 26);
    return 0;
}

// What the warp needs of a record to write its bytes, filled in by one lane:
// the nine little-endian header words of _pack_bam_aln (L551-572: block_size,
// refID, pos, bin_mq_nl, flag_nc, l_seq, next_refID, next_pos, tlen), up to
// three CIGAR ops, and the spans.
struct __align__(16) RecPlan {
    uint32_t w[12];
    const uint8_t* name;  // null: zero bytes in its place (and of SEQ)
    const uint8_t* seq;
    const uint8_t* qual;  // null: 255 in every byte
    uint32_t name_len, qlen;
    uint32_t n_cigar, rev, nm, pad;
};
static_assert(sizeof(RecPlan) == 96, "record plan layout");

__device__ __forceinline__ void plan_record(RecPlan& q, const BamDev& b, const BamRec& r) {
    const bool rev = (r.flag & 16) != 0;
    int64_t sl, sr, mid;
    clamp_clips(r, sl, sr, mid);
    if (rev) {
        const int64_t t = sl;
        sl = sr;
        sr = t;
    }
    const bool pl = placed(r);
    const int n_cigar = pl ? (sl > 0) + (mid > 0) + (sr > 0) : 0;
    const int64_t l_qname = static_cast<int64_t>(r.name_len) + 1;
    const int64_t block = static_cast<int64_t>(record_bytes(r, b.rg_n)) - 4;
    const int64_t bin = pl ? reg2bin(r.pos, r.pos + mid) : 4680;
    q.w[0] = static_cast<uint32_t>(block);
    q.w[1] = static_cast<uint32_t>(pl ? r.tid : -1);
    q.w[2] = static_cast<uint32_t>(pl ? r.pos : -1);
    q.w[3] = static_cast<uint32_t>((bin << 16) | (clamp255(r.mapq) << 8) | l_qname);
    q.w[4] = static_cast<uint32_t>((r.flag << 16) | n_cigar);
    q.w[5] = static_cast<uint32_t>(r.qlen);
    q.w[6] = static_cast<uint32_t>(r.ntid < 0 ? -1 : r.ntid);
    q.w[7] = static_cast<uint32_t>(r.ntid < 0 ? -1 : r.npos);
    q.w[8] = static_cast<uint32_t>(r.tlen);
    // the present ops of S(sl) M(mid) S(sr)
    int k = 9;
    if (pl && sl > 0) q.w[k++] = static_cast<uint32_t>((sl << 4) | 4);
    if (pl && mid > 0) q.w[k++] = static_cast<uint32_t>(mid << 4);
    if (pl && sr > 0) q.w[k++] = static_cast<uint32_t>((sr << 4) | 4);
    q.name = r.bad ? nullptr : b.arena + r.name_off;
    q.seq = r.bad ? nullptr : b.arena + r.orig_off;
    q.qual = r.has_qual ? b.arena + r.qual_off : nullptr;
    q.name_len = r.name_len;
    q.qlen = static_cast<uint32_t>(r.qlen);
    q.n_cigar = n_cigar;
    q.rev = rev;
    q.nm = static_cast<uint32_t>(clamp255(r.nm));
}

// _nt16 (L455-464) of four bases at once: A/C/G/T in either case -> 1/2/4/8,
// anything else 15; comp: _nt16_comp (L467-476) of that, A<->T, C<->G.
// Bits 1-2 of a letter tell A, C, T and G apart; the letter they stand for
// is compared with the byte to find the others.
__device__ __forceinline__ uint32_t nt16x4(uint32_t x, bool comp) {
    const uint32_t c = x & 0xdfdfdfdfu;  // upper case
    const uint32_t i = (c >> 1) & 0x03030303u;
    const uint32_t sel = __byte_perm(i | (i >> 4), 0, 0x4420);  // one nibble per base
    const uint32_t d = __byte_perm(0x47544341u, 0, sel) ^ c;
    const uint32_t code = __byte_perm(comp ? 0x02010408u : 0x04080201u, 0, sel);
    const uint32_t other = ((((d & 0x7f7f7f7fu) + 0x7f7f7f7fu) | d) >> 7) & 0x01010101u;
    return code | other * 15u;
}

// Four quality bytes: phred+33 minus 33, 255 below '!'.
__device__ __forceinline__ uint32_t qual4(uint32_t x) {
    const uint32_t hb = x & 0x80808080u;
    const uint32_t y = (x | 0x80808080u) - 0x21212121u;  // 128 + (low seven bits) - 33 in each byte, no borrow
    const uint32_t t = y & 0x80808080u;
    // bytes >= 128: y itself; below 128: y - 128, or 255 where that is negative
    return (y & ~(t & ~hb)) | (((~(hb | t) & 0x80808080u) >> 7) * 255u);
}

// Bytes of the tags RG:Z:<rg> and NM:C:<nm> but the last one, which is nm
// (L655-665).
__device__ __forceinline__ uint8_t tag_byte(const BamDev& b, uint32_t i) {
    if (i < 3) return i == 0 ? 82 : (i == 1 ? 71 : 90);
    if (i < 3 + b.rg_n) return b.rg[i - 3];
    i -= 3 + b.rg_n;
    return i == 0 ? 0 : (i == 1 ? 78 : (i == 2 ? 77 : 67));
}

// A lane's share of a record's source bytes: two name bytes, eight bases,
// eight qualities; for records of up to 63 name bytes and 256 bases that is
// all of them.
struct RecRaw {
    uint32_t n0, n1;
    Span8 seq, qual;
};
constexpr uint32_t RAW_NAME = 64;  // l_qname that one RecRaw per lane covers

__device__ __forceinline__ void load_raw(RecRaw& x, const RecPlan& q, uint32_t lane) {
    const uint8_t* name = q.name;
    const uint32_t nn = name ? q.name_len : 0;
    x.n0 = lane < nn ? __ldg(name + lane) : 0;
    x.n1 = lane + 32 < nn ? __ldg(name + lane + 32) : 0;
    x.seq = span8_load(q.seq, q.seq ? q.qlen : 0, lane, q.rev);
    x.qual = span8_load(q.qual, q.qual ? q.qlen : 0, lane, q.rev);
}

// SEQ bytes of eight bases: byte k holds bases 2k and 2k+1 of the stored
// strand; on the reverse strand base i is the complement of original base
// qlen-1-i (L617-639).  left < 8: the span's last bases.
__device__ __forceinline__ uint32_t seq_word(uint2 x, bool rev, uint32_t left) {
    const uint32_t c0 = nt16x4(x.x, rev), c1 = nt16x4(x.y, rev);
    const uint32_t v = __byte_perm((c0 << 4) | (c0 >> 8), (c1 << 4) | (c1 >> 8), 0x6420);
    return left < 8 && (left & 1) ? v & ~(15u << (4 * left - 4)) : v;  // no second base in the last byte
}

// The warp writes the planned record at dst (shared or global), _pack_bam_aln
// L520-666: lanes 0-11 the header words and CIGAR ops, then the name, SEQ,
// QUAL (all 255 without qualities of the read's length, reversed on the
// reverse strand, L640-654) and the tags; tag: this lane's tag byte.
__device__ __forceinline__ void write_record(uint8_t* dst, const BamDev& b, const RecPlan& q, const RecRaw& x,
                                             uint32_t tag, uint32_t n_tags, uint32_t lane) {
    const uint32_t qlen = q.qlen, l_qname = q.name_len + 1, n_cigar = q.n_cigar;
    const bool rev = q.rev;
    const uint8_t *seq = q.seq, *qual = q.qual;
    const uint32_t o_cig = 36 + l_qname, o_seq = o_cig + 4 * n_cigar, o_qual = o_seq + (qlen + 1) / 2;
    const uint32_t o_tag = o_qual + qlen;
    if (lane < 9 + n_cigar) put_bytes(dst + 4 * lane + (lane < 9 ? 0 : o_cig - 36), q.w[lane], 4);
    if (lane < l_qname) dst[36 + lane] = static_cast<uint8_t>(x.n0);
    if (lane + 32 < l_qname) dst[68 + lane] = static_cast<uint8_t>(x.n1);
    if (l_qname > RAW_NAME)
        for (uint32_t i = RAW_NAME + lane; i < l_qname; i += 32)
            dst[36 + i] = i + 1 < l_qname && q.name ? __ldg(q.name + i) : 0;
    for (uint32_t i = lane; 8 * i < qlen; i += 32) {
        const uint32_t left = qlen - 8 * i;
        uint32_t v = 0;
        uint2 u = make_uint2(~0u, ~0u);
        if (seq) v = seq_word(span8_bytes(i < 32 ? x.seq : span8_load(seq, qlen, i, rev), seq, qlen, rev), rev, left);
        if (qual) {
            u = span8_bytes(i < 32 ? x.qual : span8_load(qual, qlen, i, rev), qual, qlen, rev);
            u = make_uint2(qual4(u.x), qual4(u.y));
        }
        put_bytes(dst + o_seq + 4 * i, v, min(4u, (left + 1) >> 1));
        put_bytes(dst + o_qual + 8 * i, u.x, min(4u, left));
        if (left > 4) put_bytes(dst + o_qual + 8 * i + 4, u.y, min(4u, left - 4));
    }
    if (lane < n_tags) dst[o_tag + lane] = static_cast<uint8_t>(lane + 1 == n_tags ? q.nm : tag);
    if (n_tags > 32)
        for (uint32_t i = 32 + lane; i < n_tags; i += 32)
            dst[o_tag + i] = i + 1 == n_tags ? static_cast<uint8_t>(q.nm) : tag_byte(b, i);
}

// A warp takes `per` consecutive records (whole pairs).  One lane per record
// works out its fields (the mate's by shuffle); the warp then writes the
// records one after the other into its stage, placed at the destination's
// 16-byte phase, and stores the stage in 16-byte blocks when the next record
// does not fit.  A record longer than the stage is built in place.
// Bound by instruction issue: 1 M records of 314 B (150 bases) take 0.43 ms;
// with the fields worked out by every lane and byte-wise loads, conversions
// and per-pair stores it was 1.53 ms.
__global__ void __launch_bounds__(REC_WARPS * 32) bam_records_kernel(BamDev b, const uint64_t* rec_end, uint32_t per) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ __align__(16) uint8_t s_stage[REC_WARPS][REC_STAGE + 16];
    __shared__ RecPlan s_plan[REC_WARPS][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t n_rec = b.paired ? 2ull * b.n1 : b.n1;
    const uint64_t total = rec_end[n_rec - 1];
    if (blockIdx.x == 0 && threadIdx.x == 0) b.status[0] = total;
    if (total > b.cap) return;
    const uint32_t n_tags = 3 + b.rg_n + 1 + 4;
    const uint32_t tag = lane + 1 < n_tags ? tag_byte(b, lane) : 0;
    uint8_t* stage = s_stage[warp];
    RecPlan* plan = s_plan[warp];
    const uint64_t chunk_hi = static_cast<uint64_t>(b.chunk) << 32;
    const uint64_t n_warps = static_cast<uint64_t>(gridDim.x) * REC_WARPS;
    for (uint64_t base = (static_cast<uint64_t>(blockIdx.x) * REC_WARPS + warp) * per; base < n_rec;
         base += n_warps * per) {
        const uint64_t j = base + lane;
        const bool mine = lane < per && j < n_rec;
        uint64_t start = 0;
        uint32_t bytes = 0;
        BamRec r{};
        r.tid = -1;
        if (mine) {
            start = j ? rec_end[j - 1] : 0;
            bytes = static_cast<uint32_t>(rec_end[j] - start);
            b.rec[b.n_reads + j - b.meta_origin] = chunk_hi | start;
            if (b.paired) load_read(b, (j >> 1) + (j & 1) * b.n1, (j & 1) ? 128 : 64, r);
            else load_read(b, j, 64, r);
        }
        if (b.paired) {  // pair_up from this lane's side; pairs sit in lanes 2i, 2i + 1
            const int64_t mtid = __shfl_xor_sync(FULL, r.tid, 1), mpos = __shfl_xor_sync(FULL, r.pos, 1);
            const int64_t mqlen = __shfl_xor_sync(FULL, r.qlen, 1);
            if (mtid < 0) r.flag |= 8;
            if (r.tid >= 0 && r.tid == mtid) r.flag |= 2;
            if (mtid >= 0) {
                r.ntid = mtid;
                r.npos = mpos;
            }
            if (r.tid >= 0 && r.tid == mtid) {
                const int64_t p1 = (lane & 1) ? mpos : r.pos, p2 = (lane & 1) ? r.pos : mpos;
                const int64_t tl = (p2 < p1 ? p1 - p2 : p2 - p1) + ((lane & 1) ? r.qlen : mqlen);
                const int64_t t1 = p1 <= p2 ? tl : -tl;
                r.tlen = (lane & 1) ? -t1 : t1;
            }
        }
        if (mine) plan_record(plan[lane], b, r);
        __syncwarp();
        const uint32_t count = static_cast<uint32_t>(n_rec - base < per ? n_rec - base : per);
        RecRaw next;
        load_raw(next, plan[0], lane);
        span::staged_run<REC_STAGE>(b.bam + __shfl_sync(FULL, start, 0), stage, bytes, count, lane,
                                    [&](uint8_t* dst, uint32_t k) {
                                        const RecRaw x = next;  // the next record's bytes are on their way
                                        if (k + 1 < count) load_raw(next, plan[k + 1], lane);
                                        write_record(dst, b, plan[k], x, tag, n_tags, lane);
                                    });
    }
}

void check_launch(cudaError_t e, const char* what) {
    if (e != cudaSuccess) fail(MA_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

size_t align256(size_t n) { return (n + 255) & ~static_cast<size_t>(255); }

size_t scan_temp_bytes(uint64_t n_rec) {
    size_t t = 0;
    cub::DeviceScan::InclusiveSum(nullptr, t, static_cast<const uint64_t*>(nullptr),
                                  static_cast<uint64_t*>(nullptr), static_cast<int64_t>(n_rec));
    return t;
}

}  // namespace

size_t bam_scratch_bytes(uint64_t n_rec) {
    return 2 * align256(n_rec * sizeof(uint64_t)) + align256(scan_temp_bytes(n_rec));
}

const uint64_t* bam_total_in_scratch(const void* scratch, uint64_t n_rec) {
    const uint8_t* s = static_cast<const uint8_t*>(scratch);
    return reinterpret_cast<const uint64_t*>(s + align256(n_rec * sizeof(uint64_t))) + (n_rec - 1);
}

int enqueue_bam_layout(const BamDev& b, void* scratch, size_t scratch_bytes, cudaStream_t st) {
    const uint64_t n_rec = b.paired ? 2ull * b.n1 : b.n1;
    uint8_t* s = static_cast<uint8_t*>(scratch);
    uint64_t* sizes = reinterpret_cast<uint64_t*>(s);
    uint64_t* ends = reinterpret_cast<uint64_t*>(s + align256(n_rec * sizeof(uint64_t)));
    void* temp = s + 2 * align256(n_rec * sizeof(uint64_t));
    size_t temp_bytes = scratch_bytes - 2 * align256(n_rec * sizeof(uint64_t));
    const unsigned grid = static_cast<unsigned>((b.n1 + LAYOUT_THREADS - 1) / LAYOUT_THREADS);
    bam_layout_kernel<<<grid, LAYOUT_THREADS, 0, st>>>(b, sizes);
    check_launch(cudaGetLastError(), "bam_layout_kernel");
    check_launch(cub::DeviceScan::InclusiveSum(temp, temp_bytes, static_cast<const uint64_t*>(sizes), ends,
                                               static_cast<int64_t>(n_rec), st),
                 "bam record scan");
    return 3;  // the layout kernel and the scan's two
}

int enqueue_bam_records(const BamDev& b, const void* scratch, int sm_count, cudaStream_t st) {
    const uint64_t n_rec = b.paired ? 2ull * b.n1 : b.n1;
    const uint64_t* ends =
        reinterpret_cast<const uint64_t*>(static_cast<const uint8_t*>(scratch) + align256(n_rec * sizeof(uint64_t)));
    // 32 records a warp where that still gives every SM 32 warps, fewer (down
    // to 4) for a small batch: its records spread over more warps
    const uint64_t sms = static_cast<uint64_t>(sm_count > 0 ? sm_count : 148);
    uint32_t per = 32;
    while (per > 4 && (n_rec + per - 1) / per < sms * 32) per /= 2;
    const uint64_t want = (n_rec + REC_WARPS * per - 1) / (REC_WARPS * per);
    const uint64_t cap = sms * 16;
    const unsigned grid = static_cast<unsigned>(want < cap ? want : cap);
    bam_records_kernel<<<grid, REC_WARPS * 32, 0, st>>>(b, ends, per);
    check_launch(cudaGetLastError(), "bam_records_kernel");
    return 1;
}

}  // namespace ma
