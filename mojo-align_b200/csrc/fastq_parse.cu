// fastq_parse.cu - FASTQ record split on the device.
//
// Replaces the host record split of the FM path's two FASTQ readers and
// the row packing fq_pack_bases (fq2bam-meth/src/linear_fastq.mojo:454-492):
//   rules 0, the BAM path's reader (linear_fastq.mojo: _pipe_line L233-280,
//     _qname_span L308-325, _store_rec L365-417, fq_read_batch L437-451):
//     one trailing '\r' dropped per line, a record cut short is an error;
//   rules 1, the SAM path's reader (fq2bam-meth/python/fastq_batch.py:
//     _qname L18-28, FastqPairReader._one / read_batch L250-317): every
//     trailing '\r' dropped, four lines per record whatever they hold, and
//     at the end of the stream a record cut short reads its missing lines
//     as empty.  The reference walks the decompressed
// bytes one record at a time on one host thread and copies name, original
// bases, converted bases and qualities into an arena; here the uncompressed
// bytes are copied to HBM once and become the arena themselves:
//   1. nl_count_kernel / scan / nl_write_kernel: the bytes are read once, in
//      aligned 16-byte chunks, and leave a bit per byte ('\n' or not) and a
//      count per tile of 16 KB; the positions come from the bits;
//   2. fq_lines_kernel (one thread): lines, complete records, the bytes
//      consumed and the truncation error, exactly as the reference's line
//      reader sees the stream;
//   3. fq_records_kernel: one thread per record, name span (leading '@'
//      dropped, cut at ' ' or '/'), SEQ and QUAL spans without their
//      trailing '\r' (one, or all), the longest SEQ;
//   4. fq_rows_kernel: 16 bytes of the padded rows the mapper takes ('N'
//      fill) per thread.  The C->T / G->A conversion is applied by the
//      mapper's pack kernel, so the rows hold the original bases.
// The newline array is sized before the newlines are counted (a line per 32
// bytes: FASTQ of reads above ~50 bases), so all passes are enqueued at once
// and the host waits for one status copy; denser texts size it by the count
// and repeat the passes from the positions on.  340 MB of 150-base records:
// parse and rows 0.36 ms; 0.70 ms with a byte-wise row copy and name scan, the
// bytes read twice and three waits.
#include <cub/device/device_scan.cuh>

#include <string>

#include "fastq_parse.h"
#include "ma_internal.h"

namespace ma {
namespace {

constexpr int THREADS = 256;
constexpr int CHUNK = 16;                   // bytes per bit mask (uint16_t)
constexpr int TILE_CHUNKS = 4 * THREADS;    // chunks per tile: four per thread
constexpr uint64_t NL_BYTES = 32;           // text bytes per newline the array is sized for at first

void check_launch(cudaError_t e, const char* what) {
    if (e != cudaSuccess) fail(MA_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

size_t align256(size_t n) { return (n + 255) & ~static_cast<size_t>(255); }

// Bit j of the result: byte j of w is '\n'.
__device__ __forceinline__ uint32_t nl_bits(uint32_t w) {
    // '\n' bytes of w become zero bytes of x; the exact zero-byte test sets
    // 0x80 in exactly those byte lanes, the product gathers the four bits
    const uint32_t x = w ^ 0x0a0a0a0au;
    const uint32_t t = ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x | 0x7f7f7f7fu);
    return ((t >> 7) * 0x01020408u) >> 24;
}

// Chunk c covers the 16 bytes from byte 16 c - lead of the buffer on, lead =
// how far the buffer starts past a 16-byte boundary; bits of bytes outside
// the buffer stay 0.
__global__ void __launch_bounds__(THREADS) nl_count_kernel(const uint8_t* buf, uint64_t n, uint64_t n_chunks,
                                                          uint16_t* bits, uint32_t* counts) {
    __shared__ uint32_t part[THREADS / 32];
    const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(buf) & 15);
    const uint4* src = reinterpret_cast<const uint4*>(buf - lead);
    const uint64_t c0 = static_cast<uint64_t>(blockIdx.x) * TILE_CHUNKS + threadIdx.x;
    uint32_t count = 0;
    uint4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        v[k] = c0 + k * THREADS < n_chunks ? __ldg(src + c0 + k * THREADS) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint64_t c = c0 + k * THREADS;
        if (c >= n_chunks) break;
        uint32_t m = nl_bits(v[k].x) | nl_bits(v[k].y) << 4 | nl_bits(v[k].z) << 8 | nl_bits(v[k].w) << 12;
        if (c == 0) m &= 0xffffu << lead;
        const uint64_t end = n + lead - c * CHUNK;  // bytes of the chunk before the buffer's end
        if (end < CHUNK) m &= (1u << end) - 1;
        bits[c] = static_cast<uint16_t>(m);
        count += __popc(m & 0xffffu);
    }
    for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = count;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < THREADS / 32; ++w) t += part[w];
        counts[blockIdx.x] = t;
    }
}

// Positions of the tile's newlines from the bits (64 bytes of text per
// thread), the first nl_cap of them.
__global__ void __launch_bounds__(THREADS) nl_write_kernel(uint32_t lead, uint64_t n_chunks, const uint16_t* bits,
                                                          const uint32_t* tile_base, uint32_t* nl, uint64_t nl_cap) {
    __shared__ uint32_t part[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t c0 = static_cast<uint64_t>(blockIdx.x) * TILE_CHUNKS + 4 * threadIdx.x;
    uint64_t m = 0;
    if (c0 + 4 <= n_chunks) {
        m = __ldg(reinterpret_cast<const unsigned long long*>(bits + c0));
    } else {
        for (int k = 0; k < 4; ++k)
            if (c0 + k < n_chunks) m |= static_cast<uint64_t>(bits[c0 + k]) << (16 * k);
    }
    const uint32_t own = __popcll(m);
    uint32_t incl = own;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    uint64_t k = tile_base[blockIdx.x] + incl - own;
    for (int w = 0; w < warp; ++w) k += part[w];
    const uint64_t first = c0 * CHUNK - lead;  // buffer position of bit 0
    for (; m && k < nl_cap; m &= m - 1) nl[k++] = static_cast<uint32_t>(first + __ffsll(static_cast<long long>(m)) - 1);
}

// st[0] lines, [1] records, [2] bytes consumed, [3] error (0, or 1/2/3 for a
// record missing its SEQ / + / QUAL line), [4] newlines, [5] max SEQ length
// (more than nl_cap newlines: no records yet, the host repeats the passes)
__global__ void fq_lines_kernel(const uint8_t* buf, uint64_t n, int at_eof, uint64_t max_records, int rules,
                                const uint32_t* nl, uint64_t nl_cap, const uint32_t* tile_base, const uint32_t* counts,
                                uint64_t n_tiles, unsigned long long* st) {
    const uint64_t n_nl = n_tiles ? static_cast<uint64_t>(tile_base[n_tiles - 1]) + counts[n_tiles - 1] : 0;
    if (n_nl > nl_cap) {
        st[0] = st[1] = st[2] = st[3] = st[5] = 0;
        st[4] = n_nl;
        return;
    }
    const uint64_t rest = n_nl ? static_cast<uint64_t>(nl[n_nl - 1]) + 1 : 0;
    uint64_t lines = n_nl;
    if (at_eof && rest < n) {
        if (rules == 1) {
            ++lines;  // readline() returns any non-empty rest
        } else {      // the rest counts when not empty after the '\r' strip
            uint64_t e = n;
            if (buf[e - 1] == 13) --e;
            if (e > rest) ++lines;
        }
    }
    // rules 1 at the end of the stream: a header line starts a record, its
    // missing lines read as empty
    const uint64_t whole = (rules == 1 && at_eof) ? (lines + 3) / 4 : lines / 4;
    const uint64_t recs = whole < max_records ? whole : max_records;
    st[0] = lines;
    st[1] = recs;
    // the reference reads one record past the complete ones only while it
    // still wants records
    st[3] = (rules == 0 && at_eof && max_records > whole && (lines & 3)) ? (lines & 3) : 0;
    uint64_t consumed = 0;
    if (recs) {
        const uint64_t last = 4 * recs - 1;  // index of the last QUAL line
        consumed = last < n_nl ? static_cast<uint64_t>(nl[last]) + 1 : n;
    }
    st[2] = consumed;
    st[4] = n_nl;
    st[5] = 0;
}

// 0x80 in exactly the byte lanes of w that hold c.
__device__ __forceinline__ uint64_t bytes_equal(uint64_t w, uint8_t c) {
    const uint64_t x = w ^ (0x0101010101010101ull * c);
    return ~(((x & 0x7f7f7f7f7f7f7f7full) + 0x7f7f7f7f7f7f7f7full) | x | 0x7f7f7f7f7f7f7f7full);
}

// First ' ' or '/' in buf[a, b), or b: aligned 8-byte words that hold a byte
// of the span, four loaded at once.
__device__ __forceinline__ uint64_t name_end(const uint8_t* buf, uint64_t a, uint64_t b) {
    if (a >= b) return b;
    const uintptr_t base = reinterpret_cast<uintptr_t>(buf), e = base + b;
    uintptr_t q = (base + a) & ~uintptr_t(7);
    uint64_t skip = ~0ull << (8 * ((base + a) & 7));  // bytes of the first word before a
    while (q < e) {
        uint64_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = q + 8 * k < e ? __ldg(reinterpret_cast<const unsigned long long*>(q + 8 * k)) : 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t m = (bytes_equal(w[k], 32) | bytes_equal(w[k], 47)) & skip;
            skip = ~0ull;
            if (m) {
                const uint64_t at = q + 8 * k + ((__ffsll(static_cast<long long>(m)) - 1) >> 3) - base;
                return at < b ? at : b;
            }
        }
        q += 32;
    }
    return b;
}

__global__ void fq_records_kernel(const uint8_t* buf, uint64_t n, uint64_t base, int rules, const uint32_t* nl,
                                  const unsigned long long* st, FastqRecordsDev out, unsigned long long* max_len) {
    const uint64_t r = static_cast<uint64_t>(blockIdx.x) * THREADS + threadIdx.x;
    uint32_t seq_len = 0;
    if (r < st[1]) {
        const uint64_t lines = st[0], n_nl = st[4];
        uint64_t s[4], e[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t li = 4 * r + k;
            if (li >= lines) {  // past the end of the stream (rules 1): empty
                s[k] = e[k] = n;
                continue;
            }
            s[k] = li ? static_cast<uint64_t>(nl[li - 1]) + 1 : 0;
            e[k] = li < n_nl ? nl[li] : n;
            if (rules == 1) {
                while (e[k] > s[k] && buf[e[k] - 1] == 13) --e[k];
            } else if (e[k] > s[k] && buf[e[k] - 1] == 13) {
                --e[k];
            }
        }
        uint64_t ns = s[0], ne = e[0];
        if (ne > ns && buf[ns] == 64) ++ns;
        ne = name_end(buf, ns, ne);
        out.name_off[r] = base + ns;
        out.name_len[r] = static_cast<uint32_t>(ne > ns ? ne - ns : 0);
        seq_len = static_cast<uint32_t>(e[1] - s[1]);
        out.seq_off[r] = base + s[1];
        out.seq_len[r] = seq_len;
        out.qual_off[r] = base + s[3];
        out.qual_len[r] = static_cast<uint32_t>(e[3] - s[3]);
    }
    for (int o = 16; o > 0; o >>= 1) seq_len = max(seq_len, __shfl_xor_sync(0xffffffffu, seq_len, o));
    if ((threadIdx.x & 31) == 0 && seq_len) atomicMax(max_len, static_cast<unsigned long long>(seq_len));
}

// Byte i of the rows is byte i % max_len of row i / max_len.  A thread makes
// the 16 bytes of one 16-byte block of the destination: for each row that the
// block touches (one or two, more for rows under 15 bytes) the five aligned
// words that cover the row's part, loaded where they hold a byte of the SEQ
// span, and 'N' past its end.  The thread that makes a row's first byte writes
// its length.
__global__ void __launch_bounds__(THREADS) fq_rows_kernel(const uint8_t* arena, const uint64_t* seq_off,
                                                         const uint32_t* seq_len, uint64_t total, uint32_t max_len,
                                                         uint8_t* rows, uint32_t* lens) {
    __shared__ uint64_t s_row0;
    const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(rows) & 15);
    const uint64_t blk = static_cast<uint64_t>(blockIdx.x) * THREADS * 16;  // first byte of this CTA, from rows - lead
    const uint64_t cta = blk > lead ? blk - lead : 0;
    if (threadIdx.x == 0) s_row0 = cta / max_len;
    __syncthreads();
    const uint64_t row0 = s_row0, at = blk + 16 * threadIdx.x;  // the block's first byte, from rows - lead
    const uint64_t lo = at > lead ? at - lead : 0, hi = min(at + 16 - lead, total);
    if (at + 16 <= lead || lo >= hi) return;
    const uint64_t p = lo - row0 * max_len;  // below 4096 + max_len
    uint32_t left = static_cast<uint32_t>(hi - lo), put = static_cast<uint32_t>(lo + lead - at);
    uint64_t o0 = 0, o1 = 0;
    uint32_t row = static_cast<uint32_t>(p >> 32 ? p / max_len : static_cast<uint32_t>(p) / max_len);
    uint32_t col = static_cast<uint32_t>(p - static_cast<uint64_t>(row) * max_len);
    while (left) {
        const uint32_t take = min(left, max_len - col);
        const uint64_t r = row0 + row;
        const uint32_t len = __ldg(seq_len + r);
        if (col == 0 && lens) lens[r] = len;
        const uint32_t real = col < len ? min(take, len - col) : 0;  // bases, then 'N'
        uint64_t v0 = 0x4e4e4e4e4e4e4e4eull, v1 = v0;
        if (real) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(arena) + __ldg(seq_off + r) + col;
            const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
            const uint32_t nw = (static_cast<uint32_t>(a & 3) + real + 3) >> 2, sh = static_cast<uint32_t>(a & 3) * 8;
            uint32_t x[5];
#pragma unroll
            for (uint32_t k = 0; k < 5; ++k) x[k] = k < nw ? __ldg(w + k) : 0;
            const uint64_t u0 = __funnelshift_r(x[0], x[1], sh) | static_cast<uint64_t>(__funnelshift_r(x[1], x[2], sh)) << 32;
            const uint64_t u1 = __funnelshift_r(x[2], x[3], sh) | static_cast<uint64_t>(__funnelshift_r(x[3], x[4], sh)) << 32;
            const uint64_t m0 = real >= 8 ? ~0ull : (1ull << (8 * real)) - 1;
            const uint64_t m1 = real >= 16 ? ~0ull : real > 8 ? (1ull << (8 * (real - 8))) - 1 : 0;
            v0 = (u0 & m0) | (v0 & ~m0);
            v1 = (u1 & m1) | (v1 & ~m1);
        }
        // to byte `put` of the block; what lies past `take` is overwritten or not stored
        const uint64_t k0 = put >= 8 ? ~0ull : (1ull << (8 * put)) - 1;             // bytes kept of o0
        const uint64_t k1 = put > 8 ? (1ull << (8 * (put - 8))) - 1 : 0;              // bytes kept of o1
        const uint32_t b = 8 * (put & 7);
        const uint64_t s0 = put >= 8 ? 0 : v0 << b;
        const uint64_t s1 = put >= 8 ? v0 << b : (b ? (v0 >> (64 - b)) | (v1 << b) : v1);
        o0 = (o0 & k0) | (s0 & ~k0);
        o1 = (o1 & k1) | (s1 & ~k1);
        put += take;
        left -= take;
        ++row;
        col = 0;
    }
    uint8_t* d = rows + (static_cast<int64_t>(at) - static_cast<int64_t>(lead));
    if (lo + lead == at && hi - lo == 16) {
        *reinterpret_cast<ulonglong2*>(d) = make_ulonglong2(o0, o1);
    } else {
        for (uint32_t k = static_cast<uint32_t>(lo + lead - at); k < static_cast<uint32_t>(hi + lead - at); ++k)
            d[k] = static_cast<uint8_t>((k < 8 ? o0 : o1) >> (8 * (k & 7)));
    }
}

uint64_t chunks_of(uint64_t n) { return n ? (n + 15) / CHUNK + 1 : 0; }  // enough for every alignment
uint64_t tiles_of(uint64_t n_chunks) { return (n_chunks + TILE_CHUNKS - 1) / TILE_CHUNKS; }

}  // namespace

size_t fastq_scratch_bytes(uint64_t n_bytes) {
    const uint64_t n_chunks = chunks_of(n_bytes), n_tiles = tiles_of(n_chunks);
    size_t t = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, t, static_cast<const uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                  static_cast<int64_t>(n_tiles ? n_tiles : 1));
    // newline bits, tile counts, tile bases, status, scan temp
    return align256(n_chunks * 2) + 2 * align256(n_tiles * 4) + 256 + align256(t);
}

int fastq_parse_enqueue(const uint8_t* buf, uint64_t n, int at_eof, uint64_t max_records, uint64_t base, int rules,
                        const FastqRecordsDev& out, void* scratch, size_t scratch_bytes,
                        void* (*newline_buffer)(void* user, size_t bytes), void* user, cudaStream_t st,
                        unsigned long long* h_status) {
    const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(buf) & 15);
    const uint64_t n_chunks = n ? (n + lead + CHUNK - 1) / CHUNK : 0, n_tiles = tiles_of(n_chunks);
    const uint64_t max_tiles = tiles_of(chunks_of(n));
    uint8_t* s = static_cast<uint8_t*>(scratch);
    uint16_t* bits = reinterpret_cast<uint16_t*>(s);
    s += align256(chunks_of(n) * 2);
    uint32_t* counts = reinterpret_cast<uint32_t*>(s);
    s += align256(max_tiles * 4);
    uint32_t* tile_base = reinterpret_cast<uint32_t*>(s);
    s += align256(max_tiles * 4);
    unsigned long long* status = reinterpret_cast<unsigned long long*>(s);
    s += 256;
    void* temp = s;
    size_t tb = scratch_bytes - static_cast<size_t>(s - static_cast<uint8_t*>(scratch));
    int launches = 0;
    if (n_tiles) {
        nl_count_kernel<<<static_cast<unsigned>(n_tiles), THREADS, 0, st>>>(buf, n, n_chunks, bits, counts);
        check_launch(cudaGetLastError(), "nl_count_kernel");
        check_launch(cub::DeviceScan::ExclusiveSum(temp, tb, static_cast<const uint32_t*>(counts), tile_base,
                                                   static_cast<int64_t>(n_tiles), st),
                     "newline scan");
        launches += 3;
    }
    uint64_t nl_cap = n / NL_BYTES + 1024;
    unsigned long long head[6];
    for (;;) {
        uint32_t* nl = static_cast<uint32_t*>(newline_buffer(user, nl_cap * 4));
        if (n_tiles) {
            nl_write_kernel<<<static_cast<unsigned>(n_tiles), THREADS, 0, st>>>(lead, n_chunks, bits, tile_base, nl, nl_cap);
            check_launch(cudaGetLastError(), "nl_write_kernel");
            ++launches;
        }
        fq_lines_kernel<<<1, 1, 0, st>>>(buf, n, at_eof, max_records, rules, nl, nl_cap, tile_base, counts, n_tiles, status);
        check_launch(cudaGetLastError(), "fq_lines_kernel");
        ++launches;
        // at most a record per four lines, the last of them unterminated
        const uint64_t most = nl_cap / 4 + 1 < max_records ? nl_cap / 4 + 1 : max_records;
        if (most) {
            fq_records_kernel<<<static_cast<unsigned>((most + THREADS - 1) / THREADS), THREADS, 0, st>>>(
                buf, n, base, rules, nl, status, out, status + 5);
            check_launch(cudaGetLastError(), "fq_records_kernel");
            ++launches;
        }
        check_launch(cudaMemcpyAsync(head, status, sizeof(head), cudaMemcpyDeviceToHost, st), "D2H parse status");
        check_launch(cudaStreamSynchronize(st), "fastq records");
        if (head[4] <= nl_cap) break;
        nl_cap = head[4];
    }
    for (int i = 0; i < 6; ++i) h_status[i] = head[i];
    return launches;
}

int fastq_rows_enqueue(const uint8_t* arena, const uint64_t* seq_off, const uint32_t* seq_len, uint64_t n_seq,
                       uint32_t max_len, uint8_t* rows, uint32_t* lens, cudaStream_t st) {
    if (!n_seq) return 0;
    if (!max_len) {
        if (lens) check_launch(cudaMemcpyAsync(lens, seq_len, n_seq * 4, cudaMemcpyDeviceToDevice, st), "D2D lengths");
        return 0;
    }
    const uint64_t total = n_seq * max_len;
    const uint64_t blocks = ((reinterpret_cast<uintptr_t>(rows) & 15) + total + 15) / 16;
    const unsigned g = static_cast<unsigned>((blocks + THREADS - 1) / THREADS);
    fq_rows_kernel<<<g, THREADS, 0, st>>>(arena, seq_off, seq_len, total, max_len, rows, lens);
    check_launch(cudaGetLastError(), "fq_rows_kernel");
    return 1;
}

}  // namespace ma
