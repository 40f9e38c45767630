"""BGZF members inflated on the device (ma_bgzf_inflate[_device]) against the
gzip module: the same bytes for every level, and the member-level errors
(size, CRC-32, damaged deflate data) the host-run member step reports."""
from __future__ import annotations

import ctypes as C
import gzip

import numpy as np
import pytest

from fastq_cases import random_fastq
from mojoalign_b200 import GpuContext, MojoAlignError, _lib
from mojoalign_b200.fqio import bgzf_inflate, bgzf_members
from oracle import bgzf_ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = GpuContext(0)
    yield c
    c.close()


@pytest.mark.parametrize("level", [0, 1, 6, 9])
def test_inflate_matches_gzip(ctx, level):
    text = random_fastq(21 + level, 20_000, crlf=0.2)
    blob = bgzf_ref.compress(text, level)
    assert bgzf_inflate(ctx, blob) == gzip.decompress(blob) == text


def test_empty_and_single_member(ctx):
    assert bgzf_inflate(ctx, bgzf_ref.compress(b"", 1)) == b""
    assert bgzf_inflate(ctx, bgzf_ref.compress(b"@r\nACGT\n+\nIIII\n", 6, eof=False)) == b"@r\nACGT\n+\nIIII\n"


def test_bad_members_are_reported(ctx):
    text = random_fastq(30, 3000)
    blob = bgzf_ref.compress(text, 1)
    t = bgzf_members(blob)
    bad = bytearray(blob)
    # the CRC-32 of member 1 (4 bytes before its ISIZE)
    end1 = int(t["src_off"][1] + t["src_len"][1])
    bad[end1] ^= 0xFF
    with pytest.raises(MojoAlignError, match="BGZF member 1: CRC-32 mismatch"):
        bgzf_inflate(ctx, bytes(bad))


def test_device_form_status(ctx):
    import torch

    text = random_fastq(31, 5000)
    blob = bgzf_ref.compress(text, 1)
    t = bgzf_members(blob)
    dev = torch.device("cuda", 0)

    def put(a):
        a = np.ascontiguousarray(a)
        sg = {np.dtype(np.uint64): np.int64, np.dtype(np.uint32): np.int32}
        return torch.from_numpy(a.view(sg.get(a.dtype, a.dtype)).copy()).to(dev)

    d_in = put(np.frombuffer(blob, np.uint8))
    cols = {k: put(t[k]) for k in ("src_off", "src_len", "dst_off", "isize", "crc")}
    cols["crc"][2] += 1  # member 2 fails its check, the others inflate
    n = int(t["src_off"].size)
    d_out = torch.zeros(t["out_bytes"] + 8, dtype=torch.uint8, device=dev)
    d_status = torch.zeros(n, dtype=torch.int32, device=dev)
    torch.cuda.synchronize()
    _lib.check(_lib.lib.ma_bgzf_inflate_device(ctx.handle, d_in.data_ptr(), len(blob),
                                               *[cols[k].data_ptr() for k in ("src_off", "src_len", "dst_off",
                                                                              "isize", "crc")],
                                               n, d_out.data_ptr(), t["out_bytes"], d_status.data_ptr(), None),
               ctx.handle)
    torch.cuda.synchronize()
    status = d_status.cpu().numpy()
    assert status[2] == 9 and not np.delete(status, 2).any()
    out = d_out.cpu().numpy().tobytes()
    assert out[:t["out_bytes"]] == text and not any(out[t["out_bytes"]:])


def _payloads():
    """(name, raw deflate stream, its bytes) over block kinds, code shapes and
    sizes around the kernel's: 4 bytes, 130 per thread, strips of 2048, a
    member of 65280, streams of several blocks and of several rounds."""
    import zlib

    def raw(data, level=6, strategy=zlib.Z_DEFAULT_STRATEGY, mem=8, flush_every=0, mode=zlib.Z_FULL_FLUSH):
        c = zlib.compressobj(level, zlib.DEFLATED, -15, mem, strategy)
        out = b""
        if flush_every:
            for a in range(0, len(data), flush_every):
                out += c.compress(data[a:a + flush_every]) + c.flush(mode)
        else:
            out = c.compress(data)
        return out + c.flush()

    rng = np.random.default_rng(5)
    text = random_fastq(9, 1500, crlf=0.1)
    noise = rng.integers(0, 256, 70_000, dtype=np.uint8).tobytes()
    skewed = rng.choice(256, 70_000, p=np.r_[np.full(1, .9), np.full(255, .1 / 255)]).astype(np.uint8).tobytes()
    # Fibonacci-like counts: codes up to 15 bits
    deep = b"".join(bytes([k]) * int(1.6 ** k) for k in range(1, 23))[:65280]
    deep = bytes(np.random.default_rng(6).permutation(np.frombuffer(deep, np.uint8)))
    for n in (0, 1, 3, 4, 5, 129, 130, 131, 2047, 2048, 2049, 65279, 65280, 65281, 65536):
        yield f"text{n}", raw(text[:n]), text[:n]
        yield f"noise{n}", raw(noise[:n], 9), noise[:n]
    for level in (0, 1, 9):
        yield f"level{level}", raw(text[:65280], level), text[:65280]
    for name, st in (("fixed", zlib.Z_FIXED), ("huffman", zlib.Z_HUFFMAN_ONLY), ("rle", zlib.Z_RLE), ("filtered", zlib.Z_FILTERED)):
        for kind, data in (("text", text[:65280]), ("skewed", skewed[:65280]), ("deep", deep), ("noise", noise[:65280])):
            yield f"{name}_{kind}", raw(data, 6, st), data
    for n in (1, 2, 3, 258, 259, 300, 65280):
        yield f"run{n}", raw(b"F" * n), b"F" * n
        yield f"period{n}", raw((b"ACGTTGCAG" * 8000)[:n], 9), (b"ACGTTGCAG" * 8000)[:n]
    yield "small_blocks", raw(text[:60000], 6, mem=1), text[:60000]
    for every in (37, 700, 5000, 30000):
        yield f"flush{every}", raw(text[:65280], 6, flush_every=every), text[:65280]
    yield "sync_flush", raw(text[:20000], 1, flush_every=1500, mode=zlib.Z_SYNC_FLUSH), text[:20000]
    yield "trailing", raw(text[:3000]) + b"rest", text[:3000]


def _inflate_raw(ctx, members, lead=0, gap=0):
    """members: (payload, isize, crc) -> statuses and the output buffer's bytes per member."""
    import torch

    src, so, sl, do, at = bytearray(b"\0" * 5), [], [], [], lead
    for p, n, _ in members:
        so.append(len(src))
        sl.append(len(p))
        src += p + b"\xff" * 3
        do.append(at)
        at += n + gap
    dev = torch.device("cuda", 0)
    put = lambda v, t: torch.from_numpy(np.array(v, t).view(np.int64 if t == np.uint64 else np.int32)).to(dev)  # noqa: E731
    d_in = torch.frombuffer(src, dtype=torch.uint8).to(dev)
    d_out = torch.full((at + 64,), 7, dtype=torch.uint8, device=dev)
    status = torch.full((len(members),), 77, dtype=torch.int32, device=dev)
    cols = [put(so, np.uint64), put(sl, np.uint32), put(do, np.uint64), put([n for _, n, _ in members], np.uint32),
            put([c for _, _, c in members], np.uint32)]
    torch.cuda.synchronize()
    _lib.check(_lib.lib.ma_bgzf_inflate_device(ctx.handle, d_in.data_ptr(), len(src), *[c.data_ptr() for c in cols],
                                               len(members), d_out.data_ptr(), at, status.data_ptr(), None), ctx.handle)
    torch.cuda.synchronize()
    out = d_out.cpu().numpy()
    assert (out[:lead] == 7).all() and (out[at:] == 7).all()
    return status.cpu().numpy(), [out[d:d + n].tobytes() for d, (_, n, _) in zip(do, members)], out, do


@pytest.mark.parametrize("lead,gap", [(0, 0), (1, 0), (2, 3), (3, 1)])
def test_every_block_kind_and_size(ctx, lead, gap):
    import zlib

    cases = list(_payloads())
    status, got, out, do = _inflate_raw(ctx, [(p, len(d), zlib.crc32(d)) for _, p, d in cases], lead, gap)
    for (name, _, data), s, g, at in zip(cases, status, got, do):
        assert s == 0 and g == data, name
        assert (out[at + len(data):at + len(data) + gap] == 7).all(), name


def test_damaged_members_end_as_on_the_host(ctx, tmp_path_factory):
    """Truncated, altered and mislabelled members: the status is that of the
    host-run decoder, or the size or CRC-32 check's."""
    import zlib

    from test_inflate import _build, inflate

    host = _build(tmp_path_factory, "libinflate_gpu.so", ["-O2"])
    rng = np.random.default_rng(8)
    members, want = [], []
    for name, p, data in _payloads():
        if len(data) < 100 or len(data) > 65280:
            continue
        crc = zlib.crc32(data)
        made = [(p[:int(rng.integers(0, len(p)))], len(data), crc), (p, len(data) + 1, crc), (p, len(data) - 1, crc),
                (p, len(data), crc ^ 1)]
        for _ in range(4):
            q = bytearray(p)
            for at in rng.integers(0, len(p) if rng.random() < .5 else min(len(p), 90), int(rng.integers(1, 3))):
                q[at] ^= 1 << int(rng.integers(0, 8))
            made.append((bytes(q), len(data), crc))
        for q, n, c in made:
            rc, b = inflate(host, q, n)
            members.append((q, n, c))
            want.append(rc if rc else 8 if len(b) != n else 0 if zlib.crc32(b) == c else 9)
    status, _, _, _ = _inflate_raw(ctx, members)
    np.testing.assert_array_equal(status, want)


@pytest.mark.parametrize("symbols", [1, 2, 3, 5, 16, 64, 65, 200, 256])
def test_literals_in_pairs(ctx, symbols):
    """Members of literals alone, of 1 to 15 bits: pairs that fill the table's
    bits or just miss them, that straddle a segment's end, a word of the start
    marks and the member's last byte."""
    import zlib

    rng = np.random.default_rng(symbols)
    cases = []
    for n in (4, 5, 31, 32, 33, 64, 65, 2047, 30_001, 65_279, 65_280):
        for p in (np.full(symbols, 1 / symbols), np.geomspace(1, 1e-4, symbols)):
            data = rng.choice(symbols, n, p=p / p.sum()).astype(np.uint8).tobytes()
            c = zlib.compressobj(6, zlib.DEFLATED, -15, 8, zlib.Z_HUFFMAN_ONLY)
            cases.append((c.compress(data) + c.flush(), data))
    status, got, _, _ = _inflate_raw(ctx, [(p, len(d), zlib.crc32(d)) for p, d in cases])
    for i, ((_, data), s, g) in enumerate(zip(cases, status, got)):
        assert s == 0 and g == data, i


def _members(kind):
    """One to eight deflate payloads of a kind of member and their bytes."""
    import base64
    import zlib

    rng = np.random.default_rng(12)
    text = random_fastq(13, 6000)
    noise = rng.integers(0, 256, 8 * 65280, dtype=np.uint8).tobytes()
    size, data, level, strategy = {
        "small": (512, text, 6, zlib.Z_DEFAULT_STRATEGY), "whole": (65536, text, 6, zlib.Z_DEFAULT_STRATEGY),
        "zeros": (65280, bytes(65280), 6, zlib.Z_DEFAULT_STRATEGY), "stored": (4096, noise, 0, zlib.Z_DEFAULT_STRATEGY),
        "fixed": (65280, text, 6, zlib.Z_FIXED), "base64": (65280, base64.b64encode(noise), 6, zlib.Z_HUFFMAN_ONLY)}[kind]
    made = []
    for a in range(0, min(len(data), 8 * size) - size + 1, size):
        c = zlib.compressobj(level, zlib.DEFLATED, -15, 8, strategy)
        made.append((c.compress(data[a:a + size]) + c.flush(), data[a:a + size]))
    return made


@pytest.mark.parametrize("kind,many,most", [("whole", 2368, 4), ("small", 2368, 4.5), ("stored", 8000, 10),
                                            ("zeros", 2368, 8), ("fixed", 2368, 11), ("base64", 2368, 8)])
def test_many_members_of_any_kind_run_side_by_side(ctx, kind, many, most):
    """Members that a CTA does not hold, that it is slow at, or that are mostly
    its own overhead: a call of 16 members an SM (54 stored ones) takes at most
    `most` times one of a member an SM, 16 (54) times where each had an SM to
    itself.  The measured factors are 1.4, 2.3, 5.5, 4.8, 7 and 4.6."""
    import torch
    import zlib

    made = _members(kind)
    took = []
    for n in (148, many):
        src, so, sl = bytearray(), [], []
        for p, _ in made:
            so.append(len(src))
            sl.append(len(p))
            src += p
        i = np.arange(n) % len(made)
        size = len(made[0][1])
        put = lambda v, t: torch.from_numpy(np.asarray(v).astype(t)).cuda()  # noqa: E731
        cols = [put(np.array(so)[i], np.int64), put(np.array(sl)[i], np.int32), put(np.arange(n) * size, np.int64),
                put(np.full(n, size), np.int32),
                put(np.array([zlib.crc32(d) for _, d in made], np.uint32).view(np.int32)[i], np.int32)]
        d_in = torch.frombuffer(src, dtype=torch.uint8).cuda()
        d_out = torch.zeros(n * size, dtype=torch.uint8, device="cuda")
        status = torch.full((n,), 77, dtype=torch.int32, device="cuda")
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            _lib.check(_lib.lib.ma_bgzf_inflate_device(ctx.handle, d_in.data_ptr(), len(src),
                                                       *[c.data_ptr() for c in cols], n, d_out.data_ptr(), n * size,
                                                       status.data_ptr(), stream.cuda_stream), ctx.handle)
            b.record(stream)
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        took.append(float(np.median(times[2:])))
        assert not status.any()
        want = torch.frombuffer(bytearray(b"".join(d for _, d in made)), dtype=torch.uint8).cuda()
        whole = n // len(made) * len(made) * size
        assert torch.equal(d_out[:whole].view(-1, want.numel()), want.expand(whole // want.numel(), -1))
        assert torch.equal(d_out[whole:], want[:n * size - whole])
    assert took[1] < most * took[0], took


def _fixed_block(data, last):
    """Bits of a block of literals in the fixed codes, first bit first."""
    bits = [last, 1, 0]
    for x in data:
        code, n = (0x30 + x, 8) if x < 144 else (0x190 + x - 144, 9)
        bits += [code >> (n - 1 - k) & 1 for k in range(n)]
    return bits + [0] * 7


def test_edges_of_segments_strips_and_rounds(ctx):
    """Members that end around a thread's 66 bytes of the CRC, around strips of
    3968 bytes and around the 992 * 224 bits that the threads read at once;
    copies and runs across a strip's edge."""
    import zlib

    text = random_fastq(14, 400)
    cases = []

    def add(data, level=9):
        c = zlib.compressobj(level, zlib.DEFLATED, -15)
        cases.append((c.compress(data) + c.flush(), data))

    for n in (65, 66, 67, 131, 132, 133, 3967, 3968, 3969, 7935, 7936, 7937, 65279):
        add(text[:n])
    for at in (3900, 3960, 3965, 3967, 3968, 3969):
        for run in (b"F" * 300, b"ACG" * 120, text[:257], text[at - 5:at] * 60):
            add(text[:at] + run + text[:50])
    # 27776 codes of 8 bits fill the 992 segments: the end-of-block code before,
    # up to and past their end, then another block
    for a, b in ((27775, 0), (27774, 1), (27773, 2), (27776, 0), (27770, 4), (27777, 0)):
        data = bytes([65 + k % 50 for k in range(a)]) + bytes([200] * b)
        bits = _fixed_block(data, 0) + _fixed_block(text[:100], 1)
        cases.append((np.packbits(np.array(bits, np.uint8), bitorder="little").tobytes(), data + text[:100]))
    for p, d in cases:
        assert zlib.decompress(p, -15) == d
    for lead in (0, 1):
        status, got, _, _ = _inflate_raw(ctx, [(p, len(d), zlib.crc32(d)) for p, d in cases], lead)
        for i, ((_, d), s, g) in enumerate(zip(cases, status, got)):
            assert s == 0 and g == d, i


@pytest.mark.parametrize("last", [300, 600, 1500])
def test_a_small_last_member_costs_nothing(ctx, last):
    """The member that ends a file is decoded beside the others of its CTA, not
    by a warp after all of them (0.2 to 0.4 ms on top of 2.3)."""
    import torch
    import zlib

    text = random_fastq(13, 6000)
    pieces = [text[a * 65280:(a + 1) * 65280] for a in range(8)] + [text[:last]]
    src, so, sl = bytearray(), [], []
    for p in pieces:
        c = zlib.compressobj(6, zlib.DEFLATED, -15)
        d = c.compress(p) + c.flush()
        so.append(len(src))
        sl.append(len(d))
        src += d
    crc = np.array([zlib.crc32(p) for p in pieces], np.uint32).view(np.int32)
    d_in = torch.frombuffer(src, dtype=torch.uint8).cuda()
    took = []
    for n in (1036, 1037):
        i = np.arange(n) % 8
        i[1036:] = 8
        size = np.array([len(p) for p in pieces])[i]
        put = lambda v, t: torch.from_numpy(np.asarray(v).astype(t)).cuda()  # noqa: E731
        cols = [put(np.array(so)[i], np.int64), put(np.array(sl)[i], np.int32), put(np.cumsum(size) - size, np.int64),
                put(size, np.int32), put(crc[i], np.int32)]
        d_out = torch.zeros(int(size.sum()), dtype=torch.uint8, device="cuda")
        status = torch.full((n,), 77, dtype=torch.int32, device="cuda")
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        times = []
        for _ in range(13):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            _lib.check(_lib.lib.ma_bgzf_inflate_device(ctx.handle, d_in.data_ptr(), len(src),
                                                       *[c.data_ptr() for c in cols], n, d_out.data_ptr(),
                                                       d_out.numel(), status.data_ptr(), stream.cuda_stream),
                       ctx.handle)
            b.record(stream)
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        took.append(float(np.median(times[3:])))
        assert not status.any()
        assert d_out[-last if n > 1036 else -65280:].cpu().numpy().tobytes() == pieces[i[-1]]
    assert took[1] < 1.05 * took[0], took
