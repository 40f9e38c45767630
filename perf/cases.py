"""The work that is timed: calls of the framework's public entry points on
synthetic bisulfite sequencing data of the sizes and mixes its users bring.

A case is a plain dict; `kind` says which path it takes:

  map_host     map_batch on host arrays, the reference's batch step
  map_device   map_batch_device on reads that are already in HBM
  serve        a burst of requests of uneven sizes through the served form
  fastq_split  FASTQ bytes in HBM to records and mapper rows
  bam_pack     BAM records of a mapped batch
  sam_emit     SAM lines of a mapped batch
  sort_gather  coordinate sort, duplicate marking and the sorted record stream
  bgzf         a BAM record stream to BGZF members
  inflate      BGZF members (as bgzip writes them) to FASTQ bytes
  fastq_to_bam FASTQ files to a sorted, duplicate-marked BAM file

Everything is drawn on a 250 Mbp reference in 24 contigs, 45% of it in repeat
copies (the repeat-heavy model of the synthetic references): the chromosome
size of the benchmark with the repeat content of a genome.  The reference and
its resident index are what a program opens once and keeps; the reads, the
qualities, the hits and the duplicates come from the seed.

Every output is whole numbers or bytes.
"""
import math
import os
import shutil
import sys
import tempfile
import zlib
from concurrent.futures import ThreadPoolExecutor
from ctypes import byref, c_uint64
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "mojo-align_b200"))

from mojoalign_b200 import BENCH_PARAMS, GpuContext, GpuIndex, MapResult, build_index, map_batch, map_batch_device, synth  # noqa: E402
from mojoalign_b200._lib import check, lib, ma_fastq_arena, ma_fastq_records, ma_hits  # noqa: E402
from mojoalign_b200.bam import META_FIELDS, BamTile, canonical_rid_to_tid, emit_bam_device  # noqa: E402
from mojoalign_b200.fq2bam import map_fastq_to_bam  # noqa: E402
from mojoalign_b200.sam import SamContigs, emit_sam_device  # noqa: E402
from mojoalign_b200.serve import Server  # noqa: E402

GENOME = 250_000_000
CONTIGS = 24
RG = b"mojo1"
NAMES = [s + "chr%d" % (i + 1) for i in range(CONTIGS) for s in ("r", "f")]  # the index's contig order
# the form the autotuner picks for large uneven batches (see bench.py)
BATCHED = dict(seed_kernel=4, stage1_endpoints=2, reg_level=1, wave_endpoints=8, wave_loci_per_read=32)


def listed():
    return [
        # a request of a few pairs: copies, launches and synchronisations
        {"name": "map_host_32_pairs", "kind": "map_host", "n1": 32, "paired": True, "read_len": 150},
        # the reference's batch of 16384 pairs, as its mapper fires it
        {"name": "map_host_16k_pairs", "kind": "map_host", "n1": 16384, "paired": True, "read_len": 150},
        # the batched form of the benchmark: uneven single-end reads from both
        # directional and non-directional strands, the autotuned kernel form,
        # the call repeated on kept buffers (CUDA graphs on)
        {"name": "map_device_uneven_2m", "kind": "map_device", "n1": 2_000_000, "paired": False, "read_len": 0, "batched": True},
        # long pairs in the default kernel form, as the file pipelines map them
        {"name": "map_device_400k_2x250", "kind": "map_device", "n1": 400_000, "paired": True, "read_len": 250, "batched": False},
        # requests of several samples arriving at once at a running server
        {"name": "serve_burst_32", "kind": "serve", "requests": 32, "smallest": 1_000, "largest": 64_000},
        # one piece of a FASTQ file, split and laid out for the mapper
        {"name": "fastq_split_1m", "kind": "fastq_split", "records": 1_000_000, "read_len": 150, "rules": 0},
        # one mapped batch of the BAM path, and of the SAM path
        {"name": "bam_pack_500k_pairs", "kind": "bam_pack", "n1": 500_000, "paired": True, "read_len": 150},
        {"name": "sam_emit_500k_pairs", "kind": "sam_emit", "n1": 500_000, "paired": True, "read_len": 150},
        # the end of the BAM path: a tile of 4 M records
        {"name": "sort_gather_4m", "kind": "sort_gather", "n1": 2_000_000, "paired": True, "read_len": 100},
        # the file's compression at the default level
        {"name": "bgzf_256mb_level1", "kind": "bgzf", "bytes": 256_000_000, "level": 1},
        # a bgzipped FASTQ piece, inflated behind the copy of its members
        {"name": "inflate_128mb", "kind": "inflate", "bytes": 128_000_000},
        # a small sequencing run, files in and file out
        {"name": "fastq_to_bam_100k_pairs", "kind": "fastq_to_bam", "n1": 100_000, "read_len": 150},
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["map_host", "map_device", "serve", "fastq_split", "bam_pack", "sam_emit", "sort_gather", "bgzf", "inflate", "fastq_to_bam"])
    length = rng.randint(75, 251)
    paired = rng.random() < 0.6
    if kind == "map_host":
        return {"kind": kind, "n1": _log(rng, 8, 65_536), "paired": paired, "read_len": length}
    if kind == "map_device":
        uneven = rng.random() < 0.5
        return {"kind": kind, "n1": _log(rng, 20_000, 800_000), "paired": paired and not uneven, "read_len": 0 if uneven else length, "batched": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(4, 32), "smallest": _log(rng, 100, 2_000), "largest": _log(rng, 4_000, 64_000)}
    if kind == "fastq_split":
        return {"kind": kind, "records": _log(rng, 1_000, 1_000_000), "read_len": length if rng.random() < 0.6 else 0, "rules": rng.randint(0, 1)}
    if kind in ("bam_pack", "sam_emit"):
        return {"kind": kind, "n1": _log(rng, 1_000, 500_000), "paired": paired, "read_len": length}
    if kind == "sort_gather":
        return {"kind": kind, "n1": _log(rng, 5_000, 2_000_000), "paired": paired, "read_len": rng.randint(75, 101)}
    if kind == "bgzf":
        return {"kind": kind, "bytes": _log(rng, 200_000, 256_000_000), "level": rng.choice([0, 1, 1, 1, 6])}
    if kind == "inflate":
        return {"kind": kind, "bytes": _log(rng, 200_000, 128_000_000)}
    return {"kind": kind, "n1": _log(rng, 1_000, 100_000), "read_len": length}


# ---- what a program opens once ------------------------------------------


@lru_cache(maxsize=None)
def _stream():
    return torch.cuda.Stream()


@lru_cache(maxsize=None)
def _context():
    return GpuContext(torch.cuda.current_device())


def _tuned(batched):
    """The context with the batched form's tuning and graphs, or as it is made."""
    ctx = _context()
    ctx.set_tuning(**(BATCHED if batched else {}))
    ctx.set_graphs(batched)
    return ctx


def _write_reference(folder):
    fa = Path(folder) / "ref.fa"
    synth.write_reference_model(fa, GENOME, n_contigs=CONTIGS, seed=0, repeats=synth.RepeatModel())
    return fa


@lru_cache(maxsize=None)
def _genome():
    """The reference's bases (A, C, G, T = 0..3) in HBM and its contigs' starts."""
    with tempfile.TemporaryDirectory() as folder:
        text = torch.from_numpy(np.fromfile(_write_reference(folder), np.uint8)).cuda()
    newline = torch.cat([text.new_zeros(1, dtype=torch.int64) - 1, torch.nonzero(text == 10).flatten()])
    headers = torch.nonzero(text == ord(">")).flatten()
    ends = newline[torch.searchsorted(newline, headers)]
    starts, keep = [], text != 10
    for a, b in zip(headers.tolist(), ends.tolist()):
        keep[a:b] = False
        starts.append(a)
    at = torch.cumsum(keep, 0)
    starts = torch.tensor([int(at[a]) for a in starts], device="cuda")
    code = torch.zeros(256, dtype=torch.uint8, device="cuda")
    code[torch.tensor(list(b"ACGTacgt"), device="cuda")] = torch.tensor([0, 1, 2, 3] * 2, dtype=torch.uint8, device="cuda")
    return code[text[keep].int()], starts


@lru_cache(maxsize=None)
def _index():
    """The bwa-meth index of the reference, resident with the benchmark's tables."""
    folder = tempfile.mkdtemp()
    try:
        fa = _write_reference(folder)
        prefix = str(fa) + ".bwameth.c2t"
        build_index(fa, prefix, bwameth_c2t=True, sa_intv=32, device=torch.cuda.current_device())
        return GpuIndex(_context(), prefix, kmer_k=12, kmer3_k=19, at_k=28, at_seed_len=BENCH_PARAMS.seed_len)
    finally:
        shutil.rmtree(folder)


@lru_cache(maxsize=None)
def _server():
    return Server(_context(), _index(), hbm_budget_bytes=2 << 30)


# ---- synthetic reads ------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _below(g, hi, *shape):
    return torch.randint(0, hi, shape, generator=g, device="cuda")


class Reads:
    """n1 fragments sequenced as single reads or pairs: rows [n_seq][max_len]
    of ASCII (R1 rows, then R2 rows), padded with N, the lengths, and where
    each read lies.  read_len 0: lognormal lengths, 36 to 300.  Non-CpG bases
    are converted at 0.99, CpGs kept at 0.75, 0.5% substitutions, 5% random
    reads, every tenth fragment a duplicate of another; `both`: half of the
    reads from the strands that the directional protocol leaves out."""

    def __init__(self, g, n1, paired, read_len, both=False):
        self.n1, self.paired = n1, paired
        self.n_seq = n1 * (2 if paired else 1)
        if read_len:
            self.max_len = read_len
            self.lens = torch.full((self.n_seq,), read_len, device="cuda")
        else:
            self.max_len = 300
            normal = torch.randn(self.n_seq, generator=g, device="cuda")
            self.lens = (120 * torch.exp(0.35 * normal)).long().clamp(36, 300)
        frag = (350 + 50 * torch.randn(n1, generator=g, device="cuda")).long().clamp(min=300)
        start = _below(g, GENOME - 1200, n1) + 100
        bottom = _rand(g, n1) < 0.5
        copy = _rand(g, n1) < 0.1
        source = _below(g, n1, n1)
        for x in (frag, start, bottom):
            x[copy] = x[source[copy]]
        if not paired:
            frag = torch.maximum(frag, self.lens[:n1])
        far = torch.zeros(n1, dtype=torch.bool, device="cuda")
        if both:
            far = _rand(g, n1) < 0.5
        junk = _rand(g, n1) < 0.05
        self.start, self.frag, self.bottom, self.junk = start, frag, bottom, junk
        self.rows = torch.empty((self.n_seq, self.max_len), dtype=torch.uint8, device="cuda")
        for m in range(2 if paired else 1):
            for a in range(0, n1, 250_000):
                s = slice(a, min(n1, a + 250_000))
                second = torch.ones_like(far[s]) if m else far[s]
                self.rows[m * n1 + a:m * n1 + s.stop] = self._sequence(g, start[s], frag[s], bottom[s], second, junk[s], self.lens[m * n1 + a:m * n1 + s.stop])

    def _sequence(self, g, start, frag, bottom, second, junk, lens):
        genome, _ = _genome()
        n, w = start.numel(), self.max_len
        j = torch.arange(w, device="cuda").expand(n, w)
        # position in the converted fragment, 5' to 3' of its own strand
        p = torch.where(second[:, None], frag[:, None] - 1 - j, j)

        def base(p):
            x = genome[torch.where(bottom[:, None], start[:, None] + frag[:, None] - 1 - p, start[:, None] + p).clamp(0, GENOME - 1)]
            return torch.where(bottom[:, None], 3 - x, x)

        b = base(p)
        kept = _rand(g, n, w) < torch.where(base(p + 1) == 2, 0.75, 0.01)
        b = torch.where((b == 1) & ~kept, torch.full_like(b, 3), b)
        b = torch.where(second[:, None], 3 - b, b)
        b = torch.where(_rand(g, n, w) < 0.005, (b + 1 + _below(g, 3, n, w).byte()) % 4, b)
        b = torch.where(junk[:, None], _below(g, 4, n, w).byte(), b)
        letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")[b.int()]
        return torch.where(j < lens[:, None], letters, torch.full_like(letters, ord("N")))

    def hits(self, g):
        """The mapping outputs a run of the mapper would give: the drawn place
        of each read, a few of them clipped, random reads unmapped."""
        _, starts = _genome()
        n, m = self.n1, 2 if self.paired else 1
        contig = torch.searchsorted(starts, self.start, right=True) - 1
        left = self.start - starts[contig]
        out = {}
        pos, rev, un = [], [], []
        for k in range(m):
            right_end = (self.bottom if k == 0 else ~self.bottom)
            pos.append(torch.where(right_end, left + self.frag - self.lens[k * n:(k + 1) * n], left))
            rev.append(right_end)
            un.append(self.junk | (_rand(g, n) < 0.01))
        un = torch.cat(un)
        clip = lambda: torch.where(_rand(g, self.n_seq) < 0.03, _below(g, 19, self.n_seq) + 1, 0)  # noqa: E731
        out["sl"], out["sr"] = clip(), clip()
        out["rid"] = torch.where(un, -1, (2 * contig + (~self.bottom).long()).repeat(m))
        out["pos"] = torch.where(un, 0, torch.cat(pos) + out["sl"])
        out["flag"] = torch.where(un, 4, 16 * torch.cat(rev).long())
        out["mapq"] = torch.where(un, 0, torch.where(_rand(g, self.n_seq) < 0.85, 60, _below(g, 60, self.n_seq)))
        out["nm"] = torch.where(un, 0, (4 * _rand(g, self.n_seq) ** 4).long())
        return {f: out[f].int() for f in MapResult.FIELDS}


def _digits(x, width):
    """Decimal digits of x in `width` byte columns; 0 bytes in front."""
    p = 10 ** torch.arange(width - 1, -1, -1, device="cuda")
    d = (x[:, None] // p) % 10 + 48
    return torch.where((x[:, None] >= p) | (p == 1), d, 0).byte()


class Fastq:
    """The FASTQ text of reads (R1 records, then R2 records) in HBM and the
    byte offsets and lengths of every record's name, bases and qualities."""

    def __init__(self, g, reads):
        n = reads.n1
        lane, tile, x, y = 1 + _below(g, 4, n), 1101 + _below(g, 78, n), 1000 + _below(g, 31_000, n), 1000 + _below(g, 36_000, n)
        level = _rand(g, n)
        texts, self.cols = [], {}
        sizes = []
        for m in range(reads.n_seq // n):
            for a in range(0, n, 250_000):
                s = slice(a, min(n, a + 250_000))
                k = s.stop - a
                word = lambda t: torch.tensor(list(t), dtype=torch.uint8, device="cuda").expand(k, len(t))  # noqa: E731,B023
                name = torch.cat([word(b"A01182:77:HGV2DSX:"), _digits(lane[s], 1), word(b":"), _digits(tile[s], 4), word(b":"), _digits(x[s], 5), word(b":"),
                                  _digits(y[s], 5)], 1)
                note = word(b" %d:N:0:ACGTTGCA\n" % (m + 1))
                seq = reads.rows[m * n + a:m * n + s.stop]
                lens = reads.lens[m * n + a:m * n + s.stop]
                inside = torch.arange(reads.max_len, device="cuda") < lens[:, None]
                seq = torch.where(inside, seq, 0)
                # four quality bins; reads of a poor tile and read ends drop more often
                drop = _rand(g, k, reads.max_len) * (1.6 - 0.6 * level[s, None] - 0.4 * torch.arange(reads.max_len, device="cuda") / reads.max_len)
                bins = torch.tensor(list(b"#,:F"), dtype=torch.uint8, device="cuda")
                qual = bins[torch.bucketize(drop, torch.tensor([0.004, 0.02, 0.08], device="cuda"))]
                qual = torch.where(inside, qual, 0)
                record = torch.cat([word(b"@"), name, note, seq, word(b"\n+\n"), qual, word(b"\n")], 1)
                texts.append(record[record != 0])
                named = (name != 0).sum(1)
                sizes.append(torch.stack([named, lens, named + note.shape[1] + 2 * lens + 5], 1))
        sizes = torch.cat(sizes)
        self.text = torch.cat(texts)
        end = torch.cumsum(sizes[:, 2], 0)
        at = end - sizes[:, 2]
        note = len(b" 1:N:0:ACGTTGCA\n")
        self.cols["name_off"] = at + 1
        self.cols["orig_off"] = at + 1 + sizes[:, 0] + note
        self.cols["qual_off"] = end - 1 - sizes[:, 1]
        self.cols["name_len"] = sizes[:, 0].int()
        self.cols["orig_len"] = self.cols["qual_len"] = sizes[:, 1].int()
        self.first = int(end[n - 1])  # bytes of the R1 records

    def arena(self):
        return {"data": self.text.data_ptr(), **{k: v.data_ptr() for k, v in self.cols.items()}}


def _zeros(n, dtype):
    return torch.zeros(n, dtype=dtype, device="cuda")


def _pointers(tensors):
    return {k: v.data_ptr() for k, v in tensors.items()}


# ---- the cases --------------------------------------------------------------


class MapHost:
    def __init__(self, case, seed):
        g = _generator(seed)
        self.ctx, self.index = _tuned(False), _index()
        r = Reads(g, case["n1"], case["paired"], case["read_len"])
        self.n1, self.paired, self.max_len = r.n1, r.paired, r.max_len
        self.bases, self.lens = r.rows.cpu().numpy(), r.lens.cpu().numpy().astype(np.uint32)

    def run(self):
        r = map_batch(self.ctx, self.index, self.bases, self.lens, self.n1, self.paired, self.max_len, "C2T", "G2A", BENCH_PARAMS)
        return {f: getattr(r, f) for f in MapResult.FIELDS}

    @staticmethod
    def work(case):
        n, w = case["n1"] * (2 if case["paired"] else 1), case["read_len"] or 128
        # the rows and lengths, the outputs, and the text under each read
        return {"bytes": n * (w + 4 + 28 + w / 4), "flops": 0}


class MapDevice:
    def __init__(self, case, seed):
        g = _generator(seed)
        self.ctx, self.index = _tuned(case["batched"]), _index()
        r = Reads(g, case["n1"], case["paired"], case["read_len"], both=not case["paired"])
        self.n1, self.paired, self.max_len = r.n1, r.paired, r.max_len
        self.rows, self.lens = r.rows, r.lens.int()
        self.out = {f: _zeros(r.n_seq, torch.int32) for f in MapResult.FIELDS}

    def run(self):
        map_batch_device(self.ctx, self.index, self.rows.data_ptr(), self.lens.data_ptr(), self.n1, self.paired, self.max_len, _pointers(self.out), "C2T", "G2A",
                         BENCH_PARAMS, stream=_stream().cuda_stream)
        return self.out

    work = MapHost.work


class Serve:
    """Requests of log-uniform sizes from samples of several read lengths."""

    def __init__(self, case, seed):
        g = _generator(seed)
        self.server = _server()
        self.requests = []
        for k in range(case["requests"]):
            n, paired, length = self.size(case, k), k % 3 == 0, (100, 150, 0)[k % 3]
            r = Reads(g, n, paired, length)
            self.requests.append((r.rows.cpu().numpy(), r.lens.cpu().numpy().astype(np.uint32), n, paired, r.max_len))

    @staticmethod
    def size(case, k):
        step = (k * 7919 % case["requests"] + 0.5) / case["requests"]
        return int(case["smallest"] * (case["largest"] / case["smallest"]) ** step)

    def run(self):
        tickets = [self.server.submit(*r, "C2T", "G2A", BENCH_PARAMS) for r in self.requests]
        results = [self.server.wait(t) for t in tickets]
        return {f: np.concatenate([getattr(r, f) for r in results]) for f in MapResult.FIELDS}

    @staticmethod
    def work(case):
        parts = [MapHost.work({"n1": Serve.size(case, k), "paired": k % 3 == 0, "read_len": (100, 150, 0)[k % 3]}) for k in range(case["requests"])]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": 0}


class FastqSplit:
    KEYS = ("name_off", "name_len", "seq_off", "seq_len", "qual_off", "qual_len")

    def __init__(self, case, seed):
        g = _generator(seed)
        r = Reads(g, case["records"], False, case["read_len"])
        self.text = Fastq(g, r).text
        self.n, self.rules = r.n1, case["rules"]
        self.max_len = r.max_len
        self.records = {k: _zeros(self.n, torch.int64 if k.endswith("off") else torch.int32) for k in self.KEYS}
        self.rows, self.lens = _zeros(self.n * self.max_len, torch.uint8), _zeros(self.n, torch.int32)

    def run(self):
        ctx, stream, r = _context(), _stream().cuda_stream, self.records
        got = (c_uint64 * 3)()
        out = ma_fastq_records(*[r[k].data_ptr() for k in self.KEYS])
        check(lib.ma_fastq_parse_rules_device(ctx.handle, self.text.data_ptr(), self.text.numel(), 1, self.n, 0, self.rules, byref(out), got, stream), ctx.handle)
        check(lib.ma_fastq_rows_device(ctx.handle, self.text.data_ptr(), r["seq_off"].data_ptr(), r["seq_len"].data_ptr(), int(got[0]), self.max_len,
                                       self.rows.data_ptr(), self.lens.data_ptr(), stream), ctx.handle)
        return {**r, "rows": self.rows, "lens": self.lens, "taken": int(got[0]), "spanned": int(got[1]), "longest": int(got[2])}

    @staticmethod
    def work(case):
        w = case["read_len"] or 128
        return {"bytes": case["records"] * (58 + 2 * w + 36 + (case["read_len"] or 300) + 4), "flops": 0}


class Mapped:
    """A mapped batch: its FASTQ text, its hits and room for its records."""

    def __init__(self, case, g):
        r = Reads(g, case["n1"], case["paired"], case["read_len"])
        self.n1, self.n_seq, self.paired = r.n1, r.n_seq, r.paired
        self.hits = r.hits(g)
        self.fastq = Fastq(g, r)
        self.rg = torch.tensor(list(RG), dtype=torch.uint8, device="cuda")


class BamPack:
    def __init__(self, case, seed):
        g = _generator(seed)
        self.b = b = Mapped(case, g)
        self.tids = torch.from_numpy(canonical_rid_to_tid(NAMES)).cuda()
        self.cap = b.n_seq * (64 + len(RG) + 40 + 2 * case["read_len"])
        self.bam = _zeros(self.cap, torch.uint8)
        self.meta = {k: _zeros(b.n_seq, torch.int64 if t == np.uint64 else torch.int32) for k, t in META_FIELDS}
        self.status = _zeros(3, torch.int64)
        self.tile = BamTile(b.n_seq, host_meta=False)

    def run(self):
        b = self.b
        emit_bam_device(_context(), _pointers(b.hits), b.n1, b.paired, b.fastq.arena(), b.fastq.text.numel(), self.tids.data_ptr(), len(NAMES), b.rg.data_ptr(), len(RG),
                        self.bam.data_ptr(), self.cap, _pointers(self.meta), self.tile, self.status.data_ptr(), _stream().cuda_stream)
        return {"bam": self.bam, "status": self.status, **self.meta}

    @staticmethod
    def work(case):
        n, w = case["n1"] * (2 if case["paired"] else 1), case["read_len"]
        return {"bytes": n * (36 + 2 * w + 28 + 36 + 36 + 36 + 4 + 15 + 1.5 * w + 44), "flops": 0}


class SamEmit:
    def __init__(self, case, seed):
        g = _generator(seed)
        self.b = b = Mapped(case, g)
        self.contigs = SamContigs.from_names(NAMES).to_device(torch, "cuda")
        self.cap = b.n_seq * (128 + len(RG) + 16 + 40 + 2 * case["read_len"])
        self.sam = _zeros(self.cap, torch.uint8)
        self.status = _zeros(3, torch.int64)

    def run(self):
        b, a = self.b, self.b.fastq.arena()
        arena = ma_fastq_arena(a["data"], b.fastq.text.numel(), *[a[k] for k in ("name_off", "name_len", "orig_off", "orig_len", "qual_off", "qual_len")])
        hits = ma_hits(*[b.hits[f].data_ptr() for f in MapResult.FIELDS])
        emit_sam_device(_context(), hits, b.n1, b.paired, arena, self.contigs, b.rg.data_ptr(), len(RG), self.sam.data_ptr(), self.cap, self.status.data_ptr(),
                        _stream().cuda_stream)
        return {"sam": self.sam, "status": self.status}

    @staticmethod
    def work(case):
        n, w = case["n1"] * (2 if case["paired"] else 1), case["read_len"]
        return {"bytes": n * (36 + 2 * w + 28 + 36 + 36 + 2 * w + 60), "flops": 0}


class SortGather:
    def __init__(self, case, seed):
        pack = BamPack(case, seed)
        torch.cuda.synchronize()
        pack.run()
        torch.cuda.synchronize()
        self.n, self.meta, self.chunk = pack.b.n_seq, pack.meta, pack.bam
        self.size, self.cap = int(pack.status[0]), pack.cap
        self.chunks = torch.tensor([self.chunk.data_ptr()], dtype=torch.int64, device="cuda")
        self.chunk_len = torch.tensor([self.size], dtype=torch.int64, device="cuda")
        self.perm, self.is_dup = _zeros(self.n, torch.int32), _zeros(self.n, torch.int32)
        self.marked, self.status = _zeros(1, torch.int64), _zeros(2, torch.int64)
        self.out = _zeros(self.cap, torch.uint8)

    def run(self):
        ctx, stream, m = _context(), _stream().cuda_stream, _pointers(self.meta)
        check(lib.ma_sort_markdup_device(ctx.handle, self.n, m["coord"], m["dhi"], m["dlo"], m["score"], m["pair"], self.is_dup.data_ptr(), self.perm.data_ptr(), 1, None,
                                         self.marked.data_ptr(), stream), ctx.handle)
        check(lib.ma_gather_sorted_bam_device(ctx.handle, self.n, self.perm.data_ptr(), m["rec"], m["len"], self.is_dup.data_ptr(), 1, self.chunks.data_ptr(),
                                              self.chunk_len.data_ptr(), 1, self.out.data_ptr(), self.cap, self.status.data_ptr(), stream), ctx.handle)
        return {"perm": self.perm, "is_dup": self.is_dup, "marked": self.marked, "status": self.status, "stream": self.out}

    @staticmethod
    def work(case):
        n, w = case["n1"] * (2 if case["paired"] else 1), case["read_len"]
        # the keys, scores, pairs, places and sizes read, the order and flags
        # written, every record's bytes read and written
        return {"bytes": n * (24 + 8 + 12 + 8 + 2 * (36 + 36 + 4 + 15 + 1.5 * w)), "flops": 0}


class Bgzf:
    """The sorted record stream of a tile, as the BAM path hands it over."""

    def __init__(self, case, seed):
        self.level = case["level"]
        n1 = case["bytes"] // 550 + 1
        sort = SortGather({"n1": n1, "paired": True, "read_len": 150}, seed)
        torch.cuda.synchronize()
        sort.run()
        torch.cuda.synchronize()
        self.data = sort.out[: case["bytes"]].clone()
        self.cap = int(lib.ma_bgzf_bound(self.data.numel()))
        self.out = _zeros(self.cap, torch.uint8)

    def run(self):
        ctx, got = _context(), c_uint64(0)
        check(lib.ma_bgzf_compress_device(ctx.handle, self.data.data_ptr(), self.data.numel(), self.level, 1, self.out.data_ptr(), self.cap, byref(got),
                                          _stream().cuda_stream), ctx.handle)
        return {"file": self.out, "bytes": int(got.value)}

    @staticmethod
    def work(case):
        return {"bytes": case["bytes"] * (2.0 if case["level"] == 0 else 1.6), "flops": 0}


class Inflate:
    """The members that bgzip writes: 65280 bytes each, zlib at its default level."""

    def __init__(self, case, seed):
        g = _generator(seed)
        n = case["bytes"] // 340 + 1
        text = Fastq(g, Reads(g, n, False, 150)).text[: case["bytes"]].cpu().numpy()
        pieces = [text[a:a + 65280] for a in range(0, text.size, 65280)]

        def deflate(p):
            z = zlib.compressobj(6, zlib.DEFLATED, -15)
            data = z.compress(p.tobytes()) + z.flush()
            return data, zlib.crc32(p)

        with ThreadPoolExecutor(16) as pool:
            members = list(pool.map(deflate, pieces))
        raw, size = [], []
        for data, _ in members:  # 18 header bytes and 8 trailer bytes around each payload
            raw.append(b"\0" * 18 + data + b"\0" * 8)
            size.append(len(data))
        whole = np.array([len(r) for r in raw])
        put = lambda v, t: torch.from_numpy(np.asarray(v).astype(t)).cuda()  # noqa: E731
        self.data = torch.from_numpy(np.frombuffer(b"".join(raw), np.uint8).copy()).cuda()
        sizes = np.array([p.size for p in pieces])
        self.table = [put(np.cumsum(whole) - whole + 18, np.int64), put(size, np.int32), put(np.cumsum(sizes) - sizes, np.int64), put(sizes, np.int32),
                      put(np.array([c for _, c in members], np.uint32).view(np.int32), np.int32)]
        self.out, self.status = _zeros(text.size, torch.uint8), _zeros(len(pieces), torch.int32)

    def run(self):
        ctx = _context()
        check(lib.ma_bgzf_inflate_device(ctx.handle, self.data.data_ptr(), self.data.numel(), *[t.data_ptr() for t in self.table], self.status.numel(),
                                         self.out.data_ptr(), self.out.numel(), self.status.data_ptr(), _stream().cuda_stream), ctx.handle)
        return {"text": self.out, "status": self.status}

    @staticmethod
    def work(case):
        return {"bytes": case["bytes"] * 1.35, "flops": 0}


class FastqToBam:
    def __init__(self, case, seed):
        g = _generator(seed)
        self.ctx, self.index = _tuned(False), _index()
        f = Fastq(g, Reads(g, case["n1"], True, case["read_len"]))
        self.folder = tempfile.TemporaryDirectory()
        self.paths = [str(Path(self.folder.name) / p) for p in ("r1.fq", "r2.fq", "out.bam")]
        f.text[: f.first].cpu().numpy().tofile(self.paths[0])
        f.text[f.first:].cpu().numpy().tofile(self.paths[1])
        self.cap = 100_000 + 2 * case["n1"] * (160 + 2 * case["read_len"])

    def run(self):
        fq1, fq2, bam = self.paths
        mapped = map_fastq_to_bam(None, fq1, bam, fq2=fq2, bs_r1="C2T", bs_r2="G2A", params=BENCH_PARAMS, environ={}, ctx=self.ctx, index=self.index)
        size = os.path.getsize(bam)
        os.truncate(bam, self.cap)  # a length that does not depend on the reads, the rest of it zeros
        return {"mapped": int(mapped), "size": size, "file": np.memmap(bam, np.uint8, "r")}

    @staticmethod
    def work(case):
        w = case["read_len"]
        return {"bytes": 2 * case["n1"] * (58 + 2 * w + 0.6 * (91 + 1.5 * w)), "flops": 0}


KINDS = {"map_host": MapHost, "map_device": MapDevice, "serve": Serve, "fastq_split": FastqSplit, "bam_pack": BamPack, "sam_emit": SamEmit, "sort_gather": SortGather,
         "bgzf": Bgzf, "inflate": Inflate, "fastq_to_bam": FastqToBam}


def prepare(case, seed):
    state = KINDS[case["kind"]](case, seed)
    torch.cuda.synchronize()
    return state


def run(state):
    return state.run()


def work(case):
    return KINDS[case["kind"]].work(case)
