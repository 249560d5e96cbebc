"""The calls a user of this library makes, with sizes, for timing them.

Each case is one public call path over seeded synthetic input of a shape the
library's own workloads have (short reads, ultra-long reads, BCF, FASTQ, FASTA,
VCF text): the per-member codec, the batch reader, the batched engine from
device and from host memory, several formats in one engine, region serving, the
scanners over a resident batch, the record-field calls and the compressor.
Every output is whole numbers and bytes.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import fritillaria_gb300 as frt
from fritillaria_gb300 import synth

GENOME = 3_100_000_000  # 24 contigs in the proportions of the human chromosomes

# Bytes per record (or per site, base) of the synthetic shapes: inflated,
# compressed at level 6, columns written.
SHORT = (296.3, 166.0, 113.0)
LONG_READ = (41_200.0, 26_800.0, 125.0)
BCF = (2068.0, 625.0, 53.0)
FASTQ = (367.0, 177.0, 28.0)
FASTA = (1.017, 0.34, 1.0)
VCF_SAMPLE = (4.0, 0.13, 12.0)  # per genotype: text, compressed, tab and call


def listed():
    return [
        # the first members of a file, for its header: the smallest call there is
        dict(name="inflate_head", kind="inflate", records=500, level=6),
        # the members behind one region of an index, as a viewer fetches them
        dict(name="inflate_region", kind="inflate", records=20_000, level=6),
        # a BAM written by htslib read batch by batch, the reader's own batch size
        dict(name="reader_bam", kind="reader", records=150_000, level=6, packing="record", blocks=256),
        # a panel or amplicon BAM resident on the device
        dict(name="engine_bam_small", kind="engine", records=100_000, level_a=6, level_b=6),
        # the largest: a lane of short reads, members of two compression levels
        dict(name="engine_bam_large", kind="engine", records=2_000_000, level_a=1, level_b=6),
        # the same from pinned host memory, upload inside the call
        dict(name="engine_host_bam", kind="host", records=500_000, level_a=1, level_b=6),
        # unaligned nanopore reads, records over many members
        dict(name="engine_ultra_long", kind="ultra_long", reads=4_000, extra=2, level=6),
        # a variant file, its reads and its reference in one bind
        dict(name="engine_mixed", kind="mixed", sites=60_000, samples=500, reads=400_000, bases=80_000_003),
        # region queries against a few indexed files, as a browser session asks them
        dict(name="serve_regions", kind="serve", files=3, records=150_000, requests=40),
        # a population panel's VCF: framing, fixed fields and every genotype
        dict(name="vcf_panel", kind="vcf", sites=2_000, samples=2_504),
        # fields of decoded records: one tag, CIGARs, bases, payloads
        dict(name="record_fields", kind="fields", records=400_000, level=1),
        # device bytes written back as BGZF
        dict(name="compress_bam", kind="compress", records=100_000, chunk=65_280),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["inflate", "reader", "engine", "host", "ultra_long", "mixed", "serve", "vcf", "fields",
                       "compress", "fastq", "fasta", "bcf"])
    if kind == "inflate":
        return dict(kind=kind, records=_log(rng, 100, 60_000), level=rng.choice([1, 6, 9]))
    if kind == "reader":
        return dict(kind=kind, records=_log(rng, 2_000, 200_000), level=rng.choice([1, 6]),
                    packing=rng.choice(["record", "full"]), blocks=rng.choice([64, 256, 1000]))
    if kind == "engine":
        return dict(kind=kind, records=_log(rng, 3_000, 1_000_000), level_a=rng.choice([1, 6]), level_b=6)
    if kind == "host":
        return dict(kind=kind, records=_log(rng, 10_000, 600_000), level_a=1, level_b=rng.choice([1, 6]))
    if kind == "ultra_long":
        return dict(kind=kind, reads=_log(rng, 50, 5_000), extra=rng.randint(0, 3), level=rng.choice([1, 6]))
    if kind == "mixed":
        return dict(kind=kind, sites=_log(rng, 500, 60_000), samples=rng.choice([1, 100, 500]),
                    reads=_log(rng, 3_000, 400_000), bases=_log(rng, 500_000, 80_000_000))
    if kind == "serve":
        return dict(kind=kind, files=rng.randint(1, 4), records=_log(rng, 20_000, 200_000),
                    requests=rng.randint(1, 60))
    if kind == "vcf":
        return dict(kind=kind, sites=_log(rng, 100, 3_000), samples=_log(rng, 1, 3_000))
    if kind == "fields":
        return dict(kind=kind, records=_log(rng, 1_000, 400_000), level=1)
    if kind == "compress":
        return dict(kind=kind, records=_log(rng, 200, 100_000), chunk=rng.choice([65_280, 65_505, 20_011]))
    if kind == "fastq":  # a resident FASTQ batch, boundary scan and columns
        return dict(kind=kind, reads=_log(rng, 1_000, 500_000), shape=rng.choice(["illumina", "ultra_long"]))
    if kind == "fasta":  # a resident reference, compacted
        return dict(kind=kind, bases=_log(rng, 100_000, 100_000_000), contigs=rng.randint(1, 40),
                    width=rng.choice([50, 60, 61, 80]))
    return dict(kind="bcf", sites=_log(rng, 300, 60_000), samples=rng.choice([1, 100, 500]))


# ---- device arrays ------------------------------------------------------------

class _Device:
    """Device memory a handle owns, as torch sees foreign arrays; keeps the owner."""

    def __init__(self, ptr, nbytes, width, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (nbytes // width,), "typestr": {1: "|u1", 2: "<i2", 4: "<i4", 8: "<i8"}[width],
                                         "data": (ptr, False), "version": 3}


class Views:
    """Tensors over a handle's device columns, made again where the column moved."""

    def __init__(self):
        self.known = {}

    def of(self, key, ptr, nbytes, width, owner):
        at = (ptr, nbytes)
        got = self.known.get(key)
        if got is None or got[0] != at:
            t = torch.as_tensor(_Device(ptr, nbytes, width, owner), device="cuda") if ptr and nbytes else torch.empty(0, dtype=torch.uint8, device="cuda")
            self.known[key] = got = (at, t)
        return got[1]


WIDTH = {np.dtype(np.uint8): 1, np.dtype(np.uint16): 2, np.dtype(np.int32): 4, np.dtype(np.uint32): 4, np.dtype(np.int64): 8, np.dtype(np.uint64): 8}


def _columns(handle, names, views=None, tag="", owner=None):
    """{column: tensor} of a batch or engine; `names` maps a column to (id,
    dtype), `owner` is what holds the handle's memory where that is another object."""
    views = views or Views()
    out = {}
    for name, (_, dtype) in names.items():
        p, nb, _ = handle.column_ptr(name)
        out[name] = views.of(tag + name, p, nb, WIDTH[np.dtype(dtype)], (handle, owner))
    return out


def _inflated(batch):
    return Views().of("data", batch.data_ptr(), batch.byte_len(), 1, batch)


BAM = dict(frt.BAM_COLUMNS)


def _bam_result(eng, views):
    out = _columns(eng, BAM, views)
    p, nb, _ = eng.column_ptr("aux_entries")
    out["aux_entries"] = views.of("aux_entries", p, nb, 4, eng)
    p, nb = eng.inflated_ptr()
    out["inflated"] = views.of("inflated", p, nb, 1, eng)
    return out


# ---- inputs ---------------------------------------------------------------------

def _bam(kind, records, seed, levels, packing="full", extra=0):
    """(raw, BGZF) of a BAM whose records are one fixed draw of the shape, in an
    order that starts at a record the seed picks: every seed gives other
    members and columns of the same lengths."""
    raw, ends = synth.raw_bam(kind, records, 24 if kind == "short_reads" else 1, GENOME, 20, extra)
    n = len(ends) - 1
    k = int(np.random.default_rng(seed).integers(0, n))
    head, cut, size = int(ends[0]), int(ends[k]), raw.size
    raw = np.concatenate([raw[:head], raw[cut:], raw[head:cut]])
    moved = np.concatenate([ends[:1], ends[k + 1:] - np.uint64(cut - head), ends[1:k + 1] + np.uint64(size - cut)])
    return raw, synth.bgzf(raw, packing, levels, moved)


def _to_device(data):
    return torch.from_numpy(np.ascontiguousarray(data)).to("cuda")


def _engine(bgzf, stream):
    dev = _to_device(bgzf)
    torch.cuda.synchronize()
    eng = frt.BatchEngine(0, stream=stream.cuda_stream)
    eng.bind_bam(dev.data_ptr(), dev.numel())
    return eng, dev


def _resident(bgzf, stream):
    codec = frt.CudaCodec(0, stream=stream.cuda_stream)
    spans, _ = frt.discover_blocks(bgzf)
    return codec, codec.inflate_batch_device(bgzf, spans)


def prepare(case, seed):
    kind = case["kind"]
    stream = torch.cuda.Stream()
    s = dict(kind=kind, stream=stream, views=Views())
    if kind == "inflate":
        _, bgzf = _bam("short_reads", case["records"], seed, (case["level"],) * 2)
        s["spans"], _ = frt.discover_blocks(bgzf)
        s["bgzf"] = bgzf
        s["codec"] = frt.CudaCodec(0, stream=stream.cuda_stream)
    elif kind == "reader":
        _, s["bgzf"] = _bam("short_reads", case["records"], seed, (case["level"],) * 2, case["packing"])
        s["codec"] = frt.CudaCodec(0, stream=stream.cuda_stream)
        s["decoder"] = frt.BamDecoder(0, stream=stream.cuda_stream)
        s["blocks"] = case["blocks"]
    elif kind in ("engine", "host"):
        _, bgzf = _bam("short_reads", case["records"], seed, (case["level_a"], case["level_b"]))
        s["eng"], s["dev"] = _engine(bgzf, stream)
        if kind == "host":
            s["pinned"] = torch.from_numpy(bgzf).pin_memory()
            s["host"] = s["pinned"].numpy()
    elif kind == "ultra_long":
        _, bgzf = _bam("ultra_long", case["reads"], seed, (case["level"],) * 2, extra=case["extra"])
        s["eng"], s["dev"] = _engine(bgzf, stream)
    elif kind == "mixed":
        parts = [(synth.bcf(case["sites"], case["samples"], seed=seed)[1], frt.Format.BCF),
                 (synth.fastq(case["reads"], seed=seed + 1)[1], frt.Format.FASTQ),
                 (synth.fasta(24, case["bases"], seed=seed + 2)[1], frt.Format.FASTA)]
        layout, at = [], 0
        for data, fmt in parts:
            layout.append((at, data.size, fmt))
            at += data.size
        s["dev"] = _to_device(np.concatenate([p[0] for p in parts]))
        torch.cuda.synchronize()
        s["eng"] = frt.BatchEngine(0, stream=stream.cuda_stream)
        s["eng"].bind_files(s["dev"].data_ptr(), s["dev"].numel(), layout)
    elif kind == "serve":
        s["server"] = frt.RegionServer(0)
        for f in range(case["files"]):
            raw, bgzf = synth.short_read_bam(case["records"], n_contigs=24, genome_len=GENOME, seed=seed * 16 + f, levels=(1, 6))
            s["server"].add_bam(bgzf, synth.bai(raw, bgzf))
        rng = np.random.default_rng(seed)
        s["room"] = case["requests"] * (200 + case["records"] * 15_000_000 // GENOME)  # a region holds a third more reads than its share at most
        s["queries"] = []
        for _ in range(case["requests"]):  # length log-uniform 1 kb to 10 Mb
            start = int(rng.integers(1, 100_000_000))
            s["queries"].append((int(rng.integers(0, case["files"])), int(rng.integers(0, 24)), start,
                                 start + int(np.exp(rng.uniform(np.log(1e3), np.log(1e7))))))
    elif kind == "vcf":
        raw, bgzf = synth.vcf_text(case["sites"], case["samples"], seed=seed)
        s["spans"], _ = frt.discover_blocks(bgzf)
        s["bgzf"] = bgzf
        s["codec"] = frt.CudaCodec(0, stream=stream.cuda_stream)
        s["scanner"] = frt.TextScanner(0, stream=stream.cuda_stream)
        s["vcf"] = frt.VcfDecoder(0, stream=stream.cuda_stream)
        s["vcf"].set_contigs([f"chr{k + 1}" for k in range(24)])
    elif kind == "fields":
        _, bgzf = _bam("short_reads", case["records"], seed, (case["level"],) * 2)
        s["eng"], s["dev"] = _engine(bgzf, stream)
        s["eng"].run()
        s["eng"].finish()
    elif kind == "compress":
        raw, _ = _bam("short_reads", case["records"], seed, (1, 1))
        s["dev"] = _to_device(raw)
        s["bounds"] = np.append(np.arange(0, raw.size, case["chunk"], dtype=np.uint64), np.uint64(raw.size))
        s["compressor"] = frt.DeviceCompressor(0, stream=stream.cuda_stream)
        s["pinned"] = torch.zeros(66_000 * len(s["bounds"]), dtype=torch.uint8).pin_memory()
        s["out"] = s["pinned"].numpy()
    elif kind == "fastq":
        _, bgzf = synth.fastq(case["reads"] if case["shape"] == "illumina" else max(1, case["reads"] // 100), case["shape"], seed=seed, levels=(1, 1))
        s["codec"], s["batch"] = _resident(bgzf, stream)
        s["scanner"] = frt.FastqScanner(0, stream=stream.cuda_stream)
    elif kind == "fasta":
        _, bgzf = synth.fasta(case["contigs"], case["bases"], case["width"], seed=seed, levels=(1, 1))
        s["codec"], s["batch"] = _resident(bgzf, stream)
        s["scanner"] = frt.FastaCompactor(0, stream=stream.cuda_stream)
    elif kind == "bcf":
        raw, bgzf = synth.bcf(case["sites"], case["samples"], seed=seed, levels=(1, 1))
        s["codec"], s["batch"] = _resident(bgzf, stream)
        s["scanner"] = frt.BcfScanner(0, stream=stream.cuda_stream)
        s["header"] = frt.parse_bcf_header(raw)
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return s


# ---- one pass ---------------------------------------------------------------------

def _run_reader(s):
    """Every column of a BAM read batch by batch, the columns of all batches joined."""
    reader = frt.DeviceBgzfReader(s["bgzf"], s["codec"], blocks_per_batch=s["blocks"])
    parts, first = {k: [] for k in BAM}, True
    for batch in reader:
        start = batch.start
        if first:
            start, n_ref = frt.parse_header(batch.data.to_host())
            s["decoder"].set_reference_count(n_ref)
            first = False
        records = s["decoder"].decode(batch.data, start)
        for name, col in _columns(records, BAM).items():
            parts[name].append(col)
        reader.carry_from(records.tail())
    return {k: torch.cat(v) for k, v in parts.items()}


def _run_serve(s):
    server = s["server"]
    ids = [server.submit(*q) for q in s["queries"]]
    server.drain()
    out = {name: np.zeros(s["room"], dtype) for name, (_, dtype) in frt.REGION_COLUMNS.items()}
    out["records"] = np.array([server.info(r).records for r in ids], np.int64)
    ends = np.cumsum(out["records"])
    for r, end, n in zip(ids, ends, out["records"]):
        for name in frt.REGION_COLUMNS:
            out[name][end - n:end] = server.column(r, name)
        server.release(r)
    # unsigned 64-bit values as the signed ones of the same bits
    return {k: v.view(np.int64) if v.dtype == np.uint64 else v.view(np.int32) if v.dtype == np.uint32 else v.astype(np.int32) if v.dtype == np.uint16 else v
            for k, v in out.items()}


def run(s):
    kind = s["kind"]
    with torch.cuda.stream(s["stream"]):
        if kind == "inflate":
            return _inflated(s["codec"].inflate_batch_device(s["bgzf"], s["spans"]))
        if kind == "reader":
            return _run_reader(s)
        if kind in ("engine", "ultra_long"):
            s["eng"].run()
            st = s["eng"].finish()
            return {"records": int(st.records), **_bam_result(s["eng"], s["views"])}
        if kind == "host":
            st = s["eng"].run_host(s["host"])
            return {"records": int(st.records), **_bam_result(s["eng"], s["views"])}
        if kind == "mixed":
            s["eng"].run()
            s["eng"].finish()
            names = (frt.BCF_COLUMNS, frt.FASTQ_COLUMNS, frt.FASTA_COLUMNS)
            return [_columns(s["eng"].file_result(i), cols, s["views"], str(i), s["eng"]) for i, cols in enumerate(names)]
        if kind == "serve":
            return _run_serve(s)
        if kind == "vcf":
            batch = s["codec"].inflate_batch_device(s["bgzf"], s["spans"])
            text = s["scanner"].scan(batch, 0, frt.Dialect.VCF)
            return [_columns(text, frt.TEXT_COLUMNS), _columns(s["vcf"].decode(text), frt.VCF_COLUMNS),
                    _columns(s["vcf"].genotypes(text), frt.VCF_GT_COLUMNS)]
        if kind == "fields":
            eng = s["eng"]
            return [_columns(b, b._cols, owner=eng) for b in (eng.aux_lookup("NM"), eng.cigar_resolved(), eng.unpack_sequences(), eng.compact())]
        if kind == "compress":
            got = s["compressor"].compress_batch_device(s["dev"].data_ptr(), s["dev"].numel(), s["bounds"], s["out"])
            return [s["pinned"], got.offsets.view(np.int64)]
        if kind == "fastq":
            return _columns(s["scanner"].decode(s["batch"], 0), frt.FASTQ_COLUMNS)
        if kind == "fasta":
            return _columns(s["scanner"].compact(s["batch"]), frt.FASTA_COLUMNS)
        start, samples, contigs = s["header"]
        return _columns(s["scanner"].decode(s["batch"], start, samples, contigs), frt.BCF_COLUMNS)


# ---- the work of one pass -----------------------------------------------------------

def work(case):
    """Bytes of one pass: the input read once, each output written once.  There
    is no floating-point work on these paths."""
    kind = case["kind"]
    if kind == "inflate":
        b = case["records"] * (SHORT[0] + SHORT[1])
    elif kind in ("reader", "engine", "host"):
        b = case["records"] * sum(SHORT)
    elif kind == "ultra_long":
        b = case["reads"] * sum(LONG_READ) + case["extra"] * 1.6 * 500_000
    elif kind == "mixed":
        b = (case["sites"] * (68 + 4 * case["samples"] + (20 + 1.2 * case["samples"]) + BCF[2]) + case["reads"] * sum(FASTQ)
             + case["bases"] * sum(FASTA))
    elif kind == "serve":  # a mean region of 1.1 Mb and two members of cover, both sides of the inflate
        per = case["records"] * 1.1e6 / GENOME + 440
        b = case["requests"] * per * (SHORT[0] + SHORT[1] + 31)
    elif kind == "vcf":
        b = case["sites"] * (100 * 1.2 + 159 + case["samples"] * sum(VCF_SAMPLE))
    elif kind == "fields":  # columns and payloads read, values, bases and payloads written
        b = case["records"] * (36 + 60 + 36 + 75 + 158 + 2 * 260 + 40)
    elif kind == "compress":
        b = case["records"] * (SHORT[0] + SHORT[1])
    elif kind == "fastq":
        b = case["reads"] * (FASTQ[0] + FASTQ[2])
    elif kind == "fasta":
        b = case["bases"] * (FASTA[0] + FASTA[2])
    else:
        b = case["sites"] * (68 + 4 * case["samples"] + BCF[2])
    return {"bytes": float(b), "flops": 0.0}
