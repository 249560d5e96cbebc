"""Launches of many members, short ones among them or all of them short, where a
warp a member is quicker than a team: the bytes zlib gives back, the oracle's
error for a bad member among them, and no longer than the serial form takes."""

import struct
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _file(streams):
    """The streams back to back at odd distances, and their spans."""
    from fritillaria_gb300 import SPAN_DTYPE

    data, spans = bytearray(b"\x55" * 3), []
    for k, (payload, raw) in enumerate(streams):
        spans.append((len(data), len(data), len(payload), len(raw), zlib.crc32(raw)))
        data += payload + b"\xaa" * (8 + k % 5)
    return np.frombuffer(bytes(data), np.uint8), np.array(spans, dtype=SPAN_DTYPE)


def _deflate(raw, level=6, strategy=zlib.Z_DEFAULT_STRATEGY, mem=8):
    co = zlib.compressobj(level, zlib.DEFLATED, -15, mem, strategy)
    return co.compress(raw) + co.flush()


def _streams(n, rng):
    """Members of 0 to 4,000 bytes (n odd) or 500, one in 50 long (n even);
    text and runs, every level."""
    letters = np.frombuffer(b"ACGTNacgt\t\n0123456789", np.uint8)
    out = []
    for k in range(n):
        size = int(rng.integers(0, 4000 if n % 2 else 500)) if n % 2 or k % 50 else int(rng.integers(30_000, 65_537))
        raw = bytes(rng.choice(letters, size)) if k % 3 else bytes(letters[:7]) * (size // 7)
        out.append((_deflate(raw, int(rng.integers(0, 10))), raw))
    return out


@pytest.mark.parametrize("n", [1, 303, 305, 607, 608, 913, 2500, 2501, 5000, 5001])
def test_many_members_equal_zlib(gpu, n):
    """Counts around one, two, three and many members a CTA of a 152-SM grid."""
    streams = _streams(n, np.random.default_rng(n))
    data, spans = _file(streams)
    got, offs = gpu.CudaCodec(0).inflate_batch(data, spans)
    for i, (_, raw) in enumerate(streams):
        assert got[offs[i]:offs[i + 1]].tobytes() == raw, i


@pytest.mark.parametrize("bad", [0, 1500, 2999])
def test_a_bad_member_among_short_ones(gpu, bad):
    from oracle import oracle

    streams = [(_deflate(b"a%d" % k * 40), b"a%d" % k * 40) for k in range(3000)]
    payload, raw = streams[bad]
    streams[bad] = (payload[:-3], raw)
    data, spans = _file(streams)
    with pytest.raises(oracle.OracleError) as oe:
        oracle.inflate_batch(data, spans)
    with pytest.raises(gpu.FrtError) as ge:
        gpu.CudaCodec(0).inflate_batch_device(data, spans)
    assert (ge.value.code, ge.value.offset) == (oe.value.code, oe.value.offset)


@pytest.mark.parametrize("payload", [400, 1000])
def test_short_members_take_no_longer_than_serial(gpu, payload):
    """20,000 members and over, each a few records: the default took two to three
    times the serial form's time where every member had a team."""
    torch = pytest.importorskip("torch")
    from fritillaria_gb300 import synth

    raw, bgzf = synth.short_read_bam(20_000 * payload // 296, seed=9, member_payload=payload)
    dev = torch.from_numpy(bgzf).to("cuda")
    torch.cuda.synchronize()
    eng = gpu.BatchEngine(0)
    eng.bind_bam(dev.data_ptr(), dev.numel())
    team = eng.time_inflate(gpu.InflateTuning(0, 3, 0, 1), reps=5)[0]
    serial = eng.time_inflate(gpu.InflateTuning(1, 3, 0, 1), reps=5)[0]
    assert team < 1.3 * serial
    eng.run()
    assert eng.finish().status == 0 and np.array_equal(eng.inflated(), raw)


def _bam_of(members, count):
    """A BGZF file of a BAM header's member and `count` members, the given ones
    (payload, bytes) over and over; and its inflated bytes."""
    head = b"BAM\x01" + struct.pack("<II", 0, 1) + struct.pack("<I", 5) + b"chr1\0" + struct.pack("<I", 1 << 28)
    blocks = []
    for raw, d in [(head, _deflate(head))] + members:
        blocks.append(b"\x1f\x8b\x08\x04\0\0\0\0\0\xff\x06\0BC\x02\0" + struct.pack("<H", len(d) + 25) + d + struct.pack("<II", zlib.crc32(raw), len(raw)))
    turns = -(-count // len(members))
    return (np.frombuffer(blocks[0] + b"".join(blocks[1:] * turns), np.uint8),
            np.frombuffer(head + b"".join(m[0] for m in members) * turns, np.uint8))


def _engine(gpu, bgzf):
    torch = pytest.importorskip("torch")
    dev = torch.from_numpy(bgzf.copy()).to("cuda")
    torch.cuda.synchronize()
    eng = gpu.BatchEngine(0)
    eng.bind_bam(dev.data_ptr(), dev.numel())
    return eng, dev


def _short_reads(members, records=215):
    """That many members' worth of whole records."""
    from fritillaria_gb300 import synth

    raw, ends = synth.raw_bam("short_reads", members * records, 1, 1 << 28, 3)
    return [raw[int(ends[k]):int(ends[k + records])].tobytes() for k in range(0, members * records, records)]


@pytest.mark.parametrize("count,mem", [(700, 1), (1300, 2), (3000, 1), (3000, 2), (3000, 3), (3000, 8)])
def test_short_blocks_take_no_longer_than_serial(gpu, count, mem):
    """Members of 240 to 60 blocks (zlib's memLevel 1 to 3), two and ten a CTA:
    the default took up to 3.5 times the serial form's time."""
    bgzf, raw = _bam_of([(r, _deflate(r, mem=mem)) for r in _short_reads(20)], count)
    eng, _ = _engine(gpu, bgzf)
    team = eng.time_inflate(gpu.InflateTuning(0, 3, 0, 1), reps=5)[0]
    serial = eng.time_inflate(gpu.InflateTuning(1, 3, 0, 1), reps=5)[0]
    assert team < 1.3 * serial
    eng.run()
    assert eng.finish().status == 0 and np.array_equal(eng.inflated(), raw)


@pytest.mark.parametrize("n", [608, 1300, 4000])
def test_members_of_short_blocks_among_others(gpu, n):
    """Through the codec: members of short blocks, of long ones, and short ones;
    and one bad member of short blocks."""
    from oracle import oracle

    reads = _short_reads(8)
    kinds = [(_deflate(reads[k], mem=1 + 7 * (k % 2)), reads[k]) for k in range(8)] + [(_deflate(b"x" * 99), b"x" * 99)]
    streams = [kinds[k * k % 9] for k in range(n)]
    data, spans = _file(streams)
    got, offs = gpu.CudaCodec(0).inflate_batch(data, spans)
    for i, (_, raw) in enumerate(streams):
        assert got[offs[i]:offs[i + 1]].tobytes() == raw, i
    payload, raw = kinds[0]
    streams[n // 2] = (payload[:-9], raw)
    data, spans = _file(streams)
    with pytest.raises(oracle.OracleError) as oe:
        oracle.inflate_batch(data, spans)
    with pytest.raises(gpu.FrtError) as ge:
        gpu.CudaCodec(0).inflate_batch_device(data, spans)
    assert (ge.value.code, ge.value.offset) == (oe.value.code, oe.value.offset)


def _flushed(raw, every, level):
    """Blocks of `every` bytes, an empty stored block after each."""
    co = zlib.compressobj(level, zlib.DEFLATED, -15, 8)
    return b"".join(co.compress(raw[a:a + every]) + co.flush(zlib.Z_SYNC_FLUSH) for a in range(0, len(raw), every)) + co.flush()


@pytest.mark.parametrize("every", [1, 5, 40, 300, 1000, 7000, 20_000])
@pytest.mark.parametrize("n", [20, 1000])
def test_flushed_members_equal_zlib(gpu, every, n):
    """Short stored blocks and short coded ones in turn, each kind to a member."""
    raw = _short_reads(1)[0][:60_000 if every >= 300 else 200 * every + 17]
    kinds = [(_flushed(raw, every, level), raw) for level in (0, 1, 6)]
    streams = [kinds[k % 3] for k in range(n)]
    data, spans = _file(streams)
    got, offs = gpu.CudaCodec(0).inflate_batch(data, spans)
    for i in range(n):
        assert got[offs[i]:offs[i + 1]].tobytes() == raw, i


@pytest.mark.parametrize("every", [300, 1000, 3000])
def test_short_stored_blocks_take_no_longer_than_serial(gpu, every):
    """3,000 members of stored blocks: the default took up to six times the serial
    form's time."""
    bgzf, raw = _bam_of([(r, _flushed(r, every, 0)) for r in _short_reads(10, 200)], 3000)
    eng, _ = _engine(gpu, bgzf)
    team = eng.time_inflate(gpu.InflateTuning(0, 3, 0, 1), reps=5)[0]
    serial = eng.time_inflate(gpu.InflateTuning(1, 3, 0, 1), reps=5)[0]
    assert team < 1.3 * serial
    eng.run()
    assert eng.finish().status == 0 and np.array_equal(eng.inflated(), raw)


@pytest.mark.parametrize("cut", ["length", "end"])
def test_a_bad_stored_block_among_short_ones(gpu, cut):
    from oracle import oracle

    raw = _short_reads(1)[0][:40_000]
    good = _flushed(raw, 300, 0)
    for at in (310 * 5, 310 * 70, 310 * 120):  # a block of 300 bytes and an empty one take 310
        bad = good[:at] if cut == "end" else good[:at + 3] + bytes([good[at + 3] ^ 1]) + good[at + 4:]
        data, spans = _file([(good, raw), (bad, raw), (good, raw)])
        with pytest.raises(oracle.OracleError) as oe:
            oracle.inflate_batch(data, spans)
        with pytest.raises(gpu.FrtError) as ge:
            gpu.CudaCodec(0).inflate_batch_device(data, spans)
        assert (ge.value.code, ge.value.offset) == (oe.value.code, oe.value.offset), at


def test_short_payloads_of_long_members_stay_with_the_team(gpu):
    """3,000 members of 60 KB that a few hundred bytes hold: short to read, not to
    write, and the serial form's time is 1.9 times the team's."""
    raws = [struct.pack("<IiiBBHHHIiii", 60_000, 0, 5, 2, 9, 0, 0, 0, 0, -1, -1, 0) + b"q\0XXBC" + struct.pack("<I", 60_000 - 42) + bytes([k]) * (60_000 - 42)
            for k in range(10)]
    bgzf, raw = _bam_of([(r, _deflate(r)) for r in raws], 3000)
    eng, _ = _engine(gpu, bgzf)
    team = eng.time_inflate(gpu.InflateTuning(0, 3, 0, 1), reps=5)[0]
    assert team < 0.8 * eng.time_inflate(gpu.InflateTuning(1, 3, 0, 1), reps=5)[0]
    eng.run()
    assert eng.finish().status == 0 and np.array_equal(eng.inflated(), raw)
