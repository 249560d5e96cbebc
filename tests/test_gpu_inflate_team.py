"""The team form of the inflate (one CTA per member, every lane decoding) at the
sizes where it can go wrong: empty and one-byte members, a member of exactly
64 KiB, match lists past their room, blocks of a few bits and
of one segment, many blocks a member, second-level codes, stored runs between
coded blocks, and outputs at every alignment -- the bytes zlib gives back."""

import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _content(kind: str, n: int, rng) -> bytes:
    if kind == "zeros":
        return bytes(n)
    if kind == "period":  # distances shorter than a match, 1 to 40 bytes
        out = bytearray()
        while len(out) < n:
            unit = bytes(rng.integers(0, 256, int(rng.integers(1, 41)), dtype=np.uint8))
            out += unit * int(rng.integers(2, 30))
        return bytes(out[:n])
    if kind == "pairs":  # three-byte matches as dense as they come: the match list overflows
        words = [bytes(rng.integers(0, 256, 3, dtype=np.uint8)) for _ in range(300)]
        return b"".join(words[i] for i in rng.integers(0, 300, n // 3 + 1))[:n]
    if kind == "skewed":  # code lengths up to 15 bits: second-level tables
        p = 0.6 ** np.arange(60)
        return bytes(rng.choice(60, n, p=p / p.sum()).astype(np.uint8) * 4)
    if kind == "noise":
        return bytes(rng.integers(0, 256, n, dtype=np.uint8))
    half = n // 2  # "mixed": text, then noise (a stored block between coded ones)
    text = b"".join(b"chr%d\t%d\t%s\n" % (i % 23, i * 37, b"ACGT"[i % 4:i % 4 + 1] * (i % 9)) for i in range(half // 8 + 1))
    return text[:half] + bytes(rng.integers(0, 256, n - half, dtype=np.uint8))


SIZES = [0, 1, 2, 3, 15, 16, 17, 255, 4096, 12287, 12289, 32768, 65280, 65535, 65536]


def _file(streams):
    """The streams back to back at odd distances, and their spans."""
    from fritillaria_gb300 import SPAN_DTYPE

    data, spans = bytearray(b"\x55" * 5), []
    for k, (payload, raw) in enumerate(streams):
        spans.append((len(data), len(data), len(payload), len(raw), zlib.crc32(raw)))
        data += payload + b"\xaa" * (8 + k % 7)
    return np.frombuffer(bytes(data), np.uint8), np.array(spans, dtype=SPAN_DTYPE)


def _deflate(raw, level, strategy=zlib.Z_DEFAULT_STRATEGY, mem=8):
    co = zlib.compressobj(level, zlib.DEFLATED, -15, mem, strategy)
    return co.compress(raw) + co.flush()


@pytest.mark.parametrize("kind", ["zeros", "period", "pairs", "skewed", "noise", "mixed"])
def test_edges_equal_zlib(gpu, kind):
    rng = np.random.default_rng(len(kind))
    assert gpu.default_tuning().variant == 0
    streams = []
    for n in SIZES:
        raw = _content(kind, n, rng)
        for level, strategy, mem in ((1, 0, 8), (6, 0, 8), (9, 0, 1), (6, zlib.Z_HUFFMAN_ONLY, 8), (6, zlib.Z_FIXED, 9), (0, 0, 8)):
            streams.append((_deflate(raw, level, strategy, mem), raw))
    data, spans = _file(streams)
    got, offs = gpu.CudaCodec(0).inflate_batch(data, spans)
    for i, (_, raw) in enumerate(streams):
        assert got[offs[i]:offs[i + 1]].tobytes() == raw, (kind, i)


def test_a_payload_that_ends_with_a_block_header(gpu):
    """Two fixed blocks and the three bits of a third, the last of the payload:
    no symbol is left, and the member fails as the oracle's does."""
    from oracle import oracle

    for n in (6, 41, 3000):
        bits = []

        def code(value, width):  # Huffman codes go most significant bit first
            bits.extend((value >> i) & 1 for i in range(width - 1, -1, -1))

        for lits in (n, n % 5):
            bits += [0, 1, 0]  # not the last, fixed codes
            if lits == n:
                code(0x190 + 7, 9)
            for i in range(lits):
                code(0x30 + i * 7 % 144, 8)
            code(0, 7)
        bits += [0, 1, 0]
        assert len(bits) % 8 == 0
        payload = np.packbits(np.array(bits, np.uint8), bitorder="little").tobytes()
        data, spans = _file([(payload, bytes(n + n % 5 + 1))])
        with pytest.raises(oracle.OracleError) as oe:
            oracle.inflate_batch(data, spans)
        with pytest.raises(gpu.FrtError) as ge:
            gpu.CudaCodec(0).inflate_batch_device(data, spans)
        assert (ge.value.code, ge.value.offset) == (oe.value.code, oe.value.offset)


def test_a_tuning_with_a_spread_variant_keeps_the_team(gpu):
    """Fewer members than the team's grid has warps, under a tuning that names a
    serial spread variant: the bytes are zlib's, and the time of the launch is
    the team's (a serial chain takes ten times as long)."""
    torch = pytest.importorskip("torch")
    from fritillaria_gb300 import synth

    raw, bgzf = synth.short_read_bam(80_000, seed=5)
    dev = torch.from_numpy(bgzf).to("cuda")
    torch.cuda.synchronize()
    eng = gpu.BatchEngine(0)
    eng.bind_bam(dev.data_ptr(), dev.numel())
    alone = eng.time_inflate(gpu.InflateTuning(0, 3, 0, 1, spread_variant=-1))[0]
    assert eng.time_inflate(gpu.InflateTuning(0, 3, 0, 1, spread_variant=1))[0] < 3 * alone
    eng.set_tuning(gpu.InflateTuning(0, 3, 0, 1, spread_variant=1))
    eng.run()
    assert eng.finish().status == 0 and np.array_equal(eng.inflated(), raw)
